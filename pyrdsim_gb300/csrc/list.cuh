// list.cuh -- Verlet-list step kernels.
//
// At every rebuild k_nlist writes, for each particle in sorted order, the
// particles of the 3^D cells around its cell that lie within the list radius
// (range + 2 delta) and form a listed pair at that rebuild:
// interaction partners (types at the rebuild, pyrdsim.pyx:1448-1587) of
// another molecule, or bonded-list members of its own molecule (flagged with
// LIST_SAME_MOL: they count for reactions, not for pair forces).  The drift
// kernel's displacement check bounds every particle's motion since the
// rebuild by delta (Euclidean), so every pair that comes within range
// during the rebuild period is in the list, and each step kernel applies the
// same distance tests as the reference to the listed pairs only.
//
// Layout: ELL of width W, interleaved by TPP so that the TPP lanes serving
// one particle read consecutive words: entry e of particle i sits at
//   ((e / TPP) * npad + i) * TPP + e % TPP.
// A particle with more than W entries keeps its full count; the step kernels
// then regenerate its row from the cells, in the same order and on the same
// lanes as the list would have delivered it, so results do not depend on W.
//
// Step kernels run in two phases per CTA of LBLOCK threads and LBLOCK / TPP
// particles.  Phase A: TPP lanes per particle walk its list and combine with
// shuffles into shared memory.  Phase B: one thread per particle runs the
// per-particle tail (walls, bonded terms, Euler-Maruyama update; or the
// reaction draw).
//
// Neighbour staging (the period kernel).  A chunk's particles are neighbours in
// space, so their lists name the same few hundred particles over and over.
// k_nlist also writes, per chunk, the sorted indices of the particles in the
// runs its rows scan (stg_g: the touched part of every touched chunk, side by
// side) and every list row as 16-bit slot codes into that table (slot << 4,
// bit 0: same molecule), two codes per word, the word of a lane next to its
// neighbours'.  A step loads the staged particles once, coalesced, into shared
// memory as 16-byte records and walks the rows there, in list order and with
// the arithmetic of the gathers (the sums are the same bit for bit).  In small
// systems LPC lanes share what one lane would walk (period.cuh).  A row
// longer than the codes hold, or a chunk that touches more particles than fit,
// gathers from memory instead.
#pragma once

#include "kernels.cuh"

// resident CTAs per SM the step kernels are compiled for (register budget)
#ifndef RD_LIST_MIN_BLOCKS
#define RD_LIST_MIN_BLOCKS 8
#endif
// the same where every pair law is a single Lennard-Jones n = 6 law: more
// warps in flight are worth the registers there (wall fluid, 1,048,576
// particles, 40 steps: 5,220 us at 8 with the general walk; the walk of
// lj_walk 4,903 / 4,484 / 4,218 / 4,395 / 4,409 us at 8 / 10 / 12 / 14 / 16; the
// general walk at 7 / 8 / 9 / 10: ensemble of 64, 30 steps, 2,254 / 2,133 /
// 2,173 / 2,768 us, LJ fluid at 100,000, 60 steps, 1,120 / 1,125 / 1,179 / 1,405)
constexpr int LJ_MIN_BLOCKS = 12;
// list entries loaded per lane before their neighbours are gathered
#ifndef RD_LIST_BATCH
#define RD_LIST_BATCH 2
#endif

namespace rd {

constexpr int LBLOCK = BLOCK;                  // threads per CTA
constexpr int LIST_SAME_MOL = (int)0x80000000;

template <int TPP>
__device__ inline int ell_index(int e, int i, int npad) {
  return ((e / TPP) * npad + i) * TPP + (e % TPP);
}

__device__ inline void prefetch_l1(const void* p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

struct ListShared {
  SysDev sys;
  PairLaw laws[MAXI];
  WallLaw walls[MAXW];
  RxDev rx[MAXR];
};

// Run of particles number q (PER per run): computed for a single system,
// else from the chunk table.
template <int PER>
__device__ inline Chunk chunk_at(const Args& a, int q) {
  if (a.single) {
    Chunk c = a.chunk1;
    c.beg = q * PER;
    c.cnt = min(PER, a.n_total - c.beg);
    return c;
  }
  return a.chunks[q];
}

template <int PER>
__device__ inline Chunk chunk_of(const Args& a) {
  return chunk_at<PER>(a, (int)blockIdx.x);
}

// The chunk's system tables into shared memory: one round trip (all loads
// first, then the stores; the caller synchronises).
template <bool LAWS, bool WALLS, bool RX>
__device__ inline void list_tables(ListShared& sh, const Args& a, const Chunk& c) {
  constexpr int NS = (int)(sizeof(SysDev) / 4);
  constexpr int NL = LAWS ? MAXI * (int)(sizeof(PairLaw) / 4) : 0;
  constexpr int NW = WALLS ? MAXW * (int)(sizeof(WallLaw) / 4) : 0;
  constexpr int NR = RX ? MAXR * (int)(sizeof(RxDev) / 4) : 0;
  const int nl = c.nlaws * (int)(sizeof(PairLaw) / 4);
  const int nw = c.nwalls * (int)(sizeof(WallLaw) / 4);
  const int nr = c.nrx * (int)(sizeof(RxDev) / 4);
  WordLoad<NS> ls;
  WordLoad<NL> ll;
  WordLoad<NW> lw;
  WordLoad<NR> lr;
  ls.load(reinterpret_cast<const int*>(&a.sys[c.sys]), NS);
  if (LAWS) ll.load(reinterpret_cast<const int*>(a.laws + c.law0), nl);
  if (WALLS) lw.load(reinterpret_cast<const int*>(a.walls + c.wall0), nw);
  if (RX) lr.load(reinterpret_cast<const int*>(a.rx + c.rx0), nr);
  ls.store(reinterpret_cast<int*>(&sh.sys), NS);
  if (LAWS) ll.store(reinterpret_cast<int*>(sh.laws), nl);
  if (WALLS) lw.store(reinterpret_cast<int*>(sh.walls), nw);
  if (RX) lr.store(reinterpret_cast<int*>(sh.rx), nr);
}

// Prefetch into L1 the list words of this warp's particles: column block q
// (entries q*TPP .. q*TPP+TPP-1 of every particle of the warp) on lane q.
// Every lane of the warp calls it.
template <int TPP>
__device__ inline void prefetch_rows(const Args& a, const Chunk& ch, int cnt, bool active) {
  const int warp0 = ch.beg + ((int)(threadIdx.x & ~31u)) / TPP;
  const int wlast = min(warp0 + 32 / TPP, ch.beg + ch.cnt) - 1;
  const unsigned int mc = __reduce_max_sync(0xffffffffu, active ? (unsigned)min(cnt, a.W) : 0u);
  const int q = threadIdx.x & 31;
  if (wlast >= warp0 && q * TPP < (int)mc) {
    prefetch_l1(a.nbr + ell_index<TPP>(q * TPP, warp0, a.npad));
    prefetch_l1(a.nbr + ell_index<TPP>(q * TPP + TPP - 1, wlast, a.npad));
  }
}

// Cells of one row of particle cell c (offsets dy, dz): the cell index of
// x = 0 in that row and one or two runs of x cells [lo0, hi0], [lo1, hi1]
// (hi1 < lo1: none), in dx order.  False if the row lies outside a
// reflecting box.
template <int D>
__device__ inline bool row_runs(const SysDev& s, const int* c, int dy, int dz, int& row, int& lo0,
                                int& hi0, int& lo1, int& hi1) {
  const int nx = s.nc[0], cx = c[0];
  row = 0;
  if (D > 1) {
    int mult = nx;
#pragma unroll
    for (int k = 1; k < D; k++) {
      int ck = c[k] + (k == 1 ? dy : dz);
      if ((s.periodic >> k) & 1) {
        if (ck < 0) ck += s.nc[k];
        else if (ck >= s.nc[k]) ck -= s.nc[k];
      } else if (ck < 0 || ck >= s.nc[k]) {
        return false;
      }
      row += ck * mult;
      mult *= s.nc[k];
    }
  }
  lo1 = 0;
  hi1 = -1;
  if (s.halo[0] == 0) {
    lo0 = hi0 = cx;
  } else if (s.periodic & 1) {  // nx >= 3 here
    if (cx == 0) { lo0 = hi0 = nx - 1; lo1 = 0; hi1 = 1; }
    else if (cx == nx - 1) { lo0 = nx - 2; hi0 = nx - 1; lo1 = hi1 = 0; }
    else { lo0 = cx - 1; hi0 = cx + 1; }
  } else {
    lo0 = max(cx - 1, 0);
    hi0 = min(cx + 1, nx - 1);
  }
  return true;
}

// The list row of sorted particle i, generated from the cells and the
// positions at the last rebuild (xr).  Candidates are visited in a fixed
// order (rows of cells in dz, dy order; along x the adjacent cells form one
// or two contiguous runs of the sorted arrays, in dx order).  All run
// boundaries are loaded at once, then the L lanes enumerate the candidates
// of all runs together, L per round, two rounds per batch of loads.  Hits are
// numbered in candidate order and hit e is handed to lane e % L, which calls
// emit(e, entry).  Returns the number of entries.  The entry order does not
// depend on L.  All lanes of the group must call it together.
template <int D, int L, class Emit>
__device__ inline int row_scan(const SysDev& s, const Args& a, int i, int lane, Emit&& emit) {
  constexpr int NROW = D == 3 ? 9 : (D == 2 ? 3 : 1);
  constexpr int NRUN = 2 * NROW;
  constexpr int U = 2;
  const unsigned int gshift = (threadIdx.x & 31) & ~(L - 1);
  const unsigned int gmask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << gshift;
  uint32_t xi[3] = {0u, 0u, 0u};
  int c[3] = {0, 0, 0};
#pragma unroll
  for (int k = 0; k < D; k++) {
    xi[k] = a.xr[k][i];
    c[k] = cell_coord(s, k, xi[k]);
  }
  const uint32_t mi = a.meta[i];
  const int moli = a.mol[i];
  const int trbi = (mi >> 8) & 0xff, loci = (mi >> 16) & 0xff, tmi = mi >> 24;
  const unsigned int pmask = s.partner[trbi];
  const uint32_t bmask = tmi != 0xff ? a.tmpl[tmi].bondmask[loci] : 0u;
  const float Rl2 = s.Rl2;
  const int h1 = D > 1 ? s.halo[1] : 0;
  const int h2 = D > 2 ? s.halo[2] : 0;
  // runs [rb, re) of the sorted arrays, in candidate order
  int rb[NRUN], re[NRUN];
#pragma unroll
  for (int q = 0; q < NROW; q++) {
    const int dz = D == 3 ? q / 3 - 1 : 0;
    const int dy = D >= 2 ? q % 3 - 1 : 0;
    int row, lo0, hi0, lo1, hi1;
    const bool ok = dy >= -h1 && dy <= h1 && dz >= -h2 && dz <= h2 &&
                    row_runs<D>(s, c, dy, dz, row, lo0, hi0, lo1, hi1);
    const int* cs = a.cell_start + s.c0 + row;
    rb[2 * q] = ok ? cs[lo0] : 0;
    re[2 * q] = ok ? cs[hi0 + 1] : 0;
    const bool two = ok && hi1 >= lo1;
    rb[2 * q + 1] = two ? cs[lo1] : 0;
    re[2 * q + 1] = two ? cs[hi1 + 1] : 0;
  }
  int total = 0;
#pragma unroll
  for (int q = 0; q < NRUN; q++) total += re[q] - rb[q];
  int cnt = 0;
  for (int base = 0; base < total; base += U * L) {
    int jj[U];
    uint32_t xx[U][3], mj[U];
    int molj[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      // candidate t -> sorted index
      int off = base + u * L + lane, j = -1;
#pragma unroll
      for (int q = 0; q < NRUN; q++) {
        const int len = re[q] - rb[q];
        if (j < 0) {
          if (off < len) j = rb[q] + off;
          else off -= len;
        }
      }
      jj[u] = j;
      const int jl = j < 0 ? i : j;
#pragma unroll
      for (int k = 0; k < 3; k++) xx[u][k] = k < D ? a.xr[k][jl] : 0u;
      mj[u] = a.meta[jl];
      molj[u] = a.mol[jl];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (base + u * L >= total) break;  // uniform across the group
      const int j = jj[u];
      int ent = 0;
      bool hit = false;
      if (j >= 0 && j != i) {
        float r2 = 0.f;
#pragma unroll
        for (int k = 0; k < D; k++) {
          const float d = (float)(int)(xx[u][k] - xi[k]) * s.unit_hi[k];
          r2 += d * d;
        }
        if (r2 < Rl2) {
          if (molj[u] == moli) {
            hit = (bmask >> ((mj[u] >> 16) & 31)) & 1;
            ent = j | LIST_SAME_MOL;
          } else {
            hit = (pmask >> ((mj[u] >> 8) & 0xff)) & 1;
            ent = j;
          }
        }
      }
      const unsigned int m = (__ballot_sync(gmask, hit) & gmask) >> gshift;
      const int nh = __popc(m);
      const int r = (lane - cnt) & (L - 1);  // this lane takes hit cnt + r
      int src = lane;
      if (r < nh) {
        unsigned int mm = m;
        for (int q = 0; q < r; q++) mm &= mm - 1u;
        src = __ffs(mm) - 1;
      }
      const int v = __shfl_sync(gmask, ent, src, L);
      if (r < nh) emit(cnt + r, v);
      cnt += nh;
    }
  }
  return cnt;
}

// A list entry with the neighbour's current pair words and meta word.
struct Nb {
  uint32_t x[3];
  uint32_t m;
  int v;  // entry: sorted index | LIST_SAME_MOL
};

// PEND (period kernel): the neighbour's record of this step, waited for until
// it is written and its reaction draw resolved.
template <int D, bool PEND = false>
__device__ inline Nb gather(const Args& a, int v) {
  Nb n;
  const int j = v & 0x7fffffff;
  n.v = v;
  if (PEND) {
    const int st = period_n;
    uint4 r = get_rec(a, a.rec[st & 1] + j, REC_TAG, st);
    if (r.w & REC_PENDING) r = rec_wait(a, a.rec[st & 1] + j, REC_TAG, st, true);
    n.x[0] = r.x;
    n.x[1] = r.y;
    n.x[2] = r.z;
    n.m = r.w & 0xfu;
  } else {
#pragma unroll
    for (int k = 0; k < 3; k++) n.x[k] = k < D ? a.xp[k][j] : 0u;
    n.m = a.meta[j];
  }
  return n;
}

// Displacement of an entry from its pair words (the exact integer
// difference rounded once to float32, then scaled by the unit) and the
// squared distance.
template <int D>
__device__ inline float pair_geom(const SysDev& s, const uint32_t* xj, const uint32_t* xi,
                                  float* dx) {
  float r2 = 0.f;
#pragma unroll
  for (int k = 0; k < D; k++) {
    dx[k] = (float)(int)(xj[k] - xi[k]) * s.qf[k];
    r2 = fmaf(dx[k], dx[k], r2);
  }
  return r2;
}

// Visit the list entries of particle i on this lane (entries lane, lane +
// TPP, ...), from the list or, for an overflowing row, from the cells.  List
// rows are read RD_LIST_BATCH entries at a time: all index loads, then all
// neighbour loads, then the arithmetic.
template <int D, int TPP, bool PEND = false, class Fn>
__device__ inline void for_entries(const SysDev& s, const Args& a, int i, int lane, int cnt,
                                   Fn&& fn) {
  constexpr int B = RD_LIST_BATCH;
  if (cnt <= a.W) {
    for (int e0 = lane; e0 < cnt; e0 += B * TPP) {
      int v[B];
#pragma unroll
      for (int u = 0; u < B; u++) {
        const int e = e0 + u * TPP;
        v[u] = e < cnt ? a.nbr[ell_index<TPP>(e, i, a.npad)] : i;
      }
      Nb nb[B];
#pragma unroll
      for (int u = 0; u < B; u++) nb[u] = gather<D, PEND>(a, v[u]);
#pragma unroll
      for (int u = 0; u < B; u++)
        if (e0 + u * TPP < cnt) fn(nb[u]);
    }
  } else {
    row_scan<D, TPP>(s, a, i, lane, [&](int, int v) { fn(gather<D, PEND>(a, v)); });
  }
}

// Reaction prefilter of a step (sorted particle gi of type ti): the
// float64 total propensity of that step grows monotonically with every
// neighbour count, so rxA + rxB * cnt, with cnt the list entries that can come
// within a reaction radius before the next rebuild (within it plus twice the
// allowed displacement at the last one) and a relative margin far above the
// rounding of the reference's repeated additions, bounds it from above.  If dt times the bound does not exceed the step's u1 (the same
// counter-based draw the reaction kernel makes), the draw `dt * total > u1`
// (pyrdsim.pyx:2211-2213) cannot succeed and the particle keeps its type.
// The bound and the comparison are float32: rxAf, rxBf and dtf are rounded
// up, the relative margin 1e-5 covers the float32 rounding, and the uniform
// is replaced by the lower bound of its top 24 bits.  Returns true when the
// draw may succeed (pid: caller index, w0: the tag-0
// words of the next step).
template <int D>
__device__ inline bool rx_may_react(const SysDev& s, int ti, int cnt, int pid, long long step,
                                    const U4* w0) {
  if (!((s.rx_any_mask >> ti) & 1)) return false;
  uint32_t hi, lo;
  u1_words<D>(s.seed, step, pid, w0, hi, lo);
  float u1lo, u1hi;
  uniform_bounds(hi, u1lo, u1hi);
  const float ub = (s.rxAf[ti] + s.rxBf[ti] * (float)cnt) * (1.0f + 1e-5f);
  return s.dtf * ub > u1lo;
}

// The period kernel's records of sorted particle i before its first step: the
// state as step 0, "no step yet" for the other parity.
template <int D>
__device__ inline void first_records(const Args& a, int i, uint32_t mi, bool pending) {
  uint32_t p[3] = {0u, 0u, 0u}, l[3] = {0u, 0u, 0u}, h[3] = {0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < D; k++) {
    p[k] = a.xp[k][i];
    l[k] = a.xl[k][i];
    h[k] = a.xh[k][i];
  }
  const uint32_t ty = mi & 0xfu;
  a.rec[0][i] = make_uint4(p[0], p[1], p[2], rec_word(0, ty, ty, pending));
  a.recl[0][i] = make_uint4(l[0], l[1], l[2], 0u);
  a.rech[0][i] = make_uint4(h[0], h[1], h[2], 0u);
  a.rec[1][i].w = REC_NONE;
  a.recl[1][i].w = REC_NONE;
  a.rech[1][i].w = REC_NONE;
}

// The same for a launch of the period kernel that no list builder precedes.
template <int D>
__global__ void k_first_records(Args a) {
  pdl_wait();  // (no early launch of the period kernel: see F_PERIOD_FULL)
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n_total) first_records<D>(a, i, a.meta[i], false);
}

// Rebuild: every particle's list row and entry count.  With F_RX_HERE one thread
// per particle also runs the reaction prefilter of its step with the fresh
// counts, and with F_PERIOD_PREP it writes the period kernel's records of its
// particle: of step 0 (candidates of the rebuild step marked pending), and "no
// step yet" for the other parity.  Chunks' staging tables and slot codes: see
// the top of this file.
// Position, in 16-bit codes, of entry e of particle p of a chunk: chain e % TPP of
// its row is shared by LPC lanes, which take its entries in turn.
template <int TPP, int LPC>
__device__ inline int code_at(int p, int e) {
  const int k = e / TPP, m = k / LPC;
  return (((m >> 1) * LBLOCK) + (p * TPP + e % TPP) * LPC + k % LPC) * 2 + (m & 1);
}

constexpr int STG_HASH = 128;  // touched chunks of a chunk (open addressing)

struct StageHash {
  int key[STG_HASH], lo[STG_HASH], hi[STG_HASH], off[STG_HASH];
  int total, on;
};

// Two forms.  k_nlist: NT threads per particle (3 in 2D, one per row of cells)
// scan their rows' runs in candidate order, four candidates per batch of loads,
// into shared-memory buffers; the buffers are then concatenated in row order (the
// order row_scan uses).  A thread whose rows hold more than BCAP listed pairs
// scans again to write the rest.  k_nlist_lanes: 16 lanes per particle walk one
// run after the other, 16 consecutive candidates at a time; hits are numbered by
// ballots and written where they belong; lane q finds the run bounds of row q of
// cells for the others.  The rows are the same.  The lanes form is the faster one
// where rows of cells hold many candidates (in 3D the thread with a particle's
// own row outgrows its buffer: 107 us with threads, 55 with lanes at 13,824
// particles) and where few particles leave threads to spare (11.2 -> 9.2 us at
// 1,024); its set-up, done by 16 lanes for 3 rows, loses in large 2D systems (21 /
// 43 us at 65,536, 127 / 409 at 1,048,576).
__host__ __device__ constexpr bool nlist_by_lanes(int D, int lpc) { return D == 3 || lpc == 4; }
constexpr int NL_LANES = 16;
// Threads per CTA (chunks of `per` particles).
__host__ __device__ constexpr int nlist_threads(int D, int per) { return per * (D == 1 ? 1 : 3); }
__host__ __device__ constexpr int nlist_lane_threads(int per) {
  return per * NL_LANES < 512 ? per * NL_LANES : 512;
}

// LPC: see period.cuh (the period kernel's lanes per chain of a row; its chunks
// are this kernel's).
template <int D, int TPP, int LPC>
__global__ void __launch_bounds__(nlist_threads(D, LBLOCK / TPP / LPC)) k_nlist(Args a) {
  constexpr int PER = LBLOCK / TPP / LPC;
  static_assert(D < 3, "the lanes form builds rows in 3D");
  constexpr int NT = D == 1 ? 1 : 3;  // threads per particle, a row of cells each
  constexpr int NTH = PER * NT;
  constexpr int NRUN = 2;
  constexpr int U = 4;
  constexpr int BCAP = 24;
  __shared__ SysDev sys;
  __shared__ int sbuf[NTH][BCAP];
  __shared__ int2 scnt[NTH];
  __shared__ StageHash sth;
  if (!(a.flags & F_PERIOD_FULL)) pdl_trigger();
  const Chunk ch = chunk_at<PER>(a, (int)blockIdx.x);
  {
    constexpr int NS = (int)(sizeof(SysDev) / 4);
    WordLoad<NS, NTH> ls;
    ls.load(reinterpret_cast<const int*>(&a.sys[ch.sys]), NS);
    ls.store(reinterpret_cast<int*>(&sys), NS);
  }
  const bool prep = (a.flags & F_PERIOD_PREP) != 0;
  const bool stage = a.codes != nullptr;
  if (stage) {
    for (int q = (int)threadIdx.x; q < STG_HASH; q += NTH) {
      sth.key[q] = 0;
      sth.lo[q] = 0x7fffffff;
      sth.hi[q] = -1;
    }
    if (threadIdx.x == 0) {
      sth.total = 0;
      sth.on = 1;
    }
  }
  pdl_wait();
  __syncthreads();
  const SysDev& s = sys;
  const int tid = (int)threadIdx.x, pp = tid / NT, t = tid % NT;
  const bool valid = pp < ch.cnt;
  const int i = ch.beg + (valid ? pp : 0);
  uint32_t xi[3] = {0u, 0u, 0u};
  int c[3] = {0, 0, 0};
#pragma unroll
  for (int k = 0; k < D; k++) {
    xi[k] = a.xr[k][i];
    c[k] = cell_coord(s, k, xi[k]);
  }
  const uint32_t mi = a.meta[i];
  const int moli = a.mol[i];
  const int trbi = (mi >> 8) & 0xff, loci = (mi >> 16) & 0xff, tmi = mi >> 24;
  const unsigned int pmask = s.partner[trbi];
  const uint32_t bmask = tmi != 0xff ? a.tmpl[tmi].bondmask[loci] : 0u;
  const float Rl2 = s.Rl2;
  const int h1 = D > 1 ? s.halo[1] : 0;
  int rb[NRUN], re[NRUN];
  {
    const int dy = D == 2 ? t - 1 : 0;
    int row, lo0, hi0, lo1, hi1;
    const bool ok = valid && dy >= -h1 && dy <= h1 && row_runs<D>(s, c, dy, 0, row, lo0, hi0, lo1, hi1);
    const int* cs = a.cell_start + s.c0 + row;
    rb[0] = ok ? cs[lo0] : 0;
    re[0] = ok ? cs[hi0 + 1] : 0;
    const bool two = ok && hi1 >= lo1;
    rb[1] = two ? cs[lo1] : 0;
    re[1] = two ? cs[hi1 + 1] : 0;
  }
  // the listed pairs of this thread's rows, in candidate order: emit(k, entry,
  // squared distance)
  auto scan_rows = [&](auto&& emit) {
    int k = 0;
#pragma unroll
    for (int q = 0; q < NRUN; q++) {
      for (int j0 = rb[q]; j0 < re[q]; j0 += U) {
        uint32_t xx[U][3], mj[U];
        int molj[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int jl = j0 + u < re[q] ? j0 + u : i;
#pragma unroll
          for (int d = 0; d < 3; d++) xx[u][d] = d < D ? a.xr[d][jl] : 0u;
          mj[u] = a.meta[jl];
          molj[u] = a.mol[jl];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int j = j0 + u;
          if (j >= re[q] || j == i) continue;
          float r2 = 0.f;
#pragma unroll
          for (int d = 0; d < D; d++) {
            const float dd = (float)(int)(xx[u][d] - xi[d]) * s.unit_hi[d];
            r2 += dd * dd;
          }
          if (!(r2 < Rl2)) continue;
          bool hit;
          int ent;
          if (molj[u] == moli) {
            hit = (bmask >> ((mj[u] >> 16) & 31)) & 1;
            ent = j | LIST_SAME_MOL;
          } else {
            hit = (pmask >> ((mj[u] >> 8) & 0xff)) & 1;
            ent = j;
          }
          if (hit) emit(k++, ent, r2);
        }
      }
    }
    return k;
  };
  // slot of chunk key - 1 (of this system) in the hash, -1 if absent
  auto find = [&](int key, bool insert) {
    for (int q = 0, h = key & (STG_HASH - 1); q < STG_HASH; q++, h = (h + 1) & (STG_HASH - 1)) {
      const int k = insert ? atomicCAS(&sth.key[h], 0, key) : sth.key[h];
      if (k == key || (insert && k == 0)) return h;
      if (k == 0) return -1;
    }
    return -1;
  };
  if (stage && valid) {
    // the runs of the first particle of each cell: those of the others too
    bool first = pp == 0;
    if (!first) {
#pragma unroll
      for (int k = 0; k < D; k++) first = first || cell_coord(s, k, a.xr[k][i - 1]) != c[k];
    }
    if (first) {
#pragma unroll
      for (int q = 0; q < NRUN; q++)
        for (int b = rb[q]; b < re[q];) {
          const int cc = (b - s.p0) / PER, e = min(re[q], s.p0 + (cc + 1) * PER);
          const int h = find(cc + 1, true);
          if (h < 0) {
            sth.on = 0;
          } else {
            atomicMin(&sth.lo[h], b);
            atomicMax(&sth.hi[h], e - 1);
          }
          b = e;
        }
    }
  }
  int rcnt = 0;
  const int cnt = scan_rows([&](int k, int ent, float r2) {
    if (k < BCAP) sbuf[tid][k] = ent;
    rcnt += r2 < s.Rrl2 ? 1 : 0;
  });
  scnt[tid] = make_int2(cnt, rcnt);
  __syncthreads();
  int off = 0, total = 0, rtotal = 0;
#pragma unroll
  for (int u = 0; u < NT; u++) {
    const int2 cu = scnt[pp * NT + u];
    if (u < t) off += cu.x;
    total += cu.x;
    rtotal += cu.y;
  }
  if (stage) {
    // table positions, in whatever order the counter hands them out
    for (int q = tid; q < STG_HASH; q += NTH)
      if (sth.key[q]) {
        const int len = sth.hi[q] - sth.lo[q] + 1;
        sth.off[q] = atomicAdd(&sth.total, len) - sth.lo[q];
      }
    __syncthreads();
    const bool on = sth.on && sth.total <= a.stg_max;
    if (tid == 0) a.stg_n[blockIdx.x] = on ? sth.total : -1;
    if (on) {
      int* g = a.stg_g + (size_t)blockIdx.x * a.stg_max;
      for (int q = tid / 16; q < STG_HASH; q += NTH / 16)
        if (sth.key[q])
          for (int j = sth.lo[q] + tid % 16; j <= sth.hi[q]; j += 16) g[sth.off[q] + j] = j;
    }
  }
  // the slot code of entry e of this particle
  unsigned short* codes = reinterpret_cast<unsigned short*>(a.codes) +
                          (size_t)blockIdx.x * a.kw * LBLOCK * 2;
  const bool coded = stage && total <= a.kw * 2 * TPP * LPC;
  int lastc = -1, lasto = 0;
  auto put_code = [&](int e, int ent) {
    if (!coded) return;
    const int j = ent & 0x7fffffff, cc = (j - s.p0) / PER;
    if (cc != lastc) {
      const int h = find(cc + 1, false);
      lastc = cc;
      lasto = h >= 0 ? sth.off[h] : 0;
    }
    codes[code_at<TPP, LPC>(pp, e)] = (unsigned short)(((j + lasto) << 4) | (ent < 0 ? 1 : 0));
  };
  int4 rec = make_int4(0, 0, 0, 0);
  bool listed = false;
  if (valid) {
    int* nbr = a.nbr_out;
    const int W = a.W, npad = a.npad;
    const int nb = min(cnt, BCAP);
    for (int k = 0; k < nb; k++)
      if (off + k < W) {
        nbr[ell_index<TPP>(off + k, i, npad)] = sbuf[tid][k];
        put_code(off + k, sbuf[tid][k]);
      }
    if (cnt > BCAP && off + BCAP < W)
      scan_rows([&](int k, int ent, float) {
        if (k >= BCAP && off + k < W) {
          nbr[ell_index<TPP>(off + k, i, npad)] = ent;
          put_code(off + k, ent);
        }
      });
    if (t == 0) {
      a.ncnt_out[i] = total;
      a.rcnt_out[i] = rtotal;
      if (a.flags & F_RX_HERE) {  // reaction prefilter of this step (see rx_may_react)
        rec = make_int4(i, (int)mi, total, a.pid[i]);
        listed = rx_may_react<D>(s, (int)(mi & 0xff), rtotal, rec.w, eff_step(a), nullptr);
        a.meta_out[i] = mi;
      }
      if (prep) first_records<D>(a, i, mi, listed);
    }
  }
  if (a.flags & F_RX_HERE) {  // the candidate list of the per-step kernels
    const unsigned int bal = __ballot_sync(0xffffffffu, listed);
    if (bal) {
      const int l32 = threadIdx.x & 31, leader = __ffs(bal) - 1;
      const int p = rx_slot(eff_step(a));
      int base = 0;
      if (l32 == leader) base = atomicAdd(a.rx_count + p, __popc(bal));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (listed) a.rx_list[(size_t)p * a.npad + base + __popc(bal & ((1u << l32) - 1u))] = rec;
    }
  }
}

template <int D, int TPP, int LPC>
__global__ void __launch_bounds__(nlist_lane_threads(LBLOCK / TPP / LPC)) k_nlist_lanes(Args a) {
  constexpr int PER = LBLOCK / TPP / LPC;
  constexpr int NTH = nlist_lane_threads(PER), NPASS = PER * NL_LANES / NTH;
  constexpr int NROW = D == 3 ? 9 : (D == 2 ? 3 : 1);
  static_assert(NROW <= NL_LANES, "a lane per row of cells");
  __shared__ SysDev sys;
  __shared__ StageHash sth;
  __shared__ int2 scnt[PER];  // entries, and those within the reactions' reach
  if (!(a.flags & F_PERIOD_FULL)) pdl_trigger();
  const Chunk ch = chunk_at<PER>(a, (int)blockIdx.x);
  {
    constexpr int NS = (int)(sizeof(SysDev) / 4);
    WordLoad<NS, NTH> ls;
    ls.load(reinterpret_cast<const int*>(&a.sys[ch.sys]), NS);
    ls.store(reinterpret_cast<int*>(&sys), NS);
  }
  const bool prep = (a.flags & F_PERIOD_PREP) != 0;
  const bool stage = a.codes != nullptr;
  const int tid = (int)threadIdx.x, l32 = tid & 31, sub = tid % NL_LANES;
  if (stage) {
    for (int q = tid; q < STG_HASH; q += NTH) {
      sth.key[q] = 0;
      sth.lo[q] = 0x7fffffff;
      sth.hi[q] = -1;
    }
    if (tid == 0) {
      sth.total = 0;
      sth.on = 1;
    }
  }
  pdl_wait();
  __syncthreads();
  const SysDev& s = sys;
  // slot of chunk key - 1 (of this system) in the hash, -1 if absent
  auto find = [&](int key, bool insert) {
    for (int q = 0, h = key & (STG_HASH - 1); q < STG_HASH; q++, h = (h + 1) & (STG_HASH - 1)) {
      const int k = insert ? atomicCAS(&sth.key[h], 0, key) : sth.key[h];
      if (k == key || (insert && k == 0)) return h;
      if (k == 0) return -1;
    }
    return -1;
  };
  // the runs of row `sub` of the cells around the particle of each pass
  int rb[NPASS][2], re[NPASS][2];
#pragma unroll
  for (int ps = 0; ps < NPASS; ps++) {
    const int pp = ps * (NTH / NL_LANES) + tid / NL_LANES;
    const bool valid = pp < ch.cnt;
    const int i = ch.beg + (valid ? pp : 0);
    int c[3] = {0, 0, 0};
    bool first = pp == 0;
#pragma unroll
    for (int k = 0; k < D; k++) {
      c[k] = cell_coord(s, k, a.xr[k][i]);
      if (pp > 0 && valid) first = first || cell_coord(s, k, a.xr[k][i - 1]) != c[k];
    }
    const int dz = D == 3 ? sub / 3 - 1 : 0, dy = D >= 2 ? sub % 3 - 1 : 0;
    const int h1 = D > 1 ? s.halo[1] : 0, h2 = D > 2 ? s.halo[2] : 0;
    int row = 0, lo0 = 0, hi0 = 0, lo1 = 0, hi1 = 0;
    const bool ok = valid && sub < NROW && dy >= -h1 && dy <= h1 && dz >= -h2 && dz <= h2 &&
                    row_runs<D>(s, c, dy, dz, row, lo0, hi0, lo1, hi1);
    const int* cs = a.cell_start + s.c0 + row;
    const bool two = ok && hi1 >= lo1;
    rb[ps][0] = ok ? cs[lo0] : 0;
    re[ps][0] = ok ? cs[hi0 + 1] : 0;
    rb[ps][1] = two ? cs[lo1] : 0;
    re[ps][1] = two ? cs[hi1 + 1] : 0;
    // the chunks they touch (the runs of the first particle of each cell are
    // those of the others too)
    if (stage && valid && first)
#pragma unroll
      for (int q = 0; q < 2; q++)
        for (int b = rb[ps][q]; b < re[ps][q];) {
          const int cc = (b - s.p0) / PER, e = min(re[ps][q], s.p0 + (cc + 1) * PER);
          const int h = find(cc + 1, true);
          if (h < 0) {
            sth.on = 0;
          } else {
            atomicMin(&sth.lo[h], b);
            atomicMax(&sth.hi[h], e - 1);
          }
          b = e;
        }
  }
  bool staged = false;
  if (stage) {
    __syncthreads();
    // table positions, in whatever order the counter hands them out
    for (int q = tid; q < STG_HASH; q += NTH)
      if (sth.key[q]) {
        const int len = sth.hi[q] - sth.lo[q] + 1;
        sth.off[q] = atomicAdd(&sth.total, len) - sth.lo[q];
      }
    __syncthreads();
    staged = sth.on && sth.total <= a.stg_max;
    if (tid == 0) a.stg_n[blockIdx.x] = staged ? sth.total : -1;
    if (staged) {
      int* g = a.stg_g + (size_t)blockIdx.x * a.stg_max;
      for (int q = tid / 16; q < STG_HASH; q += NTH / 16)
        if (sth.key[q])
          for (int j = sth.lo[q] + tid % 16; j <= sth.hi[q]; j += 16) g[sth.off[q] + j] = j;
    }
  }
  unsigned short* codes = reinterpret_cast<unsigned short*>(a.codes) +
                          (size_t)blockIdx.x * a.kw * LBLOCK * 2;
  const int coded = staged ? min(a.W, a.kw * 2 * TPP * LPC) : 0;  // entries with a code
  const float Rl2 = s.Rl2, Rrl2 = s.Rrl2;
  const unsigned int below = (1u << sub) - 1u;
  const int shift = l32 & ~(NL_LANES - 1);
#pragma unroll
  for (int ps = 0; ps < NPASS; ps++) {
    const int pp = ps * (NTH / NL_LANES) + tid / NL_LANES;
    const bool valid = pp < ch.cnt;
    const int i = ch.beg + (valid ? pp : 0);
    uint32_t xi[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < D; k++) xi[k] = a.xr[k][i];
    const uint32_t mi = a.meta[i];
    const int moli = a.mol[i];
    const int trbi = (mi >> 8) & 0xff, loci = (mi >> 16) & 0xff, tmi = mi >> 24;
    const unsigned int pmask = s.partner[trbi];
    const uint32_t bmask = tmi != 0xff ? a.tmpl[tmi].bondmask[loci] : 0u;
    int cnt = 0, rcnt = 0, lastc = -1, lasto = 0;
#pragma unroll 1
    for (int q = 0; q < 2 * NROW; q++) {
      const int b = __shfl_sync(0xffffffffu, (q & 1) ? rb[ps][1] : rb[ps][0], q >> 1, NL_LANES);
      const int e = __shfl_sync(0xffffffffu, (q & 1) ? re[ps][1] : re[ps][0], q >> 1, NL_LANES);
      // (the particles of a warp go round together)
      const int most = __reduce_max_sync(0xffffffffu, max(e - b, 0));
      for (int t = sub; t < most + sub; t += NL_LANES) {
        const int j = b + t;
        const bool in = j < e;
        const int jl = in ? j : i;
        uint32_t xj[3] = {0u, 0u, 0u};
#pragma unroll
        for (int d = 0; d < D; d++) xj[d] = a.xr[d][jl];
        const uint32_t mj = a.meta[jl];
        const bool own = a.mol[jl] == moli;
        float r2 = 0.f;
#pragma unroll
        for (int d = 0; d < D; d++) {
          const float dd = (float)(int)(xj[d] - xi[d]) * s.unit_hi[d];
          r2 += dd * dd;
        }
        const bool hit = in && j != i && r2 < Rl2 &&
                         ((own ? bmask >> ((mj >> 16) & 31) : pmask >> ((mj >> 8) & 0xff)) & 1u);
        const unsigned int m = (__ballot_sync(0xffffffffu, hit) >> shift) & ((1u << NL_LANES) - 1u);
        const unsigned int mr = (__ballot_sync(0xffffffffu, hit && r2 < Rrl2) >> shift) &
                                ((1u << NL_LANES) - 1u);
        if (hit) {
          const int k = cnt + __popc(m & below);
          if (k < a.W) a.nbr_out[ell_index<TPP>(k, i, a.npad)] = own ? (j | LIST_SAME_MOL) : j;
          if (k < coded) {
            const int cc = (j - s.p0) / PER;
            if (cc != lastc) {
              lastc = cc;
              lasto = sth.off[find(cc + 1, false)];
            }
            codes[code_at<TPP, LPC>(pp, k)] = (unsigned short)(((j + lasto) << 4) | (own ? 1 : 0));
          }
        }
        cnt += __popc(m);
        rcnt += __popc(mr);
      }
    }
    if (valid && sub == 0) scnt[pp] = make_int2(cnt, rcnt);
  }
  __syncthreads();
  if (tid >= (PER + 31) / 32 * 32) return;
  int4 rec = make_int4(0, 0, 0, 0);
  bool listed = false;
  if (tid < ch.cnt) {
    const int i = ch.beg + tid;
    const uint32_t mi = a.meta[i];
    const int2 n = scnt[tid];
    a.ncnt_out[i] = n.x;
    a.rcnt_out[i] = n.y;
    if (a.flags & F_RX_HERE) {  // reaction prefilter of this step (see rx_may_react)
      rec = make_int4(i, (int)mi, n.x, a.pid[i]);
      listed = rx_may_react<D>(s, (int)(mi & 0xff), n.y, rec.w, eff_step(a), nullptr);
      a.meta_out[i] = mi;
    }
    if (prep) first_records<D>(a, i, mi, listed);
  }
  if (a.flags & F_RX_HERE) {  // the candidate list of the per-step kernels
    const unsigned int bal = __ballot_sync(0xffffffffu, listed);
    if (bal) {
      const int leader = __ffs(bal) - 1;
      const int p = rx_slot(eff_step(a));
      int base = 0;
      if (l32 == leader) base = atomicAdd(a.rx_count + p, __popc(bal));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (listed) a.rx_list[(size_t)p * a.npad + base + __popc(bal & ((1u << l32) - 1u))] = rec;
    }
  }
}

// Adds one listed partner (type tj before the step's reactions, pair words xj,
// sorted index j()) of particle m (type tm, pair words xm) to the counts of the
// neighbour-dependent reactions whose radius it is within.
template <int D, class J>
__device__ inline void count_partner(const SysDev& s, const RxDev* rx, const Args& a, int m, J&& j,
                                     int tm, int tj, const uint32_t* xm, const uint32_t* xj,
                                     uint32_t* cw) {
  float d[3];
  const float r2 = pair_geom<D>(s, xj, xm, d);
  if (!(r2 < s.Rrx2)) return;
  const unsigned int rmask = s.rxmatch[tm * MAXT + tj];
  double dexact = -1.0;
  for (unsigned int b = rmask; b; b &= b - 1u) {
    const int r = __ffs(b) - 1;
    const RxDev& R = rx[r];
    bool inside;
    if (r2 < R.r02_lo) inside = true;
    else if (r2 > R.r02_hi) inside = false;
    else {
      if (dexact < 0) dexact = exact_dist<D>(s, a, m, j());
      inside = dexact < R.r0;
    }
    if (inside) cw[r >> 1] += 1u << (16 * (r & 1));
  }
}

// One listed particle's reaction draw at the kernel's step, by a whole warp
// (pyrdsim.pyx:2070-2223): the lanes count, for every neighbour-dependent
// reaction, its listed partners of the right type within r0 (types before
// this step's reactions, positions of this step), and lane 0 forms the
// propensities and draws.  rec = {sorted index, meta, list entries, pid}.
// Returns the new type on lane 0.
template <int D, int TPP>
__device__ inline int resolve_listed(const SysDev& s, const RxDev* rx, const Args& a, int4 rec,
                                     int lane) {
  const int m = rec.x, cnt = rec.z, pid = rec.w;
  // lane 0's counter-based words of the draw (2D: u1 from the tag-0 words),
  // computed while the neighbour loads below are in flight
  U4 w0 = {0u, 0u, 0u, 0u};
  if (D <= 2 && lane == 0 && !(a.flags & F_INJECT)) w0 = noise_words(s.seed, eff_step(a), pid, 0u);
  const uint32_t mm = (uint32_t)rec.y;
  const int tm = mm & 0xff;
  uint32_t cw[4] = {0u, 0u, 0u, 0u};
  if ((s.rx_nb_mask >> tm) & 1) {
    uint32_t xm[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < D; k++) xm[k] = a.xp[k][m];
    auto count = [&](const Nb& nb) {
      count_partner<D>(s, rx, a, m, [&] { return nb.v & 0x7fffffff; }, tm, (int)(nb.m & 0xff), xm,
                       nb.x, cw);
    };
    if (cnt <= a.W) {
      for (int e = lane; e < cnt; e += 32) count(gather<D>(a, a.nbr[ell_index<TPP>(e, m, a.npad)]));
    } else {
      row_scan<D, 32>(s, a, m, lane, [&](int, int v) { count(gather<D>(a, v)); });
    }
#pragma unroll
    for (int w = 0; w < 4; w++) cw[w] = __reduce_add_sync(0xffffffffu, cw[w]);
  }
  return lane == 0 ? react_decide<D>(s, rx, a, pid, tm, cw,
                                     (D <= 2 && !(a.flags & F_INJECT)) ? &w0 : nullptr)
                   : tm;
}

// One listed pair's drift on particle i (type ti, pair words xo) from a
// partner with pair words xj and type tj (sorted index j(), evaluated where a
// cutoff is close), added to acc (pyrdsim.pyx:1988-2030).
template <int D, class J>
__device__ __forceinline__ void pair_eval(const ListShared& sh, const Args& a, int i, int ti,
                                          const uint32_t* xo, const uint32_t* xj, int tj, J&& j,
                                          float* acc) {
  const SysDev& s = sh.sys;
  float d[3];
  const float r2 = pair_geom<D>(s, xj, xo, d);
  if (!(r2 < s.prc2[ti * MAXT + tj])) return;  // beyond every law of the pair
  const unsigned int pp = s.ppair[ti * MAXT + tj];
  const PairLaw& L0 = sh.laws[(pp >> 5) & 0x3ff];
  float fr;
  if ((pp & 0x8000u) && r2 < L0.rc2_lo) {
    // a single Lennard-Jones n = 6 law, clear of its cutoff: eval_pair's
    // arithmetic inline
    fr = lj6_over_r(L0.c0, L0.c1, r2, recip(r2));
  } else {
    fr = pair_force<D>(s, sh.laws, a, i, j, pp, r2);
  }
#pragma unroll
  for (int k = 0; k < D; k++) acc[k] = fmaf(fr, d[k], acc[k]);
}

template <int D>
__device__ __forceinline__ void pair_term(const ListShared& sh, const Args& a, int i, int ti,
                                          const uint32_t* xo, const Nb& nb, float* acc) {
  if (nb.v < 0) return;  // same molecule: reactions only
  pair_eval<D>(sh, a, i, ti, xo, nb.x, (int)(nb.m & 0xff), [&] { return nb.v; }, acc);
}

// What the pair loop needs of a type pair in one 16-byte read: the largest
// guarded rc^2 of its laws and, for a single Lennard-Jones n = 6 law, the lower
// edge of its guard band and its constants (lo < 0: other laws).
// {rc2, lo, c0, c1} by [ti * ntypes + tj].  Whole CTA; the tables are staged.
__device__ inline void fill_rows(float4* rows, const ListShared& sh) {
  const int nt = sh.sys.ntypes;
  for (int q = threadIdx.x; q < nt * nt; q += LBLOCK) {
    const int t = q / nt * MAXT + q % nt;
    const unsigned int pp = sh.sys.ppair[t];
    const PairLaw& L = sh.laws[(pp >> 5) & 0x3ff];
    const bool lj6 = (pp & 0x8000u) != 0u;
    rows[q] = make_float4(sh.sys.prc2[t], lj6 ? L.rc2_lo : -1.f, lj6 ? L.c0 : 0.f, lj6 ? L.c1 : 0.f);
  }
}

// Phase A from the staged records of a period kernel: this lane's share
// (entries lane, lane + TPP, ...) of the pair drift of sorted particle i.
// codes: the lane's first word of the chunk's table; g, rec: the table's sorted
// indices and the records of this step.  A neighbour within range whose draw is
// pending (RX) is waited for.  The walk holds no call: at a distance in a cutoff's
// guard band it stops and returns false, and the lane walks its row again in
// staged_slow, where the float64 distance decides.  Two entries are in flight
// at a time: the loop is bound by the latency of its shared-memory reads and of
// the reciprocal.
//
// LPC > 1: LPC lanes share a chain (the entries that one lane would walk).
// Each evaluates every LPC-th entry; then the terms go round by shuffles and
// every lane adds them in list order, so the sum is that of LPC = 1.  All lanes
// of the warp call it (cnt = 0: no row), and the result is valid on each.
template <int D, int TPP, int LPC, bool RX>
__device__ __forceinline__ bool staged_walk(const ListShared& sh, const Args& a, const float4* rows,
                                            const uint4* slots, const int* g, const uint4* rec,
                                            const uint32_t* codes, int chain, int sub, int cnt,
                                            const uint32_t* xo, int ti, float* acc) {
  const SysDev& s = sh.sys;
  const float4* row = rows + ti * s.ntypes;
  // entries of this lane, and the rounds the lanes of the warp make together
  const int mine = ((cnt - chain + TPP - 1) / TPP - sub + LPC - 1) / LPC;
  const int rounds = LPC == 1 ? mine : __reduce_max_sync(0xffffffffu, max(mine, 0));
  bool ok = true;
  uint32_t next = mine > 0 ? codes[0] : 0u;
  for (int q = 0; q < rounds; q += 2) {
    const uint32_t cw = next;
    if (q + 2 < mine) next = codes[((q >> 1) + 1) * LBLOCK];
    const unsigned int code[2] = {q < mine ? cw & 0xffffu : 1u, q + 1 < mine ? cw >> 16 : 1u};
    uint4 r[2];
    float d[2][3], r2[2], fr[2];
    float4 t[2];
#pragma unroll
    for (int u = 0; u < 2; u++) r[u] = slots[code[u] >> 4];
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const uint32_t xj[3] = {r[u].x, r[u].y, r[u].z};
      t[u] = row[r[u].w & 0xfu];
      r2[u] = pair_geom<D>(s, xj, xo, d[u]);
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
      fr[u] = 0.f;
      bool in = !(code[u] & 1u);  // not of the same molecule (reactions only) or past the row
      if (RX && in && (r[u].w & REC_PENDING) && r2[u] <= s.R2) {
        r[u].w = pending_word(a, &rec[g[code[u] >> 4]].w);
        t[u] = row[r[u].w & 0xfu];
      }
      in = in && r2[u] < t[u].x;  // else beyond every law of the pair
      if (in) {
        if (r2[u] < t[u].y) {
          fr[u] = lj6_over_r(t[u].z, t[u].w, r2[u], recip(r2[u]));
        } else {
          bool close = t[u].y >= 0.f;
          if (!close)
            fr[u] = laws_over_r(sh.laws, s.ppair[ti * MAXT + (int)(r[u].w & 0xfu)], r2[u], close);
          if (close) {
            if (LPC == 1) return false;
            ok = false;
          }
        }
        if (LPC == 1) {
#pragma unroll
          for (int k = 0; k < D; k++) acc[k] = fmaf(fr[u], d[u][k], acc[k]);
        }
      }
    }
    if (LPC > 1) {
      // (no term: fr = 0 leaves the sum as it is)
#pragma unroll
      for (int u = 0; u < 2; u++) {
#pragma unroll
        for (int v = 0; v < LPC; v++) {
          const float f = __shfl_sync(0xffffffffu, fr[u], v, LPC);
#pragma unroll
          for (int k = 0; k < D; k++)
            acc[k] = fmaf(f, __shfl_sync(0xffffffffu, d[u][k], v, LPC), acc[k]);
        }
      }
    }
  }
  if (LPC > 1) {
    const unsigned int bad = __ballot_sync(0xffffffffu, !ok);
    ok = ((bad >> ((threadIdx.x & 31u) & ~(unsigned)(LPC - 1))) & ((1u << LPC) - 1u)) == 0u;
  }
  return ok;
}

// The chain of particle p of the chunk by one lane, with whatever calls it needs.
template <int D, int TPP, int LPC>
__device__ __noinline__ float3 staged_slow(const ListShared& sh, const Args& a, const uint4* slots,
                                           const int* g, const uint32_t* codes, int i, int p,
                                           int chain, int cnt, uint3 x, int ti) {
  const unsigned short* c16 = reinterpret_cast<const unsigned short*>(codes);
  const uint32_t xo[3] = {x.x, x.y, x.z};
  float acc[3] = {0.f, 0.f, 0.f};
  for (int e = chain; e < cnt; e += TPP) {
    const unsigned int code = c16[code_at<TPP, LPC>(p, e)];
    if (code & 1u) continue;  // same molecule: reactions only
    const uint4 r = slots[code >> 4];
    const uint32_t xj[3] = {r.x, r.y, r.z};
    int tj = (int)(r.w & 0xfu);
    if (r.w & REC_PENDING)
      tj = (int)(rec_wait(a, a.rec[period_n & 1] + g[code >> 4], REC_TAG, period_n, true).w & 0xfu);
    pair_eval<D>(sh, a, i, ti, xo, xj, tj, [&] { return g[code >> 4]; }, acc);
  }
  return make_float3(acc[0], acc[1], acc[2]);
}

template <int D, int TPP, bool PEND = false>
__device__ __forceinline__ void pair_drift(const ListShared& sh, const Args& a, int i, int lane,
                                           int cnt, const uint32_t* xo, uint32_t mi, float* acc) {
  const int ti = mi & 0xff;
  for_entries<D, TPP, PEND>(sh.sys, a, i, lane, cnt,
                            [&](const Nb& nb) { pair_term<D>(sh, a, i, ti, xo, nb, acc); });
}

// Phase A of the drift kernel where every pair law is a single Lennard-Jones n
// = 6 law: pair_drift's sums by a walk that holds no call and reads one row per
// type pair (fill_rows).  Bound by the latency of the gathers: the neighbour of
// the next entry and the index of the one after it are in flight while an entry
// is evaluated (4 % of the call at 1,048,576 particles; two entries at a time 1 %
// slower).  False at a distance in a cutoff's guard
// band (the lane then takes pair_drift).  Rows within the stored width only.
template <int D, int TPP>
__device__ __forceinline__ bool lj_walk(const ListShared& sh, const Args& a, const float4* rows,
                                        int i, int lane, int cnt, const uint32_t* xo, int ti,
                                        float* acc) {
  const SysDev& s = sh.sys;
  const float4* row = rows + ti * s.ntypes;
  auto entry = [&](int e) {
    return e < cnt ? a.nbr[ell_index<TPP>(e, i, a.npad)] : (i | LIST_SAME_MOL);
  };
  Nb nb = gather<D>(a, entry(lane));
  int v = entry(lane + TPP);
  for (int e = lane; e < cnt; e += TPP) {
    const Nb cur = nb;
    nb = gather<D>(a, v);
    v = entry(e + 2 * TPP);
    if (cur.v < 0) continue;  // same molecule: reactions only
    float d[3];
    const float r2 = pair_geom<D>(s, cur.x, xo, d);
    const float4 t = row[cur.m & 0xffu];
    if (!(r2 < t.x)) continue;  // beyond the pair's law
    if (!(r2 < t.y)) return false;
    const float fr = lj6_over_r(t.z, t.w, r2, recip(r2));
#pragma unroll
    for (int k = 0; k < D; k++) acc[k] = fmaf(fr, d[k], acc[k]);
  }
  return true;
}

template <int D, int TPP>
__device__ __noinline__ float3 lj_slow(const ListShared& sh, const Args& a, int i, int lane,
                                       int cnt, uint3 x, uint32_t mi) {
  const uint32_t xo[3] = {x.x, x.y, x.z};
  float acc[3] = {0.f, 0.f, 0.f};
  pair_drift<D, TPP>(sh, a, i, lane, cnt, xo, mi, acc);
  return make_float3(acc[0], acc[1], acc[2]);
}

// Drift kernel.  Phase A: TPP lanes per particle sum the pair drift over its
// list entries (pyrdsim.pyx:1988-2030).  Phase B: one thread per particle
// adds walls and bonded terms and performs the fused Euler-Maruyama update.
template <int D, int TPP, bool LJ>
__global__ void __launch_bounds__(LBLOCK, LJ ? LJ_MIN_BLOCKS : RD_LIST_MIN_BLOCKS) k_force_l(Args a) {
  constexpr int PER = LBLOCK / TPP;
  __shared__ ListShared sh;
  __shared__ float4 rows[LJ ? MAXT * MAXT : 1];
  __shared__ float sacc[3][PER];
  pdl_trigger();
  const Chunk ch = chunk_of<PER>(a);
  const int tid = threadIdx.x, g = tid / TPP, lane = tid % TPP;
  const bool active = g < ch.cnt;
  const int i = ch.beg + (active ? g : 0);
  list_tables<true, true, false>(sh, a, ch);
  pdl_wait();
  if (tid < ch.cnt) {  // phase B reads of particle beg + tid
    const int ib = ch.beg + tid;
    prefetch_l1(a.pid + ib);
#pragma unroll
    for (int k = 0; k < D; k++) prefetch_l1(a.xl[k] + ib);
  }
  const int cnt = a.ncnt[i];
  uint32_t xo[3] = {0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < D; k++) xo[k] = a.xp[k][i];
  if (a.stamps && threadIdx.x == 0)
    a.stamps[((size_t)(eff_step(a) % a.stamp_ring) * gridDim.x + blockIdx.x) * 2] = global_timer();
  const uint32_t mi = a.meta[i];
  prefetch_rows<TPP>(a, ch, cnt, active);
  __syncthreads();
  const SysDev& s = sh.sys;
  float acc[3] = {0.f, 0.f, 0.f};
  if (LJ) {
    fill_rows(rows, sh);
    __syncthreads();
    if (active) {
      bool ok = cnt <= a.W;
      if (ok) ok = lj_walk<D, TPP>(sh, a, rows, i, lane, cnt, xo, (int)(mi & 0xff), acc);
      if (!ok) {
        const float3 f = lj_slow<D, TPP>(sh, a, i, lane, cnt, make_uint3(xo[0], xo[1], xo[2]), mi);
        acc[0] = f.x;
        acc[1] = f.y;
        acc[2] = f.z;
      }
    }
  } else if (active && s.R2 > 0.f) {
    pair_drift<D, TPP>(sh, a, i, lane, cnt, xo, mi, acc);
  }
#pragma unroll
  for (int o = TPP >> 1; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < D; k++) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
  }
  if (active && lane == 0) {
#pragma unroll
    for (int k = 0; k < D; k++) sacc[k][g] = acc[k];
  }
  __syncthreads();
  const int ib = ch.beg + tid;
  bool listed = false;
  int4 rec = make_int4(0, 0, 0, 0);
  if (tid < ch.cnt) {
    uint32_t xb[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < D; k++) xb[k] = a.xh[k][ib];
    float accb[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < D; k++) accb[k] = sacc[k][tid];
    const uint32_t mb = a.meta[ib];
    const int pid = a.pid[ib];
    // one Philox call for the next step's noise and reaction uniform
    const bool words = (a.flags & F_RX_NEXT) ||
                       ((a.flags & F_EM) && !(a.flags & (F_NO_NOISE | F_INJECT)));
    U4 w0 = {0u, 0u, 0u, 0u};
    if (words) w0 = noise_words(s.seed, eff_em_step(a), pid, 0u);
    force_tail<D>(s, sh.walls, a, ib, pid, xb, mb, accb, words ? &w0 : nullptr);
    if (a.flags & F_RX_NEXT) {
      a.meta_out[ib] = mb;  // the next step's types, unless its draw succeeds
      rec = make_int4(ib, (int)mb, a.ncnt[ib], pid);
      listed = rx_may_react<D>(s, (int)(mb & 0xff), a.rcnt[ib], pid, eff_em_step(a), &w0);
    }
  }
  if (a.flags & F_RX_NEXT) {
    // append the particles whose draw may succeed (warp-aggregated)
    const unsigned int bal = __ballot_sync(0xffffffffu, listed);
    if (bal) {
      const int lane32 = threadIdx.x & 31, leader = __ffs(bal) - 1;
      const int p = rx_slot(eff_em_step(a));
      int base = 0;
      if (lane32 == leader) base = atomicAdd(a.rx_count + p, __popc(bal));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (listed) a.rx_list[(size_t)p * a.npad + base + __popc(bal & ((1u << lane32) - 1u))] = rec;
    }
  }
  // the slot of two steps ago was consumed before this kernel: empty it for
  // the drift kernel (or list builder) of the next step that appends to it
  if (blockIdx.x == 0 && threadIdx.x == 0) a.rx_count[rx_slot(eff_step(a) + 2)] = 0;
  // each warp's end: the CTA's end is their maximum (no barrier; the times
  // only grow, so a reused slot's older value never wins)
  if (a.stamps && (threadIdx.x & 31) == 0)
    atomicMax(a.stamps + ((size_t)(eff_step(a) % a.stamp_ring) * gridDim.x + blockIdx.x) * 2 + 1,
              global_timer());
}

// Spans of the stamped drift launches: per ring slot, the last CTA end minus
// the first CTA start (slots never written are skipped), summed.
static __global__ void k_stamp_spans(const unsigned long long* st, int ring, int nctas,
                              unsigned long long* sum, unsigned long long* count) {
  __shared__ unsigned long long lo[32], hi[32];
  const int slot = blockIdx.x;
  unsigned long long a0 = ~0ull, b0 = 0ull;
  for (int c = threadIdx.x; c < nctas; c += blockDim.x) {
    const unsigned long long s0 = st[((size_t)slot * nctas + c) * 2];
    const unsigned long long e0 = st[((size_t)slot * nctas + c) * 2 + 1];
    if (s0 && e0) {
      a0 = min(a0, s0);
      b0 = max(b0, e0);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    a0 = min(a0, __shfl_xor_sync(0xffffffffu, a0, o));
    b0 = max(b0, __shfl_xor_sync(0xffffffffu, b0, o));
  }
  if ((threadIdx.x & 31) == 0) {
    lo[threadIdx.x >> 5] = a0;
    hi[threadIdx.x >> 5] = b0;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      a0 = min(a0, lo[w]);
      b0 = max(b0, hi[w]);
    }
    if (b0 > a0) {
      atomicAdd(sum, b0 - a0);
      atomicAdd(count, 1ull);
    }
  }
}

// Reaction kernel.  Phase A: TPP lanes per particle count, for every
// neighbour-dependent reaction, the listed partners of the right type within
// r0 (16-bit counters, two reactions per word).  Phase B: one thread per
// particle forms the propensities, draws and writes the new type
// (pyrdsim.pyx:2070-2223).
template <int D, int TPP>
__global__ void __launch_bounds__(LBLOCK, RD_LIST_MIN_BLOCKS) k_react_l(Args a) {
  constexpr int PER = LBLOCK / TPP;
  __shared__ ListShared sh;
  __shared__ uint32_t scnt[4][PER];
  pdl_trigger();
  const Chunk ch = chunk_of<PER>(a);
  list_tables<false, false, true>(sh, a, ch);
  pdl_wait();
  const int tid = threadIdx.x, g = tid / TPP, lane = tid % TPP;
  const bool active = g < ch.cnt;
  const int i = ch.beg + (active ? g : 0);
  if (tid < ch.cnt) prefetch_l1(a.pid + ch.beg + tid);
  const int cnt = a.ncnt[i];
  const uint32_t mi = a.meta[i];
  uint32_t xo[3] = {0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < D; k++) xo[k] = a.xp[k][i];
  prefetch_rows<TPP>(a, ch, cnt, active);
  __syncthreads();
  const SysDev& s = sh.sys;
  uint32_t c0 = 0u, c1 = 0u, c2 = 0u, c3 = 0u;
  const int ti = mi & 0xff;
  if (active && ((s.rx_nb_mask >> ti) & 1)) {
    const float Rrx2 = s.Rrx2;
    for_entries<D, TPP>(s, a, i, lane, cnt, [&](const Nb& nb) {
      float d[3];
      const float r2 = pair_geom<D>(s, nb.x, xo, d);
      if (!(r2 < Rrx2)) return;
      const unsigned int rm = s.rxmatch[ti * MAXT + (nb.m & 0xff)];
      double dexact = -1.0;
      for (unsigned int mm = rm; mm; mm &= mm - 1u) {
        const int r = __ffs(mm) - 1;
        const RxDev& R = sh.rx[r];
        bool inside;
        if (r2 < R.r02_lo) inside = true;
        else if (r2 > R.r02_hi) inside = false;
        else {
          if (dexact < 0) dexact = exact_dist<D>(s, a, i, nb.v & 0x7fffffff);
          inside = dexact < R.r0;
        }
        if (inside) {
          const uint32_t inc = 1u << (16 * (r & 1));
          switch (r >> 1) {
            case 0: c0 += inc; break;
            case 1: c1 += inc; break;
            case 2: c2 += inc; break;
            default: c3 += inc; break;
          }
        }
      }
    });
  }
#pragma unroll
  for (int o = TPP >> 1; o > 0; o >>= 1) {
    c0 += __shfl_xor_sync(0xffffffffu, c0, o);
    c1 += __shfl_xor_sync(0xffffffffu, c1, o);
    c2 += __shfl_xor_sync(0xffffffffu, c2, o);
    c3 += __shfl_xor_sync(0xffffffffu, c3, o);
  }
  if (active && lane == 0) {
    scnt[0][g] = c0;
    scnt[1][g] = c1;
    scnt[2][g] = c2;
    scnt[3][g] = c3;
  }
  __syncthreads();
  if (tid < ch.cnt) {
    const int ib = ch.beg + tid;
    const uint32_t cw[4] = {scnt[0][tid], scnt[1][tid], scnt[2][tid], scnt[3][tid]};
    react_tail<D>(s, sh.rx, a, ib, a.pid[ib], a.meta[ib], cw);
  }
}

// Reaction kernel of the steps the previous drift kernel (or the list
// builder) prefiltered: that kernel copied every type forward and listed the
// particles whose draw may succeed; one warp per listed particle resolves it
// (resolve_listed) and writes its new type (pyrdsim.pyx:2070-2223).  A
// single system's tables are staged in shared memory; a batch's are read
// through L1.
template <int D, int TPP>
__global__ void __launch_bounds__(LBLOCK) k_react_listed(Args a) {
  __shared__ SysDev sys1;
  __shared__ RxDev rx1[MAXR];
  pdl_trigger();
  if (a.single) {
    constexpr int NS = (int)(sizeof(SysDev) / 4), NR = MAXR * (int)(sizeof(RxDev) / 4);
    const int nr = a.chunk1.nrx * (int)(sizeof(RxDev) / 4);
    WordLoad<NS> ls;
    WordLoad<NR> lr;
    ls.load(reinterpret_cast<const int*>(a.sys), NS);
    lr.load(reinterpret_cast<const int*>(a.rx), nr);
    ls.store(reinterpret_cast<int*>(&sys1), NS);
    lr.store(reinterpret_cast<int*>(rx1), nr);
  }
  pdl_wait();
  // the step counter, the three slots' counts and this warp's first record
  // of each slot are loaded together (one round trip instead of three)
  const int w0 = (int)((blockIdx.x * LBLOCK + threadIdx.x) >> 5);
  int nc[3];
  int4 f[3];
  const int4 zero = make_int4(0, 0, 0, 0);
#pragma unroll
  for (int q = 0; q < 3; q++) {
    nc[q] = a.rx_count[q];
    f[q] = w0 < a.npad ? a.rx_list[(size_t)q * a.npad + w0] : zero;
  }
  const int p = rx_slot(eff_step(a));
  const int n = p == 0 ? nc[0] : (p == 1 ? nc[1] : nc[2]);
  const int4 first = p == 0 ? f[0] : (p == 1 ? f[1] : f[2]);
  __syncthreads();
  const int4* list = a.rx_list + (size_t)p * a.npad;
  const int lane = threadIdx.x & 31;
  const int nwarps = (int)(gridDim.x * LBLOCK / 32);
  for (int q = w0; q < n; q += nwarps) {
    const int4 rec = q == w0 ? first : list[q];
    const SysDev& s = a.single ? sys1 : a.sys[a.sid[rec.x]];
    const RxDev* rx = a.single ? rx1 : a.rx + s.rx0;
    const int newt = resolve_listed<D, TPP>(s, rx, a, rec, lane);
    if (lane == 0) a.meta_out[rec.x] = ((uint32_t)rec.y & 0xffffff00u) | (uint32_t)newt;
  }
}

}  // namespace rd
