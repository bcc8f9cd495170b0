// observe.cuh -- float64 observables of one system at the current state.
//
// k_observe: one thread per particle (sorted order) sums, in float64, the
// pair energies and virials of its Verlet-list row (each pair once, by the
// lower sorted index), its wall energies and the bonded terms it heads
// (bond or angle whose first atom it is), and takes the minimum listed
// partner distance; a block reduction writes one partial per CTA.
// k_observe_sum adds the partials in a fixed order (deterministic results).
// Counts (pairs in range, particles per type) are integer atomics.
//
// k_rdf and k_pairs_*: pair-distance histogram and neighbour pairs.
// Particles are binned in the cells of the last rebuild and have moved by at
// most delta since, so every pair closer than r now lies within a stencil of
// h cells, h = floor((r + 2 delta) / cell length) + 1 per dimension (all
// cells once where the stencil would wrap onto itself; always all cells
// after a call that ended with a device error).
#pragma once

#include "list.cuh"

namespace rd {

constexpr int OBS_BLOCK = 128;
constexpr int OBS_NSUM = 6;  // pair, wall, bond, angle energy, virial, min distance
constexpr int RDF_MAX_BINS = 8192;

struct ObsArgs {
  const rdsim_interaction* laws;   // float64 parameters, same order as Args::laws
  const rdsim_interaction* walls;  // same order as Args::walls
  const rdsim_term* terms;         // same order as Args::terms
  double* part;                    // [CTAs][OBS_NSUM]
  double* sums;                    // [OBS_NSUM] results of k_observe_sum
  unsigned long long* counts;      // [1 + MAXT]: pairs in range, particles per type
  int sys, tpp, nblocks, pad;
};

// Potential U and force magnitude f = dU/dr of one pair law at float64
// distance r; f follows pyrdsim.pyx:1068-1130.
__device__ inline double law_potential(const rdsim_interaction& it, double r, double& f) {
  switch (it.law) {
    case RDSIM_LAW_LJ: {
      const double q = it.r0 / r, q2 = q * q;
      const double s = it.n == 6 ? q2 * q2 * q2 : pow(q, (double)it.n);
      f = -2.0 * it.n * it.u0 / r * s * (s - 1.0);
      return it.u0 * s * (s - 2.0);
    }
    case RDSIM_LAW_TANH: {
      const double t = tanh((r - it.r0) / it.a);
      f = it.u0 * (1.0 - t * t) / (2.0 * it.a);
      return 0.5 * it.u0 * (t - 1.0);
    }
    case RDSIM_LAW_YUKAWA: {
      const double e = exp(-r / it.r0);
      f = -it.u0 * (1.0 + it.r0 / r) * e / (r * it.r0);
      return it.u0 * e / r;
    }
    case RDSIM_LAW_HARMONIC:
      f = it.u0 * r;
      return 0.5 * it.u0 * r * r;
    case RDSIM_LAW_PIECEWISE_LINEAR:
      if (r < it.r0 - it.dr) {
        f = 0.0;
        return -it.u0;
      }
      f = it.u0 / it.dr;
      return f * (r - it.r0);
  }
  f = 0.0;
  return 0.0;
}

// Wall potential at coordinate y (pyrdsim.pyx:1132-1145; 9-3 wall cut at rc).
__device__ inline double wall_potential(const rdsim_interaction& w, double y) {
  if (w.law == RDSIM_LAW_WALL) return 0.5 * w.u0 * (tanh((y - w.r0) / w.a) - 1.0);
  if (y > w.rc) return 0.0;
  const double s = w.r0 / y, s3 = s * s * s, s9 = s3 * s3 * s3;
  return w.u0 * (2.0 / 15.0 * s9 - s3);
}

// Minimum-image vector x_j - x_i and distance in float64, with the same
// operations as exact_dist (pyrdsim.pyx:1619-1633).
template <int D>
__device__ inline double exact_vec(const SysDev& s, const Args& a, int gi, int gj, double* v) {
  double d2 = 0.0;
#pragma unroll
  for (int k = 0; k < D; k++) {
    const double xi = fixed_to_double(s, k, a.xh[k][gi], a.xl[k][gi]);
    const double xj = fixed_to_double(s, k, a.xh[k][gj], a.xl[k][gj]);
    double d = __dsub_rn(xj, xi);
    if (((s.periodic >> k) & 1) && !(fabs(d) < 0.49 * s.L[k]))
      d = __dsub_rn(d, __dmul_rn(s.L[k], round(__ddiv_rn(d, s.L[k]))));
    v[k] = d;
    d2 = __dadd_rn(d2, __dmul_rn(d, d));
  }
  return __dsqrt_rn(d2);
}

// Sum (or minimum, q == OBS_NSUM - 1) of OBS_NSUM values over the CTA;
// thread 0 receives the result.
template <int NT>
__device__ inline void block_reduce(double* v) {
  __shared__ double red[NT / 32][OBS_NSUM];
#pragma unroll
  for (int q = 0; q < OBS_NSUM; q++)
    for (int o = 16; o > 0; o >>= 1) {
      const double u = __shfl_down_sync(0xffffffffu, v[q], o);
      v[q] = q == OBS_NSUM - 1 ? fmin(v[q], u) : v[q] + u;
    }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < OBS_NSUM; q++) red[w][q] = v[q];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int ww = 1; ww < NT / 32; ww++)
#pragma unroll
      for (int q = 0; q < OBS_NSUM; q++)
        v[q] = q == OBS_NSUM - 1 ? fmin(v[q], red[ww][q]) : v[q] + red[ww][q];
}

// Float64 energy, virial term (-r dU/dr summed) and whether any law of the
// pair is within its cutoff.
template <int D>
__device__ inline bool pair_potential(const SysDev& s, const Args& a, const ObsArgs& o, int i,
                                      int j, unsigned int pp, double& U, double& W) {
  const double r = exact_dist<D>(s, a, i, j);
  const int nl = pp & 31, l0 = (pp >> 5) & 0x3ff;
  bool in_range = false;
  U = W = 0.0;
  for (int l = l0; l < l0 + nl; l++) {
    const rdsim_interaction& L = o.laws[s.law0 + l];
    const double rc = L.law == RDSIM_LAW_PIECEWISE_LINEAR ? L.r0 : L.rc;
    if (r > rc) continue;  // pyrdsim.pyx:1988-2030
    double f;
    U += law_potential(L, r, f);
    W += r * f;
    in_range = true;
  }
  return in_range;
}

// The float64 pair terms bound this kernel (16 cycles per warp instruction
// and SM), so a listed pair is first tested in float32 from the pair words
// (against its guarded cutoff, as the drift kernel does) and only pairs that
// pass are evaluated: every lane collects up to OBS_C of its own, the warp
// lays them side by side, evaluates 32 at a time with all lanes busy, and each
// lane adds its results in list order (the sums do not depend on the split).
// The minimum distance is evaluated in float64 only for the entries whose
// float32 distance is within its error of the warp's smallest.  65,536
// particles of the wall fluid: 43 us (232 us with every listed distance in
// float64 on the listing thread).
constexpr int OBS_C = 8;

struct ObsWarp {
  int j[OBS_C][32];
  double U[OBS_C][32], W[OBS_C][32];
  unsigned short at[OBS_C * 32];  // lane | k << 5 of the q-th collected pair
};

template <int D>
__global__ void __launch_bounds__(OBS_BLOCK) k_observe(Args a, ObsArgs o) {
  __shared__ unsigned int stype[MAXT];
  __shared__ unsigned int spairs;
  __shared__ ObsWarp swarp[OBS_BLOCK / 32];
  const SysDev& s = a.sys[o.sys];
  if (threadIdx.x < MAXT) stype[threadIdx.x] = 0u;
  if (threadIdx.x == 0) spairs = 0u;
  __syncthreads();
  double v[OBS_NSUM] = {0.0, 0.0, 0.0, 0.0, 0.0, INFINITY};
  const int i = s.p0 + (int)blockIdx.x * OBS_BLOCK + (int)threadIdx.x;
  const bool valid = i < s.p0 + s.n;
  const int lane = threadIdx.x & 31;
  ObsWarp& sw = swarp[threadIdx.x >> 5];
  const uint32_t mi = valid ? a.meta[i] : 0u;
  const int ti = mi & 0xff;
  const int cnt = valid ? a.ncnt[i] : 0;
  unsigned int npairs = 0;
  uint32_t xi[3] = {0u, 0u, 0u};
  if (valid) {
    atomicAdd(&stype[ti], 1u);
#pragma unroll
    for (int k = 0; k < D; k++) xi[k] = a.xp[k][i];
  }
  auto r2_of = [&](int j) {
    uint32_t xj[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < D; k++) xj[k] = a.xp[k][j];
    float d[3];
    return pair_geom<D>(s, xj, xi, d);
  };
  auto entry = [&](int e) { return a.nbr[((e / o.tpp) * a.npad + i) * o.tpp + e % o.tpp]; };
  // listed pairs (both directions are listed; the lower index sums)
  const int ne = cnt <= a.W ? cnt : 0;
  float r2min = INFINITY;
  for (int e = 0; __any_sync(0xffffffffu, e < ne);) {
    int found = 0;
    for (; e < ne && found < OBS_C; e++) {
      const int j = entry(e);
      if (j & LIST_SAME_MOL) continue;
      const float r2 = r2_of(j);
      r2min = fminf(r2min, r2);
      if (j > i && r2 <= s.prc2[ti * MAXT + (a.meta[j] & 0xff)]) sw.j[found++][lane] = j;
    }
    int incl = found;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int k = 0; k < found; k++) sw.at[incl - found + k] = (unsigned short)(lane | k << 5);
    __syncwarp();
    const int i0 = i - lane;
    for (int q = lane; q < total; q += 32) {
      const int l = sw.at[q] & 31, k = sw.at[q] >> 5, j = sw.j[k][l];
      const unsigned int pp =
          s.ppair[(a.meta[i0 + l] & 0xff) * MAXT + (a.meta[j] & 0xff)];
      double U, W;
      npairs += pair_potential<D>(s, a, o, i0 + l, j, pp, U, W) ? 1u : 0u;
      sw.U[k][l] = U;
      sw.W[k][l] = W;
    }
    __syncwarp();
    for (int k = 0; k < found; k++) {
      v[0] += sw.U[k][lane];
      v[4] -= sw.W[k][lane];
    }
    __syncwarp();
  }
  // the smallest partner distance (see the comment above)
  {
    float w = r2min;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) w = fminf(w, __shfl_xor_sync(0xffffffffu, w, d));
    float q = s.qf[0];
#pragma unroll
    for (int k = 1; k < D; k++) q = fmaxf(q, s.qf[k]);
    const float bound = w * 1.000004f + 16.f * q * sqrtf(w) + 64.f * q * q;
    if (w < INFINITY && r2min <= bound)
      for (int e = 0; e < ne; e++) {
        const int j = entry(e);
        if (!(j & LIST_SAME_MOL) && r2_of(j) <= bound) v[5] = fmin(v[5], exact_dist<D>(s, a, i, j));
      }
  }
  if (valid) {
    if (cnt > a.W) {  // a row beyond the stored width
      row_scan<D, 1>(s, a, i, 0, [&](int, int j) {
        if (j & LIST_SAME_MOL) return;
        v[5] = fmin(v[5], exact_dist<D>(s, a, i, j));
        if (j < i) return;
        double U, W;
        const unsigned int pp = s.ppair[ti * MAXT + (a.meta[j] & 0xff)];
        npairs += pair_potential<D>(s, a, o, i, j, pp, U, W) ? 1u : 0u;
        v[0] += U;
        v[4] -= W;
      });
    }
    // walls
    for (int w = 0; w < s.nwalls; w++) {
      const rdsim_interaction& W = o.walls[s.wall0 + w];
      if (W.type_a != ti) continue;
      const int d = W.type_b;
      v[1] += wall_potential(W, fixed_to_double(s, d, a.xh[d][i], a.xl[d][i]));
    }
    // bonded terms headed by this particle (role 0: it is atom i of the term)
    const int tm = mi >> 24;
    if (tm != 0xff) {
      const TmplDev& T = a.tmpl[tm];
      const int loc = (mi >> 16) & 0xff;
      const int mbase = a.pid[i] - loc;
      for (int e = a.atomterm[T.atom0 + loc]; e < a.atomterm[T.atom0 + loc + 1]; e++) {
        const int code = a.atomterm[e];
        if (code & 3) continue;
        const TermDev& tr = a.terms[code >> 2];
        const rdsim_term& ot = o.terms[code >> 2];
        if (tr.kind == RDSIM_TERM_BOND) {
          double dv[3];
          const double d = exact_vec<D>(s, a, i, a.slot_of[mbase + tr.j], dv);
          const double f = ot.k0 * (d - ot.p0);
          v[2] += 0.5 * f * (d - ot.p0);
          v[4] -= d * f;
        } else {
          // theta from the unit vectors as pyrdsim.pyx:1341-1364 forms them
          const int s2 = a.slot_of[mbase + tr.j], s3 = a.slot_of[mbase + tr.k];
          double v1[3], v2[3];
          const double d21 = exact_vec<D>(s, a, s2, i, v1);
          const double d23 = exact_vec<D>(s, a, s2, s3, v2);
          double c = 0.0;
#pragma unroll
          for (int k = 0; k < D; k++) c += (v1[k] / d21) * (v2[k] / d23);
          const double theta = c <= -1.0 ? 3.141592653589793 : (c >= 1.0 ? 0.0 : acos(c));
          v[3] += 0.5 * ot.k0 * (theta - ot.p0) * (theta - ot.p0);
        }
      }
    }
  }
  // counted by the lane that evaluated the pair, not by its particle's
  npairs = __reduce_add_sync(0xffffffffu, npairs);
  if (lane == 0 && npairs) atomicAdd(&spairs, npairs);
  block_reduce<OBS_BLOCK>(v);
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < OBS_NSUM; q++) o.part[(size_t)blockIdx.x * OBS_NSUM + q] = v[q];
    if (spairs) atomicAdd(o.counts, (unsigned long long)spairs);
  }
  if (threadIdx.x < MAXT && stype[threadIdx.x])
    atomicAdd(o.counts + 1 + threadIdx.x, (unsigned long long)stype[threadIdx.x]);
}

// One CTA: thread t adds the partials of CTAs t, t + 128, ... in order, then
// the fixed-shape block reduction.
__global__ void __launch_bounds__(OBS_BLOCK) k_observe_sum(ObsArgs o) {
  double v[OBS_NSUM] = {0.0, 0.0, 0.0, 0.0, 0.0, INFINITY};
  for (int b = threadIdx.x; b < o.nblocks; b += OBS_BLOCK)
#pragma unroll
    for (int q = 0; q < OBS_NSUM; q++) {
      const double u = o.part[(size_t)b * OBS_NSUM + q];
      v[q] = q == OBS_NSUM - 1 ? fmin(v[q], u) : v[q] + u;
    }
  block_reduce<OBS_BLOCK>(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < OBS_NSUM; q++) o.sums[q] = v[q];
}

// Cells around sorted particle i that can hold a particle within a given
// reach now: the cells date from the last rebuild, so they are looked up from
// the positions of that rebuild (xr), h[k] cells to either side (every cell
// once where that would wrap onto itself; h[k] >= nc[k] always means every
// cell).
struct CellBox {
  int lo[3], hi[3];
};

template <int D>
__device__ inline CellBox cell_box(const SysDev& s, const Args& a, int i, const int* h) {
  CellBox b;
#pragma unroll
  for (int k = 0; k < 3; k++) b.lo[k] = b.hi[k] = 0;
#pragma unroll
  for (int k = 0; k < D; k++) {
    const int c = cell_coord(s, k, a.xr[k][i]);
    const bool per = (s.periodic >> k) & 1;
    if (per ? 2 * h[k] + 1 >= s.nc[k] : h[k] >= s.nc[k]) {
      b.lo[k] = 0;
      b.hi[k] = s.nc[k] - 1;
    } else {
      b.lo[k] = per ? c - h[k] : max(c - h[k], 0);
      b.hi[k] = per ? c + h[k] : min(c + h[k], s.nc[k] - 1);
    }
  }
  return b;
}

// Visit the runs [jb, je) of sorted particles in the box, row of cells by row
// (cells along x are contiguous in the sorted arrays; a row that wraps is two
// runs).
template <int D, class Fn>
__device__ inline void for_runs(const SysDev& s, const Args& a, const CellBox& b, Fn&& fn) {
  const int nx = s.nc[0];
  for (int cz = b.lo[2]; cz <= b.hi[2]; cz++)
    for (int cy = b.lo[1]; cy <= b.hi[1]; cy++) {
      int row = 0;
      if (D > 1) row += (cy < 0 ? cy + s.nc[1] : (cy >= s.nc[1] ? cy - s.nc[1] : cy)) * nx;
      if (D > 2) row += (cz < 0 ? cz + s.nc[2] : (cz >= s.nc[2] ? cz - s.nc[2] : cz)) * nx * s.nc[1];
      const int* cs = a.cell_start + s.c0 + row;
      const int x0 = max(b.lo[0], 0), x1 = min(b.hi[0], nx - 1);
      fn(cs[x0], cs[x1 + 1]);
      if (b.lo[0] < 0) fn(cs[nx + b.lo[0]], cs[nx]);
      if (b.hi[0] >= nx) fn(cs[0], cs[b.hi[0] - nx + 1]);
    }
}

// Float32 squared distance from the high words (unit L / 2^32), minimum image
// in periodic dimensions whatever the distance.
template <int D>
__device__ inline float high_r2(const SysDev& s, const Args& a, const uint32_t* xi, int j) {
  float r2 = 0.f;
#pragma unroll
  for (int k = 0; k < D; k++) {
    const float d = (float)(int)(a.xh[k][j] - xi[k]) * s.unit_hi[k];
    r2 += d * d;
  }
  return r2;
}

// ---------------------------------------------------------------------------
// Neighbour list as the reference would rebuild it now (pyrdsim.pyx:1448-1587):
// bonded-list pairs plus partner-type pairs of different molecules, d <= rs,
// each once from its lower caller index, in caller order.
//
// One warp per particle walks the cells within rs of it, 32 candidates at a
// time, twice: k_pairs_count writes the row lengths by caller index, k_pairs_scan
// their running sum, and k_pairs_fill each row at its offset, ordered by
// ranking (every entry counts the smaller ones), so the list leaves the device
// sorted.  A row beyond PAIR_ROW entries is left unordered (the host orders
// it).  Only distances within the float32 error of rs are evaluated in
// float64.  Bound by the distance tests of the candidates (about 130 per
// particle here, whatever N).  Measured on the wall fluid at 16,384 particles
// (257 K pairs): count 20 us, scan 13 us, fill 24 us; testing all N^2 pairs
// took 3.8 ms per walk and the host's sort about 12 ms.
constexpr int PAIR_WARPS = 8;   // particles per CTA
constexpr int PAIR_ROW = 256;   // longest row ordered on the device

struct PairArgs {
  double rs;
  float rs2_lo, rs2_hi;           // guard band around rs^2
  int sys, pid0;                  // the system's first caller index
  int h[3];                       // stencil half-width in cells
  int* count;                     // [n] row lengths, by local caller index
  unsigned long long* start;      // [n] row offsets
  unsigned long long* total;      // [2]: pairs, longest row
  int* out;                       // [cap][2]
};

// Calls fn(hit, j's local caller index) on every lane of the warp, 32
// candidates at a time; `hit` marks a listed pair of sorted particle gi with
// a partner of larger caller index.
template <int D, class Fn>
__device__ inline void walk_pairs(const SysDev& s, const Args& a, const PairArgs& o, int gi,
                                  int lane, Fn&& fn) {
  const uint32_t mi = a.meta[gi];
  const int pi = a.pid[gi], moli = a.mol[gi];
  const int ti = mi & 0xff, loci = (mi >> 16) & 0xff, tmi = mi >> 24;
  const uint32_t bmask = tmi != 0xff ? a.tmpl[tmi].bondmask[loci] : 0u;
  uint32_t xi[3] = {0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < D; k++) xi[k] = a.xh[k][gi];
  const CellBox b = cell_box<D>(s, a, gi, o.h);
  for_runs<D>(s, a, b, [&](int jb, int je) {
    for (int j0 = jb; j0 < je; j0 += 32) {
      const int j = j0 + lane;
      bool hit = false;
      int pj = 0;
      if (j < je) {
        pj = a.pid[j];
        const float r2 = high_r2<D>(s, a, xi, j);
        if (pj > pi && r2 <= o.rs2_hi) {
          const uint32_t mj = a.meta[j];
          hit = a.mol[j] == moli ? (bmask >> ((mj >> 16) & 31)) & 1 : (s.partner[ti] >> (mj & 0xff)) & 1;
          if (hit && r2 >= o.rs2_lo) hit = exact_dist<D>(s, a, gi, j) <= o.rs;
        }
      }
      fn(hit, pj - o.pid0);
    }
  });
}

template <int D>
__global__ void __launch_bounds__(PAIR_WARPS * 32) k_pairs_count(Args a, PairArgs o) {
  const SysDev& s = a.sys[o.sys];
  const int q = (int)blockIdx.x * PAIR_WARPS + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (q >= s.n) return;
  int cnt = 0;
  walk_pairs<D>(s, a, o, s.p0 + q, lane, [&](bool hit, int) { cnt += hit ? 1 : 0; });
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) o.count[a.pid[s.p0 + q] - o.pid0] = cnt;
}

// Running sum of n row lengths in 64 bits (all pairs of a dense box may pass
// 2^31) and the longest row: one CTA, 16 rows per thread and round.
constexpr int PSCAN_T = 1024, PSCAN_I = 16;
static __global__ void __launch_bounds__(PSCAN_T) k_pairs_scan(PairArgs o, int n) {
  __shared__ unsigned long long ws[PSCAN_T / 32];
  __shared__ int wm[PSCAN_T / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  unsigned long long carry = 0ull;
  int longest = 0;
  for (int base = 0; base < n; base += PSCAN_T * PSCAN_I) {
    int v[PSCAN_I];
    unsigned long long sum = 0ull;
    const int q0 = base + tid * PSCAN_I;
    if (q0 + PSCAN_I <= n) {
#pragma unroll
      for (int e = 0; e < PSCAN_I / 4; e++) {
        const int4 u = reinterpret_cast<const int4*>(o.count + q0)[e];
        v[4 * e] = u.x;
        v[4 * e + 1] = u.y;
        v[4 * e + 2] = u.z;
        v[4 * e + 3] = u.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < PSCAN_I; e++) v[e] = q0 + e < n ? o.count[q0 + e] : 0;
    }
#pragma unroll
    for (int e = 0; e < PSCAN_I; e++) {
      sum += (unsigned)v[e];
      longest = max(longest, v[e]);
    }
    unsigned long long inc = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += u;
    }
    if (lane == 31) ws[w] = inc;
    __syncthreads();
    unsigned long long off = carry, all = carry;
    for (int u = 0; u < PSCAN_T / 32; u++) {
      if (u < w) off += ws[u];
      all += ws[u];
    }
    unsigned long long run = off + inc - sum;
#pragma unroll
    for (int e = 0; e < PSCAN_I; e++) {
      if (q0 + e < n) o.start[q0 + e] = run;
      run += (unsigned)v[e];
    }
    carry = all;
    __syncthreads();
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  if (lane == 0) wm[w] = longest;
  __syncthreads();
  if (tid == 0) {
    for (int u = 1; u < PSCAN_T / 32; u++) longest = max(longest, wm[u]);
    o.total[0] = carry;
    o.total[1] = (unsigned long long)longest;
  }
}

template <int D>
__global__ void __launch_bounds__(PAIR_WARPS * 32) k_pairs_fill(Args a, PairArgs o) {
  __shared__ int row[PAIR_WARPS][PAIR_ROW];
  const SysDev& s = a.sys[o.sys];
  const int w = (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int q = (int)blockIdx.x * PAIR_WARPS + w;
  if (q >= s.n) return;
  const int gi = s.p0 + q, pi = a.pid[gi] - o.pid0;
  const int len = o.count[pi];
  int2* out = reinterpret_cast<int2*>(o.out) + o.start[pi];
  const bool order = len <= PAIR_ROW;
  int cnt = 0;
  walk_pairs<D>(s, a, o, gi, lane, [&](bool hit, int pj) {
    const unsigned int m = __ballot_sync(0xffffffffu, hit);
    const int at = cnt + __popc(m & ((1u << lane) - 1u));
    if (hit) {
      if (order) row[w][at] = pj;
      else out[at] = make_int2(pi, pj);
    }
    cnt += __popc(m);
  });
  if (!order) return;
  __syncwarp();
  for (int e = lane; e < len; e += 32) {
    const int v = row[w][e];
    int rank = 0;
    for (int u = 0; u < len; u++) rank += row[w][u] < v ? 1 : 0;
    out[rank] = make_int2(pi, v);
  }
}

struct RdfArgs {
  unsigned long long* counts;  // [nbins]
  double r_max, width;         // bin width r_max / nbins
  float r2_hi;                 // float32 bound of r_max^2 (guard band)
  float inv_width;             // 1 / width
  float edge;                  // half-width of the guard band at bin edges, in bins
  int sys, type_a, type_b, nbins, flags;
  int h[3];                    // stencil half-width in cells
};

__device__ inline bool type_is(int t, int want) { return want < 0 || t == want; }

// Pair-distance histogram.  RDF_LANES lanes per particle walk the later
// sorted particles of the cells around it.  The bin of a pair is
// floor(r / width) with the reference's float64 distance; the float32
// distance from the high words decides wherever it lies farther from a bin
// edge than its error (o.edge bins, see rdsim_get_rdf), and only the pairs
// next to an edge, below 1 in 1,000 here, are evaluated in float64.  65,536
// particles of the wall fluid with r_max = 5 and 200 bins (1.0 M pairs): 43 us,
// against 291 us with the float64 distance of every pair, one thread per
// particle (bound by the FP64 pipe).
constexpr int RDF_LANES = 8;

template <int D>
__global__ void __launch_bounds__(OBS_BLOCK) k_rdf(Args a, RdfArgs o) {
  __shared__ unsigned int hist[RDF_MAX_BINS];
  for (int b = threadIdx.x; b < o.nbins; b += OBS_BLOCK) hist[b] = 0u;
  __syncthreads();
  const SysDev& s = a.sys[o.sys];
  const int lane = (int)threadIdx.x % RDF_LANES;
  const int step = (int)gridDim.x * (OBS_BLOCK / RDF_LANES);
  for (int q = (int)(blockIdx.x * OBS_BLOCK + threadIdx.x) / RDF_LANES; q < s.n; q += step) {
    const int i = s.p0 + q;
    const int ti = a.meta[i] & 0xff;
    if (!(type_is(ti, o.type_a) || type_is(ti, o.type_b))) continue;
    const int moli = a.mol[i];
    uint32_t xi[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < D; k++) xi[k] = a.xh[k][i];
    const CellBox b = cell_box<D>(s, a, i, o.h);
    for_runs<D>(s, a, b, [&](int jb, int je) {
      for (int j = max(jb, i + 1) + lane; j < je; j += RDF_LANES) {
        const float r2 = high_r2<D>(s, a, xi, j);
        if (r2 > o.r2_hi) continue;
        const int tj = a.meta[j] & 0xff;
        if (!((type_is(ti, o.type_a) && type_is(tj, o.type_b)) ||
              (type_is(ti, o.type_b) && type_is(tj, o.type_a))))
          continue;
        if ((o.flags & RDSIM_RDF_OTHER_MOLECULES) && a.mol[j] == moli) continue;
        const float t = sqrtf(r2) * o.inv_width, f = floorf(t);
        int bin = (int)f;
        if (t - f < o.edge || t - f > 1.0f - o.edge) {
          const double r = exact_dist<D>(s, a, i, j);
          if (!(r < o.r_max)) continue;
          bin = (int)floor(__ddiv_rn(r, o.width));
        } else if (bin >= o.nbins) {
          continue;  // beyond r_max by more than the guard band
        }
        atomicAdd(&hist[min(bin, o.nbins - 1)], 1u);
      }
    });
  }
  __syncthreads();
  for (int b = threadIdx.x; b < o.nbins; b += OBS_BLOCK)
    if (hist[b]) atomicAdd(o.counts + b, (unsigned long long)hist[b]);
}

}  // namespace rd
