// period.cuh -- the period kernel: the steps between two rebuilds in one launch.
//
// Every step of one rebuild period (the listed reactions of each step, then
// its drift with the fused update of the next step), one CTA per chunk, all
// CTAs resident.  There is no grid-wide barrier and no progress word: each
// particle's state of a step is published as 16-byte records that carry the
// step as a tag (rec: pair words and type; recl, rech: low and high words, for
// exact distances and bonded terms), written and read with 128-bit accesses
// at GPU scope, so a record and its tag are seen together.  A chunk stages the
// records of the particles its lists touch and polls each until its tag is
// the current step: the poll is the load, one L2 round trip instead of a
// progress poll, a fence and the load.  Everything else a chunk needs (its own
// words, types, the noise) stays in its shared memory for the whole launch.
//
// Records are double-buffered by the parity of the step.  The list relation is
// symmetric (the same distance and partner tests from both ends), so a chunk
// that reads a particle is waited for by that particle's chunk: before a
// particle's record of step n is overwritten (at the end of step n + 1) its
// chunk has seen the step n + 1 record of a particle of every chunk that lists
// it, and that chunk wrote it after it had read all records of step n.  (A chunk
// that stages nothing waits for what it lists by gathering it, in every step of
// a launch with reactions, whatever the laws.)  A staged run also holds particles
// that no row lists; their records may be one buffer ahead, which the tag test
// accepts (they are not used).  Bonded partners read each other's records and so
// order each other in the same way.
//
// What bounds it: latency (the staged poll, the pair loop's shared-memory reads,
// the tail of half the threads) and, with reactions, the resolution of pending
// draws, which the neighbours of ~30 particles per step wait for.  Nothing in
// the pair loop may call or spill: the spills of calls in it went to L2 (the
// L1 is small beside the shared memory) and made the step 25 % slower.
// Measured at 65,536 particles (wall fluid, 20-step launches, ncu): 201 us with
// progress flags, an acquire per step and one polling warp, 150 us with records
// and 139 with the L1 that PeriodStage leaves; the LJ fluid at 1,024 particles 70 ->
// 37 us per 10-step launch, 28 us with 4 lanes per chain.
//
// LPC lanes share a chain (the entries of a row that one lane of the per-step
// kernels walks), so that small systems, whose few chunks leave most of the
// GPU idle, take more and shorter chunks: a chunk is LBLOCK / TPP / LPC
// particles.  The sums do not depend on it (staged_walk).
//
// Reactions: the drift of step n - 1 marks the record of each particle whose
// draw of step n may succeed as pending; the particle's own chunk resolves the
// draw at the start of step n from its staged records (every record keeps the
// type before the step's reactions, so a neighbour resolved earlier does not
// matter) and rewrites the type word.  A neighbour that stages a pending record
// waits for that word alone, and only when the pair is within range.  Every
// wait ends after wait_ns of the global timer, or as soon as any CTA has
// recorded an error: RDSIM_ERR_SYNC is recorded and the CTA returns.  The
// arithmetic per particle is that of k_force_l and k_react_listed (same
// functions), so the results equal theirs bit for bit.
#pragma once

#include "list.cuh"

// Resident CTAs per SM the period kernel is compiled for: 7 x 152 SMs hold
// the 1,024 chunks of 65,536 particles with 72 registers per thread.
#ifndef RD_PERIOD_MIN_BLOCKS
#define RD_PERIOD_MIN_BLOCKS 7
#endif

namespace rd {

// Per-particle words of the chunk, kept for the launch.  The noise of the
// update of a step is computed by the threads that have no particle tail of
// their own while the tails of the step before run.  Kept small (no pair words,
// counts in 16 bits): seven chunks of a 2D system then need 164 KB of an SM and
// not 196, which leaves the L1 92 KB and not 60 for spills, bonded partners and
// the loads of the draws (65,536 particles, 10-step launch of the patchy system:
// 111 -> 100 us; 160 / 153 us per rebuild period).
constexpr unsigned int CNT_MANY = 0xffffu;  // this many or more: read it from memory
template <int D, int PER>
struct PeriodStage {
  int pid[PER];
  uint32_t cnts[PER];               // entries of the row | those in the reactions' reach << 16
  uint32_t meta[PER];
  uint32_t xr[D][PER];              // high words at the rebuild
  uint32_t xh[D][PER], xl[D][PER];
  uint32_t w[2][2][PER];            // Philox words (tag 0) the reaction draw uses, by
                                    // parity of the step
  float xi[2][D][PER];              // their standard normals

  __device__ int cnt(const Args& a, int p, int i) const {
    const unsigned int c = cnts[p] & 0xffffu;
    return c < CNT_MANY ? (int)c : a.ncnt[i];
  }
  __device__ int rcnt(const Args& a, int p, int i) const {
    const unsigned int c = cnts[p] >> 16;
    return c < CNT_MANY ? (int)c : a.rcnt[i];
  }
  // pair word of dimension k
  __device__ uint32_t xp(const SysDev& s, int k, int p) const {
    return (uint32_t)((((unsigned long long)xh[k][p] << 32) | xl[k][p]) >> s.ps[k]);
  }
};

struct PeriodShared {
  ListShared sh;
  uint32_t cmask[2][CAND_WORDS];    // listed particles of steps of parity 0/1
  long long s0;                     // first step of the launch
};

// The reaction draw of particle p of the chunk (sorted index m) at step n by
// the calling warp (resolve_listed's counts and draw, from the staged records
// where its row is staged).  Out of line: rare, and its registers stay out of
// the drift's budget.
template <int D, int TPP, int LPC>
__device__ __noinline__ void period_resolve(const ListShared& sh, const Args& a, const uint4* slots,
                                            const uint32_t* codes, bool staged, int m, int p,
                                            int cnt, int pid, uint32_t* meta, const uint32_t* xo,
                                            int n, int lane) {
  const SysDev& s = sh.sys;
  const int tm = (int)(*meta & 0xffu);
  U4 w0 = {0u, 0u, 0u, 0u};
  if (D <= 2 && lane == 0) w0 = noise_words(s.seed, eff_step(a), pid, 0u);
  uint32_t cw[4] = {0u, 0u, 0u, 0u};
  if ((s.rx_nb_mask >> tm) & 1) {
    const uint4* rec = a.rec[n & 1];
    if (staged) {
      const unsigned short* c16 = reinterpret_cast<const unsigned short*>(codes);
      for (int e = lane; e < cnt; e += 32) {
        const unsigned int code = c16[code_at<TPP, LPC>(p, e)];
        const uint4 r = slots[code >> 4];
        const uint32_t xj[3] = {r.x, r.y, r.z};
        count_partner<D>(s, sh.rx, a, m, [&] { return a.nbr[ell_index<TPP>(e, m, a.npad)] & 0x7fffffff; },
                         tm, (int)((r.w >> REC_OLD) & 0xfu), xo, xj, cw);
      }
    } else {
      auto one = [&](int v) {
        const int j = v & 0x7fffffff;
        const uint4 r = get_rec(a, rec + j, REC_TAG, n);
        const uint32_t xj[3] = {r.x, r.y, r.z};
        count_partner<D>(s, sh.rx, a, m, [&] { return j; }, tm, (int)((r.w >> REC_OLD) & 0xfu), xo,
                         xj, cw);
      };
      if (cnt <= a.W) {
        for (int e = lane; e < cnt; e += 32) one(a.nbr[ell_index<TPP>(e, m, a.npad)]);
      } else {
        row_scan<D, 32>(s, a, m, lane, [&](int, int v) { one(v); });
      }
    }
#pragma unroll
    for (int w = 0; w < 4; w++) cw[w] = __reduce_add_sync(0xffffffffu, cw[w]);
  }
  if (lane == 0) {
    const int newt = react_decide<D>(s, sh.rx, a, pid, tm, cw, D <= 2 ? &w0 : nullptr);
    *meta = (*meta & 0xffffff00u) | (uint32_t)newt;
    uint32_t* w = &a.rec[n & 1][m].w;
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(w),
                 "r"(rec_word(n, (uint32_t)newt, (uint32_t)tm, false))
                 : "memory");
  }
}

// The noise of the update of step s0 + n + 1 for particle p.
template <int D, int PER>
__device__ __forceinline__ void period_noise(PeriodStage<D, PER>& st, const SysDev& s,
                                             long long step, bool noise, int P, int p) {
  const U4 w0 = noise_words(s.seed, step, st.pid[p], 0u);
  st.w[P][0][p] = w0.z;
  st.w[P][1][p] = w0.w;
  if (noise) {
    float xi[3];
    gaussians<D>(w0, xi);
#pragma unroll
    for (int k = 0; k < D; k++) st.xi[P][k][p] = xi[k];
  }
}

// Phase A of a particle whose row or chunk is not staged.  A row beyond the
// stored width, where LPC lanes share a chain: each lane generates the whole row
// and takes its chain's entries (row_scan's lanes are adjacent threads, the
// chains here are not), so that the sums stay those of LPC = 1.
template <int D, int TPP, int LPC>
__device__ __noinline__ float3 period_gather(const ListShared& sh, const Args& a, int i, int chain,
                                             int cnt, uint3 x, uint32_t mi) {
  const uint32_t xo[3] = {x.x, x.y, x.z};
  float acc[3] = {0.f, 0.f, 0.f};
  if (LPC > 1 && cnt > a.W) {
    row_scan<D, 1>(sh.sys, a, i, 0, [&](int k, int v) {
      if (k % TPP == chain)
        pair_term<D>(sh, a, i, (int)(mi & 0xff), xo, gather<D, true>(a, v), acc);
    });
  } else {
    pair_drift<D, TPP, true>(sh, a, i, chain, cnt, xo, mi, acc);
  }
  return unless_failed(make_float3(acc[0], acc[1], acc[2]));
}

// A wait ran out, or another chunk recorded an error: the particles stay where
// this chunk's last step left them.
constexpr int GAVE_UP = 2;  // period_failed then
template <int D, int PER, bool RX>
__device__ __noinline__ void leave_state(const SysDev& s, const PeriodStage<D, PER>& st,
                                         const Args& a, int i, int p) {
#pragma unroll
  for (int k = 0; k < D; k++) {
    a.xh_out[k][i] = st.xh[k][p];
    a.xl_out[k][i] = st.xl[k][p];
    a.xp_out[k][i] = st.xp(s, k, p);
  }
  if (RX) a.meta_out[i] = st.meta[p];
}

// Records a thread loads before it looks at their tags (1, 2, 4: 2,794 / 2,789
// / 2,843 us on the wall fluid while it was the same otherwise), and its pause
// between two looks, which leaves the issue slots to the CTAs that work (0 to
// 300 ns: no difference beyond 0.5 %).
constexpr int PBATCH = 2;
constexpr int PERIOD_SLEEP_NS = 100;

// Dynamic shared memory: the chunk's staging table and slot codes (they do not
// change within the launch, and the SM's L1, mostly shared memory here, would
// not keep them: 2,789 -> 2,676 us on the wall fluid), the pair constants and
// the staged records.
struct PeriodTables {
  uint4* slots;                     // [stg_max]
  int* g;                           // [stg_max]
  uint32_t* codes;                  // [kw][LBLOCK]
  float4* rows;                     // fill_rows
};
__device__ inline PeriodTables period_tables(const Args& a, unsigned char* dyn) {
  PeriodTables t;
  t.slots = reinterpret_cast<uint4*>(dyn);
  t.rows = reinterpret_cast<float4*>(t.slots + a.stg_max);
  t.g = reinterpret_cast<int*>(t.rows + a.rows_max);
  t.codes = reinterpret_cast<uint32_t*>(t.g + a.stg_max);
  return t;
}

// Step n of the launch on the CTA's chunk (RX: reactions run).  False: a wait
// ran out.
template <int D, int TPP, int LPC, bool RX>
__device__ __forceinline__ bool period_run_step(PeriodShared& ps,
                                                PeriodStage<D, LBLOCK / TPP / LPC>& st,
                                                const PeriodTables& tb,
                                                float (*sacc)[LBLOCK / TPP / LPC],
                                                const Args& a,
                                                const PeriodArgs& p, const Chunk& ch, int nstg,
                                                int n) {
  constexpr int PER = LBLOCK / TPP / LPC;
  const int tid = threadIdx.x, warp = tid >> 5, l32 = tid & 31, P = n & 1;
  const SysDev& s = ps.sh.sys;
  const bool last = n + 1 >= p.nsteps;
  const bool rx_next = RX && !last;
  const bool noise = !(a.flags & F_NO_NOISE);
  const int* sg = tb.g;
  const uint32_t* codes = tb.codes;
  uint4* slots = tb.slots;
  if (tid == 0) {
    period_step = ps.s0 + n;
    period_n = n;
  }
  // the staged records of this step
  const uint4* rec = a.rec[P];
  for (int q0 = tid; q0 < nstg; q0 += PBATCH * LBLOCK) {
    int at[PBATCH];
    uint4 v[PBATCH];
#pragma unroll
    for (int u = 0; u < PBATCH; u++) at[u] = sg[min(q0 + u * LBLOCK, nstg - 1)];
#pragma unroll
    for (int u = 0; u < PBATCH; u++) v[u] = ld_rec(rec + at[u]);
    bool over = false;
    unsigned long long t0 = 0ull;
    for (int k = 1; !over; k++) {
      bool ready = true;
#pragma unroll
      for (int u = 0; u < PBATCH; u++)
        if (!rec_ready(v[u].w, REC_TAG, n)) {
          ready = false;
          v[u] = ld_rec(rec + at[u]);
        }
      if (ready) break;
      __nanosleep(PERIOD_SLEEP_NS);
      if (k == 1) t0 = global_timer();
      else if ((k & 31) == 0) over = wait_over(a, t0);
    }
#pragma unroll
    for (int u = 0; u < PBATCH; u++)
      if (q0 + u * LBLOCK < nstg) slots[q0 + u * LBLOCK] = v[u];
    if (over) wait_failed(a, n);
  }
  // (a chunk that stages nothing has no wait that would notice an error)
  if (__syncthreads_or(nstg < 0 && tid == 0 ? *(volatile int*)&a.err->code : period_failed)) {
    period_failed = GAVE_UP;  // (every thread: k_period looks at it without a barrier)
    return false;
  }
  const int lsmax = min(a.W, a.kw * 2 * TPP * LPC);
  // reactions of step n: each warp resolves the draws of its own particles
  // (no barrier: who needs another's type waits for its record)
  if (RX) {
    constexpr int WP = PER * 32 / LBLOCK;  // particles per warp
    const int q0 = warp * WP;
    uint32_t b = ps.cmask[P][q0 >> 5] >> (q0 & 31);
    if (WP < 32) b &= (1u << (WP & 31)) - 1u;
#pragma unroll 1
    for (; b; b &= b - 1u) {
      const int q = q0 + __ffs(b) - 1;
      uint32_t xo[3] = {0u, 0u, 0u};
#pragma unroll
      for (int d = 0; d < D; d++) xo[d] = st.xp(s, d, q);
      const int cnt = st.cnt(a, q, ch.beg + q);
      period_resolve<D, TPP, LPC>(ps.sh, a, slots, codes, nstg >= 0 && cnt <= lsmax, ch.beg + q, q,
                             cnt, st.pid[q], &st.meta[q], xo, n, l32);
      __syncwarp();
    }
  }
  // drift of step n and the update of step n + 1 (k_force_l)
  const int g = tid / (TPP * LPC), chain = tid % (TPP * LPC) / LPC, sub = tid % LPC;
  const bool active = g < ch.cnt;
  const int gq = active ? g : 0;
  const int i = ch.beg + gq;
  float acc[3] = {0.f, 0.f, 0.f};
  // (an unstaged chunk walks its rows in a system without pair laws too: the
  // gathers are its wait for the particles it lists, whose draws read its
  // records)
  if (s.R2 > 0.f || (RX && nstg < 0)) {
    const int cnt = st.cnt(a, gq, i);
    uint32_t xo[3] = {0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < D; k++) xo[k] = st.xp(s, k, gq);
    const int ti = (int)(st.meta[gq] & 0xffu);
    const bool staged = nstg >= 0 && active && cnt <= lsmax;
    const bool ok = staged_walk<D, TPP, LPC, RX>(ps.sh, a, tb.rows, slots, sg, rec, codes + tid,
                                                 chain, sub, staged ? cnt : 0, xo, ti, acc);
    if (active && (!staged || !ok)) {
      const uint3 x = make_uint3(xo[0], xo[1], xo[2]);
      const float3 f =
          staged ? staged_slow<D, TPP, LPC>(ps.sh, a, slots, sg, codes, i, g, chain, cnt, x, ti)
                 : period_gather<D, TPP, LPC>(ps.sh, a, i, chain, cnt, x, (uint32_t)ti);
      acc[0] = f.x;
      acc[1] = f.y;
      acc[2] = f.z;
    }
    __syncwarp();
  }
#pragma unroll
  for (int o = TPP >> 1; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < D; k++) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o * LPC);
  }
  if (active && chain == 0 && sub == 0) {
#pragma unroll
    for (int k = 0; k < D; k++) sacc[k][g] = acc[k];
  }
  __syncthreads();
  if (warp < (PER + 31) / 32) {
    bool listed = false;
    if (tid < ch.cnt) {
      const int ib = ch.beg + tid;
      TailIn t;
#pragma unroll
      for (int k = 0; k < 3; k++) t.xh[k] = t.xl[k] = t.xr[k] = 0u;
#pragma unroll
      for (int k = 0; k < D; k++) {
        t.xh[k] = st.xh[k][tid];
        t.xl[k] = st.xl[k][tid];
      }
      float accb[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < D; k++) accb[k] = sacc[k][tid];
      const uint32_t mb = st.meta[tid];
      const int pid = st.pid[tid];
      wall_terms<D>(s, ps.sh.walls, t.xh, t.xl, (int)(mb & 0xff), accb);
      add_bonded<D, true>(s, a, t.xh, t.xl, pid, mb, n, accb);
      // (loaded here: nothing of it lives across the bonded terms' call)
#pragma unroll
      for (int k = 0; k < D; k++) t.xr[k] = st.xr[k][tid];
      tail_checks<D>(s, a, pid, t.xh, t.xr, accb, ps.s0 + n);
      float xi[3] = {0.f, 0.f, 0.f};
      if (noise) {
#pragma unroll
        for (int k = 0; k < D; k++) xi[k] = st.xi[P][k][tid];
      }
      t.xi = xi;
      unsigned long long X[3] = {0ull, 0ull, 0ull};
      em_update_in<D>(s, a, pid, (int)(mb & 0xff), accb, ps.s0 + n + 1, a.flags, nullptr, t, X);
      U4 w0 = {0u, 0u, 0u, 0u};
      if (rx_next) w0 = U4{0u, 0u, st.w[P][0][tid], st.w[P][1][tid]};
      if (rx_next)
        listed = rx_may_react<D>(s, (int)(mb & 0xff), st.rcnt(a, tid, ib), pid, ps.s0 + n + 1, &w0);
      uint32_t h[3] = {0u, 0u, 0u}, l[3] = {0u, 0u, 0u}, q[3] = {0u, 0u, 0u};
#pragma unroll
      for (int k = 0; k < D; k++) {
        h[k] = (uint32_t)(X[k] >> 32);
        l[k] = (uint32_t)X[k];
        q[k] = (uint32_t)(X[k] >> s.ps[k]);
      }
      if (!last) {
        if ((int)blockIdx.x != p.withhold) {
          const uint32_t ty = mb & 0xfu;
          st_rec(a.rec[P ^ 1] + ib, q[0], q[1], q[2], rec_word(n + 1, ty, ty, listed));
          st_rec(a.recl[P ^ 1] + ib, l[0], l[1], l[2], (uint32_t)(n + 1));
          st_rec(a.rech[P ^ 1] + ib, h[0], h[1], h[2], (uint32_t)(n + 1));
        }
#pragma unroll
        for (int k = 0; k < D; k++) {
          st.xh[k][tid] = h[k];
          st.xl[k][tid] = l[k];
        }
      } else {
#pragma unroll
        for (int k = 0; k < D; k++) {
          a.xh_out[k][ib] = h[k];
          a.xl_out[k][ib] = l[k];
          a.xp_out[k][ib] = q[k];
        }
        if (RX) a.meta_out[ib] = mb;
      }
    }
    // the particles whose draw of step n + 1 may succeed: one word per warp
    const unsigned int bal = __ballot_sync(0xffffffffu, listed);
    if (l32 == 0) ps.cmask[P ^ 1][warp] = bal;
  }
  // the noise of the next step's update, on the threads without a tail (one
  // lane per particle: on the same threads, after it)
  const int np = tid - (LBLOCK - PER);
  if (!last && np >= 0 && np < ch.cnt)
    period_noise<D, PER>(st, s, ps.s0 + n + 2, noise, P ^ 1, np);
  return true;
}

// RX: the launch runs reactions (its pair loop then also looks for pending
// draws; a system without reactions is 7 % faster without that code).
template <int D, int TPP, int LPC, bool RX>
__global__ void __launch_bounds__(LBLOCK, RD_PERIOD_MIN_BLOCKS)
    k_period(const __grid_constant__ Args a0, PeriodArgs p) {
  constexpr int PER = LBLOCK / TPP / LPC;
  extern __shared__ __align__(16) unsigned char dyn[];
  const PeriodTables tb = period_tables(a0, dyn);
  __shared__ PeriodShared ps;
  __shared__ PeriodStage<D, PER> st;
  __shared__ float sacc[D][PER];
  // No early launch of the next kernel: its CTAs must not take the SM slots
  // that CTAs of this kernel still wait for.
  const Chunk ch = chunk_at<PER>(a0, (int)blockIdx.x);
  list_tables<true, true, true>(ps.sh, a0, ch);
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5;
  // the chunk's words, all loads in flight together
  const int nstg = a0.stg_n[blockIdx.x];
  {
    const int* sg = a0.stg_g + (size_t)blockIdx.x * a0.stg_max;
    const uint32_t* codes = a0.codes + (size_t)blockIdx.x * a0.kw * LBLOCK;
    for (int q = tid; q < nstg; q += LBLOCK) tb.g[q] = sg[q];
    if (nstg >= 0)
#pragma unroll 4
      for (int w = 0; w < a0.kw; w++) tb.codes[w * LBLOCK + tid] = codes[w * LBLOCK + tid];
  }
  if (tid == 0) {
    period_failed = 0;
    ps.s0 = a0.step_base ? *a0.step_base + a0.step : a0.step;
    if (blockIdx.x == 0) {
      // the candidate lists of the per-step kernels stay empty
      a0.rx_count[0] = 0;
      a0.rx_count[1] = 0;
      a0.rx_count[2] = 0;
    }
  }
  if (tid < 2 * CAND_WORDS) ps.cmask[tid / CAND_WORDS][tid % CAND_WORDS] = 0u;
  bool listed = false;
  if (tid < ch.cnt) {
    const int ib = ch.beg + tid;
    st.pid[tid] = a0.pid[ib];
    st.cnts[tid] = min((unsigned int)a0.ncnt[ib], CNT_MANY) |
                   min((unsigned int)a0.rcnt[ib], CNT_MANY) << 16;
    st.meta[tid] = a0.meta[ib];
#pragma unroll
    for (int k = 0; k < D; k++) {
      st.xr[k][tid] = a0.xr[k][ib];
      st.xh[k][tid] = a0.xh[k][ib];
      st.xl[k][tid] = a0.xl[k][ib];
    }
    listed = RX && p.first_rx && (a0.rec[0][ib].w & REC_PENDING);
  }
  const unsigned int bal = __ballot_sync(0xffffffffu, listed);
  __syncthreads();
  if (warp < CAND_WORDS && (tid & 31) == 0) ps.cmask[0][warp] = bal;
  const SysDev& s = ps.sh.sys;
  fill_rows(tb.rows, ps.sh);
  {
    const int np = tid - (LBLOCK - PER);
    if (np >= 0 && np < ch.cnt)
      period_noise<D, PER>(st, s, ps.s0 + 1, !(a0.flags & F_NO_NOISE), 0, np);
  }
  const long long slot = a0.stamps ? (ps.s0 / p.nsteps) % a0.stamp_ring : 0;
  if (a0.stamps && tid == 0)
    a0.stamps[((size_t)slot * gridDim.x + blockIdx.x) * 2] = global_timer();
#pragma unroll 1
  for (int n = 0; n < p.nsteps; n++)
    if (!period_run_step<D, TPP, LPC, RX>(ps, st, tb, sacc, a0, p, ch, nstg, n)) break;
  if (period_failed == GAVE_UP && tid < ch.cnt)
    leave_state<D, PER, RX>(s, st, a0, ch.beg + tid, tid);
  if (a0.stamps && (tid & 31) == 0)
    atomicMax(a0.stamps + ((size_t)slot * gridDim.x + blockIdx.x) * 2 + 1, global_timer());
}

}  // namespace rd
