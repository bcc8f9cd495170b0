// adjoint.cu -- float64 reaction-free steps, a trajectory loss and its
// discrete adjoint (gradients with respect to the initial positions and the
// pair-law parameters), for include/rdsim_adjoint.h.
//
// Every state is binned into cells (counting sort, then each cell's members
// in index order) and gets a neighbour list: the particles of the 3^D
// cells around each particle that pass a float32 distance screen, in a fixed
// order, so all sums run in a fixed order and results are deterministic.
// Float64 issue is scarce on this GPU (a warp instruction every 16 cycles per
// SM, however few lanes are active), so the float64 kernels screen the list
// entries in float32 first, queue the pairs inside a law's cutoff by kind of
// law, and evaluate 32 of a kind at a time (see PairQueue).  Forward
// (k_adj_step): pair drift of pyrdsim.pyx:1941-2067 for
// Lennard-Jones and Yukawa laws (pyrdsim.pyx:1068-1130), the loss terms of
// the state, and the Euler-Maruyama update with injected noise and periodic
// wrap (pyrdsim.pyx:2225-2292).  Backward (k_adj_back): for state x_n and
// w = c * lambda_{n+1},
//   lambda_n = g_n + lambda_{n+1} + sum_j K_ij (w_j - w_i),
//   K_ij = f' rhat rhat^T + (f / r) (I - rhat rhat^T),
// (f = dU/dr; a_i = sum_j f rhat_ij, so d a_i / d x_j = K_ij), the loss
// gradient g_n, and the parameter gradients sum over pairs of
// df/dtheta rhat . (w_i - w_j) plus the loss's own dependence.  States of
// the backward pass are recomputed segment by segment from checkpoints.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/rdsim_adjoint.h"

namespace {

constexpr int MAXT = RDSIM_MAX_TYPES;
constexpr int MAXL = RDSIM_ADJ_MAX_LAWS;
constexpr int NG = 2 * MAXL;  // parameter gradients: (u0, r0) per law
constexpr int BLK = 128;
constexpr int SCAN_T = 1024;

thread_local std::string g_err;

int fail(int code, const std::string& m) {
  g_err = m;
  return code;
}

#define CK(call)                                                                  \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess)                                                        \
      return fail(RDSIM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

struct Law {
  int law, n;
  double u0, r0, rc, ir0;       // ir0 = 1 / r0
  double Uc, dUc_du0, dUc_dr0;  // energy at rc and its parameter derivatives
  double r02, rc2;              // r0^2, rc^2
  float screen2;                // float32 screen: above rc^2
  int pad;
};

struct AdjArgs {
  int N, D, nlaws;
  int nc[3], ncell;
  double L[3], cellinv[3];
  float Lf[3], Linvf[3];
  int exact_image;              // boxes near 2 rc: float64 decides the image
  float cut2f;                  // float32 screen of the list in use
  float move2f;                 // displacement^2 allowed while a list is reused
  double c[MAXT], s[MAXT];      // dt D and sqrt(2 dt D) per type
  double wU, wW;                // loss weights 1/K and 1/(K d V)
  unsigned char lawmask[MAXT * MAXT];  // bit l: law l applies to (ti, tj)
  Law laws[MAXL];
};

enum { F_STEP = 1, F_LOSS = 2 };
constexpr int TPP = 4;  // lanes per particle in the pair kernels

// Pair terms of one law at distance r < rc (ir = 1 / r): U (unshifted),
// f = dU/dr, fp = d2U/dr2, and the derivatives of U and f by (u0, r0).
struct PairEval {
  double U, f, fp, dU[2], df[2];
};

inline double lj_power(double q, int n) {
  // (r0 / r)^n from q = r0 / r
  if (n == 6) {
    const double q2 = q * q;
    return q2 * q2 * q2;
  }
  double s = 1.0;
  for (int e = 0; e < n; e++) s *= q;
  return s;
}

inline PairEval eval_law(const Law& w, double r, double ir) {
  PairEval p;
  if (w.law == RDSIM_LAW_LJ) {
    // U = u0 (s^2 - 2 s), s = (r0/r)^n; f = -2 n u0 s (s - 1) / r
    const double n = (double)w.n;
    const double s = lj_power(w.r0 * ir, w.n);
    const double t = 2.0 * n * s * ir;
    p.U = w.u0 * s * (s - 2.0);
    p.f = -w.u0 * t * (s - 1.0);
    p.fp = w.u0 * t * ((2.0 * n + 1.0) * s - (n + 1.0)) * ir;
    p.dU[0] = s * (s - 2.0);
    p.df[0] = -t * (s - 1.0);
    // ds/dr0 = n s / r0
    p.dU[1] = 2.0 * n * w.u0 * s * (s - 1.0) * w.ir0;
    p.df[1] = -w.u0 * t * n * (2.0 * s - 1.0) * w.ir0;
  } else {
    // Yukawa: U = u0 e / r, e = exp(-r / r0)
    const double e = exp(-r * w.ir0);
    const double ir0 = w.ir0;
    const double h = ir * ir0 + ir * ir;
    p.U = w.u0 * e * ir;
    p.f = -w.u0 * e * h;
    p.fp = w.u0 * e * ir * (ir0 * ir0 + 2.0 * ir * ir0 + 2.0 * ir * ir);
    p.dU[0] = e * ir;
    p.df[0] = -e * h;
    p.dU[1] = w.u0 * e * ir0 * ir0;
    p.df[1] = -w.u0 * e * ir0 * ir0 * ir0;
  }
  return p;
}

// Cell of coordinate x along k, wrapped into [0, nc) (positions on or
// outside the box edge map to their periodic image's cell).
__device__ inline int cell_of(const AdjArgs& g, int k, double x) {
  int c = (int)floor(x * g.cellinv[k]) % g.nc[k];
  return c < 0 ? c + g.nc[k] : c;
}

template <int D>
__global__ void k_bin(AdjArgs g, const double* __restrict__ x, int* __restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  int c = 0, mult = 1;
#pragma unroll
  for (int k = 0; k < D; k++) {
    c += cell_of(g, k, x[(size_t)i * D + k]) * mult;
    mult *= g.nc[k];
  }
  atomicAdd(count + c, 1);
}

// Exclusive scan of count[0..n) into start[0..n] and cursor[0..n), one CTA.
__global__ void __launch_bounds__(SCAN_T) k_scan(const int* __restrict__ count, int n,
                                                 int* __restrict__ start, int* __restrict__ cursor) {
  __shared__ int wsum[SCAN_T / 32];
  const int t = threadIdx.x;
  const int chunk = (n + SCAN_T - 1) / SCAN_T;
  const int b = min(t * chunk, n), e = min(b + chunk, n);
  int sum = 0;
  for (int q = b; q < e; q++) sum += count[q];
  // block exclusive scan of the per-thread sums
  int v = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if ((t & 31) >= o) v += u;
  }
  if ((t & 31) == 31) wsum[t >> 5] = v;
  __syncthreads();
  if (t < 32) {
    int w = wsum[t];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, w, o);
      if (t >= o) w += u;
    }
    wsum[t] = w;  // inclusive over warps
  }
  __syncthreads();
  int run = v - sum + ((t >> 5) > 0 ? wsum[(t >> 5) - 1] : 0);
  for (int q = b; q < e; q++) {
    start[q] = run;
    cursor[q] = run;
    run += count[q];
  }
  if (t == SCAN_T - 1) start[n] = run;
}

template <int D>
__global__ void k_fill(AdjArgs g, const double* __restrict__ x, int* __restrict__ cursor,
                       int* __restrict__ idx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.N) return;
  int c = 0, mult = 1;
#pragma unroll
  for (int k = 0; k < D; k++) {
    c += cell_of(g, k, x[(size_t)i * D + k]) * mult;
    mult *= g.nc[k];
  }
  idx[atomicAdd(cursor + c, 1)] = i;
}

// Members of each cell in index order, and their float32 positions in the
// same order (the screen of the pair kernels); clears the counts for the
// next build.
template <int D>
__global__ void k_cell_sort(int ncell, const double* __restrict__ x,
                            const int* __restrict__ start, int* __restrict__ idx,
                            float* __restrict__ xs, int* __restrict__ count) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int b = start[c], e = start[c + 1];
  for (int p = b + 1; p < e; p++) {
    const int v = idx[p];
    int q = p - 1;
    while (q >= b && idx[q] > v) {
      idx[q + 1] = idx[q];
      q--;
    }
    idx[q + 1] = v;
  }
  for (int p = b; p < e; p++) {
    const int j = idx[p];
#pragma unroll
    for (int k = 0; k < D; k++) xs[(size_t)p * D + k] = (float)x[(size_t)j * D + k];
  }
  count[c] = 0;
}

// Neighbour list of one state (or of R states: the screen distance then
// includes twice the allowed displacement).  TPP lanes per particle i: lane l takes the
// members l, l + TPP, ... of each of the 3^D cells around i's cell (cells in
// a fixed order, members in index order) that pass the float32 distance
// screen and keeps them in its own sub-list nbr[(i * TPP + l) * W + e],
// e < min(count, W); ncnt[l * N + i] = count.  maxcnt receives the largest
// count (the caller enlarges W and repeats when it exceeds W).
template <int D>
__global__ void __launch_bounds__(BLK) k_adj_list(AdjArgs g, const double* __restrict__ x,
                                                  const int* __restrict__ start,
                                                  const int* __restrict__ idx,
                                                  const float* __restrict__ xs, int W,
                                                  int* __restrict__ nbr, int* __restrict__ ncnt,
                                                  int* __restrict__ maxcnt,
                                                  float* __restrict__ xr) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = t % TPP, i = t / TPP;
  int cnt = 0;
  if (i < g.N) {
    int c[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    float xf[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < D; k++) {
      const double xk = x[(size_t)i * D + k];
      xf[k] = (float)xk;
      c[k] = cell_of(g, k, xk);
      if (g.nc[k] >= 3) {
        lo[k] = c[k] - 1;
        hi[k] = c[k] + 1;
      } else {
        lo[k] = 0;
        hi[k] = g.nc[k] - 1;
      }
    }
    for (int cz = lo[2]; cz <= hi[2]; cz++)
      for (int cy = lo[1]; cy <= hi[1]; cy++)
        for (int cx = lo[0]; cx <= hi[0]; cx++) {
          const int cc[3] = {cx, cy, cz};
          int cell = 0, mult = 1;
#pragma unroll
          for (int k = 0; k < D; k++) {
            int ck = cc[k];
            if (ck < 0) ck += g.nc[k];
            else if (ck >= g.nc[k]) ck -= g.nc[k];
            cell += ck * mult;
            mult *= g.nc[k];
          }
          const int e = start[cell + 1];
          for (int p = start[cell] + lane; p < e; p += TPP) {
            float r2f = 0.f;
#pragma unroll
            for (int k = 0; k < D; k++) {
              float v = xs[(size_t)p * D + k] - xf[k];
              v -= g.Lf[k] * rintf(v * g.Linvf[k]);
              r2f += v * v;
            }
            if (r2f > g.cut2f) continue;
            const int j = idx[p];
            if (j == i) continue;
            if (cnt < W) nbr[((size_t)i * TPP + lane) * W + cnt] = j;
            cnt++;
          }
        }
    ncnt[(size_t)lane * g.N + i] = cnt;
    if (xr && lane == 0) {  // positions of this list, for the displacement check
#pragma unroll
      for (int k = 0; k < D; k++) xr[(size_t)i * D + k] = xf[k];
    }
  }
  const int m = __reduce_max_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(maxcnt, m);
}

// Float32 value of a coordinate from the high word of its float64 (20 bits of
// the significand; Law::screen2 allows for what that leaves out);
// coordinates far outside the box are wrapped first.
__device__ inline float screen_coord(const AdjArgs& g, int k, const double* p) {
  const uint32_t h = reinterpret_cast<const uint32_t*>(p)[1];
  const uint32_t m = h & 0x7fffffffu;
  const float v = __uint_as_float((m < (897u << 20) ? 0u : (m - (896u << 20)) << 3) | (h & 0x80000000u));
  if (!(fabsf(v) <= 2.f * g.Lf[k])) {
    const double x = *p;
    return (float)(x - g.L[k] * floor(x / g.L[k]));
  }
  return v;
}

// 1 / r2 to within about one ulp: the float32 reciprocal and two Newton steps.
__device__ inline double recip_d(double r2) {
  const float f = (float)r2;
  if (!(f > 1e-30f && f < 1e30f)) return 1.0 / r2;
  double w = (double)(1.0f / f);
  w = fma(w, fma(-r2, w, 1.0), w);
  return fma(w, fma(-r2, w, 1.0), w);
}

// Displacement x_j - x_i, minimum image (float64; the float32 value decides the
// image unless the box is so small that a pair in range can be half a box long).
template <int D>
__device__ inline double pair_vec(const AdjArgs& g, const double* __restrict__ x, int i, int j,
                                  double* d) {
  double r2 = 0.0;
#pragma unroll
  for (int k = 0; k < D; k++) {
    double v = __dadd_rn(x[(size_t)j * D + k], -x[(size_t)i * D + k]);
    if (g.exact_image) {
      if (!(fabs(v) < 0.49 * g.L[k])) v -= g.L[k] * rint(v / g.L[k]);
    } else {
      const float q = rintf((float)v * g.Linvf[k]);
      if (q != 0.f) v = fma(-(double)q, g.L[k], v);
    }
    d[k] = v;
    r2 = k == 0 ? __dmul_rn(v, v) : fma(v, v, r2);
  }
  return r2;
}

// One law at squared distance r2 < rc2, in the form the kernels use it:
// U, fr = f / r, fp = f' and the derivatives of U and f / r by
// (u0, r0).  Lennard-Jones laws of even power take a reciprocal, no root.
struct PairD {
  double U, fr, fp, dU[2], dfr[2], w;
};

template <bool LJ>
__device__ inline PairD eval_pair_d(const Law& l, double r2) {
  PairD p;
  if (LJ) {
    const double w = recip_d(r2), n = (double)l.n;
    double s;  // (r0 / r)^n
    if (l.n == 6) {
      const double q = __dmul_rn(l.r02, w);
      s = __dmul_rn(__dmul_rn(q, q), q);
    } else if ((l.n & 1) == 0) {
      const double q = __dmul_rn(l.r02, w);
      s = q;
      for (int e = 2; e < l.n; e += 2) s = __dmul_rn(s, q);
    } else {
      const double q = sqrt(__dmul_rn(l.r02, w));
      s = q;
      for (int e = 1; e < l.n; e++) s = __dmul_rn(s, q);
    }
    const double t = __dmul_rn(2.0 * n, __dmul_rn(s, w));  // 2 n s / r^2
    p.w = w;
    p.U = l.u0 * s * (s - 2.0);
    p.dfr[0] = __dmul_rn(-t, __dadd_rn(s, -1.0));
    p.fr = __dmul_rn(l.u0, p.dfr[0]);
    p.fp = l.u0 * t * fma(2.0 * n + 1.0, s, -(n + 1.0));
    p.dU[0] = s * (s - 2.0);
    p.dU[1] = 2.0 * n * l.u0 * s * (s - 1.0) * l.ir0;
    p.dfr[1] = -l.u0 * t * n * fma(2.0, s, -1.0) * l.ir0;
  } else {
    // Yukawa: U = u0 e / r, e = exp(-r / r0)
    const double ir = rsqrt(r2), r = __dmul_rn(r2, ir), ir0 = l.ir0;
    const double e = exp(__dmul_rn(-r, ir0));
    const double eir = __dmul_rn(e, ir);                   // e / r
    const double h = __dmul_rn(eir, __dadd_rn(ir0, ir));   // e (1 / (r r0) + 1 / r^2)
    p.w = __dmul_rn(ir, ir);
    p.U = l.u0 * eir;
    p.dfr[0] = __dmul_rn(-h, ir);
    p.fr = __dmul_rn(l.u0, p.dfr[0]);
    p.fp = l.u0 * eir * (ir0 * ir0 + 2.0 * ir * ir0 + 2.0 * p.w);
    p.dU[0] = eir;
    p.dU[1] = l.u0 * e * ir0 * ir0;
    p.dfr[1] = -l.u0 * eir * ir0 * ir0 * ir0;
  }
  return p;
}

// The pair terms of a warp's PW particles.  32 / PW lanes per particle screen
// its four sub-lists in float32; the pairs inside a law's cutoff are queued by
// kind of law, 32 of a kind are evaluated with every lane busy, and each
// sub-list's terms are added in list order (one running sum per sub-list, kind
// and component), so results do not depend on PW.  Measured on the mixture at
// 16,384 / 1,001 particles, against four lanes per particle walking their
// sub-lists: see k_adj_step and k_adj_back.
// NS: terms held per kind.
template <int NC, int PW, int NS = 128>
struct PairQueue {
  static constexpr int CH = PW * TPP;           // sub-lists of the warp
  static constexpr int CAP = NS / CH;           // terms per sub-list and kind
  static_assert(CAP >= 32 / CH, "a round fits");
  static constexpr int SLOTS = CH * CAP;
  double term[SLOTS][NC];
  double acc[CH][NC];
  int j[SLOTS];
  unsigned short slot[SLOTS];
  unsigned char law[SLOTS];
  int n[CH];
};

// Runs term(p, i, j, law, kind, out[NC]) for every pair of the warp's
// particles and adds the results to q[kind].acc.  ti, i, cnt: the lane's
// particle (p = lane / LPP of the warp), its type and its sub-list's length
// (sub-list sub % TPP); i0: the warp's first particle.
template <int D, int NC, int PW, int NS, class Term>
__device__ inline void for_pairs(const AdjArgs& g, const Law* laws, PairQueue<NC, PW, NS>* q,
                                 const double* __restrict__ x, const int* __restrict__ nbr, int W,
                                 const int* __restrict__ types, int i0, int i, int ti, int cnt,
                                 Term&& term) {
  typedef PairQueue<NC, PW, NS> Queue;
  constexpr int LPP = 32 / PW, CAP = Queue::CAP, STEP = LPP / TPP;  // entries per round
  const int l32 = threadIdx.x & 31, p = l32 / LPP, sub = l32 % LPP, c = p * TPP + sub % TPP;
  for (int e = l32; e < 2 * Queue::CH; e += 32) {
    q[e & 1].n[e >> 1] = 0;
#pragma unroll
    for (int k = 0; k < NC; k++) q[e & 1].acc[e >> 1][k] = 0.0;
  }
  __syncwarp();
  int queued[2] = {0, 0};  // the same on every lane
  auto flush = [&](auto kind) {
    constexpr int K = decltype(kind)::value;
    Queue& f = q[K];
    __syncwarp();
    for (int e = l32; e < queued[K]; e += 32) {
      const int slot = f.slot[e];
      double out[NC];
      term(kind, i0 + slot / (TPP * CAP), f.j[e], laws[f.law[e]], (int)f.law[e], out);
#pragma unroll
      for (int k = 0; k < NC; k++) f.term[slot][k] = out[k];
    }
    __syncwarp();
    for (int e = l32; e < Queue::CH * NC; e += 32) {
      const int cc = e / NC, k = e % NC, n = f.n[cc];
      double v = f.acc[cc][k];
      for (int t = 0; t < n; t++) v = __dadd_rn(v, f.term[cc * CAP + t][k]);
      f.acc[cc][k] = v;
    }
    __syncwarp();
    for (int e = l32; e < Queue::CH; e += 32) f.n[e] = 0;
    queued[K] = 0;
    __syncwarp();
  };
  float xi[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < D; k++) xi[k] = screen_coord(g, k, x + (size_t)i * D + k);
  // lanes of the same sub-list
  unsigned int peers = 0u;
#pragma unroll
  for (int e = 0; e < LPP; e++)
    if (e % TPP == sub % TPP) peers |= 1u << (p * LPP + e);
  const unsigned int below = (1u << l32) - 1u;
  const int* row = nbr + ((size_t)i * TPP + sub % TPP) * W;
  const int rounds = (__reduce_max_sync(0xffffffffu, cnt) + STEP - 1) / STEP;
  int e = sub / TPP;
  int jn = e < cnt ? row[e] : -1;
  for (int r = 0; r < rounds; r++) {
    const int j = jn;
    e += STEP;
    jn = e < cnt ? row[e] : -1;
    unsigned int m = 0u;  // laws the pair is inside of
    if (j >= 0) {
      float r2 = 0.f;
#pragma unroll
      for (int k = 0; k < D; k++) {
        float v = screen_coord(g, k, x + (size_t)j * D + k) - xi[k];
        v -= g.Lf[k] * rintf(v * g.Linvf[k]);
        r2 += v * v;
      }
      for (unsigned int mm = g.lawmask[ti * MAXT + types[j]]; mm; mm &= mm - 1u) {
        const int l = __ffs(mm) - 1;
        if (r2 < laws[l].screen2) m |= 1u << l;
      }
    }
    while (__any_sync(0xffffffffu, m)) {  // each lane's next law
      const int l = m ? __ffs(m) - 1 : 0;
      const int kind = m ? (laws[l].law == RDSIM_LAW_LJ ? 0 : 1) : -1;
      m &= m - 1u;
#pragma unroll
      for (int K = 0; K < 2; K++) {
        const unsigned int b = __ballot_sync(0xffffffffu, kind == K), mine = b & peers;
        if (!b) continue;
        Queue& f = q[K];
        const int n = f.n[c];
        __syncwarp();
        if (kind == K) {
          const int at = queued[K] + __popc(b & below);
          f.j[at] = j;
          f.law[at] = (unsigned char)l;
          f.slot[at] = (unsigned short)(c * CAP + n + __popc(mine & below));
        }
        if (!(peers & below)) f.n[c] = n + __popc(mine);
        queued[K] += __popc(b);
        __syncwarp();
        // room for another round in every sub-list
        if (__any_sync(0xffffffffu, f.n[c] > CAP - STEP)) {
          if (K == 0) flush(std::integral_constant<int, 0>{});
          else flush(std::integral_constant<int, 1>{});
        }
      }
    }
  }
  flush(std::integral_constant<int, 0>{});
  flush(std::integral_constant<int, 1>{});
}

// Component k of particle p's sum over its sub-lists and kinds (in the order of
// a xor tree over four lanes).
template <int NC, int PW, int NS>
__device__ inline double pair_sum(const PairQueue<NC, PW, NS>* q, int p, int k) {
  double c[TPP];
#pragma unroll
  for (int l = 0; l < TPP; l++) c[l] = __dadd_rn(q[0].acc[p * TPP + l][k], q[1].acc[p * TPP + l][k]);
  return __dadd_rn(__dadd_rn(c[0], c[1]), __dadd_rn(c[2], c[3]));
}

// One state: loss terms (F_LOSS, accumulated per particle into lacc) and the
// step to the next state (F_STEP).  Mixture, step only: 70 -> 35 us at 16,384
// particles (57 % of the float64 pipe), 30 -> 10 us at 1,001.
template <int D, int FL, int PW>
__global__ void __launch_bounds__(BLK) k_adj_step(AdjArgs g, const double* __restrict__ x,
                                                  const int* __restrict__ nbr,
                                                  const int* __restrict__ ncnt, int W,
                                                  const int* __restrict__ types,
                                                  const double* __restrict__ noise,
                                                  double* __restrict__ x_out,
                                                  double* __restrict__ lacc,
                                                  const float* __restrict__ xr,
                                                  int* __restrict__ moved) {
  constexpr int LPP = 32 / PW, PER = BLK / 32 * PW;
  constexpr bool LOSS = (FL & F_LOSS) != 0;
  constexpr int NC = D + (LOSS ? 1 : 0);
  __shared__ Law slaws[MAXL];
  __shared__ PairQueue<NC, PW> queue[BLK / 32][2];
  if (threadIdx.x < (unsigned)g.nlaws) slaws[threadIdx.x] = g.laws[threadIdx.x];
  __syncthreads();
  const int warp = threadIdx.x >> 5, l32 = threadIdx.x & 31, sub = l32 % LPP;
  const int i0 = (int)blockIdx.x * PER + warp * PW;
  const bool own = i0 + l32 / LPP < g.N;
  const int i = own ? i0 + l32 / LPP : g.N - 1;
  const int cnt = own ? min(ncnt[(size_t)(sub % TPP) * g.N + i], W) : 0;
  for_pairs<D>(g, slaws, queue[warp], x, nbr, W, types, i0, i, types[i], cnt,
                       [&](auto kind, int gi, int gj, const Law& w, int, double* out) {
    double d[3];
    const double r2 = pair_vec<D>(g, x, gi, gj, d);
    if (!(r2 < w.rc2)) {
#pragma unroll
      for (int k = 0; k < NC; k++) out[k] = 0.0;
      return;
    }
    const PairD e = eval_pair_d<decltype(kind)::value == 0>(w, r2);
#pragma unroll
    for (int k = 0; k < D; k++) out[k] = __dmul_rn(e.fr, d[k]);
    // each pair is seen from both ends: half of its loss on each
    if (LOSS) out[NC - 1] = 0.5 * (g.wU * (e.U - w.Uc) - g.wW * r2 * e.fr);
  });
  __syncthreads();
  // one thread per particle and component
  const int t = threadIdx.x;
  if (t >= PER * NC) return;
  const int pq = t / NC, k = t % NC, ip = (int)blockIdx.x * PER + pq;
  if (ip >= g.N) return;
  const double v = pair_sum(queue[pq / PW], pq % PW, k);
  if (LOSS && k == D) {
    lacc[ip] += v;
    return;
  }
  const int ti = types[ip];
  const double xk = x[(size_t)ip * D + k];
  if (xr && k == 0) {
    // the list in use dates from an earlier state: it holds every pair in
    // range only while no particle has moved more than the skin allows
    float d2 = 0.f;
#pragma unroll
    for (int c = 0; c < D; c++) {
      float u = (float)x[(size_t)ip * D + c] - xr[(size_t)ip * D + c];
      u -= g.Lf[c] * rintf(u * g.Linvf[c]);
      d2 += u * u;
    }
    if (d2 > g.move2f) atomicOr(moved, 1);
  }
  if (FL & F_STEP) {
    double y = fma(g.c[ti], v, xk);
    y = fma(g.s[ti], noise[(size_t)ip * D + k], y);
    const double L = k == 0 ? g.L[0] : (k == 1 ? g.L[1] : g.L[2]);
    if (!(y >= 0.0 && y < L)) y -= L * floor(y / L);
    x_out[(size_t)ip * D + k] = y;
  }
}

// One state of the backward pass (see the file comment).  gpart[block][NG]
// accumulates this CTA's parameter gradients over the steps, in step order.
// Mixture, step only / with loss terms: 128 / 162 -> 63 / 79 us at 16,384
// particles, 51 / 62 -> 13 / 14 us at 1,001.
template <int D, int FL, int PW>
__global__ void __launch_bounds__(BLK) k_adj_back(AdjArgs g, const double* __restrict__ x,
                                                  const int* __restrict__ nbr,
                                                  const int* __restrict__ ncnt, int W,
                                                  const int* __restrict__ types,
                                                  const double* __restrict__ lam_next,
                                                  double* __restrict__ lam_out,
                                                  double* __restrict__ gpart) {
  constexpr int LPP = 32 / PW, PER = BLK / 32 * PW;
  __shared__ Law slaws[MAXL];
  __shared__ PairQueue<D, PW, D == 3 ? 64 : 128> queue[BLK / 32][2];  // (48 KB in all)
  __shared__ double sgp[NG][BLK + 1];  // per-thread parameter gradients
  const int tid = threadIdx.x;
  if (tid < g.nlaws) slaws[tid] = g.laws[tid];
  for (int q = 0; q < 2 * g.nlaws; q++) sgp[q][tid] = 0.0;
  __syncthreads();
  const int warp = tid >> 5, l32 = tid & 31, sub = l32 % LPP;
  const int i0 = (int)blockIdx.x * PER + warp * PW;
  const bool own = i0 + l32 / LPP < g.N;
  const int i = own ? i0 + l32 / LPP : g.N - 1;
  const int cnt = own ? min(ncnt[(size_t)(sub % TPP) * g.N + i], W) : 0;
  for_pairs<D>(g, slaws, queue[warp], x, nbr, W, types, i0, i, types[i], cnt,
                      [&](auto kind, int gi, int gj, const Law& w, int l, double* out) {
    double d[3];
    const double r2 = pair_vec<D>(g, x, gi, gj, d);
#pragma unroll
    for (int k = 0; k < D; k++) out[k] = 0.0;
    if (!(r2 < w.rc2)) return;
    const PairD e = eval_pair_d<decltype(kind)::value == 0>(w, r2);
    double ddw = 0.0;  // d . (w_j - w_i)
    if (FL & F_STEP) {
      const double ci = g.c[types[gi]], cj = g.c[types[gj]];
      double dw[3];
#pragma unroll
      for (int k = 0; k < D; k++) {
        dw[k] = fma(cj, lam_next[(size_t)gj * D + k], -(ci * lam_next[(size_t)gi * D + k]));
        ddw = fma(d[k], dw[k], ddw);
      }
      // f' rhat rhat.dw + (f / r) (dw - rhat rhat.dw)
      const double h = (e.fp - e.fr) * e.w * ddw;
#pragma unroll
      for (int k = 0; k < D; k++) out[k] = fma(h, d[k], e.fr * dw[k]);
    }
    if (FL & F_LOSS) {
      // d loss_pair / dr times d r / d x_i = -rhat
      const double dl = g.wU * e.fr - g.wW * (e.fr + e.fp);
#pragma unroll
      for (int k = 0; k < D; k++) out[k] = fma(-dl, d[k], out[k]);
    }
    if (gj > gi) {
#pragma unroll
      for (int q = 0; q < 2; q++) {
        double v = 0.0;
        if (FL & F_STEP) v -= e.dfr[q] * ddw;  // df/dtheta rhat . (w_i - w_j)
        if (FL & F_LOSS)
          v += g.wU * (e.dU[q] - (q == 0 ? w.dUc_du0 : w.dUc_dr0)) - g.wW * r2 * e.dfr[q];
        sgp[2 * l + q][tid] += v;
      }
    }
  });
  __syncthreads();
  if (tid < PER * D) {
    const int pq = tid / D, k = tid % D, ip = (int)blockIdx.x * PER + pq;
    if (ip < g.N) {
      const double v = pair_sum(queue[pq / PW], pq % PW, k);
      lam_out[(size_t)ip * D + k] = v + ((FL & F_STEP) ? lam_next[(size_t)ip * D + k] : 0.0);
    }
  }
  // CTA sum of the parameter gradients in a fixed order (eight threads per
  // parameter), added to this CTA's slot
  static_assert(BLK == 8 * NG, "eight threads per parameter");
  {
    const int q = tid / 8, part = tid % 8;
    double v = 0.0;
    if (q < 2 * g.nlaws)
      for (int u = 0; u < BLK / 8; u++) v += sgp[q][u * 8 + part];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (part == 0 && q < 2 * g.nlaws) gpart[(size_t)blockIdx.x * NG + q] += v;
  }
}

// Sum of n values (or n rows of NG values) in a fixed order: one CTA per column,
// thread t adds entries t, t + SUM_T, ..., then a fixed tree.  (One CTA of 128
// threads for all columns: 16 us of latency; now 4 us.)
constexpr int SUM_T = 512;
__global__ void __launch_bounds__(SUM_T) k_sum_rows(const double* __restrict__ v, int n, int width,
                                                    double* __restrict__ out) {
  __shared__ double sh[SUM_T];
  const int col = blockIdx.x;
  {
    double s = 0.0;
    for (int r = threadIdx.x; r < n; r += SUM_T) s += v[(size_t)r * width + col];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = SUM_T / 2; o > 0; o >>= 1) {
      if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[col] = sh[0];
  }
}

__global__ void k_scale(double* v, size_t n, double f) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] *= f;
}

unsigned nblk(int n) { return (unsigned)((n + BLK - 1) / BLK); }
// CTAs of the list kernel (TPP lanes per particle) and of the pair kernels
unsigned lblk(int n) { return nblk(n * TPP); }
// Particles per warp of the float64 pair kernels.  Loss and gradients at 2 / 4 /
// 8 per warp: 1.45 / 1.62 / 2.24 ms for 16 steps at 1,001 particles, 3.30 / 2.97
// / 3.95 ms for 32 steps at 4,096, 7.67 / 6.15 / 6.08 ms at 16,384.
int pair_width(int n) { return n <= 2500 ? 2 : 4; }
unsigned pblk(int n) {
  const int per = BLK / 32 * pair_width(n);
  return (unsigned)((n + per - 1) / per);
}

}  // namespace

struct rdsim_adjoint {
  int device = 0;
  cudaStream_t stream = nullptr;
  AdjArgs g;
  std::vector<rdsim_interaction> laws;
  int K = 1, E = 32;
  int* types = nullptr;
  // cells of the state being listed (transient)
  int *count = nullptr, *cursor = nullptr, *start = nullptr, *idx = nullptr;
  float* xs = nullptr;             // [N][D] float32 positions in cell order
  // neighbour lists of the segment's states: E + 1 slots of nbr[W][N], ncnt[N]
  int W = 0;
  int *seg_nbr = nullptr, *seg_ncnt = nullptr;
  int* maxcnt = nullptr;
  // list reuse: one list serves R consecutive states (R divides E) when no
  // particle moves more than the skin allows in between
  int R = 1, R_used = 1;
  float cut2f_exact = 0.f, cut2f_skin = 0.f;
  float* xr = nullptr;             // [N][D] float32 positions of the forward list
  int* moved = nullptr;
  double* seg_x = nullptr;         // [E][N][D] states of the current segment
  double* ckpt = nullptr;          // [nckpt][N][D] states 0, E, 2E, ...
  size_t ckpt_cap = 0;
  double* xT = nullptr;            // [N][D] final state
  double* lacc = nullptr;          // [N] per-particle loss
  double* lam[2] = {nullptr, nullptr};
  double* gpart = nullptr;         // [blocks][NG]
  double* red = nullptr;           // [NG] reduction results
  const double* xi = nullptr;      // noise of the last forward (caller's)
  int T = -1;                      // steps of the last forward
};

namespace {

void free_adj(rdsim_adjoint* h) {
  auto F = [](void* p) {
    if (p) cudaFree(p);
  };
  F(h->types); F(h->count); F(h->cursor); F(h->start); F(h->idx); F(h->xs);
  F(h->seg_nbr); F(h->seg_ncnt); F(h->maxcnt); F(h->seg_x); F(h->xr); F(h->moved);
  F(h->ckpt); F(h->xT); F(h->lacc); F(h->lam[0]); F(h->lam[1]); F(h->gpart); F(h->red);
  if (h->stream) cudaStreamDestroy(h->stream);
}

int* slot_nbr(rdsim_adjoint* h, int s) { return h->seg_nbr + (size_t)s * h->W * TPP * h->g.N; }
int* slot_ncnt(rdsim_adjoint* h, int s) { return h->seg_ncnt + (size_t)s * TPP * h->g.N; }

// (Re)allocates the neighbour-list slots for width W.
int alloc_lists(rdsim_adjoint* h, int W) {
  if (h->seg_nbr) cudaFree(h->seg_nbr);
  h->seg_nbr = nullptr;
  h->W = 0;
  const size_t slots = (size_t)h->E + 1;
  if (cudaMalloc(&h->seg_nbr, sizeof(int) * slots * W * TPP * h->g.N) != cudaSuccess)
    return fail(RDSIM_ERR_NOMEM, "neighbour lists");
  h->W = W;
  return 0;
}

template <int D>
void build_list_d(rdsim_adjoint* h, const double* x, int slot, float* xr) {
  const AdjArgs& g = h->g;
  k_bin<D><<<nblk(g.N), BLK, 0, h->stream>>>(g, x, h->count);
  k_scan<<<1, SCAN_T, 0, h->stream>>>(h->count, g.ncell, h->start, h->cursor);
  k_fill<D><<<nblk(g.N), BLK, 0, h->stream>>>(g, x, h->cursor, h->idx);
  k_cell_sort<D><<<nblk(g.ncell), BLK, 0, h->stream>>>(g.ncell, x, h->start, h->idx, h->xs,
                                                        h->count);
  k_adj_list<D><<<lblk(g.N), BLK, 0, h->stream>>>(g, x, h->start, h->idx, h->xs, h->W,
                                                   slot_nbr(h, slot), slot_ncnt(h, slot),
                                                   h->maxcnt, xr);
}

// Cells and neighbour list of state x into list slot `slot` (and its float32
// positions into xr when given).
void build_list(rdsim_adjoint* h, const double* x, int slot, float* xr = nullptr) {
  if (h->g.D == 2) build_list_d<2>(h, x, slot, xr);
  else if (h->g.D == 3) build_list_d<3>(h, x, slot, xr);
  else build_list_d<1>(h, x, slot, xr);
}

template <int D, int FL>
void step_k(rdsim_adjoint* h, const double* x, int slot, const double* noise, double* x_out,
            const float* xr) {
  auto k = pair_width(h->g.N) == 2 ? k_adj_step<D, FL, 2> : k_adj_step<D, FL, 4>;
  k<<<pblk(h->g.N), BLK, 0, h->stream>>>(h->g, x, slot_nbr(h, slot), slot_ncnt(h, slot), h->W,
                                         h->types, noise, x_out, h->lacc, xr, h->moved);
}

template <int D>
void step_d(rdsim_adjoint* h, const double* x, int slot, const double* noise, double* x_out,
            int flags, const float* xr) {
  if (flags == F_STEP) step_k<D, F_STEP>(h, x, slot, noise, x_out, xr);
  else if (flags == F_LOSS) step_k<D, F_LOSS>(h, x, slot, noise, x_out, xr);
  else step_k<D, F_STEP | F_LOSS>(h, x, slot, noise, x_out, xr);
}

// One state's kernel (loss terms and/or the step); with xr the displacement
// since the list was built is checked.
void step(rdsim_adjoint* h, const double* x, int slot, const double* noise, double* x_out,
          int flags, const float* xr = nullptr) {
  if (h->g.D == 2) step_d<2>(h, x, slot, noise, x_out, flags, xr);
  else if (h->g.D == 3) step_d<3>(h, x, slot, noise, x_out, flags, xr);
  else step_d<1>(h, x, slot, noise, x_out, flags, xr);
}

template <int D, int FL>
void back_k(rdsim_adjoint* h, const double* x, int slot, const double* lam_next, double* lam_out) {
  auto k = pair_width(h->g.N) == 2 ? k_adj_back<D, FL, 2> : k_adj_back<D, FL, 4>;
  k<<<pblk(h->g.N), BLK, 0, h->stream>>>(h->g, x, slot_nbr(h, slot), slot_ncnt(h, slot), h->W,
                                         h->types, lam_next, lam_out, h->gpart);
}

template <int D>
void back_d(rdsim_adjoint* h, const double* x, int slot, const double* lam_next, double* lam_out,
            int flags) {
  if (flags == F_STEP) back_k<D, F_STEP>(h, x, slot, lam_next, lam_out);
  else if (flags == F_LOSS) back_k<D, F_LOSS>(h, x, slot, lam_next, lam_out);
  else back_k<D, F_STEP | F_LOSS>(h, x, slot, lam_next, lam_out);
}

void back(rdsim_adjoint* h, const double* x, int slot, const double* lam_next, double* lam_out,
          int flags) {
  if (h->g.D == 2) back_d<2>(h, x, slot, lam_next, lam_out, flags);
  else if (h->g.D == 3) back_d<3>(h, x, slot, lam_next, lam_out, flags);
  else back_d<1>(h, x, slot, lam_next, lam_out, flags);
}

}  // namespace

extern "C" {

int rdsim_adjoint_create(const rdsim_adjoint_system* s, int32_t device, rdsim_adjoint** out) {
  if (!s || !out) return fail(RDSIM_ERR_ARG, "null argument");
  *out = nullptr;
  const int D = s->n_dim, N = s->n_particles;
  if (D < 1 || D > 3) return fail(RDSIM_ERR_ARG, "n_dim must be 1, 2 or 3");
  if (N < 1) return fail(RDSIM_ERR_ARG, "no particles");
  if (s->n_types < 1 || s->n_types > MAXT) return fail(RDSIM_ERR_ARG, "n_types out of range");
  if (s->n_laws < 0 || s->n_laws > MAXL) return fail(RDSIM_ERR_UNSUPPORTED, "at most 8 laws");
  if (s->loss_steps < 1) return fail(RDSIM_ERR_ARG, "loss_steps must be >= 1");
  if (s->checkpoint_every < 1) return fail(RDSIM_ERR_ARG, "checkpoint_every must be >= 1");
  auto* h = new rdsim_adjoint();
  std::memset(&h->g, 0, sizeof h->g);
  AdjArgs& g = h->g;
  g.N = N;
  g.D = D;
  g.nlaws = s->n_laws;
  double rc_max = 0.0, V = 1.0;
  h->E = s->checkpoint_every;
  // list reuse: R states per list (R divides E); the skin covers five
  // standard deviations of R diffusion steps of the most mobile type per
  // dimension (a particle that moves farther makes the forward pass repeat
  // itself with one list per state)
  double sig = 0.0;
  for (int t = 0; t < s->n_types; t++)
    if (s->mobility[t] > 0) sig = std::max(sig, std::sqrt(2.0 * s->dt * s->mobility[t]));
  h->R = h->E % 8 == 0 ? 8 : (h->E % 4 == 0 ? 4 : (h->E % 2 == 0 ? 2 : 1));
  const double skin_half = std::max(0.05, 5.0 * sig * std::sqrt((double)h->R) * std::sqrt((double)D));
  for (int l = 0; l < s->n_laws; l++) {
    const rdsim_interaction& it = s->laws[l];
    if (it.law != RDSIM_LAW_LJ && it.law != RDSIM_LAW_YUKAWA) {
      delete h;
      return fail(RDSIM_ERR_UNSUPPORTED, "the adjoint supports lj and yukawa laws");
    }
    if (it.type_a < 0 || it.type_b < it.type_a || it.type_b >= s->n_types || !(it.rc > 0) ||
        !(it.r0 > 0) || (it.law == RDSIM_LAW_LJ && it.n < 1)) {
      delete h;
      return fail(RDSIM_ERR_ARG, "bad law");
    }
    g.lawmask[it.type_a * MAXT + it.type_b] |= (unsigned char)(1u << l);
    g.lawmask[it.type_b * MAXT + it.type_a] |= (unsigned char)(1u << l);
    rc_max = std::max(rc_max, it.rc);
    h->laws.push_back(it);
  }
  double Lmin = 1e300, Lmax = 0.0;
  for (int k = 0; k < D; k++) {
    Lmin = std::min(Lmin, s->L[k]);
    Lmax = std::max(Lmax, s->L[k]);
  }
  // screen distances: float32 positions and minimum image err by a few
  // 1e-7 L per coordinate
  const double cut_exact = rc_max + 1e-3 + 1e-6 * Lmax;
  const double cut_skin = cut_exact + 2.0 * skin_half;
  if (rc_max <= 0 || 2.0 * cut_skin > Lmin) h->R = 1;
  const double cut_cells = h->R > 1 ? cut_skin : cut_exact;
  for (int k = 0; k < D; k++)
    if (!(s->L[k] >= 2.1 * rc_max)) g.exact_image = 1;
  h->cut2f_exact = (float)(cut_exact * cut_exact * (1.0 + 1e-6));
  h->cut2f_skin = (float)(cut_skin * cut_skin * (1.0 + 1e-6));
  {
    const double mv = skin_half - 1e-4 - 1e-6 * Lmax;  // float32 check, conservative
    g.move2f = (float)(mv > 0 ? mv * mv : 0.0);
  }
  for (int k = 0; k < D; k++) {
    if (!(s->L[k] >= 2.0 * rc_max) || !(s->L[k] > 0)) {
      delete h;
      return fail(RDSIM_ERR_ARG, "box length below twice the largest cutoff");
    }
    int nc = rc_max > 0 ? (int)std::floor(s->L[k] / cut_cells) : 1;
    nc = std::min(std::max(nc, 1), 1 << 12);
    if (nc < 3) nc = 1;
    g.nc[k] = nc;
    g.L[k] = s->L[k];
    g.Lf[k] = (float)s->L[k];
    g.Linvf[k] = (float)(1.0 / s->L[k]);
    g.cellinv[k] = nc / s->L[k];
    V *= s->L[k];
  }
  for (int k = D; k < 3; k++) g.nc[k] = 1;
  g.cut2f = h->R > 1 ? h->cut2f_skin : h->cut2f_exact;
  g.ncell = g.nc[0] * g.nc[1] * g.nc[2];
  for (int t = 0; t < s->n_types; t++) {
    const double Dt = s->mobility[t];
    g.c[t] = Dt > 0 ? s->dt * Dt : 0.0;
    g.s[t] = Dt > 0 ? std::sqrt(2.0 * s->dt * Dt) : 0.0;
  }
  h->K = s->loss_steps;
  g.wU = 1.0 / h->K;
  g.wW = 1.0 / (h->K * D * V);
  std::vector<int> types(s->types, s->types + N);
  for (int t : types)
    if (t < 0 || t >= s->n_types) {
      delete h;
      return fail(RDSIM_ERR_ARG, "particle type out of range");
    }
  h->device = device;
  auto bail = [&](int rc) {
    free_adj(h);
    delete h;
    return rc;
  };
  if (cudaSetDevice(device) != cudaSuccess) return bail(fail(RDSIM_ERR_CUDA, "cudaSetDevice"));
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
    return bail(fail(RDSIM_ERR_CUDA, "cudaStreamCreate"));
  const size_t nd = (size_t)N * D;
  const size_t slots = (size_t)h->E + 1;
  bool ok = cudaMalloc(&h->types, sizeof(int) * N) == cudaSuccess &&
            cudaMalloc(&h->count, sizeof(int) * g.ncell) == cudaSuccess &&
            cudaMalloc(&h->cursor, sizeof(int) * g.ncell) == cudaSuccess &&
            cudaMalloc(&h->start, sizeof(int) * (g.ncell + 1)) == cudaSuccess &&
            cudaMalloc(&h->idx, sizeof(int) * N) == cudaSuccess &&
            cudaMalloc(&h->xs, sizeof(float) * nd) == cudaSuccess &&
            cudaMalloc(&h->seg_ncnt, sizeof(int) * slots * TPP * N) == cudaSuccess &&
            cudaMalloc(&h->maxcnt, sizeof(int)) == cudaSuccess &&
            cudaMalloc(&h->xr, sizeof(float) * nd) == cudaSuccess &&
            cudaMalloc(&h->moved, sizeof(int)) == cudaSuccess &&
            cudaMalloc(&h->seg_x, sizeof(double) * h->E * nd) == cudaSuccess &&
            cudaMalloc(&h->xT, sizeof(double) * nd) == cudaSuccess &&
            cudaMalloc(&h->lacc, sizeof(double) * N) == cudaSuccess &&
            cudaMalloc(&h->lam[0], sizeof(double) * nd) == cudaSuccess &&
            cudaMalloc(&h->lam[1], sizeof(double) * nd) == cudaSuccess &&
            cudaMalloc(&h->gpart, sizeof(double) * pblk(N) * NG) == cudaSuccess &&
            cudaMalloc(&h->red, sizeof(double) * NG) == cudaSuccess;
  if (!ok) return bail(fail(RDSIM_ERR_NOMEM, "device allocation failed"));
  {
    // sub-list width: twice the expected number of particles within the
    // screen distance per lane, plus a margin (a forward pass that finds
    // more widens it)
    const double cut = std::sqrt((double)g.cut2f);
    const double ball = D == 1 ? 2.0 * cut : (D == 2 ? M_PI * cut * cut : 4.0 / 3.0 * M_PI * cut * cut * cut);
    const double expect = std::min((double)N, N / V * ball) / TPP;
    const int W = (int)(2.0 * expect) + 8;
    int rc = alloc_lists(h, std::min(W, N));
    if (rc) return bail(rc);
  }
  if (cudaMemcpyAsync(h->types, types.data(), sizeof(int) * N, cudaMemcpyHostToDevice, h->stream) !=
          cudaSuccess ||
      cudaMemsetAsync(h->count, 0, sizeof(int) * g.ncell, h->stream) != cudaSuccess ||
      cudaStreamSynchronize(h->stream) != cudaSuccess)
    return bail(fail(RDSIM_ERR_CUDA, "upload"));
  *out = h;
  return 0;
}

int rdsim_adjoint_destroy(rdsim_adjoint* h) {
  if (!h) return 0;
  cudaSetDevice(h->device);
  free_adj(h);
  delete h;
  return 0;
}

int rdsim_adjoint_get_lists(rdsim_adjoint* h, int32_t* states_per_list, int32_t* list_width) {
  if (!h || !states_per_list || !list_width) return fail(RDSIM_ERR_ARG, "null argument");
  *states_per_list = h->R_used;
  *list_width = h->W;
  return 0;
}

int rdsim_adjoint_get_stream(rdsim_adjoint* h, void** stream) {
  if (!h || !stream) return fail(RDSIM_ERR_ARG, "null argument");
  *stream = (void*)h->stream;
  return 0;
}

int rdsim_adjoint_forward(rdsim_adjoint* h, const double* x0, const double* params,
                          const double* xi, int32_t n_steps, double* loss, double* x_final) {
  if (!h || !x0 || !params || !loss || (n_steps > 0 && !xi)) return fail(RDSIM_ERR_ARG, "null argument");
  if (n_steps < 0) return fail(RDSIM_ERR_ARG, "n_steps must be >= 0");
  if (h->K > n_steps + 1) return fail(RDSIM_ERR_ARG, "loss_steps exceeds the number of states");
  CK(cudaSetDevice(h->device));
  AdjArgs& g = h->g;
  for (int l = 0; l < g.nlaws; l++) {
    const rdsim_interaction& it = h->laws[l];
    Law& w = g.laws[l];
    w.law = it.law;
    w.n = it.n;
    w.u0 = params[2 * l];
    w.r0 = params[2 * l + 1];
    w.rc = it.rc;
    if (!(w.r0 > 0)) return fail(RDSIM_ERR_ARG, "r0 must be positive");
    w.ir0 = 1.0 / w.r0;
    w.r02 = w.r0 * w.r0;
    w.rc2 = w.rc * w.rc;
    // the screen's coordinates carry 20 bits each: at most 2^-20 of twice the
    // box per coordinate, and the float32 arithmetic a few 1e-7 of it
    double Lmax = 0.0;
    for (int k = 0; k < g.D; k++) Lmax = std::max(Lmax, g.L[k]);
    const double cut = w.rc + 8.0 * std::sqrt((double)g.D) * std::ldexp(Lmax, -20) + 1e-4;
    w.screen2 = (float)(cut * cut * (1.0 + 1e-6));
    const PairEval p = eval_law(w, w.rc, 1.0 / w.rc);
    w.Uc = p.U;
    w.dUc_du0 = p.dU[0];
    w.dUc_dr0 = p.dU[1];
  }
  const int N = g.N, D = g.D, E = h->E;
  const size_t nd = (size_t)N * D;
  const size_t nck = (size_t)n_steps / E + 1;
  if (nck * nd > h->ckpt_cap) {
    if (h->ckpt) cudaFree(h->ckpt);
    h->ckpt = nullptr;
    h->ckpt_cap = 0;
    if (cudaMalloc(&h->ckpt, sizeof(double) * nck * nd) != cudaSuccess)
      return fail(RDSIM_ERR_NOMEM, "checkpoint buffer");
    h->ckpt_cap = nck * nd;
  }
  const double* cur = nullptr;
  int R = h->R;
  for (int attempt = 0;; attempt++) {
    g.cut2f = R > 1 ? h->cut2f_skin : h->cut2f_exact;
    CK(cudaMemsetAsync(h->lacc, 0, sizeof(double) * N, h->stream));
    CK(cudaMemsetAsync(h->maxcnt, 0, sizeof(int), h->stream));
    CK(cudaMemsetAsync(h->moved, 0, sizeof(int), h->stream));
    CK(cudaMemcpyAsync(h->ckpt, x0, sizeof(double) * nd, cudaMemcpyDeviceToDevice, h->stream));
    // states between checkpoints alternate between seg_x[0] and seg_x[1]
    // (the segment buffer is free during the forward pass; E >= 2 there)
    cur = h->ckpt;
    const int slot = E;  // list slot of the forward pass
    for (int n = 0; n <= n_steps; n++) {
      int flags = n >= n_steps - h->K + 1 ? F_LOSS : 0;
      double* nxt = nullptr;
      if (n < n_steps) {
        flags |= F_STEP;
        const int m = n + 1;
        nxt = m % E == 0 ? h->ckpt + (size_t)(m / E) * nd : h->seg_x + (size_t)(m & 1) * nd;
      }
      if (n % R == 0) build_list(h, cur, slot, R > 1 ? h->xr : nullptr);
      step(h, cur, slot, n < n_steps ? xi + (size_t)n * nd : nullptr, nxt, flags,
           R > 1 ? h->xr : nullptr);
      if (nxt) cur = nxt;
    }
    CK(cudaGetLastError());
    int mx = 0, moved = 0;
    CK(cudaMemcpyAsync(&mx, h->maxcnt, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(&moved, h->moved, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (mx <= h->W && !moved) break;
    if (attempt > 2) return fail(RDSIM_ERR_CAPACITY, "neighbour list overflow");
    if (moved) {
      R = 1;  // a particle outran the skin: one list per state
    } else {
      // a list row overflowed: widen the lists and run the pass again
      int rc = alloc_lists(h, std::min(N, mx + mx / 4 + 4));
      if (rc) return rc;
    }
  }
  h->R_used = R;
  if (cur != h->xT) CK(cudaMemcpyAsync(h->xT, cur, sizeof(double) * nd, cudaMemcpyDeviceToDevice, h->stream));
  k_sum_rows<<<1, SUM_T, 0, h->stream>>>(h->lacc, N, 1, h->red);
  CK(cudaMemcpyAsync(loss, h->red, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  if (x_final) CK(cudaMemcpyAsync(x_final, h->xT, sizeof(double) * nd, cudaMemcpyDeviceToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->xi = xi;
  h->T = n_steps;
  return 0;
}

int rdsim_adjoint_backward(rdsim_adjoint* h, double dloss, double* grad_x0, double* grad_params) {
  if (!h || !grad_x0 || !grad_params) return fail(RDSIM_ERR_ARG, "null argument");
  if (h->T < 0) return fail(RDSIM_ERR_ARG, "no forward pass to differentiate");
  CK(cudaSetDevice(h->device));
  AdjArgs& g = h->g;
  const int N = g.N, D = g.D, E = h->E, T = h->T;
  const size_t nd = (size_t)N * D;
  CK(cudaMemsetAsync(h->gpart, 0, sizeof(double) * pblk(N) * NG, h->stream));
  CK(cudaMemsetAsync(h->lam[0], 0, sizeof(double) * nd, h->stream));
  const int R = h->R_used;
  g.cut2f = R > 1 ? h->cut2f_skin : h->cut2f_exact;
  const int extra = E;  // list slot of the final state when it starts a list
  int cur = 0;     // lam[cur] holds lambda_{n+1}
  int seg = -1;    // base step of the states held in seg_x
  // states b .. b + E - 1 below T recomputed from checkpoint b / E, with the
  // lists of states b, b + R, ... in slots 0, 1, ... (the forward pass used
  // the list of state floor(n / R) R for state n; R divides E)
  auto segment = [&](int b) -> int {
    if (b == seg) return 0;
    CK(cudaMemcpyAsync(h->seg_x, h->ckpt + (size_t)(b / E) * nd, sizeof(double) * nd,
                       cudaMemcpyDeviceToDevice, h->stream));
    const int last = std::min(b + E - 1, T - 1);
    for (int q = 0; q <= last - b; q++) {
      double* xq = h->seg_x + (size_t)q * nd;
      if (q > 0) step(h, xq - nd, (q - 1) / R, h->xi + (size_t)(b + q - 1) * nd, xq, F_STEP);
      if (q % R == 0) build_list(h, xq, q / R);
    }
    seg = b;
    return 0;
  };
  for (int n = T; n >= 0; n--) {
    const double* x;
    int slot;
    if (n == T) {
      x = h->xT;
      const int r0 = (T / R) * R;
      if (r0 == T) {
        slot = extra;
        build_list(h, x, slot);
      } else {
        const int b = ((T - 1) / E) * E;
        int rc = segment(b);
        if (rc) return rc;
        slot = (r0 - b) / R;
      }
    } else {
      const int b = (n / E) * E;
      int rc = segment(b);
      if (rc) return rc;
      x = h->seg_x + (size_t)(n - b) * nd;
      slot = (n - b) / R;
    }
    int flags = n >= T - h->K + 1 ? F_LOSS : 0;
    if (n < T) flags |= F_STEP;
    back(h, x, slot, h->lam[cur], h->lam[1 - cur], flags);
    cur = 1 - cur;
  }
  CK(cudaGetLastError());
  k_sum_rows<<<NG, SUM_T, 0, h->stream>>>(h->gpart, (int)pblk(N), NG, h->red);
  double gsum[NG];
  CK(cudaMemcpyAsync(gsum, h->red, sizeof gsum, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(grad_x0, h->lam[cur], sizeof(double) * nd, cudaMemcpyDeviceToDevice,
                     h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int q = 0; q < 2 * g.nlaws; q++) grad_params[q] = dloss * gsum[q];
  if (dloss != 1.0) {
    k_scale<<<(unsigned)((nd + BLK - 1) / BLK), BLK, 0, h->stream>>>(grad_x0, nd, dloss);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(h->stream));
  }
  return 0;
}

}  // extern "C"
