// period.h -- launches of the period kernel (period1.cu, period2.cu, period3.cu:
// one translation unit per dimension, compiled in parallel).
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace rd {

// A variant of the period kernel: lanes (chains) per particle, lanes per chain
// (1, 2 or 4; more than 1 only with two chains), with reactions or without.
struct PeriodVariant {
  int D, tpp, lpc;
  bool rx;
};

// One launch over `chunks` CTAs.
cudaError_t launch_period(const PeriodVariant& v, unsigned chunks, cudaStream_t st, const Args& a,
                          const PeriodArgs& p);

// CTAs that are resident per SM at once with stg_max staged particles, kw code
// words per lane and `rows` type pairs (0 if unknown); also allows the largest
// tables.
int period_blocks_per_sm(const PeriodVariant& v, int stg_max, int kw, int rows);

// Records of a launch that no list builder precedes.
void launch_first_records(int D, cudaStream_t st, const Args& a);

// The same for one dimension (its translation unit).
template <int D>
struct PeriodOf {
  static cudaError_t launch(const PeriodVariant& v, unsigned chunks, cudaStream_t st,
                            const Args& a, const PeriodArgs& p);
  static int blocks_per_sm(const PeriodVariant& v, int stg_max, int kw, int rows);
  static void first_records(cudaStream_t st, const Args& a);
};

inline cudaError_t launch_period(const PeriodVariant& v, unsigned chunks, cudaStream_t st,
                                 const Args& a, const PeriodArgs& p) {
  return v.D == 2   ? PeriodOf<2>::launch(v, chunks, st, a, p)
         : v.D == 3 ? PeriodOf<3>::launch(v, chunks, st, a, p)
                    : PeriodOf<1>::launch(v, chunks, st, a, p);
}

inline int period_blocks_per_sm(const PeriodVariant& v, int stg_max, int kw, int rows) {
  return v.D == 2   ? PeriodOf<2>::blocks_per_sm(v, stg_max, kw, rows)
         : v.D == 3 ? PeriodOf<3>::blocks_per_sm(v, stg_max, kw, rows)
                    : PeriodOf<1>::blocks_per_sm(v, stg_max, kw, rows);
}

inline void launch_first_records(int D, cudaStream_t st, const Args& a) {
  if (D == 2) PeriodOf<2>::first_records(st, a);
  else if (D == 3) PeriodOf<3>::first_records(st, a);
  else PeriodOf<1>::first_records(st, a);
}

}  // namespace rd
