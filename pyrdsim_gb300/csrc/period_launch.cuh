// period_launch.cuh -- the period kernel's variants of one dimension and their
// launches (included by period1.cu, period2.cu and period3.cu).
#pragma once

#include "launch.cuh"
#include "period.cuh"
#include "period.h"

namespace rd {
namespace {

typedef void (*PeriodKernel)(Args, PeriodArgs);

template <int D, bool RX>
PeriodKernel kernel_rx(int tpp, int lpc) {
  if (tpp == 2) return lpc == 4 ? k_period<D, 2, 4, RX> : lpc == 2 ? k_period<D, 2, 2, RX> : k_period<D, 2, 1, RX>;
  return tpp == 1 ? k_period<D, 1, 1, RX> : tpp == 8 ? k_period<D, 8, 1, RX> : k_period<D, 4, 1, RX>;
}

template <int D>
PeriodKernel kernel_of(const PeriodVariant& v) {
  return v.rx ? kernel_rx<D, true>(v.tpp, v.lpc) : kernel_rx<D, false>(v.tpp, v.lpc);
}

size_t period_shared(int stg_max, int kw, int rows) {
  return (size_t)stg_max * (sizeof(uint4) + sizeof(int)) + (size_t)rows * sizeof(float4) +
         (size_t)kw * LBLOCK * sizeof(uint32_t);
}

}  // namespace

template <int D>
cudaError_t PeriodOf<D>::launch(const PeriodVariant& v, unsigned chunks, cudaStream_t st,
                                const Args& a, const PeriodArgs& p) {
  launch_dyn(kernel_of<D>(v), chunks, LBLOCK, period_shared(a.stg_max, a.kw, a.rows_max), st, a, p);
  return cudaGetLastError();
}

template <int D>
int PeriodOf<D>::blocks_per_sm(const PeriodVariant& v, int stg_max, int kw, int rows) {
  int nb = 0;
  const size_t dyn = period_shared(stg_max, kw, rows);
  const void* k = (const void*)kernel_of<D>(v);
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)period_shared(STG_LIMIT, KW_LIMIT, MAXT * MAXT)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, LBLOCK, dyn) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nb;
}

template <int D>
void PeriodOf<D>::first_records(cudaStream_t st, const Args& a) {
  rd::launch(k_first_records<D>, (unsigned)((a.n_total + 255) / 256), 256, st, a);
}

}  // namespace rd
