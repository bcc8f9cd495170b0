// force64.cu -- translation unit of the float64 drift kernels (force64.cuh),
// compiled apart from engine.cu so that the two build in parallel.
#include "force64.h"

#include "force64.cuh"
#include "launch.cuh"

namespace rd {

namespace {

typedef void (*ForceKernel)(Args);

template <int D, int TPP>
ForceKernel kernel_of(int pw) {
  return pw == 2 ? k_force_d<D, TPP, 2> : pw == 4 ? k_force_d<D, TPP, 4> : k_force_d<D, TPP, 16>;
}

template <int D>
ForceKernel kernel_of(int tpp, int pw) {
  return tpp == 1   ? kernel_of<D, 1>(pw)
         : tpp == 2 ? kernel_of<D, 2>(pw)
         : tpp == 8 ? kernel_of<D, 8>(pw)
                    : kernel_of<D, 4>(pw);
}

}  // namespace

cudaError_t launch_force64(int D, int tpp, int pw, unsigned grid, cudaStream_t st, const Args& a) {
  launch(D == 2 ? kernel_of<2>(tpp, pw) : D == 3 ? kernel_of<3>(tpp, pw) : kernel_of<1>(tpp, pw),
         grid, LBLOCK, st, a);
  return cudaGetLastError();
}

cudaError_t launch_em64(int D, unsigned grid, cudaStream_t st, const Args& a, const int* sid) {
  if (D == 2) launch(k_em_d<2>, grid, 256, st, a, sid);
  else if (D == 3) launch(k_em_d<3>, grid, 256, st, a, sid);
  else launch(k_em_d<1>, grid, 256, st, a, sid);
  return cudaGetLastError();
}

}  // namespace rd
