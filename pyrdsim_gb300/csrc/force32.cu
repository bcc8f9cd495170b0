// force32.cu -- the float32 drift kernel's variants (a translation unit of its
// own, compiled in parallel with the engine).
#include "force32.h"

#include "launch.cuh"
#include "list.cuh"

namespace rd {
namespace {

typedef void (*ForceKernel)(Args);

template <int D, bool LJ>
ForceKernel kernel_of(int tpp) {
  return tpp == 1   ? k_force_l<D, 1, LJ>
         : tpp == 2 ? k_force_l<D, 2, LJ>
         : tpp == 8 ? k_force_l<D, 8, LJ>
                    : k_force_l<D, 4, LJ>;
}

template <int D>
ForceKernel kernel_of(int tpp, bool lj6) {
  return lj6 ? kernel_of<D, true>(tpp) : kernel_of<D, false>(tpp);
}

}  // namespace

cudaError_t launch_force32(int D, int tpp, bool lj6, unsigned chunks, cudaStream_t st,
                           const Args& a) {
  launch(D == 2 ? kernel_of<2>(tpp, lj6) : D == 3 ? kernel_of<3>(tpp, lj6) : kernel_of<1>(tpp, lj6),
         chunks, LBLOCK, st, a);
  return cudaGetLastError();
}

}  // namespace rd
