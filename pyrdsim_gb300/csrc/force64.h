// force64.h -- launches of the float64 drift kernels (force64.cu), the
// "plain method" in the reference's own precision.
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace rd {

// Particles per warp of k_force_d for n particles.  us per step of the LJ fluid
// at 2 / 4 / 16 particles per warp: 11.8 / 12.7 / 23.4 at 1,024, 15.5 / 19.3 /
// 28.5 at 4,096, 26.9 / 23.3 / 42.0 at 8,192, 38.9 / 40.6 / 54.1 at 16,384, 129 /
// 106 / 101 at 65,536.
inline int force64_particles(int n) { return n <= 6000 ? 2 : (n <= 40000 ? 4 : 16); }
// Particles per CTA of k_force_d.
inline int force64_chunk(int pw) { return BLOCK / 32 * pw; }

// k_force_d<D, tpp, pw> over `grid` CTAs (runs of force64_chunk(pw) particles).
cudaError_t launch_force64(int D, int tpp, int pw, unsigned grid, cudaStream_t st, const Args& a);
// k_em_d<D>: the stand-alone float64 Euler-Maruyama update.
cudaError_t launch_em64(int D, unsigned grid, cudaStream_t st, const Args& a, const int* sid);

}  // namespace rd
