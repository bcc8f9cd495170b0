// force32.h -- launches of the float32 drift kernel (force32.cu).
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace rd {

// Chunks from which the Lennard-Jones walk's 12 CTAs per SM pay: two rounds of
// the GPU.  With fewer, the next launch finds no free slot to stage its tables
// in (us per step with the general walk / with it: 18.9 / 20.0 at 100,000
// particles, 28.5 / 28.8 at 200,000, 33.9 / 32.9 at 250,000, 130 / 105 at 1,048,576).
constexpr unsigned LJ_MIN_CHUNKS = 2 * 12 * 152;

// lj6: the Lennard-Jones walk (every pair law of every system is then a single
// Lennard-Jones n = 6 law).
cudaError_t launch_force32(int D, int tpp, bool lj6, unsigned chunks, cudaStream_t st,
                           const Args& a);

}  // namespace rd
