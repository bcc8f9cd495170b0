// force32.h -- launches of the float32 drift kernel (force32.cu).
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace rd {

// lj6: every pair law of every system is a single Lennard-Jones n = 6 law.
cudaError_t launch_force32(int D, int tpp, bool lj6, unsigned chunks, cudaStream_t st,
                           const Args& a);

}  // namespace rd
