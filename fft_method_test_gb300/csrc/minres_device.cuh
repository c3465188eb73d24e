// minres_device.cuh -- the MINRES scalar steps that the last block of a kernel
// runs (kernels_minres.cu, and the inverse x pass of fft_fast.cuh).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"
#include "internal.h"

namespace fp {

// true in every thread of the block that finishes last among the nblk blocks
// of one problem (its partial sums are then all in memory); the counter is reset
__device__ __forceinline__ bool last_block(unsigned int* counter, unsigned int nblk) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned int t = atomicAdd(counter, 1u);
        last = t == nblk - 1;
        if (last) *counter = 0u;
    }
    __syncthreads();
    return last;
}

// z mean and alpha = v . (z_raw - mean) from the apply's partial rows, by one
// whole block; red holds 4 * 32 doubles
__device__ __forceinline__ void alpha_body(MinresScalars* sc, const double* partials, int nparts,
                                           double inv_nb, double* red) {
    if (sc->done) return;
    double o[4];
    sum_rows<4, 4>(partials, nparts, red, o);
    if (threadIdx.x == 0) {
        double corr = 0.0;
        for (int c = 0; c < 3; ++c) {
            sc->zmean[c] = o[c] * inv_nb;
            corr += sc->zmean[c] * sc->vsum[c];
        }
        sc->alpha = o[3] - corr;
    }
}

}  // namespace fp
