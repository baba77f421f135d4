// overlap3c_prep.cuh -- device helpers shared by the set-up kernels of the 3-center overlap.
#pragma once

#include "aok_internal.h"

namespace aok {

constexpr int kOrder3Max = 2048;
constexpr int kOrder3Threads = 256;
constexpr int kOrder3Per = kOrder3Max / kOrder3Threads;

// Inclusive scan of one value per thread over the kOrder3Threads threads.
__device__ __forceinline__ long long block_scan3(long long v, long long* wtot) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) wtot[w] = v;
    __syncthreads();
    if (w == 0) {
        long long t = lane < kOrder3Threads / 32 ? wtot[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        if (lane < kOrder3Threads / 32) wtot[lane] = t;
    }
    __syncthreads();
    if (w > 0) v += wtot[w - 1];
    __syncthreads();
    return v;
}

}  // namespace aok
