// error_reduce.cuh -- the end of the quality kernels: a CTA's six sums into the
// caller's accumulators, and the totals to the host.
#pragma once
#include <cstdint>

#include "decode.h"

namespace goofy_gpu {

// Called by threads 0 .. THREADS - 1 of the CTA (others may have left): sums s
// over them (shuffles, shared memory), adds the totals with one atomic each
// and, with result.host, lets the last CTA of the grid hand them over
// (decode.h).
template <uint32_t THREADS>
__device__ __forceinline__ void reduce_errors(const uint64_t (&in)[6], unsigned long long (*part)[THREADS / 32],
                                              unsigned long long* __restrict__ sums, const ErrorResult& result)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); };
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        unsigned long long v = in[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) part[c][warp] = v;
    }
    sync();
    if (threadIdx.x < 6) {
        unsigned long long t = 0;
        for (uint32_t k = 0; k < THREADS / 32; ++k) t += part[threadIdx.x][k];
        if (t) atomicAdd(&sums[threadIdx.x], t);
    }
    if (!result.host) return;
    __shared__ bool last;
    __threadfence();  // this CTA's sums before its tick
    sync();
    if (threadIdx.x == 0) last = atomicAdd(result.finished, 1u) == gridDim.x - 1u;
    sync();
    if (!last || warp != 0) return;
    __threadfence();  // every CTA's sums after the last tick
    if (lane < 6) result.host[lane] = atomicExch(&sums[lane], 0ull);
    if (lane == 6) *result.finished = 0u;
    __threadfence_system();  // before the word that the host polls
    __syncwarp();
    if (lane == 0)
        asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(result.flag), "r"(result.serial) : "memory");
}

}  // namespace goofy_gpu
