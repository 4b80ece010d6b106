// error_reduce.cuh -- the end of the quality kernels: a CTA's error sums into the
// caller's accumulators, and the totals to the host.
#pragma once
#include <cstdint>

#include "block_error.cuh"
#include "decode.h"

namespace goofy_gpu {

// The warp's total of a 32-bit sum, 16 bits at a time.
__device__ __forceinline__ unsigned long long warp_total(uint32_t v)
{
    return __reduce_add_sync(0xffffffffu, v & 0xffffu) +
           ((unsigned long long)__reduce_add_sync(0xffffffffu, v >> 16) << 16);
}

__device__ __forceinline__ unsigned long long warp_total(int32_t v)  // two's complement
{
    return __reduce_add_sync(0xffffffffu, (uint32_t)v & 0xffffu) +
           ((unsigned long long)(long long)__reduce_add_sync(0xffffffffu, v >> 16) << 16);
}

// Called by threads 0 .. THREADS - 1 of the CTA (others may have left): sums e
// and bad over them, adds the totals with one atomic each and, with
// result.host, lets the last CTA of the grid hand them over (decode.h), with
// a kGaveUp for each warp with a lane that `gave_up`.  A
// synchronous call waits for all of this after its last block, so it is kept
// short: the luminosity sum, linear in the others, is formed from the CTA's
// totals; one warp does everything behind the one barrier; the host polls the
// totals themselves, so nothing is fenced for it.  (A 4096^2 BC1 call from Python
// 27.2 us before, 25.0 now.)
template <uint32_t THREADS>
__device__ __forceinline__ void reduce_errors(const ErrorSums& e, uint32_t bad, bool gave_up,
                                              unsigned long long* __restrict__ sums, const ErrorResult& result)
{
    constexpr uint32_t W = THREADS / 32;
    __shared__ unsigned long long part[8][W];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned long long t[8] = {warp_total(e.sq[0]),
                                     warp_total(e.sq[1]),
                                     warp_total(e.sq[2]),
                                     warp_total(e.sq[3]),
                                     warp_total(bad) +
                                         (__any_sync(0xffffffffu, gave_up) && result.host ? kGaveUp : 0ull),
                                     warp_total((int32_t)(e.pos[0] - e.neg[0])),
                                     warp_total((int32_t)(e.pos[1] - e.neg[1])),
                                     warp_total((int32_t)(e.pos[2] - e.neg[2]))};
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 8; ++k) part[k][warp] = t[k];
    asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    if (warp != 0) return;
    unsigned long long v = 0;  // of sum lane / 4
#pragma unroll
    for (uint32_t w = lane & 3u; w < W; w += 4) v += part[lane >> 2][w];
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    const auto of = [&](int k) { return __shfl_sync(0xffffffffu, v, 4 * k); };
    const long long cross = 21 * 72 * (long long)of(5) + 21 * 7 * (long long)of(6) + 72 * 7 * (long long)of(7);
    const unsigned long long luma = 441ull * of(2) + 5184ull * of(1) + 49ull * of(0) + (unsigned long long)(2 * cross);
    v = of(lane & 7u);
    if (lane == 5) v = luma;
    if (lane < 6 && v) atomicAdd(&sums[lane], v);
    if (!result.host) return;
    __threadfence();  // this CTA's sums before its tick
    __syncwarp();
    uint32_t tick = 0;
    if (lane == 0) tick = atomicAdd(result.finished, 1u);
    if (__shfl_sync(0xffffffffu, tick, 0) != gridDim.x - 1u) return;
    __threadfence();  // every CTA's sums after the last tick
    if (lane < 6) {
        const unsigned long long total = atomicExch(&sums[lane], 0ull);
        asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(result.host + lane), "l"(total) : "memory");
    }
    if (lane == 6) *result.finished = 0u;
}

}  // namespace goofy_gpu
