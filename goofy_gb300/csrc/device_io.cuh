// device_io.cuh -- global-memory access helpers shared by the encoder kernels.
#pragma once
#include <cstdint>

#include "block_codec.cuh"

namespace goofy_gpu {

// Source pixels are read exactly once: 128-bit loads that skip L1.
//
// These loads are volatile and not .nc: kernels issue them behind pdl_wait(),
// and the compiler may move an asm without a memory operand, and the assembler
// a load of constant memory (.nc, __ldg), ahead of that wait, where the data
// is still the previous kernel's to write (seen with .nc loads in a grid of two
// blocks a thread).
__device__ __forceinline__ uint4 ld_once16(const uint8_t* p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
        : "l"(p));
    return v;
}

// An encoded block.
__device__ __forceinline__ uint2 load_block8(const uint8_t* p)
{
    uint2 v;
    asm volatile("ld.global.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Encoded blocks are written once and not read back by the kernel: streaming store.
__device__ __forceinline__ void st_stream8(uint8_t* p, uint2 v)
{
    asm volatile("st.global.cs.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}

// The same for rows that the next kernel reads again.  Behind the loads above it
// finds less of them in L2 (a 4096^2 texture: mips, then all levels encoded,
// 32.4 us with those, 29.7 with these).
__device__ __forceinline__ uint4 ld_keep16(const uint8_t* p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ uint2 ld_keep8(const uint8_t* p)
{
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t ld_keep4(const uint8_t* p)
{
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// 16 pixel words of the block at `p`: 16-byte aligned rows use one vector load
// each, 4-byte aligned rows four word loads.  Those leave their lines in L1:
// each of a warp's four loads touches every sector of the row, which crossed
// L2 four times without (1996x1532 BC1 4.45 / 3.4 us, ETC1s 5.2 / 4.7).
__device__ __forceinline__ void load_block_rows(const uint8_t* p, size_t stride, bool vec16, uint32_t (&w)[16])
{
    if (vec16) {
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const uint4 v = ld_once16(p + (size_t)y * stride);
            w[4 * y + 0] = v.x;
            w[4 * y + 1] = v.y;
            w[4 * y + 2] = v.z;
            w[4 * y + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int x = 0; x < 4; ++x) w[4 * y + x] = ld_keep4(p + (size_t)y * stride + 4 * x);
    }
}

// Asks L2 for the line at p.  A hint: L2 stays coherent with every later write to it.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// n / d for n < 2^32 with magic = floor((2^32 - 1) / d): the estimate is low by
// at most one, so a single correction makes it exact.
__device__ __forceinline__ uint32_t div_magic(uint32_t n, uint32_t d, uint32_t magic, uint32_t& rem)
{
    uint32_t q = __umulhi(n, magic);
    uint32_t r = n - q * d;
    if (r >= d) {
        ++q;
        r -= d;
    }
    rem = r;
    return q;
}

// Largest i < n with first_unit[i] <= u (first_unit[0] == 0, ascending): the
// image a work unit of a batch belongs to.
__device__ __forceinline__ uint32_t find_image(const uint32_t* first_unit, uint32_t n, uint32_t u)
{
    uint32_t lo = 0, hi = n;  // invariant: first_unit[lo] <= u < first_unit[hi] (first_unit[n] = inf)
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (first_unit[mid] <= u) lo = mid;
        else hi = mid;
    }
    return lo;
}

// etc1BrighnessRangeTocontrolByte (goofy_tc.h:1040-1057) as 128 bytes indexed by range >> 1.
__device__ __forceinline__ void fill_ctrl_lut(uint8_t* lut)
{
    for (uint32_t i = threadIdx.x; i < 128; i += blockDim.x) lut[i] = (uint8_t)etc_control_byte(2 * i);
}

}  // namespace goofy_gpu
