// error_emulation.h -- TEST ONLY.  CPU definitions of the further intrinsics
// block_error.cuh uses.
#pragma once
#include <cstdint>

// __vabsdiffu4: per-byte absolute difference of unsigned bytes
static inline uint32_t __vabsdiffu4(uint32_t a, uint32_t b)
{
    uint32_t r = 0;
    for (int n = 0; n < 4; ++n) {
        const int x = (a >> (8 * n)) & 0xff, y = (b >> (8 * n)) & 0xff;
        r |= (uint32_t)(x > y ? x - y : y - x) << (8 * n);
    }
    return r;
}

namespace goofy_gpu {
// prmt.b32 with selector nibbles 0..7; fails on any other
static inline uint32_t pick(uint32_t a, uint32_t b, uint32_t sel)
{
    if (sel & 0x8888u) __builtin_trap();
    return __byte_perm(a, b, sel);
}
}  // namespace goofy_gpu
