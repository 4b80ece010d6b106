// error_emulation.h -- TEST ONLY.  CPU definition of the further intrinsic
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
