// block_error_host.cpp -- TEST ONLY.  block_error.cuh compiled for the CPU: the
// error sums of whole images, for comparison with the oracle.
#include <cstring>

#include "block_error.cuh"

// sums[6]: squares of bytes 0..3, unsupported blocks, luminosity squares.
// The 32-bit sums are flushed every `every` blocks.
extern "C" void host_emu_errors(int codec, const uint8_t* blocks, const uint8_t* src, unsigned width, unsigned height,
                                unsigned stride, unsigned every, uint64_t* sums)
{
    const unsigned bw = width / 4, bh = height / 4;
    goofy_gpu::ErrorSums s{};
    uint32_t store[8];
    unsigned n = 0;
    auto flush = [&] {
        for (int c = 0; c < 4; ++c) sums[c] += s.sq[c];
        sums[5] += goofy_gpu::luma_sum_of(s);
        s = goofy_gpu::ErrorSums{};
        n = 0;
    };
    for (unsigned by = 0; by < bh; ++by)
        for (unsigned bx = 0; bx < bw; ++bx) {
            uint32_t w[16];
            for (int y = 0; y < 4; ++y)
                std::memcpy(&w[4 * y], src + (size_t)(4 * by + y) * stride + 16 * (size_t)bx, 16);
            uint2 blk;
            std::memcpy(&blk.x, blocks + 8 * ((size_t)by * bw + bx), 4);
            std::memcpy(&blk.y, blocks + 8 * ((size_t)by * bw + bx) + 4, 4);
            const bool ok = codec == 0 ? goofy_gpu::add_block_errors<goofy_gpu::kBC1>(w, blk, store, 1, s)
                                       : goofy_gpu::add_block_errors<goofy_gpu::kETC1S>(w, blk, store, 1, s);
            sums[4] += ok ? 0 : 1;
            if (++n == every) flush();
        }
    flush();
}
