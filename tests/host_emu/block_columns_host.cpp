// block_columns_host.cpp -- TEST ONLY.  The encoders of block_codec.cuh on
// blocks whose columns x lie in the places x ^ q (q as the kernels take it
// from the lane), compiled for the CPU through host_emulation.h.
#include <cstring>

#include "block_codec.cuh"

// `blocks`: n blocks of 64 bytes.  codec 2: {BC1, ETC1s} pairs of 16 bytes.
extern "C" void host_emu_encode_columns(int codec, uint8_t* out, const uint8_t* blocks, unsigned n, unsigned q)
{
    uint8_t lut[128];
    for (uint32_t i = 0; i < 128; ++i) lut[i] = (uint8_t)goofy_gpu::etc_control_byte(2 * i);
    for (unsigned k = 0; k < n; ++k) {
        uint32_t px[16], w[16];
        std::memcpy(px, blocks + 64 * (size_t)k, 64);
        for (unsigned y = 0; y < 4; ++y)
            for (unsigned x = 0; x < 4; ++x) w[4 * y + x] = px[4 * y + (x ^ q)];
        if (codec == 2) {
            const uint4 r = goofy_gpu::encode_both<true>(w, lut, q);
            std::memcpy(out + 16 * (size_t)k, &r, 16);
        } else {
            const uint2 r = codec == 0 ? goofy_gpu::encode_block<goofy_gpu::kBC1, true>(w, lut, q)
                                       : goofy_gpu::encode_block<goofy_gpu::kETC1S, true>(w, lut, q);
            std::memcpy(out + 8 * (size_t)k, &r, 8);
        }
    }
}
