// block_error.cuh -- squared errors of one encoded block against its source
// pixels, without decoding it to pixels.
//
// The reference decodes a block to RGBA and subtracts (getMsePsnr,
// Src/main.cpp:403-469).  Here a block's palette is held as one word per
// channel, colour k of the channel in byte k, and a row's four palette
// indices are the selector of a byte permute: one instruction gives the four
// decoded values of a channel.  The row's source pixels are regrouped by
// channel in eight byte permutes; squares are byte dot products of absolute
// differences.  The harness's luminosity error, the square of
// 21 d2 + 72 d1 + 7 d0 in hundredths (dk the difference of byte k), is a
// quadratic form of the channel differences, so only the products
// d2 d1, d2 d0, d1 d0 are summed besides the squares -- each as four dot
// products, (a - p)(b - q) = ab + pq - aq - pb -- and combined once at the end
// (luma_sum_of).  All sums are exact integers.
#pragma once
#include <cstdint>

#include "block_codec.cuh"
#include "block_decode.cuh"

#if defined(GOOFY_HOST_EMULATION)
#include "error_emulation.h"
#endif

namespace goofy_gpu {

#if !defined(GOOFY_HOST_EMULATION)
// Byte permute whose selector nibbles are known to be 0..7 (__byte_perm masks
// a selector that is not a constant); only the low four nibbles count.
GOOFY_FN uint32_t pick(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
#endif

// Sums over at most kErrorSumBlocks blocks: 16 * 255^2 a block in a square,
// twice that in each half of a product.
constexpr uint32_t kErrorSumBlocks = 2048;
struct ErrorSums {
    uint32_t sq[4];           // squares of the differences of bytes 0..3
    uint32_t pos[3], neg[3];  // products of bytes (2, 1), (2, 0), (1, 0): pos - neg
};

// Four RGBA words to one word per byte position.
GOOFY_FN void channel_words(const uint32_t* px, uint32_t (&c)[4])
{
    const uint32_t t0 = perm(px[0], px[1], 0x5140u), t1 = perm(px[2], px[3], 0x5140u);
    const uint32_t t2 = perm(px[0], px[1], 0x7362u), t3 = perm(px[2], px[3], 0x7362u);
    c[0] = perm(t0, t1, 0x5410u);
    c[1] = perm(t0, t1, 0x7632u);
    c[2] = perm(t2, t3, 0x5410u);
    c[3] = perm(t2, t3, 0x7632u);
}

// One row: source and decoded channel words.
GOOFY_FN void add_row(const uint32_t (&a)[4], const uint32_t (&p)[4], ErrorSums& s)
{
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t d = __vabsdiffu4(a[c], p[c]);
        s.sq[c] = __dp4a(d, d, s.sq[c]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int i = k < 2 ? 2 : 1, j = k == 0 ? 1 : 0;
        s.pos[k] = __dp4a(p[i], p[j], __dp4a(a[i], a[j], s.pos[k]));
        s.neg[k] = __dp4a(p[i], a[j], __dp4a(a[i], p[j], s.neg[k]));
    }
}

// The squared luminosity differences (hundredths) behind the sums.
GOOFY_FN uint64_t luma_sum_of(const ErrorSums& s)
{
    const int64_t cross = 21 * 72 * (int64_t)(int32_t)(s.pos[0] - s.neg[0]) +
                          21 * 7 * (int64_t)(int32_t)(s.pos[1] - s.neg[1]) +
                          72 * 7 * (int64_t)(int32_t)(s.pos[2] - s.neg[2]);
    return 441ull * s.sq[2] + 5184ull * s.sq[1] + 49ull * s.sq[0] + (uint64_t)(2 * cross);
}

// Palette word of a BC1 channel from its two endpoints in 16-bit lanes;
// k1, m1, m2 as set by the endpoint order (bc1_palette in block_decode.cuh):
// colour 2 is (2x + y) / 3 or (x + y) >> 1, colour 3 (x + 2y) / 3 or 0, as the
// third byte of a product.
GOOFY_FN uint32_t bc1_channel(uint32_t lanes, uint32_t k1, uint32_t m1, uint32_t m2)
{
    const uint32_t x = lanes & 0xffffu, y = lanes >> 16;
    const uint32_t q1 = (x * k1 + y) * m1, q2 = (x + 2u * y) * m2;
    return perm(perm(lanes, 0u, 0x4420u), perm(q1, q2, 0x4462u), 0x5410u);
}

// Palette word of an ETC1s channel: base + {small, large, -small, -large}
// clamped to 0..255; sl holds small and large in 16-bit lanes.
GOOFY_FN uint32_t etc1s_channel(uint32_t base, uint32_t sl)
{
    const uint32_t b = base * 0x00010001u;
    const uint32_t up = vmin2(b + sl, 0x00ff00ffu), down = vmax2(b + 0x01000100u - sl, 0x01000100u);
    return perm(up, down, 0x6420u);
}

// Eight 2-bit codes (bits 0..15) to nibbles.
GOOFY_FN uint32_t spread_nibbles(uint32_t x)
{
    x = (x | x << 8) & 0x00ff00ffu;
    x = (x | x << 4) & 0x0f0f0f0fu;
    return (x | x << 2) & 0x33333333u;
}

// Adds one block's errors.  `store` (stride as for decode_block) is used only
// by ETC1 blocks of another shape than ETC1s.  False: an unsupported block
// (compared as zeros).
template <int CODEC>
GOOFY_FN bool add_block_errors(const uint32_t (&w)[16], uint2 blk, uint32_t* store, uint32_t stride, ErrorSums& s)
{
    uint32_t pal[4];
    if constexpr (CODEC == kBC1) {
        const bool four = (blk.x & 0xffffu) > blk.x >> 16;
        const uint32_t k1 = four ? 2u : 1u, m1 = four ? 21846u : 32768u, m2 = four ? 21846u : 0u;
        pal[0] = bc1_channel((((blk.x >> 11) & 0x001f001fu) * 33u >> 2) & 0x00ff00ffu, k1, m1, m2);
        pal[1] = bc1_channel((((blk.x >> 5) & 0x003f003fu) * 65u >> 4) & 0x00ff00ffu, k1, m1, m2);
        pal[2] = bc1_channel(((blk.x & 0x001f001fu) * 33u >> 2) & 0x00ff00ffu, k1, m1, m2);
        pal[3] = four ? 0xffffffffu : 0x00ffffffu;
        const uint32_t n[2] = {spread_nibbles(blk.y & 0xffffu), spread_nibbles(blk.y >> 16)};
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const uint32_t sel = n[y >> 1] >> (16 * (y & 1));
            uint32_t a[4];
            channel_words(w + 4 * y, a);
            const uint32_t p[4] = {pick(pal[0], 0u, sel), pick(pal[1], 0u, sel), pick(pal[2], 0u, sel),
                                   pick(pal[3], 0u, sel)};
            add_row(a, p, s);
        }
        return true;
    } else {
        const uint32_t w0 = perm(blk.x, 0u, 0x0123u), w1 = perm(blk.y, 0u, 0x0123u);
        if ((w0 & 0x07070702u) == 0x00000002u && ((w0 >> 5) & 7u) == ((w0 >> 2) & 7u)) {
            // ETC1s shape, as in decode_block
            const uint32_t c5 = (w0 >> 3) & 0x1f1f1f00u;
            const uint32_t e = ((c5 << 3) & 0xf8f8f800u) | ((c5 >> 2) & 0x07070700u);  // R, G, B in bytes 3, 2, 1
            const uint32_t table = (w0 >> 5) & 7u;
            const uint32_t sl = (uint32_t)etc1_small(table) | (uint32_t)etc1_large(table) << 16;
            pal[0] = etc1s_channel(e >> 24, sl);
            pal[1] = etc1s_channel((e >> 16) & 0xffu, sl);
            pal[2] = etc1s_channel((e >> 8) & 0xffu, sl);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                // pixel (x, y) keeps its low bit at 4x + y and its high bit at 16 + 4x + y: nibble x
                const uint32_t t = (w1 >> y) & 0x11111111u, sel = t + (t >> 15);
                uint32_t a[4];
                channel_words(w + 4 * y, a);
                const uint32_t p[4] = {pick(pal[0], 0u, sel), pick(pal[1], 0u, sel), pick(pal[2], 0u, sel),
                                       0xffffffffu};
                add_row(a, p, s);
            }
            return true;
        }
        uint32_t px[16];
        const bool ok = decode_block<CODEC>(blk, store, stride, px);
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            uint32_t a[4], p[4];
            channel_words(w + 4 * y, a);
            channel_words(px + 4 * y, p);
            add_row(a, p, s);
        }
        return ok;
    }
}

}  // namespace goofy_gpu
