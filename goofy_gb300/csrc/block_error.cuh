// block_error.cuh -- squared errors of one encoded block against its source
// pixels, without decoding it to pixels.
//
// The reference decodes a block to RGBA and subtracts (getMsePsnr,
// Src/main.cpp:403-469).  Here a row's decoded values stay in the channel
// words that the palette gives (block_decode.cuh) and the row's source pixels
// are regrouped by channel in eight byte permutes; squares are byte dot
// products of absolute differences.  The harness's luminosity error, the square of
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

// x, in a register of its own as far as the compiler can tell.
GOOFY_FN uint32_t opaque(uint32_t x)
{
#if !defined(GOOFY_HOST_EMULATION)
    asm volatile("" : "+r"(x));
#endif
    return x;
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

// Adds one block's errors.  False: an unsupported block (compared as zeros).
//
// ETC1 blocks of other shapes than ETC1s (other encoders') go through palette
// words too: a byte permute picks from those of both sub-blocks at once.
// (Blocks of every mode, 4096^2 back to back on the ring: 20.6 us decoded to
// pixels through shared memory, 16.1 so.)
template <int CODEC>
GOOFY_FN bool add_block_errors(const uint32_t (&w)[16], uint2 blk, ErrorSums& s)
{
    uint32_t a[4], p[4];
    if constexpr (CODEC == kBC1) {
        uint32_t pal[4], sel[4];
        bc1_palette(blk.x, pal);
        bc1_selectors(blk.y, sel);
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            channel_words(w + 4 * y, a);
            pick_row(pal, sel[y], p);
            add_row(a, p, s);
        }
        return true;
    } else {
        const uint32_t w0 = perm(blk.x, 0u, 0x0123u), w1 = perm(blk.y, 0u, 0x0123u);
        if (etc1s_shape(w0)) {
            uint32_t pal[4];
            etc1s_palette(w0, pal);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                channel_words(w + 4 * y, a);
                pick_row(pal, etc1_selector(w1, y), p);
                add_row(a, p, s);
            }
            return true;
        }
        // Copies of the rows: the compiler would regroup them once, ahead of the branch, and the words kept for that
        // cost the ETC1s side 3 % (4096^2 in L2 12.3 against 12.0 us).
        uint32_t v[16], pal[3], pal1[3];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = opaque(w[k]);
        const bool ok = etc1_palettes(w0, pal, pal1, p[3]);
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            channel_words(v + 4 * y, a);
            const uint32_t sel = etc1_selector(w1, y) | etc1_half(w0, y);
#pragma unroll
            for (int k = 0; k < 3; ++k) p[k] = pick(pal[k], pal1[k], sel);
            add_row(a, p, s);
        }
        return ok;
    }
}

#if defined(GOOFY_HOST_EMULATION)
// As the host tests call it, with the palette store that decode_block takes.
template <int CODEC>
GOOFY_FN bool add_block_errors(const uint32_t (&w)[16], uint2 blk, uint32_t*, uint32_t, ErrorSums& s)
{
    return add_block_errors<CODEC>(w, blk, s);
}
#endif

}  // namespace goofy_gpu
