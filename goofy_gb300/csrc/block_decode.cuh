// block_decode.cuh -- per-block BC1 / ETC1 decoding, branch-free.
//
// The reference harness's decoders (Src/decoder.cpp: DecompressColour
// :799-871 with decodeBlockDXT1 :933-943; decompressBlockDiffFlipC :388-678
// with decodeBlockETC1 :958-971) restated as a palette per block and a
// palette slot per pixel.  BC1 blocks and ETC1 blocks of the ETC1s shape
// (differential, zero deltas, one table: every block this encoder writes)
// hold their palette as one word per channel, colour k in byte k, and a row's
// four slots as the selector of a byte permute: one instruction gives a
// channel of four pixels.  Other ETC1 blocks, decoded to pixels, put 4 RGBA
// words per sub-block (8) into a per-thread column of a store (shared memory on the device: entry
// k of thread t at store[k * stride + t], bank-conflict free) and take each
// pixel with one indexed load.  (All blocks through the store: decoding took
// 1-4 % longer, 4096^2 ETC1s 12.7 against 12.3 us.)
//
// ETC1 differential blocks whose second colour leaves 0..31 are ETC2 modes the
// harness does not decode (decoder.cpp:740-760); they decode to zeros and are
// reported as unsupported.
#pragma once
#include <cstdint>

#include "block_codec.cuh"

namespace goofy_gpu {

// Byte permute whose selector nibbles are known to be 0..7 (__byte_perm masks
// a selector that is not a constant); only the low four nibbles count.
GOOFY_FN uint32_t pick(uint32_t a, uint32_t b, uint32_t sel)
{
#if defined(GOOFY_HOST_EMULATION)
    return perm(a, b, sel);
#else
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
#endif
}

// Palette word of a BC1 channel from its two endpoints x, y in 16-bit lanes:
// {x, y, (2x + y) / 3 or (x + y) >> 1, (x + 2y) / 3 or 0}, the last two as the
// third byte of a product (division by 3 of n <= 765 is (n * 21846) >> 16).
GOOFY_FN uint32_t bc1_channel(uint32_t lanes, uint32_t k1, uint32_t m1, uint32_t m2)
{
    const uint32_t x = lanes & 0xffffu, y = lanes >> 16;
    const uint32_t q1 = (x * k1 + y) * m1, q2 = (x + 2u * y) * m2;
    return perm(perm(lanes, 0u, 0x4420u), perm(q1, q2, 0x4462u), 0x5410u);
}

// Palette words R, G, B, A of a BC1 block (DecompressColour): c0 > c1 gives
// the 1/3 and 2/3 points as colours 2 and 3, otherwise colour 2 is the
// midpoint and colour 3 transparent black.  Endpoints expand by bit
// replication, both at once.
GOOFY_FN void bc1_palette(uint32_t ends, uint32_t (&pal)[4])
{
    const bool four = (ends & 0xffffu) > ends >> 16;
    const uint32_t k1 = four ? 2u : 1u, m1 = four ? 21846u : 32768u, m2 = four ? 21846u : 0u;
    pal[0] = bc1_channel((((ends >> 11) & 0x001f001fu) * 33u >> 2) & 0x00ff00ffu, k1, m1, m2);
    pal[1] = bc1_channel((((ends >> 5) & 0x003f003fu) * 65u >> 4) & 0x00ff00ffu, k1, m1, m2);
    pal[2] = bc1_channel(((ends & 0x001f001fu) * 33u >> 2) & 0x00ff00ffu, k1, m1, m2);
    pal[3] = four ? 0xffffffffu : 0x00ffffffu;
}

// Eight 2-bit codes (bits 0..15) to nibbles.
GOOFY_FN uint32_t spread_nibbles(uint32_t x)
{
    x = (x | x << 8) & 0x00ff00ffu;
    x = (x | x << 4) & 0x0f0f0f0fu;
    return (x | x << 2) & 0x33333333u;
}

// Row selectors (low four nibbles) of a BC1 index word.
GOOFY_FN void bc1_selectors(uint32_t idx, uint32_t (&sel)[4])
{
    sel[0] = spread_nibbles(idx & 0xffffu);
    sel[1] = sel[0] >> 16;
    sel[2] = spread_nibbles(idx >> 16);
    sel[3] = sel[2] >> 16;
}

// One channel's palette words picked for a row.
GOOFY_FN void pick_row(const uint32_t (&pal)[4], uint32_t sel, uint32_t (&c)[4])
{
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = pick(pal[k], 0u, sel);
}

// Four channel words of a row to its four RGBA words.
GOOFY_FN void pixel_words(const uint32_t (&c)[4], uint32_t* px)
{
    const uint32_t t0 = perm(c[0], c[1], 0x5140u), t1 = perm(c[0], c[1], 0x7362u);  // RGRG of pixels 0, 1 / 2, 3
    const uint32_t t2 = perm(c[2], c[3], 0x5140u), t3 = perm(c[2], c[3], 0x7362u);
    px[0] = perm(t0, t2, 0x5410u);
    px[1] = perm(t0, t2, 0x7632u);
    px[2] = perm(t1, t3, 0x5410u);
    px[3] = perm(t1, t3, 0x7632u);
}

// Base colours (bytes R, G, B) of the two sub-blocks of the big-endian word
// w0: 4+4-bit individual colours, or a 5-bit colour and a 3-bit signed delta.
// False for a differential second colour outside 0..31.
GOOFY_FN bool etc1_bases(uint32_t w0, uint32_t& base0, uint32_t& base1)
{
    const bool diff = (w0 >> 1) & 1u;
    bool ok = true;
    base0 = base1 = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const uint32_t h = (w0 >> (24 - 8 * c)) & 0xffu;
        const uint32_t i0 = (h >> 4) * 17u, i1 = (h & 15u) * 17u;
        const int c5 = (int)(h >> 3), d = (int)(h & 3u) - (int)(h & 4u);  // 3-bit two's complement
        const int c52 = c5 + d;
        ok = ok && (!diff || (c52 >= 0 && c52 <= 31));
        const int cl = min(max(c52, 0), 31);
        const uint32_t d0 = (uint32_t)(c5 << 3 | c5 >> 2), d1 = (uint32_t)(cl << 3 | cl >> 2);
        base0 |= (diff ? d0 : i0) << (8 * c);
        base1 |= (diff ? d1 : i1) << (8 * c);
    }
    return ok;
}

// Intensity modifier tables (compressParams, decoder.cpp:391-408): the small and large
// magnitude of each of the 8 tables, one byte each, picked with a byte permute.
GOOFY_FN int etc1_small(uint32_t table) { return (int)(perm(0x0D090502u, 0x2F211812u, table) & 0xffu); }
GOOFY_FN int etc1_large(uint32_t table) { return (int)(perm(0x2A1D1108u, 0xB76A503Cu, table) & 0xffu); }

// The 4 colours of a sub-block, slot = pixel index (msb << 1 | lsb):
// base + {small, large, -small, -large}, each channel clamped to 0..255.
// R and B are clamped together in 16-bit lanes biased by 256.
GOOFY_FN void etc1_subpalette(uint32_t base, uint32_t table, uint32_t* pal)
{
    const int s = etc1_small(table), l = etc1_large(table);
    const int mod[4] = {s, l, -s, -l};
    const uint32_t rb = base & 0x00ff00ffu;
    const int g = (int)((base >> 8) & 0xffu);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t v = vmin2(vmax2(rb + (uint32_t)(256 + mod[k]) * 0x00010001u, 0x01000100u), 0x01ff01ffu) -
                           0x01000100u;
        pal[k] = v | (uint32_t)min(max(g + mod[k], 0), 255) << 8 | 0xff000000u;
    }
}

// Differential with zero deltas and one table for both halves.
GOOFY_FN bool etc1s_shape(uint32_t w0)
{
    return (w0 & 0x07070702u) == 0x00000002u && ((w0 >> 5) & 7u) == ((w0 >> 2) & 7u);
}

// Palette word of an ETC1s channel: base + {small, large, -small, -large}
// clamped to 0..255; sl holds small and large in 16-bit lanes.
GOOFY_FN uint32_t etc1s_channel(uint32_t base, uint32_t sl)
{
    const uint32_t b = base * 0x00010001u;
    const uint32_t up = vmin2(b + sl, 0x00ff00ffu), down = vmax2(b + 0x01000100u - sl, 0x01000100u);
    return perm(up, down, 0x6420u);
}

// Palette words R, G, B, A of an ETC1s-shaped block: both sub-blocks have the
// 5-bit colour (bits 31..27, 23..19, 15..11) expanded by bit replication as
// base.
GOOFY_FN void etc1s_palette(uint32_t w0, uint32_t (&pal)[4])
{
    const uint32_t c5 = (w0 >> 3) & 0x1f1f1f00u;  // R5, G5, B5 in bytes 3, 2, 1
    const uint32_t e = ((c5 << 3) & 0xf8f8f800u) | ((c5 >> 2) & 0x07070700u);
    const uint32_t table = (w0 >> 5) & 7u;
    const uint32_t sl = (uint32_t)etc1_small(table) | (uint32_t)etc1_large(table) << 16;
    pal[0] = etc1s_channel(e >> 24, sl);
    pal[1] = etc1s_channel((e >> 16) & 0xffu, sl);
    pal[2] = etc1s_channel((e >> 8) & 0xffu, sl);
    pal[3] = 0xffffffffu;
}

// Palette words R, G, B of both sub-blocks of any ETC1 block, and their alpha.
// False, and zeros, for an unsupported one.
GOOFY_FN bool etc1_palettes(uint32_t w0, uint32_t (&pal)[3], uint32_t (&pal1)[3], uint32_t& alpha)
{
    uint32_t b0, b1;
    const bool ok = etc1_bases(w0, b0, b1);
    const uint32_t t0 = (w0 >> 5) & 7u, t1 = (w0 >> 2) & 7u;
    const uint32_t sl0 = (uint32_t)etc1_small(t0) | (uint32_t)etc1_large(t0) << 16;
    const uint32_t sl1 = (uint32_t)etc1_small(t1) | (uint32_t)etc1_large(t1) << 16;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        pal[k] = ok ? etc1s_channel((b0 >> (8 * k)) & 0xffu, sl0) : 0u;
        pal1[k] = ok ? etc1s_channel((b1 >> (8 * k)) & 0xffu, sl1) : 0u;
    }
    alpha = ok ? 0xffffffffu : 0u;
    return ok;
}

// Which nibbles of row y's selector pick from the second sub-block (4 added):
// the lower rows with flip, the right columns without.
GOOFY_FN uint32_t etc1_half(uint32_t w0, int y) { return (w0 & 1u) ? (y < 2 ? 0u : 0x4444u) : 0x4400u; }

// Selector (low four nibbles) of pixel row y: pixel (x, y) keeps its low bit
// at 4x + y of the index word and its high bit at 16 + 4x + y, nibble x.
GOOFY_FN uint32_t etc1_selector(uint32_t w1, int y)
{
    const uint32_t t = (w1 >> y) & 0x11111111u;
    return t + (t >> 15);
}

// 2-bit palette index of every pixel, pixel k = 4x + y at bits 2k..2k+1, from
// the lsb plane (bits 0..15) and msb plane (bits 16..31) of the index word.
GOOFY_FN uint32_t spread_bits16(uint32_t x)
{
    x = (x | x << 8) & 0x00ff00ffu;
    x = (x | x << 4) & 0x0f0f0f0fu;
    x = (x | x << 2) & 0x33333333u;
    return (x | x << 1) & 0x55555555u;
}

GOOFY_FN uint32_t etc1_codes(uint32_t w1) { return spread_bits16(w1 & 0xffffu) | spread_bits16(w1 >> 16) << 1; }

// Decodes one block into 16 row-major RGBA words; ETC1 blocks of other shapes
// than ETC1s use store[k * stride] (k < 8) for the palette.  Returns false
// for an unsupported ETC1 block.
template <int CODEC>
GOOFY_FN bool decode_block(uint2 blk, uint32_t* store, uint32_t stride, uint32_t (&px)[16])
{
    if constexpr (CODEC == kBC1) {
        uint32_t pal[4], sel[4], c[4];
        bc1_palette(blk.x, pal);
        bc1_selectors(blk.y, sel);
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            pick_row(pal, sel[y], c);
            pixel_words(c, px + 4 * y);
        }
        return true;
    } else {
        // the block is big-endian: bytes 0..3 of blk.x are bits 63..32
        const uint32_t w0 = perm(blk.x, 0u, 0x0123u), w1 = perm(blk.y, 0u, 0x0123u);
        if (etc1s_shape(w0)) {
            uint32_t pal[4], c[4];
            etc1s_palette(w0, pal);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                pick_row(pal, etc1_selector(w1, y), c);
                pixel_words(c, px + 4 * y);
            }
            return true;
        }
        const bool flip = w0 & 1u;
        uint32_t b0, b1, pal[4];
        const bool ok = etc1_bases(w0, b0, b1);
        // equal halves have one palette: it is built and stored once
        const bool one = b0 == b1 && ((w0 >> 5) & 7u) == ((w0 >> 2) & 7u);
        etc1_subpalette(b0, (w0 >> 5) & 7u, pal);
#pragma unroll
        for (int k = 0; k < 4; ++k) store[k * stride] = ok ? pal[k] : 0u;
        if (!one) {
            etc1_subpalette(b1, (w0 >> 2) & 7u, pal);
#pragma unroll
            for (int k = 0; k < 4; ++k) store[(4 + k) * stride] = ok ? pal[k] : 0u;
        }
        const uint32_t codes = etc1_codes(w1);
        if (one) {  // no sub-block offsets
#pragma unroll
            for (int y = 0; y < 4; ++y)
#pragma unroll
                for (int x = 0; x < 4; ++x) px[4 * y + x] = store[((codes >> (2 * (4 * x + y))) & 3u) * stride];
            return ok;
        }
        // sub-block 1: right half (x >= 2) without flip, bottom half (y >= 2) with flip
        const uint32_t s1 = 4u * stride;
        const uint32_t lower_right = s1, upper_right = flip ? 0u : s1, lower_left = flip ? s1 : 0u;
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const uint32_t sub = x < 2 ? (y < 2 ? 0u : lower_left) : (y < 2 ? upper_right : lower_right);
                px[4 * y + x] = store[sub + ((codes >> (2 * (4 * x + y))) & 3u) * stride];
            }
        return ok;
    }
}

}  // namespace goofy_gpu
