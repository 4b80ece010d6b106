// encode_tma.cu -- the image encoder fed by bulk asynchronous copies.
//
// A resident grid of CTAs, each with one producer warp and C compute warps
// (C = threads / 32).  Work is cut into units of 32 * C * BPT consecutive
// blocks of the image in row-major order; CTA b takes units b, b + grid, ...
// The producer's elected lane copies each unit's pixel rows (16 bytes per
// block, contiguous in the source; four pieces for every block row that the
// unit touches) into the next free stage of a shared-memory ring with
// cp.async.bulk, counted on that stage's "full" mbarrier; compute warps wait
// for it, pull their blocks into registers with conflict-free 128-bit shared
// loads (lane l of a warp reads 16 contiguous bytes, the warp 512: block k of
// a unit lies at 16 * k of each of the stage's four planes, whatever rows it
// came from), run the
// same block codec as every other kernel, store 8 bytes per block with
// streaming stores and release the stage on its "empty" mbarrier.  Global
// loads never sit in the compute warps' registers, so the integer math of one
// unit overlaps the HBM reads of the next stages.
//
// Units run on across block rows, so every stage but the last is full at any
// width.  Tiles that ended with their row left a stage half empty at 2048
// pixels and added a nearly empty one to each row a little wider than a
// stage: 4100x4096 BC1 16.7, ETC1s 20.1, both 24.6 us then, 11.1, 12.3 and
// 14.7 us so (floor 11.3 us at 4.5 B/px of measured HBM; 4096^2 unchanged at
// 11.0, 12.2 and 14.4 us).  The producer stays one lane: copies issued by
// several lanes at once cost more (ETC1s 4096^2 12.5 us), and so did tiles
// of several rows and part of the width (short row copies; 15.4 us).
//
// Launched with programmatic dependent launch (pdl.cuh): the prologue
// (barriers, control-byte table) runs while the previous kernel in the stream
// drains, and no copy is issued before that kernel has completed.
//
// Word-aligned rows (a part of an atlas at an odd pixel offset, a padded
// stride) take the same kernel: whole 16-byte granules are copied and the
// shift is taken out when the words leave shared memory.  The
// register-loading kernel reads such a block with sixteen 4-byte loads
// (launch_image has both sides' times).
//
// Every wait is bounded (async_copy.cuh): a stuck barrier ends the kernel with
// a counted time-out instead of a hang, and the producer then waits (bounded)
// for the copies it issued before its CTA exits.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "async_copy.cuh"
#include "batch.h"
#include "block_codec.cuh"
#include "block_error.cuh"
#include "decode.h"
#include "device_io.cuh"
#include "error_reduce.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace goofy_gpu {

__device__ unsigned int g_pipeline_timeouts;

// CTAs per SM each instantiation is compiled for (register caps that keep
// that many resident; every ring fits that many times in shared memory).  With
// two blocks a thread the ETC1s codec wants about 80 registers, so the
// 512-thread CTA runs alone on its SM; the 256-thread one is capped at 72 to
// fit 3.  The 128-thread CTA stays at 4: 5 would put 7 warps on one scheduler,
// whose quarter of the register file then caps them at 72 with spills.
__host__ __device__ constexpr int tma_min_ctas(uint32_t bpt, uint32_t compute_threads)
{
    return bpt == 1 ? (compute_threads == 512 ? 2 : compute_threads == 256 ? 4 : 7)
                    : (compute_threads == 512 ? 1 : compute_threads == 256 ? 3 : 4);
}

struct TmaLayout {
    uint32_t tile_blocks, row_bytes, stage_bytes, stages;
};

// Word-aligned rows: a run of nb blocks is copied as the 16-byte granules that
// hold it, up to nb + 1 of them, so every plane has room for one more granule
// per block row that a unit touches (and the one read past the last block).
// kWordSlack of them serve units of up to 5 block rows' width.
constexpr uint32_t kWordSlack = 8;
__host__ __device__ constexpr bool word_rows_fit(uint32_t tile_blocks, uint32_t bw) { return tile_blocks <= 5u * bw; }

__host__ __device__ constexpr TmaLayout tma_layout(uint32_t compute_threads, uint32_t bpt, bool word = false)
{
    TmaLayout l{};
    l.tile_blocks = compute_threads * bpt;
    l.row_bytes = 16u * (l.tile_blocks + (word ? kWordSlack : 0u));
    l.stage_bytes = 4u * l.row_bytes;
    // ring budget scaled with the CTA (112 KB at 512 compute threads), so the
    // CTAs the registers allow per SM also fit in shared memory; at least 3
    // stages for a CTA alone on its SM (a stage is released only once it has
    // been encoded, so 2 would leave that SM a single stage of lookahead)
    const uint32_t s = (114688u / 512u * compute_threads) / (64u * l.tile_blocks);
    const uint32_t lo = tma_min_ctas(bpt, compute_threads) == 1 ? 3u : 2u;
    l.stages = s < lo ? lo : s > 6u ? 6u : s;
    return l;
}

constexpr size_t tma_smem_bytes(const TmaLayout& l) { return (size_t)l.stages * (l.stage_bytes + 16u) + 128u; }

// Tiles (batch: units) of a CTA whose rows its producer asks L2 for before
// the dependency wait, while the previous kernel drains.  Two of the three
// stages measured best: with all three the launch starts later (8192^2
// ETC1s 45.3 against 44.8 us, 4096^2 13.9 against 13.2 us), with one the
// first copies find less in L2.
#ifndef GOOFY_L2_PREFETCH_TILES
#define GOOFY_L2_PREFETCH_TILES 2
#endif
__host__ __device__ constexpr uint32_t l2_prefetch_tiles(const TmaLayout& l)
{
    return (uint32_t)GOOFY_L2_PREFETCH_TILES < l.stages ? (uint32_t)GOOFY_L2_PREFETCH_TILES : l.stages;
}

// Encodes the blocks of one stage held in shared memory (four pixel rows of
// row_bytes, block k of the unit at 16 * k in each) and stores those below nb
// at out + 8 * k (and out2, for both codecs).  Thread `lane` of compute warp
// `warp` takes blocks (warp * BPT + j) * 32 + lane.  Every thread loads and
// encodes all its slots, also past nb (the image's last, shorter unit): such
// a slot holds whatever an earlier unit left in the stage, which nothing
// writes while the stage is held, and its result is dropped.  Only the
// stores are conditional, so the loads and the codec run without branches.
// WORD: block k's pixel row y starts shift[y] bytes into granule
// k + (its block row - the unit's first) of plane y and is read word by word.
// In column order that puts four lanes on a bank (64 wavefronts a warp and
// block instead of 16), so with XOR_COLUMNS lane l reads column x ^ (l >> 3)
// into w[4y + x]: the eight lanes of a group are 4 words apart and the four
// groups a word apart, so no two share a bank.  The codec gives the same block
// but for the order of its indices (swap_columns in block_codec.cuh).
// Measured against column order (400 MB of inputs): 4096^2 BC1 13.2 -> 12.2,
// ETC1s 14.1 -> 13.9 us.  Four addresses a block plus uniform row offsets:
// added the other way round (a row's base plus the column) the sixteen sums
// cost more than the conflicts at 2376x2628.
template <int BPT, bool WORD, bool XOR_COLUMNS>
__device__ __forceinline__ void load_stage(const uint8_t* buf, uint32_t row_bytes, uint32_t warp, uint32_t lane,
                                           uint32_t nb, uint32_t bx0, uint32_t bw, uint32_t bw_magic,
                                           const uint32_t (&shift)[4], uint32_t (&w)[BPT][16])
{
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
        const uint32_t b = (warp * BPT + j) * 32u + lane;
        if constexpr (WORD) {
            uint32_t x;
            const uint32_t s = div_magic(min(bx0 + b, bx0 + nb - 1u), bw, bw_magic, x);
            const uint8_t* p = buf + 16u * (min(b, nb - 1u) + s);
            const uint32_t q = XOR_COLUMNS ? (lane >> 1) & 12u : 0u;
            const uint8_t* const col[4] = {p + q, p + (q ^ 4u), p + (q ^ 8u), p + (q ^ 12u)};
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    w[j][4 * r + i] = *reinterpret_cast<const uint32_t*>(col[i] + (r * row_bytes + shift[r]));
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint4 v = *reinterpret_cast<const uint4*>(buf + r * row_bytes + 16u * b);
                w[j][4 * r + 0] = v.x;
                w[j][4 * r + 1] = v.y;
                w[j][4 * r + 2] = v.z;
                w[j][4 * r + 3] = v.w;
            }
        }
    }
}

template <int CODEC, int BPT, bool WORD>
__device__ __forceinline__ void encode_stage(const uint8_t* buf, uint32_t row_bytes, uint32_t warp, uint32_t lane,
                                             uint32_t nb, uint8_t* out, uint8_t* out2, const uint8_t* ctrl_lut,
                                             uint32_t bx0, uint32_t bw, uint32_t bw_magic,
                                             const uint32_t (&shift)[4])
{
    uint32_t w[BPT][16];
    load_stage<BPT, WORD, WORD>(buf, row_bytes, warp, lane, nb, bx0, bw, bw_magic, shift, w);
    const uint32_t q = WORD ? lane >> 3 : 0u;
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
        const uint32_t b = (warp * BPT + j) * 32u + lane;
        if constexpr (CODEC == kBoth) {
            const uint4 e = encode_both<WORD>(w[j], ctrl_lut, q);
            if (b < nb) {
                st_stream8(out + 8u * (size_t)b, make_uint2(e.x, e.y));
                st_stream8(out2 + 8u * (size_t)b, make_uint2(e.z, e.w));
            }
        } else {
            const uint2 e = encode_block<CODEC, WORD>(w[j], ctrl_lut, q);
            if (b < nb) st_stream8(out + 8u * (size_t)b, e);
        }
    }
}

// Calls f(k, nb, p) for every run of unit blocks [first, first + n) in one
// block row of the image: unit blocks k .. k + nb - 1, whose first pixel row
// starts at p.
template <typename F>
__device__ __forceinline__ void for_unit_rows(const uint8_t* src, size_t stride, uint32_t bw, uint32_t bw_magic,
                                              uint32_t first, uint32_t n, F f)
{
    uint32_t bx;
    const uint32_t by = div_magic(first, bw, bw_magic, bx);
    const uint8_t* p = src + (size_t)by * 4u * stride + 16u * (size_t)bx;
    uint32_t nb = min(bw - bx, n);
    f(0u, nb, p);
    for (uint32_t k = nb; k < n; k += nb) {
        p += 4u * stride - 16u * (size_t)bx;
        bx = 0u;
        nb = min(bw, n - k);
        f(k, nb, p);
    }
}

// The image behind a ring.  WORD: its rows are only 4-byte aligned.
// 4 * stride is then a multiple of 16, so pixel row y of every block row
// starts shift[y] = (src + y * stride) % 16 bytes past a 16-byte boundary; the
// copies take whole granules from that boundary on (the first and last may
// hold bytes of other pixels, never of another allocation's page) and the
// compute warps read at the shift.
template <bool WORD>
struct RingImage {
    const uint8_t* src;
    size_t stride;
    uint32_t bw, bw_magic, total;
    uint32_t shift[4];

    __device__ __forceinline__ RingImage(const uint8_t* src_, size_t stride_, uint32_t bw_, uint32_t magic, uint32_t n)
        : src(src_), stride(stride_), bw(bw_), bw_magic(magic), total(n)
    {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            shift[r] = WORD ? (uint32_t)(reinterpret_cast<uintptr_t>(src) + r * stride) & 15u : 0u;
    }

    // bytes of pixel row r's piece of nb blocks
    __device__ __forceinline__ uint32_t piece(uint32_t nb, int r) const
    {
        return WORD ? (16u * nb + shift[r] + 15u) & ~15u : 16u * nb;
    }
};

// One lane, before the dependency wait: while the previous kernel in the
// stream drains, ask L2 for the rows of this CTA's first units.  Only a hint:
// no data enters the CTA before pdl_wait(), and L2 is coherent with the
// previous kernel's writes, so the copies after the wait still read what it
// wrote.
template <bool WORD>
__device__ __forceinline__ void prefetch_units(const RingImage<WORD>& im, const TmaLayout& L)
{
    const uint32_t unit = L.tile_blocks, step = gridDim.x * unit;
    uint32_t c = 0;
    for (uint32_t first = blockIdx.x * unit; first < im.total && c < l2_prefetch_tiles(L); first += step, ++c)
        for_unit_rows(im.src, im.stride, im.bw, im.bw_magic, first, min(unit, im.total - first),
                      [&](uint32_t, uint32_t nb, const uint8_t* row) {
#pragma unroll
                          for (int r = 0; r < 4; ++r)
                              bulk_prefetch_l2(row + r * im.stride - im.shift[r], im.piece(nb, r));
                      });
}

// The producer's one lane: copies the rows of units blockIdx.x, + gridDim.x,
// ... into the ring, each stage once its compute warps have released it.
template <bool WORD>
__device__ __forceinline__ void produce_units(const RingImage<WORD>& im, const TmaLayout& L, uint8_t* smem,
                                              uint64_t* full, uint64_t* empty, volatile uint32_t* abort_flag,
                                              uint64_t policy)
{
    const uint32_t unit = L.tile_blocks, step = gridDim.x * unit;
    uint32_t issued = 0, slot = 0, phase = 0;
    for (uint32_t first = blockIdx.x * unit; first < im.total; first += step) {
        if (issued >= L.stages && !mbar_wait(&empty[slot], phase ^ 1u, abort_flag, &g_pipeline_timeouts)) break;
        const uint32_t n = min(unit, im.total - first);
        uint32_t bytes = 64u * n, s = 0;
        if constexpr (WORD) {
            bytes = 0;
            for_unit_rows(im.src, im.stride, im.bw, im.bw_magic, first, n,
                          [&](uint32_t, uint32_t nb, const uint8_t*) {
#pragma unroll
                              for (int r = 0; r < 4; ++r) bytes += im.piece(nb, r);
                          });
        }
        mbar_arrive_expect_tx(&full[slot], bytes);
        uint8_t* buf = smem + slot * L.stage_bytes;
        for_unit_rows(im.src, im.stride, im.bw, im.bw_magic, first, n,
                      [&](uint32_t k, uint32_t nb, const uint8_t* row) {
#pragma unroll
                          for (int r = 0; r < 4; ++r)
                              bulk_copy_g2s_hint(buf + r * L.row_bytes + 16u * (k + s),
                                                 row + r * im.stride - im.shift[r], im.piece(nb, r), &full[slot],
                                                 policy);
                          if constexpr (WORD) ++s;
                      });
        ++issued;
        if (++slot == L.stages) {
            slot = 0;
            phase ^= 1u;
        }
    }
    if (*abort_flag) {
        // the copies of the last stages may still be landing: wait for them (bounded) before exiting
        const uint32_t n = issued < L.stages ? issued : L.stages;
        for (uint32_t i = issued - n; i < issued; ++i)
            mbar_wait(&full[i % L.stages], (i / L.stages) & 1u, nullptr, &g_pipeline_timeouts);
    }
}

// One thread, at a CTA's start.
__device__ __forceinline__ void init_ring(uint64_t* full, uint64_t* empty, uint32_t stages, uint32_t compute_warps,
                                          uint32_t* abort_flag)
{
    for (uint32_t s = 0; s < stages; ++s) {
        mbar_init(&full[s], 1u);
        mbar_init(&empty[s], compute_warps);
    }
    *abort_flag = 0u;
    mbar_init_fence();
}

template <int CODEC, int BPT, int COMPUTE, bool WORD>
__global__ void __launch_bounds__(COMPUTE + 32, tma_min_ctas(BPT, COMPUTE))
    encode_image_tma(const uint8_t* __restrict__ src, size_t stride, uint8_t* __restrict__ dst,
                     uint8_t* __restrict__ dst2, uint32_t bw, uint32_t bw_magic, uint32_t total)
{
    pdl_launch_dependents();
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t abort_flag;
    constexpr uint32_t compute_warps = COMPUTE / 32;
    constexpr TmaLayout L = tma_layout(COMPUTE, BPT, WORD);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.stages * L.stage_bytes);
    uint64_t* empty = full + L.stages;
    uint8_t* ctrl_lut = reinterpret_cast<uint8_t*>(empty + L.stages);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const RingImage<WORD> im(src, stride, bw, bw_magic, total);

    if (threadIdx.x == 0) init_ring(full, empty, L.stages, compute_warps, &abort_flag);
    if constexpr (CODEC != kBC1) fill_ctrl_lut(ctrl_lut);
    __syncthreads();
    if (warp == compute_warps && lane == 0) prefetch_units(im, L);
    pdl_wait();  // no global memory access before the previous kernel in the stream is done

    if (warp == compute_warps) {  // producer
        // Rows are read once: evict-first in L2 (single-codec launches back to
        // back: 4096^2 ETC1s 12.3 against 13.2 us, BC1 11.2 against 12.4 us).
        // The two-codec pass marks half of them: with all it measured 0.9 us
        // slower at 8192^2; with half, as fast there and 0.4 us faster at 4096^2.
        if (lane == 0)
            produce_units(im, L, smem, full, empty, &abort_flag,
                          CODEC == kBoth ? l2_evict_first_half_policy() : l2_evict_first_policy());
        return;
    }

    constexpr uint32_t unit = L.tile_blocks;
    const uint32_t step = gridDim.x * unit;  // units blockIdx.x, + gridDim.x, ...
    uint32_t slot = 0, phase = 0;
    for (uint32_t first = blockIdx.x * unit; first < total; first += step) {
        if (!mbar_wait(&full[slot], phase, &abort_flag, &g_pipeline_timeouts)) break;
        const uint32_t nb = min(unit, total - first);
        const uint8_t* buf = smem + slot * L.stage_bytes;
        const size_t o = (size_t)first * 8u;
        uint32_t bx0 = 0;
        if constexpr (WORD) div_magic(first, bw, bw_magic, bx0);
        if (warp * (BPT * 32u) < nb)  // warps wholly past the unit's last block skip it
            encode_stage<CODEC, BPT, WORD>(buf, L.row_bytes, warp, lane, nb, dst + o,
                                           CODEC == kBoth ? dst2 + o : nullptr, ctrl_lut, bx0, bw, bw_magic, im.shift);
        // Release the stage only now.  An arrival right after the shared loads
        // can overtake them: the loads wait in the load/store queue (behind
        // other kernels' global loads when SMs are shared) while the arrival
        // completes at once, and the producer's next copy into the stage then
        // lands before they read it (seen with a concurrent register-loading
        // kernel: rows of the stage's next tile inside this tile's blocks).
        // The stores cannot issue before the blocks they write are encoded
        // from every loaded word, and the arrival (a release) stays after them.
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        if (++slot == L.stages) {
            slot = 0;
            phase ^= 1u;
        }
    }
}


// ---------------------------------------------------------------------------
// The quality measurement on the same ring: the compute warps compare each
// block with its rows (block_error.cuh) instead of encoding it.  A thread's
// codes of the next unit are loaded while it works on this one.  Bound by
// HBM at 8192^2 (42.6 us, 7.09 TB/s); with the rows loaded into registers a
// block ahead it is short of bytes in flight there (44.2 us).  Smaller images
// do better by the registers (launch_block_error has both sides).
// ---------------------------------------------------------------------------
template <int CODEC, int BPT, int COMPUTE, bool WORD>
__global__ void __launch_bounds__(COMPUTE + 32, 1)
    error_image_tma(const uint8_t* __restrict__ blocks, const uint8_t* __restrict__ src, size_t stride, uint32_t bw,
                    uint32_t bw_magic, uint32_t total, unsigned long long* __restrict__ sums, ErrorResult result)
{
    pdl_launch_dependents();
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t abort_flag;
    constexpr uint32_t compute_warps = COMPUTE / 32;
    constexpr TmaLayout L = tma_layout(COMPUTE, BPT, WORD);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.stages * L.stage_bytes);
    uint64_t* empty = full + L.stages;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const RingImage<WORD> im(src, stride, bw, bw_magic, total);

    if (threadIdx.x == 0) init_ring(full, empty, L.stages, compute_warps, &abort_flag);
    __syncthreads();
    if (warp == compute_warps && lane == 0) prefetch_units(im, L);
    pdl_wait();

    if (warp == compute_warps) {
        if (lane == 0) produce_units(im, L, smem, full, empty, &abort_flag, l2_evict_first_policy());
        return;
    }

    constexpr uint32_t unit = L.tile_blocks;
    const uint32_t step = gridDim.x * unit;
    uint32_t first = blockIdx.x * unit, slot = 0, phase = 0, bad = 0;
    ErrorSums e{};  // at most kErrorSumBlocks blocks a thread (launch_error_tma)
    bool gave_up = false;
    uint2 next[BPT];
    auto load_codes = [&](uint32_t at) {
#pragma unroll
        for (int j = 0; j < BPT; ++j) {
            const uint32_t b = at + (warp * BPT + j) * 32u + lane;
            next[j] = b < total ? load_block8(blocks + 8u * (size_t)b) : make_uint2(0u, 0u);
        }
    };
    if (first < total) load_codes(first);
    for (; first < total; first += step) {
        uint2 code[BPT];
#pragma unroll
        for (int j = 0; j < BPT; ++j) code[j] = next[j];
        if (first + step < total) load_codes(first + step);
        if (!mbar_wait(&full[slot], phase, &abort_flag, &g_pipeline_timeouts)) {
            // This lane leaves its blocks out, here and in the units that follow, but lanes of its warp whose last
            // try succeeded still need it at the __syncwarp below.
            gave_up = true;
            for (; first < total; first += step) __syncwarp();
            break;
        }
        const uint32_t nb = min(unit, total - first);
        uint32_t bx0 = 0, w[BPT][16];
        if constexpr (WORD) div_magic(first, bw, bw_magic, bx0);
        load_stage<BPT, WORD, false>(smem + slot * L.stage_bytes, L.row_bytes, warp, lane, nb, bx0, bw, bw_magic, im.shift, w);
#pragma unroll
        for (int j = 0; j < BPT; ++j)
            if ((warp * BPT + j) * 32u + lane < nb) bad += add_block_errors<CODEC>(w[j], code[j], e) ? 0u : 1u;
        // Release the stage only now (see encode_image_tma): every loaded word has gone into these sums.
        asm volatile("" ::"r"(e.sq[0]), "r"(e.sq[1]), "r"(e.sq[2]), "r"(e.sq[3]) : "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        if (++slot == L.stages) {
            slot = 0;
            phase ^= 1u;
        }
    }
    reduce_errors<COMPUTE>(e, bad, gave_up, sums, result);
}

// ---------------------------------------------------------------------------
// The batch kernel on the same pipeline (tile `pipeline` = 1).  A work unit is
// one stage: up to COMPUTE * BPT consecutive blocks of one image (they may
// span several block rows).  CTA b takes units b, b + grid, ... (equal units
// balance like the image kernel's tiles, and no work counter is needed); its
// producer finds each unit's image, writes the stage's unit record and copies
// the unit's rows: for each block row segment of nb blocks, its 4 pixel rows
// (16 * nb bytes each) land one after another, so block k of a segment that
// starts at unit block ks sits at 64 * ks + 16 * (k - ks) + r * 16 * nb.
// Units of images with 4-byte aligned rows, or narrower than an eighth of a
// unit, are not copied: their record says so and the compute warps load those
// blocks themselves.  A record with no blocks ends the CTA's work.
// ---------------------------------------------------------------------------
struct UnitRec {
    const uint8_t* src;
    uint8_t* dst;
    uint32_t stride, bw, bw_magic, codec;
    uint32_t first, n;  // first block of the unit in its image, blocks in the unit (0: no more units)
    uint32_t direct;    // 1: rows not copied (4-byte aligned source), blocks read from global memory
    uint32_t reserved;
};
static_assert(sizeof(UnitRec) == 48, "UnitRec layout");

constexpr size_t batch_tma_smem_bytes(const TmaLayout& l)
{
    return (size_t)l.stages * (l.stage_bytes + 16u + sizeof(UnitRec)) + 128u;
}

// PARAM_TABLES: the descriptor and first-unit tables are the kernel's
// parameter (readable before the dependency wait); otherwise they are device
// memory the stream wrote before this launch.
template <int BPT, int COMPUTE, bool PARAM_TABLES>
__device__ __forceinline__ void batch_tma_body(const BatchImage* __restrict__ images, uint32_t n_images,
                                               const uint32_t* __restrict__ first_unit, uint32_t total_units)
{
    pdl_launch_dependents();
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t abort_flag;
    constexpr uint32_t compute_warps = COMPUTE / 32;
    constexpr TmaLayout L = tma_layout(COMPUTE, BPT);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.stages * L.stage_bytes);
    uint64_t* empty = full + L.stages;
    UnitRec* rec = reinterpret_cast<UnitRec*>(empty + L.stages);
    uint8_t* ctrl_lut = reinterpret_cast<uint8_t*>(rec + L.stages);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;

    if (threadIdx.x == 0) init_ring(full, empty, L.stages, compute_warps, &abort_flag);
    fill_ctrl_lut(ctrl_lut);
    __syncthreads();
    if constexpr (PARAM_TABLES) {
        if (warp == compute_warps && lane == 0) {
            // While the previous kernel in the stream drains, ask L2 for the rows
            // of this CTA's first units (a hint, as in encode_image_tma: nothing
            // enters the CTA and nothing is written before pdl_wait()).
            uint32_t ii = 0;
            for (uint32_t u = blockIdx.x, k = 0; u < total_units && k < l2_prefetch_tiles(L); u += gridDim.x, ++k) {
                ii += find_image(first_unit + ii, n_images - ii, u);
                const BatchImage& im = images[ii];
                if (!im.vec16 || im.bw * 8u < L.tile_blocks) continue;  // units the compute warps load themselves
                const uint32_t first = (u - im.first_unit) * L.tile_blocks;
                const uint32_t n = min(L.tile_blocks, im.bw * im.bh - first);
                for (uint32_t gb = first; gb < first + n;) {
                    uint32_t bx;
                    const uint32_t by = div_magic(gb, im.bw, im.bw_magic, bx);
                    const uint32_t nb = min(im.bw - bx, first + n - gb);
                    const uint8_t* row = im.src + (size_t)by * 4u * im.stride + 16u * (size_t)bx;
#pragma unroll
                    for (int rr = 0; rr < 4; ++rr) bulk_prefetch_l2(row + (size_t)rr * im.stride, 16u * nb);
                    gb += nb;
                }
            }
        }
    }
    pdl_wait();  // no copy and no store before the previous kernel in the stream is done

    if (warp == compute_warps) {  // producer
        if (lane != 0) return;
        // Units u = blockIdx.x, + gridDim.x, ...: the image of the next unit and
        // its descriptor are looked up right after the current unit's copies are
        // issued, while the compute warps work; the search starts at the current
        // image (units only grow), so a batch of large images rarely searches.
        // Rows are read once: evict-first in L2, as in encode_image_tma.
        const uint64_t policy = l2_evict_first_policy();
        uint32_t issued = 0, slot = 0, phase = 0;
        uint32_t u = blockIdx.x, ii = 0;
        BatchImage im{};
        if (u < total_units) {
            ii = find_image(first_unit, n_images, u);
            im = images[ii];
        }
        for (;;) {
            if (issued >= L.stages && !mbar_wait(&empty[slot], phase ^ 1u, &abort_flag, &g_pipeline_timeouts))
                break;
            UnitRec& r = rec[slot];
            if (u >= total_units) {
                r.n = 0;  // published by the arrival (release), read after the wait (acquire)
                mbar_arrive(&full[slot]);
                ++issued;
                break;
            }
            const uint32_t first = (u - im.first_unit) * L.tile_blocks;
            const uint32_t n = min(L.tile_blocks, im.bw * im.bh - first);
            r.src = im.src;
            r.dst = im.dst;
            r.stride = im.stride;
            r.bw = im.bw;
            r.bw_magic = im.bw_magic;
            r.codec = im.codec;
            r.first = first;
            r.n = n;
            // narrow images would take many small copies per unit (one per pixel row of every
            // block row): a unit is copied only when it spans at most about 9 block rows
            const bool copy = im.vec16 && im.bw * 8u >= L.tile_blocks;
            r.direct = copy ? 0u : 1u;
            if (copy) {
                mbar_arrive_expect_tx(&full[slot], 64u * n);
                uint8_t* buf = smem + slot * L.stage_bytes;
                for (uint32_t g = first; g < first + n;) {
                    uint32_t bx;
                    const uint32_t by = div_magic(g, im.bw, im.bw_magic, bx);
                    const uint32_t nb = min(im.bw - bx, first + n - g);
                    const uint8_t* row = im.src + (size_t)by * 4u * im.stride + 16u * (size_t)bx;
                    uint8_t* d = buf + 64u * (g - first);
#pragma unroll
                    for (int rr = 0; rr < 4; ++rr)
                        bulk_copy_g2s_hint(d + rr * 16u * nb, row + (size_t)rr * im.stride, 16u * nb, &full[slot],
                                           policy);
                    g += nb;
                }
            } else {
                mbar_arrive(&full[slot]);
            }
            ++issued;
            if (++slot == L.stages) {
                slot = 0;
                phase ^= 1u;
            }
            u += gridDim.x;
            if (u < total_units && ii + 1 < n_images && first_unit[ii + 1] <= u) {
                ii += find_image(first_unit + ii, n_images - ii, u);
                im = images[ii];
            }
        }
        if (*static_cast<volatile uint32_t*>(&abort_flag)) {
            const uint32_t n = issued < L.stages ? issued : L.stages;
            for (uint32_t i = issued - n; i < issued; ++i)
                mbar_wait(&full[i % L.stages], (i / L.stages) & 1u, nullptr, &g_pipeline_timeouts);
        }
        return;
    }

    uint32_t slot = 0, phase = 0;
    for (;;) {
        if (!mbar_wait(&full[slot], phase, &abort_flag, &g_pipeline_timeouts)) break;
        const UnitRec r = rec[slot];
        if (r.n == 0) break;
        const uint8_t* buf = smem + slot * L.stage_bytes;
        uint32_t w[BPT][16];
#pragma unroll
        for (int j = 0; j < BPT; ++j) {
            const uint32_t k = (warp * BPT + j) * 32u + lane;
            if (k < r.n) {
                uint32_t bx;
                const uint32_t by = div_magic(r.first + k, r.bw, r.bw_magic, bx);
                if (r.direct) {
                    load_block_rows(r.src + (size_t)by * 4u * r.stride + 16u * (size_t)bx, r.stride, false, w[j]);
                } else {
                    const uint32_t row0 = by * r.bw;  // first block of this block row
                    const uint32_t ks = row0 > r.first ? row0 - r.first : 0u;
                    const uint32_t nb = min(row0 + r.bw, r.first + r.n) - max(row0, r.first);
                    const uint8_t* p = buf + 64u * ks + 16u * (k - ks);
#pragma unroll
                    for (int rr = 0; rr < 4; ++rr) {
                        const uint4 v = *reinterpret_cast<const uint4*>(p + rr * 16u * nb);
                        w[j][4 * rr + 0] = v.x;
                        w[j][4 * rr + 1] = v.y;
                        w[j][4 * rr + 2] = v.z;
                        w[j][4 * rr + 3] = v.w;
                    }
                }
            }
        }
#pragma unroll
        for (int j = 0; j < BPT; ++j) {
            const uint32_t k = (warp * BPT + j) * 32u + lane;
            if (k < r.n) {
                const uint2 e = r.codec == kBC1 ? encode_bc1(w[j]) : encode_etc1s(w[j], ctrl_lut);
                st_stream8(r.dst + 8u * (size_t)(r.first + k), e);
            }
        }
        // released only after the stores, which wait for every loaded word (see encode_image_tma)
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[slot]);
        if (++slot == L.stages) {
            slot = 0;
            phase ^= 1u;
        }
    }
}

// Descriptor and first-unit tables in device memory (uploaded per call).
template <int BPT, int COMPUTE>
__global__ void __launch_bounds__(COMPUTE + 32, tma_min_ctas(BPT, COMPUTE))
    encode_batch_tma(const BatchImage* __restrict__ images, uint32_t n_images, const uint32_t* __restrict__ first_unit,
                     uint32_t total_units)
{
    batch_tma_body<BPT, COMPUTE, false>(images, n_images, first_unit, total_units);
}

// The same tables in the kernel's parameter space (small batches).
template <int BPT, int COMPUTE>
__global__ void __launch_bounds__(COMPUTE + 32, tma_min_ctas(BPT, COMPUTE))
    encode_batch_tma_inline(const __grid_constant__ InlineBatch batch, uint32_t n_images, uint32_t total_units)
{
    batch_tma_body<BPT, COMPUTE, true>(batch.images, n_images, batch.first_unit, total_units);
}

namespace {

// Resident CTAs of a ring kernel on the current device, kept per device in
// `resident`; the first call opts in to its shared memory.
template <typename K>
cudaError_t resident_ctas_of(K kernel, uint32_t threads, size_t smem, std::atomic<int> (&resident)[64], int* out)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    int ctas = resident[dev].load(std::memory_order_relaxed);
    if (ctas == 0) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)threads, smem);
        if (e != cudaSuccess) return e;
        ctas = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
        resident[dev].store(ctas, std::memory_order_relaxed);
    }
    *out = ctas;
    return cudaSuccess;
}

template <int CODEC, int BPT, int COMPUTE, bool WORD>
cudaError_t launch_tma_t(const uint8_t* src, size_t stride, uint8_t* dst, uint8_t* dst2, uint32_t bw, uint32_t bh,
                         cudaStream_t stream)
{
    constexpr TmaLayout L = tma_layout(COMPUTE, BPT, WORD);
    const size_t smem = tma_smem_bytes(L);
    const auto kernel = encode_image_tma<CODEC, BPT, COMPUTE, WORD>;
    static std::atomic<int> resident[64];
    int ctas = 0;
    const cudaError_t e = resident_ctas_of(kernel, COMPUTE + 32, smem, resident, &ctas);
    if (e != cudaSuccess) return e;
    const uint32_t total = bw * bh, units = (total + L.tile_blocks - 1) / L.tile_blocks;
    const uint32_t grid = std::min(units, (uint32_t)ctas);
    return launch_pdl(kernel, dim3(grid), dim3(COMPUTE + 32), smem, stream, src, stride, dst, dst2, bw,
                      0xffffffffu / bw, total);
}

template <int CODEC, int BPT>
cudaError_t launch_tma_bpt(const uint8_t* src, size_t stride, uint8_t* dst, uint8_t* dst2, uint32_t bw, uint32_t bh,
                           uint32_t threads, cudaStream_t stream)
{
    switch (threads) {
    case 128: return launch_tma_t<CODEC, BPT, 128, false>(src, stride, dst, dst2, bw, bh, stream);
    case 256: return launch_tma_t<CODEC, BPT, 256, false>(src, stride, dst, dst2, bw, bh, stream);
    case 512: return launch_tma_t<CODEC, BPT, 512, false>(src, stride, dst, dst2, bw, bh, stream);
    default: return cudaErrorInvalidValue;
    }
}

// Word-aligned rows come in two shapes, 512 x 2 and 128 x 1.
template <int CODEC>
cudaError_t launch_tma_word(const uint8_t* src, size_t stride, uint8_t* dst, uint8_t* dst2, uint32_t bw, uint32_t bh,
                            bool big, cudaStream_t stream)
{
    return big ? launch_tma_t<CODEC, 2, 512, true>(src, stride, dst, dst2, bw, bh, stream)
               : launch_tma_t<CODEC, 1, 128, true>(src, stride, dst, dst2, bw, bh, stream);
}

}  // namespace

cudaError_t launch_image_tma(int codec, const uint8_t* src, size_t stride, uint8_t* dst, uint32_t width,
                             uint32_t height, Tile tile, SrcAccess access, cudaStream_t stream, uint8_t* dst2)
{
    const uint32_t bw = width / 4, bh = height / 4;
    if (bw == 0 || bh == 0) return cudaSuccess;
    const uint32_t align = access == SrcAccess::kVec16 ? 16 : 4;
    if (reinterpret_cast<uintptr_t>(src) % align || stride % align) return cudaErrorInvalidValue;
    if (codec == kBoth && !dst2) return cudaErrorInvalidValue;
    if (access == SrcAccess::kWord4) {
        const bool big = tile.threads == 512 && tile.bpt == 2;
        if (!word_rows_fit(big ? 1024 : 128, bw)) return cudaErrorInvalidValue;
        if (codec == kBC1) return launch_tma_word<kBC1>(src, stride, dst, nullptr, bw, bh, big, stream);
        if (codec == kETC1S) return launch_tma_word<kETC1S>(src, stride, dst, nullptr, bw, bh, big, stream);
        if (codec == kBoth) return launch_tma_word<kBoth>(src, stride, dst, dst2, bw, bh, big, stream);
        return cudaErrorInvalidValue;
    }
    if (codec == kBC1) {
        if (tile.bpt == 1) return launch_tma_bpt<kBC1, 1>(src, stride, dst, nullptr, bw, bh, tile.threads, stream);
        if (tile.bpt == 2) return launch_tma_bpt<kBC1, 2>(src, stride, dst, nullptr, bw, bh, tile.threads, stream);
    } else if (codec == kETC1S) {
        if (tile.bpt == 1) return launch_tma_bpt<kETC1S, 1>(src, stride, dst, nullptr, bw, bh, tile.threads, stream);
        if (tile.bpt == 2) return launch_tma_bpt<kETC1S, 2>(src, stride, dst, nullptr, bw, bh, tile.threads, stream);
    } else if (codec == kBoth) {
        if (tile.bpt == 1) return launch_tma_bpt<kBoth, 1>(src, stride, dst, dst2, bw, bh, tile.threads, stream);
        if (tile.bpt == 2) return launch_tma_bpt<kBoth, 2>(src, stride, dst, dst2, bw, bh, tile.threads, stream);
    }
    return cudaErrorInvalidValue;
}

namespace {

template <int CODEC, bool WORD>
cudaError_t launch_error_t(const uint8_t* blocks, const uint8_t* src, size_t stride, uint32_t bw, uint32_t bh,
                           unsigned long long* sums, ErrorResult result, cudaStream_t stream)
{
    constexpr int BPT = 2, COMPUTE = 512;
    constexpr TmaLayout L = tma_layout(COMPUTE, BPT, WORD);
    constexpr size_t smem = (size_t)L.stages * (L.stage_bytes + 16u);
    const auto kernel = error_image_tma<CODEC, BPT, COMPUTE, WORD>;
    static std::atomic<int> resident[64];
    int ctas = 0;
    const cudaError_t e = resident_ctas_of(kernel, COMPUTE + 32, smem, resident, &ctas);
    if (e != cudaSuccess) return e;
    const uint32_t total = bw * bh, units = (total + L.tile_blocks - 1) / L.tile_blocks;
    // a thread's sums hold kErrorSumBlocks blocks
    const uint32_t least = (uint32_t)(((uint64_t)units * BPT + kErrorSumBlocks - 1) / kErrorSumBlocks);
    const uint32_t grid = std::max(least, std::min(units, (uint32_t)ctas));
    return launch_pdl(kernel, dim3(grid), dim3(COMPUTE + 32), smem, stream, blocks, src, stride, bw, 0xffffffffu / bw,
                      total, sums, result);
}

}  // namespace

cudaError_t launch_error_tma(int codec, const uint8_t* blocks, const uint8_t* src, uint32_t width, uint32_t height,
                             size_t stride, bool vec16, unsigned long long* sums, ErrorResult result,
                             cudaStream_t stream)
{
    const uint32_t bw = width / 4, bh = height / 4;
    if (!vec16 && !word_rows_fit(1024, bw)) return cudaErrorInvalidValue;
    if (codec == kBC1)
        return vec16 ? launch_error_t<kBC1, false>(blocks, src, stride, bw, bh, sums, result, stream)
                     : launch_error_t<kBC1, true>(blocks, src, stride, bw, bh, sums, result, stream);
    return vec16 ? launch_error_t<kETC1S, false>(blocks, src, stride, bw, bh, sums, result, stream)
                 : launch_error_t<kETC1S, true>(blocks, src, stride, bw, bh, sums, result, stream);
}

namespace {

template <int BPT, int COMPUTE>
int batch_tma_ctas_t(int dev)
{
    constexpr TmaLayout L = tma_layout(COMPUTE, BPT);
    constexpr size_t smem = batch_tma_smem_bytes(L);
    static std::atomic<int> resident[64];
    if (dev < 0 || dev >= 64) return 0;
    int ctas = resident[dev].load(std::memory_order_relaxed);
    if (ctas == 0) {
        if (cudaFuncSetAttribute(encode_batch_tma<BPT, COMPUTE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem) != cudaSuccess ||
            cudaFuncSetAttribute(encode_batch_tma<BPT, COMPUTE>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared) != cudaSuccess)
            return 0;
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_batch_tma<BPT, COMPUTE>, COMPUTE + 32,
                                                          smem) != cudaSuccess)
            return 0;
        ctas = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
        resident[dev].store(ctas, std::memory_order_relaxed);
    }
    return ctas;
}

template <int BPT, int COMPUTE>
cudaError_t launch_batch_tma_t(const BatchImage* images, uint32_t n_images, const uint32_t* first_unit,
                               uint32_t total_units, uint32_t* work_counter, uint32_t ctas, cudaStream_t stream)
{
    (void)work_counter;  // units are dealt to CTAs statically
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const int resident = batch_tma_ctas_t<BPT, COMPUTE>(dev);
    if (resident == 0) return cudaErrorInvalidValue;
    if (ctas > (uint32_t)resident) ctas = (uint32_t)resident;
    constexpr size_t smem = batch_tma_smem_bytes(tma_layout(COMPUTE, BPT));
    return launch_pdl(encode_batch_tma<BPT, COMPUTE>, dim3(ctas ? ctas : 1u), dim3(COMPUTE + 32), smem, stream,
                      images, n_images, first_unit, total_units);
}

template <int BPT, int COMPUTE>
cudaError_t launch_batch_tma_inline_t(const InlineBatch& batch, uint32_t n_images, uint32_t total_units, uint32_t ctas,
                                      cudaStream_t stream)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const int resident = batch_tma_ctas_t<BPT, COMPUTE>(dev);
    if (resident == 0 || dev < 0 || dev >= 64) return cudaErrorInvalidValue;
    constexpr size_t smem = batch_tma_smem_bytes(tma_layout(COMPUTE, BPT));
    static std::atomic<bool> ready[64];
    if (!ready[dev].load(std::memory_order_relaxed)) {
        e = cudaFuncSetAttribute(encode_batch_tma_inline<BPT, COMPUTE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(encode_batch_tma_inline<BPT, COMPUTE>,
                                     cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        ready[dev].store(true, std::memory_order_relaxed);
    }
    if (ctas > (uint32_t)resident) ctas = (uint32_t)resident;
    return launch_pdl(encode_batch_tma_inline<BPT, COMPUTE>, dim3(ctas ? ctas : 1u), dim3(COMPUTE + 32), smem,
                      stream, batch, n_images, total_units);
}

}  // namespace

cudaError_t launch_batch_tma_inline(const InlineBatch& batch, uint32_t n_images, uint32_t total_units,
                                    const BatchTile& tile, uint32_t ctas, cudaStream_t stream)
{
    if (total_units == 0) return cudaSuccess;
    if (n_images > kInlineImages || tile.unit_blocks != tile.threads * tile.bpt) return cudaErrorInvalidValue;
    const uint32_t t = tile.threads;
    if (tile.bpt == 1) {
        if (t == 128) return launch_batch_tma_inline_t<1, 128>(batch, n_images, total_units, ctas, stream);
        if (t == 256) return launch_batch_tma_inline_t<1, 256>(batch, n_images, total_units, ctas, stream);
        if (t == 512) return launch_batch_tma_inline_t<1, 512>(batch, n_images, total_units, ctas, stream);
    } else if (tile.bpt == 2) {
        if (t == 128) return launch_batch_tma_inline_t<2, 128>(batch, n_images, total_units, ctas, stream);
        if (t == 256) return launch_batch_tma_inline_t<2, 256>(batch, n_images, total_units, ctas, stream);
        if (t == 512) return launch_batch_tma_inline_t<2, 512>(batch, n_images, total_units, ctas, stream);
    }
    return cudaErrorInvalidValue;
}

int batch_tma_resident_ctas(uint32_t threads, uint32_t bpt)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    int n = 0;
    if (bpt == 1) n = threads == 128 ? batch_tma_ctas_t<1, 128>(dev) : threads == 256 ? batch_tma_ctas_t<1, 256>(dev)
                                                                                      : batch_tma_ctas_t<1, 512>(dev);
    else n = threads == 128 ? batch_tma_ctas_t<2, 128>(dev) : threads == 256 ? batch_tma_ctas_t<2, 256>(dev)
                                                                             : batch_tma_ctas_t<2, 512>(dev);
    return n > 0 ? n : 1;
}

cudaError_t launch_batch_tma(const BatchImage* images, uint32_t n_images, const uint32_t* first_unit,
                             uint32_t total_units, uint32_t* work_counter, const BatchTile& tile, uint32_t ctas,
                             cudaStream_t stream)
{
    if (total_units == 0) return cudaSuccess;
    if (tile.unit_blocks != tile.threads * tile.bpt) return cudaErrorInvalidValue;
    const uint32_t t = tile.threads;
    if (tile.bpt == 1) {
        if (t == 128) return launch_batch_tma_t<1, 128>(images, n_images, first_unit, total_units, work_counter, ctas, stream);
        if (t == 256) return launch_batch_tma_t<1, 256>(images, n_images, first_unit, total_units, work_counter, ctas, stream);
        if (t == 512) return launch_batch_tma_t<1, 512>(images, n_images, first_unit, total_units, work_counter, ctas, stream);
    } else if (tile.bpt == 2) {
        if (t == 128) return launch_batch_tma_t<2, 128>(images, n_images, first_unit, total_units, work_counter, ctas, stream);
        if (t == 256) return launch_batch_tma_t<2, 256>(images, n_images, first_unit, total_units, work_counter, ctas, stream);
        if (t == 512) return launch_batch_tma_t<2, 512>(images, n_images, first_unit, total_units, work_counter, ctas, stream);
    }
    return cudaErrorInvalidValue;
}

// Thread 0 waits on an mbarrier that expects one arrival and gets none.
// Nothing is copied into the CTA, so nothing is in flight when it returns.
__global__ void bounded_wait_selftest_kernel(unsigned int* counter, uint32_t* out)
{
    __shared__ uint64_t bar;
    __shared__ uint32_t abort_flag;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1u);
    abort_flag = 0u;
    mbar_init_fence();
    const bool completed = mbar_wait(&bar, 0u, &abort_flag, counter);
    out[0] = completed ? 1u : 0u;
    out[1] = abort_flag;
}

cudaError_t bounded_wait_selftest(bool* completed, bool* aborted, unsigned int* counted)
{
    uint32_t* d = nullptr;  // {counter, wait result, abort flag}
    cudaError_t e = cudaMalloc(&d, 3 * sizeof(uint32_t));
    if (e != cudaSuccess) return e;
    uint32_t h[3] = {0, 0, 0};
    e = cudaMemset(d, 0, 3 * sizeof(uint32_t));
    if (e == cudaSuccess) {
        bounded_wait_selftest_kernel<<<1, 32>>>(d, d + 1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(d);
    *counted = h[0];
    *completed = h[1] != 0;
    *aborted = h[2] != 0;
    return e;
}

cudaError_t pipeline_timeouts(unsigned int* count, bool reset)
{
    cudaError_t e = cudaMemcpyFromSymbol(count, g_pipeline_timeouts, sizeof(unsigned int));
    if (e == cudaSuccess && reset) {
        const unsigned int zero = 0;
        e = cudaMemcpyToSymbol(g_pipeline_timeouts, &zero, sizeof(unsigned int));
    }
    return e;
}

}  // namespace goofy_gpu
