// encode_kernels.cu -- image encoder kernels for sm_103a.
//
// Replaces the reference's image driver loops (goofy::compressDXT1 /
// compressETC1, GoofyTC/goofy_tc.h:1497-1557: block rows x 16-pixel strips,
// 4 blocks per goofySimdEncode call) with a grid over 4x4 blocks.
//
// Mapping: one warp owns a segment of 32*BPT consecutive blocks of the image
// in row-major order; lane l encodes blocks l, l+32, ..., l+32*(BPT-1) of the
// segment.  For each of the 4 pixel rows a warp-wide 128-bit load instruction
// therefore reads 512 contiguous bytes (every 32-byte sector fully used; two
// runs where the segment crosses into the next block row), and each 8-byte
// block store of the warp writes 256 contiguous bytes.  Segments that ended
// with their block row left most lanes idle on narrow images (120x8000 ETC1s:
// 7.0 us then, 2.0 us so).  Source rows are
// read once (L1 no-allocate) and blocks are written with streaming stores:
// the kernel moves 4 B/px in and 0.5 B/px out and is meant to sit on the HBM
// roofline.  Launched with programmatic dependent launch (pdl.cuh): CTAs may
// start while the previous kernel in the stream drains and wait for it before
// their first load.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "block_codec.cuh"
#include "device_io.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace goofy_gpu {

// Where a grid's rows are and whether it asks L2 for them early.  Launches on
// rows in host memory give shared memory the largest share of L1: 2048^2 ETC1s
// 96.4 us a call against 98.7, BC1 96.5 against 99.2 (device rows lose by it:
// 2048^2 ETC1s 4.4 against 3.9).
enum class Rows { kDevice, kAhead, kHost };

template <SrcAccess ACCESS>
__device__ __forceinline__ void load_block(const uint8_t* p, size_t stride, uint32_t (&w)[16])
{
    load_block_rows(p, stride, ACCESS == SrcAccess::kVec16, w);
}

// The first pixel of block b of the image in row-major order.
__device__ __forceinline__ const uint8_t* block_address(const uint8_t* src, size_t stride, uint32_t bw,
                                                        uint32_t bw_magic, uint32_t b)
{
    uint32_t bx;
    const uint32_t by = div_magic(b, bw, bw_magic, bx);
    return src + (size_t)by * 4u * stride + 16u * (size_t)bx;
}

// Loads this lane's blocks of segment `seg`: blocks b0, b0 + 32, ... of the
// image in row-major order (b0 returned), so a segment runs on from one block
// row into the next and only the image's last one is short.
template <int BPT, SrcAccess ACCESS>
__device__ __forceinline__ uint32_t load_segment(const uint8_t* __restrict__ src, size_t stride, uint32_t bw,
                                                 uint32_t bw_magic, uint32_t total, uint32_t seg, uint32_t lane,
                                                 uint32_t (&w)[BPT][16])
{
    const uint32_t b0 = seg * (32u * BPT) + lane;
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
        const uint32_t b = b0 + 32u * j;
        if (b < total) load_block<ACCESS>(block_address(src, stride, bw, bw_magic, b), stride, w[j]);
    }
    return b0;
}

template <int CODEC, int BPT, typename Lut>
__device__ __forceinline__ void encode_segment(uint8_t* __restrict__ dst, uint8_t* __restrict__ dst2, uint32_t total,
                                               uint32_t b0, const uint32_t (&w)[BPT][16], Lut ctrl_lut)
{
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
        const uint32_t b = b0 + 32u * j;
        if (b < total) {
            if constexpr (CODEC == kBoth) {
                const uint4 e = encode_both(w[j], ctrl_lut);
                st_stream8(dst + 8u * (size_t)b, make_uint2(e.x, e.y));
                st_stream8(dst2 + 8u * (size_t)b, make_uint2(e.z, e.w));
            } else {
                st_stream8(dst + 8u * (size_t)b, encode_block<CODEC>(w[j], ctrl_lut));
            }
        }
    }
}

// One segment per warp: every lane issues its 4*BPT row loads up front.
//
// PREFETCH (device memory): before the dependency wait, while the previous
// kernel in the stream drains, the warp asks L2 for the lines of its rows
// (every eighth lane's addresses are 128 bytes apart).  Only a hint: the loads
// after the wait read what that kernel wrote.  An image whose CTAs are all
// resident at once is then on its way to L2 before its turn comes.  Launches
// back to back, inputs of 400 MB in all, without / with (us): 256^2 BC1 1.6 / 1.2,
// ETC1s 1.8 / 1.3, 2048^2 BC1 4.6 / 3.7, 8192^2 BC1 45.5 / 43.  Segments of two
// to four steps a warp, all asked for ahead, were slower at every size.
//
// The register caps are for CTAs that fit on an SM (CTAs of 512 a cap allows).
// Without PREFETCH, on images of more than a wave, two blocks a thread of ETC1s
// or both codecs are held to 64: at the 66 to 73 that they take by themselves
// an SM has one CTA of 512 threads instead of two (8192^2 ETC1s 67.8 against
// 51.3 us, both 76.4 / 59.8) and three of 256 instead of four (53.1 / 50.5).
// Word-aligned ETC1s takes 62 anyway and would spill.
template <int CODEC, int BPT, SrcAccess ACCESS, bool PREFETCH>
constexpr int grid_min_ctas()
{
    if (!PREFETCH) return BPT == 2 && (CODEC == kBoth || (CODEC == kETC1S && ACCESS == SrcAccess::kVec16)) ? 2 : 1;
    return BPT > 1 || ACCESS == SrcAccess::kWord4 ? 1 : CODEC == kBC1 ? 4 : 3;
}

template <int CODEC, int BPT, SrcAccess ACCESS, bool PREFETCH>
__global__ void __launch_bounds__(512, (grid_min_ctas<CODEC, BPT, ACCESS, PREFETCH>()))
    encode_image_kernel(const uint8_t* __restrict__ src, size_t stride, uint8_t* __restrict__ dst,
                        uint8_t* __restrict__ dst2, uint32_t bw, uint32_t bw_magic, uint32_t total)
{
    pdl_launch_dependents();
    constexpr bool kLut = CODEC != kBC1 && BPT * (CODEC == kBoth ? 2 : 1) >= 4;  // see control_byte
    __shared__ uint8_t ctrl_lut[kLut ? 128 : 1];
    if constexpr (kLut) {
        fill_ctrl_lut(ctrl_lut);
        __syncthreads();
    }
    const uint32_t seg = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (seg * (32u * BPT) >= total) return;
    const uint32_t b0 = seg * (32u * BPT) + lane;
    const uint8_t* p[BPT];
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
        p[j] = block_address(src, stride, bw, bw_magic, min(b0 + 32u * j, total - 1u));
        if (PREFETCH && !(lane & 7u)) {
#pragma unroll
            for (int y = 0; y < 4; ++y) prefetch_l2(p[j] + y * stride);
        }
    }
    pdl_wait();
    uint32_t w[BPT][16];
#pragma unroll
    for (int j = 0; j < BPT; ++j)
        if (b0 + 32u * j < total) load_block<ACCESS>(p[j], stride, w[j]);
    if constexpr (kLut) encode_segment<CODEC, BPT, const uint8_t*>(dst, dst2, total, b0, w, ctrl_lut);
    else encode_segment<CODEC, BPT>(dst, dst2, total, b0, w, NoLut{});
}

// Persistent grid: warp-segments are dealt round-robin to the resident warps;
// each warp loads its next segment before encoding the current one, so the
// 64*BPT bytes per lane of the next segment are in flight during the math.
template <int CODEC, int BPT, SrcAccess ACCESS>
__global__ void __launch_bounds__(512) encode_image_persistent(const uint8_t* __restrict__ src, size_t stride,
                                                               uint8_t* __restrict__ dst, uint32_t bw,
                                                               uint32_t bw_magic, uint32_t total)
{
    pdl_launch_dependents();
    __shared__ uint8_t ctrl_lut[128];
    if constexpr (CODEC == kETC1S) {
        fill_ctrl_lut(ctrl_lut);
        __syncthreads();
    }
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp_stride = gridDim.x * (blockDim.x >> 5);
    const uint32_t segs = (total + 32u * BPT - 1u) / (32u * BPT);
    uint32_t seg = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    uint32_t a[BPT][16], b[BPT][16], ba = 0, bb = 0;
    if (seg < segs) ba = load_segment<BPT, ACCESS>(src, stride, bw, bw_magic, total, seg, lane, a);
    while (seg < segs) {
        uint32_t next = seg + warp_stride;
        if (next < segs) bb = load_segment<BPT, ACCESS>(src, stride, bw, bw_magic, total, next, lane, b);
        encode_segment<CODEC, BPT, const uint8_t*>(dst, nullptr, total, ba, a, ctrl_lut);
        seg = next;
        if (seg >= segs) break;
        next = seg + warp_stride;
        if (next < segs) ba = load_segment<BPT, ACCESS>(src, stride, bw, bw_magic, total, next, lane, a);
        encode_segment<CODEC, BPT, const uint8_t*>(dst, nullptr, total, bb, b, ctrl_lut);
        seg = next;
    }
}

template <int CODEC, int BPT, SrcAccess ACCESS>
static int resident_ctas(uint32_t threads)
{
    // cached per instantiation, device and block size
    static std::atomic<int> cached[64][3];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    const int slot = threads == 128 ? 0 : threads == 256 ? 1 : 2;
    int n = cached[dev][slot].load(std::memory_order_relaxed);
    if (n == 0) {
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_image_persistent<CODEC, BPT, ACCESS>, threads, 0);
        n = (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
        cached[dev][slot].store(n, std::memory_order_relaxed);
    }
    return n;
}

template <int CODEC, int BPT, SrcAccess ACCESS>
static cudaError_t launch_t(const uint8_t* src, size_t stride, uint8_t* dst, uint8_t* dst2, uint32_t bw, uint32_t bh,
                            uint32_t threads, bool persistent, Rows rows, cudaStream_t stream)
{
    constexpr bool kHasPersistent = BPT <= 2 && CODEC != kBoth;
    const uint32_t total = bw * bh, magic = 0xffffffffu / bw;
    const uint32_t per_cta = threads * BPT;
    uint64_t ctas = ((uint64_t)total + per_cta - 1) / per_cta;
    if constexpr (kHasPersistent) {
        if (persistent) {
            const uint64_t resident = (uint64_t)resident_ctas<CODEC, BPT, ACCESS>(threads);
            if (ctas > resident) ctas = resident;
            return launch_pdl(encode_image_persistent<CODEC, BPT, ACCESS>, dim3((unsigned)ctas), dim3(threads), 0,
                              stream, src, stride, dst, bw, magic, total);
        }
    }
    return launch_pdl_carveout(rows == Rows::kHost ? 100 : -1,
                               rows == Rows::kAhead ? encode_image_kernel<CODEC, BPT, ACCESS, true>
                                                    : encode_image_kernel<CODEC, BPT, ACCESS, false>,
                               dim3((unsigned)ctas), dim3(threads), 0, stream, src, stride, dst, dst2, bw, magic, total);
}

template <int CODEC, SrcAccess ACCESS>
static cudaError_t launch_bpt(const uint8_t* src, size_t stride, uint8_t* dst, uint8_t* dst2, uint32_t bw,
                              uint32_t bh, Tile tile, Rows rows, cudaStream_t stream)
{
    switch (tile.bpt) {
    case 1: return launch_t<CODEC, 1, ACCESS>(src, stride, dst, dst2, bw, bh, tile.threads, tile.persistent, rows, stream);
    case 2: return launch_t<CODEC, 2, ACCESS>(src, stride, dst, dst2, bw, bh, tile.threads, tile.persistent, rows, stream);
    case 4:
        if constexpr (CODEC != kBoth) return launch_t<CODEC, 4, ACCESS>(src, stride, dst, dst2, bw, bh, tile.threads, false, rows, stream);
        return cudaErrorInvalidValue;
    default: return cudaErrorInvalidValue;
    }
}

template <int CODEC>
static cudaError_t launch_access(const uint8_t* src, size_t stride, uint8_t* dst, uint8_t* dst2, uint32_t bw,
                                 uint32_t bh, Tile tile, SrcAccess access, Rows rows, cudaStream_t stream)
{
    if (access == SrcAccess::kVec16)
        return launch_bpt<CODEC, SrcAccess::kVec16>(src, stride, dst, dst2, bw, bh, tile, rows, stream);
    return launch_bpt<CODEC, SrcAccess::kWord4>(src, stride, dst, dst2, bw, bh, tile, rows, stream);
}

cudaError_t launch_image(int codec, const uint8_t* src, size_t stride, uint8_t* dst, uint32_t width,
                         uint32_t height, Tile tile, SrcAccess access, cudaStream_t stream, uint8_t* dst2, bool host_rows)
{
    if (!tile_valid(tile) || (host_rows && tile.persistent == 2)) return cudaErrorInvalidValue;
    if (codec != kBC1 && codec != kETC1S && (codec != kBoth || !dst2)) return cudaErrorInvalidValue;
    const uint32_t bw = width / 4, bh = height / 4;
    if (bw == 0 || bh == 0) return cudaSuccess;
    constexpr uint64_t kMostBlocks = 1u << 30;  // a launch numbers its blocks in 32 bits
    if ((uint64_t)bw * bh > kMostBlocks) {      // in bands of block rows (a row has fewer: its stride is 32 bits)
        const uint32_t band = (uint32_t)(kMostBlocks / bw);
        for (uint32_t y = 0; y < bh; y += std::min(band, bh - y)) {
            const size_t out = (size_t)y * bw * 8u;
            const cudaError_t e = launch_image(codec, src + (size_t)y * 4u * stride, stride, dst + out, width,
                                               4u * std::min(band, bh - y), tile, access, stream,
                                               dst2 ? dst2 + out : nullptr, host_rows);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    Rows rows = host_rows ? Rows::kHost : Rows::kDevice;
    if (tile.persistent == 2) {
        // Launches back to back over inputs of 400 MB in all (us), BC1 / ETC1s / both:
        //                            grid 128x1           grid 128x2           bulk copy 128x1      bulk copy 512x2
        //   256^2     (4096 blocks)   1.2 / 1.3 / 1.35     1.3 / 1.4 / 1.5      1.6 / 1.7 / 1.7      4.1 / 4.4 / 4.7
        //   512^2     (16384)         1.35 / 2.0 / 2.4     1.4 / 2.4 / 2.4      2.2 / 2.3 / 2.8      3.1 / 3.5 / 3.8
        //   1024^2    (65536)         2.25 / 2.7 / 3.05    2.8 / 2.7 / 2.8      2.6 / 2.45 / 3.05    2.8 / 3.2 / 3.4
        //   2048x1800 (230400)        3.4 / 3.8 / 4.2      3.7 / 4.1 / 4.4      4.3 / 4.55 / 5.2
        //   2048^2    (262144)        3.65 / 4.8 / 5.2     3.8 / 4.4 / 5.0      4.55 / 4.9 / 5.65    4.8 / 5.5 / 6.1
        //   2400x2048 (307200)        4.1 / 5.3 / 5.8      4.15 / 6.45 / 7.15   5.0 / 5.45 / 6.3
        //   3000x2048 (384000)         -  / 6.2 / 6.75      -  / 6.6 / 8.2       -  / 6.1 / 7.0
        //   3840x2160 (518400)        6.25 / 8.8 / 9.7     6.5 / 8.0 / 8.95     6.65 / 7.3 / 8.4     7.1 / 8.1 / 9.0
        //   4096x3000 (768000)        8.7 / 12.0 / 13.2    9.1 / 12.3 / 12.6    9.6 / 10.4 / 12.8    9.3 / 10.4 / 12.0
        //   4096^2    (1048576)      11.6 / 14.7 / 16.5   11.9 / 14.9 / 16.6   12.3 / 13.45 / 15.55 11.5 / 12.6 / 14.7
        //   8192^2    (4194304)      43.0 / 54.1 / 61.0   43.7 / 49.4 / 66.8   48.6 / 47.5 / 52.8   45.8 / 45.8 / 50.1
        //   256x32768 (524288)        6.2 / 8.6 / 9.9      7.2 / 7.7 / 8.8      6.8 / 7.8 / 8.4     13.2 / 13.5 / 14.2
        //   64x16000  (64000)         2.1 / 2.7 / 3.2      1.8 / 2.5 / 2.35     3.2 / 3.0 / 3.7     10.0 / 10.3 / 10.7
        // (With 3 inputs, mostly in L2, ETC1s and both, grid 128x1 / bulk copy: 2400x2048 4.6 / 4.9 and 5.1 / 5.35,
        // 3000x2048 5.3 / 5.7 and 5.95 / 6.3.)  Word-aligned rows, BC1 / ETC1s, both where given:
        //   1024^2    (65536)         2.8 / 2.9 / 3.0      2.8 / 4.0 / 3.6      2.9 / 2.75 / 3.3
        //   1996x1532 (191117)        3.4 / 4.4 / 4.6      4.4 / 4.7 / 4.1      4.1 / 4.6 / 5.1
        //   2048x1800 (230400)        3.6 / 4.85 / 5.1     4.6 / 4.7 / 4.8      4.8 / 5.1 / 5.6
        //   2376x2628 (390258)        5.9 / 7.4 / 7.85     5.7 / 7.45 / 7.9     6.2 / 6.75 / 7.8
        //   3840x2160 (518400)        7.2 / 9.5            7.15 / 8.8           7.3 / 8.5
        //   4096^2                   13.2 / 17.9          13.2 / 17.0          13.4 / 14.9          12.3 / 13.9
        //
        // A grid whose CTAs are all resident at once has its rows prefetched while the launch before it drains; two
        // blocks a thread let a few more of them be resident.  Beyond, BC1 keeps enough warps in flight to stay at the
        // memory's rate up to about a million blocks (8192^2: 43 to 45.7 us, the pipeline 44.9 to 45.8), 600,000 where
        // each row takes four loads; the other codecs' longer blocks do not, and from 1.7 waves on take the pipeline,
        // whose copies run ahead of the codec.  One big CTA a SM leaves SMs idle in its last round on images of few
        // units, and its one copy queue is slow on short rows.
        constexpr uint32_t kTinyBlocks = 20000, kTinyRow = 32, kBigBlocks = 600000, kBigRow = 256;
        const bool word = access == SrcAccess::kWord4;
        // One block a thread up to grid1, two (where it can be) up to grid2.  With 16-byte rows these are the blocks
        // resident at 128x1 and 128x2, by the kernels' registers.  Word-aligned kernels take more (BC1 34, ETC1s 53 at
        // 128x1: waves of 233,472 and 175,104 blocks; both 73 at 128x2: 233,472), but a little past a wave the next
        // choice is still slower, in L2 / from HBM: BC1 1940x1944 (235,710) 3.6 / 4.0 against 4.2 / 4.5, 2180^2
        // (297,025) 4.2 / 4.6 against 4.4 / 4.7, from 2228^2 (310,249) on alike; ETC1s 1760x1756 (193,160) 3.9 / 4.4
        // against 4.6 / 4.8; both 2048^2 4.9 / 6.45 against 5.9 / 6.5.
        const uint32_t grid1 = kSms * 128 * (codec == kBC1 ? 16 : !word ? 12 : codec == kETC1S ? 10 : 9);
        const uint32_t grid2 = kSms * 256 * (word && codec == kETC1S ? 8 : 7);
        const uint32_t blocks = bw * bh;
        const bool by_size = tile.threads == 512 && tile.bpt == 2;
        bool grid = blocks < kTinyBlocks || bw < kTinyRow;
        if (by_size) grid |= blocks <= (codec == kBC1 ? (word ? 600000 : 900000) : word ? grid2 : 400000);
        if (!grid) {
            if (by_size && (blocks < kBigBlocks || bw < kBigRow)) tile = Tile{128, 1, 2};
            return launch_image_tma(codec, src, stride, dst, width, height, tile, access, stream, dst2);
        }
        const bool two = blocks > grid1 && (word || (codec != kBC1 && blocks <= grid2));
        tile = Tile{128, two ? 2u : 1u, 0};
        rows = Rows::kAhead;
    } else if (tile.persistent == 0 && !host_rows) {
        // A grid asked for by its shape has its rows prefetched as well, without / with, us, in L2 and from HBM:
        //   128x1 BC1    2048^2 3.9 / 3.5, 4.7 / 3.8    4096^2 12.0 / 10.25, 12.1 / 10.9    6000x4000 16.1 / 18.0
        //   128x2 ETC1s  2048^2 3.8 / 3.6, 5.4 / 4.3    4096^2 14.6 / 12.7, 14.8 / 14.2
        //   128x4 ETC1s  2048^2 5.2 / 4.15, 6.9 / 4.9   4096^2 16.5 / 13.8, 16.6 / 15.5
        // but not on images far larger than the GPU holds at once, where BC1 loses and, next to an ETC1s pipeline launch,
        // the two calls do (8192^2, both codecs in turn: 89-90.6 us, both on the pipeline 87); nor on word-aligned rows
        // (3072^2 128x1 ETC1s 9.5 / 10.4 from HBM); nor, in two blocks a thread of the longer codecs, with CTAs of which
        // fewer fit on an SM than under the cap of the plain kernel, unless it is all one wave (256x2 ETC1s: 2048^2 5.8 / 6.3,
        // 3072^2 9.9 / 9.6; 1024^2 both 4.6 / 3.05).
        const uint32_t blocks = bw * bh;
        const bool word = access == SrcAccess::kWord4, fewer = tile.bpt == 2 && codec != kBC1;
        const uint32_t wave = kSms * 2u * tile.threads * (tile.threads == 128 ? 7u : tile.threads == 256 ? 3u : 1u);
        if (fewer && (word || tile.threads > 128) ? blocks <= wave : !word && blocks <= 1250000u) rows = Rows::kAhead;
    }
    if (codec == kBC1) return launch_access<kBC1>(src, stride, dst, nullptr, bw, bh, tile, access, rows, stream);
    if (codec == kETC1S) return launch_access<kETC1S>(src, stride, dst, nullptr, bw, bh, tile, access, rows, stream);
    return launch_access<kBoth>(src, stride, dst, dst2, bw, bh, tile, access, rows, stream);
}

}  // namespace goofy_gpu
