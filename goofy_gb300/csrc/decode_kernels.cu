// decode_kernels.cu -- BC1 / ETC1 block decoding and the encode-quality error
// reduction on sm_103a.
//
// The reference checks quality on the CPU: it decodes every block with its
// harness decoders (Src/decoder.cpp: DecompressColour :819-871 for BC1,
// decompressBlockDiffFlipC :388-678 for ETC1) and sums squared channel
// differences in getMsePsnr (Src/main.cpp:403-469).  Here one thread decodes
// one block (BC1: both endpoint orders; ETC1: individual and differential
// modes, both flips; ETC2-only differential overflows are counted as
// unsupported and decoded as black) and either stores the 16 pixels or, in
// the quality kernels, compares the block with its source pixels
// (block_error.cuh), summing squared differences per channel exactly in
// integers (32-bit per thread, then 64-bit through shuffles and shared memory,
// one atomic per CTA and sum).
#include <cuda_runtime.h>

#include <atomic>

#include "batch.h"
#include "block_codec.cuh"
#include "block_decode.cuh"
#include "block_error.cuh"
#include "decode.h"
#include "device_io.cuh"
#include "error_reduce.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace goofy_gpu {

// Threads per CTA of every decoding kernel: the palette column stride, a
// constant so that a pixel's palette address is a shift and an add.
constexpr uint32_t kDecodeThreads = 256;

// CTAs resident at once.  A grid within it asks L2 for its blocks while the
// kernel before it drains (us, inputs of 400 MB in all, BC1: 256^2 1.66 / 1.38,
// 1024^2 2.7 / 2.4, 2048^2 3.75 / 3.55, 3840x2160 6.1 / 6.0); a larger one's later
// CTAs start too late for that and would only wait longer (1384x3800 5.05 / 5.2).
constexpr uint32_t kDecodeWave = kSms * 8;

// N blocks a thread, 32 apart, so each store of a warp writes 512 contiguous
// bytes of a pixel row.
template <int CODEC, int N>
__global__ void __launch_bounds__(kDecodeThreads) decode_image_kernel(const uint8_t* __restrict__ blocks, uint32_t bw,
                                                                      uint32_t bw_magic, uint32_t nblk,
                                                                      uint8_t* __restrict__ rgba, size_t stride,
                                                                      unsigned long long* __restrict__ unsupported)
{
    pdl_launch_dependents();
    __shared__ uint32_t pal[CODEC == kBC1 ? 1 : 8 * kDecodeThreads];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t i0 = (blockIdx.x * (kDecodeThreads / 32u) + (threadIdx.x >> 5)) * (32u * N) + lane;
    uint2 code[N];
    uint32_t bad = 0;
    if (gridDim.x <= kDecodeWave && !(lane & 15u)) {  // (each such lane's block starts a 128-byte line)
#pragma unroll
        for (int j = 0; j < N; ++j) prefetch_l2(blocks + 8u * (size_t)min(i0 + 32u * j, nblk - 1u));
    }
    pdl_wait();
#pragma unroll
    for (int j = 0; j < N; ++j)
        code[j] = i0 + 32u * j < nblk ? load_block8(blocks + 8u * (size_t)(i0 + 32u * j)) : make_uint2(0u, 0u);
#pragma unroll
    for (int j = 0; j < N; ++j) {
        const uint32_t i = i0 + 32u * j;
        if (i < nblk) {
            uint32_t bx, px[16];
            const uint32_t by = div_magic(i, bw, bw_magic, bx);
            if (!decode_block<CODEC>(code[j], pal + threadIdx.x, kDecodeThreads, px)) ++bad;
            uint8_t* row = rgba + (size_t)by * 4u * stride + 16u * (size_t)bx;
#pragma unroll
            for (int y = 0; y < 4; ++y)
                *reinterpret_cast<uint4*>(row + (size_t)y * stride) = make_uint4(px[4 * y], px[4 * y + 1], px[4 * y + 2],
                                                                                 px[4 * y + 3]);
        }
    }
    if constexpr (CODEC != kBC1) {
        bad = __reduce_add_sync(0xffffffffu, bad);
        if (bad && lane == 0) atomicAdd(unsupported, (unsigned long long)bad);
    }
}

// All but large images, which take error_image_tma (encode_tma.cu).  Resident
// grid: each thread walks blocks with a grid stride, then the CTA reduces and
// adds its six totals.  Register caps for 4 (BC1) / 3 (ETC1) CTAs per SM, no
// spills (ETC1 with 4: 3.9 -> 4.4 us at 1024^2).  While the previous kernel in
// the stream drains, the first blocks' rows are asked of L2 (a hint: the loads
// after the wait read what that kernel wrote): BC1 / ETC1s back to back over
// 400 MB, without / with (us): 1024^2 4.4 / 4.0 and 3.9 / 3.4, 2048^2 6.75 / 5.75
// and 6.3 / 5.2.
template <int CODEC>
__global__ void __launch_bounds__(kDecodeThreads, CODEC == kBC1 ? 4 : 3)
    block_error_kernel(const uint8_t* __restrict__ blocks, uint32_t bw, uint32_t nblk, const uint8_t* __restrict__ src,
                       size_t stride, bool vec16, unsigned long long* __restrict__ sums, ErrorResult result)
{
    pdl_launch_dependents();
    const uint32_t bw_magic = 0xffffffffu / bw;
    ErrorSums e{};  // at most kErrorSumBlocks blocks a thread (launch_block_error)
    uint32_t bad = 0;
    const uint32_t step = gridDim.x * kDecodeThreads;
    uint32_t i = blockIdx.x * kDecodeThreads + threadIdx.x;
    uint32_t bx0;
    const uint32_t by0 = div_magic(min(i, nblk - 1u), bw, bw_magic, bx0);
    const uint8_t* p0 = src + (size_t)by0 * 4u * stride + 16u * (size_t)bx0;
    if (!(threadIdx.x & 7u)) {  // eight blocks' rows are 128 bytes, sixteen codes
#pragma unroll
        for (int y = 0; y < 4; ++y) prefetch_l2(p0 + (size_t)y * stride);
        if (!(threadIdx.x & 15u)) prefetch_l2(blocks + 8u * (size_t)min(i, nblk - 1u));
    }
    pdl_wait();
    // software pipeline: the next block's source rows and code are loaded
    // before this block is compared
    uint32_t w[16];
    uint2 blk = make_uint2(0, 0);
    if (i < nblk) {
        load_block_rows(p0, stride, vec16, w);
        blk = load_block8(blocks + 8u * (size_t)i);
    }
    for (; i < nblk; i += step) {
        uint32_t cur[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) cur[k] = w[k];
        const uint2 cur_blk = blk;
        if (i + step < nblk) {
            uint32_t bx;
            const uint32_t by = div_magic(i + step, bw, bw_magic, bx);
            load_block_rows(src + (size_t)by * 4u * stride + 16u * (size_t)bx, stride, vec16, w);
            blk = load_block8(blocks + 8u * (size_t)(i + step));
        }
        if (!add_block_errors<CODEC>(cur, cur_blk, e)) ++bad;
    }
    reduce_errors<kDecodeThreads>(e, bad, false, sums, result);
}

// The error sums of every image of a batch (the request server's quality
// measurement): the batch's work units, pulled from a counter as in the
// encoder's batch kernel, decode the image's blocks (`dst`) and compare them
// with its source; a warp sums its unit and adds six totals to the image's
// sums[6 * image + c].
__global__ void __launch_bounds__(kDecodeThreads) quality_batch_kernel(const BatchImage* __restrict__ images, uint32_t n_images,
                                                            const uint32_t* __restrict__ first_unit,
                                                            uint32_t total_units, uint32_t unit_blocks,
                                                            uint32_t* __restrict__ work_counter,
                                                            unsigned long long* __restrict__ sums)
{
    const uint32_t lane = threadIdx.x & 31u;
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(work_counter, 1u);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= total_units) return;
        const uint32_t ii = find_image(first_unit, n_images, u);
        const BatchImage im = images[ii];
        const uint32_t first = (u - im.first_unit) * unit_blocks, last = min(first + unit_blocks, im.bw * im.bh);
        ErrorSums e{};  // a lane has at most kErrorSumBlocks blocks of a unit (launch_quality_batch)
        uint32_t bad = 0;
        for (uint32_t b = first + lane; b < last; b += 32u) {
            uint32_t bx;
            const uint32_t by = div_magic(b, im.bw, im.bw_magic, bx);
            uint32_t w[16];
            const uint2 blk = load_block8(im.dst + 8u * (size_t)b);
            load_block_rows(im.src + (size_t)by * 4u * im.stride + 16u * (size_t)bx, im.stride, im.vec16 != 0, w);
            const bool ok = im.codec == kBC1 ? add_block_errors<kBC1>(w, blk, e) : add_block_errors<kETC1S>(w, blk, e);
            bad += ok ? 0u : 1u;
        }
        unsigned long long t[6] = {e.sq[0], e.sq[1], e.sq[2], e.sq[3], bad, luma_sum_of(e)};
#pragma unroll
        for (int c = 0; c < 6; ++c) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
        }
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < 6; ++c)
                if (t[c]) atomicAdd(&sums[6u * ii + c], t[c]);
    }
}

cudaError_t launch_quality_batch(const BatchImage* images, uint32_t n_images, const uint32_t* first_unit,
                                 uint32_t total_units, uint32_t unit_blocks, uint32_t* work_counter,
                                 unsigned long long* sums, cudaStream_t stream)
{
    if (total_units == 0) return cudaSuccess;
    if (unit_blocks > 32u * kErrorSumBlocks) return cudaErrorInvalidValue;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t warps = total_units, ctas = (warps + 7) / 8;
    const uint32_t grid = (uint32_t)(ctas < (uint64_t)sms * 8u ? ctas : (uint64_t)sms * 8u);
    quality_batch_kernel<<<grid, kDecodeThreads, 0, stream>>>(images, n_images, first_unit, total_units, unit_blocks,
                                                   work_counter, sums);
    return cudaGetLastError();
}

namespace {

template <int CODEC, int N>
cudaError_t launch_decode_t(const uint8_t* blocks, uint32_t bw, uint32_t nblk, uint8_t* rgba, size_t stride,
                            unsigned long long* unsupported, cudaStream_t stream)
{
    const uint32_t grid = (nblk + N * kDecodeThreads - 1) / (N * kDecodeThreads);
    return launch_pdl(decode_image_kernel<CODEC, N>, dim3(grid), dim3(kDecodeThreads), 0, stream, blocks, bw,
                      0xffffffffu / bw, nblk, rgba, stride, unsupported);
}

}  // namespace

cudaError_t launch_decode(int codec, const uint8_t* blocks, uint32_t width, uint32_t height, uint8_t* rgba,
                          size_t stride, unsigned long long* unsupported, cudaStream_t stream)
{
    const uint32_t bw = width / 4, nblk = bw * (height / 4);
    if (nblk == 0) return cudaSuccess;
    // A wave is 152 SMs x 2048 threads = 311296 blocks.  Two blocks a thread where one would leave a second wave
    // mostly empty, up to two full waves of two (us, one / two, BC1 and ETC1s): 3840x2160 (518400 blocks) 6.3 / 6.1
    // and 6.5 / 6.2, 4096^2 (1048576) 12.0 / 11.6 and 12.2 / 11.7.  Below and above one is as fast or faster: 3000x2048
    // (384000) 4.8 / 5.4 and 5.0 / 5.6, 5000x4096 (1280000) 14.7 / 14.6 and 14.8 / 14.7, 8192^2 44.2 / 44.7 and 44.8 / 44.9.
    const bool two = nblk >= 430000 && nblk <= 1250000;
    if (codec == kBC1)
        return two ? launch_decode_t<kBC1, 2>(blocks, bw, nblk, rgba, stride, unsupported, stream)
                   : launch_decode_t<kBC1, 1>(blocks, bw, nblk, rgba, stride, unsupported, stream);
    return two ? launch_decode_t<kETC1S, 2>(blocks, bw, nblk, rgba, stride, unsupported, stream)
               : launch_decode_t<kETC1S, 1>(blocks, bw, nblk, rgba, stride, unsupported, stream);
}

namespace {

// Resident CTAs of `kernel` per SM on device `dev` (cached per device and
// slot), at least 1.
template <typename K>
uint32_t resident_per_sm(K kernel, int dev, int slot)
{
    static std::atomic<uint32_t> cache[64][2];
    if (dev < 0 || dev >= 64) dev = 0;
    uint32_t n = cache[dev][slot].load(std::memory_order_relaxed);
    if (n == 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kDecodeThreads, 0) != cudaSuccess) {
            cudaGetLastError();
            per_sm = 0;
        }
        n = per_sm > 0 ? (uint32_t)per_sm : 1u;
        cache[dev][slot].store(n, std::memory_order_relaxed);
    }
    return n;
}

}  // namespace

cudaError_t launch_block_error(int codec, const uint8_t* blocks, const uint8_t* src, uint32_t width, uint32_t height,
                               size_t stride, bool vec16, unsigned long long* sums, cudaStream_t stream,
                               ErrorResult result)
{
    const uint32_t bw = width / 4, nblk = bw * (height / 4);
    if (nblk == 0) return cudaSuccess;
    // The ring keeps more bytes in flight but has to fill first and ends in an uneven round: it is for large images,
    // and larger ones where nothing runs before or behind the launch to hide that (a synchronous call) or where it
    // copies word-aligned rows in granules.  This kernel / the ring, BC1, us, image in L2 and from HBM:
    //                    launches back to back              synchronous calls from Python
    //   1024^2          3.1 / 3.2      4.0 / 3.75         13.4 / 13.7    14.0 / 14.3
    //   2048^2          5.15 / 5.1     5.75 / 5.75        15.5 / 16.5    16.4 / 17.75
    //   2816^2          7.7 / 7.55     8.0 / 8.8
    //   3072^2          8.8 / 7.9      9.05 / 8.7         19.4 / 19.5    19.9 / 20.5
    //   3300^2          9.7 / 9.2      9.75 / 10.0        20.2 / 20.9    20.4 / 22.2
    //   3800^2         12.1 / 11.0    12.1 / 11.5
    //   4096^2         13.1 / 12.0    13.2 / 12.9         23.8 / 24.3    24.0 / 25.15
    //   6000x4000      17.75 / 16.4   17.8 / 16.9         28.1 / 29.05   28.5 / 29.7
    //   8192^2         43.2 / 40.0    44.2 / 42.6         54.0 / 52.6    55.0 / 55.5
    //   128x65536       7.6 / 8.9      8.1 / 9.6          18.2 / 20.2    18.9 / 20.3
    //   512x32768      13.1 / 12.6    13.2 / 13.8         23.8 / 24.8    23.85 / 25.3
    // word-aligned 4096^2 13.2 / 14.8, 15.0 / 15.0; 6000x4000 18.3 / 19.8, 19.7 / 20.0; 8192^2 49.0 / 46.8.  ETC1s alike.
    const bool late = result.host || !vec16;
    if (nblk >= (late ? 2500000u : 580000u) && bw >= 256)
        return launch_error_tma(codec, blocks, src, width, height, stride, vec16, sums, result, stream);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // One wave: as many CTAs as fit on the GPU at once, each thread striding
    // over its share of the blocks (more for an image so long and narrow that
    // a thread's 32-bit sums would run over).
    const uint32_t per_sm = codec == kBC1 ? resident_per_sm(block_error_kernel<kBC1>, dev, 0)
                                          : resident_per_sm(block_error_kernel<kETC1S>, dev, 1);
    const uint32_t most = (nblk + kDecodeThreads - 1) / kDecodeThreads, least = (most + kErrorSumBlocks - 1) / kErrorSumBlocks;
    const uint32_t grid = max(least, min(most, (uint32_t)(sms > 0 ? sms : 1) * per_sm));
    if (codec == kBC1)
        return launch_pdl(block_error_kernel<kBC1>, dim3(grid), dim3(kDecodeThreads), 0, stream, blocks, bw, nblk, src, stride,
                          vec16, sums, result);
    return launch_pdl(block_error_kernel<kETC1S>, dim3(grid), dim3(kDecodeThreads), 0, stream, blocks, bw, nblk, src, stride,
                      vec16, sums, result);
}

}  // namespace goofy_gpu
