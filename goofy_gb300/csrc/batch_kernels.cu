// batch_kernels.cu -- many images of uneven sizes (textures, mip levels) in
// one persistent launch.
//
// The reference encodes one image per call (goofy::compressDXT1/ETC1,
// GoofyTC/goofy_tc.h:1497-1557); here a batch of images is flattened into
// work units of `unit_blocks` consecutive 4x4 blocks of one image (the last
// unit of an image may be short).  A resident grid of warps pulls units from
// a device work counter (one atomicAdd per unit, by lane 0), finds the unit's
// image by binary search over the per-image first-unit table, and encodes the
// unit's blocks with the same per-block codec as the image kernel.  Codec and
// load mode are uniform per unit, so warps never diverge on them.  There is no
// waiting: a warp that draws a unit number past the end exits.
//
// Up to about two thousand images, the descriptors are the kernel's parameter
// instead (encode_batch_params): no upload and no counter to zero ahead of
// the kernel, units sized to the work.  A call (us), uploaded / as parameter
// (both before the prefetches below) / now: 24 tiles of 128x128 12.3 / 3.1 / 3.1
// (from Python: the host's time), a 2048^2 mip chain 12 / 4 / 4, the first 20 textures of the mixed batch 19.2 / 9.2
// / 7.0, 100 53.2 / 40.3 / 37.4 (floor 35.5 at 4.5 B/px of measured HBM), 380 (993
// images) 148 / 137 / 128 (134), 600 (two launches) 201 / 195 / 182.  Each further
// launch drains the GPU once, about 4 us: with 1000 textures (three launches,
// 2642 images) 323 against 317-320 uploaded, which takes 304 now (306).
#include <cuda_runtime.h>

#include "batch.h"
#include "block_codec.cuh"
#include "device_io.cuh"
#include "pdl.cuh"

namespace goofy_gpu {

// This lane's blocks of the step at b0: their addresses, and (PREFETCH) L2
// asked for their lines, every eighth lane's block being 128 bytes on.  Blocks
// past the unit's last are the last.
template <int BPT>
__device__ __forceinline__ void step_addresses(const BatchImage& im, uint32_t b0, uint32_t last, uint32_t lane,
                                               bool prefetch, const uint8_t* (&p)[BPT])
{
#pragma unroll
    for (int j = 0; j < BPT; ++j) {
        uint32_t bx;
        const uint32_t by = div_magic(min(b0 + lane + 32u * j, last - 1u), im.bw, im.bw_magic, bx);
        p[j] = im.src + (size_t)by * 4u * im.stride + 16u * (size_t)bx;
        if (prefetch && !(lane & 7u)) {
#pragma unroll
            for (int y = 0; y < 4; ++y) prefetch_l2(p[j] + (size_t)y * im.stride);
        }
    }
}

// Encodes blocks [first, last) of one image, 32 * BPT at a time, `p` being the
// first step's addresses.  While a step waits for its rows and encodes them,
// the next step's are on their way to L2: a warp's own steps are a serial
// chain, and memory latency is most of each.  Whole calls without / with (us):
// 1000 textures 319 / 304, 600 197 / 182, 380 139 / 128, 100 40.3 / 37.4.
// Loading the next step's words into registers instead leaves too few warps
// (1000 textures 344).
//
// MODE: the images' codec where it is one and all rows are 16-byte aligned,
// else kMixed.
template <int BPT, int MODE, typename Lut>
__device__ __forceinline__ void encode_unit(const BatchImage& im, uint32_t first, uint32_t last, uint32_t lane,
                                            const uint8_t* (&p)[BPT], Lut ctrl_lut)
{
    const bool vec16 = MODE != kMixed || im.vec16 != 0;
    for (uint32_t b0 = first; b0 < last; b0 += 32u * BPT) {
        uint32_t w[BPT][16];
        const uint8_t* n[BPT];  // asked for ahead of this step's loads (behind them: 2 us more on 600 textures)
        if (b0 + 32u * BPT < last) step_addresses<BPT>(im, b0 + 32u * BPT, last, lane, true, n);
#pragma unroll
        for (int j = 0; j < BPT; ++j) {  // also past the last block (it is read again): no branch ahead of the loads
            load_block_rows(p[j], im.stride, vec16, w[j]);
            p[j] = n[j];
        }
#pragma unroll
        for (int j = 0; j < BPT; ++j) {
            const uint32_t b = b0 + lane + 32u * j;
            if (b < last) {
                const bool bc1 = MODE == kMixed ? im.codec == kBC1 : MODE == kBC1;
                st_stream8(im.dst + 8u * (size_t)b, bc1 ? encode_bc1(w[j]) : encode_etc1s(w[j], ctrl_lut));
            }
        }
    }
}

template <int BPT>
__global__ void __launch_bounds__(512) encode_batch_kernel(const BatchImage* __restrict__ images, uint32_t n_images,
                                                           const uint32_t* __restrict__ first_unit,
                                                           uint32_t total_units, uint32_t unit_blocks,
                                                           uint32_t* __restrict__ work_counter)
{
    __shared__ uint8_t ctrl_lut[128];
    fill_ctrl_lut(ctrl_lut);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    for (;;) {
        uint32_t u = 0;
        if (lane == 0) u = atomicAdd(work_counter, 1u);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= total_units) return;
        const uint32_t ii = find_image(first_unit, n_images, u);
        const BatchImage im = images[ii];
        const uint32_t first = (u - im.first_unit) * unit_blocks, last = min(first + unit_blocks, im.bw * im.bh);
        const uint8_t* p[BPT];
        step_addresses<BPT>(im, first, last, lane, false, p);
        encode_unit<BPT, kMixed, const uint8_t*>(im, first, last, lane, p, ctrl_lut);
    }
}

template <uint32_t N>
struct ParamTable {
    ParamImage images[N];
};

// The same work with the descriptors as the kernel's parameter and one work
// unit a warp, dealt by the CTA scheduler: nothing is uploaded, no counter is
// zeroed or shared, and the launch overlaps its predecessor's tail.  128
// threads a CTA: a warp's slot is free again only when its CTA is done (380
// textures 137 us, 141 with 256 threads).
//
// A launch whose images share a codec and 16-byte rows (a texture's mip chain,
// most sets of tiles) runs code for just that, in fewer registers: the BC1
// chain of 2048^2 5.3 / 4.6 us, its mips and that together 10.75 / 10.15.
template <int BPT, uint32_t N, int MODE>
__global__ void __launch_bounds__(512) encode_batch_params(const __grid_constant__ ParamTable<N> t, uint32_t n_images,
                                                           uint32_t total_units)
{
    pdl_launch_dependents();
    const uint32_t u = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (u >= total_units) return;
    // largest i with images[i].first_unit <= u (an image without blocks shares its successor's)
    uint32_t lo = 0, hi = n_images;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (t.images[mid].first_unit <= u) lo = mid;
        else hi = mid;
    }
    const ParamImage& p = t.images[lo];
    BatchImage im;
    im.src = p.src;
    im.dst = p.dst;
    im.stride = p.stride;
    im.bw = p.bw();
    im.bh = p.bh();
    im.bw_magic = 0xffffffffu / im.bw;
    im.codec = p.codec();
    im.vec16 = p.vec16();
    const uint32_t unit = (32u * BPT) << p.unit_class(), first = (u - p.first_unit) * unit;
    const uint32_t last = min(first + unit, im.bw * im.bh), lane = threadIdx.x & 31u;
    // the first step's rows, while the previous kernel drains (20 textures 9.2 / 8.3 us); nothing
    // of them enters the SM before the wait
    const uint8_t* rows[BPT];
    step_addresses<BPT>(im, first, last, lane, true, rows);
    pdl_wait();  // no global memory access before the previous kernel in the stream is done
    encode_unit<BPT, MODE>(im, first, last, lane, rows, NoLut{});
}

int batch_resident_ctas(uint32_t threads, uint32_t bpt, uint32_t pipeline)
{
    if (pipeline) return batch_tma_resident_ctas(threads, bpt);
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (bpt == 1) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_batch_kernel<1>, threads, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_batch_kernel<2>, threads, 0);
    return sms * (per_sm > 0 ? per_sm : 1);
}

cudaError_t launch_batch(const BatchImage* images, uint32_t n_images, const uint32_t* first_unit,
                         uint32_t total_units, uint32_t* work_counter, const BatchTile& tile, uint32_t ctas,
                         cudaStream_t stream)
{
    if (total_units == 0) return cudaSuccess;
    if (tile.pipeline) return launch_batch_tma(images, n_images, first_unit, total_units, work_counter, tile, ctas, stream);
    if (tile.bpt == 1)
        encode_batch_kernel<1><<<ctas, tile.threads, 0, stream>>>(images, n_images, first_unit, total_units,
                                                                   tile.unit_blocks, work_counter);
    else
        encode_batch_kernel<2><<<ctas, tile.threads, 0, stream>>>(images, n_images, first_unit, total_units,
                                                                   tile.unit_blocks, work_counter);
    return cudaGetLastError();
}

namespace {

template <int BPT, uint32_t N, int MODE>
cudaError_t launch_params_t(const ParamLaunch& l, uint32_t threads, cudaStream_t stream)
{
    const uint32_t wpc = threads / 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((l.units + wpc - 1) / wpc);
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {l.images, const_cast<uint32_t*>(&l.count),
                    const_cast<uint32_t*>(&l.units)};
    return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(&encode_batch_params<BPT, N, MODE>), args);
}

template <int BPT, int MODE>
cudaError_t launch_params(const ParamLaunch& l, uint32_t threads, cudaStream_t stream)
{
    if (l.count <= 32) return launch_params_t<BPT, 32, MODE>(l, threads, stream);
    if (l.count <= 256) return launch_params_t<BPT, 256, MODE>(l, threads, stream);
    return launch_params_t<BPT, kParamImages, MODE>(l, threads, stream);
}

}  // namespace

cudaError_t launch_batch_params(const ParamLaunch& l, const BatchTile& tile, cudaStream_t stream)
{
    if (l.units == 0) return cudaSuccess;
    if (tile.bpt != 1) return launch_params<2, kMixed>(l, tile.threads, stream);
    if (l.mode == kBC1) return launch_params<1, kBC1>(l, tile.threads, stream);
    if (l.mode == kETC1S) return launch_params<1, kETC1S>(l, tile.threads, stream);
    return launch_params<1, kMixed>(l, tile.threads, stream);
}

}  // namespace goofy_gpu
