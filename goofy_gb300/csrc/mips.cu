// mips.cu -- mip-chain generation on the device, feeding the batch encoder.
//
// The reference has no mip generator (its harness only builds an RGB565 x2
// downsample as a quality baseline, Src/main.cpp:501-557); textures with mip
// chains are encoded level by level from levels the caller made.  Here each
// level is produced from the one above by a 2x2 box filter with rounding,
// (a + b + c + d + 2) >> 2 per channel, an axis that is already 4 pixels
// being copied instead of halved -- the rule of the workload generator's
// goofy_synth_downsample, so device and host chains are bit-identical.  While
// both axes halve, one launch makes up to 6 levels from shared-memory tiles
// (mip_fused_kernel), or the whole chain of 512^2 and 1024^2
// (mip_chain_kernel); small levels behind them take one launch in all
// (mip_tail_kernel), larger ones a launch each, a thread per output pixel.
// Channel pairs are summed in 16-bit lanes.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/goofy_gpu.h"
#include "device_io.cuh"
#include "host_util.h"
#include "pdl.cuh"

namespace {

__device__ __forceinline__ uint32_t box4(uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    const uint32_t m = 0x00ff00ffu;
    const uint32_t rb = (a & m) + (b & m) + (c & m) + (d & m) + 0x00020002u;
    const uint32_t ga = ((a >> 8) & m) + ((b >> 8) & m) + ((c >> 8) & m) + ((d >> 8) & m) + 0x00020002u;
    return ((rb >> 2) & m) | (((ga >> 2) & m) << 8);
}

// One output pixel per thread.  FX = 2 (the level halves horizontally) with
// 8-byte aligned rows reads the two source pixels of each row with one 8-byte
// load; otherwise four 4-byte loads.
template <bool PAIR>
__global__ void __launch_bounds__(256) mip_level_kernel(const uint8_t* __restrict__ src, size_t src_stride,
                                                        uint8_t* __restrict__ dst, size_t dst_stride, uint32_t dw,
                                                        uint32_t dh, uint32_t fx, uint32_t fy)
{
    goofy_gpu::pdl_launch_dependents();
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (x >= dw || y >= dh) return;
    goofy_gpu::pdl_wait();
    const uint8_t* r0 = src + (size_t)(y * fy) * src_stride + 4u * (size_t)(x * fx);
    const uint8_t* r1 = r0 + src_stride * (fy - 1);
    uint32_t a, b, c, d;
    if constexpr (PAIR) {
        const uint2 p = goofy_gpu::ld_keep8(r0), q = goofy_gpu::ld_keep8(r1);
        a = p.x;
        b = p.y;
        c = q.x;
        d = q.y;
    } else {
        a = goofy_gpu::ld_keep4(r0);
        b = goofy_gpu::ld_keep4(r0 + 4 * (fx - 1));
        c = goofy_gpu::ld_keep4(r1);
        d = goofy_gpu::ld_keep4(r1 + 4 * (fx - 1));
    }
    *reinterpret_cast<uint32_t*>(dst + (size_t)y * dst_stride + 4u * (size_t)x) = box4(a, b, c, d);
}

// Up to 6 levels per launch: a CTA takes a tile of up to 64x64 pixels of the
// level above.  Each thread reads a 4x4 patch (four 16-byte row loads), makes
// the 2x2 quad of the first new level and the one pixel of the second from it
// in registers, the third level comes from the 2x2 neighbourhood of second-
// level pixels held by lanes t^1, t^w, t^w^1 of the same warp (shuffles), and
// the remaining levels (at most 8x8 pixels per tile) go through shared
// memory.  Used while both axes halve; every level is the same box4 of the
// level above as in the one-level kernel, so the results are identical.
template <int LEVELS>
struct MipLevels {
    uint8_t* data[LEVELS];
    uint32_t pitch[LEVELS];
};
using MipOut = MipLevels<6>;

template <typename Out>
__device__ __forceinline__ void store_px(const Out& o, int l, uint32_t row, uint32_t col, uint32_t v)
{
    *reinterpret_cast<uint32_t*>(o.data[l] + (size_t)row * o.pitch[l] + 4u * col) = v;
}

// One tile's levels from the 4x4 patches `r` (already loaded) of its 256
// threads, of which this is number t.  Returns thread 0's pixel of the sixth
// level, if there is one.  A CTA calls it for all its tiles at once.
template <typename Out>
__device__ __forceinline__ uint32_t mip_tile(const uint4 (&r)[4], uint32_t t, bool act, uint32_t tx, uint32_t ty,
                                             uint32_t tw_log2, uint32_t th_log2, uint32_t nlev, const Out& out,
                                             uint32_t (*buf)[64])
{
    const uint32_t w2_log2 = tw_log2 - 2, h2_log2 = th_log2 - 2, w2 = 1u << w2_log2;
    const uint32_t x2 = t & (w2 - 1u), y2 = t >> w2_log2;
    uint32_t v2 = 0;
    if (act) {
        const uint32_t q00 = box4(r[0].x, r[0].y, r[1].x, r[1].y), q01 = box4(r[0].z, r[0].w, r[1].z, r[1].w);
        const uint32_t q10 = box4(r[2].x, r[2].y, r[3].x, r[3].y), q11 = box4(r[2].z, r[2].w, r[3].z, r[3].w);
        const uint32_t row1 = (ty << (th_log2 - 1)) + 2u * y2, col1 = (tx << (tw_log2 - 1)) + 2u * x2;
        *reinterpret_cast<uint2*>(out.data[0] + (size_t)row1 * out.pitch[0] + 4u * col1) = make_uint2(q00, q01);
        *reinterpret_cast<uint2*>(out.data[0] + (size_t)(row1 + 1) * out.pitch[0] + 4u * col1) = make_uint2(q10, q11);
        v2 = box4(q00, q01, q10, q11);
        if (nlev > 1) store_px(out, 1, (ty << h2_log2) + y2, (tx << w2_log2) + x2, v2);
    }
    if (nlev <= 2) return 0;
    // third level: lanes with even x2 and y2 combine their 2x2 neighbourhood
    const uint32_t b = __shfl_xor_sync(0xffffffffu, v2, 1), c = __shfl_xor_sync(0xffffffffu, v2, w2),
                   d = __shfl_xor_sync(0xffffffffu, v2, w2 ^ 1u);
    const uint32_t w3_log2 = w2_log2 - 1, h3_log2 = h2_log2 - 1;
    if (act && !(x2 & 1u) && !(y2 & 1u)) {
        const uint32_t v3 = box4(v2, b, c, d), x3 = x2 >> 1, y3 = y2 >> 1;
        store_px(out, 2, (ty << h3_log2) + y3, (tx << w3_log2) + x3, v3);
        buf[0][(y3 << w3_log2) + x3] = v3;
    }
    uint32_t cw_log2 = w3_log2, ch_log2 = h3_log2, v = 0;
#pragma unroll
    for (uint32_t l = 3; l < 6; ++l) {  // unrolled: the level indexes `out` as a constant (no stack copy)
        if (l >= nlev) break;
        __syncthreads();
        const uint32_t* in = buf[(l - 3) & 1];
        uint32_t* next = buf[(l - 2) & 1];
        const uint32_t nw_log2 = cw_log2 - 1, nh_log2 = ch_log2 - 1, cw = 1u << cw_log2;
        if (t < (1u << (nw_log2 + nh_log2))) {
            const uint32_t ox = t & ((1u << nw_log2) - 1u), oy = t >> nw_log2;
            const uint32_t* r0 = in + (2u * oy) * cw + 2u * ox;
            v = box4(r0[0], r0[1], r0[cw], r0[cw + 1]);
            next[t] = v;
            store_px(out, (int)l, (ty << nh_log2) + oy, (tx << nw_log2) + ox, v);
        }
        cw_log2 = nw_log2;
        ch_log2 = nh_log2;
    }
    __syncthreads();  // the next tile of this CTA reuses buf
    return v;
}

// Before the dependency wait, while the previous kernel in the stream drains:
// asks L2 for the 128-byte lines at a patch's rows (every eighth lane's cover
// the eight patches beside it).  A hint: the loads after the wait read what
// that kernel wrote.  Whole chains without / with (us): 1024^2 3.8 / 3.4 with
// inputs of 400 MB in all, 2048^2 7.25 / 6.0, 4096^2 17.7 / 16.4.
__device__ __forceinline__ void prefetch_patch_rows(const uint8_t* patch, size_t src_stride)
{
#pragma unroll
    for (int j = 0; j < 4; ++j) goofy_gpu::prefetch_l2(patch + j * src_stride);
}

// TILES horizontally adjacent tiles per CTA: every patch load of all of them
// is issued before the first tile is reduced, so more bytes are in flight.
template <int TILES>
__global__ void __launch_bounds__(256) mip_fused_kernel(const uint8_t* __restrict__ src, size_t src_stride,
                                                        uint32_t tw_log2, uint32_t th_log2, uint32_t nlev, MipOut out)
{
    goofy_gpu::pdl_launch_dependents();
    __shared__ uint32_t buf[2][64];
    const uint32_t t = threadIdx.x, ty = blockIdx.y;
    const uint32_t w2_log2 = tw_log2 - 2, h2_log2 = th_log2 - 2, w2 = 1u << w2_log2;
    const bool act = t < (1u << (w2_log2 + h2_log2));
    const uint32_t x2 = t & (w2 - 1u), y2 = t >> w2_log2;
    uint4 r[TILES][4];
    if (act && !(t & 7u)) {
#pragma unroll
        for (int k = 0; k < TILES; ++k)
            prefetch_patch_rows(src + (((size_t)ty << th_log2) + 4u * y2) * src_stride +
                                    (((size_t)(blockIdx.x * TILES + k) << tw_log2) + 4u * x2) * 4u,
                                src_stride);
    }
    goofy_gpu::pdl_wait();  // the level above may come from the previous launch
#pragma unroll
    for (int k = 0; k < TILES; ++k) {
        if (act) {
            const uint32_t tx = blockIdx.x * TILES + k;
            const uint8_t* patch = src + (((size_t)ty << th_log2) + 4u * y2) * src_stride +
                                   (((size_t)tx << tw_log2) + 4u * x2) * 4u;
#pragma unroll
            for (int j = 0; j < 4; ++j) r[k][j] = goofy_gpu::ld_keep16(patch + (size_t)j * src_stride);
        }
    }
#pragma unroll
    for (int k = 0; k < TILES; ++k) mip_tile(r[k], t, act, blockIdx.x * TILES + k, ty, tw_log2, th_log2, nlev, out, buf);
}

// Whole square chains of 7 and 8 levels (512^2, 1024^2) in one launch: a
// cluster of CTAs takes a square of K x K tiles of 64x64 pixels, 256 threads a
// tile; each tile's last pixel goes to the first CTA's shared memory, and that
// CTA makes the levels above.  Against two launches, mips / mips and the
// encode behind them (us): 512^2 2.55 / 4.36 -> 2.12 / 3.71, 1024^2 3.52 / 6.88 ->
// 3.14 / 5.16, and 1.5 us of host time.  2048^2 stays at two launches (5.7 us
// for the mips): as 16 clusters of 64 tiles it took 6.5 (16 CTAs of 512
// threads) to 10 us, clusters that large leaving SMs without one.
__host__ __device__ constexpr int chain_cluster(int k) { return k == 2 ? 4 : 8; }
__host__ __device__ constexpr int chain_tiles(int k) { return k * k / chain_cluster(k); }  // a CTA's
__host__ __device__ constexpr int chain_levels(int k) { return k == 2 ? 7 : 8; }

template <int K>
__global__ void __cluster_dims__(chain_cluster(K), 1, 1) __launch_bounds__(256 * chain_tiles(K), 1)
    mip_chain_kernel(const uint8_t* __restrict__ src, size_t src_stride, uint32_t squares_x,
                     const __grid_constant__ MipLevels<chain_levels(K)> out)
{
    goofy_gpu::pdl_launch_dependents();
    constexpr uint32_t kCtas = chain_cluster(K);
    __shared__ uint32_t buf[chain_tiles(K)][2][64];
    __shared__ uint32_t top[K * K];  // the first CTA's: the tiles' last pixels
    const uint32_t group = threadIdx.x >> 8, t = threadIdx.x & 255u, rank = blockIdx.x % kCtas;
    const uint32_t square = blockIdx.x / kCtas, sx = square % squares_x, sy = square / squares_x;
    const uint32_t tile = rank * chain_tiles(K) + group, tx = sx * K + tile % K, ty = sy * K + tile / K;
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    const uint8_t* patch = src + (size_t)(64u * ty + 4u * (t >> 4)) * src_stride + 4u * (64u * tx + 4u * (t & 15u));
    if (!(t & 7u)) prefetch_patch_rows(patch, src_stride);
    goofy_gpu::pdl_wait();
    uint4 r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) r[j] = goofy_gpu::ld_keep16(patch + (size_t)j * src_stride);
    const uint32_t last = mip_tile(r, t, true, tx, ty, 6u, 6u, 6u, out, buf[group]);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // the first CTA has started
    if (t == 0) {
        uint32_t at = (uint32_t)__cvta_generic_to_shared(&top[tile]), remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(at));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(last) : "memory");
    }
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (rank != 0) return;
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (threadIdx.x >= 32) return;
    constexpr uint32_t n = K / 2;
    const uint32_t lane = threadIdx.x, x = lane % n, y = lane / n;
    uint32_t v = 0;
    if (lane < n * n) {
        const uint32_t* p = top + 2u * y * K + 2u * x;
        v = box4(p[0], p[1], p[K], p[K + 1]);
        store_px(out, 6, sy * n + y, sx * n + x, v);
    }
#pragma unroll
    for (uint32_t d = 1, l = 7; 2 * d <= n; d *= 2, ++l) {  // neighbours are d pixels apart
        const uint32_t b = __shfl_xor_sync(0xffffffffu, v, d), c = __shfl_xor_sync(0xffffffffu, v, d * n),
                       e = __shfl_xor_sync(0xffffffffu, v, d * n ^ d);
        v = box4(v, b, c, e);
        if (lane < n * n && !(x & (2 * d - 1)) && !(y & (2 * d - 1)))
            store_px(out, (int)l, sy * (n / (2 * d)) + y / (2 * d), sx * (n / (2 * d)) + x / (2 * d), v);
    }
}

// The end of a chain in one CTA: levels of at most kTailPixels pixels, each
// made from the one above, which is kept in shared memory.  Used where the
// fused kernel would not reach the chain's last level, because one axis is at
// 4 first and the rest would take a launch a level.  Whole chains (us), a
// launch a level / one: 4096x256 5.7 / 4.3, 1024x256 3.4 / 3.0, 4096x1024 7.1 /
// 6.2, 64x16 2.7 / 1.7, 8192x64 9.9 / 6.9, and 1.5 us of host time a launch.
constexpr uint32_t kTailPixels = 4096, kTailLevels = 16, kTailThreads = 512;
struct TailOut {
    uint8_t* data[kTailLevels];
    uint32_t pitch[kTailLevels];
};

__global__ void __launch_bounds__(kTailThreads) mip_tail_kernel(const uint8_t* __restrict__ src, size_t src_stride,
                                                                uint32_t w, uint32_t h, uint32_t nlev,
                                                                const __grid_constant__ TailOut out)
{
    goofy_gpu::pdl_launch_dependents();
    __shared__ uint32_t buf[2][kTailPixels];
    goofy_gpu::pdl_wait();
    for (uint32_t l = 0; l < nlev; ++l) {
        const uint32_t fx = w > 4 ? 2 : 1, fy = h > 4 ? 2 : 1, dw = w / fx, dh = h / fy;
        const uint32_t* in = buf[(l + 1) & 1];
        uint32_t* next = buf[l & 1];
        for (uint32_t t = threadIdx.x; t < dw * dh; t += kTailThreads) {
            const uint32_t x = t & (dw - 1u), y = t / dw;
            uint32_t a, b, c, d;
            if (l == 0) {
                const uint8_t* r0 = src + (size_t)(y * fy) * src_stride + 4u * (size_t)(x * fx);
                const uint8_t* r1 = r0 + src_stride * (fy - 1);
                a = goofy_gpu::ld_keep4(r0);
                b = goofy_gpu::ld_keep4(r0 + 4 * (fx - 1));
                c = goofy_gpu::ld_keep4(r1);
                d = goofy_gpu::ld_keep4(r1 + 4 * (fx - 1));
            } else {
                const uint32_t* r0 = in + (y * fy) * w + x * fx;
                const uint32_t* r1 = r0 + w * (fy - 1);
                a = r0[0];
                b = r0[fx - 1];
                c = r1[0];
                d = r1[fx - 1];
            }
            const uint32_t v = box4(a, b, c, d);
            next[t] = v;
            *reinterpret_cast<uint32_t*>(out.data[l] + (size_t)y * out.pitch[l] + 4u * x) = v;
        }
        w = dw;
        h = dh;
        __syncthreads();
    }
}

template <int K>
cudaError_t launch_chain(const goofy_gpu_level* levels, uint32_t i, cudaStream_t stream)
{
    MipLevels<chain_levels(K)> out{};
    for (int l = 0; l < chain_levels(K); ++l) {
        out.data[l] = static_cast<uint8_t*>(levels[i + l].data);
        out.pitch[l] = levels[i + l].stride;
    }
    const goofy_gpu_level& up = levels[i - 1];
    const uint32_t sx = up.width / (64u * K), sy = up.height / (64u * K);
    return goofy_gpu::launch_pdl(mip_chain_kernel<K>, dim3(sx * sy * chain_cluster(K)), dim3(256 * chain_tiles(K)), 0,
                                 stream, static_cast<const uint8_t*>(up.data), (size_t)up.stride, sx, out);
}

bool pow2(uint32_t v) { return v && !(v & (v - 1)); }

uint32_t log2u(uint32_t v)
{
    uint32_t l = 0;
    while (v > 1) {
        v >>= 1;
        ++l;
    }
    return l;
}

size_t pitch_of(uint32_t w) { return ((size_t)4 * w + 255) & ~(size_t)255; }

}  // namespace

extern "C" {

GOOFY_EXPORT uint32_t goofy_gpu_mip_count(uint32_t width, uint32_t height)
{
    if (!pow2(width) || !pow2(height) || width < 4 || height < 4) return 0;
    uint32_t n = 1;
    while (width > 4 || height > 4) {
        width = width / 2 >= 4 ? width / 2 : 4;
        height = height / 2 >= 4 ? height / 2 : 4;
        ++n;
    }
    return n;
}

GOOFY_EXPORT size_t goofy_gpu_mip_arena_bytes(uint32_t width, uint32_t height)
{
    const uint32_t n = goofy_gpu_mip_count(width, height);
    size_t bytes = 0;
    for (uint32_t i = 1; i < n; ++i) {
        width = width / 2 >= 4 ? width / 2 : 4;
        height = height / 2 >= 4 ? height / 2 : 4;
        bytes += pitch_of(width) * height;
    }
    return bytes;
}

GOOFY_EXPORT int goofy_gpu_generate_mips(const void* src, uint32_t width, uint32_t height, uint32_t stride,
                                         void* arena, size_t arena_bytes, goofy_gpu_level* levels,
                                         uint32_t max_levels, uint32_t* nlevels, void* stream)
{
    const uint32_t n = goofy_gpu_mip_count(width, height);
    if (n == 0) return goofy_gpu::fail(GOOFY_ERR_WIDTH, "mips: sizes must be powers of two >= 4");
    if (!src || !levels || !nlevels || (n > 1 && !arena)) return GOOFY_ERR_INVALID;
    if ((uint64_t)stride < 4ull * width || stride % 4 || reinterpret_cast<uintptr_t>(src) % 4)
        return GOOFY_ERR_ALIGNMENT;
    if (max_levels < n) return goofy_gpu::fail(GOOFY_ERR_TOO_LARGE, "mips: level array too small");
    if (arena_bytes < goofy_gpu_mip_arena_bytes(width, height) || reinterpret_cast<uintptr_t>(arena) % 256)
        return goofy_gpu::fail(GOOFY_ERR_TOO_LARGE, "mips: arena too small or not 256-byte aligned");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    levels[0] = goofy_gpu_level{const_cast<void*>(src), width, height, stride};
    uint8_t* out = static_cast<uint8_t*>(arena);
    for (uint32_t i = 1; i < n; ++i) {  // the arena layout: levels 1.. back to back, 256-byte rows
        const goofy_gpu_level& up = levels[i - 1];
        const uint32_t dw = up.width / 2 >= 4 ? up.width / 2 : 4, dh = up.height / 2 >= 4 ? up.height / 2 : 4;
        const size_t pitch = pitch_of(dw);
        levels[i] = goofy_gpu_level{out, dw, dh, (uint32_t)pitch};
        out += pitch * dh;
    }
    for (uint32_t i = 1; i < n;) {
        const goofy_gpu_level& up = levels[i - 1];
        // levels from here on that halve both axes (an axis at 4 stays 4)
        uint32_t both = 0;
        for (uint32_t w = up.width, h = up.height; i + both < n && w > 4 && h > 4; w /= 2, h /= 2) ++both;
        const bool vec16 = reinterpret_cast<uintptr_t>(up.data) % 16 == 0 && up.stride % 16 == 0;
        if (vec16 && both == n - i && (both == 7 || both == 8)) {
            GOOFY_CUDA_TRY(both == 7 ? launch_chain<2>(levels, i, st) : launch_chain<4>(levels, i, st));
            break;
        }
        uint32_t f = log2u(up.width < up.height ? up.width : up.height);
        f = f < both ? f : both;
        f = f < 6 ? f : 6;
        // square tiles of 2^f pixels make exactly f levels (one pixel of the last);
        // the tail of a chain thus gets many small tiles instead of a few large ones
        const uint32_t tw = 1u << f, th = 1u << f;
        const goofy_gpu_level& lv = levels[i];
        if (n - i > 1 && f < n - i && n - i <= kTailLevels && (uint64_t)lv.width * lv.height <= kTailPixels) {
            TailOut to{};
            for (uint32_t l = 0; i + l < n; ++l) {
                to.data[l] = static_cast<uint8_t*>(levels[i + l].data);
                to.pitch[l] = levels[i + l].stride;
            }
            GOOFY_CUDA_TRY(goofy_gpu::launch_pdl(mip_tail_kernel, dim3(1), dim3(kTailThreads), 0, st,
                                                 static_cast<const uint8_t*>(up.data), (size_t)up.stride, up.width,
                                                 up.height, n - i, to));
            break;
        }
        if (f >= 2 && vec16) {
            MipOut mo{};
            for (uint32_t l = 0; l < f; ++l) {
                mo.data[l] = static_cast<uint8_t*>(levels[i + l].data);
                mo.pitch[l] = levels[i + l].stride;
            }
            const uint32_t gx = up.width / tw, gy = up.height / th;
            const uint8_t* up_data = static_cast<const uint8_t*>(up.data);
            const size_t up_stride = up.stride;
            if (gx % 2 == 0 && (uint64_t)gx * gy >= 2048)  // two tiles a CTA (faster than one or four) on large grids
                GOOFY_CUDA_TRY(goofy_gpu::launch_pdl(mip_fused_kernel<2>, dim3(gx / 2, gy), dim3(256), 0, st, up_data,
                                                     up_stride, log2u(tw), log2u(th), f, mo));
            else
                GOOFY_CUDA_TRY(goofy_gpu::launch_pdl(mip_fused_kernel<1>, dim3(gx, gy), dim3(256), 0, st, up_data,
                                                     up_stride, log2u(tw), log2u(th), f, mo));
            i += f;
            continue;
        }
        const uint32_t fx = up.width > lv.width ? 2 : 1, fy = up.height > lv.height ? 2 : 1;
        const bool pair = fx == 2 && reinterpret_cast<uintptr_t>(up.data) % 8 == 0 && up.stride % 8 == 0;
        const dim3 grid((lv.width + 255) / 256, lv.height);
        const uint8_t* up_data = static_cast<const uint8_t*>(up.data);
        uint8_t* lv_data = static_cast<uint8_t*>(lv.data);
        const size_t up_stride = up.stride, lv_stride = lv.stride;
        if (pair)
            GOOFY_CUDA_TRY(goofy_gpu::launch_pdl(mip_level_kernel<true>, grid, dim3(256), 0, st, up_data, up_stride,
                                                 lv_data, lv_stride, lv.width, lv.height, fx, fy));
        else
            GOOFY_CUDA_TRY(goofy_gpu::launch_pdl(mip_level_kernel<false>, grid, dim3(256), 0, st, up_data, up_stride,
                                                 lv_data, lv_stride, lv.width, lv.height, fx, fy));
        ++i;
    }
    *nlevels = n;
    return GOOFY_OK;
}

}  // extern "C"
