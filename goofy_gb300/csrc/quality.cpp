// quality.cpp -- C ABI of the GPU decoder and the encode-quality measurement
// (the reference harness's check: decode with Src/decoder.cpp, compare with
// getMsePsnr, Src/main.cpp:403-469).
#include <cuda.h>  // driver types for the context queries (entry points fetched at run time)
#include <cuda_runtime.h>

#include <cfloat>
#include <algorithm>
#include <chrono>
#include <cmath>
#include <mutex>

#include "../../include/goofy_gpu.h"
#include "context_slots.h"
#include "decode.h"
#include "host_util.h"

namespace {

int check(int codec, const void* a, const void* b, uint32_t width, uint32_t height)
{
    if (codec != GOOFY_CODEC_BC1 && codec != GOOFY_CODEC_ETC1S) return GOOFY_ERR_INVALID;
    if (width % 4) return GOOFY_ERR_WIDTH;
    if (height % 4) return GOOFY_ERR_HEIGHT;
    if (width == 0 || height == 0) return GOOFY_OK;
    if (!a || !b) return GOOFY_ERR_INVALID;
    if ((uint64_t)(width / 4) * (height / 4) > 0x7fffffffull) return GOOFY_ERR_TOO_LARGE;
    return 1;
}

// Unique id of the calling thread's current context, 0 if it has none.
uint64_t current_context_id()
{
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(p);
        p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(p);
        cudaGetLastError();
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

// Accumulators of the synchronous quality calls, per context.  Zero between
// calls: the error kernel's last CTA moves its totals to `host` and clears
// them, so a call is one launch and a short wait.  With a memset before the
// kernel and a copy behind it a call took 31.4 us at 4096^2 BC1 from Python,
// 29.3 us without both, 27.2 us with a completion word polled, 25.0 us with the
// totals themselves polled and a shorter end of the kernel (error_reduce.cuh).
struct Accumulators {
    unsigned long long* sums = nullptr;  // six sums and the finished-CTA count
    unsigned long long* host = nullptr;  // mapped: six totals
};
std::mutex g_mu;
goofy_gpu::ContextSlots<Accumulators, 64> g_acc;

// Those of the current context, which cudaDeviceReset ends with its memory:
// pointers kept for the device would be written after that, by the host below
// and by the kernel.
int accumulators(Accumulators** out)
{
    uint64_t id = current_context_id();
    if (id == 0) {
        GOOFY_CUDA_TRY(cudaFree(nullptr));  // makes the device's primary context current
        id = current_context_id();
    }
    if (id == 0) return goofy_gpu::fail(GOOFY_ERR_CUDA, "quality: the driver names no current context");
    Accumulators& a = g_acc.at(id);
    *out = &a;
    if (a.host) return GOOFY_OK;
    if (!a.sums) GOOFY_CUDA_TRY(cudaMalloc(&a.sums, 7 * sizeof(unsigned long long)));
    GOOFY_CUDA_TRY(cudaMemset(a.sums, 0, 7 * sizeof(unsigned long long)));  // on the stream of the launches
    unsigned long long* host = nullptr;
    GOOFY_CUDA_TRY(cudaHostAlloc(&host, 6 * sizeof(unsigned long long), cudaHostAllocMapped | cudaHostAllocPortable));
    a.host = host;
    return GOOFY_OK;
}

// Waits until the GPU has replaced all six kNoTotal of `host` and copies them
// to h: polls for a few milliseconds, then waits for the stream, which also
// reports a launch that failed.  (Launch and stream synchronisation of an
// empty kernel take 9.5 us on this GPU, launch and polling 7.0.)
cudaError_t wait_for(const unsigned long long* host, unsigned long long h[6], cudaStream_t stream)
{
    const auto read = [&] {
        bool all = true;
        for (int k = 0; k < 6; ++k) {
            h[k] = __atomic_load_n(&host[k], __ATOMIC_ACQUIRE);
            all = all && h[k] != goofy_gpu::kNoTotal;
        }
        return all;
    };
    const auto t0 = std::chrono::steady_clock::now();
    do {
        for (int i = 0; i < 256; ++i)
            if (read()) return cudaSuccess;
    } while (std::chrono::steady_clock::now() - t0 < std::chrono::milliseconds(5));
    const cudaError_t e = cudaStreamSynchronize(stream);
    return e != cudaSuccess ? e : read() ? cudaSuccess : cudaErrorUnknown;
}

// The launch behind both forms of the measurement, arguments of check() passed.
int block_error(int codec, const void* blocks, const void* src, uint32_t width, uint32_t height, uint32_t stride,
                unsigned long long* sums, cudaStream_t stream, goofy_gpu::ErrorResult result)
{
    if ((uint64_t)stride < 4ull * width) return GOOFY_ERR_INVALID;
    const uintptr_t s = reinterpret_cast<uintptr_t>(src);
    if (s % 4 || stride % 4 || reinterpret_cast<uintptr_t>(blocks) % 8) return GOOFY_ERR_ALIGNMENT;
    GOOFY_CUDA_TRY(goofy_gpu::launch_block_error(codec, static_cast<const uint8_t*>(blocks),
                                                 static_cast<const uint8_t*>(src), width, height, stride,
                                                 s % 16 == 0 && stride % 16 == 0, sums, stream, result));
    return GOOFY_OK;
}

}  // namespace

extern "C" {

GOOFY_EXPORT int goofy_gpu_decode_device(int codec, void* rgba, uint32_t rgba_stride, const void* blocks,
                                         uint32_t width, uint32_t height, uint64_t* d_unsupported, void* stream)
{
    int rc = check(codec, rgba, blocks, width, height);
    if (rc <= 0) return rc;
    if (!d_unsupported || reinterpret_cast<uintptr_t>(d_unsupported) % 8) return GOOFY_ERR_INVALID;
    if ((uint64_t)rgba_stride < 4ull * width) return GOOFY_ERR_INVALID;
    if (reinterpret_cast<uintptr_t>(rgba) % 16 || rgba_stride % 16 || reinterpret_cast<uintptr_t>(blocks) % 8)
        return GOOFY_ERR_ALIGNMENT;
    GOOFY_CUDA_TRY(goofy_gpu::launch_decode(codec, static_cast<const uint8_t*>(blocks), width, height,
                                            static_cast<uint8_t*>(rgba), rgba_stride,
                                            reinterpret_cast<unsigned long long*>(d_unsupported),
                                            static_cast<cudaStream_t>(stream)));
    return GOOFY_OK;
}

GOOFY_EXPORT int goofy_gpu_block_error_device(int codec, const void* blocks, const void* src, uint32_t width,
                                              uint32_t height, uint32_t stride, uint64_t* d_sums, void* stream)
{
    int rc = check(codec, blocks, src, width, height);
    if (rc <= 0) return rc;
    if (!d_sums || reinterpret_cast<uintptr_t>(d_sums) % 8) return GOOFY_ERR_INVALID;
    return block_error(codec, blocks, src, width, height, stride, reinterpret_cast<unsigned long long*>(d_sums),
                       static_cast<cudaStream_t>(stream), {});
}

}  // extern "C"

namespace {

// getPSNR, Src/main.cpp:386-395
double psnr_of(double mse, double peak) { return mse < 0.0000001 ? DBL_MAX : 10.0 * std::log10((peak * peak) / mse); }

// Runs the error kernel on the current device and reads the six sums back.
int error_sums(int codec, const void* blocks, const void* src, uint32_t width, uint32_t height, uint32_t stride,
               unsigned long long h[6])
{
    int rc = check(codec, blocks, src, width, height);
    if (rc <= 0) return rc == GOOFY_OK ? GOOFY_ERR_INVALID : rc;
    std::lock_guard<std::mutex> lk(g_mu);
    Accumulators* acc = nullptr;
    if ((rc = accumulators(&acc)) != GOOFY_OK) return rc;
    const Accumulators& a = *acc;
    cudaStream_t st = nullptr;
    const goofy_gpu::ErrorResult result{a.host, reinterpret_cast<unsigned int*>(a.sums + 6)};
    for (int k = 0; k < 6; ++k) __atomic_store_n(&a.host[k], goofy_gpu::kNoTotal, __ATOMIC_RELEASE);
    if ((rc = block_error(codec, blocks, src, width, height, stride, a.sums, st, result)) != GOOFY_OK) return rc;
    GOOFY_CUDA_TRY(wait_for(a.host, h, st));
    if (!goofy_gpu::complete(h))
        return goofy_gpu::fail(GOOFY_ERR_TIMEOUT, "quality: a bounded wait of the bulk-copy ring gave up");
    return GOOFY_OK;
}

}  // namespace

extern "C" {

GOOFY_EXPORT int goofy_gpu_psnr_rgb(int codec, const void* blocks, const void* src, uint32_t width, uint32_t height,
                                    uint32_t stride, double* psnr_rgb, uint64_t* sums_out)
{
    unsigned long long h[6];
    const int rc = error_sums(codec, blocks, src, width, height, stride, h);
    if (rc != GOOFY_OK) return rc;
    if (sums_out)
        for (int i = 0; i < 5; ++i) sums_out[i] = h[i];
    // getPSNR(mseRGB, 768), Src/main.cpp:455, :466
    const double mse = (double)(h[0] + h[1] + h[2]) / ((double)width * (double)height);
    if (psnr_rgb) *psnr_rgb = psnr_of(mse, 768.0);
    return GOOFY_OK;
}

GOOFY_EXPORT int goofy_gpu_mse_psnr(int codec, const void* blocks, const void* src, uint32_t width, uint32_t height,
                                    uint32_t stride, goofy_gpu_quality* out)
{
    if (!out) return GOOFY_ERR_INVALID;
    unsigned long long h[6];
    const int rc = error_sums(codec, blocks, src, width, height, stride, h);
    if (rc != GOOFY_OK) return rc;
    // Src/main.cpp:456-468; the harness's r is byte 2 and its b byte 0
    const double n = (double)(uint32_t)(width * height);
    goofy_gpu_quality& r = *out;
    r.mse_r = (double)h[2] / n;
    r.mse_g = (double)h[1] / n;
    r.mse_b = (double)h[0] / n;
    r.mse_a = (double)h[3] / n;
    r.mse_rgb = (double)(h[0] + h[1] + h[2]) / n;
    r.mse_y = (double)h[5] / 10000.0 / n;
    r.mse_max = std::max(std::max(r.mse_r, r.mse_g), std::max(r.mse_b, r.mse_a));
    r.psnr_r = psnr_of(r.mse_r, 255.0);
    r.psnr_g = psnr_of(r.mse_g, 255.0);
    r.psnr_b = psnr_of(r.mse_b, 255.0);
    r.psnr_a = psnr_of(r.mse_a, 255.0);
    r.psnr_min = std::min(std::min(r.psnr_r, r.psnr_g), std::min(r.psnr_b, r.psnr_a));
    r.psnr_rgb = psnr_of(r.mse_rgb, 768.0);
    r.psnr_y = psnr_of(r.mse_y, 255.0);
    r.unsupported_blocks = h[4];
    return GOOFY_OK;
}

}  // extern "C"
