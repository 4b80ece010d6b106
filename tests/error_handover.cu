// error_handover.cu -- TEST ONLY.  The end of the quality kernels
// (error_reduce.cuh) on sums made up here: CTAs of 128 threads, each thread
// with sq = {1, 2, 3, 4} and one unsupported block; the warps of `gave_up`
// (bit: CTA * 4 + warp) report a wait that gave up.  No kernel here waits.
#include <cuda_runtime.h>

#include "error_reduce.cuh"

__global__ void handover_kernel(unsigned gave_up, unsigned long long* sums, goofy_gpu::ErrorResult result)
{
    goofy_gpu::ErrorSums e{};
    for (int c = 0; c < 4; ++c) e.sq[c] = c + 1;
    goofy_gpu::reduce_errors<128>(e, 1u, gave_up >> (blockIdx.x * 4 + threadIdx.x / 32) & 1u, sums, result);
}

// totals[6] as handed to the host (host = 1) or as the launch left them in
// its accumulators; -1 for a CUDA error, else complete().
extern "C" int handover(unsigned ctas, unsigned gave_up, int host, unsigned long long* totals)
{
    unsigned long long *dev = nullptr, *mapped = nullptr;
    bool ok = cudaMalloc(&dev, 7 * sizeof *dev) == cudaSuccess && cudaMemset(dev, 0, 7 * sizeof *dev) == cudaSuccess &&
              cudaHostAlloc(&mapped, 6 * sizeof *mapped, cudaHostAllocMapped) == cudaSuccess;
    if (ok) {
        goofy_gpu::ErrorResult r;
        if (host) r = {mapped, reinterpret_cast<unsigned*>(dev + 6)};
        handover_kernel<<<ctas, 128>>>(gave_up, dev, r);
        ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
        if (ok && host) for (int k = 0; k < 6; ++k) totals[k] = mapped[k];
        else if (ok) ok = cudaMemcpy(totals, dev, 6 * sizeof *dev, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    cudaFreeHost(mapped);
    cudaFree(dev);
    return ok ? goofy_gpu::complete(totals) : -1;
}

extern "C" int complete_totals(const unsigned long long* totals) { return goofy_gpu::complete(totals); }
