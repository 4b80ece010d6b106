// batch_noalloc.cu -- batch encoding that allocates nothing.
//
// Some callers may not allocate on the path that encodes: a texture-streaming
// thread working inside a renderer's frame budget, where cudaMalloc / cudaFree
// can stall or synchronise the whole device, or a host engine that owns every
// byte of GPU memory through its own allocator and does not let libraries call
// the CUDA allocator.  goofy_gpu_batch_create allocates, so those callers
// cannot use it.  Here a call is one launch of the batch kernel that takes the
// descriptors as its by-value parameter: no device scratch at all, nothing
// shared between calls, and nothing read from the calling thread's memory
// after the call returns.  Inputs and outputs are the caller's device buffers.
// (With the tables written into a device array by a first kernel, 24 tiles of
// 128x128 took 12.3 us a call from Python; the one launch takes 3.1 us, the
// host's cost of making it.)
#include <cuda_runtime.h>

#include <cstdio>

#include "../../include/goofy_gpu.h"
#include "batch.h"
#include "host_util.h"

static_assert(GOOFY_NOALLOC_MAX_IMAGES == 256, "a call is one launch with room for 256 images");

extern "C" GOOFY_EXPORT int goofy_gpu_batch_encode_noalloc(const goofy_gpu_image* images, uint32_t count,
                                                           void* stream)
{
    if (count > GOOFY_NOALLOC_MAX_IMAGES) {
        char msg[128];
        std::snprintf(msg, sizeof msg, "goofy_gpu_batch_encode_noalloc: at most %u images per call, got %u",
                      GOOFY_NOALLOC_MAX_IMAGES, count);
        return goofy_gpu::fail(GOOFY_ERR_TOO_LARGE, msg);
    }
    if (count == 0) return GOOFY_OK;
    if (!images) return goofy_gpu::fail(GOOFY_ERR_INVALID, "goofy_gpu_batch_encode_noalloc: images is NULL");
    const goofy_gpu::BatchTile tile{128, 1, 256, 0};
    goofy_gpu::ParamImage table[GOOFY_NOALLOC_MAX_IMAGES];  // 8 KB of this thread's stack; the launch copies it
    goofy_gpu::ParamLaunch l{table, 0, 0, goofy_gpu::kMixed};
    const int rc = goofy_gpu::validate_and_fill(images, count, tile, &l);
    if (rc != GOOFY_OK) return rc;  // nothing launched for an invalid batch
    GOOFY_CUDA_TRY(goofy_gpu::launch_batch_params(l, tile, static_cast<cudaStream_t>(stream)));
    return GOOFY_OK;
}
