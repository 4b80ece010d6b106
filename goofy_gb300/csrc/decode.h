// decode.h -- launchers of the block decoder and the squared-error reduction.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace goofy_gpu {

// Decode (width/4)*(height/4) blocks into RGBA8 rows (`rgba`, `stride`: both
// 16-byte aligned).  Adds the count of unsupported ETC1 blocks to *unsupported.
cudaError_t launch_decode(int codec, const uint8_t* blocks, uint32_t width, uint32_t height, uint8_t* rgba,
                          size_t stride, unsigned long long* unsupported, cudaStream_t stream);

// Where the sums go when the launch is their only user (`sums` and *finished
// zero before it): the last CTA to finish writes the six totals to `host`
// (mapped host memory) and leaves `sums` and *finished zero for the next
// launch.  A total is never kNoTotal: with that in all six before the launch,
// the host need not wait for the stream.
//
// Total 4 is the unsupported-block count (below 2^31) and, for every warp that
// left blocks out because a bounded wait of the ring gave up, kGaveUp: the
// sums are then too low, and complete() is false.
constexpr unsigned long long kNoTotal = ~0ull, kGaveUp = 1ull << 40;
inline bool complete(const unsigned long long totals[6]) { return totals[4] < kGaveUp; }
struct ErrorResult {
    unsigned long long* host = nullptr;
    unsigned int* finished = nullptr;
};

// Adds the per-channel sums of squared differences between `src` and the
// decoded blocks to sums[0..3], the unsupported-block count to sums[4] and the
// sum of squared luminosity differences (hundredths) to sums[5].
cudaError_t launch_block_error(int codec, const uint8_t* blocks, const uint8_t* src, uint32_t width, uint32_t height,
                               size_t stride, bool vec16, unsigned long long* sums, cudaStream_t stream,
                               ErrorResult result = {});

// The same on the bulk-copy ring (encode_tma.cu), for rows of 205 blocks and
// more.
cudaError_t launch_error_tma(int codec, const uint8_t* blocks, const uint8_t* src, uint32_t width, uint32_t height,
                             size_t stride, bool vec16, unsigned long long* sums, ErrorResult result,
                             cudaStream_t stream);

struct BatchImage;

// Adds the six error sums of every image of a batch (blocks at `dst`, source
// at `src`) to sums[6 * i + c]; work units as for the batch encoder
// (`first_unit`, `unit_blocks`), `work_counter` reading 0 at the start.
cudaError_t launch_quality_batch(const BatchImage* images, uint32_t n_images, const uint32_t* first_unit,
                                 uint32_t total_units, uint32_t unit_blocks, uint32_t* work_counter,
                                 unsigned long long* sums, cudaStream_t stream);

}  // namespace goofy_gpu
