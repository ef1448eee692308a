// af_xfer.h -- host<->device copies of row blocks (the fields a caller hands
// in or reads back) at the link's rate whether or not the host memory is
// pinned.
//
// Pinned (page-locked) host memory, and any copy under 2 MB, goes straight to
// the driver.  Larger copies of pageable memory, which the driver would move
// with one thread at a fraction of the link's rate (19 GB/s, about 10 from or to
// memory that no cache holds or that is touched for the first time), go
// through a ring of pinned buffers of this library instead: up to eight host
// threads fill (or drain) chunks while the DMA of others runs.  Such a copy
// returns when the host side is done with the caller's memory (for a copy to
// the device: when the data has left this library's buffers too).  Copies
// through the buffers run one at a time per process.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace af {

// Same arguments as cudaMemcpy2DAsync (pitches and width in bytes).
cudaError_t copy2d_h2d(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                       size_t rows, cudaStream_t st);
cudaError_t copy2d_d2h(void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                       size_t rows, cudaStream_t st);

}  // namespace af
