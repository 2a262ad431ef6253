// Large copies between the caller's (pageable) memory and the device.
//
// The driver moves pageable memory through one staging thread: 11 GB/s up, 17-21
// down, and 2 GB/s down into pages that the caller has not touched yet, against
// 54 GB/s of the link; a two-dimensional copy that changes the row pitch moves
// 0.8 GB/s.  Here up to eight threads copy pieces through a pinned ring, each
// with two slots, so that the host copies (and the page faults) run in parallel
// and overlap the transfers: 41-46 GB/s both ways at 256 MB, 22-32 at 4-16 MB.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace b200 {

// `rows` rows of row_bytes, pitched on either side; going up, the device rows'
// bytes past row_bytes are zeroed.
struct XferSeg {
    void *host;
    size_t host_pitch;
    void *dev;
    size_t dev_pitch, row_bytes, rows;
};

// Copies all segments, ordered after the work on stream s.  Up: returns with the
// transfers enqueued on s and the host memory read; down: with the host memory
// written.  False: not taken (too small, page-locked dense rows, the ring in use
// by another thread, not set up yet, another device, s being captured or the
// calling thread's own default stream) -- nothing was done and the caller copies
// by other means; e: the error of a copy that was taken.
bool xfer_up(const XferSeg *segs, int n, cudaStream_t s, cudaError_t &e);
bool xfer_down(const XferSeg *segs, int n, cudaStream_t s, cudaError_t &e);

// Host memory that is page-locked (such rows need no ring).
bool host_pinned(const void *p);

// One segment, either way, with the driver's copy where the ring does not take
// it (up: like cudaMemcpy2DAsync from pageable memory; down: synchronises).
cudaError_t copy_up(const XferSeg &seg, cudaStream_t s);
cudaError_t copy_down(const XferSeg &seg, cudaStream_t s);

} // namespace b200
