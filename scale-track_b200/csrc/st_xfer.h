/*
 * st_xfer.h -- copies between device memory and the caller's host arrays (st_xfer.cu).
 */
#ifndef ST_XFER_H
#define ST_XFER_H

#include <cstddef>
#include <cuda_runtime.h>

namespace st {

/* One contiguous copy: `host` in the caller's memory (pageable or pinned), `dev` on the device. */
struct XferSeg {
    void* host;
    void* dev;
    size_t bytes;
};

/* Copies the segments in the order of stream `s` and returns when they have arrived (down:
 * device to host, up: host to device).  Call with `device` current.  ahead: bytes that the caller
 * goes on to copy in the same call. */
cudaError_t xfer_down(const XferSeg* seg, int n, int device, cudaStream_t s, size_t ahead = 0);
cudaError_t xfer_up(const XferSeg* seg, int n, int device, cudaStream_t s, size_t ahead = 0);

/* The pinned staging buffer is shared by the process: made once enough has been copied, given
 * back when the last handle is destroyed. */
void xfer_retain();
void xfer_release();

}  // namespace st

#endif
