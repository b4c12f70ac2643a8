// Copies between the caller's host memory and the device's staging buffer.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace ym {

// A context or ensemble that may transfer: the pinned slots below live while any does.
void transfer_retain();
void transfer_release();
struct TransferUser {
    TransferUser() { transfer_retain(); }
    ~TransferUser() { transfer_release(); }
    TransferUser(const TransferUser&) = delete;
    TransferUser& operator=(const TransferUser&) = delete;
};

// Host to device (upload) or device to host, ordered after what `st` holds.
// The device side is enqueued on `st`; host memory has been read (upload: and
// `st` need not be synchronised for the caller to reuse it) or written when
// the call returns, except for memory that is pinned already, which is copied
// by `st` itself: synchronise `st` before touching that.
cudaError_t transfer_upload(int device, void* dev, const void* host, size_t bytes, cudaStream_t st);
cudaError_t transfer_download(int device, void* host, const void* dev, size_t bytes, cudaStream_t st);

}  // namespace ym
