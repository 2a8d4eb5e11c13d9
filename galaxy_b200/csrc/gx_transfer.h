// gx_transfer.h -- host <-> device copies of callers' arrays (gx_transfer.cpp).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace gx {

struct HostPiece {
  void* host;       // null: skipped
  const void* dev;
  size_t bytes;
};

// Pageable outputs of at most this many bytes together go through the caller's own pinned
// buffer of this size.
constexpr size_t kSmallOut = size_t{1} << 16;

// dst (device) <- src (host), in order on st. src has been read when it returns, unless it
// is pinned (then it must stay until the copy has run, as for cudaMemcpyAsync). The device
// is the current one.
cudaError_t copy_in(int device, cudaStream_t st, void* dst, const void* src, size_t bytes);
// The pieces' device memory, after the work enqueued on st, to the host: complete, and the
// stream idle, when it returns. small: kSmallOut bytes of pinned memory that only this call
// uses, or null.
cudaError_t copy_out(int device, cudaStream_t st, const HostPiece* pieces, int count, char* small = nullptr);
// Every handle and batch holds a reference; with the last one go the staging buffers but one.
void transfer_ref();
void transfer_unref();

}  // namespace gx
