// host_copy.h -- copies between device arrays and a caller's pageable host
// arrays (host_copy.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace zg {
namespace host {

// A piece of a copy: `host` and `dev` hold `bytes` each.
struct Piece {
    void *host;
    const void *dev;
    size_t bytes;
};

// One library context more / fewer: the staging memory goes with the last.
void retain();
void release();

// Device to host (to_host) or host to device, after the work queued on
// `stream` and before the work queued on it later; returns when the host
// arrays may be read or reused.
cudaError_t copy(int device, cudaStream_t stream, const Piece *pieces, int n, bool to_host);

}  // namespace host
}  // namespace zg
