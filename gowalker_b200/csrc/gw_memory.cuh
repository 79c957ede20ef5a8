// Device memory of the library (internal to libgowalker.so).
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

struct gw_handle;

namespace gw {

// cudaMalloc.  On a full device the index of a resident CSR, which walks can do
// without, gives way: that of any engine on the current device that no call is
// using, and that of `self` (the engine whose call this is, or null).
cudaError_t device_malloc_any(void **p, size_t bytes, gw_handle *self = nullptr);
template <class T>
inline cudaError_t device_malloc(T **p, size_t bytes)
{
    return device_malloc_any((void **)p, bytes);
}

// The driver takes memory 2 MB at a time and keeps what is left of such a piece
// for smaller allocations: those cost 5 us where they find room, and 600 us, like
// every larger one, where they do not.  So buffers of this size and more are
// worth one allocation together, smaller ones each their own.
constexpr size_t kShareBytes = 3u << 19;

}  // namespace gw
