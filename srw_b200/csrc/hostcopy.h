// Copies between the caller's pageable arrays and the device, by several threads over a ring of
// pinned blocks.
//
// A cudaMemcpyAsync of pageable memory runs through the driver's own staging on one thread: at the
// 64 MB of a 2048 x 2048 result it moved 4.5 GB/s, most of it the page faults of an array that was
// just allocated, while the link takes 50.  Here each thread owns two pinned blocks, so its memcpy of
// one block (and the page faults it takes) runs beside the other block's transfer and beside the
// other threads.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace srwg {

struct CopySeg {
    void* host;
    void* dev;
    size_t bytes;
};

// The pinned blocks of one device, kept between calls (HOSTCOPY_THREADS x 2 x HOSTCOPY_BLOCK bytes,
// 16 MiB in all, allocated by the first copy that needs them).
struct HostRing {
    char* pinned = nullptr;
    cudaEvent_t* ev = nullptr;
};

constexpr int HOSTCOPY_THREADS = 16;
constexpr size_t HOSTCOPY_BLOCK = 1u << 19;

// Copies the segments in stream order: host to device (toDevice; the host arrays have been read when
// it returns, the device sees the data in stream order) or device to host (the host arrays hold the
// data when it returns).  Not thread-safe for one ring: the callers hold the library's lock.
cudaError_t copy_segments(HostRing& ring, int dev, const CopySeg* segs, int n, bool toDevice, cudaStream_t st);

}  // namespace srwg
