// Copies between a caller's pageable arrays and device memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace gtd {

struct HostSpan {
    void *host;
    void *dev;
    size_t bytes;
};

// The arrays of one copy.
struct HostSpans {
    HostSpan span[8];
    int count = 0;
    void add(const void *host, void *dev, size_t bytes) { span[count++] = {const_cast<void *>(host), dev, bytes}; }
};

// A handle's pinned staging ring, made when its large copies have come to what that pays for, and freed
// with the handle.
constexpr int kRingThreads = 8, kRingSlotsEach = 2;
struct HostRing {
    char *mem = nullptr;
    size_t moved = 0;  // bytes of large copies, up to that point
    cudaEvent_t events[kRingThreads * kRingSlotsEach] = {};  // one per slot
};
void release_host_ring(HostRing &ring);

// Copies the spans behind what `stream` has queued.  copy_to_host returns when every byte has arrived;
// after copy_to_device the caller's arrays may change once the stream has been synchronised.  Small
// copies, arrays that are pinned already, and all of them where the ring cannot be pinned, go through the
// driver; large ones are cut into chunks that a few threads move between the caller's arrays and pinned
// slots while the copy engine moves the slots: one thread copies, and takes the page faults of a fresh
// array, at 5 to 15 GB/s (88 bytes of each of 2^20 bodies to fresh arrays: 17.7 ms, 4.8 with the threads).
int copy_to_host(HostRing &ring, int device, cudaStream_t stream, const HostSpans &spans);
int copy_to_device(HostRing &ring, int device, cudaStream_t stream, const HostSpans &spans);

}  // namespace gtd
