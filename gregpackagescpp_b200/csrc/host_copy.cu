// Copies between a caller's pageable arrays and device memory (host_copy.cuh).
#include "host_copy.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

#include "gtd_internal.cuh"

namespace gtd {

constexpr size_t kSlotBytes = (size_t)512 << 10;
constexpr int kSlots = kRingThreads * kRingSlotsEach;
constexpr size_t kRingFrom = (size_t)4 << 20;  // smaller copies: starting the threads costs what they save
// Making the ring takes 4 to 7 ms; its threads save 0.05 ms a MB of arrays in use and 0.14 of fresh ones, 0.1
// over an upload and a download.  So it pays after 40 to 70 MB, and a handle's ring is made once the large
// copies of its life, this one included, come to the lower end of that: two calls of 262144 bodies, host
// arrays in and out, run at 3.03e12 pair-interactions/s with it and at 2.7 to 3.0e12 with 64 MiB.
constexpr size_t kRingPays = (size_t)40 << 20;

void release_host_ring(HostRing &ring) {
    for (cudaEvent_t &e : ring.events) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    cudaFreeHost(ring.mem);
    ring.mem = nullptr;
}

// Whether the ring is there.  Where it cannot be made the copies go on through the driver, and the next
// attempt waits for as many bytes again.
static bool ensure_ring(HostRing &ring) {
    if (ring.mem) return true;
    bool ok = true;
    for (cudaEvent_t &e : ring.events) ok = ok && (e || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess);
    ok = ok && cudaMallocHost(&ring.mem, kSlots * kSlotBytes) == cudaSuccess;
    if (ok) return true;
    cudaGetLastError();
    ring.mem = nullptr;
    ring.moved = 0;
    return false;
}

// One thread's chunks (every `threads`-th of the spans in ring_mask), through its own slots.
static cudaError_t copy_chunks(HostRing &ring, int device, cudaStream_t stream, const HostSpans &spans, unsigned ring_mask,
                               int thread, int threads, bool to_host) {
    cudaError_t e = cudaSetDevice(device);
    HostSpan held[kRingSlotsEach] = {};  // the chunk a slot is in use for
    auto drain = [&](int s) {
        if (e != cudaSuccess || !held[s].bytes) return;
        const int slot = thread * kRingSlotsEach + s;
        e = cudaEventSynchronize(ring.events[slot]);
        if (e == cudaSuccess && to_host) memcpy(held[s].host, ring.mem + slot * kSlotBytes, held[s].bytes);
        held[s].bytes = 0;
    };
    int s = 0, k = 0;
    for (int a = 0; a < spans.count; ++a) {
        if (!(ring_mask >> a & 1u)) continue;
        const HostSpan &span = spans.span[a];
        for (size_t at = 0; at < span.bytes && e == cudaSuccess; at += kSlotBytes, ++k) {
            if (k % threads != thread) continue;
            drain(s);
            if (e != cudaSuccess) break;
            const HostSpan c{static_cast<char *>(span.host) + at, static_cast<char *>(span.dev) + at,
                             std::min(kSlotBytes, span.bytes - at)};
            const int slot = thread * kRingSlotsEach + s;
            char *pinned = ring.mem + slot * kSlotBytes;
            if (!to_host) memcpy(pinned, c.host, c.bytes);
            e = to_host ? cudaMemcpyAsync(pinned, c.dev, c.bytes, cudaMemcpyDeviceToHost, stream)
                        : cudaMemcpyAsync(c.dev, pinned, c.bytes, cudaMemcpyHostToDevice, stream);
            if (e == cudaSuccess) e = cudaEventRecord(ring.events[slot], stream);
            held[s] = c;
            s = (s + 1) % kRingSlotsEach;
        }
    }
    for (int q = 0; q < kRingSlotsEach; ++q) drain((s + q) % kRingSlotsEach);
    return e;
}

static bool pageable(const void *p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

static int copy_spans(HostRing &ring, int device, cudaStream_t stream, const HostSpans &spans, bool to_host) {
    size_t total = 0;
    for (int a = 0; a < spans.count; ++a) total += spans.span[a].bytes;
    const int cores = (int)std::thread::hardware_concurrency();
    if (total >= kRingFrom && ring.moved < kRingPays) ring.moved += total;
    unsigned ring_mask = 0;  // the spans that go through the ring
    if (total >= kRingFrom && cores >= 4 && ring.moved >= kRingPays) {
        for (int a = 0; a < spans.count; ++a)
            if (spans.span[a].bytes && pageable(spans.span[a].host)) ring_mask |= 1u << a;
        if (ring_mask && !ensure_ring(ring)) ring_mask = 0;
    }
    for (int a = 0; a < spans.count; ++a) {
        const HostSpan &s = spans.span[a];
        if (ring_mask >> a & 1u) continue;
        GTD_CUDA(to_host ? cudaMemcpyAsync(s.host, s.dev, s.bytes, cudaMemcpyDeviceToHost, stream)
                         : cudaMemcpyAsync(s.dev, s.host, s.bytes, cudaMemcpyHostToDevice, stream));
    }
    if (ring_mask) {
        const int threads = std::min(kRingThreads, cores / 2);
        std::atomic<int> error{cudaSuccess};
        auto work = [&](int t) {
            const cudaError_t e = copy_chunks(ring, device, stream, spans, ring_mask, t, threads, to_host);
            if (e != cudaSuccess) error.store((int)e);
        };
        std::thread pool[kRingThreads];
        int started = 1;  // this thread takes part 0
        try {
            for (; started < threads; ++started) pool[started] = std::thread(work, started);
        } catch (...) {  // no more threads: their parts are done here
        }
        work(0);
        for (int t = started; t < threads; ++t) work(t);
        for (int t = 1; t < started; ++t) pool[t].join();
        if (error.load() != cudaSuccess) {
            cudaStreamSynchronize(stream);  // nothing is left in the slots
            GTD_CUDA((cudaError_t)error.load());
        }
    }
    if (to_host) GTD_CUDA(cudaStreamSynchronize(stream));
    return GTD_OK;
}

int copy_to_host(HostRing &ring, int device, cudaStream_t stream, const HostSpans &spans) {
    return copy_spans(ring, device, stream, spans, true);
}

int copy_to_device(HostRing &ring, int device, cudaStream_t stream, const HostSpans &spans) {
    return copy_spans(ring, device, stream, spans, false);
}

}  // namespace gtd
