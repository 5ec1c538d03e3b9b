// Copies between a caller's pageable arrays and device memory (host_copy.cuh).
#include "host_copy.cuh"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>

#include "gtd_internal.cuh"

namespace gtd {

constexpr size_t kSlotBytes = (size_t)512 << 10;
constexpr int kThreadsMost = 8, kSlotsEach = 2;
constexpr size_t kRingFrom = (size_t)4 << 20;  // smaller copies: starting the threads costs what they save
// Pinning the ring takes 3.7 ms and the threads save 0.15 ms a MB: a handle's ring is made once the large
// copies of its life, this one included, come to what that pays for.
constexpr size_t kRingPays = (size_t)40 << 20;

void release_host_ring(HostRing &ring) {
    for (cudaEvent_t e : ring.events) cudaEventDestroy(e);
    ring.events.clear();
    cudaFreeHost(ring.mem);
    ring.mem = nullptr;
}

static int ensure_ring(HostRing &ring) {
    if (ring.mem) return GTD_OK;
    constexpr int slots = kThreadsMost * kSlotsEach;
    while ((int)ring.events.size() < slots) {
        cudaEvent_t e;
        GTD_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        ring.events.push_back(e);
    }
    GTD_CUDA(cudaMallocHost(&ring.mem, slots * kSlotBytes));
    return GTD_OK;
}

// One thread's chunks (every `threads`-th), through its own slots.
static cudaError_t copy_chunks(HostRing &ring, int device, cudaStream_t stream, const std::vector<HostSpan> &chunks,
                               int thread, int threads, bool to_host) {
    cudaError_t e = cudaSetDevice(device);
    HostSpan held[kSlotsEach] = {};  // to_host: the chunk a slot is being filled with
    auto drain = [&](int s) {
        if (e != cudaSuccess || !held[s].bytes) return;
        const int slot = thread * kSlotsEach + s;
        e = cudaEventSynchronize(ring.events[(size_t)slot]);
        if (e == cudaSuccess && to_host) memcpy(held[s].host, ring.mem + slot * kSlotBytes, held[s].bytes);
        held[s].bytes = 0;
    };
    int s = 0;
    for (size_t k = (size_t)thread; k < chunks.size() && e == cudaSuccess; k += (size_t)threads, s = (s + 1) % kSlotsEach) {
        drain(s);
        if (e != cudaSuccess) break;
        const HostSpan &c = chunks[k];
        const int slot = thread * kSlotsEach + s;
        char *pinned = ring.mem + slot * kSlotBytes;
        if (!to_host) memcpy(pinned, c.host, c.bytes);
        e = to_host ? cudaMemcpyAsync(pinned, c.dev, c.bytes, cudaMemcpyDeviceToHost, stream)
                    : cudaMemcpyAsync(c.dev, pinned, c.bytes, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaEventRecord(ring.events[(size_t)slot], stream);
        held[s] = c;
    }
    for (int q = 0; q < kSlotsEach; ++q) drain((s + q) % kSlotsEach);
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

static int copy_spans(HostRing &ring, int device, cudaStream_t stream, const std::vector<HostSpan> &spans, bool to_host) {
    size_t total = 0;
    for (const HostSpan &s : spans) total += s.bytes;
    const int cores = (int)std::thread::hardware_concurrency();
    if (total >= kRingFrom && ring.moved < kRingPays) ring.moved += total;
    const bool threaded = total >= kRingFrom && cores >= 4 && ring.moved >= kRingPays;
    std::vector<HostSpan> chunks;
    std::vector<std::thread> pool;
    for (const HostSpan &s : spans) {
        if (!threaded || !pageable(s.host)) {
            GTD_CUDA(to_host ? cudaMemcpyAsync(s.host, s.dev, s.bytes, cudaMemcpyDeviceToHost, stream)
                             : cudaMemcpyAsync(s.dev, s.host, s.bytes, cudaMemcpyHostToDevice, stream));
            continue;
        }
        for (size_t at = 0; at < s.bytes; at += kSlotBytes)
            chunks.push_back({static_cast<char *>(s.host) + at, static_cast<char *>(s.dev) + at, std::min(kSlotBytes, s.bytes - at)});
    }
    if (!chunks.empty()) {
        int rc = ensure_ring(ring);
        if (rc) return rc;
        const int threads = std::min(kThreadsMost, cores / 2);
        std::atomic<int> error{cudaSuccess};
        auto work = [&](int t) {
            const cudaError_t e = copy_chunks(ring, device, stream, chunks, t, threads, to_host);
            if (e != cudaSuccess) error.store((int)e);
        };
        pool.reserve((size_t)threads);
        int started = 1;  // this thread takes part 0
        try {
            for (; started < threads; ++started) pool.emplace_back(work, started);
        } catch (...) {  // no more threads: their parts are done here
        }
        work(0);
        for (int t = started; t < threads; ++t) work(t);
        for (std::thread &t : pool) t.join();
        GTD_CUDA((cudaError_t)error.load());
    }
    if (to_host) GTD_CUDA(cudaStreamSynchronize(stream));
    return GTD_OK;
}

int copy_to_host(HostRing &ring, int device, cudaStream_t stream, const std::vector<HostSpan> &spans) {
    return copy_spans(ring, device, stream, spans, true);
}

int copy_to_device(HostRing &ring, int device, cudaStream_t stream, const std::vector<HostSpan> &spans) {
    return copy_spans(ring, device, stream, spans, false);
}

}  // namespace gtd
