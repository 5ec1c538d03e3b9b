// Host copies through the pinned ring (csrc/host_copy.cu) over a CUDA runtime of this file's own: device
// memory is host memory, and a copy happens only when somebody waits for it or for a later event, so that
// a slot that is used again, or read, without its wait shows as wrong bytes.
#include "host_copy.cu"

#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>
#include <mutex>
#include <random>
#include <vector>

namespace {

struct Op {
    void *dst = nullptr;
    const void *src = nullptr;
    size_t bytes = 0;
    long event = -1;  // marks an event's record instead of a copy
};
std::recursive_mutex mu;
std::deque<Op> queue_;
long recorded = 0, passed = 0;           // records made, records reached
std::map<cudaEvent_t, long> last_record;  // event -> its record
std::map<const char *, size_t> pinned;
bool pin_fails = false;
int events_alive = 0, copy_fails_after = -1;
long ring_copies = 0;  // copies from or to a pinned block

void run_until(long record) {
    while (passed < record && !queue_.empty()) {
        const Op op = queue_.front();
        queue_.pop_front();
        if (op.event >= 0) passed = op.event;
        else std::memcpy(op.dst, op.src, op.bytes);
    }
}
bool in_pinned(const void *p) {
    auto it = pinned.upper_bound((const char *)p);
    return it != pinned.begin() && (const char *)p < (--it)->first + it->second;
}

}  // namespace

namespace gtd {
int fail(int code, const char *, ...) { return code; }
int cuda_fail(cudaError_t, const char *, const char *, int) { return GTD_ERR_CUDA; }
}  // namespace gtd

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    if (pin_fails) return cudaErrorMemoryAllocation;
    *p = std::malloc(n);
    pinned[(const char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    pinned.erase((const char *)p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    ++events_alive;
    *e = (cudaEvent_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    --events_alive;
    std::free((void *)e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> l(mu);
    Op op;
    op.event = last_record[e] = ++recorded;
    queue_.push_back(op);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> l(mu);
    run_until(last_record[e]);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    std::lock_guard<std::recursive_mutex> l(mu);
    while (!queue_.empty()) run_until(passed + 1);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    *a = cudaPointerAttributes{};
    a->type = in_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (copy_fails_after == 0) return cudaErrorUnknown;
    if (copy_fails_after > 0) --copy_fails_after;
    const void *host = kind == cudaMemcpyHostToDevice ? src : dst;
    if (in_pinned(host)) {
        ++ring_copies;
        queue_.push_back({dst, src, n, -1});
    } else {  // the driver stages pageable memory: done on return
        while (!queue_.empty()) run_until(passed + 1);
        std::memcpy(dst, src, n);
    }
    return cudaSuccess;
}
}

using namespace gtd;

static int bad(const char *what) {
    std::printf("%s\n", what);
    return 1;
}

// Six arrays of a handle of n bodies there and back; array `pin` (or none) is pinned already.
static int round_trip(HostRing &ring, size_t n, int pin, unsigned seed) {
    const size_t words[6] = {3, 3, 3, 1, 1, 1};
    std::vector<std::vector<char>> host, dev, back;
    std::mt19937_64 rng(seed);
    HostSpans up, down;
    char *block = nullptr;
    for (int a = 0; a < 6; ++a) {
        const size_t bytes = words[a] * 8 * n;
        host.emplace_back(bytes);
        dev.emplace_back(bytes, 1);
        back.emplace_back(bytes, 2);
        for (size_t k = 0; k + 8 <= bytes; k += 8) *(uint64_t *)&host[a][k] = rng();
    }
    if (pin >= 0) {
        cudaHostAlloc((void **)&block, host[pin].size(), 0);
        if (block) std::memcpy(block, host[pin].data(), host[pin].size());
    }
    for (int a = 0; a < 6; ++a) {
        up.add(a == pin && block ? block : host[a].data(), dev[a].data(), host[a].size());
        down.add(a == pin && block ? block : back[a].data(), dev[a].data(), host[a].size());
    }
    if (copy_to_device(ring, 0, nullptr, up)) return bad("copy to the device failed");
    cudaStreamSynchronize(nullptr);
    for (int a = 0; a < 6; ++a)
        if (dev[a] != host[a]) return bad("wrong bytes on the device");
    if (block) std::memset(block, 0, host[pin].size());
    if (copy_to_host(ring, 0, nullptr, down)) return bad("copy to the host failed");
    for (int a = 0; a < 6; ++a)
        if (std::memcmp(a == pin && block ? block : back[a].data(), host[a].data(), host[a].size())) return bad("wrong bytes on the host");
    if (block) cudaFreeHost(block);
    return 0;
}

int main() {
    const bool threads = std::thread::hardware_concurrency() >= 4;
    HostRing ring, other;
    // small copies never make the ring
    for (int k = 0; k < 40; ++k)
        if (round_trip(ring, 10007, -1, 1)) return 1;
    if (ring.mem || ring_copies) return bad("small copies made a ring");
    // large ones do, once they have paid for it; sizes with partial last chunks and a whole number of them
    for (size_t n : {(size_t)262144, (size_t)262145, (size_t)65536 * 3, (size_t)150001, (size_t)300007})
        for (int pin : {-1, 0, 4})
            if (round_trip(ring, n, pin, (unsigned)n)) return 1;
    if (threads && (!ring.mem || ring_copies == 0)) return bad("large copies made no ring");
    // a second handle beside it has its own
    for (int k = 0; k < 3; ++k)
        if (round_trip(other, 400009, -1, 7) || round_trip(ring, 270001, -1, 8)) return 1;
    if (threads && (!other.mem || other.mem == ring.mem)) return bad("handles share a ring");
    release_host_ring(other);
    if (round_trip(ring, 262147, 2, 9)) return 1;
    // memory that cannot be pinned: the driver's copy
    HostRing none;
    pin_fails = true;
    for (int k = 0; k < 4; ++k)
        if (round_trip(none, 400009, -1, 11)) return 1;
    if (none.mem) return bad("a ring without memory");
    pin_fails = false;
    for (int k = 0; k < 4; ++k)
        if (round_trip(none, 400009, -1, 12)) return 1;
    if (threads && !none.mem) return bad("no ring once memory can be pinned again");
    // an error in the middle is returned, with nothing left under way
    std::vector<char> h(48 << 20), d(48 << 20);
    HostSpans one;
    one.add(h.data(), d.data(), h.size());
    copy_fails_after = 20;
    if (copy_to_device(ring, 0, nullptr, one) == GTD_OK || !queue_.empty()) return bad("an error in the middle");
    copy_fails_after = -1;
    if (round_trip(ring, 262147, -1, 13)) return 1;
    release_host_ring(ring);
    release_host_ring(none);
    release_host_ring(none);
    if (events_alive || !pinned.empty()) return bad("something is not given back");
    std::printf("ok%s\n", threads ? "" : " (too few cores for the ring)");
    return 0;
}
