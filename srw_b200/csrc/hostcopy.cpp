#include "hostcopy.h"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <new>
#include <thread>

namespace srwg {

// Copies of fewer bytes than this run on the calling thread alone: starting threads costs about 0.1 ms.
constexpr size_t HOSTCOPY_THREADED = 4u << 20;

static bool pageable(const void* p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

static bool ring_ready(HostRing& r)
{
    if (r.pinned != nullptr) return true;
    const int nb = 2 * HOSTCOPY_THREADS;
    char* p = nullptr;
    if (cudaMallocHost((void**)&p, nb * HOSTCOPY_BLOCK) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    cudaEvent_t* ev = new (std::nothrow) cudaEvent_t[nb];
    int made = 0;
    while (ev != nullptr && made < nb && cudaEventCreateWithFlags(&ev[made], cudaEventDisableTiming) == cudaSuccess) made++;
    if (made < nb) {
        cudaGetLastError();
        for (int i = 0; i < made; i++) cudaEventDestroy(ev[i]);
        delete[] ev;
        cudaFreeHost(p);
        return false;
    }
    r.pinned = p;
    r.ev = ev;
    return true;
}

static cudaError_t copy_plain(const CopySeg* segs, int n, bool toDevice, cudaStream_t st)
{
    for (int i = 0; i < n; i++) {
        const cudaError_t e = toDevice
                                  ? cudaMemcpyAsync(segs[i].dev, segs[i].host, segs[i].bytes, cudaMemcpyHostToDevice, st)
                                  : cudaMemcpyAsync(segs[i].host, segs[i].dev, segs[i].bytes, cudaMemcpyDeviceToHost, st);
        if (e != cudaSuccess) return e;
    }
    return toDevice ? cudaSuccess : cudaStreamSynchronize(st);
}

namespace {
struct Job {
    const CopySeg* segs;
    int n;
    bool toDevice;
    cudaStream_t st;
    int dev;
    char* pinned;
    cudaEvent_t* ev;
    std::atomic<size_t> next{0};
    std::atomic<int> err{0};

    bool block(size_t k, char** h, char** d, size_t* bytes) const
    {
        for (int i = 0; i < n; i++) {
            const size_t nb = (segs[i].bytes + HOSTCOPY_BLOCK - 1) / HOSTCOPY_BLOCK;
            if (k < nb) {
                const size_t off = k * HOSTCOPY_BLOCK;
                *h = (char*)segs[i].host + off;
                *d = (char*)segs[i].dev + off;
                *bytes = std::min(HOSTCOPY_BLOCK, segs[i].bytes - off);
                return true;
            }
            k -= nb;
        }
        return false;
    }
    bool ok(cudaError_t e)
    {
        if (e == cudaSuccess) return true;
        int none = 0;
        err.compare_exchange_strong(none, (int)e);
        return false;
    }
    // thread t: its two blocks in turn
    void work(int t)
    {
        if (!ok(cudaSetDevice(dev))) return;
        char* slot[2] = {pinned + (2 * t) * HOSTCOPY_BLOCK, pinned + (2 * t + 1) * HOSTCOPY_BLOCK};
        cudaEvent_t* e = ev + 2 * t;
        char *h, *d;
        size_t bytes;
        if (toDevice) {
            for (int s = 0; err.load() == 0 && block(next.fetch_add(1), &h, &d, &bytes); s ^= 1) {
                if (!ok(cudaEventSynchronize(e[s]))) return;     // the slot's last transfer has read it
                memcpy(slot[s], h, bytes);
                if (!ok(cudaMemcpyAsync(d, slot[s], bytes, cudaMemcpyHostToDevice, st))) return;
                if (!ok(cudaEventRecord(e[s], st))) return;
            }
            return;
        }
        char* hp[2] = {nullptr, nullptr};                        // where the block in flight goes
        size_t nb[2] = {0, 0};
        for (int s = 0;; s ^= 1) {
            if (hp[s] != nullptr) {
                if (!ok(cudaEventSynchronize(e[s]))) return;
                memcpy(hp[s], slot[s], nb[s]);
                hp[s] = nullptr;
            }
            if (err.load() == 0 && block(next.fetch_add(1), &h, &d, &bytes)) {
                if (!ok(cudaMemcpyAsync(slot[s], d, bytes, cudaMemcpyDeviceToHost, st))) return;
                if (!ok(cudaEventRecord(e[s], st))) return;
                hp[s] = h;
                nb[s] = bytes;
            } else if (hp[s ^ 1] == nullptr) {
                return;
            }
        }
    }
};
}  // namespace

cudaError_t copy_segments(HostRing& ring, int dev, const CopySeg* segs, int n, bool toDevice, cudaStream_t st)
{
    size_t bytes = 0, total = 0;
    bool ours = true;
    for (int i = 0; i < n; i++) {
        bytes += segs[i].bytes;
        total += (segs[i].bytes + HOSTCOPY_BLOCK - 1) / HOSTCOPY_BLOCK;
        // pinned and managed arrays transfer directly; what the driver refuses it refuses
        ours = ours && pageable(segs[i].host);
        // segments that share host memory land in their order
        for (int j = 0; j < i; j++)
            ours = ours && ((const char*)segs[i].host >= (const char*)segs[j].host + segs[j].bytes ||
                                  (const char*)segs[j].host >= (const char*)segs[i].host + segs[i].bytes);
    }
    if (!ours || !ring_ready(ring)) return copy_plain(segs, n, toDevice, st);

    Job job;
    job.segs = segs;
    job.n = n;
    job.toDevice = toDevice;
    job.st = st;
    job.dev = dev;
    job.pinned = ring.pinned;
    job.ev = ring.ev;
    int nt = 1;
    if (bytes >= HOSTCOPY_THREADED)
        nt = (int)std::min<size_t>(std::min((unsigned)HOSTCOPY_THREADS, std::max(1u, std::thread::hardware_concurrency())),
                                   (total + 1) / 2);
    std::thread th[HOSTCOPY_THREADS];
    int made = 0;
    try {
        for (; made < nt - 1; made++) th[made] = std::thread([&job, made]() { job.work(made + 1); });
    } catch (const std::exception&) {
        // no thread or no memory for one: the threads that did start, and this one, take all blocks
    }
    job.work(0);
    for (int i = 0; i < made; i++) th[i].join();
    return (cudaError_t)job.err.load();
}

}  // namespace srwg
