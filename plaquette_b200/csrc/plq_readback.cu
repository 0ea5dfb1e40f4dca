// plq_readback.cu -- see plq_readback.h.
//
// The driver's copy into pageable memory runs one host thread over one staging
// buffer, 5 GB/s into freshly allocated pages: 27.5 ms for a 512^3 configuration,
// whose transfer takes 3.  Here a few threads each own a pinned buffer, take the
// next piece, wait for its transfer and copy it out, so that transfers, copies and
// the target's page faults overlap: 134 MB in 7 ms (10.6 the first time, when the
// buffers are made).  Smaller targets are as a rule pages the process has already,
// where the driver's copy makes 20 GB/s (16.8 MB: 0.85 ms, 1.4 with the threads);
// pieces of 4 MB were 1 ms faster and took 10 ms more the first time.
#include "plq_readback.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

namespace {

constexpr size_t kPiece = size_t(1) << 20;
constexpr int kWorkers = 8;
constexpr size_t kKept = 2;  // sets kept for later calls (8 MiB of pinned memory each) until a context ends

// A set of pinned buffers and their events, one a worker; used by one call at a time.
struct Staging {
    int device = 0;
    uint8_t *buffers = nullptr;
    cudaEvent_t landed[kWorkers] = {};
};

std::mutex g_mutex;
std::vector<Staging *> g_idle;

void destroy(Staging *s) {
    if (s->buffers) cudaFreeHost(s->buffers);
    for (cudaEvent_t e : s->landed)
        if (e) cudaEventDestroy(e);
    delete s;
}

Staging *acquire(int device) {
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        for (size_t k = 0; k < g_idle.size(); ++k)
            if (g_idle[k]->device == device) {
                Staging *s = g_idle[k];
                g_idle.erase(g_idle.begin() + (long)k);
                return s;
            }
    }
    Staging *s = new (std::nothrow) Staging();
    if (!s) return nullptr;
    s->device = device;
    bool ok = cudaHostAlloc((void **)&s->buffers, kPiece * kWorkers, cudaHostAllocPortable) == cudaSuccess;
    for (cudaEvent_t &e : s->landed)
        ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (ok) return s;
    (void)cudaGetLastError();
    destroy(s);
    return nullptr;
}

void give_back(Staging *s) {
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        if (g_idle.size() < kKept) {
            try {
                g_idle.push_back(s);
                return;
            } catch (const std::bad_alloc &) {
            }
        }
    }
    destroy(s);
}

}  // namespace

void plq_readback_release(int device) {
    for (;;) {
        Staging *s = nullptr;
        {
            std::lock_guard<std::mutex> lock(g_mutex);
            for (size_t k = 0; k < g_idle.size() && !s; ++k)
                if (g_idle[k]->device == device) {
                    s = g_idle[k];
                    g_idle.erase(g_idle.begin() + (long)k);
                }
        }
        if (!s) return;
        destroy(s);
    }
}

cudaError_t plq_readback(void *dst, const void *src, size_t bytes, int device, cudaStream_t stream) {
    cudaPointerAttributes attr;
    Staging *s = nullptr;
    if (bytes >= kReadbackStaged) {
        const cudaError_t e = cudaPointerGetAttributes(&attr, dst);
        if (e != cudaSuccess) (void)cudaGetLastError();
        if (e == cudaSuccess && attr.type == cudaMemoryTypeUnregistered) s = acquire(device);
    }
    if (!s) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
    const size_t pieces = (bytes + kPiece - 1) / kPiece;
    std::atomic<size_t> next{0};
    std::atomic<int> failure{(int)cudaSuccess};
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(device);
        uint8_t *buffer = s->buffers + (size_t)w * kPiece;
        while (e == cudaSuccess) {
            const size_t k = next.fetch_add(1);
            if (k >= pieces) break;
            const size_t n = std::min(kPiece, bytes - k * kPiece);
            e = cudaMemcpyAsync(buffer, static_cast<const uint8_t *>(src) + k * kPiece, n, cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaEventRecord(s->landed[w], stream);
            if (e == cudaSuccess) e = cudaEventSynchronize(s->landed[w]);
            if (e == cudaSuccess) std::memcpy(static_cast<uint8_t *>(dst) + k * kPiece, buffer, n);
        }
        if (e != cudaSuccess) {
            next.store(pieces);
            failure.store((int)e);
        }
    };
    std::thread threads[kWorkers];
    const unsigned hw = std::thread::hardware_concurrency();
    const int workers = (int)std::min<size_t>(pieces, std::min<unsigned>(kWorkers, hw ? hw : 1u));
    for (int w = 1; w < workers; ++w) {
        try {
            threads[w] = std::thread(work, w);
        } catch (const std::system_error &) {
            break;  // the threads there are take all the pieces
        }
    }
    work(0);
    for (std::thread &t : threads)
        if (t.joinable()) t.join();
    const cudaError_t e = (cudaError_t)failure.load();
    // (after a failure a transfer may still be on its way into a buffer)
    if (e != cudaSuccess) (void)cudaStreamSynchronize(stream);
    give_back(s);
    return e;
}
