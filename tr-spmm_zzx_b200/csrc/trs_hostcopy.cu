// Copies between pageable host memory and the device, for the entries that take and return plain host arrays
// (the reference's calling convention).
//
// What bounds such a copy is the host side: cudaMemcpy on pageable memory stages through one driver
// thread, which also takes the page faults of freshly allocated results - 33 MB came back at 2.4 GB/s, while
// the link does 55.  Here the staging is a ring of pinned chunks (kSlots * kChunk bytes, allocated on first
// use, freed by trs_pool_trim), the calling thread drives the copy engine, and a few worker threads move
// chunks between the ring and the caller's memory, page faults included.
#include <string.h>
#include <sys/mman.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "trs_common.cuh"

namespace trs {
namespace {

constexpr size_t kChunk = (size_t)1 << 20;
constexpr size_t kSmallChunk = (size_t)256 << 10, kRamp = (size_t)2 << 20;
constexpr int kSlots = 32;
constexpr int kMaxWorkers = 8;
constexpr size_t kStageFrom = (size_t)512 << 10;  // below, the driver's own path is as fast

struct Chunk {
    unsigned char* host;
    unsigned char* dev;
    size_t bytes;
};

inline void relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}

// Into the pinned ring: the copy engine reads the chunk next, the cores never do, so the stores bypass the caches.
inline void copy_out_of_cache(unsigned char* dst, const unsigned char* src, size_t bytes) {
    size_t i = 0;
#if defined(__SSE2__)
    for (; i + 64 <= bytes; i += 64) {   // dst is a chunk of the ring: aligned
        const __m128i a = _mm_loadu_si128((const __m128i*)(src + i)), b = _mm_loadu_si128((const __m128i*)(src + i + 16));
        const __m128i c = _mm_loadu_si128((const __m128i*)(src + i + 32)), d = _mm_loadu_si128((const __m128i*)(src + i + 48));
        _mm_stream_si128((__m128i*)(dst + i), a);
        _mm_stream_si128((__m128i*)(dst + i + 16), b);
        _mm_stream_si128((__m128i*)(dst + i + 32), c);
        _mm_stream_si128((__m128i*)(dst + i + 48), d);
    }
    _mm_sfence();
#endif
    if (i < bytes) memcpy(dst + i, src + i, bytes - i);
}

// Fresh result arrays are not backed by memory yet: 2 MB pages instead of 4 KB ones take a fifth of the faults' time
// (33 MB: 3.0 -> 1.9 ms).  Only whole 2 MB blocks inside the array; a hint, whatever it returns.
inline void ask_for_large_pages(const HostSegment& s) {
#if defined(MADV_HUGEPAGE)
    const uintptr_t big = (uintptr_t)2 << 20, a = ((uintptr_t)s.host + big - 1) & ~(big - 1), e = ((uintptr_t)s.host + s.bytes) & ~(big - 1);
    if (e > a) madvise((void*)a, e - a, MADV_HUGEPAGE);
#endif
}

// One operation runs at a time (`busy`); a second thread takes the driver's path instead of waiting.
struct Copier {
    std::mutex busy;
    unsigned char* ring = nullptr;
    cudaEvent_t ev[kSlots] = {};
    int ev_device = -1;
    bool in_flight[kSlots] = {};

    std::mutex m;
    std::condition_variable wake;
    int workers = 0;
    unsigned long long op = 0;

    // state of the running operation
    const Chunk* chunks = nullptr;
    std::atomic<int> n{0};
    bool to_host = false;
    std::atomic<int> next{0};      // next chunk to claim
    std::atomic<int> allowed{0};   // chunks the workers may touch: [0, allowed)
    std::atomic<int> active{0};    // workers inside the operation
    std::vector<std::atomic<int>> done;

    void work() {
        while (true) {
            const int i = next.fetch_add(1, std::memory_order_relaxed);
            if (i >= n.load(std::memory_order_relaxed)) return;
            for (int spins = 0; allowed.load(std::memory_order_acquire) <= i; ++spins) {
                if (spins < 4096) relax();
                else std::this_thread::yield();
            }
            const Chunk& c = chunks[i];
            unsigned char* slot = ring + (size_t)(i % kSlots) * kChunk;
            if (c.bytes) {
                if (to_host) memcpy(c.host, slot, c.bytes);
                else copy_out_of_cache(slot, c.host, c.bytes);
            }
            done[i].store(1, std::memory_order_release);
        }
    }
    void worker_main() {
        unsigned long long seen = 0;
        while (true) {
            {
                std::unique_lock<std::mutex> lock(m);
                wake.wait(lock, [&] { return op != seen; });
                seen = op;
                if (n == 0) continue;   // the operation is already over
                active.fetch_add(1, std::memory_order_relaxed);
            }
            work();
            active.fetch_sub(1, std::memory_order_release);
        }
    }
    static void wait_done(std::atomic<int>& f) {
        for (int spins = 0; !f.load(std::memory_order_acquire); ++spins) {
            if (spins < 4096) relax();
            else std::this_thread::yield();
        }
    }
    int prepare() {
        int dev = 0;
        TRS_CUDA(cudaGetDevice(&dev));
        if (ev_device != dev) {   // events belong to the device they were made on
            int rc = drain();
            if (rc) return rc;
            for (cudaEvent_t& e : ev) {
                if (e) cudaEventDestroy(e);
                e = nullptr;
            }
            for (cudaEvent_t& e : ev) TRS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            ev_device = dev;
        }
        if (!ring) TRS_CUDA(cudaHostAlloc((void**)&ring, kChunk * kSlots, cudaHostAllocPortable));
        if (workers == 0) {
            const int hw = (int)std::thread::hardware_concurrency();
            const int want = hw >= 4 ? (hw / 2 < kMaxWorkers ? hw / 2 : kMaxWorkers) : 1;
            try {
                for (; workers < want; ++workers) std::thread([this] { worker_main(); }).detach();
            } catch (const std::system_error&) {   // no more threads to be had: those that there are do the work
            }
        }
        return drain();
    }
    int drain() {   // copies to the device still reading the ring
        for (int i = 0; i < kSlots; ++i)
            if (in_flight[i]) {
                TRS_CUDA(cudaEventSynchronize(ev[i]));
                in_flight[i] = false;
            }
        return 0;
    }
    void start(const std::vector<Chunk>& list, bool down) {
        std::lock_guard<std::mutex> lock(m);
        chunks = list.data();
        to_host = down;
        if (done.size() < list.size()) done = std::vector<std::atomic<int>>(list.size());
        for (size_t i = 0; i < list.size(); ++i) done[i].store(0, std::memory_order_relaxed);
        next.store(0, std::memory_order_relaxed);
        allowed.store(0, std::memory_order_relaxed);
        n = (int)list.size();
        ++op;
        wake.notify_all();
    }
    // No worker is left inside the operation when this returns.
    void finish() {
        {
            std::lock_guard<std::mutex> lock(m);
            allowed.store(n.load(), std::memory_order_release);   // after an error: let waiting workers run out
            n = 0;
        }
        while (active.load(std::memory_order_acquire)) std::this_thread::yield();
    }
    int down(const std::vector<Chunk>& list, cudaStream_t st) {
        start(list, true);
        const int total = (int)list.size();
        cudaError_t e = cudaSuccess;
        // Chunks go out as slots come free, arrived ones go to the workers at once, and neither waits for the other: with the
        // next arrival held back until a slot was free the workers took turns, 48 MB in 2.46 ms instead of 1.25.
        for (int issued = 0, arrived = 0; arrived < total && e == cudaSuccess;) {
            if (issued < total && issued == arrived && issued >= kSlots) wait_done(done[issued - kSlots]);
            while (issued < total && e == cudaSuccess && (issued < kSlots || done[issued - kSlots].load(std::memory_order_acquire))) {
                const int s = issued % kSlots;
                e = cudaMemcpyAsync(ring + (size_t)s * kChunk, list[issued].dev, list[issued].bytes, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev[s], st);
                ++issued;
                if (arrived < issued - 4) break;   // look at the arrivals in between
            }
            if (e == cudaSuccess) e = cudaEventSynchronize(ev[arrived % kSlots]);
            if (e == cudaSuccess) allowed.store(++arrived, std::memory_order_release);
        }
        if (e != cudaSuccess) { abandon(); return (int)e; }
        for (int i = 0; i < total; ++i) wait_done(done[i]);
        finish();
        return 0;
    }
    int up(const std::vector<Chunk>& list, cudaStream_t st) {
        start(list, false);
        const int total = (int)list.size();
        cudaError_t e = cudaSuccess;
        allowed.store(total < kSlots ? total : kSlots, std::memory_order_release);
        for (int i = 0; i < total && e == cudaSuccess; ++i) {
            const int s = i % kSlots;
            wait_done(done[i]);
            e = cudaMemcpyAsync(list[i].dev, ring + (size_t)s * kChunk, list[i].bytes, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(ev[s], st);
            in_flight[s] = e == cudaSuccess;
            // the slot half a ring back is free for its next chunk when its copy is through
            const int j = i - kSlots / 2;
            if (e == cudaSuccess && j >= 0 && j + kSlots < total) {
                e = cudaEventSynchronize(ev[j % kSlots]);
                allowed.store(j + kSlots + 1, std::memory_order_release);
            }
        }
        if (e != cudaSuccess) { abandon(); return (int)e; }
        finish();
        return 0;
    }
    // After a CUDA error the workers may still hold chunks: they are let through (the chunks' memory is the
    // caller's until the call returns, the ring's content is worthless by then).
    void abandon() {
        cudaDeviceSynchronize();
        finish();
    }
};

Copier& copier() {
    static Copier* c = new Copier();   // never destroyed: detached workers wait on it
    return *c;
}

// Memory that the copy engine reads or writes directly, after the call has returned if nothing waits for it.
bool page_locked(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type != cudaMemoryTypeUnregistered;
}

int plain(const HostSegment* seg, int n, bool to_host, cudaStream_t st) {
    bool wait = to_host;
    for (int i = 0; i < n; ++i) {
        if (!seg[i].bytes) continue;
        if (to_host) TRS_CUDA(cudaMemcpyAsync(seg[i].host, seg[i].dev, seg[i].bytes, cudaMemcpyDeviceToHost, st));
        else TRS_CUDA(cudaMemcpyAsync(seg[i].dev, seg[i].host, seg[i].bytes, cudaMemcpyHostToDevice, st));
        wait = wait || page_locked(seg[i].host);
    }
    if (wait) TRS_CUDA(cudaStreamSynchronize(st));
    return 0;
}

int staged(const HostSegment* all, int n_all, bool to_host, cudaStream_t st) {
    // Page-locked arrays need no staging: the copy engine takes them directly (57 GB/s; through the ring host memory
    // is crossed three times and 36 - 38 GB/s are left).  Downloads wait for them at the end.
    std::vector<HostSegment> rest;
    bool direct = false;
    for (int i = 0; i < n_all; ++i) {
        if (all[i].bytes >= kStageFrom && page_locked(all[i].host)) {
            if (to_host) TRS_CUDA(cudaMemcpyAsync(all[i].host, all[i].dev, all[i].bytes, cudaMemcpyDeviceToHost, st));
            else TRS_CUDA(cudaMemcpyAsync(all[i].dev, all[i].host, all[i].bytes, cudaMemcpyHostToDevice, st));
            direct = true;
        } else {
            rest.push_back(all[i]);
        }
    }
    struct Wait {   // the host memory is the caller's again when this returns
        cudaStream_t st;
        bool on;
        ~Wait() { if (on) cudaStreamSynchronize(st); }
    } wait{st, direct};
    const HostSegment* seg = rest.data();
    const int n = (int)rest.size();
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += seg[i].bytes;
    Copier& c = copier();
    std::unique_lock<std::mutex> lock(c.busy, std::defer_lock);
    if (total < kStageFrom || !lock.try_lock()) return plain(seg, n, to_host, st);
    const int rc = c.prepare();
    if (rc) return rc;
    if (c.workers == 0) return plain(seg, n, to_host, st);
    if (to_host)
        for (int i = 0; i < n; ++i) ask_for_large_pages(seg[i]);
    // Chunks of 1 MiB, but small ones where nothing else runs beside them: at the start of an upload (the copy engine waits for
    // the first chunk to be filled) and at the end of a download (the call waits for the last one to be emptied); a
    // download also leaves its small arrays for the end.
    std::vector<HostSegment> order(seg, seg + n);
    if (to_host) std::stable_sort(order.begin(), order.end(), [](const HostSegment& x, const HostSegment& y) { return x.bytes > y.bytes; });
    std::vector<Chunk> list;
    list.reserve(total / kChunk + n + 2 * kRamp / kSmallChunk);
    size_t before = 0;
    for (const HostSegment& g : order)
        for (size_t o = 0; o < g.bytes;) {
            const size_t most = (to_host ? total - before <= kRamp : before < kRamp) ? kSmallChunk : kChunk;
            const size_t bytes = g.bytes - o < most ? g.bytes - o : most;
            list.push_back(Chunk{(unsigned char*)g.host + o, (unsigned char*)g.dev + o, bytes});
            o += bytes;
            before += bytes;
        }
    return to_host ? c.down(list, st) : c.up(list, st);
}

}  // namespace

int copy_to_host(const HostSegment* seg, int n, cudaStream_t st) { return staged(seg, n, true, st); }
int copy_to_device(const HostSegment* seg, int n, cudaStream_t st) { return staged(seg, n, false, st); }

void release_host_ring() {
    Copier& c = copier();
    std::unique_lock<std::mutex> lock(c.busy, std::try_to_lock);
    if (!lock.owns_lock() || !c.ring) return;
    c.drain();
    cudaFreeHost(c.ring);
    c.ring = nullptr;
}

}  // namespace trs

static int segments(int n, void* const* host, void* const* dev, const size_t* bytes, std::vector<trs::HostSegment>* seg) {
    if (n < 0 || (n > 0 && (!host || !dev || !bytes))) return TRS_E_ARG;
    for (int i = 0; i < n; ++i) {
        if (!bytes[i]) continue;
        if (!host[i] || !dev[i]) return TRS_E_ARG;
        seg->push_back(trs::HostSegment{host[i], dev[i], bytes[i]});
    }
    return TRS_OK;
}

extern "C" int trs_host_register(void* host, size_t bytes) {
    if (!host || !bytes) return TRS_E_ARG;
    const cudaError_t e = cudaHostRegister(host, bytes, cudaHostRegisterPortable);
    if (e != cudaSuccess) cudaGetLastError();
    return (int)e;
}

extern "C" int trs_host_unregister(void* host) {
    if (!host) return TRS_E_ARG;
    const cudaError_t e = cudaHostUnregister(host);
    if (e != cudaSuccess) cudaGetLastError();
    return (int)e;
}

extern "C" int trs_copy_to_host(int n, void* const* host, const void* const* dev, const size_t* bytes, void* stream) try {
    std::vector<trs::HostSegment> seg;
    const int rc = segments(n, host, (void* const*)dev, bytes, &seg);
    return rc ? rc : trs::copy_to_host(seg.data(), (int)seg.size(), (cudaStream_t)stream);
} TRS_CATCH

extern "C" int trs_copy_to_device(int n, const void* const* host, void* const* dev, const size_t* bytes, void* stream) try {
    std::vector<trs::HostSegment> seg;
    const int rc = segments(n, (void* const*)host, dev, bytes, &seg);
    return rc ? rc : trs::copy_to_device(seg.data(), (int)seg.size(), (cudaStream_t)stream);
} TRS_CATCH
