// Host-buffer entry points of the C ABI: the reference's calling convention (CPU arrays in,
// CPU result out; mGCN_online.cpp:760-1138) on top of the device-resident plan API.
#include <string.h>

#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#include "trs_common.cuh"

using namespace trs;

extern "C" const char* trs_strerror(int code) {
    switch (code) {
        case TRS_OK: return "ok";
        case TRS_E_ARG: return "invalid argument (null pointer, non-positive size or unsupported value)";
        case TRS_E_WINDOW: return "window must be in 1..16 (and exactly 16 when dense TC blocks are present)";
        case TRS_E_OFFSETS: return "a prefix/offset array is not monotone or does not start at 0";
        case TRS_E_SHAPE: return "array lengths are inconsistent with each other";
        case TRS_E_COLUMN: return "a column id lies outside [-1, kOri)";
        case TRS_E_ROW: return "a row id lies outside [0, mOri)";
        case TRS_E_WORKSPACE: return "workspace missing or too small";
        case TRS_E_NOT_CANONICAL: return "CSR input is not canonical (columns must ascend without duplicates in a row)";
        case TRS_E_NO_DEVICE: return "no usable CUDA device (this library has no CPU fallback)";
        case TRS_E_LIMIT: return "size exceeds a fixed limit of this entry point";
        default: break;
    }
    if (code > 0) return cudaGetErrorString((cudaError_t)code);
    return "unknown error";
}

extern "C" int trs_version(void) { return 100; }

extern "C" int trs_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) return 0;
    return n;
}

namespace trs {

namespace {
constexpr int kPoolDevices = 64;
cudaMemPool_t g_pool[kPoolDevices] = {};
std::mutex g_pool_mutex;

int device_pool(cudaMemPool_t* out) {
    int dev = 0;
    TRS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kPoolDevices) return TRS_E_LIMIT;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    if (!g_pool[dev]) {
        cudaMemPoolProps props;
        memset(&props, 0, sizeof(props));
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        TRS_CUDA(cudaMemPoolCreate(&pool, &props));
        unsigned long long keep = kPoolKeepBytes;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        g_pool[dev] = pool;
    }
    *out = g_pool[dev];
    return TRS_OK;
}
}  // namespace

int pool_alloc(void** p, size_t bytes, cudaStream_t st) {
    *p = nullptr;
    cudaMemPool_t pool;
    const int rc = device_pool(&pool);
    if (rc) return rc;
    const cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    if (e != cudaSuccess) { *p = nullptr; cudaGetLastError(); }
    return (int)e;
}

void pool_free(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}

}  // namespace trs

// Returns to the driver what the library holds for later calls: the current device's pool, the pinned ring.
extern "C" int trs_pool_trim(void) {
    trs::release_host_ring();
    int dev = 0;
    TRS_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(trs::g_pool_mutex);
    if (dev >= 0 && dev < trs::kPoolDevices && trs::g_pool[dev]) TRS_CUDA(cudaMemPoolTrimTo(trs::g_pool[dev], 0));
    return TRS_OK;
}

namespace {

// Owns the device copies made for one host-format upload.  Arrays are first noted (put / raw), then get their
// places in one block from the pool and are filled in one go (commit).
struct Upload {
    struct Part { const void* host; size_t bytes; void** dev; };
    std::vector<Part> parts;
    std::vector<void*> blocks;
    cudaStream_t st = nullptr;
    int device = 0;
    ~Upload() {
        if (blocks.empty()) return;
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev != device) cudaSetDevice(device);
        cudaDeviceSynchronize();   // whatever still uses them, on any stream
        for (void* p : blocks) pool_free(p, nullptr);
        if (dev != device) cudaSetDevice(dev);
    }
    template <class T>
    int put(const T* host, size_t n, const T** dev) {
        *dev = nullptr;
        if (n == 0) return 0;
        if (!host) return TRS_E_ARG;
        parts.push_back(Part{host, n * sizeof(T), (void**)dev});
        return 0;
    }
    template <class T>
    void raw(size_t n, T** dev) {
        *dev = nullptr;
        if (n) parts.push_back(Part{nullptr, n * sizeof(T), (void**)dev});
    }
    int commit() {
        std::vector<Part> noted;   // forgotten whatever happens: their `dev` may live on a caller's stack
        noted.swap(parts);
        size_t total = 0;
        for (const Part& p : noted) total += (p.bytes + 255) & ~(size_t)255;
        if (total == 0) return 0;
        TRS_CUDA(cudaGetDevice(&device));
        void* block;
        int rc = pool_alloc(&block, total, st);
        if (rc) return rc;
        blocks.push_back(block);
        std::vector<HostSegment> seg;
        unsigned char* at = (unsigned char*)block;
        for (const Part& p : noted) {
            *p.dev = at;
            if (p.host) seg.push_back(HostSegment{(void*)p.host, at, p.bytes});
            at += (p.bytes + 255) & ~(size_t)255;
        }
        return copy_to_device(seg.data(), (int)seg.size(), st);
    }
    template <class T>
    int now(size_t n, T** dev) {   // one array by itself
        raw(n, dev);
        return commit();
    }
};

// A stream and an event for work beside the caller's, kept between calls: as many exist as were ever in use at once.
struct SideStream {
    cudaStream_t st = nullptr;
    cudaEvent_t ready = nullptr;
    int device = 0;
};
std::mutex g_side_mutex;
std::vector<SideStream> g_side;

int take_side(SideStream* s) {
    int device = 0;
    TRS_CUDA(cudaGetDevice(&device));
    {
        std::lock_guard<std::mutex> lock(g_side_mutex);
        for (size_t i = g_side.size(); i-- > 0;)
            if (g_side[i].device == device) {
                *s = g_side[i];
                g_side.erase(g_side.begin() + i);
                return TRS_OK;
            }
    }
    s->device = device;
    TRS_CUDA(cudaEventCreateWithFlags(&s->ready, cudaEventDisableTiming));
    TRS_CUDA(cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking));
    return TRS_OK;
}

// Makes a plan on a thread and a stream of its own, behind what `after` holds so far.
class PlanThread {
    std::thread t_;
    SideStream side_;
    int rc_ = TRS_OK;

public:
    int start(const trs_format& dev, int m_rows, int k_cols, int window, bool first_ids, cudaStream_t after, trs_spmm_plan** out) {
        const int rc = take_side(&side_);
        if (rc) return rc;
        TRS_CUDA(cudaEventRecord(side_.ready, after));
        TRS_CUDA(cudaStreamWaitEvent(side_.st, side_.ready, 0));
        try {
            t_ = std::thread([=] {
                const cudaError_t e = cudaSetDevice(side_.device);
                rc_ = e != cudaSuccess ? (int)e : spmm_plan_create(&dev, m_rows, k_cols, window, 1, first_ids, side_.st, out);
            });
        } catch (const std::system_error&) {   // no thread to be had: the caller makes the plan itself
        }
        return TRS_OK;
    }
    bool started() const { return t_.joinable(); }
    int join() {
        if (t_.joinable()) t_.join();
        return rc_;
    }
    ~PlanThread() {
        join();
        if (!side_.st) return;
        std::lock_guard<std::mutex> lock(g_side_mutex);
        g_side.push_back(side_);
    }
};

// Host-side checks that need no device (the reference's TORCH_CHECKs, mGCN_online.cpp:888-932)
// and that make the array lengths below trustworthy.
int host_lengths(const trs_format& h, size_t* tc_nnz, size_t* c_nnz, size_t* cs_nnz) {
    *tc_nnz = *c_nnz = *cs_nnz = 0;
    if (h.parts_t < 0 || h.blocks < 0 || h.parts_c < 0 || h.parts_c_short < 0 || h.num_windows < 0 || h.tiles < 0)
        return TRS_E_ARG;
    if (h.parts_t > 0) {
        if (!h.t_row_offset || !h.t_block_offset) return TRS_E_ARG;
        if (h.t_row_offset[0] != 0 || h.t_block_offset[0] != 0) return TRS_E_OFFSETS;
        if (h.t_row_offset[h.parts_t] != h.blocks) return TRS_E_SHAPE;
        if (h.t_block_offset[h.blocks] < 0) return TRS_E_OFFSETS;
        *tc_nnz = (size_t)h.t_block_offset[h.blocks];
    } else if (h.blocks != 0) return TRS_E_SHAPE;
    if (h.parts_c > 0) {
        if (!h.c_row_offset) return TRS_E_ARG;
        if (h.c_row_offset[0] != 0 || h.c_row_offset[h.parts_c] < 0) return TRS_E_OFFSETS;
        *c_nnz = (size_t)h.c_row_offset[h.parts_c];
    }
    if (h.parts_c_short > 0) {
        if (!h.cs_row_offset) return TRS_E_ARG;
        if (h.cs_row_offset[0] != 0 || h.cs_row_offset[h.parts_c_short] < 0) return TRS_E_OFFSETS;
        *cs_nnz = (size_t)h.cs_row_offset[h.parts_c_short];
    }
    if (h.num_windows > 0) {
        if (!h.s_window_tile_offset) return TRS_E_ARG;
        if (h.s_window_tile_offset[0] != 0) return TRS_E_OFFSETS;
        if (h.s_window_tile_offset[h.num_windows] != h.tiles) return TRS_E_SHAPE;
    } else if (h.tiles != 0) return TRS_E_SHAPE;
    return TRS_OK;
}

int upload_format(const trs_format& h, Upload& up, trs_format* d) {
    size_t tc_nnz, c_nnz, cs_nnz;
    int rc = host_lengths(h, &tc_nnz, &c_nnz, &cs_nnz);
    if (rc) return rc;
    *d = h;
    const bool tc = h.parts_t > 0;
    if ((rc = up.put(h.t_row_offset, tc ? (size_t)h.parts_t + 1 : 0, &d->t_row_offset))) return rc;
    if ((rc = up.put(h.t_block_offset, tc ? (size_t)h.blocks + 1 : 0, &d->t_block_offset))) return rc;
    if ((rc = up.put(h.t_column, tc ? (size_t)h.blocks * 8 : 0, &d->t_column))) return rc;
    if ((rc = up.put(h.t_value, tc ? tc_nnz : 0, &d->t_value))) return rc;
    if ((rc = up.put(h.t_window_row, tc ? (size_t)h.parts_t : 0, &d->t_window_row))) return rc;
    if ((rc = up.put(h.t_binary, tc ? (size_t)h.blocks * 2 : 0, &d->t_binary))) return rc;
    const bool c = h.parts_c > 0;
    if ((rc = up.put(h.c_row_offset, c ? (size_t)h.parts_c + 1 : 0, &d->c_row_offset))) return rc;
    if ((rc = up.put(h.c_row, c ? (size_t)h.parts_c : 0, &d->c_row))) return rc;
    if ((rc = up.put(h.c_column, c_nnz, &d->c_column))) return rc;
    if ((rc = up.put(h.c_value, c_nnz, &d->c_value))) return rc;
    const bool cs = h.parts_c_short > 0;
    if ((rc = up.put(h.cs_row_offset, cs ? (size_t)h.parts_c_short + 1 : 0, &d->cs_row_offset))) return rc;
    if ((rc = up.put(h.cs_row, cs ? (size_t)h.parts_c_short : 0, &d->cs_row))) return rc;
    if ((rc = up.put(h.cs_column, cs_nnz, &d->cs_column))) return rc;
    if ((rc = up.put(h.cs_value, cs_nnz, &d->cs_value))) return rc;
    const bool s = h.num_windows > 0;
    if ((rc = up.put(h.s_window_tile_offset, s ? (size_t)h.num_windows + 1 : 0, &d->s_window_tile_offset))) return rc;
    if ((rc = up.put(h.s_tile_column, (size_t)h.tiles * 16, &d->s_tile_column))) return rc;
    if ((rc = up.put(h.s_packed_a, (size_t)h.tiles * 64, &d->s_packed_a))) return rc;
    if ((rc = up.put(h.s_packed_meta, (size_t)h.tiles * 8, &d->s_packed_meta))) return rc;
    return TRS_OK;
}

struct EventPair {
    cudaEvent_t a = nullptr, b = nullptr;
    int init() {
        TRS_CUDA(cudaEventCreate(&a));
        TRS_CUDA(cudaEventCreate(&b));
        return 0;
    }
    ~EventPair() {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
    float ms() {
        float m = 0.f;
        cudaEventElapsedTime(&m, a, b);
        return m;
    }
};

}  // namespace

// Host-buffer handle.  Three streams (host->device, kernels, device->host) and two buffer slots
// let consecutive calls overlap: the input copy of call i+1 runs beside the kernels and the
// output copy of call i (PCIe is full duplex), and inside one call the result rows of a window
// chunk go back to the host while the next chunk is computed.
constexpr int kSlots = 2;
constexpr int kMaxChunks = 16;
constexpr int kSlabDim = 64;   // features per slab of the blocking call

struct ResidentSlot {
    trs_half* d_rhs = nullptr;
    void* d_out = nullptr;
    cudaEvent_t in_done = nullptr, k_done = nullptr, out_done = nullptr;
    cudaEvent_t chunk_done[kMaxChunks] = {};
};

struct trs_resident {
    Upload up;
    trs_format dev;
    trs_spmm_plan* plan = nullptr;
    ResidentSlot slot[kSlots];
    void* d_ws = nullptr;
    size_t ws_bytes = 0;
    int m_rows = 0, k_cols = 0, max_dim = 0, window = 0, num_windows = 0;
    cudaStream_t stream = nullptr;  // kernels
    cudaStream_t s_in = nullptr, s_out = nullptr;
    cudaEvent_t t_ev[6] = {};       // timing of the synchronous call
    std::vector<cudaEvent_t> slab_ev;   // before and after the kernels of each of its slabs
    unsigned long long seq = 0;     // calls submitted so far
    int pending_rc = TRS_OK;        // first error of a submitted call, reported by wait
};

namespace {

int slot_init(trs_resident* h, int i) {
    ResidentSlot& s = h->slot[i];
    if (s.d_rhs) return TRS_OK;
    h->up.raw<trs_half>((size_t)h->k_cols * h->max_dim, &s.d_rhs);
    h->up.raw<unsigned char>((size_t)h->m_rows * h->max_dim * sizeof(float), (unsigned char**)&s.d_out);
    const int rc = h->up.commit();
    if (rc) return rc;
    TRS_CUDA(cudaStreamSynchronize(h->up.st));   // the pool's memory is ordered after this stream only
    TRS_CUDA(cudaEventCreateWithFlags(&s.in_done, cudaEventDisableTiming));
    TRS_CUDA(cudaEventCreateWithFlags(&s.k_done, cudaEventDisableTiming));
    TRS_CUDA(cudaEventCreateWithFlags(&s.out_done, cudaEventDisableTiming));
    for (int c = 0; c < kMaxChunks; ++c) TRS_CUDA(cudaEventCreateWithFlags(&s.chunk_done[c], cudaEventDisableTiming));
    return TRS_OK;
}

int resident_finish_create(trs_resident* h, int mOri, int kOri, int window, int max_dimN) {
    h->m_rows = mOri; h->k_cols = kOri; h->max_dim = max_dimN; h->window = window;
    // (slabs of a wider product are 64 features wide)
    int rc = spmm_plan_create(&h->dev, mOri, kOri, window, 1, max_dimN >= kFirstIdsFrom, nullptr, &h->plan);
    if (!rc) rc = trs_spmm_workspace_bytes(h->plan, max_dimN, &h->ws_bytes);
    if (!rc) rc = h->up.now<unsigned char>(h->ws_bytes, (unsigned char**)&h->d_ws);
    if (!rc) rc = slot_init(h, 0);  // the second slot is allocated by the first overlapping submit
    if (rc) return rc;
    h->num_windows = trs_spmm_num_windows(h->plan);
    TRS_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
    TRS_CUDA(cudaStreamCreateWithFlags(&h->s_in, cudaStreamNonBlocking));
    TRS_CUDA(cudaStreamCreateWithFlags(&h->s_out, cudaStreamNonBlocking));
    for (int i = 0; i < 6; ++i) TRS_CUDA(cudaEventCreate(&h->t_ev[i]));
    return TRS_OK;
}

// How many window chunks one call's output copy is cut into: the copy of a chunk overlaps the
// kernels of the next one, so chunks only pay when the output is large.
int resident_chunks(const trs_resident* h, size_t out_bytes) {
    static const int forced = [] { const char* v = getenv("TRS_RESIDENT_CHUNKS"); return v ? atoi(v) : 0; }();
    int k = forced > 0 ? forced : (out_bytes >= ((size_t)32 << 20) ? 8 : 1);
    if (k > kMaxChunks) k = kMaxChunks;
    if (k > h->num_windows) k = h->num_windows > 0 ? h->num_windows : 1;
    return k;
}

int resident_drain(trs_resident* h) {
    cudaError_t e1 = cudaStreamSynchronize(h->s_in);
    cudaError_t e2 = cudaStreamSynchronize(h->stream);
    cudaError_t e3 = cudaStreamSynchronize(h->s_out);
    if (e1 != cudaSuccess) return (int)e1;
    if (e2 != cudaSuccess) return (int)e2;
    if (e3 != cudaSuccess) return (int)e3;
    return TRS_OK;
}

// Workspace for a width that needs more than max_dimN does (a padded copy of B): grown once, after the
// calls in flight have left the old one.
int resident_workspace(trs_resident* h, int dimN) {
    size_t need = 0;
    int rc = trs_spmm_workspace_bytes(h->plan, dimN, &need);
    if (rc || need <= h->ws_bytes) return rc;
    rc = resident_drain(h);
    if (rc) return rc;
    void* grown = nullptr;   // the old one stays with the handle until it is destroyed
    rc = h->up.now<unsigned char>(need, (unsigned char**)&grown);
    if (!rc) rc = (int)cudaStreamSynchronize(h->up.st);
    if (rc) return rc;
    h->d_ws = grown;
    h->ws_bytes = need;
    return TRS_OK;
}

// The blocking call in feature slabs: while the input copy of slab s + 1 runs, slab s is multiplied and copied
// back - the only overlap of the two directions that one call has.  A slab's rows are cut out of the host rows by 2-D
// copies, which wants page-locked memory (pageable rows go through the driver piece by piece: R-MAT 18, F = 256, 27 -> 36 ms) and
// pieces of whole 64 bytes: 128-byte pieces move at 51 GB/s (64-byte ones at 35 - 41, whole rows at 55), so slabs
// have 64 features, and widths that are no multiple of 32 lose more than they gain (R-MAT 18, F = 128 / 160 / 192 / 256 in
// fp32 3.74 / 4.66 / 5.55 / 7.38 -> 3.45 / 4.36 / 4.78 / 6.17 ms; F = 130 / 136 / 200 / 232 3.87 / 4.02 / 5.84 / 6.74 -> 4.51 /
// 4.37 / 6.21 / 6.90).
bool in_pieces(const void* host) {
    cudaPointerAttributes a;
    if (((uintptr_t)host & 63) != 0) return false;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeHost;
}
int resident_slabs(int dimN, size_t in_bytes, const void* in, const void* out) {
    const bool slabs = dimN >= 2 * kSlabDim && dimN % 32 == 0 && in_bytes >= ((size_t)8 << 20) && in_pieces(in) && in_pieces(out);
    return slabs ? dimN / kSlabDim : 1;
}

int resident_enqueue_slabs(trs_resident* h, const trs_half* rhs_host, void* out_host, int dimN, int out_dtype, int slabs, bool timed) {
    ResidentSlot& s = h->slot[h->seq % kSlots];
    int rc = slot_init(h, (int)(h->seq % kSlots));
    const int last_dim = dimN - kSlabDim * (slabs - 1);
    if (rc) return rc;
    const size_t elt = out_dtype == TRS_OUT_F16 ? 2 : 4;
    TRS_CUDA(cudaStreamWaitEvent(h->s_in, s.k_done, 0));
    TRS_CUDA(cudaStreamWaitEvent(h->stream, s.out_done, 0));
    while (timed && h->slab_ev.size() < 2 * (size_t)slabs) {
        cudaEvent_t e;
        TRS_CUDA(cudaEventCreate(&e));
        h->slab_ev.push_back(e);
    }
    if (timed) cudaEventRecord(h->t_ev[0], h->s_in);
    for (int i = 0; i < slabs; ++i) {
        const int d0 = i * kSlabDim, d = i + 1 < slabs ? kSlabDim : last_dim;
        trs_half* in = s.d_rhs + (size_t)h->k_cols * d0;
        unsigned char* out = (unsigned char*)s.d_out + (size_t)h->m_rows * d0 * elt;
        TRS_CUDA(cudaMemcpy2DAsync(in, d * sizeof(trs_half), rhs_host + d0, dimN * sizeof(trs_half), d * sizeof(trs_half),
                                   h->k_cols, cudaMemcpyHostToDevice, h->s_in));
        TRS_CUDA(cudaEventRecord(s.in_done, h->s_in));
        TRS_CUDA(cudaStreamWaitEvent(h->stream, s.in_done, 0));
        if (timed) cudaEventRecord(h->slab_ev[2 * i], h->stream);
        SpmmHow how;
        how.width = dimN;
        rc = spmm_run(h->plan, in, out, d, out_dtype, h->d_ws, h->ws_bytes, h->stream, 0, h->num_windows, how);
        if (rc) return rc;
        if (timed) cudaEventRecord(h->slab_ev[2 * i + 1], h->stream);
        TRS_CUDA(cudaEventRecord(s.chunk_done[0], h->stream));
        TRS_CUDA(cudaStreamWaitEvent(h->s_out, s.chunk_done[0], 0));
        if (timed && i == 0) cudaEventRecord(h->t_ev[4], h->s_out);
        TRS_CUDA(cudaMemcpy2DAsync((unsigned char*)out_host + d0 * elt, dimN * elt, out, d * elt, d * elt, h->m_rows,
                                   cudaMemcpyDeviceToHost, h->s_out));
    }
    if (timed) {
        cudaEventRecord(h->t_ev[1], h->s_in);
        cudaEventRecord(h->t_ev[5], h->s_out);
    }
    TRS_CUDA(cudaEventRecord(s.k_done, h->stream));
    TRS_CUDA(cudaEventRecord(s.out_done, h->s_out));
    ++h->seq;
    return TRS_OK;
}

// Enqueue one call on the three streams; returns without waiting.  `timed` records the six
// timing events of the synchronous entry.

int resident_enqueue(trs_resident* h, const trs_half* rhs_host, void* out_host, int dimN, int out_dtype, bool timed) {
    const int si = (int)(h->seq % kSlots);
    int rc = slot_init(h, si);
    if (!rc) rc = resident_workspace(h, dimN);
    if (rc) return rc;
    ResidentSlot& s = h->slot[si];
    const size_t elt = out_dtype == TRS_OUT_F16 ? 2 : 4;
    const size_t row_bytes = (size_t)dimN * elt;
    const size_t out_bytes = (size_t)h->m_rows * row_bytes;
    // input: the slot's B buffer is free once the kernels of the call two back are done
    TRS_CUDA(cudaStreamWaitEvent(h->s_in, s.k_done, 0));
    if (timed) cudaEventRecord(h->t_ev[0], h->s_in);
    TRS_CUDA(cudaMemcpyAsync(s.d_rhs, rhs_host, (size_t)h->k_cols * dimN * sizeof(trs_half), cudaMemcpyHostToDevice, h->s_in));
    if (timed) cudaEventRecord(h->t_ev[1], h->s_in);
    TRS_CUDA(cudaEventRecord(s.in_done, h->s_in));
    // kernels: need this call's B and the slot's C buffer drained by the call two back
    TRS_CUDA(cudaStreamWaitEvent(h->stream, s.in_done, 0));
    TRS_CUDA(cudaStreamWaitEvent(h->stream, s.out_done, 0));
    if (timed) cudaEventRecord(h->t_ev[2], h->stream);
    const int chunks = resident_chunks(h, out_bytes);
    for (int c = 0; c < chunks; ++c) {
        const int w0 = (int)((long long)h->num_windows * c / chunks);
        const int w1 = (int)((long long)h->num_windows * (c + 1) / chunks);
        if (w1 <= w0) continue;
        SpmmHow how;   // rows of B that need a copy get it once for all chunks
        how.rows = c == 0 ? SpmmHow::FOR_ALL_RUNS : SpmmHow::COPIED;
        rc = spmm_run(h->plan, s.d_rhs, s.d_out, dimN, out_dtype, h->d_ws, h->ws_bytes, h->stream, w0, w1, how);
        if (rc) return rc;
        TRS_CUDA(cudaEventRecord(s.chunk_done[c], h->stream));
        TRS_CUDA(cudaStreamWaitEvent(h->s_out, s.chunk_done[c], 0));
        if (timed && c == 0) cudaEventRecord(h->t_ev[4], h->s_out);
        const size_t r0 = (size_t)w0 * h->window;
        size_t r1 = (size_t)w1 * h->window;
        if (r1 > (size_t)h->m_rows) r1 = (size_t)h->m_rows;
        if (r1 > r0)
            TRS_CUDA(cudaMemcpyAsync((char*)out_host + r0 * row_bytes, (const char*)s.d_out + r0 * row_bytes,
                                     (r1 - r0) * row_bytes, cudaMemcpyDeviceToHost, h->s_out));
    }
    if (timed) cudaEventRecord(h->t_ev[3], h->stream);
    TRS_CUDA(cudaEventRecord(s.k_done, h->stream));
    if (timed) cudaEventRecord(h->t_ev[5], h->s_out);
    TRS_CUDA(cudaEventRecord(s.out_done, h->s_out));
    ++h->seq;
    return TRS_OK;
}

int resident_check_args(trs_resident* h, const trs_half* rhs_host, void* out_host, int dimN, int out_dtype) {
    if (!h || !rhs_host || !out_host || dimN <= 0 || dimN > h->max_dim) return TRS_E_ARG;
    if (out_dtype != TRS_OUT_F32 && out_dtype != TRS_OUT_F16) return TRS_E_ARG;
    return TRS_OK;
}

}  // namespace

extern "C" int trs_resident_create(const trs_format* host_format, int mOri, int kOri, int window, int max_dimN,
                                   trs_resident** out) try {
    if (!host_format || !out || max_dimN <= 0) return TRS_E_ARG;
    *out = nullptr;
    if (mOri <= 0 || kOri <= 0) return TRS_E_ARG;
    if (window <= 0 || window > 16) return TRS_E_WINDOW;
    if (trs_device_count() == 0) return TRS_E_NO_DEVICE;
    trs_resident* h = new trs_resident();
    int rc = upload_format(*host_format, h->up, &h->dev);
    if (!rc) rc = h->up.commit();
    if (!rc) rc = resident_finish_create(h, mOri, kOri, window, max_dimN);
    if (rc) { trs_resident_destroy(h); return rc; }
    *out = h;
    return TRS_OK;
} TRS_CATCH

extern "C" int trs_resident_create_device(const trs_format* dev_format, int mOri, int kOri, int window, int max_dimN,
                                          trs_resident** out) try {
    if (!dev_format || !out || max_dimN <= 0) return TRS_E_ARG;
    *out = nullptr;
    if (mOri <= 0 || kOri <= 0) return TRS_E_ARG;
    if (window <= 0 || window > 16) return TRS_E_WINDOW;
    if (trs_device_count() == 0) return TRS_E_NO_DEVICE;
    trs_resident* h = new trs_resident();
    h->dev = *dev_format;
    int rc = resident_finish_create(h, mOri, kOri, window, max_dimN);
    if (rc) { trs_resident_destroy(h); return rc; }
    *out = h;
    return TRS_OK;
} TRS_CATCH

extern "C" int trs_resident_destroy(trs_resident* h) {
    if (!h) return TRS_OK;
    if (h->stream) resident_drain(h);
    if (h->plan) trs_spmm_plan_destroy(h->plan);
    for (int i = 0; i < kSlots; ++i) {
        ResidentSlot& s = h->slot[i];
        if (s.in_done) cudaEventDestroy(s.in_done);
        if (s.k_done) cudaEventDestroy(s.k_done);
        if (s.out_done) cudaEventDestroy(s.out_done);
        for (int c = 0; c < kMaxChunks; ++c)
            if (s.chunk_done[c]) cudaEventDestroy(s.chunk_done[c]);
    }
    for (int i = 0; i < 6; ++i)
        if (h->t_ev[i]) cudaEventDestroy(h->t_ev[i]);
    for (cudaEvent_t e : h->slab_ev) cudaEventDestroy(e);
    if (h->stream) cudaStreamDestroy(h->stream);
    if (h->s_in) cudaStreamDestroy(h->s_in);
    if (h->s_out) cudaStreamDestroy(h->s_out);
    delete h;
    return TRS_OK;
}

extern "C" int trs_resident_forward(trs_resident* h, const trs_half* rhs_host, void* out_host, int dimN, int out_dtype,
                                    trs_timing* timing) try {
    int rc = resident_check_args(h, rhs_host, out_host, dimN, out_dtype);
    if (rc) return rc;
    if (timing) memset(timing, 0, sizeof(*timing));
    const int slabs = resident_slabs(dimN, (size_t)h->k_cols * dimN * sizeof(trs_half), rhs_host, out_host);
    rc = slabs > 1 ? resident_enqueue_slabs(h, rhs_host, out_host, dimN, out_dtype, slabs, timing != nullptr)
                   : resident_enqueue(h, rhs_host, out_host, dimN, out_dtype, timing != nullptr);
    const int drc = resident_drain(h);
    if (!rc) rc = drc;
    if (!rc && h->pending_rc) { rc = h->pending_rc; }
    h->pending_rc = TRS_OK;
    if (rc) return rc;
    if (timing) {
        cudaEventElapsedTime(&timing->h2d_ms, h->t_ev[0], h->t_ev[1]);
        if (slabs > 1) {   // the kernels of the slabs, without what they waited for
            for (int i = 0; i < slabs; ++i) {
                float ms = 0.f;
                cudaEventElapsedTime(&ms, h->slab_ev[2 * i], h->slab_ev[2 * i + 1]);
                timing->total_ms += ms;
            }
        } else {
            cudaEventElapsedTime(&timing->total_ms, h->t_ev[2], h->t_ev[3]);
        }
        cudaEventElapsedTime(&timing->d2h_ms, h->t_ev[4], h->t_ev[5]);
    }
    return TRS_OK;
} TRS_CATCH

extern "C" int trs_resident_submit(trs_resident* h, const trs_half* rhs_host, void* out_host, int dimN, int out_dtype) try {
    int rc = resident_check_args(h, rhs_host, out_host, dimN, out_dtype);
    if (rc) return rc;
    rc = resident_enqueue(h, rhs_host, out_host, dimN, out_dtype, false);
    if (rc && !h->pending_rc) h->pending_rc = rc;
    return rc;
} TRS_CATCH

extern "C" int trs_resident_wait(trs_resident* h) {
    if (!h) return TRS_E_ARG;
    int rc = resident_drain(h);
    if (!rc) rc = h->pending_rc;
    h->pending_rc = TRS_OK;
    return rc;
}

extern "C" int trs_spmm_forward_host(const trs_format* host_format, const trs_half* rhs_host, float* out_host, int dimN,
                                     int mOri, int kOri, int window, int epoches, trs_timing* timing) try {
    if (!host_format || !rhs_host || !out_host) return TRS_E_ARG;
    if (dimN <= 0 || mOri <= 0 || kOri <= 0 || epoches <= 0) return TRS_E_ARG;
    if (window <= 0 || window > 16) return TRS_E_WINDOW;
    if (trs_device_count() == 0) return TRS_E_NO_DEVICE;
    // everything in two blocks of the pool (inputs and result; the plan's own), on the thread's stream
    cudaStream_t st = cudaStreamPerThread;
    Upload up;
    up.st = st;
    trs_format dev;
    trs_half* d_rhs = nullptr;
    float* d_out = nullptr;
    int rc = upload_format(*host_format, up, &dev);
    if (rc) return rc;
    const size_t rhs_bytes = (size_t)kOri * dimN * sizeof(trs_half);
    up.raw((size_t)kOri * dimN, &d_rhs);
    up.raw((size_t)mOri * dimN, &d_out);
    if ((rc = up.commit())) return rc;
    struct PlanOwner {
        trs_spmm_plan* p = nullptr;
        ~PlanOwner() { trs_spmm_plan_destroy(p); }
    } plan;
    // the plan needs the format only: it is made (some twenty small kernels and two read-backs) while the dense operand goes up
    {
        PlanThread maker;
        const bool first_ids = dimN >= kFirstIdsFrom && dimN <= kFirstIdsTo;
        if (rhs_bytes >= ((size_t)2 << 20)) rc = maker.start(dev, mOri, kOri, window, first_ids, st, &plan.p);
        const HostSegment in{(void*)rhs_host, d_rhs, rhs_bytes};
        if (!rc) rc = copy_to_device(&in, 1, st);
        const int plan_rc = maker.started() ? maker.join() : (rc ? rc : spmm_plan_create(&dev, mOri, kOri, window, 1, first_ids, st, &plan.p));
        if (rc || plan_rc) return rc ? rc : plan_rc;
    }
    size_t ws_bytes = 0;
    unsigned char* ws = nullptr;
    if ((rc = trs_spmm_workspace_bytes(plan.p, dimN, &ws_bytes))) return rc;
    if ((rc = up.now(ws_bytes, &ws))) return rc;
    // one untimed run, then `epoches` timed ones (mGCNkernel_online.cu:1604-1687 warms up and
    // averages over epoches the same way); C is fully rewritten by every run
    EventPair ev;
    rc = ev.init();
    if (!rc) rc = trs_spmm_run(plan.p, d_rhs, d_out, dimN, TRS_OUT_F32, ws, ws_bytes, st);
    if (!rc) cudaEventRecord(ev.a, st);
    for (int i = 0; i < epoches && !rc; ++i) rc = trs_spmm_run(plan.p, d_rhs, d_out, dimN, TRS_OUT_F32, ws, ws_bytes, st);
    if (!rc) cudaEventRecord(ev.b, st);
    const HostSegment back{out_host, d_out, (size_t)mOri * dimN * sizeof(float)};
    if (!rc) rc = copy_to_host(&back, 1, st);
    if (!rc && timing) {
        memset(timing, 0, sizeof(*timing));
        timing->total_ms = ev.ms() / (float)epoches;
    }
    return rc;
} TRS_CATCH

extern "C" int trs_sptc_unpacked_forward_host(const int32_t* s_column, const float* s_value, const int8_t* s_pos,
                                              const int32_t* s_window, const int32_t* s_offsets, int groups,
                                              int num_windows, const trs_half* rhs_host, float* out_host, int window,
                                              int dimN, int mOri, int kOri, int epoches, trs_timing* timing) try {
    if (!rhs_host || !out_host || groups < 0) return TRS_E_ARG;
    if (dimN <= 0 || mOri <= 0 || kOri <= 0 || epoches <= 0) return TRS_E_ARG;
    if (window <= 0 || window > 16) return TRS_E_WINDOW;
    if (groups > 0 && (!s_column || !s_value || !s_pos)) return TRS_E_ARG;
    if (!s_offsets && !s_window && groups > 0) return TRS_E_ARG;
    if (trs_device_count() == 0) return TRS_E_NO_DEVICE;
    const int W = trs::ceil_div(mOri, window);
    // per-window group offsets: given, or derived from the per-group window ids (sorted)
    std::vector<int> off;
    if (s_offsets) {
        if (num_windows < 0) return TRS_E_ARG;
        off.assign(s_offsets, s_offsets + num_windows + 1);
        if (off[0] != 0) return TRS_E_OFFSETS;
        if (off[num_windows] != groups) return TRS_E_SHAPE;
        for (int w = 0; w < num_windows; ++w)
            if (off[w + 1] < off[w]) return TRS_E_OFFSETS;
    } else {
        num_windows = W;
        off.assign(W + 1, 0);
        for (int g = 0; g < groups; ++g) {
            const int w = s_window[g];
            if (w < 0 || w >= W) return TRS_E_ROW;
            if (g > 0 && s_window[g - 1] > w) return TRS_E_OFFSETS;
            off[w + 1]++;
        }
        for (int w = 0; w < W; ++w) off[w + 1] += off[w];
    }
    std::vector<int> tile_window, tile_group, tile_off(num_windows + 1, 0);
    for (int w = 0; w < num_windows; ++w) {  // mGCN_online.cpp:914-926
        for (int g = off[w]; g < off[w + 1]; g += 4) { tile_window.push_back(w); tile_group.push_back(g); }
        tile_off[w + 1] = (int)tile_window.size();
    }
    const int tiles = (int)tile_window.size();
    Upload up;
    up.st = cudaStreamPerThread;
    const int *d_col, *d_off, *d_tw, *d_tg; const float* d_val; const int8_t* d_pos;
    int rc;
    if ((rc = up.put(s_column, (size_t)groups * 4, &d_col))) return rc;
    if ((rc = up.put(s_value, (size_t)groups * window * 2, &d_val))) return rc;
    if ((rc = up.put(s_pos, (size_t)groups * window * 2, &d_pos))) return rc;
    if ((rc = up.put(off.data(), off.size(), &d_off))) return rc;
    if ((rc = up.put(tile_window.data(), tile_window.size(), &d_tw))) return rc;
    if ((rc = up.put(tile_group.data(), tile_group.size(), &d_tg))) return rc;
    int* d_tcol; uint32_t *d_pa, *d_pm;
    up.raw((size_t)tiles * 16, &d_tcol);
    up.raw((size_t)tiles * 64, &d_pa);
    up.raw((size_t)tiles * 8, &d_pm);
    if ((rc = up.commit())) return rc;
    if ((rc = trs::pack_tiles(d_col, d_val, d_pos, d_off, d_tw, d_tg, tiles, window, d_tcol, d_pa, d_pm, up.st))) return rc;
    TRS_CUDA(cudaStreamSynchronize(up.st));
    // download the packed tiles and go through the common host path (keeps one code path)
    std::vector<int> h_tcol((size_t)tiles * 16);
    std::vector<uint32_t> h_pa((size_t)tiles * 64), h_pm((size_t)tiles * 8);
    if (tiles) {
        TRS_CUDA(cudaMemcpy(h_tcol.data(), d_tcol, h_tcol.size() * 4, cudaMemcpyDeviceToHost));
        TRS_CUDA(cudaMemcpy(h_pa.data(), d_pa, h_pa.size() * 4, cudaMemcpyDeviceToHost));
        TRS_CUDA(cudaMemcpy(h_pm.data(), d_pm, h_pm.size() * 4, cudaMemcpyDeviceToHost));
    }
    trs_format f;
    memset(&f, 0, sizeof(f));
    f.s_window_tile_offset = tile_off.data();
    f.s_tile_column = h_tcol.data();
    f.s_packed_a = h_pa.data();
    f.s_packed_meta = h_pm.data();
    f.num_windows = num_windows;
    f.tiles = tiles;
    return trs_spmm_forward_host(&f, rhs_host, out_host, dimN, mOri, kOri, window, epoches, timing);
} TRS_CATCH
