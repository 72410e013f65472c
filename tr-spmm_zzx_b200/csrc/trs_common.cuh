// Shared helpers for libtrspmm's translation units (sm_100a only).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>
#include <exception>
#include <new>

#include "trspmm.h"

// An error that a call returns does not stay the thread's last one: the check behind a later launch would return it again.
#define TRS_CUDA(expr)                                     \
    do {                                                   \
        cudaError_t _e = (expr);                           \
        if (_e != cudaSuccess) {                           \
            (void)cudaGetLastError();                      \
            return (int)_e;                                \
        }                                                  \
    } while (0)

#define TRS_LAUNCH_CHECK()                                 \
    do {                                                   \
        cudaError_t _e = cudaGetLastError();               \
        if (_e != cudaSuccess) return (int)_e;             \
    } while (0)

// Ends a function-try-block of a C entry: no C++ exception crosses it.
#define TRS_CATCH                                                                     \
    catch (const std::bad_alloc&) { return (int)cudaErrorMemoryAllocation; }          \
    catch (const std::exception&) { return (int)cudaErrorOperatingSystem; }

namespace trs {

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline long long ceil_div64(long long a, long long b) { return (a + b - 1) / b; }

// Caller-owned device memory handed to a call that would otherwise allocate: blocks are cut off
// the front (256-byte aligned); a block given back is kept on a free list and handed out again
// to the next request it fits, which is what keeps the footprint of a pass with many temporaries
// near its peak instead of its sum.  Not thread-safe: one arena serves one call at a time.
struct Arena {
    unsigned char* base = nullptr;
    size_t cap = 0, used = 0, high = 0;
    struct Free { unsigned char* p; size_t bytes; };
    Free free_list[64];
    int n_free = 0;
    unsigned char* take(size_t bytes) {
        bytes = (bytes + 255) & ~(size_t)255;
        if (bytes == 0) bytes = 256;
        int best = -1;
        for (int i = 0; i < n_free; ++i)
            if (free_list[i].bytes >= bytes && (best < 0 || free_list[i].bytes < free_list[best].bytes)) best = i;
        if (best >= 0 && free_list[best].bytes <= bytes + bytes / 4) {   // close fit: reuse whole
            unsigned char* p = free_list[best].p;
            free_list[best] = free_list[--n_free];
            return p;
        }
        if (used + bytes > cap) return nullptr;
        unsigned char* p = base + used;
        used += bytes;
        if (used > high) high = used;
        return p;
    }
    void give_back(void* p, size_t bytes) {
        bytes = (bytes + 255) & ~(size_t)255;
        if (bytes == 0) bytes = 256;
        if ((unsigned char*)p + bytes == base + used) { used -= bytes; return; }   // last block: shrink
        if (n_free < 64) free_list[n_free++] = Free{(unsigned char*)p, bytes};
    }
};

// Device memory from the library's stream-ordered pool (one per device, trs_api.cu).  A cudaMalloc /
// cudaFree pair costs 80 - 400 us here and stops the device; the pool gives memory that an earlier call
// freed back in about a microsecond.  It keeps at most kPoolKeepBytes between calls (trs_pool_trim returns that
// too), may be used from any thread, and hands memory freed on one stream to another only after the
// free has been reached on the first.
constexpr size_t kPoolKeepBytes = (size_t)4 << 30;
int pool_alloc(void** p, size_t bytes, cudaStream_t st);
void pool_free(void* p, cudaStream_t st);

// Temporaries of one call: blocks cut out of the caller's arena, or out of chunks from the pool.
struct TempSpace {
    Arena* arena = nullptr;
    cudaStream_t st = nullptr;
    size_t chunk_bytes = (size_t)16 << 20;
    static constexpr int kMaxChunks = 32;
    Arena chunk[kMaxChunks];
    int n_chunks = 0;
    int take(size_t bytes, void** out) {
        *out = nullptr;
        if (arena) { *out = arena->take(bytes); return *out ? 0 : TRS_E_WORKSPACE; }
        for (int i = n_chunks; i-- > 0;)
            if ((*out = chunk[i].take(bytes))) return 0;
        if (n_chunks == kMaxChunks) return (int)cudaErrorMemoryAllocation;
        Arena& c = chunk[n_chunks];
        c = Arena();
        c.cap = (bytes > chunk_bytes ? bytes : chunk_bytes) + 256;
        const int rc = pool_alloc((void**)&c.base, c.cap, st);
        if (rc) return rc;
        ++n_chunks;
        *out = c.take(bytes);
        return *out ? 0 : (int)cudaErrorMemoryAllocation;
    }
    template <class T>
    int get(size_t n, T** out) {
        void* d;
        const int rc = take((n ? n : 1) * sizeof(T), &d);
        *out = (T*)d;
        return rc;
    }
    // gives a block back early, so that later requests can use it
    template <class T>
    void drop(T* p, size_t n) {
        const size_t bytes = (n ? n : 1) * sizeof(T);
        if (arena) { arena->give_back(p, bytes); return; }
        for (int i = 0; i < n_chunks; ++i)
            if ((unsigned char*)p >= chunk[i].base && (unsigned char*)p < chunk[i].base + chunk[i].cap) chunk[i].give_back(p, bytes);
    }
    ~TempSpace() {
        for (int i = 0; i < n_chunks; ++i) pool_free(chunk[i].base, st);
    }
};

// Simple owning device buffer for plan-lifetime index arrays; with an arena the memory is the
// caller's and release() only forgets it.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    bool owned = true;
    int alloc(size_t count) { return alloc_from(nullptr, count); }
    int alloc_from(Arena* arena, size_t count) {
        n = count;
        if (count == 0) { p = nullptr; return 0; }
        if (arena) {
            p = (T*)arena->take(count * sizeof(T));
            owned = false;
            return p ? 0 : TRS_E_WORKSPACE;
        }
        owned = true;
        TRS_CUDA(cudaMalloc((void**)&p, count * sizeof(T)));
        return 0;
    }
    void release() {
        if (p && owned) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// 16-byte asynchronous global->shared copy; src_bytes = 0 writes zeros instead.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}
template <int OFF>
__device__ __forceinline__ void cp_async16_at(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0+%2], [%1], 16;\n" ::"r"(dst), "l"(src), "n"(OFF));
}
template <int OFF>
__device__ __forceinline__ void ldmatrix_x4_trans_at(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                                     uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4+%5];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr), "n"(OFF));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// A kernel launched behind another one of the same call (`behind`) is brought onto the SMs as that one's CTAs leave them; it
// waits for its end before it touches anything that it wrote.  At least one thread has to wait: a later kernel waits only
// for this one.  (Letting it come earlier, when the first one's CTAs have all started, gained nothing more, and the
// instruction for that cost short items of the product 5 %: R-MAT 20, F = 13 216 -> 227 us.)
__device__ __forceinline__ void wait_for_kernel_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
int launch_behind(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool behind, Args... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = behind ? 1 : 0;
    TRS_CUDA(cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
    return TRS_OK;
}
// A launch whose error is its own: cudaGetLastError behind one also returns what an earlier call left with the thread.
template <class... Params, class... Args>
int launch(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    return launch_behind(kernel, grid, threads, smem, st, false, args...);
}

// More than 48 KB of dynamic shared memory for a kernel, and with `carveout` as much of an SM's memory as can be for it; once per device
// and kernel (`done`: the attributes belong to the device's copy of the kernel).
template <class Kernel>
int allow_smem(Kernel kernel, int smem, bool carveout, std::atomic<unsigned long long>& done) {
    if (smem <= 48 * 1024 && !carveout) return TRS_OK;
    int dev = 0;
    TRS_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (dev < 64 && (done.load(std::memory_order_relaxed) & bit)) return TRS_OK;
    if (smem > 48 * 1024) TRS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (carveout) TRS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (dev < 64) done.fetch_or(bit, std::memory_order_relaxed);
    return TRS_OK;
}

// D(16x8,f32) += A(16x16 with 2:4 sparsity, stored 16x8 f16) * B(16x8 f16).
// `meta`: bits 4c..4c+3 = the two kept positions (p0 | p1<<2, p0<p1) of 4-column chunk c for
// row lane/4; bits 16+4c.. the same for row lane/4+8.  All four lanes of a quad pass the same
// word, so the thread selector is immaterial.
__device__ __forceinline__ void mma_sp_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, uint32_t b1,
                                             uint32_t meta) {
    asm volatile(
        "mma.sp::ordered_metadata.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
        "{%0,%1,%2,%3}, {%4,%5}, {%6,%7}, {%0,%1,%2,%3}, %8, 0x0;\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0), "r"(b1), "r"(meta));
}

// D(16x8,f32) += A(16x16 f16) * B(16x8 f16)
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// trs_hostcopy.cu: pageable host memory <-> device, ordered after the work on `st`.  copy_to_host returns when
// the host memory is written, copy_to_device when it has been read (the copies are then queued on `st`).
struct HostSegment {
    void* host;
    void* dev;
    size_t bytes;
};
int copy_to_host(const HostSegment* seg, int n, cudaStream_t st);
int copy_to_device(const HostSegment* seg, int n, cudaStream_t st);
void release_host_ring();

// trs_spmm.cu: trs_spmm_plan_create for callers that know whether a width is to come that reads `first_ids` (49 to 64).
constexpr int kFirstIdsFrom = 49, kFirstIdsTo = 64;
int spmm_plan_create(const trs_format* dev_format, int m_rows, int k_cols, int window, int validate, bool first_ids, cudaStream_t st,
                     trs_spmm_plan** out);

// trs_spmm.cu: trs_spmm_run_windows for callers that cut one product into several runs.
struct SpmmHow {
    int width = 0;   // the product's own width where `F` is a slab of it: what goes by the width goes by that
    // Rows of B off 16-byte boundaries: copied to the workspace if the run pays for that, if all runs of the plan's windows
    // together do, or already there from a run of the second kind.
    enum Rows { FOR_THIS_RUN, FOR_ALL_RUNS, COPIED } rows = FOR_THIS_RUN;
};
int spmm_run(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, void* workspace, size_t workspace_bytes,
             cudaStream_t st, int w0, int w1, const SpmmHow& how);

// trs_pack.cu
int pack_tiles(const int* s_column, const float* s_value, const int8_t* s_pos, const int* s_offset,
               const int* tile_window, const int* tile_group, long long tiles, int window, int* s_tile_column,
               uint32_t* packed_a, uint32_t* packed_meta, cudaStream_t st);

}  // namespace trs
