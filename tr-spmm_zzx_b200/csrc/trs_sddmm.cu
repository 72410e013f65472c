// SDDMM: out[e] = fp16( sum_k fp32(X[row(e),k]) * fp32(Y[col(e),k]) ) for every CSR entry e.
//
// The reference has no SDDMM operator; the definition is fixed by the benchmark
// configuration (X, Y dense fp16, fp32 accumulate, fp16 result in CSR order).
//
// Both kernels below contract on the tensor cores (mma m16n8k16, fp32 accumulate) over the feature
// dimension, which is contiguous in both operands, so fragments are filled by plain 16-byte pieces:
// lane (g, t) takes bytes [64 c + 16 t, +16) of its row for every 32-feature chunk c - the same feature
// positions on both sides, which is all the MMA needs (the order of k inside a chunk is free).
// Rows that do not start on 16-byte boundaries are copied to padded ones first.
#include <limits.h>
#include <stdlib.h>
#include <string.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <cub/cub.cuh>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <mutex>
#include <thread>
#include <vector>

#include "trs_common.cuh"

namespace trs {

// ----------------------------------------------------------------------------------------------
// Entry-parallel SDDMM (patterns used once)
// ----------------------------------------------------------------------------------------------
// Work is split by ENTRY, not by row, so power-law rows cost nothing extra.  Eight consecutive entries, of
// whatever rows, are one MMA: row g of A is the X row of entry g, column g of B its Y row, and the
// diagonal of the product is the result (lane 4 g + g / 2 holds it).  That wastes the other products but replaces
// conversions, FMAs and shuffles, which were 19 warp instructions per entry at K = 64, by 2 loads and 2 MMAs per
// 32 features and 8 entries; what is left is the gather of one Y row per entry through L2.
// Uniform 50 021 rows x 17 entries, K = 96: 112 -> 27 us with every step's loads behind the one before, 22 us with the next
// step's ids loaded ahead and no branch between the batches of a step.
//
// Inputs are not validated by a pass of their own on this entry (trs_sddmm_plan_create does that for
// planned patterns), so the kernel bounds what it dereferences: rows stop at the last one, and an
// entry whose column lies outside [0, n_cols) reads row 0 of Y and is written as NaN.
constexpr int kEntryWarps = 8;   // warps per CTA
// CTAs per SM, and batches of 8 entries whose loads the compiler may put side by side: narrow rows want warps, wide ones
// registers.  R-MAT 20, us, 5 CTAs x 4 batches against 4 x 2: K = 32 446 / 511, K = 64 579 / 619, K = 96 793 / 739, K = 128 1055 /
// 983, K = 256 3088 / 2217.
__host__ __device__ constexpr int entry_ctas(int kch) { return kch <= 2 ? 5 : 4; }
__host__ __device__ constexpr int entry_batches(int kch) { return kch <= 2 ? 4 : 2; }

// Largest r in [0, n) with a[r] <= x (a ascending, a[0] <= x), by the whole warp: 32 probes per round.
__device__ __forceinline__ int warp_find(const int* __restrict__ a, int n, int x, int lane) {
    int lo = 0, len = n;   // the answer is in [lo, lo + len)
    while (len > 1) {
        const int step = (len + 31) / 32;
        const int at = lo + lane * step;
        const unsigned le = __ballot_sync(0xffffffffu, lane * step < len && a[at] <= x);
        const int k = 31 - __clz(le | 1u);
        lo += k * step;
        len = min(step, len - k * step);
    }
    return lo;
}

// Results are fp16 values; callers that go on in fp32 (the gradient of fp32 edge weights) take them widened.
__device__ __forceinline__ void store_result(void* out, int f32, long long i, __half v) {
    if (f32) ((float*)out)[i] = __half2float(v);
    else ((__half*)out)[i] = v;
}

// The ends of the row pointers for the host, and a word that says that they are there (pinned memory).
__device__ __forceinline__ void publish_ends(const int* __restrict__ rowptr, int n_rows, int* ends) {
    ends[0] = rowptr[0];
    ends[1] = rowptr[n_rows];
    __threadfence_system();
    *(volatile int*)(ends + 2) = 1;
}

// KCH: 32-feature chunks per pass; FULL: one pass, all of it (otherwise K is looped over and its end tested)
template <int KCH, bool FULL>
__global__ void __launch_bounds__(32 * kEntryWarps, entry_ctas(KCH)) k_sddmm(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                            const __half* __restrict__ X, const __half* __restrict__ Y,
                                                            void* __restrict__ out, int out_f32, int n_rows, int n_cols, int K,
                                                            int ld, int* ends) {
    if (ends && blockIdx.x == 0 && threadIdx.x == 0) publish_ends(rowptr, n_rows, ends);
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int nnz = rowptr[0] == 0 ? rowptr[n_rows] : 0;   // anything else is an error the caller reports
    const int pieces = (K + 7) / 8, ld16 = ld / 8;
    // a warp's share of the entries, in chunks of 32 to 256
    const int per_warp = min(max((nnz / (int)(gridDim.x * kEntryWarps) + 31) & ~31, 32), 256);
    for (long long warp = (long long)blockIdx.x * kEntryWarps + (threadIdx.x >> 5);; warp += (long long)gridDim.x * kEntryWarps) {
        const long long first = warp * per_warp;
        if (first >= nnz) return;
        const int e_end = (int)min(first + per_warp, (long long)nnz);
        int row = warp_find(rowptr, n_rows, (int)first, lane);   // row of the chunk's first entry
        // columns and row ends of the next 32 entries are loaded while the present ones are multiplied
        auto load_col = [&](unsigned e0) { return col[min(e0 + lane, (unsigned)e_end - 1u)]; };
        auto load_bound = [&]() { return row + 1 + lane < n_rows ? rowptr[row + 1 + lane] : 0x7fffffff; };
        int c_next = load_col((unsigned)first), bound_next = load_bound();
        for (unsigned e0 = (unsigned)first; e0 < (unsigned)e_end; e0 += 32) {   // unsigned: may step past 2^31 - 1
            // columns and rows of 32 entries, one per lane
            const int e = (int)min(e0 + lane, (unsigned)e_end - 1u);
            const int bound = bound_next;
            int c = c_next;
            const bool bad = (unsigned)c >= (unsigned)n_cols;
            if (bad) c = 0;
            int r = 0;   // how many of the next 32 rows start at or before e
#pragma unroll
            for (int s = 16; s; s >>= 1)
                if (__shfl_sync(0xffffffffu, bound, r + s - 1) <= e) r += s;
            r += __shfl_sync(0xffffffffu, bound, 31) <= e ? 1 : 0;
            r += row;
            if (__any_sync(0xffffffffu, r - row > 31)) {   // many empty rows in between
                int lo = 0, hi = n_rows;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (rowptr[mid] <= e) lo = mid; else hi = mid;
                }
                r = lo;
            }
            row = __shfl_sync(0xffffffffu, r, 31);
            const unsigned bad_mask = __ballot_sync(0xffffffffu, bad);
            if (e0 + 32 < (unsigned)e_end) {
                c_next = load_col(e0 + 32);
                bound_next = load_bound();
            }
            // entries past the end repeat the last one and are not stored
#pragma unroll entry_batches(KCH)
            for (int b = 0; b < 4; ++b) {
                const uint4* x = (const uint4*)X + (size_t)__shfl_sync(0xffffffffu, r, 8 * b + g) * ld16 + t;
                const uint4* y = (const uint4*)Y + (size_t)__shfl_sync(0xffffffffu, c, 8 * b + g) * ld16 + t;
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                for (int p0 = 0; p0 < (FULL ? 1 : pieces); p0 += 4 * KCH) {
                    uint4 xv[KCH], yv[KCH];
#pragma unroll
                    for (int ch = 0; ch < KCH; ++ch) {
                        const bool in = FULL || p0 + 4 * ch + t < pieces;
                        xv[ch] = in ? __ldg(x + p0 + 4 * ch) : make_uint4(0, 0, 0, 0);
                        yv[ch] = in ? __ldg(y + p0 + 4 * ch) : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (int ch = 0; ch < KCH; ++ch) {
                        mma_16816(d, xv[ch].x, 0u, xv[ch].y, 0u, yv[ch].x, yv[ch].y);
                        mma_16816(d, xv[ch].z, 0u, xv[ch].w, 0u, yv[ch].z, yv[ch].w);
                    }
                }
                const int i = 8 * b + g;
                if (t == (g >> 1) && e0 + i < (unsigned)e_end) {
                    const float v = (g & 1) ? d[1] : d[0];
                    store_result(out, out_f32, e0 + i, (bad_mask >> i) & 1u ? __ushort_as_half((unsigned short)0x7e00) : __float2half_rn(v));
                }
            }
        }
    }
}

// The same product on rows of any alignment, a warp per entry, where there is no memory for copies of X and Y.
__global__ void __launch_bounds__(256) k_sddmm_plain(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                     const __half* __restrict__ X, const __half* __restrict__ Y,
                                                     void* __restrict__ out, int out_f32, int n_rows, int n_cols, int K, int* ends) {
    if (ends && blockIdx.x == 0 && threadIdx.x == 0) publish_ends(rowptr, n_rows, ends);
    const int lane = threadIdx.x & 31, nnz = rowptr[0] == 0 ? rowptr[n_rows] : 0;
    const long long step = (long long)gridDim.x * 8;
    for (long long e = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); e < nnz; e += step) {
        const int row = warp_find(rowptr, n_rows, (int)e, lane);
        const int c = col[e];
        const bool bad = (unsigned)c >= (unsigned)n_cols;
        const __half *x = X + (size_t)row * K, *y = Y + (size_t)(bad ? 0 : c) * K;
        float s = 0.f;
        for (int k = lane; k < K; k += 32) s = fmaf(__half2float(x[k]), __half2float(y[k]), s);
#pragma unroll
        for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane == 0) store_result(out, out_f32, e, bad ? __ushort_as_half((unsigned short)0x7e00) : __float2half_rn(s));
    }
}

// Rows of `K` halfs copied to rows of `ld` halfs (a multiple of 8, zero-filled), the `rows` of X and then those of Y: one thread
// per 16 bytes.  One launch for both: plan of 8000 uniform rows, K = 47 14.5 -> 12.2 us, 60000 clustered ones 31.1 -> 29.0.
__global__ void k_sddmm_pad(const __half* __restrict__ X, const __half* __restrict__ Y, long long rows, long long pieces, int K, int per_row,
                            __half* __restrict__ dst) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pieces) return;
    const long long r = i / per_row;
    const int k = (int)(i - r * per_row) * 8;
    const unsigned short* s = (const unsigned short*)(r < rows ? X + r * K : Y + (r - rows) * K) + k;
    unsigned short v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = k + j < K ? s[j] : (unsigned short)0;
    ((uint4*)dst)[i] = make_uint4(v[0] | (uint32_t)v[1] << 16, v[2] | (uint32_t)v[3] << 16, v[4] | (uint32_t)v[5] << 16,
                                  v[6] | (uint32_t)v[7] << 16);
}

__global__ void k_sddmm_ends(const int* __restrict__ rowptr, int n_rows, int* __restrict__ ends) {
    publish_ends(rowptr, n_rows, ends);
}

// ----------------------------------------------------------------------------------------------
// Planned, tensor-core SDDMM
// ----------------------------------------------------------------------------------------------
// With a plan over the pattern the work is done per (16-row window, column) PAIR: the distinct columns of a window,
// ascending, are cut into quads of 32 (four MMA blocks of 8).  A quad has a header, 32 column ids (unused slots of its last
// block repeat the first column) and the list of its entries in CSR order: (CSR index - first one of the window) << 9 |
// row << 5 | column.  That holds windows of up to 2^23 entries; a pattern with a larger one runs the entry-parallel kernel.
// The pattern must be canonical CSR (columns ascending and unique per row).
constexpr int kPosBits = 9;   // row (4) and column (5) of an entry inside its quad
struct __align__(16) SddmmQuad {
    int window;
    int first;           // CSR index of the window's first entry
    int entries_blocks;  // entries << 3 | blocks of 8 columns in use
    int list;            // first entry in the list
};

__device__ __forceinline__ int row_of_entry(const int* __restrict__ rowptr, int n_rows, long long e) {
    int lo = 0, hi = n_rows;  // largest r with rowptr[r] <= e
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if ((long long)rowptr[mid] <= e) lo = mid; else hi = mid;
    }
    return lo;
}

// err |= 8 for a decreasing row pointer: the lists place entries by them.
__global__ void ksp_rows(const int* __restrict__ rowptr, int n_rows, int* __restrict__ err) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n_rows && rowptr[r + 1] < rowptr[r]) atomicOr(err, 8);
}

// Also validates the pattern: err |= 1 for a column outside [0, n_cols), |= 2 for columns that are
// not strictly ascending inside a row (the plan's entry addressing relies on canonical CSR).
__global__ void ksp_keys(const int* __restrict__ rowptr, const int* __restrict__ col, int n_rows, int n_cols,
                         long long nnz, unsigned long long* __restrict__ key, int* __restrict__ ent,
                         int* __restrict__ err) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    const int r = row_of_entry(rowptr, n_rows, e);
    const int c = col[e];
    if (c < 0 || c >= n_cols) { atomicOr(err, 1); return; }
    if (e > (long long)rowptr[r] && col[e - 1] >= c) atomicOr(err, 2);
    key[e] = ((unsigned long long)(r >> 4) << 32) | (unsigned)col[e];
    ent[e] = (int)e;
}

__global__ void ksp_heads(const unsigned long long* __restrict__ key, long long nnz, int* __restrict__ head) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnz) return;
    head[i] = (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
}

// first_pair[w] = number of distinct (window, column) pairs in windows < w, for w in [0, W]
__global__ void ksp_window_pairs(const unsigned long long* __restrict__ key, const int* __restrict__ pair_idx,
                                 long long nnz, int total_pairs, int W, int* __restrict__ first_pair,
                                 int* __restrict__ quads_of, int* __restrict__ n_blocks) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > W) return;
    auto lower = [&](int win) -> int {  // pairs before the first sorted entry of window >= win
        long long lo = 0, hi = nnz;     // first i with key[i] >> 32 >= win
        while (lo < hi) {
            const long long mid = (lo + hi) >> 1;
            if ((int)(key[mid] >> 32) < win) lo = mid + 1; else hi = mid;
        }
        return lo < nnz ? pair_idx[lo] : total_pairs;
    };
    const int mine = lower(w);
    first_pair[w] = mine;
    if (w < W) {
        const int n = lower(w + 1) - mine;
        quads_of[w] = (n + 31) >> 5;
        if (n > 0) atomicAdd(n_blocks, (n + 7) >> 3);
    } else {
        quads_of[w] = 0;
    }
}

// Column ids, and where a quad's entries begin among the sorted ones (they are contiguous).
__global__ void ksp_columns(const unsigned long long* __restrict__ key, const int* __restrict__ pair_idx,
                            const int* __restrict__ head, const int* __restrict__ first_pair, const int* __restrict__ quad_off,
                            long long nnz, int* __restrict__ ids, int* __restrict__ begin) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nnz || !head[i]) return;
    const unsigned long long k = key[i];
    const int w = (int)(k >> 32);
    const int local = pair_idx[i] - first_pair[w];
    const size_t q = (size_t)quad_off[w] + (local >> 5);
    ids[q * 32 + (local & 31)] = (int)(unsigned)k;
    if ((local & 31) == 0) begin[q] = (int)i;
}

// CTAs per SM, by shared memory and registers (K = 64 with 8 CTAs of 64 registers spills: 85 against 81 us, clustered).  Single
// warps take longer to launch than CTAs of four (4096 rows, K = 256: 7.9 against 6.3 us).
constexpr int kRingClasses = 8, kRingWarps = 4;
__host__ __device__ constexpr int ring_ctas(int kch) { return kch == 1 ? 8 : kch == 2 ? 7 : kch <= 4 ? 5 : kch <= 6 ? 4 : 3; }
// What a quad costs a warp: overhead, blocks of 8 rows, entries to put in place, and the rows of X where a window begins (with
// the wait for them).
__host__ __device__ constexpr unsigned quad_cost(int blocks, int entries, bool new_window) {
    return 4 + 2 * blocks + 2 * ((entries + 31) / 32) + (new_window ? 8 : 0);
}
// One wave of warps takes equal shares of the quads, or by a table of first quads equal shares of their cost: hub windows
// have full quads, most windows of a power-law graph one that is nearly empty.  R-MAT 18, K = 32 / 64 / 128 / 256: equal numbers
// 101 / 127 / 187 / 354 us (SMs busy 73 % of the time), equal cost 82 / 104 / 155 / 322; weights of 4, 2, 1, 4 or of 2, 2, 2, 4 take 5
// to 10 % more, 16 for a window 4 %.  The table is another load to wait for, so it is used only where the largest share gets
// smaller by an eighth and warps have two quads or more (40000 clustered rows, K = 64, 6 quads a warp: 13.3 us without, 13.7 with;
// 4096 uniform rows, K = 256, 1.3 quads a warp: 6.2 and 7.2).
struct RingShares {
    int warps;                    // of a wave
    int offset;                   // of its table, where there is one
    unsigned worst, worst_cost;   // largest share of equal numbers, of equal cost
};
struct RingTables {
    RingShares of[kRingClasses];
    int total;
};
__device__ __forceinline__ int first_quad(const unsigned* __restrict__ cost_before, int n_quads, int i, int warps) {
    const unsigned long long want = (unsigned long long)cost_before[n_quads] * (unsigned)i / (unsigned)warps;
    int lo = 0, hi = n_quads;   // first quad with `want` or more before it
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cost_before[mid] < want) lo = mid + 1; else hi = mid;
    }
    return lo;
}
// A wave that gets less than two quads a warp has no table; without any such wave (fewer than 24 quads per SM) the costs are not
// summed either.
__host__ __device__ __forceinline__ bool may_have_table(int n_quads, int warps) { return n_quads / 2 >= warps; }
__global__ void ksp_shares(const unsigned* __restrict__ cost_before, int n_quads, RingTables s, int* __restrict__ starts,
                           unsigned* __restrict__ worst /* [kRingClasses][2] */) {
    const int c = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x, warps = s.of[c].warps;
    if (!may_have_table(n_quads, warps)) return;
    unsigned number = 0, cost = 0;
    if (i <= warps) {
        const int at = first_quad(cost_before, n_quads, i, warps);
        starts[s.of[c].offset + i] = at;
        if (i < warps) {
            const long long per = (n_quads + warps - 1) / warps, end = min((i + 1) * per, (long long)n_quads);
            number = cost_before[end] - cost_before[min(i * per, end)];
            cost = cost_before[first_quad(cost_before, n_quads, i + 1, warps)] - cost_before[at];
        }
    }
    number = __reduce_max_sync(0xffffffffu, number);
    cost = __reduce_max_sync(0xffffffffu, cost);
    if ((threadIdx.x & 31) != 0) return;
    atomicMax(worst + 2 * c, number);
    atomicMax(worst + 2 * c + 1, cost);
}

// One warp per quad: header, repeated columns, and the entries in CSR order, placed by row masks.
__global__ void ksp_quads(const unsigned long long* __restrict__ key, const int* __restrict__ ent, const int* __restrict__ pair_idx,
                          const int* __restrict__ first_pair, const int* __restrict__ begin, const int* __restrict__ rowptr,
                          int n_rows, int nnz, int n_quads, SddmmQuad* __restrict__ quads, int* __restrict__ ids,
                          unsigned* __restrict__ list, unsigned* __restrict__ cost, int* __restrict__ err) {
    __shared__ unsigned s_mask[8][16];
    __shared__ int s_before[8][16];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int q = blockIdx.x * 8 + wid;
    if (q >= n_quads) return;
    const int b = begin[q], e = q + 1 < n_quads ? begin[q + 1] : nnz;
    const int w = (int)(key[b] >> 32), pair0 = pair_idx[b];
    const int cols = pair_idx[e - 1] - pair0 + 1;
    const int e0 = rowptr[w * 16];
    if (lane < 16) s_mask[wid][lane] = 0u;
    __syncwarp();
    auto place = [&](int i, int& r, int& n) {
        const int x = ent[i];
        n = pair_idx[i] - pair0;
        r = 0;
        for (int k = 1; k < 16 && w * 16 + k < n_rows; ++k) r += rowptr[w * 16 + k] <= x;
    };
    for (int i = b + lane; i < e; i += 32) {
        int r, n;
        place(i, r, n);
        atomicOr(&s_mask[wid][r], 1u << n);
    }
    __syncwarp();
    int count = lane < 16 ? __popc(s_mask[wid][lane]) : 0, incl = count;
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane < 16) s_before[wid][lane] = incl - count;
    __syncwarp();
    for (int i = b + lane; i < e; i += 32) {
        int r, n;
        place(i, r, n);
        const int rel = ent[i] - e0;
        if (rel >= 1 << (32 - kPosBits)) atomicOr(err, 4);
        list[b + s_before[wid][r] + __popc(s_mask[wid][r] & ((1u << n) - 1u))] = ((unsigned)rel << kPosBits) | (unsigned)(r << 5 | n);
    }
    const int blocks = (cols + 7) / 8;
    if (lane >= cols && lane < blocks * 8) ids[(size_t)q * 32 + lane] = ids[(size_t)q * 32];
    if (lane == 0) {
        quads[q] = SddmmQuad{w, e0, (e - b) << 3 | blocks, b};
        if (cost) {
            cost[q] = quad_cost(blocks, e - b, pair0 == first_pair[w]);
            if (q + 1 == n_quads) cost[n_quads] = 0;
        }
    }
}

// One warp walks a contiguous range of quads, one block of 8 columns at a time: the window's X tile (16 x K) sits
// in registers as A fragments (the next window's is loaded while results are put in place: 5 % of the clustered pattern), the 8 gathered Y rows are the B fragments.  Column ids (one per lane) and
// headers come from memory two quads ahead, the Y rows kRowAhead blocks ahead as 16-byte cp.async copies into the
// warp's ring; a lane copies exactly the pieces it reads back, so no lane waits for another.  (The odd Y rows land with
// the two 64-byte halves of every 128 bytes swapped: chunk c at position c ^ 4.  A 16-byte access is served eight lanes
// at a time - two consecutive rows g with four chunks each - and the swap puts the two rows into different halves of the
// 128-byte bank line.)  The 16 x 32 products of a quad are rounded to fp16 into a small tile, and its list of
// entries - in CSR order, so that neighbours in the list are mostly neighbours in `out` - says which of them go where.
//
// What bounds it: instruction issue and the LSU pipe.  With a bitmap per block and four predicated 2-byte stores per
// lane a block took 99 instructions and, on a power-law pattern, 9 to 16 scattered store sectors one at a time;
// with lists it is about 35, and what is left is the L2 gather (38 us of the clustered pattern's 0.57 GB at K = 64).
constexpr int kRowAhead = 3, kRowStages = 4;
constexpr int kTilePitch = 80;    // bytes per row of the 16 x 32 fp16 tile: the quad's stores hit 32 different banks
constexpr int kListAhead = 3;     // entries of the list that a lane holds from the start of the quad

template <int KCH>
struct SddmmRing {
    static constexpr int ROWB = KCH * 64;                 // bytes of a Y row in the ring
    static constexpr int CPR = KCH * 4;                   // 16-byte chunks per row
    static constexpr bool SWAP = CPR % 8 == 0;            // rows of 64 (mod 128) bytes alternate halves by themselves
    static constexpr int STAGE = 8 * ROWB;
    static constexpr int WARP_SMEM = kRowStages * STAGE + 16 * kTilePitch;
    static constexpr int SMEM = kRingWarps * WARP_SMEM;
};
template <int N, int I = 0, class Fn>
__device__ __forceinline__ void sddmm_for(Fn&& fn) {
    if constexpr (I < N) {
        fn(std::integral_constant<int, I>());
        sddmm_for<N, I + 1>(fn);
    }
}

template <int OFFSET, int FROM>
__device__ __forceinline__ void cp_async16_to(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0+%2], [%1+%3], 16;\n" ::"r"(dst), "l"(src), "n"(OFFSET), "n"(FROM));
}

// TAIL: K is not a multiple of 32; the chunks past the end of a row are zero on both sides.
template <int KCH, bool TAIL, bool F32>
__global__ void __launch_bounds__(32 * kRingWarps, ring_ctas(KCH)) k_sddmm_tc_ring(
    const SddmmQuad* __restrict__ quads, const int* __restrict__ ids, const unsigned* __restrict__ list,
    const int* __restrict__ starts, int n_quads, int quads_per_warp, const __half* __restrict__ X, const __half* __restrict__ Y,
    void* __restrict__ out, int n_rows, int pieces, int ld16) {
    using R = SddmmRing<KCH>;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int warp = blockIdx.x * kRingWarps + wid;   // a table has an entry behind the last CTA's last warp
    const int q0 = starts ? starts[warp] : warp * quads_per_warp;
    const int nq = (starts ? starts[warp + 1] : min(q0 + quads_per_warp, n_quads)) - q0;
    if (nq <= 0) return;
    unsigned char* const ring = smem + wid * R::WARP_SMEM;
    unsigned char* const tile = ring + kRowStages * R::STAGE;
    const uint32_t rows0 = smem_u32(ring);
    const unsigned char* Xq = (const unsigned char*)(X + 8 * t);
    const unsigned char* Yq = (const unsigned char*)(Y + 8 * t);
    const uint32_t pitch = (uint32_t)ld16 * 16u;
    const uint32_t swap = R::SWAP ? (uint32_t)(g & 1) * 64u : 0u;
    const uint32_t row_at = rows0 + g * R::ROWB + t * 16;
    const uint32_t at_even = row_at + swap, at_odd = row_at + (swap ^ 64u);
    quads += q0;
    ids += (size_t)q0 * 32 + lane;

    auto load_ids = [&](int q) { return q < nq ? __ldg(ids + (size_t)q * 32) : 0; };
    auto load_head = [&](int q) {   // behind the last one: no blocks of the same window
        int4 h = __ldg((const int4*)(quads + min(q, nq - 1)));
        if (q >= nq) h.z = 0;
        return h;
    };
    auto issue_rows = [&](int c, auto stage) {
        constexpr int S = decltype(stage)::value * R::STAGE;
        const unsigned char* src = Yq + (unsigned long long)(uint32_t)c * pitch;
        sddmm_for<KCH>([&](auto ii) {
            constexpr int i = decltype(ii)::value;
            const uint32_t at = R::SWAP ? ((i & 1) ? at_odd : at_even) : row_at;
            constexpr int off = S + (R::SWAP ? (i / 2) * 128 : i * 64);
            if constexpr (!TAIL) cp_async16_to<off, i * 64>(at, src);
            else cp_async16(at + off, 4 * i + t < pieces ? src + i * 64 : src, 4 * i + t < pieces ? 16 : 0);
        });
    };
    // blocks of 8 columns in a quad; z: entries << 3 | blocks
    auto blocks_of = [](const int4& h) { return h.z & 7; };

    int id = load_ids(0), id1 = load_ids(1);
    int4 head = load_head(0), head1 = load_head(1);
    sddmm_for<kRowAhead>([&](auto u) {
        constexpr int b = decltype(u)::value;
        if (b < blocks_of(head)) issue_rows(__shfl_sync(0xffffffffu, id, 8 * b + g), u);
        cp_async_commit();
    });
    int cur_w = -1;
    uint4 xa[KCH], xb[KCH];
#pragma unroll
    for (int c = 0; c < KCH; ++c) xa[c] = xb[c] = make_uint4(0, 0, 0, 0);

    auto load_x = [&](int w) {
        cur_w = w;
        const unsigned char* ra = Xq + (size_t)min(w * 16 + g, n_rows - 1) * pitch;
        const unsigned char* rb = Xq + (size_t)min(w * 16 + g + 8, n_rows - 1) * pitch;
#pragma unroll
        for (int ch = 0; ch < KCH; ++ch) {
            if (!TAIL || 4 * ch + t < pieces) {
                xa[ch] = __ldg((const uint4*)(ra + ch * 64));
                xb[ch] = __ldg((const uint4*)(rb + ch * 64));
            }
        }
    };
    load_x(head.x);

    for (int q = 0; q < nq; ++q) {
        const int id2 = load_ids(q + 2);
        const int4 head2 = load_head(q + 2);
        const int nb = blocks_of(head), nb1 = blocks_of(head1), n_ent = head.z >> 3;
        const unsigned* entries = list + (unsigned)head.w;
        unsigned ent[kListAhead];
#pragma unroll
        for (int i = 0; i < kListAhead; ++i) ent[i] = 32 * i + lane < n_ent ? __ldg(entries + 32 * i + lane) : 0u;
        // group 4 q + b carries the rows of block b; all but the newest kRowAhead - 1 groups are complete
        const bool full = nb == 4 && nb1 == 4;
        auto blocks = [&](auto all) {
        sddmm_for<4>([&](auto uu) {
            constexpr bool ALL = decltype(all)::value;
            constexpr int b = decltype(uu)::value, bn = (b + kRowAhead) & 3;
            cp_async_wait<kRowAhead - 1>();
            if constexpr (b + kRowAhead < 4) {
                if (ALL || bn < nb) issue_rows(__shfl_sync(0xffffffffu, id, 8 * bn + g), std::integral_constant<int, bn>());
            } else {
                if (ALL || bn < nb1) issue_rows(__shfl_sync(0xffffffffu, id1, 8 * bn + g), std::integral_constant<int, bn>());
            }
            cp_async_commit();
            if (ALL || b < nb) {
                float d[4] = {0.f, 0.f, 0.f, 0.f}, d2[4] = {0.f, 0.f, 0.f, 0.f};   // two chains
                sddmm_for<KCH>([&](auto ii) {
                    constexpr int i = decltype(ii)::value;
                    constexpr int off = b * R::STAGE + (R::SWAP ? (i / 2) * 128 : i * 64);
                    uint4 y;
                    const uint32_t at = R::SWAP ? ((i & 1) ? at_odd : at_even) : row_at;
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w) : "r"(at), "n"(off));
                    mma_16816(d, xa[i].x, xb[i].x, xa[i].y, xb[i].y, y.x, y.y);
                    mma_16816(d2, xa[i].z, xb[i].z, xa[i].w, xb[i].w, y.z, y.w);
                });
#pragma unroll
                for (int i = 0; i < 4; ++i) d[i] += d2[i];
                *(__half2*)(tile + g * kTilePitch + b * 16 + t * 4) = __floats2half2_rn(d[0], d[1]);
                *(__half2*)(tile + (g + 8) * kTilePitch + b * 16 + t * 4) = __floats2half2_rn(d[2], d[3]);
            }
        });
        };
        if (full) blocks(std::true_type()); else blocks(std::false_type());
        if (head1.x != cur_w) load_x(head1.x);   // warp-uniform; under way while the results are put in place
        __syncwarp();
        const long long o = (unsigned)head.y;
        auto put = [&](unsigned e) {
            const unsigned pos = e & ((1u << kPosBits) - 1u);
            store_result(out, F32, o + (e >> kPosBits), *(const __half*)(tile + (pos >> 5) * kTilePitch + (pos & 31u) * 2));
        };
#pragma unroll
        for (int i = 0; i < kListAhead; ++i)
            if (32 * i + lane < n_ent) put(ent[i]);
        for (int i = 32 * kListAhead + lane; i < n_ent; i += 32) put(__ldg(entries + i));
        __syncwarp();
        id = id1; id1 = id2;
        head = head1; head1 = head2;
    }
    cp_async_wait<0>();
}

}  // namespace trs

struct trs_sddmm_plan {
    const int32_t* rowptr = nullptr;  // caller-owned pattern (used by the fallback kernel)
    const int32_t* col = nullptr;
    int n_rows = 0, n_cols = 0;
    long long nnz = 0, n_blocks = 0, n_pairs = 0;
    int n_quads = 0;
    bool wide = false;   // a window with too many entries for the lists
    int device = 0;
    void* block = nullptr;        // pool memory of the arrays below (a cudaMalloc each took up to milliseconds)
    trs::SddmmQuad* quads = nullptr;
    int* ids = nullptr;           // [quads][32]
    unsigned* list = nullptr;     // [nnz]
    trs::RingTables shares;
    const int* starts = nullptr;  // the tables, behind the ids; null where no wave can have one
    // whether a wave of the kernel for `kch` chunks goes by its table
    bool by_table(int kch) const {
        const trs::RingShares& sh = shares.of[kch - 1];
        return starts && trs::may_have_table(n_quads, sh.warps) && sh.worst_cost + sh.worst_cost / 8 < sh.worst;
    }
};

extern "C" int trs_sddmm_plan_destroy(trs_sddmm_plan* p) {
    if (!p) return TRS_OK;
    if (p->block) {
        // kernels on any stream may still read the plan: wait as cudaFree would
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev != p->device) cudaSetDevice(p->device);
        cudaDeviceSynchronize();
        trs::pool_free(p->block, nullptr);
        if (dev != p->device) cudaSetDevice(dev);
    }
    delete p;
    return TRS_OK;
}

extern "C" int trs_sddmm_plan_create(const int32_t* rowptr, const int32_t* col, int n_rows, int n_cols, void* stream,
                                     trs_sddmm_plan** out) try {
    using namespace trs;
    if (!out) return TRS_E_ARG;
    *out = nullptr;
    if (!rowptr || n_rows <= 0 || n_cols <= 0) return TRS_E_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return TRS_E_NO_DEVICE;
    cudaStream_t st = (cudaStream_t)stream;
    int ends[2] = {0, 0};
    TRS_CUDA(cudaMemcpyAsync(&ends[0], rowptr, sizeof(int), cudaMemcpyDeviceToHost, st));
    TRS_CUDA(cudaMemcpyAsync(&ends[1], rowptr + n_rows, sizeof(int), cudaMemcpyDeviceToHost, st));
    TRS_CUDA(cudaStreamSynchronize(st));
    if (ends[0] != 0 || ends[1] < 0) return TRS_E_OFFSETS;
    const long long nnz = ends[1];
    if (nnz > 0 && !col) return TRS_E_ARG;
    trs_sddmm_plan* p = new trs_sddmm_plan();
    p->rowptr = rowptr; p->col = col; p->n_rows = n_rows; p->n_cols = n_cols; p->nnz = nnz;
    if (nnz == 0) { *out = p; return TRS_OK; }

    const int W = (n_rows + 15) / 16;
    int dev = 0, sms = 1;
    TRS_CUDA(cudaGetDevice(&dev));
    TRS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TempSpace ts;
    ts.st = st;
    ts.chunk_bytes = (size_t)nnz * 38 + ((size_t)W + 1) * 12 + ((size_t)8 << 20);
    unsigned long long *key_a, *key_b;
    int *ent_a, *ent_b, *head, *pair_idx, *first_pair, *quads_of, *quad_off, *begin, *d_err;
    auto fail = [&](int code) { trs_sddmm_plan_destroy(p); return code; };
    int rc = ts.get(nnz, &key_a);
    if (!rc) rc = ts.get(nnz, &key_b);
    if (!rc) rc = ts.get(nnz, &ent_a);
    if (!rc) rc = ts.get(nnz, &ent_b);
    if (!rc) rc = ts.get(nnz, &head);
    if (!rc) rc = ts.get(nnz, &pair_idx);
    if (!rc) rc = ts.get((size_t)W + 1, &first_pair);
    if (!rc) rc = ts.get((size_t)W + 1, &quads_of);
    if (!rc) rc = ts.get((size_t)W + 1, &quad_off);
    if (!rc) rc = ts.get(nnz, &begin);
    if (!rc) rc = ts.get(2 + 2 * kRingClasses, &d_err);   // error bits, number of 8-column blocks, largest shares
    if (rc) return fail(rc);
    auto grid = [](long long n) { return (unsigned)((n + 255) / 256); };
    cudaMemsetAsync(d_err, 0, (2 + 2 * kRingClasses) * sizeof(int), st);
    ksp_rows<<<grid(n_rows), 256, 0, st>>>(rowptr, n_rows, d_err);
    ksp_keys<<<grid(nnz), 256, 0, st>>>(rowptr, col, n_rows, n_cols, nnz, key_a, ent_a, d_err);
    {
        int herr = 0;
        cudaError_t ee = cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (ee == cudaSuccess) ee = cudaStreamSynchronize(st);
        if (ee != cudaSuccess) return fail((int)ee);
        if (herr & 8) return fail(TRS_E_OFFSETS);
        if (herr & 1) return fail(TRS_E_COLUMN);
        if (herr & 2) return fail(TRS_E_NOT_CANONICAL);
    }
    int wbits = 1;
    while ((1ll << wbits) < W) ++wbits;
    cub::DoubleBuffer<unsigned long long> kb(key_a, key_b);
    cub::DoubleBuffer<int> vb(ent_a, ent_b);
    size_t bytes = 0, bytes2 = 0, bytes3 = 0, bytes4 = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, bytes, kb, vb, (int)nnz, 0, 32 + wbits, st);
    if (e == cudaSuccess) e = cub::DeviceScan::InclusiveSum(nullptr, bytes2, head, pair_idx, (int)nnz, st);
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, bytes3, quads_of, quad_off, W + 1, st);
    // costs of the quads: no more of them than entries
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, bytes4, (unsigned*)nullptr, (unsigned*)nullptr, nnz + 1, st);
    if (e != cudaSuccess) return fail((int)e);
    bytes = std::max(std::max(bytes, bytes4), std::max(bytes2, bytes3));
    unsigned char* tmp;
    if ((rc = ts.get(bytes + 16, &tmp))) return fail(rc);
    e = cub::DeviceRadixSort::SortPairs(tmp, bytes, kb, vb, (int)nnz, 0, 32 + wbits, st);
    if (e != cudaSuccess) return fail((int)e);
    const unsigned long long* key = kb.Current();
    const int* ent = vb.Current();
    ksp_heads<<<grid(nnz), 256, 0, st>>>(key, nnz, head);
    e = cub::DeviceScan::InclusiveSum(tmp, bytes, head, pair_idx, (int)nnz, st);  // pair id + 1
    if (e != cudaSuccess) return fail((int)e);
    int total_pairs = 0;
    e = cudaMemcpyAsync(&total_pairs, pair_idx + (nnz - 1), sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail((int)e);
    // pair_idx holds inclusive sums: pair id of sorted entry i = pair_idx[i] - 1.  Only differences against
    // first_pair, which is taken from the same array, are used.
    ksp_window_pairs<<<grid(W + 1), 256, 0, st>>>(key, pair_idx, nnz, total_pairs + 1, W, first_pair, quads_of, d_err + 1);
    e = cub::DeviceScan::ExclusiveSum(tmp, bytes, quads_of, quad_off, W + 1, st);
    if (e != cudaSuccess) return fail((int)e);
    int n_quads = 0, n_blocks = 0;
    e = cudaMemcpyAsync(&n_quads, quad_off + W, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&n_blocks, d_err + 1, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail((int)e);
    p->n_quads = n_quads;
    p->n_blocks = n_blocks;
    p->n_pairs = total_pairs;
    RingTables& sh = p->shares;
    sh.total = 0;
    int least = INT_MAX, most = 0;   // warps of a wave
    for (int c = 0; c < kRingClasses; ++c) {
        sh.of[c] = RingShares{sms * ring_ctas(c + 1) * kRingWarps, sh.total, 0u, 0u};
        sh.total += sh.of[c].warps + 1;
        least = std::min(least, sh.of[c].warps);
        most = std::max(most, sh.of[c].warps);
    }
    const bool tables = may_have_table(n_quads, least);
    p->device = dev;
    const size_t quad_bytes = (size_t)n_quads * sizeof(SddmmQuad), id_bytes = (size_t)n_quads * 32 * sizeof(int);
    const size_t start_bytes = tables ? (size_t)sh.total * sizeof(int) : 0;
    if ((rc = pool_alloc(&p->block, quad_bytes + id_bytes + start_bytes + (size_t)nnz * sizeof(unsigned), st))) return fail(rc);
    unsigned char* at = (unsigned char*)p->block;
    p->quads = (SddmmQuad*)at; at += quad_bytes;
    p->ids = (int*)at; at += id_bytes;
    int* const starts = (int*)at;
    if (tables) p->starts = starts;
    at += start_bytes;
    p->list = (unsigned*)at;
    unsigned *cost = nullptr, *cost_before = nullptr;
    if (tables && (rc = ts.get((size_t)n_quads + 1, &cost))) return fail(rc);
    if (tables && (rc = ts.get((size_t)n_quads + 1, &cost_before))) return fail(rc);
    ksp_columns<<<grid(nnz), 256, 0, st>>>(key, pair_idx, head, first_pair, quad_off, nnz, p->ids, begin);
    ksp_quads<<<(unsigned)ceil_div(n_quads, 8), 256, 0, st>>>(key, ent, pair_idx, first_pair, begin, rowptr, n_rows, (int)nnz, n_quads,
                                                              p->quads, p->ids, p->list, cost, d_err);
    if (tables) {
        e = cub::DeviceScan::ExclusiveSum(tmp, bytes, cost, cost_before, n_quads + 1, st);
        if (e != cudaSuccess) return fail((int)e);
        ksp_shares<<<dim3(grid(most + 1), kRingClasses), 256, 0, st>>>(cost_before, n_quads, sh, starts, (unsigned*)d_err + 2);
    }
    int back[2 + 2 * kRingClasses];
    e = cudaMemcpyAsync(back, d_err, sizeof(back), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail((int)e);
    p->wide = (back[0] & 4) != 0;
    for (int c = 0; c < kRingClasses; ++c) {
        sh.of[c].worst = (unsigned)back[2 + 2 * c];
        sh.of[c].worst_cost = (unsigned)back[3 + 2 * c];
    }
    *out = p;
    return TRS_OK;
} TRS_CATCH

extern "C" int trs_sddmm_plan_info(const trs_sddmm_plan* p, long long* n_pairs, long long* n_blocks) {
    if (!p) return TRS_E_ARG;
    if (n_pairs) *n_pairs = p->n_pairs;
    if (n_blocks) *n_blocks = p->n_blocks;
    return TRS_OK;
}

extern "C" int trs_sddmm_plan_shares(const trs_sddmm_plan* p, int K, int* warps, unsigned* by_number, unsigned* by_cost, int* table) {
    const int kch = (K + 31) / 32;
    if (!p || K <= 0 || kch > trs::kRingClasses) return TRS_E_ARG;
    const trs::RingShares none{0, 0, 0u, 0u}, &sh = p->nnz > 0 ? p->shares.of[kch - 1] : none;
    if (warps) *warps = sh.warps;
    if (by_number) *by_number = sh.worst;
    if (by_cost) *by_cost = sh.worst_cost;
    if (table) *table = p->nnz > 0 && p->by_table(kch);
    return TRS_OK;
}

namespace {

using namespace trs;

// X and Y as the kernels want them: rows on 16-byte boundaries, `ld` halfs apart.  Otherwise padded copies in
// pool memory, given back to the pool behind the kernel; ld = 0: there is no memory for them.
struct Operands {
    const __half *X = nullptr, *Y = nullptr;
    int ld = 0;
    void* copy = nullptr;
    cudaStream_t st = nullptr;
    int prepare(const trs_half* x, const trs_half* y, int n_rows, int n_cols, int K, cudaStream_t stream) {
        st = stream;
        X = (const __half*)x; Y = (const __half*)y; ld = K;
        if (K % 8 == 0 && (((uintptr_t)x | (uintptr_t)y) & 15) == 0) return TRS_OK;
        ld = (K + 15) & ~15;   // whole 32-byte sectors
        const int per_row = ld / 8;
        const int rc = pool_alloc(&copy, ((size_t)n_rows + n_cols) * ld * sizeof(__half), st);
        if (rc == (int)cudaErrorMemoryAllocation) { ld = 0; return TRS_OK; }
        if (rc) return rc;
        __half* xp = (__half*)copy;
        __half* yp = xp + (size_t)n_rows * ld;
        const long long pieces = ((long long)n_rows + n_cols) * per_row;
        k_sddmm_pad<<<(unsigned)ceil_div64(pieces, 256), 256, 0, st>>>(X, Y, n_rows, pieces, K, per_row, xp);
        TRS_LAUNCH_CHECK();
        X = xp; Y = yp;
        return TRS_OK;
    }
    ~Operands() { pool_free(copy, st); }
};

int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    int n = cached[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cached[dev].store(n, std::memory_order_relaxed);
    }
    return n > 0 ? n : 1;
}

// `ends`: three words of pinned memory for publish_ends, or null.  An error is the launch's own, not one that an earlier call left
// with the thread: it says that nothing will write the words.
int launch_entries(const int32_t* rowptr, const int32_t* col, const Operands& o, void* out, int out_f32, int n_rows, int n_cols,
                   int K, int* ends, cudaStream_t st) {
    if (o.ld == 0)
        return launch(k_sddmm_plain, dim3(sm_count() * 8), 256, 0, st, rowptr, col, o.X, o.Y, out, out_f32, n_rows, n_cols, K, ends);
    auto go = [&](auto kernel, int ctas) {
        return launch(kernel, dim3(sm_count() * ctas), 32 * kEntryWarps, 0, st, rowptr, col, o.X, o.Y, out, out_f32, n_rows, n_cols, K, o.ld, ends);
    };
    if (K == 32) return go(k_sddmm<1, true>, entry_ctas(1));
    if (K < 32) return go(k_sddmm<1, false>, entry_ctas(1));
    if (K == 64) return go(k_sddmm<2, true>, entry_ctas(2));
    if (K < 64) return go(k_sddmm<2, false>, entry_ctas(2));
    if (K == 96) return go(k_sddmm<3, true>, entry_ctas(3));
    if (K < 96) return go(k_sddmm<3, false>, entry_ctas(3));
    if (K == 128) return go(k_sddmm<4, true>, entry_ctas(4));
    return go(k_sddmm<4, false>, entry_ctas(4));
}

template <int KCH, bool TAIL, bool F32>
int launch_ring(const trs_sddmm_plan* p, const Operands& o, void* out, int K, cudaStream_t st) {
    using R = SddmmRing<KCH>;
    auto kernel = k_sddmm_tc_ring<KCH, TAIL, F32>;
    static std::atomic<unsigned long long> done{0};
    const int rc = allow_smem(kernel, R::SMEM, false, done);
    if (rc) return rc;
    const RingShares& sh = p->shares.of[KCH - 1];
    const bool table = p->by_table(KCH);
    const int per_warp = ceil_div(p->n_quads, sh.warps);
    const int warps = table ? sh.warps : ceil_div(p->n_quads, per_warp);
    kernel<<<ceil_div(warps, kRingWarps), 32 * kRingWarps, R::SMEM, st>>>(p->quads, p->ids, p->list, table ? p->starts + sh.offset : nullptr,
                                                                        p->n_quads, per_warp, o.X, o.Y, out, p->n_rows, (K + 7) / 8, o.ld / 8);
    TRS_LAUNCH_CHECK();
    return TRS_OK;
}

template <int KCH>
int launch_ring_k(const trs_sddmm_plan* p, const Operands& o, void* out, int out_f32, int K, cudaStream_t st) {
    if (out_f32) return K == 32 * KCH ? launch_ring<KCH, false, true>(p, o, out, K, st) : launch_ring<KCH, true, true>(p, o, out, K, st);
    return K == 32 * KCH ? launch_ring<KCH, false, false>(p, o, out, K, st) : launch_ring<KCH, true, false>(p, o, out, K, st);
}

// Three ints the device writes and the host reads (pinned, mapped).  Taken for one call, kept for the next ones: as many
// exist as calls ever ran at the same time.
struct EndsWord {
    volatile int* p = nullptr;
    int device = 0;
};
std::mutex g_ends_mutex;
std::vector<EndsWord> g_ends;

int take_ends(EndsWord* w) {
    int dev = 0;
    TRS_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lock(g_ends_mutex);
        for (size_t i = g_ends.size(); i-- > 0;)
            if (g_ends[i].device == dev) {
                *w = g_ends[i];
                g_ends.erase(g_ends.begin() + i);
                w->p[2] = 0;
                return TRS_OK;
            }
    }
    w->device = dev;
    TRS_CUDA(cudaHostAlloc((void**)&w->p, 3 * sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
    w->p[2] = 0;
    return TRS_OK;
}
void give_ends(const EndsWord& w) {
    std::lock_guard<std::mutex> lock(g_ends_mutex);
    g_ends.push_back(w);
}
// Until the device has written the word; an error of the stream ends the wait.  The word comes as the product begins, so behind
// short work it is looked at all the time; behind a long queue that would cost a core for as long as the queue lasts (and, with every
// look at the stream, a lock of the driver), so after two milliseconds the thread sleeps between looks, a sixty-fourth of the time waited so
// far at once (behind 2.05 / 10.2 / 254 ms of work the call takes 2.04 / 2.3 / 5.6 ms of the core's time and returns 0.09 / 0.03 / 0.15
// ms later).
cudaError_t wait_for_ends(const EndsWord& w, cudaStream_t st) {
    using namespace std::chrono;
    constexpr microseconds kSpin{2000}, kLook{100}, kShort{50}, kLong{250};
    steady_clock::time_point start{}, looked{};
    for (unsigned i = 0; !w.p[2]; ++i) {
#if defined(__SSE2__)
        _mm_pause();
#endif
        if (i % 64 != 0) continue;
        const auto now = steady_clock::now();
        if (i == 0) { start = looked = now; continue; }
        if (now - looked < kLook) continue;
        const cudaError_t e = cudaStreamQuery(st);
        if (e != cudaSuccess) (void)cudaGetLastError();   // not an error of a later launch
        if (e != cudaSuccess && e != cudaErrorNotReady) return e;
        if (e == cudaSuccess && !w.p[2]) return cudaErrorUnknown;   // all done, and nothing was written
        looked = now;
        if (now - start < kSpin) continue;
        std::this_thread::sleep_for(std::min(std::max(duration_cast<microseconds>((now - start) / 64), kShort), kLong));
        i = 63;   // look again at once
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return cudaSuccess;
}

}  // namespace

extern "C" int trs_sddmm_plan_run(const trs_sddmm_plan* p, const trs_half* X, const trs_half* Y, trs_half* out, int K,
                                  void* stream) {
    return trs_sddmm_plan_run_ex(p, X, Y, out, K, TRS_OUT_F16, stream);
}

extern "C" int trs_sddmm_plan_run_ex(const trs_sddmm_plan* p, const trs_half* X, const trs_half* Y, void* out, int K,
                                     int out_dtype, void* stream) {
    if (!p || !X || !Y || K <= 0) return TRS_E_ARG;
    if (out_dtype != TRS_OUT_F32 && out_dtype != TRS_OUT_F16) return TRS_E_ARG;
    const int out_f32 = out_dtype == TRS_OUT_F32;
    if (p->nnz == 0) return TRS_OK;
    if (!out) return TRS_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    Operands o;
    const int rc = o.prepare(X, Y, p->n_rows, p->n_cols, K, st);
    if (rc) return rc;
    switch (p->wide || o.ld == 0 ? 0 : (K + 31) / 32) {
        case 1: return launch_ring_k<1>(p, o, out, out_f32, K, st);
        case 2: return launch_ring_k<2>(p, o, out, out_f32, K, st);
        case 3: return launch_ring_k<3>(p, o, out, out_f32, K, st);
        case 4: return launch_ring_k<4>(p, o, out, out_f32, K, st);
        case 5: return launch_ring_k<5>(p, o, out, out_f32, K, st);
        case 6: return launch_ring_k<6>(p, o, out, out_f32, K, st);
        case 7: return launch_ring_k<7>(p, o, out, out_f32, K, st);
        case 8: return launch_ring_k<8>(p, o, out, out_f32, K, st);
        default: break;   // a window's X tile no longer fits the registers
    }
    return launch_entries(p->rowptr, p->col, o, out, out_f32, p->n_rows, p->n_cols, K, nullptr, st);
}

extern "C" int trs_sddmm(const int32_t* rowptr, const int32_t* col, const trs_half* X, const trs_half* Y, trs_half* out,
                         int n_rows, int n_cols, int K, void* stream) try {
    if (!rowptr || !X || !Y || n_rows <= 0 || n_cols <= 0 || K <= 0) return TRS_E_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return TRS_E_NO_DEVICE;
    cudaStream_t st = (cudaStream_t)stream;
    // The ends of rowptr decide whether this is an error, and only the device has them.  The product's own kernel looks at
    // them and passes them on as it begins; the host waits for that, after earlier work of the stream, and for nothing else.  (A kernel
    // of their own before the product took 3 of 28 us: uniform 50 021 rows, K = 96.)
    // A graph has no row pointers to look at when it is captured: refused before anything is queued, so that nothing is
    // left that could write the words later.
    cudaStreamCaptureStatus capture;
    TRS_CUDA(cudaStreamIsCapturing(st, &capture));
    if (capture != cudaStreamCaptureStatusNone) return (int)cudaErrorStreamCaptureUnsupported;
    EndsWord ends;
    int rc = take_ends(&ends);
    if (rc) return rc;
    Operands o;
    if (col && out) {
        rc = o.prepare(X, Y, n_rows, n_cols, K, st);
        if (!rc) rc = launch_entries(rowptr, col, o, out, 0, n_rows, n_cols, K, (int*)ends.p, st);
    } else {
        rc = launch(k_sddmm_ends, dim3(1), 1, 0, st, rowptr, n_rows, (int*)ends.p);
    }
    if (rc) {   // the kernel that writes the words was refused, or not asked for
        give_ends(ends);
        return rc;
    }
    const cudaError_t e = wait_for_ends(ends, st);
    if (e != cudaSuccess) return (int)e;   // the words stay with what may still write them
    const int first = ends.p[0], last = ends.p[1];
    give_ends(ends);
    if (first != 0 || last < 0) return TRS_E_OFFSETS;
    if (last > 0 && (!col || !out)) return TRS_E_ARG;
    return TRS_OK;
} TRS_CATCH
