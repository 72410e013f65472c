// GPU format builder: CSR -> the reference's three-way hybrid format, bit-exact.
//
// Replaces block_sptc_2to4_online (TR-source/Block/block_online.cpp:545-871), which walks the
// windows serially on one CPU thread with hash maps and an O(U^2) unit graph.  Here every stage
// is a data-parallel pass over device arrays:
//
//   1. windows by size: a CTA per window sorts its entries by column in shared memory (hub windows:
//      device-wide sorts)                                          -> per-window column lists
//      (the reference's col_info map, block_online.cpp:589-603)
//   2. runs of equal columns -> one record per (window, column): count, 16-bit row mask, first entry
//   3. stable sort by 16 - count: the (count desc, column asc) order both funnels
//      use (block_online.cpp:226-230, 281-285)
//   4. TC funnel: leading columns with count >= density in chunks of 8, kept when
//      nnz/(window*8) >= tc_min_util (block_online.cpp:215-253).  Counts descend, so the kept chunks
//      are the first ones and everything that follows is arithmetic on three numbers per window.
//   5. units = consecutive pairs of the remaining columns (the first-fit of
//      block_online.cpp:287-326 always takes the next column because its bit test cannot fail)
//   6. matching (block_online.cpp:332-392): the unit graph is complete, so degrees are all
//      equal, the node order is libstdc++ std::sort of unit nnz (emulated, see trs_stdsort.cuh)
//      and the partner of a node is the lowest-index unmatched other unit
//   7. group emission, per-row (value, position) slots with the reference's "first two kept,
//      the rest dropped" rule (block_online.cpp:629-703), and the 16x16 mma.sp tile of four groups
//      (block_online.cpp:190-210, 796-841), all by one warp per tile
//   8. TC blocks, bitmaps, values, parts (block_online.cpp:444-540)
//   9. CUDA-core row parts from the columns of an unmatched sparse unit (block_online.cpp:397-439,
//      706-733)
//
// Input contract: canonical CSR (columns strictly ascending inside a row), window in 1..16.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/transform_iterator.h>
#include <thrust/iterator/transform_output_iterator.h>
#include <thrust/iterator/zip_iterator.h>
#include <thrust/iterator/counting_iterator.h>

#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <vector>

#include "trs_common.cuh"
#include "trs_stdsort.cuh"

namespace trs {

typedef unsigned long long u64;

struct BuildCfg {
    int part_t, part_c, short_size, density, window;
    float tc_min_util;
    int skip_tc, unit_min_nnz;
    int strict;  // 1: lossless — entries the reference drops go to the CUDA-core parts instead
};

// ---------------------------------------------------------------------------------------------
// 0. the sizes, the row pointers and the windows by size: one pass, one read-back
// ---------------------------------------------------------------------------------------------
// Classes of windows: up to 256 entries, and up to 512 and 1024 where no row has more than a sixteenth of that, sorted by
// one warp in registers; up to 1024 otherwise and then up to 8192 by one CTA in shared memory; by device-wide passes over all
// larger ones together beyond (hub windows).  A power-law graph's windows above 256 have one long row nearly always, and
// sorted from scratch by a warp they take longer than a CTA merging their rows (builds of R-MAT 15 / 18 505 / 1163 against 493 /
// 1140 us); windows of equal rows of 1025 to 2048 entries are as fast in a CTA (703 and 698 us).
constexpr int kSortClasses = 7, kWarpClasses = 3;
__host__ __device__ constexpr int sort_cap(int c) { return c < kWarpClasses ? 256 << c : 1024 << (c - kWarpClasses); }
__device__ __forceinline__ int sort_class_of(long long n, int longest_row) {
    if (n <= 0) return kSortClasses + 1;   // no class
    if (n <= sort_cap(0)) return 0;
    for (int c = 1; c < kWarpClasses; ++c)
        if (n <= sort_cap(c) && longest_row <= sort_cap(c) / 16) return c;
    for (int c = kWarpClasses; c < kSortClasses; ++c)
        if (n <= sort_cap(c)) return c;
    return kSortClasses;
}

struct InputInfo {
    int first, last;  // rowptr[0], rowptr[n_rows]
    int max_col;
    int err;          // 1: decreasing row pointer, 2: columns negative, not ascending or repeated
    int windows[kSortClasses + 1];   // windows per class, hubs last
    u64 hub_entries;
};

// Words that the host looks at, copied into pinned memory by the kernel that finishes them.
struct Publish {
    const int* a;
    int* host_a;
    int na;
    const int* b;
    int* host_b;
    int nb;
    __device__ __forceinline__ void by_block() const {
        for (int i = threadIdx.x; i < na; i += blockDim.x) host_a[i] = __ldcg(a + i);
        for (int i = threadIdx.x; i < nb; i += blockDim.x) host_b[i] = __ldcg(b + i);
    }
};

__global__ void kb_input_info(const int* __restrict__ rowptr, const int* __restrict__ col, int n_rows, int window, int W,
                              int* __restrict__ sel /* [kSortClasses + 1][W] */, int* __restrict__ ncol /* [W], cleared */,
                              InputInfo* info, unsigned* done /* cleared */, Publish pub) {
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    const int first = rowptr[0], nnz = rowptr[n_rows];
    if (t0 == 0) { info->first = first; info->last = nnz; }
    bool bad = false;
    for (long long r = t0; r < n_rows; r += step) bad |= rowptr[r + 1] < rowptr[r];
    if (bad) atomicOr(&info->err, 1);
    const int lane = threadIdx.x & 31;
    for (long long w0 = t0 - lane; w0 < W; w0 += step) {   // whole warps
        const long long w = w0 + lane;
        long long n = 0;
        int longest_row = 0;
        if (w < W) {
            const long long r1 = min((w + 1) * window, (long long)n_rows);
            int from = rowptr[w * window];
            n = (long long)rowptr[r1] - from;
            ncol[w] = 0;
            if (n > sort_cap(0) && n <= sort_cap(kWarpClasses - 1))
                for (long long r = w * window + 1; r <= r1; ++r) {
                    const int to = rowptr[r];
                    longest_row = max(longest_row, to - from);
                    from = to;
                }
        }
        const int c = sort_class_of(n, longest_row);
        for (int i = 0; i <= kSortClasses; ++i) {
            const unsigned in = __ballot_sync(0xffffffffu, c == i);
            if (!in) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(&info->windows[i], __popc(in));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (c == i) sel[(size_t)i * W + at + __popc(in & ((1u << lane) - 1u))] = (int)w;
        }
        if (c == kSortClasses) atomicAdd(&info->hub_entries, (u64)n);
    }
    if (first == 0 && col) {
        int m = -1;
        for (long long e = t0; e < nnz; e += step) m = max(m, col[e]);
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0 && m > __ldcg(&info->max_col)) atomicMax(&info->max_col, m);
    }
    // the last block to get here passes everything on to the host
    __shared__ bool s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(done, 1u) + 1 == gridDim.x;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    pub.by_block();
}

// Exclusive scan of a few thousand values by one CTA: the device-wide scan and the copy of its sum for the host are three
// launches, this is one.  What bounds it is one SM's load and store rate, so up to 4608 values (builds of 9000 uniform rows 222 ->
// 201 us, of 20000 clustered ones 278 -> 252, with the other read-backs made by the kernels that finish them; 16385 windows of
// four words a build of 567 -> 612).
constexpr int kSmallScan = 4608;
template <class T, class Shuffle>
__device__ __forceinline__ T shuffle_words(const T& x, Shuffle&& shuffle) {
    static_assert(sizeof(T) % 4 == 0, "");
    T y;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); ++i) ((int*)&y)[i] = shuffle(((const int*)&x)[i]);
    return y;
}
template <class T, class Op>
__device__ __forceinline__ T warp_inclusive(T x, Op op, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = shuffle_words(x, [&](int w) { return __shfl_up_sync(0xffffffffu, w, d); });
        if (lane >= d) x = op(y, x);
    }
    return x;
}
template <class T, class Op, class In, class Out>
__global__ void __launch_bounds__(1024) kb_scan_small(In in, Out out, Op op, T zero, int n, Publish pub) {
    constexpr int kItems = 4;   // consecutive ones per thread and round (one: 1.2 us a round of 1024 four-word values)
    __shared__ T s_warp[2][32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    T before = zero, next[kItems];
    auto load = [&](int base) {
#pragma unroll
        for (int i = 0; i < kItems; ++i) next[i] = base + tid * kItems + i < n ? in(base + tid * kItems + i) : zero;
    };
    load(0);
    for (int base = 0, k = 0; base < n; base += 1024 * kItems, k ^= 1) {
        T x[kItems];
        T mine = zero;
#pragma unroll
        for (int i = 0; i < kItems; ++i) { x[i] = next[i]; mine = op(mine, x[i]); }
        load(base + 1024 * kItems);
        const T incl = warp_inclusive(mine, op, lane);
        if (lane == 31) s_warp[k][wid] = incl;
        __syncthreads();
        const T warps = warp_inclusive(s_warp[k][lane], op, lane);
        T at = before;   // everything before this thread's values
        if (wid > 0) at = op(at, shuffle_words(warps, [&](int w) { return __shfl_sync(0xffffffffu, w, max(wid - 1, 0)); }));
        const T prev = shuffle_words(incl, [&](int w) { return __shfl_up_sync(0xffffffffu, w, 1); });
        if (lane > 0) at = op(at, prev);
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            if (base + tid * kItems + i < n) out(base + tid * kItems + i, at);
            at = op(at, x[i]);
        }
        before = op(before, shuffle_words(warps, [&](int w) { return __shfl_sync(0xffffffffu, w, 31); }));
    }
    __syncthreads();
    pub.by_block();
}
template <class T>
struct FromArray {
    const T* p;
    __device__ __forceinline__ T operator()(int i) const { return p[i]; }
};
template <class T>
struct ToArray {
    T* p;
    __device__ __forceinline__ void operator()(int i, const T& x) const { p[i] = x; }
};
struct IntSum {
    __host__ __device__ __forceinline__ int operator()(int a, int b) const { return a + b; }
};

// ---------------------------------------------------------------------------------------------
// 1. - 3. the columns of every window
// ---------------------------------------------------------------------------------------------
// The entries of a window are contiguous in the input, so a window's part of every array below starts at
// the index of its first entry, and no global position has to be found.  What comes out, per window:
//   rec    one record per column, in (count desc, column asc) order
//   cnt    their counts
//   sval   the values in (column, row) order; record r's are sval[r.start .. r.start + count)
//   ncol   how many records
struct __align__(16) Record {   // one (window, column): its first sorted entry, the rows it has, the first value
    int col, start;
    unsigned mask;
    float value;
};

struct WindowOut {
    Record* rec;
    unsigned char* cnt;
    float* sval;
    int* ncol;
};

// Windows that do not go to kb_sort_warp: one CTA per window of at most CAP entries, everything in shared memory; 12 bytes read
// and 4 + 17 per column written per entry.  The rows of a window are sorted already, so four rounds merge them two by two: a thread finds where its
// outputs begin by binary search along the diagonal (merge path) and then takes them one by one.  A record's place in the
// (count desc, column asc) order is counted, not sorted.
//
// What bounds it: issue and the shared-memory pipe.  Device-wide sorts of (window, column) keys with their key, head and
// record passes moved ten times the bytes: 0.69 of the 1.30 ms of a build of the clustered graph.  A radix sort of the block
// instead of the merge took 262 us on its windows of 780 entries whatever its digits, a merge with a binary search per entry and
// round 305, this 201 (a warp, where they go now, 151), and 32 in place of 53 on windows of 510.
template <int T, int CAP, class Key>
struct WindowSort {
    static constexpr int PB = CAP <= 256 ? 8 : CAP <= 512 ? 9 : CAP <= 1024 ? 10 : CAP <= 2048 ? 11 : CAP <= 4096 ? 12 : 13;   // bits of a place in the window
    static_assert(CAP <= 1 << PB, "");
    struct Smem {
        Key key[2][CAP];           // column << PB | place in the window
        unsigned char row[CAP];    // row whose entries begin at or before a position
        unsigned short start[CAP]; // of the records
        unsigned mask[CAP / 2];    // of the records, two in a word
        unsigned heads[CAP / 32];  // entries where the column changes
        int chunk[CAP / 32];       // records that begin in a chunk of 32 entries, then before it
        int bound[17];             // first entry of every row, from the window's first
        int warp_sum[32];
    };
};

template <int T, int CAP, class Key>
__global__ void __launch_bounds__(T) kb_sort_window(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                    const float* __restrict__ val, int n_rows, int window,
                                                    const int* __restrict__ sel, WindowOut out, InputInfo* __restrict__ info) {
    using S = WindowSort<T, CAP, Key>;
    constexpr int PB = S::PB;
    constexpr unsigned kPlace = (1u << PB) - 1u;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    typename S::Smem& s = *reinterpret_cast<typename S::Smem*>(smem_raw);
    unsigned short* const cells = reinterpret_cast<unsigned short*>(s.key[1]);   // free after the merge; 16 per chunk of records
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int w = sel[blockIdx.x];
    const int base = rowptr[(size_t)w * window];
    if (tid < 17) s.bound[tid] = rowptr[min((long long)w * window + min(tid, window), (long long)n_rows)] - base;
    __syncthreads();
    const int n = s.bound[16];
    bool bad = false;
    for (int i = tid; i < n; i += T) {
        const int c = col[base + i];
        int row = 0;
#pragma unroll
        for (int d = 8; d; d >>= 1)
            if (row + d < window && s.bound[row + d] <= i) row += d;
        s.key[0][i] = (Key)(unsigned)c << PB | (Key)(unsigned)i;
        s.row[i] = (unsigned char)row;
        bad |= c < 0 || (i + 1 < s.bound[row + 1] && col[base + i + 1] <= c);
    }
    for (int i = tid; i < (n + 1) / 2; i += T) s.mask[i] = 0u;
    if (__syncthreads_or(bad)) {   // nothing below holds for unsorted rows
        if (tid == 0) atomicOr(&info->err, 2);
        return;
    }
    // outputs per thread and round; odd, so that the threads' stores fall into different banks
    const int per = ((n + T - 1) / T) | 1, o0 = tid * per, o1 = min(o0 + per, n);
    constexpr Key kNone = ~(Key)0;
#pragma unroll
    for (int L = 0; L < 4; ++L) {
        const Key* const src = s.key[L & 1];
        Key* const dst = s.key[1 - (L & 1)];
        if (o0 < n) {
            int pair = s.row[o0] >> (L + 1);
            int s0 = s.bound[pair << (L + 1)], s1 = s.bound[(2 * pair + 1) << L], s2 = s.bound[(pair + 1) << (L + 1)];
            // how many of the pair's first o0 - s0 outputs come from its first run
            const int d = o0 - s0;
            int lo = max(0, d - (s2 - s1)), hi = min(d, s1 - s0);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (src[s0 + mid] < src[s1 + d - 1 - mid]) lo = mid + 1; else hi = mid;
            }
            int i = s0 + lo, j = s1 + d - lo;
            Key a = i < s1 ? src[i] : kNone, b = j < s2 ? src[j] : kNone;
            for (int p = o0;;) {
                const bool first = a < b;
                dst[p] = first ? a : b;
                if (++p == o1) break;
                if (p == s2) {   // on to the next pair that has entries
                    do {
                        ++pair;
                        s0 = s2;
                        s1 = s.bound[(2 * pair + 1) << L];
                        s2 = s.bound[(pair + 1) << (L + 1)];
                    } while (s2 == s0);
                    i = s0; j = s1;
                    a = i < s1 ? src[i] : kNone;
                    b = j < s2 ? src[j] : kNone;
                } else if (first) {
                    ++i;
                    a = i < s1 ? src[i] : kNone;
                } else {
                    ++j;
                    b = j < s2 ? src[j] : kNone;
                }
            }
        }
        __syncthreads();
    }
    const Key* const key = s.key[0];
    // records begin where the column changes
    const int chunks = (n + 31) / 32;
    for (int c = wid; c < chunks; c += T / 32) {
        const int i = c * 32 + lane;
        const bool head = i < n && (i == 0 || (key[i] >> PB) != (key[i > 0 ? i - 1 : 0] >> PB));
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        if (lane == 0) {
            s.heads[c] = heads;
            s.chunk[c] = __popc(heads);
        }
    }
    __syncthreads();
    if (tid < 32) {
        int before = 0;
        for (int c0 = 0; c0 < chunks; c0 += 32) {
            const int x = c0 + lane < chunks ? s.chunk[c0 + lane] : 0;
            int sum = x;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sum, d);
                if (lane >= d) sum += y;
            }
            if (c0 + lane < chunks) s.chunk[c0 + lane] = before + sum - x;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) s.warp_sum[0] = before;
    }
    __syncthreads();
    const int D = s.warp_sum[0];
    for (int c = wid; c < chunks; c += T / 32) {
        const int i = c * 32 + lane;
        const unsigned heads = s.heads[c], upto = heads & (0xffffffffu >> (31 - lane));
        const int r = s.chunk[c] + __popc(upto) - 1, seg = upto ? 31 - __clz(upto) : 0;   // no head yet: a record goes on
        unsigned m = 0u;
        if (i < n) {
            const unsigned place = (unsigned)key[i] & kPlace;
            out.sval[base + i] = val[base + place];
            m = 1u << s.row[place];
        }
#pragma unroll
        for (int d = 1; d < 16; d <<= 1) {   // at most 16 entries share a column
            const unsigned y = __shfl_up_sync(0xffffffffu, m, d);
            if (lane - d >= seg) m |= y;
        }
        if (i < n) {
            if ((heads >> lane) & 1u) s.start[r] = (unsigned short)i;
            if (lane == 31 || i + 1 == n || ((heads >> (lane + 1)) & 1u)) atomicOr(&s.mask[r >> 1], m << (16 * (r & 1)));
        }
    }
    // (count desc, column asc): records keep their order inside a count, so a record's place is the number of records of
    // larger counts, of its count in earlier chunks of 32, and of its count before it in its own chunk
    const unsigned short* const masks = (const unsigned short*)s.mask;
    const int rchunks = (D + 31) / 32, ncells = 16 * rchunks;
    for (int i = tid; i < ncells; i += T) cells[i] = 0;
    __syncthreads();
    for (int c = wid; c < rchunks; c += T / 32) {
        const int q = c * 32 + lane;
        const int k = q < D ? 16 - __popc((unsigned)masks[q]) : 16;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k < 16 && (same & lt) == 0) cells[k * rchunks + c] = (unsigned short)__popc(same);
    }
    __syncthreads();
    int before = 0;   // exclusive sums over the cells, T at a time
    for (int c0 = 0; c0 < ncells; c0 += T) {
        const int i = c0 + tid, x = i < ncells ? cells[i] : 0;
        int sum = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += y;
        }
        if (lane == 31) s.warp_sum[wid] = sum;
        __syncthreads();
        int at = before + sum - x;
#pragma unroll
        for (int q = 0; q < T / 32; ++q) {
            if (q < wid) at += s.warp_sum[q];
            before += s.warp_sum[q];
        }
        if (i < ncells) cells[i] = (unsigned short)at;
        __syncthreads();
    }
    for (int c = wid; c < rchunks; c += T / 32) {
        const int q = c * 32 + lane;
        const int k = q < D ? 16 - __popc((unsigned)masks[q]) : 16;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k == 16) continue;
        const int st = s.start[q];
        const Key first = key[st];
        const size_t o = (size_t)base + cells[k * rchunks + c] + __popc(same & lt);
        out.rec[o] = Record{(int)(first >> PB), base + st, masks[q], val[base + ((unsigned)first & kPlace)]};
        out.cnt[o] = (unsigned char)(16 - k);
    }
    if (tid == 0) out.ncol[w] = D;
}

// One warp per window of at most 32 KPL entries, the keys in registers, KPL consecutive ones per lane: a bitonic merge whose
// stages are two min / max per pair of keys (and a shuffle where the pair lies in two lanes), without an address, a bank or
// a branch.  Every row takes two lanes, so that only the four rounds that merge rows are left; where a row has more than 2 KPL
// entries, which the classes leave to KPL = 8, the keys are sorted from scratch.  The mask of a record is the difference of
// two prefix sums over 1 << row: rows of one column are distinct.
//
// What bounds it: issue.  The merge of a CTA in shared memory (kb_sort_window) took 11900 warp instructions per window of the
// clustered graph (780 entries) and 201 us at 89 % of the issue slots; this takes 5400 and 151 us at 60 % (its code does not stay in
// the innermost instruction cache).  The loads of all keys go out at once: eight at a time took 202 us.
template <int KPL>
struct WarpSort {
    static constexpr int CAP = 32 * KPL;
    static constexpr int PB = KPL == 8 ? 8 : KPL == 16 ? 9 : 10;
    static constexpr int LP = PB - 4;     // rows of 2 KPL places
    static_assert(1 << PB == CAP, "");
    struct __align__(16) Smem {   // the keys are read and written 16 bytes at a time
        unsigned key[CAP];                // key i at at(i)
        unsigned short before[CAP + 2];   // of the records: sum of 1 << row over the entries before, modulo 2^16
        unsigned short start[CAP + 2];    // of the records
        union {
            unsigned char row[CAP];                // of an entry, where rows have no places of their own
            unsigned short cells[16 * KPL];        // afterwards: records per count and chunk of 32
        };
        int bound[17];                    // first entry of every row, from the window's first
    };
    // The four keys that a lane reads or writes at a time lie where the eight lanes of a phase meet eight different bank groups,
    // and 32 consecutive keys are still in 32 different banks.
    __device__ static __forceinline__ int swizzle(int owner) { return KPL == 8 ? (owner >> 2) & 1 : KPL == 16 ? (owner >> 1) & 3 : owner & 7; }
    __device__ static __forceinline__ int at(int i) { return i ^ (swizzle(i / KPL) << 2); }
    static constexpr int CTAS = KPL <= 16 ? 9 : 6;   // of kSortWarps, by shared memory and registers
};

template <int N, int P, int K, int J = 0>
__device__ __forceinline__ void odd_even_stage(unsigned (&v)[N]) {   // Batcher's odd-even merge: pairs K apart, runs of P
#pragma unroll
    for (int x = K % P; x + K < N; ++x)
        if ((x - K % P) / K % 2 == 0 && x / (2 * P) == (x + K) / (2 * P)) {
            const unsigned a = v[x], b = v[x + K];
            v[x] = min(a, b);
            v[x + K] = max(a, b);
        }
    if constexpr (K > 1) odd_even_stage<N, P, K / 2>(v);
    else if constexpr (2 * P < N) odd_even_stage<N, 2 * P, 2 * P>(v);
}

constexpr int kSortWarps = 4;
template <int KPL>
__global__ void __launch_bounds__(32 * kSortWarps, WarpSort<KPL>::CTAS) kb_sort_warp(const int* __restrict__ rowptr, const int* __restrict__ col,
                                                                const float* __restrict__ val, int n_rows, int window,
                                                                const int* __restrict__ sel, int count, WindowOut out,
                                                                InputInfo* __restrict__ info) {
    using S = WarpSort<KPL>;
    constexpr int PB = S::PB, LP = S::LP, CAP = S::CAP;
    constexpr unsigned kPad = 0xffffffffu;   // columns have 31 - PB bits at most
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    typename S::Smem& s = reinterpret_cast<typename S::Smem*>(smem_raw)[wid];
    const int which = blockIdx.x * kSortWarps + wid;
    if (which >= count) return;
    const int w = sel[which];
    const int base = rowptr[(size_t)w * window];
    if (lane < 17) s.bound[lane] = rowptr[min((long long)w * window + min(lane, window), (long long)n_rows)] - base;
    __syncwarp();
    const int n = s.bound[16];
    const bool rows_fit = KPL > 8 || __reduce_max_sync(0xffffffffu, lane < 16 ? s.bound[lane + 1] - s.bound[lane] : 0) <= 2 * KPL;
    unsigned v[KPL];
    bool bad = false;
    if (rows_fit) {
#pragma unroll
        for (int i = 0; i < KPL; ++i) {
            const int place = i * 32 + lane, row = place >> LP, e = s.bound[row] + (place & (2 * KPL - 1));
            const bool have = e < s.bound[row + 1];
            const int c = have ? col[base + e] : 0;
            bad |= c < 0;
            v[i] = have ? (unsigned)c << PB | (unsigned)place : kPad;
        }
    } else {
#pragma unroll 4
        for (int i = 0; i < KPL; ++i) {
            const int e = i * 32 + lane;
            unsigned key = kPad;
            if (e < n) {
                const int c = col[base + e];
                int row = 0;
#pragma unroll
                for (int d = 8; d; d >>= 1)
                    if (row + d < window && s.bound[row + d] <= e) row += d;
                s.row[e] = (unsigned char)row;
                key = (unsigned)c << PB | (unsigned)e;
                bad |= c < 0 || (e + 1 < s.bound[row + 1] && col[base + e + 1] <= c);
            }
            s.key[S::at(e)] = key;
        }
    }
    if (rows_fit) {
#pragma unroll
        for (int i = 0; i < KPL; ++i) s.key[S::at(i * 32 + lane)] = v[i];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < KPL; i += 4) {
        const uint4 x = *(const uint4*)(s.key + S::at(lane * KPL + i));
        v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
    }
    if (rows_fit) {   // a row's columns ascend: pairs of neighbours, behind the row's end a pad
#pragma unroll
        for (int i = 0; i + 1 < KPL; ++i) bad |= v[i] != kPad && (v[i] >> PB) >= (v[i + 1] >> PB);
        const unsigned across = __shfl_down_sync(0xffffffffu, v[0], 1);
        bad |= (lane & 1) == 0 && v[KPL - 1] != kPad && (v[KPL - 1] >> PB) >= (across >> PB);
    }
    if (__any_sync(0xffffffffu, bad)) {   // nothing below holds for unsorted rows
        if (lane == 0) atomicOr(&info->err, 2);
        return;
    }
    auto inner = [&]() {   // the last stages of a merge, inside the lanes
#pragma unroll
        for (int d = KPL / 2; d; d >>= 1)
#pragma unroll
            for (int i = 0; i < KPL; ++i)
                if (!(i & d)) {
                    const unsigned a = v[i], b = v[i + d];
                    v[i] = min(a, b);
                    v[i + d] = max(a, b);
                }
    };
    if (!rows_fit) odd_even_stage<KPL, 1, 1>(v);
    // sorted runs of m lanes become runs of 2 m: the first stage pairs a run with the next one backwards, so that all stages ascend
#pragma unroll 1
    for (int m = rows_fit ? 2 : 1; m < 32; m <<= 1) {
        const bool low = !(lane & m);
#pragma unroll
        for (int i = 0; i < KPL / 2; ++i) {
            const unsigned a = v[i], b = v[KPL - 1 - i];
            const unsigned x = __shfl_xor_sync(0xffffffffu, b, 2 * m - 1), y = __shfl_xor_sync(0xffffffffu, a, 2 * m - 1);
            v[i] = (a < x) == low ? a : x;
            v[KPL - 1 - i] = (b < y) == low ? b : y;
        }
#pragma unroll 1
        for (int d = m >> 1; d; d >>= 1) {
            const bool first = !(lane & d);
#pragma unroll
            for (int i = 0; i < KPL; ++i) {
                const unsigned x = __shfl_xor_sync(0xffffffffu, v[i], d);
                v[i] = (v[i] < x) == first ? v[i] : x;
            }
        }
        inner();
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < KPL; i += 4) *(uint4*)(s.key + S::at(lane * KPL + i)) = make_uint4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    // records begin where the column changes
    const int mine = min(max(n - lane * KPL, 0), KPL);
    unsigned rowbit_sum = 0;
    int heads = 0;
    const unsigned last = __shfl_up_sync(0xffffffffu, v[KPL - 1], 1);
    auto is_head = [&](int i) -> bool {
        if (i >= mine) return false;
        if (i == 0) return lane == 0 || (v[0] >> PB) != (last >> PB);
        return (v[i] ^ v[i - 1]) >> PB != 0u;
    };
    auto row_bit = [&](int i) -> unsigned { return 1u << (rows_fit ? (v[i] >> LP) & 15u : (unsigned)s.row[v[i] & (CAP - 1)]); };
#pragma unroll
    for (int i = 0; i < KPL; ++i) {
        heads += is_head(i);
        if (i < mine) rowbit_sum += row_bit(i);
    }
    int r = heads;
    unsigned sum = rowbit_sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, r, d);
        const unsigned z = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) { r += y; sum += z; }
    }
    const int D = __shfl_sync(0xffffffffu, r, 31);
    if (lane == 31) { s.start[D] = (unsigned short)n; s.before[D] = (unsigned short)sum; }
    r -= heads;
    sum -= rowbit_sum;
#pragma unroll
    for (int i = 0; i < KPL; ++i) {
        if (is_head(i)) {
            s.start[r] = (unsigned short)(lane * KPL + i);
            s.before[r] = (unsigned short)sum;
            ++r;
        }
        if (i < mine) sum += row_bit(i);
    }
    __syncwarp();
    auto entry = [&](unsigned key) -> int {   // of the window
        const int place = (int)(key & (CAP - 1));
        return rows_fit ? s.bound[place >> LP] + (place & (2 * KPL - 1)) : place;
    };
#pragma unroll 1
    for (int i0 = lane; i0 < n; i0 += 32 * 8) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = i0 + 32 * i < n ? val[base + entry(s.key[S::at(i0 + 32 * i)])] : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i0 + 32 * i < n) out.sval[base + i0 + 32 * i] = x[i];
    }
    // (count desc, column asc), as in kb_sort_window
    const unsigned lt = (1u << lane) - 1u;
    const int rchunks = (D + 31) / 32, ncells = 16 * rchunks;
    for (int i = lane; i < ncells; i += 32) s.cells[i] = 0;
    __syncwarp();
    for (int c = 0; c < rchunks; ++c) {
        const int q = c * 32 + lane, k = q < D ? 16 - (s.start[q + 1] - s.start[q]) : 16;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k < 16 && (same & lt) == 0) s.cells[k * rchunks + c] = (unsigned short)__popc(same);
    }
    __syncwarp();
    int before = 0;
    for (int c0 = 0; c0 < ncells; c0 += 32) {
        const int i = c0 + lane, x = i < ncells ? s.cells[i] : 0;
        int incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        if (i < ncells) s.cells[i] = (unsigned short)(before + incl - x);
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();
    for (int c = 0; c < rchunks; ++c) {
        const int q = c * 32 + lane, st = q < D ? s.start[q] : 0, k = q < D ? 16 - (s.start[q + 1] - st) : 16;
        const unsigned same = __match_any_sync(0xffffffffu, k);
        if (k == 16) continue;
        const unsigned first = s.key[S::at(st)];
        const size_t o = (size_t)base + s.cells[k * rchunks + c] + __popc(same & lt);
        out.rec[o] = Record{(int)(first >> PB), base + st, (unsigned)(unsigned short)(s.before[q + 1] - s.before[q]), val[base + entry(first)]};
        out.cnt[o] = (unsigned char)(16 - k);
    }
    if (lane == 0) out.ncol[w] = D;
}

// Hub windows: the same through device-wide sorts, keys (hub << col_bits | column), payload the place in the window.
struct HubView {
    const int* sel;   // [H] windows
    const int* off;   // [H + 1] first entry in the compact arrays
    int n;
};
__device__ __forceinline__ int find_hub(const HubView& h, int x) {
    int lo = 0, hi = h.n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (h.off[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}
// local row of an entry: rows of the window that start at or before it
__device__ __forceinline__ int local_row(const int* __restrict__ rowptr, int n_rows, int w, int window, int e) {
    int lo = 0, hi = min(window, n_rows - w * window);
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (rowptr[w * window + mid] <= e) lo = mid; else hi = mid;
    }
    return lo;
}

struct HubSizes {
    const int *rowptr, *sel;
    int n_rows, window, n;
    __host__ __device__ __forceinline__ int operator()(int h) const {
        return h < n ? rowptr[min((long long)(sel[h] + 1) * window, (long long)n_rows)] - rowptr[(size_t)sel[h] * window] : 0;
    }
};

template <class Key>
__global__ void kb_hub_keys(const int* __restrict__ rowptr, const int* __restrict__ col, int n_rows, int window, HubView hub, int E,
                            int col_bits, Key* __restrict__ keys, int* __restrict__ place, InputInfo* __restrict__ info) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= E) return;
    const int h = find_hub(hub, x), w = hub.sel[h];
    const int at = x - hub.off[h], e = rowptr[(size_t)w * window] + at;
    const int c = col[e], r = w * window + local_row(rowptr, n_rows, w, window, e);
    if (c < 0 || (e + 1 < rowptr[r + 1] && col[e + 1] <= c)) atomicOr(&info->err, 2);
    keys[x] = ((Key)h << col_bits) | (Key)(unsigned)max(c, 0);
    place[x] = at;
}

template <class Key>
struct IsHead {
    const Key* keys;
    __device__ __forceinline__ bool operator()(int i) const { return i == 0 || keys[i] != keys[i - 1]; }
};

template <class Key>
__global__ void kb_hub_records(const Key* __restrict__ keys, const int* __restrict__ place, const int* __restrict__ rowptr,
                               const float* __restrict__ val, int n_rows, int window, HubView hub, const int* __restrict__ start,
                               int D, int E, int col_bits, Record* __restrict__ record, unsigned* __restrict__ key2,
                               int* __restrict__ ord, int* __restrict__ first_rec) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= D) return;
    const int b = start[j], e = j + 1 < D ? start[j + 1] : E;
    const int h = (int)(keys[b] >> col_bits), w = hub.sel[h];
    const int base = rowptr[(size_t)w * window];
    unsigned mask = 0;
    for (int i = b; i < e; ++i) mask |= 1u << local_row(rowptr, n_rows, w, window, base + place[i]);
    record[j] = Record{(int)(keys[b] & (((Key)1 << col_bits) - 1)), base + b - hub.off[h], mask, val[base + place[b]]};
    key2[j] = ((unsigned)h << 4) | (unsigned)(16 - (e - b));
    ord[j] = j;
    if (b == hub.off[h]) first_rec[h] = j;
}

__global__ void kb_hub_place(const unsigned* __restrict__ key2, const int* __restrict__ ord, const Record* __restrict__ record, int D,
                             const int* __restrict__ rowptr, int window, HubView hub, const int* __restrict__ first_rec, WindowOut out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= D) return;
    const unsigned k = key2[p];
    const int h = (int)(k >> 4), w = hub.sel[h], o = p - first_rec[h];
    const size_t at = (size_t)rowptr[(size_t)w * window] + o;
    out.rec[at] = record[ord[p]];
    out.cnt[at] = (unsigned char)(16u - (k & 15u));
    if (p + 1 == D || (key2[p + 1] >> 4) != (unsigned)h) out.ncol[w] = o + 1;
}

__global__ void kb_hub_values(const int* __restrict__ place, const int* __restrict__ rowptr, const float* __restrict__ val, int window,
                              HubView hub, int E, float* __restrict__ sval) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= E) return;
    const int h = find_hub(hub, x), base = rowptr[(size_t)hub.sel[h] * window];
    sval[base + x - hub.off[h]] = val[base + place[x]];
}

// ---------------------------------------------------------------------------------------------
// 4., 5. per window: TC columns, units, pair slots, TC blocks, TC parts
// ---------------------------------------------------------------------------------------------
struct Win {          // prefixes over windows (W + 1 of them) after the scan
    int blocks, units, slots, parts;
};
struct WinSum {
    __host__ __device__ __forceinline__ Win operator()(const Win& a, const Win& b) const {
        return Win{a.blocks + b.blocks, a.units + b.units, a.slots + b.slots, a.parts + b.parts};
    }
};
struct WindowView {
    const int* rec;    // [W] first record of the window
    const int* end;    // [W] behind its last one
    const int* tc;     // [W] TC columns: records [rec, rec + tc) in (count desc, column asc) order
    const Win* pre;    // [W + 1]
};

constexpr int kWarpUnits = 2048;    // matching: windows up to here get a warp each,
constexpr int kBlockUnits = 14336;  // up to here a block with 56 KB for the units, beyond a whole SM's memory
constexpr int kSmemUnits = 52224;

struct MatchCounts {
    int n_block, n_huge;
    int max_warp, max_huge;   // units of the largest window of the warp and of the last tier
    u64 records;
};

__global__ void kb_windows(const int* __restrict__ rowptr, const int* __restrict__ ncol, const unsigned char* __restrict__ cnt,
                           int W, BuildCfg cfg, int* __restrict__ rec, int* __restrict__ end, int* __restrict__ tc,
                           Win* __restrict__ win, int* __restrict__ sel_block, int* __restrict__ sel_huge,
                           MatchCounts* __restrict__ mc) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = w < W ? ncol[w] : 0;
    const int sum = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&mc->records, (u64)sum);
    if (w > W) return;
    if (w == W) { win[W] = Win{0, 0, 0, 0}; return; }
    const int b = rowptr[(size_t)w * cfg.window];
    rec[w] = b;
    end[w] = b + n;
    auto count = [&](int o) -> int { return cnt[b + o]; };  // o-th largest column
    int cand = 0;
    if (!cfg.skip_tc) {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if (count(mid) >= cfg.density) lo = mid + 1; else hi = mid;
        }
        cand = lo;
    }
    int lo = 0, hi = (cand + 7) / 8;  // chunks kept
    while (lo < hi) {
        const int mid = lo + (hi - lo) / 2;
        int nnz = 0;
        for (int o = mid * 8; o < min(mid * 8 + 8, cand); ++o) nnz += count(o);
        const float util = __fdiv_rn((float)nnz, (float)(cfg.window * 8));
        if (!(util < cfg.tc_min_util)) lo = mid + 1; else hi = mid;
    }
    const int t = min(lo * 8, cand);
    const int units = (n - t + 1) / 2;
    tc[w] = t;
    win[w] = Win{lo, units, (units + 1) / 2, lo == 0 ? 0 : (lo + cfg.part_t - 1) / cfg.part_t};
    if (units > kBlockUnits) { sel_huge[atomicAdd(&mc->n_huge, 1)] = w; atomicMax(&mc->max_huge, units); }
    else if (units > kWarpUnits) sel_block[atomicAdd(&mc->n_block, 1)] = w;
    else if (units > mc->max_warp) atomicMax(&mc->max_warp, units);
}

__device__ __forceinline__ int find_window(const int* __restrict__ prefix, int W, int x) {
    // largest w in [0, W) with prefix[w] <= x   (prefix non-decreasing, prefix[W] > x)
    int lo = 0, hi = W;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= x) lo = mid; else hi = mid;
    }
    return lo;
}

// ---------------------------------------------------------------------------------------------
// 6. matching of a window's units
// ---------------------------------------------------------------------------------------------
// A unit is one word: nnz << 26 | index, so that the sort touches one array (in shared memory for
// all but enormous windows: every step of the sort and of the greedy pass is a dependent access, and
// from L2 each cost ten times as much).  The order of equal keys is libstdc++'s, reproduced as follows.
//   * Partition (Hoare, unguarded): the k-th element >= pivot from the left swaps with the k-th element
//     <= pivot from the right while the former lies left of the latter; the cut is
//     min(next left stopper, last swapped right position).  A warp finds the stoppers 32 at a time.
//   * A range of equal keys - most of a hub window - is not sorted at all: there each partition moves
//     the middle element to the front and reverses the rest, so every position can be traced back
//     through the log2(n / 16) levels on its own.
//   * Ranges of at most 16 are finished by one lane each (insertion sort), 32 at a time.
// The result goes to order_out as unit indices.
constexpr unsigned kUnitBits = 26;
constexpr unsigned kUnitMask = (1u << kUnitBits) - 1u;

struct UnitWordLess {
    __host__ __device__ bool operator()(int a, int b) const { return ((unsigned)a >> kUnitBits) > ((unsigned)b >> kUnitBits); }
};
__device__ __forceinline__ unsigned unit_key(int word) { return (unsigned)word >> kUnitBits; }

// Where introsort puts the element at position s of a range of n > 16 equal keys: every partition brings the middle one to
// the front and reverses the rest.
__device__ __forceinline__ int equal_range_target(int n, int s) {
    int f = 0, l = n;
    while (l - f > 16) {
        const int mid = f + (l - f) / 2, cut = f + 1 + (l - f - 1) / 2;
        s = s == mid ? f : f + l - (s == f ? mid : s);
        if (s < cut) l = cut; else f = cut;
    }
    return s;
}
__device__ __forceinline__ int equal_range_depth(int n) {  // partitions on the longest path
    int d = 0;
    for (; n > 16; ++d) n = max(1 + (n - 1) / 2, n - 1 - (n - 1) / 2);
    return d;
}

// One warp partitions [first, last) of a as introsort does (median of three to the front included);
// `sl` / `sr`: 32 ints of shared memory each.
__device__ __forceinline__ int warp_partition(int* a, int first, int last, int* sl, int* sr, int lane) {
    const int mid = first + (last - first) / 2;
    const int vf = a[first], va = a[first + 1], vb = a[mid], vc = a[last - 1];
    const unsigned ka = unit_key(va), kb = unit_key(vb), kc = unit_key(vc);
    const int median = ka > kb ? (kb > kc ? mid : ka > kc ? last - 1 : first + 1) : (ka > kc ? first + 1 : kb > kc ? last - 1 : mid);
    const int vm = median == first + 1 ? va : median == mid ? vb : vc;
    __syncwarp();
    if (lane == 0) { a[first] = vm; a[median] = vf; }
    __syncwarp();
    const unsigned pv = unit_key(vm);
    const unsigned lt = (1u << lane) - 1u;
    int lb = first + 1 - 32, rb = last - 1 + 32;  // the blocks start at lb (upwards) and rb (downwards)
    unsigned lm = 0, rm = 0;                       // stoppers of the blocks not used yet
    int last_r = 0x7fffffff;                       // right position of the last swap
    while (true) {
        while (lm == 0) {
            lb += 32;
            if (lb >= last) break;
            const int i = lb + lane;
            lm = __ballot_sync(0xffffffffu, i < last && unit_key(a[i]) <= pv);
        }
        while (rm == 0) {
            rb -= 32;
            if (rb <= first) break;
            const int i = rb - lane;
            rm = __ballot_sync(0xffffffffu, i > first && unit_key(a[i]) >= pv);
        }
        if (lm == 0 || rm == 0) break;
        const int t = min(__popc(lm), __popc(rm));
        if ((lm >> lane) & 1u) sl[__popc(lm & lt)] = lb + lane;
        if ((rm >> lane) & 1u) sr[__popc(rm & lt)] = rb - lane;
        __syncwarp();
        int pl = 0, pr = 0;
        bool ok = false;
        if (lane < t) {
            pl = sl[lane]; pr = sr[lane];
            ok = pl < pr;
        }
        const int n_ok = __popc(__ballot_sync(0xffffffffu, ok));
        if (ok) { const int x = a[pl]; a[pl] = a[pr]; a[pr] = x; }
        if (n_ok > 0) last_r = __shfl_sync(0xffffffffu, pr, n_ok - 1);
        __syncwarp();
        if (n_ok < t) return min(sl[n_ok], last_r);  // sl[n_ok]: the next left stopper
        // drop the t lowest bits of both masks
        const bool keep_l = ((lm >> lane) & 1u) && __popc(lm & lt) >= t;
        const bool keep_r = ((rm >> lane) & 1u) && __popc(rm & lt) >= t;
        lm = __ballot_sync(0xffffffffu, keep_l);
        rm = __ballot_sync(0xffffffffu, keep_r);
    }
    const int next_l = lm ? lb + __ffs(lm) - 1 : 0x7fffffff;
    return min(next_l, last_r);
}

struct SortRange {
    int first, last, depth;
};

// Introsort of a[first, first + n), n <= 32, by one warp, an element per lane; unit indices to out[first ..).  The stoppers
// of a partition and their partners are counted in ballots.  What is left below 17 elements the library insertion-sorts,
// which is stable and never crosses a cut, so the whole range ends up stably sorted: an element's place is the number of
// larger keys and of equal ones before it, from one ballot per bit.  In shared memory a partition takes some 700 cycles
// whatever its length, and most are of this length (matching of the clustered graph 130 -> 100 us with the pairs below).
__device__ void warp_sort_lanes(int* a, int* __restrict__ out, int first, int n, int depth, int* sl, int* sr, int lane) {
    int v = lane < n ? a[first + lane] : 0;
    const unsigned lt = (1u << lane) - 1u, gt = ~lt << 1;
    for (int f = 0, l = n; l - f > 16;) {
        if (depth == 0) {
            if (lane < n) a[first + lane] = v;
            __syncwarp();
            if (lane == 0) StdSort<UnitWordLess>(a, UnitWordLess()).heap_sort(first + f, l - f);
            __syncwarp();
            if (lane < n) v = a[first + lane];
            break;
        }
        --depth;
        const int pa = f + 1, pb = f + (l - f) / 2, pc = l - 1;
        const unsigned ka = unit_key(__shfl_sync(0xffffffffu, v, pa)), kb = unit_key(__shfl_sync(0xffffffffu, v, pb)),
                       kc = unit_key(__shfl_sync(0xffffffffu, v, pc));
        const int median = ka > kb ? (kb > kc ? pb : ka > kc ? pc : pa) : (ka > kc ? pa : kb > kc ? pc : pb);
        const int vf = __shfl_sync(0xffffffffu, v, f), vm = __shfl_sync(0xffffffffu, v, median);
        if (lane == f) v = vm;
        if (lane == median) v = vf;
        const unsigned key = unit_key(v), pivot = unit_key(vm);
        const bool in = lane > f && lane < l, is_l = in && key <= pivot, is_r = in && key >= pivot;
        const unsigned lm = __ballot_sync(0xffffffffu, is_l), rm = __ballot_sync(0xffffffffu, is_r);
        const int rl = __popc(lm & lt), rr = __popc(rm & gt);   // ranks, from the left and from the right
        const int swaps = __popc(__ballot_sync(0xffffffffu, is_l && rr > rl));
        const bool swap_l = is_l && rl < swaps, swap_r = is_r && rr < swaps;
        if (swap_l) sl[rl] = lane;
        if (swap_r) sr[rr] = lane;
        __syncwarp();
        const int partner = swap_l ? sr[rl] : swap_r ? sl[rr] : lane;
        v = __shfl_sync(0xffffffffu, v, partner);
        const unsigned next_l = __ballot_sync(0xffffffffu, is_l && rl >= swaps), last_r = __ballot_sync(0xffffffffu, swap_r);
        const int cut = min(next_l ? __ffs(next_l) - 1 : 32, last_r ? __ffs(last_r) - 1 : 32);
        if (l - cut > cut - f) f = cut; else l = cut;   // at most one side has more than 16
    }
    const unsigned key = unit_key(v);
    unsigned eq = n < 32 ? (1u << n) - 1u : 0xffffffffu, larger = 0;
#pragma unroll
    for (int b = 31 - kUnitBits; b >= 0; --b) {
        const bool one = (key >> b) & 1u;
        const unsigned ones = __ballot_sync(0xffffffffu, one);
        if (!one) larger |= eq & ones;
        eq &= one ? ones : ~ones;
    }
    if (lane < n) out[first + __popc(larger) + __popc(eq & lt)] = v & (int)kUnitMask;
    __syncwarp();
}

// Introsort of a[first0, last0) by one warp; unit indices to out[first0, last0).
// `stack`: 40 ranges, `sl`, `sr`: 32 ints, all in shared memory and this warp's own.
__device__ void warp_introsort(int* a, int* __restrict__ out, int first0, int last0, int depth0, SortRange* stack, int* sl,
                               int* sr, int lane) {
    int sp = 0;
    int first = first0, last = last0, depth = depth0;
    StdSort<UnitWordLess> S(a, UnitWordLess());
    while (true) {
        const int n = last - first;
        bool done = false;
        if (n <= 32) {
            warp_sort_lanes(a, out, first, n, depth, sl, sr, lane);
            done = true;
        } else {
            const unsigned k0 = unit_key(a[first]);
            bool equal = false;
            if (k0 == unit_key(a[last - 1]) && k0 == unit_key(a[first + n / 2]) && depth >= equal_range_depth(n)) {
                equal = true;
                for (int i = first + lane; i - lane < last; i += 32)
                    if (__ballot_sync(0xffffffffu, i < last && unit_key(a[i]) != k0)) { equal = false; break; }
            }
            if (equal) {
                for (int i = lane; i < n; i += 32) out[first + equal_range_target(n, i)] = a[first + i] & (int)kUnitMask;
                done = true;
            } else if (depth == 0) {
                if (lane == 0) S.heap_sort(first, n);
                __syncwarp();
                for (int i = first + lane; i < last; i += 32) out[i] = a[i] & (int)kUnitMask;
                done = true;
            }
        }
        if (done) {
            if (sp == 0) break;
            --sp;
            __syncwarp();
            first = stack[sp].first; last = stack[sp].last; depth = stack[sp].depth;
            continue;
        }
        const int cut = warp_partition(a, first, last, sl, sr, lane);
        --depth;
        // the longer part waits, so that the stack stays short
        const bool right_first = last - cut < cut - first;
        if (lane == 0) stack[sp] = right_first ? SortRange{first, cut, depth} : SortRange{cut, last, depth};
        ++sp;
        __syncwarp();
        if (right_first) first = cut; else last = cut;
    }
}

// Greedy pass over the sorted order (block_online.cpp:365-386) by one warp.  The next unmatched unit of the
// order is paired with the lowest unmatched unit, again and again.  Two windows of 32 are open at a
// time: entries of the order (`alive`: still unmatched) and the bitmask word of the lowest unmatched units
// (`cur`).  While no alive entry lies in that word the two are independent, and the k-th alive entry
// simply gets the k-th free bit; otherwise the pairs are made one by one until the word or the entries are used up.
// `freem`: a bit per unmatched unit, `sl`: 32 ints of shared memory.  Returns the number of pairs; *left: the
// unit that stays alone (-1: none).
__device__ __forceinline__ int warp_greedy(int U, unsigned* freem, const int* order, int* __restrict__ pa, int* __restrict__ pb,
                                           int* sl, int lane, int* left) {
    const int words = (U + 31) / 32;
    const unsigned lt = (1u << lane) - 1u;
    int wpos = 0, G = 0;
    unsigned cur = U > 0 ? freem[0] : 0u;
    *left = -1;
    auto advance = [&]() {   // to the next word with an unmatched unit; cur = 0: there is none
        __syncwarp();
        for (wpos += 1; wpos < words; wpos += 32) {
            const unsigned f = wpos + lane < words ? freem[wpos + lane] : 0u;
            const unsigned some = __ballot_sync(0xffffffffu, f != 0);
            if (!some) continue;
            const int at = __ffs(some) - 1;
            wpos += at;
            cur = __shfl_sync(0xffffffffu, f, at);
            return;
        }
    };
    int next = lane < U ? order[lane] : -1;
    for (int k0 = 0; k0 < U; k0 += 32) {
        const int idx = next;
        next = k0 + 32 + lane < U ? order[k0 + 32 + lane] : -1;
        __syncwarp();
        const int word = idx >> 5;
        unsigned f = 0;   // units in words before wpos are all matched
        if (idx >= 0 && word >= wpos) f = word == wpos ? cur : freem[word];
        unsigned alive = __ballot_sync(0xffffffffu, (f >> (idx & 31)) & 1u);
        while (alive) {
            if (cur == 0) advance();
            const bool mine = (alive >> lane) & 1u;
            if (__ballot_sync(0xffffffffu, mine && word == wpos) == 0) {
                const int t = min(__popc(alive), __popc(cur));
                const int ra = __popc(alive & lt), rb = __popc(cur & lt);
                const bool bit = (cur >> lane) & 1u;
                if (bit) sl[rb] = lane;
                __syncwarp();
                if (mine && ra < t) {
                    pa[G + ra] = idx;
                    pb[G + ra] = wpos * 32 + sl[ra];
                    atomicAnd(freem + word, ~(1u << (idx & 31)));
                }
                G += t;
                alive = __ballot_sync(0xffffffffu, mine && ra >= t);
                cur = __ballot_sync(0xffffffffu, bit && rb >= t);
                continue;
            }
            // units of the lowest free word are among the next alive ones: pair by pair, in registers (80 cycles a pair; with
            // the free words updated in shared memory 390).  Lane i knows which bit of the word its unit is, lane b which
            // alive unit bit b is; lane p keeps the p-th pair.
            const unsigned drop_bit = mine && word == wpos ? 1u << (idx & 31) : 0u;
            sl[lane] = -1;
            __syncwarp();
            if (drop_bit) sl[idx & 31] = lane;
            __syncwarp();
            const int at = sl[lane];
            const unsigned drop_lane = at >= 0 ? 1u << at : 0u;
            int px = 0, py = 0, n = 0;
            bool waits = false;   // the last unit taken from the order finds its partner in a later word
            while (alive) {
                const int i = __ffs(alive) - 1;
                alive &= alive - 1;
                cur &= ~__shfl_sync(0xffffffffu, drop_bit, i);
                if (lane == n) px = i;
                if (cur == 0) { waits = true; break; }
                const int y = __ffs(cur) - 1;
                cur &= cur - 1;
                alive &= ~__shfl_sync(0xffffffffu, drop_lane, y);
                if (lane == n) py = y;
                ++n;
                if (cur == 0) break;
            }
            const int x = __shfl_sync(0xffffffffu, idx, px);
            if (lane < n + waits) {
                if ((x >> 5) != wpos) atomicAnd(freem + (x >> 5), ~(1u << (x & 31)));
                pa[G + lane] = x;
                if (lane < n) pb[G + lane] = wpos * 32 + py;
            }
            G += n;
            if (waits) {
                advance();
                const int alone = __shfl_sync(0xffffffffu, x, n);
                if (cur == 0) { *left = alone; return G; }
                const int y = wpos * 32 + __ffs(cur) - 1;
                cur &= cur - 1;
                alive &= ~__ballot_sync(0xffffffffu, idx == y);
                if (lane == 0) pb[G] = y;
                ++G;
            }
        }
    }
    return G;
}

struct MatchOut {
    int* order;       // [units] scratch: sorted unit indices
    int* pair_a;      // [slots] groups in emission order: matched pairs, then the unmatched unit if it is kept
    int* pair_b;
    int* groups;      // [W + 1]
    int* cuda_unit;   // [W] unmatched unit that goes to the CUDA cores, -1: none
};

__device__ __forceinline__ int unit_word(const unsigned char* __restrict__ cnt, int rec0, int ncol, int u) {
    int nnz = cnt[rec0 + 2 * u];
    if (2 * u + 1 < ncol) nnz += cnt[rec0 + 2 * u + 1];
    return (int)(((unsigned)nnz << kUnitBits) | (unsigned)u);
}

__device__ __forceinline__ void match_finish(int w, int G, int left, int left_nnz, int unit_min_nnz, const MatchOut& o, int slot0) {
    int cuda = -1;
    if (left >= 0) {
        if (left_nnz >= unit_min_nnz) { o.pair_a[slot0 + G] = left; o.pair_b[slot0 + G] = -1; ++G; }
        else cuda = left;
    }
    o.groups[w] = G;
    o.cuda_unit[w] = cuda;
}

constexpr int kMatchWarps = 4;
struct MatchWarpSmem {
    SortRange stack[40];
    int sl[32], sr[32];
};

// Windows of at most `max_units` units, one warp each.  Dynamic shared memory: per warp max_units words
// and the bitmask.
__global__ void __launch_bounds__(32 * kMatchWarps) kb_match_warp(WindowView v, int W, const unsigned char* __restrict__ cnt,
                                                                  int unit_min_nnz, int max_units, MatchOut o) {
    extern __shared__ int dyn[];
    __shared__ MatchWarpSmem s_warp[kMatchWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int w = blockIdx.x * kMatchWarps + wid;
    if (w > W) return;
    if (w == W) { if (lane == 0) { o.groups[W] = 0; } return; }
    const Win p0 = v.pre[w];
    const int U = v.pre[w + 1].units - p0.units;
    if (U > max_units) return;
    const int rec0 = v.rec[w] + v.tc[w], ncol = v.end[w] - rec0;
    int* a = dyn + wid * (max_units + (max_units + 31) / 32);
    unsigned* freem = (unsigned*)(a + max_units);
    int* order = o.order + p0.units;
    for (int i = lane; i < U; i += 32) a[i] = unit_word(cnt, rec0, ncol, i);
    for (int i = lane; i < (U + 31) / 32; i += 32) freem[i] = U - 32 * i >= 32 ? 0xffffffffu : (1u << (U - 32 * i)) - 1u;
    __syncwarp();
    MatchWarpSmem& m = s_warp[wid];
    // units come in descending order already: an insertion sort of at most 16 of them moves nothing
    if (U > 16) {
        warp_introsort(a, order, 0, U, 2 * StdSort<UnitWordLess>::floor_log2(U), m.stack, m.sl, m.sr, lane);
    } else if (lane < U) {
        order[lane] = lane;
    }
    __syncwarp();   // `order` is read back by the lanes of the warp that wrote it
    int left;
    const int G = warp_greedy(U, freem, order, o.pair_a + p0.slots, o.pair_b + p0.slots, m.sl, lane, &left);
    if (lane == 0) match_finish(w, G, left, left >= 0 ? (int)unit_key(unit_word(cnt, rec0, ncol, left)) : 0, unit_min_nnz, o, p0.slots);
}

// Hub windows, one block each: long ranges are partitioned or traced by the whole block, ranges of
// at most kWarpRange units are left to single warps.  The words live in dynamic shared memory when
// they fit (smem_units), in `words_global` otherwise; the bitmask takes the same memory afterwards
// (or `mask_global`).
constexpr int kBlockThreads = 512, kWarpRange = 1024, kMaxRanges = 256;

__global__ void __launch_bounds__(kBlockThreads) kb_match_block(WindowView v, const unsigned char* __restrict__ cnt, int unit_min_nnz,
                                                                int smem_units, int* __restrict__ words_global,
                                                                unsigned* __restrict__ mask_global, const int* __restrict__ sel,
                                                                MatchOut o) {
    extern __shared__ int dyn[];
    __shared__ MatchWarpSmem s_warp[kBlockThreads / 32];
    __shared__ SortRange s_stack[64], s_small[kMaxRanges];
    __shared__ int s_scan[kBlockThreads / 32];
    __shared__ int s_sp, s_nsmall, s_take, s_lnext;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int w = sel[blockIdx.x];
    const Win p0 = v.pre[w];
    const int U = v.pre[w + 1].units - p0.units;
    const int rec0 = v.rec[w] + v.tc[w], ncol = v.end[w] - rec0;
    const bool in_smem = U <= smem_units;
    int* a = in_smem ? dyn : words_global + p0.units;
    int* order = o.order + p0.units;
    int* swapL = o.pair_a + p0.slots;   // scratch during the sort, pair list afterwards
    int* swapR = o.pair_b + p0.slots;
    for (int i = tid; i < U; i += kBlockThreads) a[i] = unit_word(cnt, rec0, ncol, i);
    if (tid == 0) {
        s_stack[0] = SortRange{0, U, 2 * StdSort<UnitWordLess>::floor_log2(U)};
        s_sp = 1; s_nsmall = 0;
    }
    __syncthreads();
    StdSort<UnitWordLess> S(a, UnitWordLess());

    auto block_excl_scan = [&](int x, int& total) -> int {
        int incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        if (lane == 31) s_scan[wid] = incl;
        __syncthreads();
        int before = 0;
        total = 0;
#pragma unroll
        for (int q = 0; q < kBlockThreads / 32; ++q) {
            if (q < wid) before += s_scan[q];
            total += s_scan[q];
        }
        __syncthreads();
        return before + incl - x;
    };
    auto run_small = [&]() {   // the warps take the waiting ranges one after the other
        __syncthreads();
        if (tid == 0) s_take = 0;
        __syncthreads();
        const int n = s_nsmall;
        while (true) {
            int q = 0;
            if (lane == 0) q = atomicAdd(&s_take, 1);
            q = __shfl_sync(0xffffffffu, q, 0);
            if (q >= n) break;
            const SortRange r = s_small[q];
            warp_introsort(a, order, r.first, r.last, r.depth, s_warp[wid].stack, s_warp[wid].sl, s_warp[wid].sr, lane);
        }
        __syncthreads();
        if (tid == 0) s_nsmall = 0;
        __syncthreads();
    };

    while (true) {
        __syncthreads();
        const int sp = s_sp;
        if (sp == 0) break;
        const SortRange r = s_stack[sp - 1];
        __syncthreads();
        const int first = r.first, last = r.last, n = last - first;
        if (n <= kWarpRange) {
            if (tid == 0) { s_small[s_nsmall++] = r; s_sp = sp - 1; }
            __syncthreads();
            if (s_nsmall == kMaxRanges) run_small();
            continue;
        }
        const unsigned k0 = unit_key(a[first]);
        const bool maybe_equal = k0 == unit_key(a[last - 1]) && k0 == unit_key(a[first + n / 2]) && r.depth >= equal_range_depth(n);
        __syncthreads();   // everyone has looked before anything moves
        if (maybe_equal) {
            int differ = 0;
            for (int i = first + tid; i < last; i += kBlockThreads) differ |= unit_key(a[i]) != k0;
            if (!__syncthreads_or(differ)) {
                for (int i = tid; i < n; i += kBlockThreads) order[first + equal_range_target(n, i)] = a[first + i] & (int)kUnitMask;
                if (tid == 0) s_sp = sp - 1;
                continue;
            }
        }
        if (r.depth == 0) {
            if (tid == 0) { S.heap_sort(first, n); s_sp = sp - 1; }
            __syncthreads();
            for (int i = first + tid; i < last; i += kBlockThreads) order[i] = a[i] & (int)kUnitMask;
            continue;
        }
        if (tid == 0) S.move_median_to_first(first, first + 1, first + n / 2, last - 1);
        __syncthreads();
        const unsigned pvk = unit_key(a[first]);
        const int lo = first + 1, m = last - lo;
        const int chunk = ((m + kBlockThreads - 1) / kBlockThreads) | 1;   // odd: the threads read from different banks
        const int cb = min(lo + tid * chunk, last), ce = min(cb + chunk, last);
        // pass 1: stoppers per chunk (left: key <= pivot, right: key >= pivot)
        int cL = 0, cR = 0;
        for (int i = cb; i < ce; ++i) {
            const unsigned k = unit_key(a[i]);
            cL += (k <= pvk);
            cR += (k >= pvk);
        }
        int totL, totR;
        const int baseL = block_excl_scan(cL, totL);
        const int exR = block_excl_scan(cR, totR);
        const int baseRright = totR - exR - cR;   // right stoppers in later chunks
        // pass 2a: which left stoppers swap; K = their number
        int lrank = baseL, rem = cR, myswaps = 0;
        for (int i = cb; i < ce; ++i) {
            const unsigned k = unit_key(a[i]);
            int right_of_i = baseRright + rem;
            if (k >= pvk) { right_of_i -= 1; rem -= 1; }
            if (k <= pvk) {
                ++lrank;
                if (right_of_i >= lrank) { swapL[lrank - 1] = i; ++myswaps; }
            }
        }
        int K;
        (void)block_excl_scan(myswaps, K);
        if (tid == 0) s_lnext = 0x7fffffff;
        __syncthreads();
        // pass 2b: the partners on the right, and the (K+1)-th left stopper
        lrank = baseL; rem = cR;
        for (int i = cb; i < ce; ++i) {
            const unsigned k = unit_key(a[i]);
            if (k >= pvk) {
                const int rrank = baseRright + rem;   // rank from the right, 1-based
                if (rrank <= K) swapR[rrank - 1] = i;
                rem -= 1;
            }
            if (k <= pvk) {
                ++lrank;
                if (lrank == K + 1) s_lnext = i;
            }
        }
        __syncthreads();
        if (tid == 0) {
            const int cut = min(s_lnext, K >= 1 ? swapR[K - 1] : 0x7fffffff);
            s_stack[sp - 1] = SortRange{cut, last, r.depth - 1};
            s_stack[sp] = SortRange{first, cut, r.depth - 1};
            s_sp = sp + 1;
        }
        for (int k0 = tid; k0 < K; k0 += 4 * kBlockThreads) {   // four pairs' loads under way
            int x[4], y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int k = k0 + j * kBlockThreads;
                x[j] = k < K ? swapL[k] : -1;
                y[j] = k < K ? swapR[k] : -1;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (x[j] >= 0) { const int t = a[x[j]]; a[x[j]] = a[y[j]]; a[y[j]] = t; }
        }
    }
    run_small();

    // the bitmask: in shared memory up to 32 * smem_units units
    const int words = (U + 31) / 32;
    unsigned* gmask = mask_global + p0.units / 32 + w;
    const bool mask_in_smem = words <= smem_units;
    for (int i = tid; i < words; i += kBlockThreads) {
        const unsigned all = U - 32 * i >= 32 ? 0xffffffffu : (1u << (U - 32 * i)) - 1u;
        if (mask_in_smem) dyn[i] = (int)all; else gmask[i] = all;
    }
    __syncthreads();
    if (wid > 0) return;
    int left;
    const int G = mask_in_smem ? warp_greedy(U, (unsigned*)dyn, order, swapL, swapR, s_warp[0].sl, lane, &left)
                               : warp_greedy(U, gmask, order, swapL, swapR, s_warp[0].sl, lane, &left);
    if (lane == 0) match_finish(w, G, left, left >= 0 ? (int)unit_key(unit_word(cnt, rec0, ncol, left)) : 0, unit_min_nnz, o, p0.slots);
}

// ---------------------------------------------------------------------------------------------
// 7. groups and tiles
// ---------------------------------------------------------------------------------------------
struct __align__(8) GroupsTiles {   // of a window, scanned together
    int groups, tiles;
};
struct GroupsTilesSum {
    __host__ __device__ __forceinline__ GroupsTiles operator()(const GroupsTiles& a, const GroupsTiles& b) const {
        return GroupsTiles{a.groups + b.groups, a.tiles + b.tiles};
    }
};
struct WithTiles {
    __host__ __device__ __forceinline__ GroupsTiles operator()(int groups) const { return GroupsTiles{groups, (groups + 3) / 4}; }
};
struct GroupsFrom {
    const int* groups;
    __device__ __forceinline__ GroupsTiles operator()(int i) const { return WithTiles()(groups[i]); }
};
struct GroupsTo {
    int *groups, *tiles;
    __device__ __forceinline__ void operator()(int i, const GroupsTiles& x) const { groups[i] = x.groups; tiles[i] = x.tiles; }
};
struct ToTuple {
    __host__ __device__ __forceinline__ thrust::tuple<int, int> operator()(const GroupsTiles& g) const { return {g.groups, g.tiles}; }
};

struct __align__(16) TileSource {   // where a tile's columns come from
    int slot;    // of its first group in the pair lists
    int rec;     // first record of the window that is in a unit
    int ncol;    // how many of them
    int groups;  // of the tile, 1 .. 4
};
__global__ void kb_tiles(const int* __restrict__ tile_off, const int* __restrict__ s_offset, WindowView v, int W, int T,
                         int* __restrict__ s_tile_window, int* __restrict__ s_tile_group, TileSource* __restrict__ source) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int w = find_window(tile_off, W, t), first = 4 * (t - tile_off[w]);
    s_tile_window[t] = w;
    s_tile_group[t] = s_offset[w] + first;
    const int rec = v.rec[w] + v.tc[w];
    source[t] = TileSource{v.pre[w].slots + first, rec, v.end[w] - rec, min(4, s_offset[w + 1] - s_offset[w] - first)};
}

struct RecordView {
    const Record* rec;
    const float* sval;
    // value of the record's k-th entry (most records of a power-law graph have one)
    __device__ __forceinline__ float value(int start, float first, int k) const { return k == 0 ? first : sval[start + k]; }
};

struct GroupOut {
    int* s_column;
    unsigned char* s_mask;
    float* s_value;
    signed char* s_pos;
    int* s_window;
    int* s_tile_column;
    uint32_t* packed_a;
    uint32_t* packed_meta;
};

// Non-zeros beyond the second one of a row inside a group, which the reference drops: counted, and
// in strict mode recorded (key = row << 32 | column) so that they can join the row's CUDA-core part.
constexpr int kDropCounters = 64;
struct ExtraOut {
    u64* count; // strict: length of the list; otherwise kDropCounters counters, one per block number modulo
    u64* key;
    int* at;    // place in sval
};

// One warp per tile of four groups: lane (q, g) = (lane / 8, lane % 8) owns rows g and g + 8 of group q,
// which are also the two rows of its word pair in the packed tile.  One pass writes the un-packed arrays
// (196 bytes per group) and the tile (352 bytes).  A record is the end of a chain of three loads of up to a thousand
// cycles each: with a tile per warp they were two thirds of its time (clustered graph: 159 us), so a warp works on many
// tiles and has the source of the tile after the next, the units of the next and its records under way (106 us).  Few
// instructions matter too: the four records of a group
// are loaded by one lane each, ranked by column with three shuffles and read back from shared memory by
// position; the positions of a row's first two entries, and the tile's metadata for them, come from tables
// indexed by the row's occupancy pattern.  With all four records in every lane's registers, sorted by a network
// and picked by selects, a tile took 590 instructions instead of 320 (clustered graph: 270 against 159 us).
constexpr unsigned kFirstPos = 0x12131210u;          // 2 bits per pattern: position of the first entry
constexpr unsigned kSecondPos = 0x6b7c6840u;         // of the second
constexpr u64 kTilePos = 0x498e4dcc49884444ull;      // 4 bits: p0 | p1 << 2, the tile's two kept positions p0 < p1 (a
                                                     // missing entry gets a position holding 0.0)
constexpr unsigned kLoneLater = 0x114u;              // patterns with one entry, not in position 0: it is the second kept one

template <bool STRICT>
__global__ void __launch_bounds__(256) kb_emit_tiles(const TileSource* __restrict__ source, RecordView r,
                                                     const int* __restrict__ tile_window, const int* __restrict__ tile_group,
                                                     int T, int window, const int* __restrict__ pair_a,
                                                     const int* __restrict__ pair_b, GroupOut o, ExtraOut x) {
    // strict mode: a warp's extras wait in shared memory for a common place in the list (a tile has at
    // most 128; one atomic per tile on the one counter would be the slowest part)
    constexpr int kWait = STRICT ? 256 : 1;
    __shared__ u64 s_key[8][kWait];
    __shared__ int s_at[8][kWait];
    __shared__ Record s_rec[8][4][4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, q = lane >> 3, g = lane & 7;
    int waiting = 0;
    auto flush = [&]() {
        __syncwarp();
        u64 at = 0;
        if (lane == 0) at = atomicAdd(x.count, (u64)waiting);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int i = lane; i < waiting; i += 32) { x.key[at + i] = s_key[wid][i]; x.at[at + i] = s_at[wid][i]; }
        waiting = 0;
        __syncwarp();
    };
    int dropped = 0;
    const int step = gridDim.x * 8;
    auto source_of = [&](int t) -> int4 { return t < T ? __ldg((const int4*)source + t) : make_int4(0, 0, 0, 0); };
    // lane g < 4 brings one of its group's columns
    auto unit_of = [&](const int4& at) -> int { return g < 4 && q < at.w ? (g < 2 ? pair_a : pair_b)[at.x + q] : -1; };
    auto record_of = [&](const int4& at, int u) -> Record {
        const int ls = 2 * u + (g & 1);
        return u >= 0 && ls < at.z ? r.rec[at.y + ls] : Record{0x7fffffff, 0, 0u, 0.f};
    };
    int t = blockIdx.x * 8 + wid;
    int4 at0 = source_of(t), at1 = source_of(t + step), at2 = source_of(t + 2 * step);
    Record next = record_of(at0, unit_of(at0));
    int u1 = unit_of(at1);
    for (; t < T; t += step) {
        const int w = tile_window[t], gid = tile_group[t] + q;
        const bool live = q < at0.w;
        Record c = next;
        next = record_of(at1, u1);
        u1 = unit_of(at2);
        at0 = at1;
        at1 = at2;
        at2 = source_of(t + 3 * step);
        int rank = 0;
#pragma unroll
        for (int i = 1; i < 4; ++i) {
            const int other = __shfl_xor_sync(0xffffffffu, c.col, i);
            rank += other < c.col || (other == c.col && (g ^ i) < g);
        }
        if (g < 4) {
            if (c.mask == 0u) c.col = -1;
            s_rec[wid][q][rank] = c;
        }
        __syncwarp();
        const Record* const group = s_rec[wid][q];
        // occupancy of rows g (low byte) and g + 8
        unsigned both = 0;
#pragma unroll
        for (int p = 0; p < 4; ++p) both |= ((group[p].mask >> g) & 0x101u) << p;
        uint32_t meta = 0, word[2];
        int n_extra = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int lr = g + 8 * h;
            const unsigned bits = (both >> (8 * h)) & 15u, below = (1u << lr) - 1u;
            const int slots = __popc(bits);
            dropped += max(slots - 2, 0);
            const int p0 = (kFirstPos >> (2 * bits)) & 3, p1 = (kSecondPos >> (2 * bits)) & 3;
            const Record a = group[p0], b = group[p1];
            const int ka = __popc(a.mask & below), kb = __popc(b.mask & below);
            float va = slots > 0 ? a.value : 0.f, vb = slots > 1 ? b.value : 0.f;
            if (slots > 0 && ka) va = r.sval[a.start + ka];
            if (slots > 1 && kb) vb = r.sval[b.start + kb];
            if constexpr (STRICT) n_extra |= (int)(((bits & (bits - 1u)) & ((bits & (bits - 1u)) - 1u)) >> 2) << (2 * h);
            if (live && lr < window) {
                const size_t i = (size_t)gid * window + lr;
                o.s_mask[i] = (unsigned char)bits;
                *(float2*)(o.s_value + 2 * i) = make_float2(va, vb);
                *(char2*)(o.s_pos + 2 * i) = make_char2((signed char)(slots > 0 ? p0 : -1), (signed char)(slots > 1 ? p1 : -1));
            }
            meta |= (uint32_t)((kTilePos >> (4 * bits)) & 15u) << (q * 4 + 16 * h);
            if ((kLoneLater >> bits) & 1u) { vb = va; va = 0.f; }
            const __half2 pair = __floats2half2_rn(va, vb);
            word[h] = *(const uint32_t*)&pair;
        }
        if constexpr (STRICT) {
            // n_extra: bit 2 h + i says that row g + 8 h has a third or fourth entry, in position 2 + i
            int incl = __popc(n_extra);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            int put = waiting + incl - __popc(n_extra);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if ((n_extra >> i) & 1) {
                    const int lr = g + 8 * (i >> 1);
                    const Record e = group[2 + (i & 1)];
                    s_key[wid][put] = ((u64)(unsigned)(w * window + lr) << 32) | (unsigned)e.col;
                    s_at[wid][put] = e.start + __popc(e.mask & ((1u << lr) - 1u));
                    ++put;
                }
            waiting += __shfl_sync(0xffffffffu, incl, 31);
            if (waiting > 128) flush();
        }
        *(uint2*)(o.packed_a + (size_t)t * 64 + g * 8 + q * 2) = make_uint2(word[0], word[1]);
        meta |= __shfl_xor_sync(0xffffffffu, meta, 8);
        meta |= __shfl_xor_sync(0xffffffffu, meta, 16);
        if (q == 0) o.packed_meta[(size_t)t * 8 + g] = meta;
        if (g == 0) {
            const int4 cols = make_int4(group[0].col, group[1].col, group[2].col, group[3].col);
            *(int4*)(o.s_tile_column + (size_t)t * 16 + q * 4) = cols;
            if (live) {
                *(int4*)(o.s_column + (size_t)gid * 4) = cols;
                o.s_window[gid] = w;
            }
        }
        __syncwarp();   // the records are overwritten by the next tile's
    }
    if constexpr (STRICT) {
        if (waiting > 0) flush();
        return;
    }
    dropped = __reduce_add_sync(0xffffffffu, dropped);
    if (lane == 0 && dropped) atomicAdd(x.count + blockIdx.x % kDropCounters, (u64)dropped);
}

// ---------------------------------------------------------------------------------------------
// 8. TC blocks
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ int find_block_window(const Win* __restrict__ pre, int W, int b) {
    int lo = 0, hi = W;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid].blocks <= b) lo = mid; else hi = mid;
    }
    return lo;
}

// one thread per TC block: columns ascending, bitmaps, value count; the record of every slot for kb_tc_values
__global__ void kb_tc_blocks(WindowView v, RecordView r, int W, int NB, int* __restrict__ t_column,
                             long long* __restrict__ t_binary, int* __restrict__ blk_nnz, int* __restrict__ slot_rec) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > NB) return;
    if (b == NB) { blk_nnz[NB] = 0; return; }
    const int w = find_block_window(v.pre, W, b);
    const int o0 = 8 * (b - v.pre[w].blocks), len = min(8, v.tc[w] - o0);
    const int p0 = v.rec[w] + o0;
    int ids[8], cols[8];
    for (int i = 0; i < len; ++i) { ids[i] = p0 + i; cols[i] = r.rec[p0 + i].col; }
    for (int i = 1; i < len; ++i) {
        const int c = cols[i], id = ids[i];
        int k = i - 1;
        while (k >= 0 && cols[k] > c) { cols[k + 1] = cols[k]; ids[k + 1] = ids[k]; --k; }
        cols[k + 1] = c; ids[k + 1] = id;
    }
    u64 lo = 0, hi = 0;
    for (int k = 0; k < 8; ++k) {
        t_column[(size_t)b * 8 + k] = k < len ? cols[k] : -1;
        slot_rec[(size_t)b * 8 + k] = k < len ? ids[k] : -1;
        if (k >= len) continue;
        const unsigned m = r.rec[ids[k]].mask;
        for (int i = 0; i < 8; ++i) {
            if ((m >> i) & 1u) lo |= 1ull << (i * 8 + k);
            if ((m >> (i + 8)) & 1u) hi |= 1ull << (i * 8 + k);
        }
    }
    t_binary[(size_t)b * 2] = (long long)lo;
    t_binary[(size_t)b * 2 + 1] = (long long)hi;
    blk_nnz[b] = __popcll(lo) + __popcll(hi);
}

// one thread per (block, slot, row): its value, in bitmap order
__global__ void kb_tc_values(RecordView r, const int* __restrict__ slot_rec, int NB, const long long* __restrict__ t_binary,
                             const int* __restrict__ t_block_offset, float* __restrict__ t_value) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)NB * 128) return;
    const int b = (int)(i >> 7), lr = (int)(i >> 3) & 15, k = (int)(i & 7);
    const int id = slot_rec[(size_t)b * 8 + k];
    if (id < 0) return;
    const Record c = r.rec[id];
    if (!((c.mask >> lr) & 1u)) return;
    const float value = r.value(c.start, c.value, __popc(c.mask & ((1u << lr) - 1u)));
    const u64 lo = (u64)t_binary[(size_t)b * 2], hi = (u64)t_binary[(size_t)b * 2 + 1];
    const int bit = (lr & 7) * 8 + k;
    const u64 below = (1ull << bit) - 1ull;
    const int rank = lr < 8 ? __popcll(lo & below) : __popcll(lo) + __popcll(hi & below);
    t_value[(size_t)t_block_offset[b] + rank] = value;
}

__global__ void kb_tc_parts(WindowView v, const int* __restrict__ win_cuda_unit, int W, int part_t,
                            int* __restrict__ t_row_offset, int* __restrict__ t_window_row, int* __restrict__ t_atomic) {
    int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w == 0) t_row_offset[0] = 0;
    if (w >= W) return;
    const int bb = v.pre[w].blocks, nb = v.pre[w + 1].blocks - bb;
    const int p0 = v.pre[w].parts, np = v.pre[w + 1].parts - p0;
    for (int q = 0; q < np; ++q) {
        t_row_offset[p0 + q + 1] = bb + min((q + 1) * part_t, nb);
        t_window_row[p0 + q] = w * 16;
        t_atomic[p0 + q] = np > 1 || win_cuda_unit[w] >= 0 ? 1 : 0;
    }
}

// ---------------------------------------------------------------------------------------------
// 9. CUDA-core leftovers: the (at most two) columns of the window's rejected unit.  Per row the
// entries come in ascending column order = CSR order.
// ---------------------------------------------------------------------------------------------
struct CudaRow {
    int n;
    int cols[2];
    int at[2];   // places in sval
};
__device__ __forceinline__ CudaRow cuda_row(int row, int window, const int* __restrict__ win_cuda_unit, const WindowView& v,
                                            const RecordView& r) {
    CudaRow out;
    out.n = 0;
    const int w = row / window, lr = row - w * window;
    const int u = win_cuda_unit[w];
    if (u < 0) return out;
    const int rec0 = v.rec[w] + v.tc[w], ncol = v.end[w] - rec0;
    for (int i = 0; i < 2; ++i) {
        const int ls = 2 * u + i;
        if (ls >= ncol) break;
        const Record c = r.rec[rec0 + ls];
        if (!((c.mask >> lr) & 1u)) continue;
        out.cols[out.n] = c.col;
        out.at[out.n] = c.start + __popc(c.mask & ((1u << lr) - 1u));
        ++out.n;
    }
    if (out.n == 2 && out.cols[0] > out.cols[1]) {
        int t = out.cols[0]; out.cols[0] = out.cols[1]; out.cols[1] = t;
        t = out.at[0]; out.at[0] = out.at[1]; out.at[1] = t;
    }
    return out;
}

// Strict mode: the row's dropped entries in the list sorted by (row, column).
struct Extras {
    const u64* key;
    const int* at;
    int n;
    __device__ __forceinline__ int first(int row) const {
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if ((long long)(key[mid] >> 32) < row) lo = mid + 1; else hi = mid;
        }
        return lo;
    }
};

// split rule of block_online.cpp:415-439: long parts, short parts, long nnz, short nnz
struct Parts {
    int nl, ns, zl, zs;
};
struct PartsSum {
    __host__ __device__ __forceinline__ Parts operator()(const Parts& a, const Parts& b) const {
        return Parts{a.nl + b.nl, a.ns + b.ns, a.zl + b.zl, a.zs + b.zs};
    }
};
__device__ __forceinline__ Parts split_counts(int n, int part_c, int short_size) {
    if (n <= 0) return Parts{0, 0, 0, 0};
    if (n <= short_size) return Parts{0, 1, 0, n};
    if (n <= part_c) return Parts{1, 0, n, 0};
    Parts p{n / part_c, 0, n / part_c * part_c, 0};
    const int residue = n % part_c;
    if (residue > 0) {
        if (residue <= short_size) { p.ns = 1; p.zs = residue; }
        else { p.nl += 1; p.zl += residue; }
    }
    return p;
}

// Where a row's parts begin: the sum over the rows before it in its block of kPartRows rows, and over the blocks before.
// A device-wide scan of all rows' 16-byte counts took 18 us behind 4 for the counts (262144 rows), the blocks' sums 5.
constexpr int kPartRows = 256;
struct PartsAt {
    const Parts* inside;   // [n_rows + 1]
    const Parts* before;   // [blocks + 1], the last one: all
    __device__ __forceinline__ Parts operator[](int row) const { return PartsSum()(inside[row], before[row / kPartRows]); }
};
__global__ void __launch_bounds__(kPartRows) kb_cuda_count(int n_rows, int window, int part_c, int short_size,
                                                           const int* __restrict__ win_cuda_unit, WindowView v, RecordView r, Extras x,
                                                           Parts* __restrict__ inside, Parts* __restrict__ block) {
    __shared__ Parts s_warp[kPartRows / 32];
    const int row = blockIdx.x * kPartRows + threadIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int n = 0;
    if (row < n_rows) {
        n = cuda_row(row, window, win_cuda_unit, v, r).n;
        if (x.n > 0) n += x.first(row + 1) - x.first(row);
    }
    const Parts own = split_counts(n, part_c, short_size);
    Parts incl = own;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Parts y{__shfl_up_sync(0xffffffffu, incl.nl, d), __shfl_up_sync(0xffffffffu, incl.ns, d),
                      __shfl_up_sync(0xffffffffu, incl.zl, d), __shfl_up_sync(0xffffffffu, incl.zs, d)};
        if (lane >= d) incl = PartsSum()(incl, y);
    }
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    Parts before{0, 0, 0, 0}, all{0, 0, 0, 0};
    for (int q = 0; q < kPartRows / 32; ++q) {
        if (q == wid) before = all;
        all = PartsSum()(all, s_warp[q]);
    }
    if (row <= n_rows)
        inside[row] = Parts{before.nl + incl.nl - own.nl, before.ns + incl.ns - own.ns, before.zl + incl.zl - own.zl,
                            before.zs + incl.zs - own.zs};
    if (threadIdx.x == 0) {
        block[blockIdx.x] = all;
        if (blockIdx.x + 1 == gridDim.x) block[gridDim.x] = Parts{0, 0, 0, 0};
    }
}

struct PartsOut {
    int *c_row_offset, *c_row, *c_atomic, *c_column;
    float* c_value;
    int *cs_row_offset, *cs_row, *cs_atomic, *cs_column;
    float* cs_value;
    // entry i of a row's list: the long parts come first
    __device__ __forceinline__ void put(const Parts& o, int row_long, int i, int col, float value) const {
        if (i < row_long) { c_column[o.zl + i] = col; c_value[o.zl + i] = value; }
        else { cs_column[o.zs + i - row_long] = col; cs_value[o.zs + i - row_long] = value; }
    }
};

// A row's list is the (at most two) entries of the window's rejected unit merged with the row's strict-mode
// extras, by column.  One thread per row writes its parts and the unit's entries, one per extra its place:
// its rank among the row's extras plus the unit entries before it (a hub row has thousands).
__global__ void kb_cuda_rows(int n_rows, int window, int part_c, int short_size, const int* __restrict__ win_cuda_unit,
                             WindowView v, RecordView r, Extras x, PartsAt off, PartsOut po, Publish pub) {
    int row = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0) pub.by_block();
    if (row == 0) { po.c_row_offset[0] = 0; po.cs_row_offset[0] = 0; }
    if (row >= n_rows) return;
    const Parts o = off[row], e = off[row + 1];
    const int row_long = e.zl - o.zl, nl = e.nl - o.nl, n = row_long + e.zs - o.zs;
    if (n <= 0) return;
    const int w = row / window;
    const int atomic = n > part_c ? 1 : (v.pre[w + 1].blocks > v.pre[w].blocks ? 1 : 0);
    for (int i = 0; i < nl; ++i) {
        po.c_row[o.nl + i] = row;
        po.c_atomic[o.nl + i] = atomic;
        po.c_row_offset[o.nl + i + 1] = o.zl + min((i + 1) * part_c, row_long);
    }
    if (e.ns > o.ns) {
        po.cs_row[o.ns] = row;
        po.cs_atomic[o.ns] = atomic;
        po.cs_row_offset[o.ns + 1] = e.zs;
    }
    const CudaRow cr = cuda_row(row, window, win_cuda_unit, v, r);
    if (cr.n == 0) return;
    const int xb = x.n > 0 ? x.first(row) : 0, xe = x.n > 0 ? x.first(row + 1) : 0;
    for (int i = 0; i < cr.n; ++i) {
        int lo = xb, hi = xe;   // extras with a smaller column
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if ((int)(x.key[mid] & 0xffffffffull) < cr.cols[i]) lo = mid + 1; else hi = mid;
        }
        po.put(o, row_long, i + lo - xb, cr.cols[i], r.sval[cr.at[i]]);
    }
}

__global__ void kb_cuda_extras(int window, const int* __restrict__ win_cuda_unit, WindowView v, RecordView r, Extras x,
                               PartsAt off, PartsOut po) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= x.n) return;
    const int row = (int)(x.key[i] >> 32), c = (int)(x.key[i] & 0xffffffffull);
    int rank = i - x.first(row);
    const CudaRow cr = cuda_row(row, window, win_cuda_unit, v, r);
    for (int k = 0; k < cr.n; ++k) rank += cr.cols[k] < c;
    const Parts o = off[row];
    po.put(o, off[row + 1].zl - o.zl, rank, c, r.sval[x.at[i]]);
}

// Words for the host where no kernel above can do it: a copy of a few words took 3.4 us behind a gap of up to 8 on the copy
// engine, this takes 2 behind 1.
__global__ void kb_publish(Publish p) { p.by_block(); }

__global__ void kb_to_half(const float* __restrict__ src, long long n, __half* __restrict__ dst) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __float2half_rn(src[i]);
}

}  // namespace trs

// ---------------------------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------------------------
using namespace trs;

struct trs_builder {
    BuildCfg cfg;
    Arena arena_store;
    Arena* arena = nullptr;            // set: outputs and scratch come from the caller's memory
    trs_build_alloc alloc = nullptr;   // set: outputs come from the caller's allocator
    void* alloc_ctx = nullptr;
    int n_rows = 0, W = 0;
    long long nnz = 0;
    // the 29 arrays, reference order (block_online.cpp:844-870)
    DevBuf<int> t_row_offset, t_block_offset, t_column, t_window_row, t_atomic;
    DevBuf<float> t_value;
    DevBuf<long long> t_binary;
    DevBuf<int> c_row_offset, c_row, c_atomic, c_column;
    DevBuf<float> c_value;
    DevBuf<int> cs_row_offset, cs_row, cs_atomic, cs_column;
    DevBuf<float> cs_value;
    DevBuf<int> s_column, s_window, s_offset, s_tile_window, s_tile_group, s_tile_column, s_window_tile_offset;
    DevBuf<unsigned char> s_mask;
    DevBuf<float> s_value;
    DevBuf<signed char> s_pos;
    DevBuf<uint32_t> s_packed_a, s_packed_meta;
    DevBuf<__half> t_value_h, c_value_h, cs_value_h;
    long long sizes[TRS_BUILD_NUM_ARRAYS];
    unsigned long long dropped = 0;
    long long distinct_cols = 0, units = 0;
    float build_ms = 0.f;

    // array `id` with `count` elements
    template <class T>
    int out(DevBuf<T>& buf, int id, size_t count) {
        if (!alloc || count == 0) return buf.alloc_from(arena, count);
        buf.n = count;
        buf.owned = false;
        buf.p = (T*)alloc(alloc_ctx, id, count * sizeof(T));
        return buf.p ? 0 : (int)cudaErrorMemoryAllocation;
    }
    void release() {
        t_row_offset.release(); t_block_offset.release(); t_column.release(); t_window_row.release();
        t_atomic.release(); t_value.release(); t_binary.release();
        c_row_offset.release(); c_row.release(); c_atomic.release(); c_column.release(); c_value.release();
        cs_row_offset.release(); cs_row.release(); cs_atomic.release(); cs_column.release(); cs_value.release();
        s_column.release(); s_window.release(); s_offset.release(); s_tile_window.release(); s_tile_group.release();
        s_tile_column.release(); s_window_tile_offset.release(); s_mask.release(); s_value.release(); s_pos.release();
        s_packed_a.release(); s_packed_meta.release(); t_value_h.release(); c_value_h.release(); cs_value_h.release();
    }
};

namespace {

inline unsigned grid_for(long long n, int block = 256) { return (unsigned)((n + block - 1) / block); }

int bits_for(long long max_value) {  // bits needed to store values in [0, max_value]
    int b = 1;
    while ((1ll << b) <= max_value && b < 62) ++b;
    return b;
}

#define TRS_TRY(expr) do { int _rc = (expr); if (_rc) return _rc; } while (0)

// CUB's temporary storage, kept between calls and grown when one needs more
struct Cub {
    TempSpace& ts;
    cudaStream_t st;
    unsigned char* tmp = nullptr;
    size_t cap = 0;
    Cub(TempSpace& t, cudaStream_t s) : ts(t), st(s) {}
    template <class Call>
    int run(Call&& call) {
        size_t bytes = 0;
        TRS_CUDA(call((void*)nullptr, bytes));
        if (bytes > cap || !tmp) {
            if (tmp) ts.drop(tmp, cap);
            TRS_TRY(ts.get<unsigned char>(bytes, &tmp));
            cap = bytes;
        }
        TRS_CUDA(call((void*)tmp, bytes));
        return 0;
    }
    template <class In, class Out, class T, class Op>
    int exclusive_scan(In in, Out out, Op op, T zero, long long n) {
        return run([&](void* t, size_t& b) { return cub::DeviceScan::ExclusiveScan(t, b, in, out, op, zero, n, st); });
    }
    template <class K, class V>
    int sort_pairs(K* k_in, K* k_out, V* v_in, V* v_out, long long n, int end_bit, K** k_res, V** v_res) {
        cub::DoubleBuffer<K> kb(k_in, k_out);
        cub::DoubleBuffer<V> vb(v_in, v_out);
        TRS_TRY(run([&](void* t, size_t& b) { return cub::DeviceRadixSort::SortPairs(t, b, kb, vb, n, 0, end_bit, st); }));
        *k_res = kb.Current();
        *v_res = vb.Current();
        return 0;
    }
};

// Pinned memory for the few words a build reads back; as many blocks exist as builds ever ran at the same time.
struct Mirror {
    static constexpr size_t kBytes = 2048;
    unsigned char* p = nullptr;
    cudaStream_t st = nullptr;
    bool pending = true;   // a kernel on `st` may still write here
    static std::mutex& lock() { static std::mutex m; return m; }
    static std::vector<unsigned char*>& idle() { static std::vector<unsigned char*> v; return v; }
    int take(cudaStream_t stream) {
        st = stream;
        {
            std::lock_guard<std::mutex> g(lock());
            if (!idle().empty()) { p = idle().back(); idle().pop_back(); return 0; }
        }
        TRS_CUDA(cudaHostAlloc((void**)&p, kBytes, cudaHostAllocPortable));
        return 0;
    }
    ~Mirror() {
        if (!p) return;
        if (pending) cudaStreamSynchronize(st);
        std::lock_guard<std::mutex> g(lock());
        idle().push_back(p);
    }
};

// what a build reads back, from the device into a Mirror; the host may look after an event or a synchronisation behind it
template <class A, class B>
Publish words(const A* a, A* host_a, const B* b, B* host_b) {
    return Publish{(const int*)a, (int*)host_a, (int)(sizeof(A) / 4), (const int*)b, (int*)host_b, (int)(sizeof(B) / 4)};
}
template <class T>
Publish words(const T* dev, T* host) { return Publish{(const int*)dev, (int*)host, (int)(sizeof(T) / 4), nullptr, nullptr, 0}; }
int publish(const Publish& p, cudaStream_t st) {
    kb_publish<<<1, 128, 0, st>>>(p);
    TRS_LAUNCH_CHECK();
    return 0;
}
template <class T>
int read_back(const T* dev, T* host, cudaStream_t st) {
    TRS_TRY(publish(words(dev, host), st));
    TRS_CUDA(cudaStreamSynchronize(st));
    return 0;
}

// Streams on which the hub tiers of the matching run beside the others (two per device, made once).
// Work on the side streams that the caller's stream has not been made to wait for: a call that fails in between waits
// here, before the memory goes back.
struct SideWork {
    cudaStream_t s[2] = {nullptr, nullptr};
    bool open = false;
    ~SideWork() {
        if (open)
            for (cudaStream_t x : s) cudaStreamSynchronize(x);
    }
};
int side_streams(cudaStream_t out[2]) {
    static cudaStream_t made[64][2] = {};
    static std::mutex m;
    int dev = 0;
    TRS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return TRS_E_LIMIT;
    std::lock_guard<std::mutex> lock(m);
    for (int i = 0; i < 2; ++i) {
        if (!made[dev][i]) TRS_CUDA(cudaStreamCreateWithFlags(&made[dev][i], cudaStreamNonBlocking));
        out[i] = made[dev][i];
    }
    return 0;
}
struct Event {
    cudaEvent_t e = nullptr;
    int record(cudaStream_t st) {
        if (!e) TRS_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        TRS_CUDA(cudaEventRecord(e, st));
        return 0;
    }
    int wait() const {
        TRS_CUDA(cudaEventSynchronize(e));
        return 0;
    }
    ~Event() { if (e) cudaEventDestroy(e); }
};

struct HubBack {   // what the host sees of the hub windows before their records are made
    int records, err;
};
struct Records {   // stages 1 - 3
    WindowOut w{};
    int* sel = nullptr;   // [kSortClasses + 1][W]
};

template <int T, class Key, int C>
int sort_class_as(const InputInfo& info, const int* rowptr, const int* col, const float* val, const trs_builder* B, const Records& R,
                  InputInfo* d_info, cudaStream_t st) {
    constexpr int CAP = sort_cap(C), smem = (int)sizeof(typename WindowSort<T, CAP, Key>::Smem);
    auto kernel = kb_sort_window<T, CAP, Key>;
    static std::atomic<unsigned long long> done{0};
    TRS_TRY(allow_smem(kernel, smem, false, done));
    kernel<<<info.windows[C], T, smem, st>>>(rowptr, col, val, B->n_rows, B->cfg.window, R.sel + (size_t)C * B->W, R.w, d_info);
    TRS_LAUNCH_CHECK();
    return 0;
}
template <int T, int C>
int sort_class(const InputInfo& info, const int* rowptr, const int* col, const float* val, const trs_builder* B, int col_bits,
               const Records& R, InputInfo* d_info, cudaStream_t st) {
    if (info.windows[C] == 0) return 0;
    if constexpr (C < kWarpClasses) {
        using S = WarpSort<sort_cap(C) / 32>;
        if (col_bits + S::PB <= 31) {   // larger columns would need keys of 64 bits, which a warp has no registers for
            constexpr int smem = (int)sizeof(typename S::Smem) * kSortWarps;
            auto kernel = kb_sort_warp<sort_cap(C) / 32>;
            static std::atomic<unsigned long long> done{0};
            TRS_TRY(allow_smem(kernel, smem, false, done));
            kernel<<<ceil_div(info.windows[C], kSortWarps), 32 * kSortWarps, smem, st>>>(rowptr, col, val, B->n_rows, B->cfg.window,
                                                                                        R.sel + (size_t)C * B->W, info.windows[C], R.w, d_info);
            TRS_LAUNCH_CHECK();
            return 0;
        }
    }
    return col_bits + WindowSort<T, sort_cap(C), unsigned>::PB <= 32
               ? sort_class_as<T, unsigned, C>(info, rowptr, col, val, B, R, d_info, st)
               : sort_class_as<T, u64, C>(info, rowptr, col, val, B, R, d_info, st);
}

// `meanwhile` queues what does not depend on the hub windows
template <class Key, class Other>
int sort_hubs(trs_builder* B, const int* rowptr, const int* col, const float* val, const InputInfo& info, InputInfo* d_info,
              int* d_count, HubBack* back, int col_bits, TempSpace& ts, Cub& cub_, cudaStream_t st, const Records& R, Other&& meanwhile) {
    const int H = info.windows[kSortClasses], E = (int)info.hub_entries, n = B->n_rows, window = B->cfg.window;
    const int h_bits = bits_for(H - 1);
    const int* sel = R.sel + (size_t)kSortClasses * B->W;
    int *off, *first_rec, *place_a, *place_b, *place;
    Key *keys_a, *keys_b, *keys;
    TRS_TRY(ts.get((size_t)H + 1, &off));
    TRS_TRY(ts.get((size_t)H, &first_rec));
    TRS_TRY(ts.get(E, &keys_a));
    TRS_TRY(ts.get(E, &keys_b));
    TRS_TRY(ts.get(E, &place_a));
    TRS_TRY(ts.get(E, &place_b));
    const HubSizes size{rowptr, sel, n, window, H};
    if (H + 1 <= kSmallScan) {
        kb_scan_small<<<1, 1024, 0, st>>>(size, ToArray<int>{off}, IntSum(), 0, H + 1, Publish{});
        TRS_LAUNCH_CHECK();
    } else {
        TRS_TRY(cub_.exclusive_scan(thrust::make_transform_iterator(thrust::counting_iterator<int>(0), size), off, IntSum(), 0, (long long)H + 1));
    }
    const HubView hub{sel, off, H};
    kb_hub_keys<Key><<<grid_for(E), 256, 0, st>>>(rowptr, col, n, window, hub, E, col_bits, keys_a, place_a, d_info);
    TRS_LAUNCH_CHECK();
    TRS_TRY(cub_.sort_pairs(keys_a, keys_b, place_a, place_b, (long long)E, col_bits + h_bits, &keys, &place));
    // first entries, into the key buffer that is free now
    int* start = (int*)(keys == keys_a ? keys_b : keys_a);
    IsHead<Key> is_head{keys};
    TRS_TRY(cub_.run([&](void* t, size_t& b) {
        return cub::DeviceSelect::If(t, b, thrust::counting_iterator<int>(0), start, d_count, E, is_head, st);
    }));
    TRS_TRY(publish(words((const int*)d_count, &back->records, (const int*)&d_info->err, &back->err), st));
    TRS_TRY(meanwhile());
    TRS_CUDA(cudaStreamSynchronize(st));
    if (back->err & 2) return TRS_E_NOT_CANONICAL;   // a repeated column may have more entries than a record counts
    const int D = back->records;
    Record* record;
    unsigned *key2_a, *key2_b, *key2;
    int *ord_a, *ord_b, *ord;
    TRS_TRY(ts.get(D, &record));
    TRS_TRY(ts.get(D, &key2_a));
    TRS_TRY(ts.get(D, &key2_b));
    TRS_TRY(ts.get(D, &ord_a));
    TRS_TRY(ts.get(D, &ord_b));
    kb_hub_records<Key><<<grid_for(D), 256, 0, st>>>(keys, place, rowptr, val, n, window, hub, start, D, E, col_bits, record, key2_a, ord_a, first_rec);
    TRS_LAUNCH_CHECK();
    TRS_TRY(cub_.sort_pairs(key2_a, key2_b, ord_a, ord_b, (long long)D, 4 + h_bits, &key2, &ord));  // stable
    kb_hub_place<<<grid_for(D), 256, 0, st>>>(key2, ord, record, D, rowptr, window, hub, first_rec, R.w);
    TRS_LAUNCH_CHECK();
    kb_hub_values<<<grid_for(E), 256, 0, st>>>(place, rowptr, val, window, hub, E, R.w.sval);
    TRS_LAUNCH_CHECK();
    ts.drop(ord_b, D); ts.drop(ord_a, D); ts.drop(key2_b, D); ts.drop(key2_a, D); ts.drop(record, D);
    ts.drop(place_b, E); ts.drop(place_a, E); ts.drop(keys_b, E); ts.drop(keys_a, E);
    return 0;
}

// The hub windows are a chain of small launches with a read-back in it (R-MAT 15: 160 us) and the classes keep the chip
// half busy one after the other (R-MAT 18: 180 us): with more than one of them in a graph, two other streams take the
// classes beside the chain (whole build of R-MAT 15 662 -> 541 us, of R-MAT 18 1470 -> 1338, with the sizes read back by kernels).
int make_records(trs_builder* B, const int* rowptr, const int* col, const float* val, const InputInfo& info, InputInfo* d_info,
                 int* d_count, HubBack* back, TempSpace& ts, Cub& cub_, cudaStream_t st, Records* R) {
    const int col_bits = bits_for(info.max_col), W = B->W;
    const size_t nnz = (size_t)B->nnz;
    TRS_TRY(ts.get(nnz, &R->w.rec));
    TRS_TRY(ts.get(nnz, &R->w.sval));
    TRS_TRY(ts.get(nnz, &R->w.cnt));
    int parts = 0;
    for (int c = 0; c <= kSortClasses; ++c) parts += info.windows[c] > 0;
    const bool fork = parts > 1;
    cudaStream_t side[2] = {st, st};
    Event ready, done[2];
    if (fork) {
        TRS_TRY(side_streams(side));
        TRS_TRY(ready.record(st));
        for (cudaStream_t s : side) TRS_CUDA(cudaStreamWaitEvent(s, ready.e, 0));
    }
    auto classes = [&]() -> int {
        TRS_TRY((sort_class<1024, 6>(info, rowptr, col, val, B, col_bits, *R, d_info, side[0])));
        TRS_TRY((sort_class<512, 5>(info, rowptr, col, val, B, col_bits, *R, d_info, side[1])));
        TRS_TRY((sort_class<256, 4>(info, rowptr, col, val, B, col_bits, *R, d_info, side[1])));
        TRS_TRY((sort_class<128, 3>(info, rowptr, col, val, B, col_bits, *R, d_info, side[0])));
        TRS_TRY((sort_class<128, 2>(info, rowptr, col, val, B, col_bits, *R, d_info, side[1])));
        TRS_TRY((sort_class<128, 1>(info, rowptr, col, val, B, col_bits, *R, d_info, side[0])));
        return sort_class<64, 0>(info, rowptr, col, val, B, col_bits, *R, d_info, side[1]);
    };
    int rc = 0;
    if (info.windows[kSortClasses] > 0) {
        const int h_bits = bits_for(info.windows[kSortClasses] - 1);
        rc = col_bits + h_bits <= 32 ? sort_hubs<unsigned>(B, rowptr, col, val, info, d_info, d_count, back, col_bits, ts, cub_, st, *R, classes)
                                     : sort_hubs<u64>(B, rowptr, col, val, info, d_info, d_count, back, col_bits, ts, cub_, st, *R, classes);
    } else {
        rc = classes();
    }
    if (fork)
        for (int i = 0; i < 2; ++i) {   // after an error too: what is freed next may still be in use
            TRS_TRY(done[i].record(side[i]));
            TRS_CUDA(cudaStreamWaitEvent(st, done[i].e, 0));
        }
    return rc;
}

int empty_outputs(trs_builder* B, cudaStream_t st) {
    TRS_TRY(B->out(B->s_offset, 22, (size_t)B->W + 1));
    TRS_TRY(B->out(B->s_window_tile_offset, 28, (size_t)B->W + 1));
    TRS_TRY(B->out(B->t_row_offset, 0, 1));
    TRS_TRY(B->out(B->t_block_offset, 1, 1));
    TRS_TRY(B->out(B->c_row_offset, 7, 1));
    TRS_TRY(B->out(B->cs_row_offset, 12, 1));
    TRS_CUDA(cudaMemsetAsync(B->s_offset.p, 0, sizeof(int) * ((size_t)B->W + 1), st));
    TRS_CUDA(cudaMemsetAsync(B->s_window_tile_offset.p, 0, sizeof(int) * ((size_t)B->W + 1), st));
    for (DevBuf<int>* b : {&B->t_row_offset, &B->t_block_offset, &B->c_row_offset, &B->cs_row_offset})
        TRS_CUDA(cudaMemsetAsync(b->p, 0, sizeof(int), st));
    return 0;
}

int do_build(trs_builder* B, const int* rowptr, const int* col, const float* val, cudaStream_t st) {
    const BuildCfg& cfg = B->cfg;
    const int n = B->n_rows, window = cfg.window, W = B->W;
    int dev = 0, sms = 1;
    TRS_CUDA(cudaGetDevice(&dev));
    TRS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TempSpace ts;
    ts.arena = B->arena;
    ts.st = st;
    Cub cub_(ts, st);

    // ---- sizes of the input ---------------------------------------------------------------------
    struct Counts { InputInfo info; MatchCounts mc; };
    struct Head { Counts counts; u64 dropped[kDropCounters]; int hub_records; unsigned info_blocks; };
    struct Back { Head head; HubBack hub; Win total; Parts parts; int groups, tiles, tc_nnz; };   // what the host sees of it
    static_assert(sizeof(Back) <= Mirror::kBytes, "");
    Mirror mirror;
    TRS_TRY(mirror.take(st));
    Back* const back = (Back*)mirror.p;
    Head* d_head;
    TRS_TRY(ts.get(1, &d_head));
    TRS_CUDA(cudaMemsetAsync(d_head, 0, sizeof(Head), st));
    Records R;
    TRS_TRY(ts.get((size_t)(kSortClasses + 1) * W, &R.sel));
    TRS_TRY(ts.get((size_t)W, &R.w.ncol));
    kb_input_info<<<2 * sms, 512, 0, st>>>(rowptr, col, n, window, W, R.sel, R.w.ncol, &d_head->counts.info, &d_head->info_blocks,
                                         words(&d_head->counts.info, &back->head.counts.info));
    TRS_LAUNCH_CHECK();
    TRS_CUDA(cudaStreamSynchronize(st));
    const InputInfo info = back->head.counts.info;
    if (info.first != 0 || info.last < 0 || (info.err & 1)) return TRS_E_OFFSETS;
    const long long nnz = B->nnz = info.last;
    if (nnz == 0) return empty_outputs(B, st);
    if (!col || !val) return TRS_E_ARG;
    ts.chunk_bytes = std::max((size_t)16 << 20, (size_t)nnz * 28);

    // ---- 1. - 3. columns of every window in (count desc, col asc) order ---------------------------
    TRS_TRY(make_records(B, rowptr, col, val, info, &d_head->counts.info, &d_head->hub_records, &back->hub, ts, cub_, st, &R));
    const RecordView rv{R.w.rec, R.w.sval};

    // Scans by one CTA where they are short (`from`, `to`), by device-wide passes over the iterators otherwise; `pub` goes to the
    // host behind them.
    auto scan = [&](auto from, auto to, auto in, auto out, auto op, auto zero, long long count, const Publish& pub) -> int {
        if (count <= kSmallScan) {
            kb_scan_small<<<1, 1024, 0, st>>>(from, to, op, zero, (int)count, pub);
            TRS_LAUNCH_CHECK();
            return 0;
        }
        TRS_TRY(cub_.exclusive_scan(in, out, op, zero, count));
        return pub.na > 0 ? publish(pub, st) : 0;
    };
    // ---- 4., 5. TC columns, units, sizes per window ---------------------------------------------
    int *rec, *end, *tc, *sel_block, *sel_huge;
    Win *win, *pre;
    TRS_TRY(ts.get((size_t)W + 1, &rec));
    TRS_TRY(ts.get((size_t)W + 1, &end));
    TRS_TRY(ts.get((size_t)W + 1, &tc));
    TRS_TRY(ts.get((size_t)W + 1, &win));
    TRS_TRY(ts.get((size_t)W + 1, &pre));
    TRS_TRY(ts.get((size_t)W + 1, &sel_block));
    TRS_TRY(ts.get((size_t)W + 1, &sel_huge));
    kb_windows<<<grid_for(W + 1, 128), 128, 0, st>>>(rowptr, R.w.ncol, R.w.cnt, W, cfg, rec, end, tc, win, sel_block, sel_huge, &d_head->counts.mc);
    TRS_LAUNCH_CHECK();
    TRS_TRY(scan(FromArray<Win>{win}, ToArray<Win>{pre}, win, pre, WinSum(), Win{0, 0, 0, 0}, W + 1,
                 words(&d_head->counts, &back->head.counts, (const Win*)pre + W, &back->total)));
    const WindowView v{rec, end, tc, pre};
    Event sized, grouped, counted;
    TRS_TRY(sized.record(st));

    // ---- 6. matching ------------------------------------------------------------------------------
    MatchOut mo;
    auto match_arrays = [&](size_t units, size_t slots) -> int {
        TRS_TRY(ts.get(units, &mo.order));
        TRS_TRY(ts.get(slots, &mo.pair_a));
        TRS_TRY(ts.get(slots, &mo.pair_b));
        TRS_TRY(ts.get((size_t)W + 1, &mo.groups));
        return ts.get((size_t)W + 1, &mo.cuda_unit);
    };
    auto match_warps = [&](int max_units) -> int {
        const int units = std::max(32, (max_units + 31) & ~31);
        const size_t smem = (size_t)kMatchWarps * (units + units / 32) * 4;
        kb_match_warp<<<grid_for(W + 1, kMatchWarps), 32 * kMatchWarps, smem, st>>>(v, W, R.w.cnt, cfg.unit_min_nnz, units, mo);
        TRS_LAUNCH_CHECK();
        return 0;
    };
    // the sizes of the groups go to the host before the TC blocks are made, so that it lays out their arrays meanwhile
    auto group_sizes = [&]() -> int {
        TRS_TRY(B->out(B->s_offset, 22, (size_t)W + 1));
        TRS_TRY(B->out(B->s_window_tile_offset, 28, (size_t)W + 1));
        const auto both = thrust::make_transform_iterator((const int*)mo.groups, WithTiles());
        const auto out = thrust::make_transform_output_iterator(
            thrust::make_zip_iterator(thrust::make_tuple(B->s_offset.p, B->s_window_tile_offset.p)), ToTuple());
        TRS_TRY(scan(GroupsFrom{mo.groups}, GroupsTo{B->s_offset.p, B->s_window_tile_offset.p}, both, out, GroupsTilesSum(), GroupsTiles{0, 0}, W + 1,
                     words((const int*)B->s_offset.p + W, &back->groups, (const int*)B->s_window_tile_offset.p + W, &back->tiles)));
        return grouped.record(st);
    };
    // Without large windows the bounds are close enough to start before the sizes have come back (30 us of 870 on the
    // clustered graph).  With them the words of every warp would take the shared memory of many.
    bool ahead = true;
    int largest = 0;
    for (int c = 0; c <= kSortClasses; ++c) {
        if (info.windows[c] == 0) continue;
        largest = c;
        ahead &= c < kSortClasses - 2;
    }
    static_assert(sort_cap(kSortClasses - 3) / 2 <= kWarpUnits, "");
    if (ahead) {
        TRS_TRY(match_arrays((size_t)nnz / 2 + W, (size_t)nnz / 4 + W));
        TRS_TRY(match_warps(sort_cap(largest) / 2));
        TRS_TRY(group_sizes());
    }
    TRS_TRY(sized.wait());
    if (back->head.counts.info.err & 2) return TRS_E_NOT_CANONICAL;
    const Win total = back->total;
    const MatchCounts mc = back->head.counts.mc;
    B->distinct_cols = (long long)mc.records;
    const int NB = total.blocks, NP = total.parts, TU = total.units, TS = total.slots;
    B->units = TU;
    if (!ahead) TRS_TRY(match_arrays(TU, TS));
    if (mc.max_huge >= (int)kUnitMask) return TRS_E_LIMIT;
    // one long chain per hub window: the tiers run side by side
    SideWork work;
    cudaStream_t* const side = work.s;
    TRS_TRY(side_streams(side));
    Event ready, done[2];
    if (mc.n_huge + mc.n_block > 0) {
        TRS_TRY(ready.record(st));
        TRS_CUDA(cudaFuncSetAttribute(kb_match_block, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemUnits * 4));
        work.open = true;
    }
    if (mc.n_huge > 0) {
        const int smem_units = mc.max_huge <= kSmemUnits ? mc.max_huge : kSmemUnits;
        int* words = nullptr;
        unsigned* mask = nullptr;
        if (mc.max_huge > kSmemUnits) {
            TRS_TRY(ts.get(TU, &words));
            TRS_TRY(ts.get((size_t)TU / 32 + W + 2, &mask));
        }
        TRS_CUDA(cudaStreamWaitEvent(side[0], ready.e, 0));
        kb_match_block<<<mc.n_huge, kBlockThreads, (size_t)smem_units * 4, side[0]>>>(v, R.w.cnt, cfg.unit_min_nnz, smem_units, words, mask,
                                                                                 sel_huge, mo);
        TRS_LAUNCH_CHECK();
    }
    if (mc.n_block > 0) {
        TRS_CUDA(cudaStreamWaitEvent(side[1], ready.e, 0));
        kb_match_block<<<mc.n_block, kBlockThreads, (size_t)kBlockUnits * 4, side[1]>>>(v, R.w.cnt, cfg.unit_min_nnz, kBlockUnits, nullptr,
                                                                                   nullptr, sel_block, mo);
        TRS_LAUNCH_CHECK();
    }
    if (!ahead) TRS_TRY(match_warps(mc.max_warp));

    // ---- 8. TC blocks (their values need the block offsets) --------------------------------------
    int *blk_nnz, *slot_rec;
    TRS_TRY(ts.get((size_t)NB + 1, &blk_nnz));
    TRS_TRY(ts.get((size_t)NB * 8, &slot_rec));
    TRS_TRY(B->out(B->t_block_offset, 1, (size_t)NB + 1));
    TRS_TRY(B->out(B->t_column, 2, (size_t)NB * 8));
    TRS_TRY(B->out(B->t_binary, 6, (size_t)NB * 2));
    kb_tc_blocks<<<grid_for(NB + 1, 128), 128, 0, st>>>(v, rv, W, NB, B->t_column.p, B->t_binary.p, blk_nnz, slot_rec);
    TRS_LAUNCH_CHECK();
    TRS_TRY(scan(FromArray<int>{blk_nnz}, ToArray<int>{B->t_block_offset.p}, (const int*)blk_nnz, B->t_block_offset.p, IntSum(), 0, (long long)NB + 1,
                 Publish{}));
    if (!ahead) {   // the hub windows are matched by now
        if (mc.n_huge > 0) { TRS_TRY(done[0].record(side[0])); TRS_CUDA(cudaStreamWaitEvent(st, done[0].e, 0)); }
        if (mc.n_block > 0) { TRS_TRY(done[1].record(side[1])); TRS_CUDA(cudaStreamWaitEvent(st, done[1].e, 0)); }
        work.open = false;
        TRS_TRY(group_sizes());
    }
    TRS_TRY(B->out(B->t_row_offset, 0, (size_t)NP + 1));
    TRS_TRY(B->out(B->t_window_row, 4, NP));
    TRS_TRY(B->out(B->t_atomic, 5, NP));
    kb_tc_parts<<<grid_for(W), 256, 0, st>>>(v, mo.cuda_unit, W, cfg.part_t, B->t_row_offset.p, B->t_window_row.p, B->t_atomic.p);
    TRS_LAUNCH_CHECK();

    // ---- 9. CUDA-core parts: counted now, or in strict mode when the dropped entries are known ------
    Parts *inside, *block, *before;
    const unsigned part_blocks = grid_for((long long)n + 1, kPartRows);
    TRS_TRY(ts.get((size_t)n + 1, &inside));
    TRS_TRY(ts.get((size_t)part_blocks + 1, &block));
    TRS_TRY(ts.get((size_t)part_blocks + 1, &before));
    const PartsAt off{inside, before};
    Extras x{nullptr, nullptr, 0};
    auto count_parts = [&](const Publish& pub) -> int {
        kb_cuda_count<<<part_blocks, kPartRows, 0, st>>>(n, window, cfg.part_c, cfg.short_size, mo.cuda_unit, v, rv, x, inside, block);
        TRS_LAUNCH_CHECK();
        return scan(FromArray<Parts>{block}, ToArray<Parts>{before}, block, before, PartsSum(), Parts{0, 0, 0, 0}, (long long)part_blocks + 1, pub);
    };
    if (cfg.strict) {
        TRS_TRY(publish(words((const int*)B->t_block_offset.p + NB, &back->tc_nnz), st));
    } else {
        TRS_TRY(count_parts(words((const int*)B->t_block_offset.p + NB, &back->tc_nnz, (const Parts*)before + part_blocks, &back->parts)));
    }
    TRS_TRY(counted.record(st));

    // ---- 7. groups and tiles ------------------------------------------------------------------------
    TRS_TRY(grouped.wait());
    const int G = back->groups, T = back->tiles;
    TRS_TRY(B->out(B->s_column, 17, (size_t)G * 4));
    TRS_TRY(B->out(B->s_mask, 18, (size_t)G * window));
    TRS_TRY(B->out(B->s_value, 19, (size_t)G * window * 2));
    TRS_TRY(B->out(B->s_pos, 20, (size_t)G * window * 2));
    TRS_TRY(B->out(B->s_window, 21, G));
    TRS_TRY(B->out(B->s_tile_window, 23, T));
    TRS_TRY(B->out(B->s_tile_group, 24, T));
    TRS_TRY(B->out(B->s_tile_column, 25, (size_t)T * 16));
    TRS_TRY(B->out(B->s_packed_a, 26, (size_t)T * 64));
    TRS_TRY(B->out(B->s_packed_meta, 27, (size_t)T * 8));
    u64 *xkey_a = nullptr, *xkey_b = nullptr;
    int *xat_a = nullptr, *xat_b = nullptr;
    if (cfg.strict) {   // at least two of a row's entries in a group are kept, so at most half are dropped
        TRS_TRY(ts.get((size_t)nnz / 2 + 1, &xkey_a));
        TRS_TRY(ts.get((size_t)nnz / 2 + 1, &xat_a));
    }
    if (T > 0) {
        TileSource* source;
        TRS_TRY(ts.get(T, &source));
        kb_tiles<<<grid_for(T), 256, 0, st>>>(B->s_window_tile_offset.p, B->s_offset.p, v, W, T, B->s_tile_window.p, B->s_tile_group.p, source);
        TRS_LAUNCH_CHECK();
        const GroupOut go{B->s_column.p, B->s_mask.p, B->s_value.p, B->s_pos.p, B->s_window.p, B->s_tile_column.p,
                          B->s_packed_a.p, B->s_packed_meta.p};
        const ExtraOut xo{d_head->dropped, xkey_a, xat_a};
        auto emit = cfg.strict ? kb_emit_tiles<true> : kb_emit_tiles<false>;
        // as many blocks as are resident
        emit<<<std::min(grid_for(T, 8), (unsigned)sms * 4u), 256, 0, st>>>(source, rv, B->s_tile_window.p, B->s_tile_group.p, T, window,
                                                                           mo.pair_a, mo.pair_b, go, xo);
        TRS_LAUNCH_CHECK();
    }
    // the values of the TC blocks fill the last wave of the tiles
    TRS_TRY(counted.wait());
    TRS_TRY(B->out(B->t_value, 3, back->tc_nnz));
    Event valued;
    if (NB > 0) {
        work.open = true;
        TRS_CUDA(cudaStreamWaitEvent(side[0], counted.e, 0));
        kb_tc_values<<<grid_for((long long)NB * 128), 256, 0, side[0]>>>(rv, slot_rec, NB, B->t_binary.p, B->t_block_offset.p, B->t_value.p);
        TRS_LAUNCH_CHECK();
        TRS_TRY(valued.record(side[0]));
    }
    if (NB > 0) {
        TRS_CUDA(cudaStreamWaitEvent(st, valued.e, 0));
        work.open = false;
    }
    if (cfg.strict) {
        TRS_TRY(read_back(&d_head->dropped, &back->head.dropped, st));
        const u64 n_extra = back->head.dropped[0];
        if (n_extra > 0) {
            u64* key;
            int* at;
            TRS_TRY(ts.get(n_extra, &xkey_b));
            TRS_TRY(ts.get(n_extra, &xat_b));
            TRS_TRY(cub_.sort_pairs(xkey_a, xkey_b, xat_a, xat_b, (long long)n_extra, 32 + bits_for(n), &key, &at));
            x = Extras{key, at, (int)n_extra};
        }
        TRS_TRY(count_parts(words((const Parts*)before + part_blocks, &back->parts)));
        TRS_CUDA(cudaStreamSynchronize(st));
    }
    const Parts p = back->parts;
    TRS_TRY(B->out(B->c_row_offset, 7, (size_t)p.nl + 1));
    TRS_TRY(B->out(B->c_row, 8, p.nl));
    TRS_TRY(B->out(B->c_atomic, 9, p.nl));
    TRS_TRY(B->out(B->c_column, 10, p.zl));
    TRS_TRY(B->out(B->c_value, 11, p.zl));
    TRS_TRY(B->out(B->cs_row_offset, 12, (size_t)p.ns + 1));
    TRS_TRY(B->out(B->cs_row, 13, p.ns));
    TRS_TRY(B->out(B->cs_atomic, 14, p.ns));
    TRS_TRY(B->out(B->cs_column, 15, p.zs));
    TRS_TRY(B->out(B->cs_value, 16, p.zs));
    const PartsOut po{B->c_row_offset.p, B->c_row.p, B->c_atomic.p, B->c_column.p, B->c_value.p,
                      B->cs_row_offset.p, B->cs_row.p, B->cs_atomic.p, B->cs_column.p, B->cs_value.p};
    kb_cuda_rows<<<grid_for(n), 256, 0, st>>>(n, window, cfg.part_c, cfg.short_size, mo.cuda_unit, v, rv, x, off, po,
                                             words(&d_head->dropped, &back->head.dropped));
    TRS_LAUNCH_CHECK();
    if (x.n > 0) {
        kb_cuda_extras<<<grid_for(x.n), 256, 0, st>>>(window, mo.cuda_unit, v, rv, x, off, po);
        TRS_LAUNCH_CHECK();
    }
    TRS_CUDA(cudaStreamSynchronize(st));
    mirror.pending = false;
    B->dropped = 0;
    if (!cfg.strict)   // nothing is lost in strict mode
        for (u64 d : back->head.dropped) B->dropped += d;
    TRS_LAUNCH_CHECK();
    return TRS_OK;
}

void fill_sizes(trs_builder* B) {
    long long* z = B->sizes;
    z[0] = B->t_row_offset.n; z[1] = B->t_block_offset.n; z[2] = B->t_column.n; z[3] = B->t_value.n;
    z[4] = B->t_window_row.n; z[5] = B->t_atomic.n; z[6] = B->t_binary.n;
    z[7] = B->c_row_offset.n; z[8] = B->c_row.n; z[9] = B->c_atomic.n; z[10] = B->c_column.n; z[11] = B->c_value.n;
    z[12] = B->cs_row_offset.n; z[13] = B->cs_row.n; z[14] = B->cs_atomic.n; z[15] = B->cs_column.n; z[16] = B->cs_value.n;
    z[17] = B->s_column.n; z[18] = B->s_mask.n; z[19] = B->s_value.n; z[20] = B->s_pos.n; z[21] = B->s_window.n;
    z[22] = B->s_offset.n; z[23] = B->s_tile_window.n; z[24] = B->s_tile_group.n; z[25] = B->s_tile_column.n;
    z[26] = B->s_packed_a.n; z[27] = B->s_packed_meta.n; z[28] = B->s_window_tile_offset.n;
}

const void* array_ptr(const trs_builder* B, int id, size_t* elem) {
    switch (id) {
        case 0: *elem = 4; return B->t_row_offset.p;    case 1: *elem = 4; return B->t_block_offset.p;
        case 2: *elem = 4; return B->t_column.p;        case 3: *elem = 4; return B->t_value.p;
        case 4: *elem = 4; return B->t_window_row.p;    case 5: *elem = 4; return B->t_atomic.p;
        case 6: *elem = 8; return B->t_binary.p;        case 7: *elem = 4; return B->c_row_offset.p;
        case 8: *elem = 4; return B->c_row.p;           case 9: *elem = 4; return B->c_atomic.p;
        case 10: *elem = 4; return B->c_column.p;       case 11: *elem = 4; return B->c_value.p;
        case 12: *elem = 4; return B->cs_row_offset.p;  case 13: *elem = 4; return B->cs_row.p;
        case 14: *elem = 4; return B->cs_atomic.p;      case 15: *elem = 4; return B->cs_column.p;
        case 16: *elem = 4; return B->cs_value.p;       case 17: *elem = 4; return B->s_column.p;
        case 18: *elem = 1; return B->s_mask.p;         case 19: *elem = 4; return B->s_value.p;
        case 20: *elem = 1; return B->s_pos.p;          case 21: *elem = 4; return B->s_window.p;
        case 22: *elem = 4; return B->s_offset.p;       case 23: *elem = 4; return B->s_tile_window.p;
        case 24: *elem = 4; return B->s_tile_group.p;   case 25: *elem = 4; return B->s_tile_column.p;
        case 26: *elem = 4; return B->s_packed_a.p;     case 27: *elem = 4; return B->s_packed_meta.p;
        case 28: *elem = 4; return B->s_window_tile_offset.p;
    }
    *elem = 0;
    return nullptr;
}

}  // namespace

static int build_impl(const int32_t* rowptr, const int32_t* col, const float* values, int n_rows,
                      const trs_build_config* cfg, void* arena, size_t arena_bytes, bool use_arena, trs_build_alloc alloc,
                      void* ctx, void* stream, trs_builder** out) try {
    if (!rowptr || !cfg || !out || n_rows <= 0) return TRS_E_ARG;
    *out = nullptr;
    if (cfg->window <= 0 || cfg->window > 16) return TRS_E_WINDOW;
    if (cfg->part_t <= 0 || cfg->part_c <= 0 || cfg->short_size < 0 || cfg->density < 0) return TRS_E_ARG;
    if (use_arena && (!arena || ((uintptr_t)arena & 255))) return TRS_E_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return TRS_E_NO_DEVICE;
    trs_builder* B = new trs_builder();
    if (use_arena) {
        B->arena_store.base = (unsigned char*)arena;
        B->arena_store.cap = arena_bytes;
        B->arena = &B->arena_store;
    }
    B->alloc = alloc;
    B->alloc_ctx = ctx;
    B->cfg = BuildCfg{cfg->part_t, cfg->part_c, cfg->short_size, cfg->density, cfg->window, cfg->tc_min_util,
                      cfg->skip_tc, cfg->unit_min_nnz, cfg->strict ? 1 : 0};
    B->n_rows = n_rows;
    B->W = ceil_div(n_rows, cfg->window);
    cudaStream_t st = (cudaStream_t)stream;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0); cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    int rc = do_build(B, rowptr, col, values, st);
    cudaEventRecord(e1, st);
    cudaError_t es = cudaStreamSynchronize(st);
    if (!rc && es != cudaSuccess) rc = (int)es;
    if (!rc) cudaEventElapsedTime(&B->build_ms, e0, e1);
    cudaEventDestroy(e0); cudaEventDestroy(e1);
    if (rc) { B->release(); delete B; return rc; }
    fill_sizes(B);
    *out = B;
    return TRS_OK;
} TRS_CATCH

extern "C" int trs_build_create(const int32_t* rowptr, const int32_t* col, const float* values, int n_rows,
                                const trs_build_config* cfg, void* stream, trs_builder** out) {
    return build_impl(rowptr, col, values, n_rows, cfg, nullptr, 0, false, nullptr, nullptr, stream, out);
}

extern "C" int trs_build_create_into(const int32_t* rowptr, const int32_t* col, const float* values, int n_rows,
                                     const trs_build_config* cfg, trs_build_alloc alloc, void* ctx, void* stream,
                                     trs_builder** out) {
    if (!alloc) return TRS_E_ARG;
    return build_impl(rowptr, col, values, n_rows, cfg, nullptr, 0, false, alloc, ctx, stream, out);
}

// Upper bound of the device memory one build can need (outputs + temporaries), from the sizes
// alone: every count the builder allocates by is bounded by the number of entries (distinct
// (window, column) pairs <= nnz, units <= pairs / 2 + windows, groups <= pairs / 4 + windows, ...).
extern "C" int trs_build_query(int n_rows, long long nnz, const trs_build_config* cfg, size_t* arena_bytes) {
    if (!cfg || !arena_bytes || n_rows <= 0 || nnz < 0) return TRS_E_ARG;
    if (cfg->window <= 0 || cfg->window > 16) return TRS_E_WINDOW;
    const size_t W = (size_t)ceil_div(n_rows, cfg->window) + 1;
    const size_t e = (size_t)nnz;
    size_t b = 0;
    b += e * 40;                      // row ids, two 64-bit key buffers, two edge buffers, heads, running counts
    b += e * 72;                      // per-(window, column) records, their two sort buffers, TC / SPTC index maps
    b += (e / 2 + W) * 8 + (e / 4 + W) * 24;   // units, pairs, group column lists
    if (cfg->strict) b += e * 28 + (size_t)n_rows * 8;
    b += W * 4 * 34;                  // per-window counters and prefixes
    b += e / 2 + ((size_t)64 << 20);  // CUB temporary storage
    // outputs: SPTC groups (196 B each) and tiles (360 B each), TC blocks, CSR parts, fp16 value copies
    b += (e / 4 + W) * 196 + (e / 16 + 2 * W) * 360;
    b += e * 12 + (e / 8 + W) * 64 + e * 14 + W * 32;
    b += 256 * 160;                   // alignment of every block
    *arena_bytes = b;
    return TRS_OK;
}

extern "C" int trs_build_fill(const int32_t* rowptr, const int32_t* col, const float* values, int n_rows,
                              const trs_build_config* cfg, void* arena, size_t arena_bytes, void* stream,
                              trs_builder** out) {
    return build_impl(rowptr, col, values, n_rows, cfg, arena, arena_bytes, true, nullptr, nullptr, stream, out);
}

extern "C" int trs_build_arena_used(const trs_builder* B, size_t* bytes) {
    if (!B || !bytes) return TRS_E_ARG;
    *bytes = B->arena ? B->arena->high : 0;
    return TRS_OK;
}

extern "C" int trs_build_destroy(trs_builder* B) {
    if (!B) return TRS_OK;
    B->release();
    delete B;
    return TRS_OK;
}

extern "C" int trs_build_sizes(const trs_builder* B, long long* sizes) {
    if (!B || !sizes) return TRS_E_ARG;
    memcpy(sizes, B->sizes, sizeof(B->sizes));
    return TRS_OK;
}

extern "C" int trs_build_stats(const trs_builder* B, trs_build_stats_t* s) {
    if (!B || !s) return TRS_E_ARG;
    s->nnz = B->nnz;
    s->dropped_nnz = (long long)B->dropped;
    s->distinct_window_columns = B->distinct_cols;
    s->units = B->units;
    s->tc_nnz = B->sizes[3];
    s->csr_nnz = B->sizes[11] + B->sizes[16];
    s->groups = B->sizes[21];
    s->tiles = B->sizes[23];
    s->tc_blocks = B->sizes[2] / 8;
    s->build_ms = B->build_ms;
    return TRS_OK;
}

extern "C" const void* trs_build_array(const trs_builder* B, int id) {
    size_t elem;
    return B ? array_ptr(B, id, &elem) : nullptr;
}

extern "C" int trs_build_copy(const trs_builder* B, int id, void* dst, int dst_is_host, void* stream) {
    if (!B || id < 0 || id >= TRS_BUILD_NUM_ARRAYS) return TRS_E_ARG;
    size_t elem;
    const void* src = array_ptr(B, id, &elem);
    const size_t bytes = (size_t)B->sizes[id] * elem;
    if (bytes == 0) return TRS_OK;
    if (!dst) return TRS_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    TRS_CUDA(cudaMemcpyAsync(dst, src, bytes, dst_is_host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, st));
    if (dst_is_host) TRS_CUDA(cudaStreamSynchronize(st));
    return TRS_OK;
}

extern "C" int trs_build_format(trs_builder* B, trs_format* out, void* stream) {
    if (!B || !out) return TRS_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    struct Conv { DevBuf<float>* src; DevBuf<__half>* dst; } conv[3] = {
        {&B->t_value, &B->t_value_h}, {&B->c_value, &B->c_value_h}, {&B->cs_value, &B->cs_value_h}};
    for (auto& c : conv) {
        if (c.dst->p || c.src->n == 0) continue;
        int rc = c.dst->alloc_from(B->arena, c.src->n);
        if (rc) return rc;
        kb_to_half<<<grid_for((long long)c.src->n), 256, 0, st>>>(c.src->p, (long long)c.src->n, c.dst->p);
        TRS_LAUNCH_CHECK();
    }
    memset(out, 0, sizeof(*out));
    out->t_row_offset = B->t_row_offset.p; out->t_block_offset = B->t_block_offset.p; out->t_column = B->t_column.p;
    out->t_value = (const trs_half*)B->t_value_h.p; out->t_window_row = B->t_window_row.p;
    out->t_binary = (const int64_t*)B->t_binary.p;
    out->parts_t = (int)B->t_window_row.n; out->blocks = (int)(B->t_column.n / 8);
    out->c_row_offset = B->c_row_offset.p; out->c_row = B->c_row.p; out->c_column = B->c_column.p;
    out->c_value = (const trs_half*)B->c_value_h.p; out->parts_c = (int)B->c_row.n;
    out->cs_row_offset = B->cs_row_offset.p; out->cs_row = B->cs_row.p; out->cs_column = B->cs_column.p;
    out->cs_value = (const trs_half*)B->cs_value_h.p; out->parts_c_short = (int)B->cs_row.n;
    out->s_window_tile_offset = B->s_window_tile_offset.p; out->s_tile_column = B->s_tile_column.p;
    out->s_packed_a = B->s_packed_a.p; out->s_packed_meta = B->s_packed_meta.p;
    out->num_windows = B->W; out->tiles = (int)B->s_tile_window.n;
    return TRS_OK;
}

namespace {
struct UnitLess {
    const unsigned char* nnz;
    __host__ __device__ bool operator()(int a, int b) const { return nnz[a] > nnz[b]; }
};
}  // namespace

// Host-side run of the std::sort emulation (the same code the matching kernel runs), so that
// it can be checked against libstdc++ without a GPU.
extern "C" int trs_debug_stdsort_order(const unsigned char* keys, int n, int* out, int* heap_sorts) {
    if (n < 0 || (n > 0 && (!keys || !out))) return TRS_E_ARG;
    for (int i = 0; i < n; ++i) out[i] = i;
    StdSort<UnitLess> s(out, UnitLess{keys});
    s.sort(n);
    if (heap_sorts) *heap_sorts = s.heap_sorts;
    return TRS_OK;
}
