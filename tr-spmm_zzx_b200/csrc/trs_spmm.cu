// Fused per-window SpMM over the reference's hybrid format, for sm_100a.
//
// One work item = a 16-row window (or a slice of a heavy window's k-steps) and up to 128 output
// features of it.  A "k-step" is 16 columns of the window:
//   * a packed 2:4 tile  (s_tile_column / s_packed_a / s_packed_meta, block_online.cpp:796-841)
//     -> one mma.sp m16n8k16 per 8 features, or
//   * a pair of dense 16x8 TC blocks (t_column / t_binary / t_value, block_online.cpp:444-540), or
//   * 16 entries of the window's CSR remainder (c_* / cs_* arrays, block_online.cpp:397-439; kernels
//     mGCNkernel.cu:976-1042, 1119-1171), entry k in column k of a 16 x 16 tile
//     -> one dense mma m16n8k16 per 8 features.
// The plan lays the steps of every item out as one stream: 16 column ids per step (64 bytes, the
// items one after the other), and for the dense steps the 16 x 16 A tile expanded in fragment order
// (512 bytes, 16 per lane).  A kernel then needs nothing but a running step number.
//
// Every item belongs to one warp; where the whole matrix is too small to give every SM its warps, to the
// four warps of a CTA (a quarter of the steps each, added through shared memory at the end).  A warp gathers the 16 B rows of a step with 16-byte cp.async
// into its own shared-memory ring, feeds them to the tensor cores with ldmatrix.trans and keeps
// the fp32 accumulators of all 16 x FS outputs in registers across the item.  No block-wide barrier
// exists in the loop.  C is written exactly once: no memset, no atomics, no second output buffer,
// no add kernel (compare mGCNkernel_online.cu:1589-1590, 1689-1712).  Heavy windows are cut into
// several items that write fp32 partial sums to scratch; a second kernel adds them in a fixed order,
// so results are bit-identical from run to run.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <string.h>

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <mutex>
#include <vector>

#include "trs_common.cuh"

namespace trs {

struct Item {        // 32 bytes: everything a warp needs to start
    int window;      // window id
    int slot;        // -1: write C; >=0: write partial sums to scratch slot
    int step0;       // first step of the item in the plan's step stream
    int nsparse;     // steps [0, nsparse) are packed tiles, the rest dense 16 x 16 tiles
    int nsteps;
    int tile0;       // packed tile of step 0
    int dense0;      // dense tile of step nsparse
    int open;        // first packed step of the window, in the stream, with an open slot
};

struct Heavy {
    int window;
    int slot_begin;
    int slot_end;
};

struct WindowRanges {
    int* blk_begin;  // TC block range per window
    int* blk_end;
    int* c_begin;    // long CSR parts per window
    int* c_end;
    int* cs_begin;   // short CSR parts per window
    int* cs_end;
};

struct KernelArgs {
    const Item* items;             // longest first, in window order for a range of windows
    int n_items;
    int w_begin, w_end;            // window range of this run (RANGE instances: items outside return at once)
    const int* ids;                // [steps + kIdSpare][16] column ids of the step stream
    const int* first_ids;          // [n_items][kIdBlock][16] those of the first block of every item, or null
    const uint32_t* packed_a;      // [tiles][64]
    const uint32_t* packed_meta;   // [tiles][8]
    const uint4* dense;            // [dense steps][32] A tiles in fragment order, one uint4 per lane
    const __half* B;
    void* C;
    float* scratch;                // [slots][16][ldS]
    int ldb;                       // elements from one row of B to the next
    int ldS;
    int F;                         // features of C
    int bchunks;                   // 16-byte chunks a row of B really has
    int m_rows, window, out_half;
    int vec_out;                   // rows of C are 16-byte aligned
    int relu;                      // 1: C = max(A'B, 0) (GCN layer epilogue)
    void* peers[8];                // fused exchange: the fp16 rows are written into every one of these
    int n_peers;                   //   [N_total, F] buffers (this GPU's and its NVLink peers'), 0 = off
    long long peer_row0;           //   at global row peer_row0 + local row
    bool behind;                   // host: launched behind the kernel that copies B
};

// ----------------------------------------------------------------------------------------------
// plan preparation kernels
// ----------------------------------------------------------------------------------------------
__global__ void k_part_ranges(const int* __restrict__ key, const int* __restrict__ prefix, int n, int div,
                              int num_windows, int* __restrict__ begin, int* __restrict__ end, int use_prefix) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    int w = key[p] / div;
    if (w < 0 || w >= num_windows) return;  // reported by validation
    int lo = use_prefix ? prefix[p] : p;
    int hi = use_prefix ? prefix[p + 1] : p + 1;
    if (p == 0 || key[p - 1] / div != w) begin[w] = lo;
    if (p == n - 1 || key[p + 1] / div != w) end[w] = hi;
}

// Entries of a window's CSR remainder: long parts first, then short parts.
__device__ __forceinline__ int csr_entries(const trs_format& f, const WindowRanges& wr, int w, int pass) {
    const int b = pass ? wr.cs_begin[w] : wr.c_begin[w], e = pass ? wr.cs_end[w] : wr.c_end[w];
    const int* off = pass ? f.cs_row_offset : f.c_row_offset;
    return e > b ? max(off[e] - off[b], 0) : 0;
}
struct WindowSteps {
    int tiles, tc, ce;  // packed tiles, pairs of TC blocks, groups of 16 CSR entries
};
__device__ __forceinline__ WindowSteps window_steps(const trs_format& f, const WindowRanges& wr, int w) {
    WindowSteps s;
    s.tiles = w < f.num_windows ? f.s_window_tile_offset[w + 1] - f.s_window_tile_offset[w] : 0;
    s.tc = (wr.blk_end[w] - wr.blk_begin[w] + 1) / 2;
    s.ce = (csr_entries(f, wr, w, 0) + csr_entries(f, wr, w, 1) + 15) / 16;
    return s;
}

// Per-window counts (arrays of W + 1, the last entry zero, scanned afterwards): steps and dense
// steps first, then items, split-window flag and scratch slots, which depend on the total.
constexpr int kWindowCounts = 5;
enum { WC_STEPS, WC_DENSE, WC_ITEMS, WC_HEAVY, WC_SLOTS };
__global__ void k_count_steps(trs_format f, WindowRanges wr, int num_windows, int* __restrict__ cnt) {
    int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > num_windows) return;
    const size_t stride = (size_t)num_windows + 1;
    WindowSteps s = {0, 0, 0};
    if (w < num_windows) s = window_steps(f, wr, w);
    cnt[WC_STEPS * stride + w] = s.tiles + s.tc + s.ce;
    cnt[WC_DENSE * stride + w] = s.tc + s.ce;
}

// Longest run of steps one item takes.  An item should not be longer than the average share of a warp
// slot (16 warps per SM at 128 features), or the longest ones are still running when the rest is
// done; below 32 steps the extra partial sums cost more than the shorter tail gives, above 512 nothing
// is left to gain.  Measured best at R-MAT scale 14 / 16 / 17 / 18 / 19 / 20 / 21, F = 128: 32 / 48 / 96 / 192 / 256 / 384 / 512
// steps; 256 for all of them took 57 / 66 / 118 / 148 / 277 / 589 / 2080 us against 21 / 43 / 74 / 143 / 277 / 554 / 2049.
// With less than six steps per warp slot items get four warps each anyway (warps_per_item) and may be four times as long.
// Windows of ordinary length are left whole, though: cutting nearly all of them in two doubles the time (uniform 24000, 32
// entries per row, 33 steps per window, F = 32 / 128 / 512: 17 / 40 / 126 us in items of 17 steps, 10 / 20 / 58 whole).  A matrix
// of few long windows needs the cuts to fill the GPU: below one window per four warp slots they stop at 128 steps.
constexpr int kWarpsPerSm = 16, kFewSteps = 6;
__host__ __device__ __forceinline__ int item_steps(int total_steps, int windows, int sms) {
    const int share = total_steps / (sms * kWarpsPerSm);
    if (share < kFewSteps) return 128;
    const int whole = min((int)(3ll * total_steps / (2 * windows)), 4 * windows < sms * kWarpsPerSm ? 128 : 512);
    return min(max(max(share, 32), whole), 512);
}

// One warp per item or four.  A step of a lone warp takes about five times as long as the SM needs for one with its warps
// all at work, a warp's start and end as long as twelve steps in the one sense and three in the other; an item of four
// warps adds twenty (it ends with two barriers and a sum).  So, in steps of an SM, the time is the longer of its longest
// item and of all its items.  R-MAT 13, F = 64 / 128 / 512, 1 -> 4 warps: 27 / 34 / 38 -> 14 / 18 / 31 us; uniform 8192, 32
// entries per row, F = 128 / 256: 12.4 / 15.4 -> 11.2 / 18.5; uniform 32768, 4 entries per row, F = 64 / 256: 8.0 / 14.4 -> 11.0 / 28.7.
static int warps_per_item(int items, long long steps, int longest, int slabs, int sms) {
    const long long one = std::max(5ll * (longest + 12), slabs * (steps + 3ll * items) / sms);
    const long long four = std::max(5ll * (longest / 4 + 12), slabs * (steps + 20ll * items) / sms);
    return four < one ? 4 : 1;
}

// Where scratch for the partial sums is short (the fixed array of trs_spmm_run_static), windows are cut at 256 steps and no
// earlier: a matrix below R-MAT scale 19 has several times the slots otherwise.
constexpr int kCoarseSteps = 256;
struct Cut {          // of all windows together
    int items, heavy, slots;
    int longest;      // steps of the longest item
};
__device__ __forceinline__ int cut_window(int steps, int chunk) { return max(1, (steps + chunk - 1) / chunk); }

__global__ void k_count_items(int num_windows, int chunk, int sms, const int* __restrict__ step_off, int* __restrict__ cnt,
                              int* __restrict__ longest, Cut* __restrict__ coarse) {
    int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (chunk <= 0) chunk = item_steps(step_off[num_windows], num_windows, sms);
    const bool live = w < num_windows;
    const int steps = live ? step_off[w + 1] - step_off[w] : 0, lane = threadIdx.x & 31;
    const int items = live ? cut_window(steps, chunk) : 0;
    const int most = __reduce_max_sync(0xffffffffu, live ? (steps + items - 1) / items : 0);
    if (lane == 0 && most > *longest) atomicMax(longest, most);
    if (chunk < kCoarseSteps) {
        const int n = live ? cut_window(steps, kCoarseSteps) : 0;
        const int all = __reduce_add_sync(0xffffffffu, n), heavy = __popc(__ballot_sync(0xffffffffu, n > 1));
        const int slots = __reduce_add_sync(0xffffffffu, n > 1 ? n : 0);
        const int coarsest = __reduce_max_sync(0xffffffffu, live ? (steps + n - 1) / n : 0);
        if (lane == 0) {
            atomicAdd(&coarse->items, all);
            if (heavy) { atomicAdd(&coarse->heavy, heavy); atomicAdd(&coarse->slots, slots); }
            if (coarsest > coarse->longest) atomicMax(&coarse->longest, coarsest);
        }
    }
    if (w > num_windows) return;
    const size_t stride = (size_t)num_windows + 1;
    cnt[WC_ITEMS * stride + w] = items;
    cnt[WC_HEAVY * stride + w] = items > 1 ? 1 : 0;
    cnt[WC_SLOTS * stride + w] = items > 1 ? items : 0;
}

// The items of window w: n of them from items[0], the slots from slot0 if there is more than one.
__device__ __forceinline__ void fill_window(const trs_format& f, int w, int num_windows, const int* __restrict__ off, int n, int slot0,
                                            int open, Item* __restrict__ items, Heavy* __restrict__ heavy) {
    const size_t stride = (size_t)num_windows + 1;
    const int step0 = off[WC_STEPS * stride + w], steps = off[WC_STEPS * stride + w + 1] - step0;
    const int dense0 = off[WC_DENSE * stride + w];
    const int tile0 = w < f.num_windows ? f.s_window_tile_offset[w] : 0;
    const int tiles = w < f.num_windows ? f.s_window_tile_offset[w + 1] - tile0 : 0;
    // split evenly so that no item is much shorter than the others
    const int per = (steps + n - 1) / n;
    for (int i = 0; i < n; ++i) {
        const int b = min(i * per, steps), e = min(b + per, steps);
        items[i] = Item{w, n > 1 ? slot0 + i : -1, step0 + b, min(max(tiles - b, 0), e - b), e - b, tile0 + b,
                        dense0 + max(b - tiles, 0), open};
    }
    if (n > 1) *heavy = Heavy{w, slot0, slot0 + n};
}

__global__ void k_fill_items(trs_format f, int num_windows, const int* __restrict__ off, Item* __restrict__ items,
                             Heavy* __restrict__ heavy) {
    int w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= num_windows) return;
    const size_t stride = (size_t)num_windows + 1;
    const int i0 = off[WC_ITEMS * stride + w];
    fill_window(f, w, num_windows, off, off[WC_ITEMS * stride + w + 1] - i0, off[WC_SLOTS * stride + w], 0x7fffffff, items + i0,
                heavy + off[WC_HEAVY * stride + w]);
}

// The coarse items, in no particular order (their windows' partial sums are still added in theirs).  `made`: cleared.
__global__ void k_fill_coarse(trs_format f, int num_windows, const int* __restrict__ off, const int* __restrict__ open,
                              Cut* __restrict__ made, Item* __restrict__ items, Heavy* __restrict__ heavy) {
    const int w = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const int* const step_off = off + WC_STEPS * ((size_t)num_windows + 1);
    const int n = w < num_windows ? cut_window(step_off[w + 1] - step_off[w], kCoarseSteps) : 0, s = n > 1 ? n : 0;
    int items_to = n, slots_to = s;   // up to this lane's
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, items_to, d), z = __shfl_up_sync(0xffffffffu, slots_to, d);
        if (lane >= d) { items_to += y; slots_to += z; }
    }
    const unsigned split = __ballot_sync(0xffffffffu, n > 1);
    int i0 = 0, slot0 = 0, h0 = 0;
    if (lane == 31) {
        i0 = atomicAdd(&made->items, items_to);
        if (split) { slot0 = atomicAdd(&made->slots, slots_to); h0 = atomicAdd(&made->heavy, __popc(split)); }
    }
    i0 = __shfl_sync(0xffffffffu, i0, 31) + items_to - n;
    slot0 = __shfl_sync(0xffffffffu, slot0, 31) + slots_to - s;
    h0 = __shfl_sync(0xffffffffu, h0, 31) + __popc(split & ((1u << lane) - 1u));
    if (n > 0) fill_window(f, w, num_windows, off, n, slot0, open[w], items + i0, heavy + h0);
}

// The step stream, one warp per item.  An unused column slot of a step repeats the step's first column, so that the gather
// needs no special case.  Its A entries are zero, but zero times an infinity is not: where the multiplication looks at such
// a slot - always in a dense tile, in a packed one if a row's metadata names it - the slot stays open (-1), and the
// gather fills it with zeros.  `open[w]`: the window's first packed step with an open slot.
__global__ void k_fill_steps(trs_format f, WindowRanges wr, const Item* __restrict__ items, int n_items,
                             const int* __restrict__ off, int num_windows, int window, int* __restrict__ ids,
                             uint4* __restrict__ dense, int* __restrict__ open) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= n_items) return;
    const Item it = items[i];
    const int w = it.window;
    for (int j = 0; j < it.nsparse; ++j) {
        int c = -1;
        if (lane < 16) c = f.s_tile_column[(size_t)(it.tile0 + j) * 16 + lane];
        const unsigned have = __ballot_sync(0xffffffffu, c >= 0);
        const int dup = have ? __shfl_sync(0xffffffffu, c, __ffs(have) - 1) : 0;
        bool is_open = false;
        if (have != 0xffffu) {
            unsigned used = 0;   // slots that a row's two positions per group name
            if (lane < 8) {
                const unsigned m = f.s_packed_meta[(size_t)(it.tile0 + j) * 8 + lane];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    used |= ((1u << ((m >> (4 * i)) & 3u)) | (1u << ((m >> (4 * i + 2)) & 3u))) << (4 * (i & 3));
            }
            is_open = (__reduce_or_sync(0xffffffffu, used) & ~have) != 0;
            if (is_open && lane == 0) atomicMin(open + w, it.step0 + j);
        }
        if (lane < 16) ids[((size_t)it.step0 + j) * 16 + lane] = c >= 0 ? c : is_open ? -1 : dup;
    }
    if (it.nsteps == it.nsparse) return;
    const WindowSteps ws = window_steps(f, wr, w);
    const int blk0 = wr.blk_begin[w], blk_end = wr.blk_end[w];
    const int n_long = csr_entries(f, wr, w, 0), n_short = csr_entries(f, wr, w, 1);
    const int rel = it.dense0 - off[WC_DENSE * ((size_t)num_windows + 1) + w];  // dense steps of the window before this item
    const int g = lane >> 2, t = lane & 3;
    for (int j = it.nsparse; j < it.nsteps; ++j) {
        const int d = rel + j - it.nsparse;
        int c = -1;
        uint32_t a[4] = {0u, 0u, 0u, 0u};
        if (d < ws.tc) {
            const int b = blk0 + 2 * d + ((lane >> 3) & 1);
            if (lane < 16 && b < blk_end) c = f.t_column[(size_t)b * 8 + (lane & 7)];
            // fragment word q: row g + 8 (q & 1), columns 2t, 2t + 1 of block q >> 1
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int bq = blk0 + 2 * d + (q >> 1);
                if (bq >= blk_end) continue;
                const unsigned long long lo = (unsigned long long)f.t_binary[(size_t)bq * 2];
                const unsigned long long hi = (unsigned long long)f.t_binary[(size_t)bq * 2 + 1];
                const unsigned long long m = (q & 1) ? hi : lo;
                const __half* v = (const __half*)f.t_value + f.t_block_offset[bq];
                const int bit = g * 8 + 2 * t;
                int rank = __popcll(m & ((1ull << bit) - 1ull)) + ((q & 1) ? __popcll(lo) : 0);
                if ((m >> bit) & 1ull) { a[q] = __half_as_ushort(v[rank]); ++rank; }
                if ((m >> (bit + 1)) & 1ull) a[q] |= (uint32_t)__half_as_ushort(v[rank]) << 16;
            }
        } else {
            // lane k < 16 finds entry k of the group: its part by binary search in the window's prefix
            const int e = (d - ws.tc) * 16 + lane;
            uint32_t ent = 0xffffu << 16;  // value | local row << 16; row 0xffff matches no row
            if (lane < 16 && e < n_long + n_short) {
                const bool is_short = e >= n_long;
                const int* roff = is_short ? f.cs_row_offset : f.c_row_offset;
                int lo = is_short ? wr.cs_begin[w] : wr.c_begin[w], hi = is_short ? wr.cs_end[w] : wr.c_end[w];
                const int at = roff[lo] + (is_short ? e - n_long : e);
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (roff[mid] <= at) lo = mid; else hi = mid;
                }
                const int row = (is_short ? f.cs_row : f.c_row)[lo];
                c = (is_short ? f.cs_column : f.c_column)[at];
                ent = (uint32_t)((is_short ? f.cs_value : f.c_value)[at]) | ((uint32_t)(row - w * window) << 16);
            }
            // fragment word q: row g + 8 (q & 1), entries 2t + 8 (q >> 1) and the next one
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t row = (uint32_t)(g + 8 * (q & 1));
                const uint32_t e0 = __shfl_sync(0xffffffffu, ent, 2 * t + 8 * (q >> 1));
                const uint32_t e1 = __shfl_sync(0xffffffffu, ent, 2 * t + 8 * (q >> 1) + 1);
                if ((e0 >> 16) == row) a[q] = e0 & 0xffffu;
                if ((e1 >> 16) == row) a[q] |= e1 << 16;
            }
        }
        if (lane < 16) ids[((size_t)it.step0 + j) * 16 + lane] = c;
        dense[((size_t)it.dense0 + j - it.nsparse) * 32 + lane] = make_uint4(a[0], a[1], a[2], a[3]);
    }
}

// The first block of column ids of every item, one warp each (it may go past the item's and the stream's end: kIdSpare).
__global__ void k_first_ids(const Item* __restrict__ items, int n_items, const int* __restrict__ ids, int* __restrict__ first) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i < n_items) ((int4*)first)[(size_t)i * 32 + lane] = ((const int4*)(ids + (size_t)items[i].step0 * 16))[lane];
}

// Validation: every violated rule ORs one bit into *err.
enum { V_OFFSETS = 1, V_COLUMN = 2, V_ROW = 4, V_SHAPE = 8 };

__global__ void k_check_prefix(const int* __restrict__ a, int n, int expect_last, int* err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0 && a[0] != 0) atomicOr(err, V_OFFSETS);
    if (i + 1 < n && a[i + 1] < a[i]) atomicOr(err, V_OFFSETS);
    if (i == n - 1 && expect_last >= 0 && a[i] != expect_last) atomicOr(err, V_SHAPE);
}
__global__ void k_check_range(const int* __restrict__ a, long long n, int lo, int hi, int bit, int* err) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int v = a[i];
    if (v < lo || v >= hi) atomicOr(err, bit);
}
// Launch-order class of an item: long items first, so that the last wave of the grid consists of
// short ones.  Classes of 8 steps (four classes over the whole range measured 4 - 6 % slower).
constexpr int kClassBits = 6;
__global__ void k_item_class(Item* __restrict__ items, int n, const int* __restrict__ open, unsigned char* __restrict__ cls) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    cls[i] = (unsigned char)(63 - min(items[i].nsteps / 8, 63));
    items[i].open = open[items[i].window];
}

// The TC kernels read t_value[t_block_offset[b] + rank] with rank taken from the block's two
// bitmaps, so the bitmaps' population must equal the block's share of t_value.
__global__ void k_check_tc_popcount(const long long* __restrict__ t_binary, const int* __restrict__ t_block_offset,
                                    int blocks, int* err) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= blocks) return;
    const int bits = __popcll((unsigned long long)t_binary[2 * (size_t)b]) + __popcll((unsigned long long)t_binary[2 * (size_t)b + 1]);
    if (bits != t_block_offset[b + 1] - t_block_offset[b]) atomicOr(err, V_SHAPE);
}
__global__ void k_check_sorted(const int* __restrict__ a, int n, int* err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i + 1 < n && a[i + 1] < a[i]) atomicOr(err, V_OFFSETS);
}

// ----------------------------------------------------------------------------------------------
// The kernel: one warp per work item, no block-wide synchronisation in the loop.
// ----------------------------------------------------------------------------------------------
// What bounds it: one 16-byte-chunked row of B per (window, column) pair has to come through L2 - 27.5 GB
// at R-MAT scale 21, F = 128, 1.83 ms for a kernel that does nothing else.  With four warps per
// scheduler the rate at which a warp gets through its own instruction stream decides how close a
// kernel comes; hence no predicates, no address arithmetic but one multiply-add per row, constant
// ring offsets in the instructions, and a loop of its own for packed tiles: 95 instructions per step instead
// of 223, 2.64 -> 2.05 ms at scale 21 (13.4 TB/s), 0.76 -> 0.55 ms at scale 20, 0.128 -> 0.097 ms clustered.
//
// FS = features per warp (a multiple of 16 up to 128; F > 128 adds feature slabs on gridDim.y).
// Per k-step the warp copies the 16 gathered rows (FS * 2 bytes each) with FS / 16 cp.async
// instructions of 16 bytes per lane into a stage of its own ring - rows unpadded, the 16-byte chunks
// of a row swizzled by the row number so that ldmatrix is conflict-free.  Column ids come in blocks
// of 8 steps (512 bytes, one cp.async per lane).  The A operand goes straight into registers
// STAGES - 1 steps ahead, so the ring holds gathered rows only.
constexpr int kIdBlock = 8;   // steps per block of column ids
// Step j of an item, j a multiple of kIdBlock, asks for the ids of steps j + kIdBlock .. j + 2 kIdBlock - 1, whether the
// item has them or not, so the array goes on that far behind the last step.
constexpr int kIdSpare = 2 * kIdBlock;

template <int FS, int STAGES>
struct WarpTile {
    static constexpr int NT = FS / 8;               // n-tiles (8 features) per warp
    static constexpr int CPR = FS / 8;              // 16-byte chunks per gathered row
    static constexpr int NCP = CPR / 2;             // cp.async instructions per lane and step
    static constexpr bool POW2 = (CPR & (CPR - 1)) == 0;
    static constexpr int ROWB = FS * 2;             // no padding: the chunks of a row are swizzled
    static constexpr int STAGE = 16 * ROWB;
    static constexpr int AHEAD = STAGES - 1;        // rows and A operand run this many steps ahead
    static constexpr int IDS = 2 * kIdBlock * 64;
    static constexpr int SMEM = STAGE * STAGES + IDS;
    static_assert(FS % 16 == 0 && FS <= 128 && STAGES >= 2 && AHEAD <= kIdBlock, "");
    static_assert(SMEM >= 16 * (FS * 4 + 16), "the epilogue stages a 16 x FS fp32 tile in the ring");
    // chunk c of row r sits at position c ^ swz(r): the 8 rows one ldmatrix phase reads land in 8
    // different 16-byte bank groups (a row is FS / 8 chunks long; an odd multiple of 2 chunks needs one
    // swizzle bit, an odd multiple of 4 two, a multiple of 8 three)
    __device__ static constexpr int swz(int r) {
        return (FS / 16) & 1 ? ((r >> 2) & 1) : ((FS / 32) & 1 ? ((r >> 1) & 3) : (r & 7));
    }
};

// Rows of the item's result leave the warp's (drained) ring: `tile` holds 16 rows of FS fp32 (or fp16
// when HALF) with the given pitch.  Called by `nthreads` threads numbered `tid`.
template <int FS>
__device__ __forceinline__ void store_rows(const unsigned char* tile, bool half_tile, const Item& it, const KernelArgs& a,
                                           int fbase, int tid, int nthreads) {
    const bool partial = it.slot >= 0;
    if (half_tile) {
        constexpr int PITCH = FS * 2 + 16, CPR = FS / 8;
        if (a.vec_out) {
            for (int c = tid; c < 16 * CPR; c += nthreads) {
                const int lr = c / CPR, ch = c % CPR;
                const int f = fbase + ch * 8;
                const long long row = (long long)it.window * a.window + lr;
                if (lr >= a.window || row >= a.m_rows || f >= a.F) continue;
                const uint4 v = *(const uint4*)(tile + lr * PITCH + ch * 16);
                if (a.n_peers > 0) {
                    const size_t off = (size_t)(a.peer_row0 + row) * (size_t)a.F + f;
                    for (int d = 0; d < a.n_peers; ++d) *(uint4*)((__half*)a.peers[d] + off) = v;
                } else {
                    __stcs((uint4*)((__half*)a.C + (size_t)row * a.F + f), v);
                }
            }
        } else {
            for (int c = tid; c < 16 * FS; c += nthreads) {
                const int lr = c / FS, f = fbase + c % FS;
                const long long row = (long long)it.window * a.window + lr;
                if (lr >= a.window || row >= a.m_rows || f >= a.F) continue;
                ((__half*)a.C)[(size_t)row * a.F + f] = *(const __half*)(tile + lr * PITCH + (c % FS) * 2);
            }
        }
        return;
    }
    constexpr int PITCH = FS * 4 + 16, CPR = FS / 4;
    if (partial || a.vec_out) {
        float* dst = partial ? a.scratch + (size_t)it.slot * 16 * (size_t)a.ldS : (float*)a.C;
        const int ld = partial ? a.ldS : a.F;
        for (int c = tid; c < 16 * CPR; c += nthreads) {
            const int lr = c / CPR, ch = c % CPR;
            const int f = fbase + ch * 4;
            const long long row = (long long)it.window * a.window + lr;
            if (f >= ld) continue;
            if (!partial && (lr >= a.window || row >= a.m_rows)) continue;
            const float4 v = *(const float4*)(tile + lr * PITCH + ch * 16);
            float4* d = (float4*)(dst + (partial ? (size_t)lr : (size_t)row) * ld + f);
            if (partial) *d = v;
            else __stcs(d, v);
        }
    } else {
        for (int c = tid; c < 16 * FS; c += nthreads) {
            const int lr = c / FS, f = fbase + c % FS;
            const long long row = (long long)it.window * a.window + lr;
            if (lr >= a.window || row >= a.m_rows || f >= a.F) continue;
            ((float*)a.C)[(size_t)row * a.F + f] = *(const float*)(tile + lr * PITCH + (c % FS) * 4);
        }
    }
}

// Accumulators are in mma fragment layout: acc[n][2h + i] = row g + 8h, feature 8n + 2t + i.
template <int FS>
__device__ __forceinline__ void stage_acc(const float (&acc)[FS / 8][4], bool half_tile, unsigned char* tile, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < FS / 8; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (half_tile) *(__half2*)(tile + (g + 8 * h) * (FS * 2 + 16) + (8 * n + 2 * t) * 2) = __floats2half2_rn(acc[n][2 * h], acc[n][2 * h + 1]);
            else *(float2*)(tile + (g + 8 * h) * (FS * 4 + 16) + (8 * n + 2 * t) * 4) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
        }
}

// 8 features of a B row that does not start on a 16-byte boundary
__device__ __forceinline__ uint4 load_unaligned8(const __half* p, int n) {
    unsigned short v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i < n ? __ldg((const unsigned short*)p + i) : (unsigned short)0;
    return make_uint4(v[0] | (uint32_t)v[1] << 16, v[2] | (uint32_t)v[3] << 16, v[4] | (uint32_t)v[5] << 16,
                      v[6] | (uint32_t)v[7] << 16);
}

template <int N, int I = 0, class Fn>
__device__ __forceinline__ void static_for(Fn&& fn) {
    if constexpr (I < N) {
        fn(std::integral_constant<int, I>());
        static_for<N, I + 1>(fn);
    }
}
template <int FS, int BASE, bool SPARSE, int H = 0>
__device__ __forceinline__ void compute_steps(float (&acc)[FS / 8][4], const uint32_t (&laddr)[4], const uint4& av) {
    if constexpr (H < FS / 16) {
        uint32_t b0, b1, b2, b3;
        ldmatrix_x4_trans_at<(H >> 2) * 128 + BASE>(laddr[H & 3], b0, b1, b2, b3);
        if constexpr (SPARSE) {
            mma_sp_16816(acc[2 * H], av.x, av.y, b0, b1, av.z);
            mma_sp_16816(acc[2 * H + 1], av.x, av.y, b2, b3, av.z);
        } else {
            mma_16816(acc[2 * H], av.x, av.y, av.z, av.w, b0, b1);
            mma_16816(acc[2 * H + 1], av.x, av.y, av.z, av.w, b2, b3);
        }
        compute_steps<FS, BASE, SPARSE, H + 1>(acc, laddr, av);
    }
}

// WPI warps share an item (each takes a contiguous share of its steps, the shares are added in
// warp order at the end).  ALIGNED: rows of B start on 16-byte boundaries; otherwise they are
// gathered with 2-byte loads (callers that can neither align B nor lend memory for a padded copy).
template <int FS, int STAGES, int WPI, int MINB, bool ALIGNED, bool RANGE, bool RAGGED>
__global__ void __launch_bounds__(32 * WPI, MINB) k_window_spmm_warp(const KernelArgs a) {
    using T = WarpTile<FS, STAGES>;
    extern __shared__ __align__(128) unsigned char smem_all[];
    const int lane = threadIdx.x & 31;
    const int wid = WPI > 1 ? threadIdx.x >> 5 : 0;
    unsigned char* const smem = smem_all + wid * T::SMEM;
    const int fbase = blockIdx.y * FS;

    // The first column ids do not wait for the item where they lie beside it: a start is one trip to memory shorter.  64 features
    // alone: the instance spills less with it too (262144 clustered rows 63.7 -> 61.7 us, 131072 uniform ones 34.9 -> 33.3, R-MAT 18
    // lossless 93.3 -> 90.4); 128 gain nothing, 16, 32 and 96 lose 2 to 7 %.
    const bool beside = FS == 64 && WPI == 1 && ALIGNED && !RANGE && a.first_ids;
    if (beside) cp_async16(smem_u32(smem) + T::STAGE * STAGES + lane * 16, a.first_ids + (size_t)blockIdx.x * (kIdBlock * 16) + lane * 4);
    const Item it = a.items[blockIdx.x];
    if constexpr (RANGE) {   // a test in the whole-matrix instance costs up to 20 % (it delays the first ids of short items)
        if (it.window < a.w_begin || it.window >= a.w_end) return;
    }
    int first = 0, nsteps = it.nsteps;
    if constexpr (WPI > 1) {
        const int per = (it.nsteps + WPI - 1) / WPI;
        first = min(wid * per, it.nsteps);
        nsteps = min(first + per, it.nsteps) - first;
    }
    const int nsparse = min(max(it.nsparse - first, 0), nsteps);
    const int nclosed = min(max(it.open - it.step0 - first, 0), nsparse);   // packed tiles before the first with an open slot
    const int* const ids = a.ids + ((size_t)it.step0 + first) * 16;
    const uint32_t* const pa = a.packed_a + (size_t)(it.tile0 + first) * 64 + lane * 2;
    const uint32_t* const pm = a.packed_meta + (size_t)(it.tile0 + first) * 8 + (lane >> 2);
    const uint4* const pd = a.dense + ((long long)it.dense0 + max(first - it.nsparse, 0) - nsparse) * 32 + lane;

    const uint32_t smem0 = smem_u32(smem);
    constexpr int ids_at = T::STAGE * STAGES;

    // gather role of this lane: T::NCP pieces of 16 bytes, piece k = chunk pc[k] of row pr[k]
    int pr[T::NCP], pc[T::NCP];
    uint32_t pdst[T::NCP];
#pragma unroll
    for (int k = 0; k < T::NCP; ++k) {
        if (T::POW2) { pr[k] = lane / T::CPR * T::NCP + k; pc[k] = lane % T::CPR; }
        else { pr[k] = (k * 32 + lane) / T::CPR; pc[k] = (k * 32 + lane) % T::CPR; }
        pdst[k] = smem0 + pr[k] * T::ROWB + ((pc[k] ^ T::swz(pr[k])) << 4);
    }
    const uint32_t pitch = (uint32_t)a.ldb * 2u;
    // A chunk beyond the end of the row repeats the last one, or, RAGGED, is not copied; its features are not stored
    const unsigned char* src0[T::POW2 ? 1 : T::NCP];
    bool in_row[T::POW2 ? 1 : T::NCP];
#pragma unroll
    for (int k = 0; k < (T::POW2 ? 1 : T::NCP); ++k) {
        in_row[k] = !RAGGED || fbase / 8 + pc[k] < a.bchunks;
        src0[k] = (const unsigned char*)a.B + (size_t)(min(fbase / 8 + pc[k], a.bchunks - 1)) * 16;
    }
    auto src_of = [&](int k) -> const unsigned char* { return src0[T::POW2 ? 0 : k]; };
    // ldmatrix role: matrix lane / 8 -> k rows (m & 1) * 8 .., features (m >> 1) * 8 ..
    const int lrow = (lane & 7) + ((lane >> 3) & 1) * 8, lchunk = lane >> 4;
    uint32_t laddr[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) laddr[q] = smem0 + lrow * T::ROWB + (((2 * q + lchunk) ^ T::swz(lrow)) << 4);

    float acc[T::NT][4];
#pragma unroll
    for (int i = 0; i < T::NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    auto issue_ids = [&](int blk) {   // ids of steps 8 blk .. 8 blk + 7
        cp_async16(smem0 + ids_at + (blk & 1) * (kIdBlock * 64) + lane * 16, ids + blk * (kIdBlock * 16) + lane * 4);
    };
    // `tested`: the step may have open slots
    auto gather = [&](int j, auto stage, auto tested) {
        const unsigned char* idp = smem + ids_at + (j & (2 * kIdBlock - 1)) * 64;
        int c[T::NCP];
        if constexpr (T::POW2 && T::NCP >= 4) {
#pragma unroll
            for (int k = 0; k < T::NCP; k += 4) {
                const int4 x = *(const int4*)(idp + pr[k] * 4);
                c[k] = x.x; c[k + 1] = x.y; c[k + 2] = x.z; c[k + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < T::NCP; ++k) c[k] = *(const int*)(idp + pr[k] * 4);
        }
#pragma unroll
        for (int k = 0; k < T::NCP; ++k) {
            if constexpr (ALIGNED) {
                if (!in_row[T::POW2 ? 0 : k]) continue;
                if constexpr (decltype(tested)::value)   // without a branch: 105 against 109 - 113 us with one (clustered, F = 128)
                    cp_async16(pdst[k] + decltype(stage)::value * T::STAGE,
                               src_of(k) + (unsigned long long)(uint32_t)max(c[k], 0) * pitch, (~c[k] >> 27) & 16);
                else
                    cp_async16_at<decltype(stage)::value * T::STAGE>(pdst[k], src_of(k) + (unsigned long long)(uint32_t)c[k] * pitch);
            } else {
                const int f = fbase + pc[k] * 8;
                *(uint4*)(smem + (pdst[k] - smem0) + decltype(stage)::value * T::STAGE) = load_unaligned8(a.B + (size_t)max(c[k], 0) * a.ldb + f, c[k] < 0 ? 0 : a.F - f);
            }
        }
    };
    // A operand of step j: a packed tile gives this lane its 8 bytes of values (x, y) and its metadata
    // word (z), a dense tile the four fragment words
    auto load_a = [&](int j) -> uint4 {
        uint4 r;
        if (j < nsparse) {
            const uint2 v = __ldg((const uint2*)(pa + (size_t)j * 64));
            r = make_uint4(v.x, v.y, __ldg(pm + (size_t)j * 8), 0u);
        } else {
            r = __ldg(pd + (size_t)j * 32);
        }
        return r;
    };
    auto compute_sparse = [&](auto stage, const uint4& av) {
        compute_steps<FS, decltype(stage)::value * T::STAGE, true>(acc, laddr, av);
    };
    auto compute = [&](int j, auto stage, const uint4& av) {
        if (j < nsparse) compute_steps<FS, decltype(stage)::value * T::STAGE, true>(acc, laddr, av);
        else compute_steps<FS, decltype(stage)::value * T::STAGE, false>(acc, laddr, av);
    };
    // rows and A operand of step j, and with every eighth step the ids of the block after its own:
    // they land before the first step that reads them is gathered (AHEAD <= 8 steps earlier), in the
    // half of the id ring whose last reader was the step before j
    // Outside the whole rounds, steps that have no open slots may be asked for instead of tested, a branch against two
    // instructions per piece.  Seven graphs, against steps that are all taken as closed: F = 16 / 48 / 56 / 72 0.98 / 0.99 / 1.06 /
    // 1.04 times tested, 0.97 / 0.93 / 1.00 / 0.97 asked for; F = 32 / 96 / 128 the other way round by 1 to 4 %.
    constexpr bool kAsk = FS == 16 || FS == 48 || FS == 64 || FS == 80;
    uint4 areg[STAGES];
    auto fetch = [&](int j, auto stage) {
        if ((j & (kIdBlock - 1)) == 0) issue_ids(j / kIdBlock + 1);
        if (kAsk && j < nclosed) {
            const uint2 v = __ldg((const uint2*)(pa + (size_t)j * 64));
            areg[decltype(stage)::value] = make_uint4(v.x, v.y, __ldg(pm + (size_t)j * 8), 0u);
            gather(j, stage, std::false_type());
        } else {
            areg[decltype(stage)::value] = load_a(j);
            gather(j, stage, std::true_type());
        }
    };

    if (nsteps > 0) {
        if (!beside) issue_ids(0);
        cp_async_commit();
        wait_for_kernel_before();   // the copy of B, where there is one
        cp_async_wait<0>();
        __syncwarp();
    }
    static_for<T::AHEAD>([&](auto u) {
        constexpr int j = decltype(u)::value;
        if (j < nsteps) fetch(j, u);
        cp_async_commit();
    });
    // group j carries the rows of step j; at iteration j all groups but the newest STAGES - 2 are complete
    int j = 0;
    // whole rounds of packed tiles without open slots
    for (; j + STAGES + T::AHEAD <= nclosed; j += STAGES) {
        static_for<STAGES>([&](auto uu) {
            constexpr int u = decltype(uu)::value, un = (u + T::AHEAD) % STAGES;
            cp_async_wait<STAGES - 2>();
            __syncwarp();
            const int jn = j + u + T::AHEAD;
            if ((jn & (kIdBlock - 1)) == 0) issue_ids(jn / kIdBlock + 1);
            {
                const uint2 v = __ldg((const uint2*)(pa + (size_t)jn * 64));
                areg[un] = make_uint4(v.x, v.y, __ldg(pm + (size_t)jn * 8), 0u);
            }
            gather(jn, std::integral_constant<int, un>(), std::false_type());
            cp_async_commit();
            compute_sparse(uu, areg[u]);
        });
    }
    for (; j < nsteps; j += STAGES) {
        if (j >= nsparse && j + STAGES + T::AHEAD <= nsteps) {   // a whole round of dense tiles
            static_for<STAGES>([&](auto uu) {
                constexpr int u = decltype(uu)::value, un = (u + T::AHEAD) % STAGES;
                cp_async_wait<STAGES - 2>();
                __syncwarp();
                const int jn = j + u + T::AHEAD;
                if ((jn & (kIdBlock - 1)) == 0) issue_ids(jn / kIdBlock + 1);
                areg[un] = __ldg(pd + (size_t)jn * 32);
                gather(jn, std::integral_constant<int, un>(), std::true_type());
                cp_async_commit();
                compute_steps<FS, u * T::STAGE, false>(acc, laddr, areg[u]);
            });
            continue;
        }
        static_for<STAGES>([&](auto uu) {
            constexpr int u = decltype(uu)::value, un = (u + T::AHEAD) % STAGES;
            if (j + u < nsteps) {
                cp_async_wait<STAGES - 2>();
                __syncwarp();
                if (j + u + T::AHEAD < nsteps) fetch(j + u + T::AHEAD, std::integral_constant<int, un>());
                cp_async_commit();
                compute(j + u, uu, areg[u]);
            }
        });
    }
    cp_async_wait<0>();
    __syncwarp();

    // ---- epilogue: the single write of the item's result -----------------------------------------
    const bool partial = it.slot >= 0;
    const bool half_out = !partial && (a.out_half || a.n_peers > 0);
    if constexpr (WPI == 1) {
        if (a.relu && !partial) {
#pragma unroll
            for (int n = 0; n < T::NT; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[n][i] = fmaxf(acc[n][i], 0.f);
        }
        stage_acc<FS>(acc, half_out, smem, lane);
        __syncwarp();
        store_rows<FS>(smem, half_out, it, a, fbase, lane, 32);
    } else {
        stage_acc<FS>(acc, false, smem, lane);
        __syncthreads();
        // thread sums its 4-feature pieces over the warps' tiles, in warp order, in place in warp 0's
        constexpr int PITCH = FS * 4 + 16;
        for (int c = threadIdx.x; c < 16 * (FS / 4); c += 32 * WPI) {
            const int at = c / (FS / 4) * PITCH + c % (FS / 4) * 16;
            float4 v = *(const float4*)(smem_all + at);
#pragma unroll
            for (int q = 1; q < WPI; ++q) {
                const float4 x = *(const float4*)(smem_all + q * T::SMEM + at);
                v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
            }
            if (a.relu && !partial) { v.x = fmaxf(v.x, 0.f); v.y = fmaxf(v.y, 0.f); v.z = fmaxf(v.z, 0.f); v.w = fmaxf(v.w, 0.f); }
            *(float4*)(smem_all + at) = v;
        }
        __syncthreads();
        if (half_out) {
            // repack the fp32 tile as fp16 into warp 1's part (already consumed)
            unsigned char* ht = smem_all + T::SMEM;
            for (int c = threadIdx.x; c < 16 * (FS / 4); c += 32 * WPI) {
                const int r = c / (FS / 4), q = c % (FS / 4);
                const float4 v = *(const float4*)(smem_all + r * PITCH + q * 16);
                *(__half2*)(ht + r * (FS * 2 + 16) + q * 8) = __floats2half2_rn(v.x, v.y);
                *(__half2*)(ht + r * (FS * 2 + 16) + q * 8 + 4) = __floats2half2_rn(v.z, v.w);
            }
            __syncthreads();
            store_rows<FS>(ht, true, it, a, fbase, threadIdx.x, 32 * WPI);
        } else {
            store_rows<FS>(smem_all, false, it, a, fbase, threadIdx.x, 32 * WPI);
        }
    }
}

// B with rows padded to a multiple of 16 features (32-byte sectors), for widths whose rows do not
// start on 16-byte boundaries: one pass over B against 2-byte gathers of every (window, column) pair.
// One thread writes 8 features.
__global__ void k_pad_rows(const __half* __restrict__ B, long long pieces, int F, int per_row, __half* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= pieces) return;
    const long long r = i / per_row;
    const int f = (int)(i - r * per_row) * 8;
    ((uint4*)out)[i] = load_unaligned8(B + r * F + f, F - f);
}

// Adds the partial sums of a split window in slot order and writes its 16 rows of C.
struct PeerDst {
    void* ptr[8];
    int n;
    long long row0;
};

// One thread owns 4 features of one row; the slots are read 8 at a time (independent loads) and added
// one by one.
__global__ void __launch_bounds__(128) k_reduce_heavy(const Heavy* __restrict__ heavy, const float* __restrict__ scratch,
                                                      void* C, int F, int ldS, int m_rows, int window, int out_half,
                                                      int relu, int w_begin, int w_end, PeerDst pd) {
    const Heavy h = heavy[blockIdx.x];
    wait_for_kernel_before();
    if (h.window < w_begin || h.window >= w_end) return;
    const int quads = ldS / 4;
    const int i = blockIdx.y * blockDim.x + threadIdx.x;
    const int lr = i / quads, f = (i - lr * quads) * 4;
    const long long row = (long long)h.window * window + lr;
    if (lr >= window || row >= m_rows) return;
    const float4* src = (const float4*)scratch + (size_t)h.slot_begin * 16 * quads + i;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    const int n = h.slot_end - h.slot_begin;
    for (int k = 0; k < n; k += 8) {
        float4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            v[u] = k + u < n ? __ldcs(src + (size_t)(k + u) * 16 * quads) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 8; ++u) { s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w; }
    }
    float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (f + q >= F) break;
        if (relu) r[q] = fmaxf(r[q], 0.f);
        const size_t at = (size_t)row * F + f + q;
        if (pd.n > 0) {
            for (int d = 0; d < pd.n; ++d) ((__half*)pd.ptr[d])[(size_t)pd.row0 * F + at] = __float2half_rn(r[q]);
        } else if (out_half) ((__half*)C)[at] = __float2half_rn(r[q]);
        else ((float*)C)[at] = r[q];
    }
}

}  // namespace trs

// ----------------------------------------------------------------------------------------------
// host side
// ----------------------------------------------------------------------------------------------
using namespace trs;

struct ItemSet {
    Item* items = nullptr;   // long ones first
    Heavy* heavy = nullptr;
    int n_items = 0, n_heavy = 0, n_slots = 0;
    int longest = 0;         // steps of the longest item
};

struct trs_spmm_plan {
    trs_format f;
    int m_rows, k_cols, window, num_windows;
    int device = 0;
    void* block = nullptr;   // the arrays below
    ItemSet fine, coarse;    // the coarse one only where it needs fewer slots
    Item* by_window = nullptr;   // the fine items in window order, for runs of a range of windows
    // first item, first split window and first step of every per_sample-th window
    int per_sample = 1;
    std::vector<int> item_at, heavy_at, step_at;
    int* ids = nullptr;      // [steps + kIdSpare][16] column ids of the step stream
    int* first_ids = nullptr;   // [fine items][kIdBlock][16] the first ones of the items in launch order, or null
    uint4* dense = nullptr;  // [dense steps][32] A tiles of the dense steps in fragment order
    int n_steps, sms;        // of all items; SMs of the device
};

static int env_int(const char* name, int dflt) {
    const char* v = getenv(name);
    return v ? atoi(v) : dflt;
}

// What the plan reads back while it is made.
struct PlanInfo {
    int err;                      // V_* bits
    int c_entries, cs_entries;    // last prefix entries of the CSR parts
    int totals[kWindowCounts];
    int longest;                  // steps of the longest item
    Cut coarse, made;
};

__global__ void k_plan_lasts(trs_format f, PlanInfo* info) {
    if (f.parts_c > 0) info->c_entries = f.c_row_offset[f.parts_c];
    if (f.parts_c_short > 0) info->cs_entries = f.cs_row_offset[f.parts_c_short];
}
// Where every per_sample-th window begins, so that a run of a range of windows launches little more than its own items
// (the windows in front of it and behind it up to a sample return at once); all of them would be a read-back of megabytes.
constexpr int kSamples = 1024;
struct PlanSamples {
    int item[kSamples + 1], heavy[kSamples + 1], step[kSamples + 1];
};
struct PlanBack {
    PlanInfo info;
    PlanSamples at;
};
__global__ void k_plan_totals(const int* __restrict__ off, int num_windows, int per_sample, PlanBack* back) {
    const size_t stride = (size_t)num_windows + 1;
    if (threadIdx.x < kWindowCounts) back->info.totals[threadIdx.x] = off[threadIdx.x * stride + num_windows];
    for (int i = threadIdx.x; i <= kSamples; i += blockDim.x) {
        const long long w = min((long long)i * per_sample, (long long)num_windows);
        back->at.item[i] = off[WC_ITEMS * stride + w];
        back->at.heavy[i] = off[WC_HEAVY * stride + w];
        back->at.step[i] = off[WC_STEPS * stride + w];
    }
}

static int verdict(int err) {
    if (err & V_OFFSETS) return TRS_E_OFFSETS;
    if (err & V_SHAPE) return TRS_E_SHAPE;
    if (err & V_COLUMN) return TRS_E_COLUMN;
    if (err & V_ROW) return TRS_E_ROW;
    return TRS_OK;
}

template <class T>
static int read_info(const T* dev, T* host, cudaStream_t st) {
    TRS_CUDA(cudaMemcpyAsync(host, dev, sizeof(*host), cudaMemcpyDeviceToHost, st));
    TRS_CUDA(cudaStreamSynchronize(st));
    return TRS_OK;
}

// Queues the checks of the format arrays; the ones that size their reads by prefix entries wait for the verdict
// on the prefixes.  Bits end up in info->err, which the caller reads with the plan's totals.
static int validate_on_device(const trs_format& f, int m_rows, int k_cols, int num_windows, PlanInfo* info, cudaStream_t st) {
    int* d_err = &info->err;
    auto grid = [](long long n) { return (unsigned)((n + 255) / 256); };
    if (f.parts_t > 0) {
        k_check_prefix<<<grid(f.parts_t + 1), 256, 0, st>>>(f.t_row_offset, f.parts_t + 1, f.blocks, d_err);
        k_check_prefix<<<grid(f.blocks + 1), 256, 0, st>>>(f.t_block_offset, f.blocks + 1, -1, d_err);
        k_check_range<<<grid((long long)f.blocks * 8), 256, 0, st>>>(f.t_column, (long long)f.blocks * 8, -1, k_cols, V_COLUMN, d_err);
        k_check_range<<<grid(f.parts_t), 256, 0, st>>>(f.t_window_row, f.parts_t, 0, num_windows * 16, V_ROW, d_err);
        k_check_sorted<<<grid(f.parts_t), 256, 0, st>>>(f.t_window_row, f.parts_t, d_err);
    }
    for (int pass = 0; pass < 2; ++pass) {
        const int n = pass ? f.parts_c_short : f.parts_c;
        if (n <= 0) continue;
        const int* off = pass ? f.cs_row_offset : f.c_row_offset;
        const int* row = pass ? f.cs_row : f.c_row;
        k_check_prefix<<<grid(n + 1), 256, 0, st>>>(off, n + 1, -1, d_err);
        k_check_range<<<grid(n), 256, 0, st>>>(row, n, 0, m_rows, V_ROW, d_err);
        k_check_sorted<<<grid(n), 256, 0, st>>>(row, n, d_err);
    }
    if (f.num_windows > 0) {
        k_check_prefix<<<grid(f.num_windows + 1), 256, 0, st>>>(f.s_window_tile_offset, f.num_windows + 1, f.tiles, d_err);
        if (f.tiles > 0)
            k_check_range<<<grid((long long)f.tiles * 16), 256, 0, st>>>(f.s_tile_column, (long long)f.tiles * 16, -1, k_cols, V_COLUMN, d_err);
    }
    k_plan_lasts<<<1, 1, 0, st>>>(f, info);
    PlanInfo h;
    const int rc = read_info(info, &h, st);
    if (rc) return rc;
    if (h.err & (V_OFFSETS | V_SHAPE)) return verdict(h.err);
    if (f.blocks > 0)
        k_check_tc_popcount<<<grid(f.blocks), 256, 0, st>>>((const long long*)f.t_binary, f.t_block_offset, f.blocks, d_err);
    if (h.c_entries > 0) k_check_range<<<grid(h.c_entries), 256, 0, st>>>(f.c_column, h.c_entries, 0, k_cols, V_COLUMN, d_err);
    if (h.cs_entries > 0) k_check_range<<<grid(h.cs_entries), 256, 0, st>>>(f.cs_column, h.cs_entries, 0, k_cols, V_COLUMN, d_err);
    return TRS_OK;
}

// First ids beside the items take 512 bytes an item.  Nobody is to miss that room: beyond 256 MB (8 M rows) they are left out where they
// would be more than a sixteenth of what the device has left, and no plan fails for want of them.  Asking for that takes 60 to 150
// us, so smaller ones are not asked for (plans of 9000 rows / R-MAT 20 with the question 250 / 1250 us, without 190 / 1060).
static bool room_for_first_ids(size_t bytes) {
    if (bytes <= (size_t)256 << 20) return true;
    size_t left = 0, total = 0;
    if (cudaMemGetInfo(&left, &total) != cudaSuccess) { (void)cudaGetLastError(); return false; }
    return bytes <= left / 16;
}

// CSR value-count checks need the last prefix entry; done with the column range check so that a
// short column array cannot be over-read: the caller states the lengths implicitly through the
// prefix arrays, exactly as the reference does (mGCN_online.cpp:982-1042 copies numel() items).
extern "C" int trs_spmm_plan_create(const trs_format* dev_format, int m_rows, int k_cols, int window, int validate,
                                    void* stream, trs_spmm_plan** out_plan) {
    return spmm_plan_create(dev_format, m_rows, k_cols, window, validate, true, (cudaStream_t)stream, out_plan);
}

int trs::spmm_plan_create(const trs_format* dev_format, int m_rows, int k_cols, int window, int validate, bool first_ids,
                          cudaStream_t st, trs_spmm_plan** out_plan) try {
    if (!dev_format || !out_plan) return TRS_E_ARG;
    *out_plan = nullptr;
    if (m_rows <= 0 || k_cols <= 0) return TRS_E_ARG;
    if (window <= 0 || window > 16) return TRS_E_WINDOW;
    const trs_format& f = *dev_format;
    if (f.parts_t < 0 || f.blocks < 0 || f.parts_c < 0 || f.parts_c_short < 0 || f.num_windows < 0 || f.tiles < 0)
        return TRS_E_ARG;
    if (f.blocks > 0 && window != 16) return TRS_E_WINDOW;  // TC parts address rows as window_id * 16
    if (f.parts_t > 0 && !(f.t_row_offset && f.t_block_offset && f.t_column && f.t_value && f.t_window_row && f.t_binary))
        return TRS_E_ARG;
    if (f.parts_c > 0 && !(f.c_row_offset && f.c_row && f.c_column && f.c_value)) return TRS_E_ARG;
    if (f.parts_c_short > 0 && !(f.cs_row_offset && f.cs_row && f.cs_column && f.cs_value)) return TRS_E_ARG;
    if (f.num_windows > 0 && !f.s_window_tile_offset) return TRS_E_ARG;
    if (f.tiles > 0 && !(f.s_tile_column && f.s_packed_a && f.s_packed_meta)) return TRS_E_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return TRS_E_NO_DEVICE;

    const int W = max(ceil_div(m_rows, window), f.num_windows);
    TempSpace ts;
    ts.st = st;
    const size_t stride = (size_t)W + 1;
    ts.chunk_bytes = ((size_t)6 + 2 * kWindowCounts) * stride * sizeof(int) + ((size_t)1 << 20);
    PlanBack* d_back;
    int *ranges, *cnt, *off;
    int rc = ts.get(1, &d_back);
    PlanInfo* const d_info = &d_back->info;
    if (!rc) rc = ts.get((size_t)6 * W, &ranges);
    if (!rc) rc = ts.get(kWindowCounts * stride, &cnt);
    if (!rc) rc = ts.get(kWindowCounts * stride, &off);
    if (rc) return rc;
    TRS_CUDA(cudaMemsetAsync(d_info, 0, sizeof(PlanInfo), st));
    if (validate && (rc = validate_on_device(f, m_rows, k_cols, W, d_info, st))) return rc;

    const int forced_chunk = env_int("TRS_CHUNK_STEPS", 0);
    const int chunk = forced_chunk > 0 ? max(8, forced_chunk) : 0;
    int dev = 0, sms = 0;
    TRS_CUDA(cudaGetDevice(&dev));
    TRS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // per-window ranges of TC blocks and CSR parts
    TRS_CUDA(cudaMemsetAsync(ranges, 0, sizeof(int) * (size_t)6 * W, st));
    WindowRanges wr{ranges, ranges + W, ranges + 2 * W, ranges + 3 * W, ranges + 4 * W, ranges + 5 * W};
    auto grid = [](long long n) { return (unsigned)((n + 255) / 256); };
    if (f.parts_t > 0)
        k_part_ranges<<<grid(f.parts_t), 256, 0, st>>>(f.t_window_row, f.t_row_offset, f.parts_t, 16, W,
                                                        wr.blk_begin, wr.blk_end, 1);
    if (f.parts_c > 0)
        k_part_ranges<<<grid(f.parts_c), 256, 0, st>>>(f.c_row, nullptr, f.parts_c, window, W, wr.c_begin, wr.c_end, 0);
    if (f.parts_c_short > 0)
        k_part_ranges<<<grid(f.parts_c_short), 256, 0, st>>>(f.cs_row, nullptr, f.parts_c_short, window, W,
                                                              wr.cs_begin, wr.cs_end, 0);
    // counts -> exclusive scans (kWindowCounts arrays of W + 1)
    size_t tmp_bytes = 0;
    unsigned char* tmp;
    TRS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, cnt, off, W + 1, st));
    if ((rc = ts.get(tmp_bytes + 16, &tmp))) return rc;
    auto scan = [&](int i) { return cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, cnt + i * stride, off + i * stride, W + 1, st); };
    k_count_steps<<<grid(W + 1), 256, 0, st>>>(f, wr, W, cnt);
    TRS_CUDA(scan(WC_STEPS));
    TRS_CUDA(scan(WC_DENSE));
    k_count_items<<<grid(W + 1), 256, 0, st>>>(W, chunk, sms, off + WC_STEPS * stride, cnt, &d_info->longest, &d_info->coarse);
    TRS_CUDA(scan(WC_ITEMS));
    TRS_CUDA(scan(WC_HEAVY));
    TRS_CUDA(scan(WC_SLOTS));
    const int per_sample = ceil_div(W, kSamples);
    k_plan_totals<<<1, 256, 0, st>>>(off, W, per_sample, d_back);
    PlanBack back;
    if ((rc = read_info(d_back, &back, st))) return rc;
    const PlanInfo& info = back.info;
    if ((rc = verdict(info.err))) return rc;
    const int n_items = info.totals[WC_ITEMS], n_heavy = info.totals[WC_HEAVY];
    const int n_steps = info.totals[WC_STEPS], n_dense = info.totals[WC_DENSE];
    if (n_steps < 0 || n_dense < 0 || n_items < 0) return TRS_E_OFFSETS;

    // the plan's own memory, one block
    trs_spmm_plan* p = new trs_spmm_plan();
    p->f = f;
    p->m_rows = m_rows; p->k_cols = k_cols; p->window = window; p->num_windows = W; p->device = dev;
    p->n_steps = n_steps; p->sms = sms;
    p->per_sample = per_sample;
    p->item_at.assign(back.at.item, back.at.item + kSamples + 1);
    p->heavy_at.assign(back.at.heavy, back.at.heavy + kSamples + 1);
    p->step_at.assign(back.at.step, back.at.step + kSamples + 1);
    ItemSet &fine = p->fine, &coarse = p->coarse;
    fine.n_items = n_items; fine.n_heavy = n_heavy; fine.n_slots = info.totals[WC_SLOTS]; fine.longest = info.longest;
    if (chunk == 0 && info.coarse.items > 0 && info.coarse.slots < fine.n_slots) {
        coarse.n_items = info.coarse.items; coarse.n_heavy = info.coarse.heavy; coarse.n_slots = info.coarse.slots;
        coarse.longest = info.coarse.longest;
    }
    const size_t ids_bytes = ((size_t)n_steps + kIdSpare) * 64, dense_bytes = (size_t)n_dense * 512;
    const size_t items_bytes = ((size_t)2 * n_items + coarse.n_items) * sizeof(Item);
    const size_t heavy_bytes = ((size_t)n_heavy + coarse.n_heavy) * sizeof(Heavy);
    // the kernels read the packed values 8 bytes per lane; an array that does not allow that is copied
    const size_t packed_bytes = ((uintptr_t)f.s_packed_a & 7) != 0 ? (size_t)f.tiles * 256 : 0;
    auto fail = [&](int code) { trs_spmm_plan_destroy(p); return code; };
    // the temporaries first: what the plan can do without comes last
    int* open;
    unsigned char *cls, *sort_tmp;
    size_t sort_bytes = 0;
    Item*& by_window = p->by_window;
    auto sort = [&](void* t) {
        return cub::DeviceRadixSort::SortPairs(t, sort_bytes, cls, cls + n_items, by_window, fine.items, n_items, 0, kClassBits, st);
    };
    rc = ts.get((size_t)2 * n_items, &cls);
    if (!rc) rc = ts.get((size_t)W, &open);
    if (rc) return fail(rc);
    cudaError_t e = sort(nullptr);
    if (e == cudaSuccess && (rc = ts.get(sort_bytes + 16, &sort_tmp))) return fail(rc);
    const size_t needed = ids_bytes + dense_bytes + packed_bytes + items_bytes + heavy_bytes;
    // 512 bytes an item, so not where most have next to no steps
    size_t first_bytes = first_ids && n_steps / 2 >= n_items ? (size_t)n_items * (kIdBlock * 64) : 0;
    if (!room_for_first_ids(first_bytes)) first_bytes = 0;
    rc = pool_alloc(&p->block, needed + first_bytes, st);
    if (rc == (int)cudaErrorMemoryAllocation && first_bytes > 0) {
        first_bytes = 0;
        rc = pool_alloc(&p->block, needed, st);
    }
    if (rc) return fail(rc);
    unsigned char* at = (unsigned char*)p->block;
    p->ids = (int*)at; at += ids_bytes;
    if (first_bytes) p->first_ids = (int*)at;
    at += first_bytes;
    p->dense = (uint4*)at; at += dense_bytes;
    if (packed_bytes) {
        const cudaError_t copied = cudaMemcpyAsync(at, f.s_packed_a, packed_bytes, cudaMemcpyDeviceToDevice, st);
        if (copied != cudaSuccess) return fail((int)copied);
        p->f.s_packed_a = (const uint32_t*)at; at += packed_bytes;
    }
    by_window = (Item*)at; fine.items = by_window + n_items; coarse.items = fine.items + n_items; at += items_bytes;
    fine.heavy = (Heavy*)at; coarse.heavy = fine.heavy + n_heavy;

    if (e == cudaSuccess) e = cudaMemsetAsync(open, 0x7f, sizeof(int) * (size_t)W, st);
    if (e == cudaSuccess) {
        k_fill_items<<<grid(W), 256, 0, st>>>(f, W, off, by_window, fine.heavy);
        k_fill_steps<<<grid((long long)n_items * 32), 256, 0, st>>>(f, wr, by_window, n_items, off, W, window, p->ids, p->dense, open);
        k_item_class<<<grid(n_items), 256, 0, st>>>(by_window, n_items, open, cls);
        if (coarse.n_items > 0)
            k_fill_coarse<<<grid(W), 256, 0, st>>>(f, W, off, open, &d_info->made, coarse.items, coarse.heavy);
        e = sort(sort_tmp);
    }
    if (e == cudaSuccess && p->first_ids) k_first_ids<<<grid((long long)n_items * 32), 256, 0, st>>>(fine.items, n_items, p->ids, p->first_ids);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail((int)e);
    *out_plan = p;
    return TRS_OK;
} TRS_CATCH

// No kernel of this library spins on a flag or a barrier that another kernel sets: the window kernels synchronise inside one warp
// or one CTA, and what the sums of split windows (and a product behind a copy of B) wait for is the end of the kernel launched before
// them, which waits for nothing of theirs.  So there is no wait that could give up, and the status word is always 0.  Kept
// for callers of earlier versions.
extern "C" int trs_spmm_status(const trs_spmm_plan* p, int* status) {
    if (!p || !status) return TRS_E_ARG;
    *status = 0;
    return TRS_OK;
}

extern "C" int trs_spmm_plan_destroy(trs_spmm_plan* p) {
    if (!p) return TRS_OK;
    if (p->block) {
        // kernels on any stream may still read the plan: wait as cudaFree would
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev != p->device) cudaSetDevice(p->device);
        cudaDeviceSynchronize();
        pool_free(p->block, nullptr);
        if (dev != p->device) cudaSetDevice(dev);
    }
    delete p;
    return TRS_OK;
}

// Partial sums: 16 rows per slot, rows padded to whole 16-byte pieces.
static int scratch_ld(int F) { return (F + 3) & ~3; }
static size_t set_scratch_bytes(const ItemSet& s, int F) { return (size_t)s.n_slots * 16 * (size_t)scratch_ld(F) * sizeof(float); }
static size_t items_scratch_bytes(const trs_spmm_plan* p, int F) { return set_scratch_bytes(p->fine, F); }
// The items a run with so much scratch takes: the fine ones, or the coarse ones where those need more than there is.
static const ItemSet& items_for(const trs_spmm_plan* p, int F, size_t scratch_bytes) {
    return p->coarse.n_items == 0 || items_scratch_bytes(p, F) <= scratch_bytes ? p->fine : p->coarse;
}
// Widths whose rows do not all start on 16-byte boundaries run on a copy of B with padded rows, kept in
// the workspace behind the partial sums.
static int padded_ld(int F) { return (F + 15) & ~15; }
static size_t padded_at(const ItemSet& s, int F) { return (set_scratch_bytes(s, F) + 255) & ~(size_t)255; }
// The copy takes 0.04 - 0.08 ns per row of B, 2-byte gathers 0.4 - 1 ns more per step than aligned ones, so it pays from
// a step per ten rows on (a matrix of 1 M rows with 10000 entries, F = 100: 190 us with the copy, 100 without).
static bool copy_pays(const trs_spmm_plan* p, long long steps) { return 10 * steps >= p->k_cols; }
static size_t padded_bytes(const trs_spmm_plan* p, int F) { return (size_t)p->k_cols * padded_ld(F) * sizeof(__half); }

extern "C" int trs_spmm_workspace_bytes(const trs_spmm_plan* p, int F, size_t* bytes) {
    if (!p || !bytes || F <= 0) return TRS_E_ARG;
    *bytes = F % 8 == 0 || !copy_pays(p, p->n_steps) ? items_scratch_bytes(p, F) : padded_at(p->fine, F) + padded_bytes(p, F);
    return TRS_OK;
}

extern "C" int trs_spmm_static_scratch_bytes(const trs_spmm_plan* p, int F, size_t* bytes) {
    if (!p || !bytes || F <= 0) return TRS_E_ARG;
    *bytes = set_scratch_bytes(items_for(p, F, TRS_STATIC_SCRATCH_BYTES), F);
    return TRS_OK;
}

extern "C" int trs_spmm_launches(const trs_spmm_plan* p) {
    if (!p) return 0;
    return p->fine.n_heavy > 0 ? 2 : 1;
}

template <int FS, int STAGES, int WPI, int MINB, bool ALIGNED, bool RANGE, bool RAGGED>
static int launch_instance(const KernelArgs& a, int slabs, cudaStream_t st) {
    auto kernel = k_window_spmm_warp<FS, STAGES, WPI, MINB, ALIGNED, RANGE, RAGGED>;
    constexpr int smem = WarpTile<FS, STAGES>::SMEM * WPI;
    static std::atomic<unsigned long long> done{0};
    const int rc = allow_smem(kernel, smem, true, done);
    if (rc) return rc;
    return launch_behind(kernel, dim3(a.n_items, slabs), 32 * WPI, smem, st, a.behind, a);
}

template <int FS, int STAGES, int MINB, int MINB4, bool RAGGED>
static int launch_items(const KernelArgs& a, int slabs, bool few_items, bool range, cudaStream_t st) {
    if (few_items) return range ? launch_instance<FS, STAGES, 4, MINB4, true, true, RAGGED>(a, slabs, st)
                                : launch_instance<FS, STAGES, 4, MINB4, true, false, RAGGED>(a, slabs, st);
    return range ? launch_instance<FS, STAGES, 1, MINB, true, true, RAGGED>(a, slabs, st)
                 : launch_instance<FS, STAGES, 1, MINB, true, false, RAGGED>(a, slabs, st);
}
// Rows that do not fill the slabs' 16-byte chunks leave out the chunks that are not there: two lanes that ask for one piece
// cost as much as two pieces.  Clustered graph of 262144 rows, F = 136 / 168 / 200 / 232 / 264: 234 / 256 / 302 / 316 / 376
// us with the last chunk repeated, 195 / 224 / 253 / 280 / 342 without; R-MAT 18 316 / 332 / 442 / 395 / 473 and 258 / 291 / 326 /
// 355 / 441.  The test takes up to a tenth where every chunk is there (F = 64 97 against 110).
template <int FS, int STAGES, int MINB, int MINB4>
static int launch_sized(const KernelArgs& a, int slabs, bool few_items, bool range, cudaStream_t st) {
    return a.bchunks < slabs * (FS / 8) ? launch_items<FS, STAGES, MINB, MINB4, true>(a, slabs, few_items, range, st)
                                            : launch_items<FS, STAGES, MINB, MINB4, false>(a, slabs, few_items, range, st);
}

static int launch_window_kernel(const KernelArgs& a, bool aligned, const trs_spmm_plan* p, const ItemSet& set, int width, bool range, cudaStream_t st) {
    // As few slabs as 128 features allow (64-feature slabs for F = 128: 2678 against 2120 us at R-MAT scale 21),
    // all of the same width rounded up to 16.  There is no instance of 112: its seven pieces per lane lie in rows of
    // their own, and F = 104 / 112 / 200 / 208 take 68 / 55 / 129 / 109 us there and 64 / 55 / 118 / 104 in the one of 128 without
    // the missing chunks (uniform 131072; R-MAT 18 188 / 160 / 360 / 339 and 173 / 156 / 326 / 300).  Stages and warps per
    // SM fill the shared memory; measured at R-MAT scale 20, us: F = 32 with 4 / 6 / 8 stages 215 / 220 / 223 (scale 18,
    // where the serial chain counts: 86 / 74 / 70), F = 64 with 3 / 4 / 5 stages 344 / 335 / 337 (137 / 110 / 93), F = 96
    // with 3 / 4 stages 494 / 467, F = 128 with 3 / 4 / 5 stages (16 / 12 / 10 warps) 577 / 627 / 650.  F = 80 with 18 warps
    // (96 registers, some spilled) takes 3 % more than with 16.
    const int slabs = ceil_div(a.F, 128);
    const int fs = ceil_div(ceil_div(a.F, slabs), 16);
    // by the whole plan and the whole width, so that a range of windows or a slab gets the bits it gets in a whole run
    const bool few_items = warps_per_item(set.n_items, p->n_steps, set.longest, ceil_div(width, 128), p->sms) == 4;
    if (!aligned) {
        if (few_items) return fs <= 4 ? launch_instance<64, 3, 4, 4, false, true, false>(a, ceil_div(a.F, 64), st)
                                      : launch_instance<128, 3, 4, 3, false, true, false>(a, ceil_div(a.F, 128), st);
        return fs <= 4 ? launch_instance<64, 3, 1, 16, false, true, false>(a, ceil_div(a.F, 64), st)
                       : launch_instance<128, 3, 1, 12, false, true, false>(a, ceil_div(a.F, 128), st);
    }
    switch (fs) {
        case 1: return launch_sized<16, 6, 32, 8>(a, slabs, few_items, range, st);
        case 2: return launch_sized<32, 6, 28, 7>(a, slabs, few_items, range, st);
        case 3: return launch_sized<48, 4, 26, 6>(a, slabs, few_items, range, st);
        case 4: return launch_sized<64, 4, 22, 5>(a, slabs, few_items, range, st);
        case 5: return launch_sized<80, 4, 16, 4>(a, slabs, few_items, range, st);
        case 6: return launch_sized<96, 4, 15, 4>(a, slabs, few_items, range, st);
        default: return launch_sized<128, 3, 16, 4>(a, slabs, few_items, range, st);
    }
}

extern "C" int trs_spmm_run(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, void* workspace,
                            size_t workspace_bytes, void* stream) {
    return trs_spmm_run_ex(p, B, C, F, out_dtype, 0, workspace, workspace_bytes, stream);
}

static int run_impl(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, int flags, void* workspace,
                    size_t workspace_bytes, void* stream, void* const* peers = nullptr, int n_peers = 0,
                    long long peer_row0 = 0, int w0 = 0, int w1 = -1, const SpmmHow& how = SpmmHow());

extern "C" int trs_spmm_run_ex(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, int flags,
                               void* workspace, size_t workspace_bytes, void* stream) {
    return run_impl(p, B, C, F, out_dtype, flags, workspace, workspace_bytes, stream);
}

extern "C" int trs_spmm_run_windows(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, int flags,
                                    void* workspace, size_t workspace_bytes, void* stream, int window_begin,
                                    int window_end) {
    if (window_end < 0) return TRS_E_ARG;
    return run_impl(p, B, C, F, out_dtype, flags, workspace, workspace_bytes, stream, nullptr, 0, 0, window_begin, window_end);
}

int trs::spmm_run(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, void* workspace, size_t workspace_bytes,
                  cudaStream_t st, int w0, int w1, const SpmmHow& how) {
    return run_impl(p, B, C, F, out_dtype, 0, workspace, workspace_bytes, st, nullptr, 0, 0, w0, w1, how);
}

extern "C" int trs_spmm_num_windows(const trs_spmm_plan* p) { return p ? p->num_windows : TRS_E_ARG; }

extern "C" int trs_spmm_run_bcast(const trs_spmm_plan* p, const trs_half* B, void* const* dst, int n_dst, long long row0,
                                  int F, int flags, void* workspace, size_t workspace_bytes, void* stream) {
    if (!p || !dst || n_dst < 1 || n_dst > 8 || row0 < 0) return TRS_E_ARG;
    for (int d = 0; d < n_dst; ++d)
        if (!dst[d] || ((uintptr_t)dst[d] & 15)) return TRS_E_ARG;
    if (F % 8 != 0 || ((uintptr_t)B & 15)) return TRS_E_ARG;  // the 16-byte row pieces need it
    return run_impl(p, B, dst[0], F, TRS_OUT_F16, flags, workspace, workspace_bytes, stream, dst, n_dst, row0);
}

static int run_impl(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype, int flags, void* workspace,
                    size_t workspace_bytes, void* stream, void* const* peers, int n_peers, long long peer_row0, int w0,
                    int w1, const SpmmHow& how) {
    if (!p || !B || !C || F <= 0) return TRS_E_ARG;
    if (w1 < 0) w1 = p->num_windows;
    if (w0 < 0 || w0 > w1 || w1 > p->num_windows) return TRS_E_ARG;
    if (w0 == w1) return TRS_OK;
    if (flags & ~TRS_EPILOGUE_RELU) return TRS_E_ARG;
    if (out_dtype != TRS_OUT_F32 && out_dtype != TRS_OUT_F16) return TRS_E_ARG;
    const ItemSet& set = items_for(p, F, workspace ? workspace_bytes : 0);
    const size_t need = set_scratch_bytes(set, F);
    if (need > 0 && (!workspace || workspace_bytes < need)) return TRS_E_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    KernelArgs a;
    a.behind = false;
    a.items = set.items; a.n_items = set.n_items;
    const Heavy* heavy = set.heavy;
    int n_heavy = set.n_heavy;
    const bool whole = w0 == 0 && w1 == p->num_windows;
    const int s0 = w0 / p->per_sample, s1 = ceil_div(w1, p->per_sample);
    if (!whole && &set == &p->fine) {
        heavy += p->heavy_at[s0]; n_heavy = p->heavy_at[s1] - p->heavy_at[s0];
        // a third of a matrix with hub windows still gains more from long items first than it loses by the items of others
        // (halves of R-MAT 20, F = 128: 378 us, in window order 490; eighths 230 either way)
        const int n = p->item_at[s1] - p->item_at[s0];
        if (set.n_heavy == 0 || n < set.n_items / 3) { a.items = p->by_window + p->item_at[s0]; a.n_items = n; }
    }
    a.w_begin = w0; a.w_end = w1;
    a.ids = p->ids; a.dense = p->dense;
    a.first_ids = a.items == p->fine.items ? p->first_ids : nullptr;
    a.packed_a = p->f.s_packed_a; a.packed_meta = p->f.s_packed_meta;
    a.B = (const __half*)B; a.C = C; a.scratch = (float*)workspace;
    a.ldb = F; a.ldS = scratch_ld(F); a.F = F; a.bchunks = ceil_div(F, 8);
    a.m_rows = p->m_rows; a.window = p->window; a.out_half = out_dtype == TRS_OUT_F16;
    a.vec_out = ((uintptr_t)C & 15) == 0 && F % (a.out_half ? 8 : 4) == 0;
    a.relu = (flags & TRS_EPILOGUE_RELU) ? 1 : 0;
    a.n_peers = n_peers; a.peer_row0 = peer_row0;
    for (int d = 0; d < 8; ++d) a.peers[d] = d < n_peers ? peers[d] : nullptr;
    // The kernel gathers B in 16-byte pieces.  Rows that do not start on 16-byte boundaries are copied to
    // padded ones first when that pays and the workspace has room (trs_spmm_workspace_bytes asks for it).
    bool aligned = F % 8 == 0 && ((uintptr_t)B & 15) == 0;
    if (((uintptr_t)workspace & 15) && need > 0) return TRS_E_WORKSPACE;
    const bool pays = copy_pays(p, how.rows == SpmmHow::FOR_THIS_RUN && !whole ? p->step_at[s1] - p->step_at[s0] : p->n_steps);
    if (!aligned && pays && n_peers == 0 && workspace && workspace_bytes >= padded_at(set, F) + padded_bytes(p, F) &&
        ((uintptr_t)workspace & 15) == 0) {
        __half* Bp = (__half*)((unsigned char*)workspace + padded_at(set, F));
        a.ldb = padded_ld(F);
        a.bchunks = a.ldb / 8;
        const long long pieces = (long long)p->k_cols * a.bchunks;
        if (how.rows != SpmmHow::COPIED) {
            // The product's CTAs may arrive while this ends, which saves two to four microseconds (8000 uniform rows, F = 47: 12.3 -> 10.3
            // us; R-MAT 17, lossless 66 -> 61 with the sums below).  An SM divides its memory anew only when it is empty: with little
            // shared memory for this kernel, few of the others would fit beside it and behind it (R-MAT 17: 84 us).  A run of a
            // range may have no item that waits, so it is launched when this has ended.
            a.behind = whole;
            static std::atomic<unsigned long long> done{0};
            const int rc = allow_smem(k_pad_rows, 0, true, done);
            if (rc) return rc;
            k_pad_rows<<<(unsigned)ceil_div64(pieces, 256), 256, 0, st>>>(a.B, pieces, F, a.bchunks, Bp);
            TRS_LAUNCH_CHECK();
        }
        a.B = Bp;
        aligned = true;
    }
    if (!aligned && n_peers > 0) return TRS_E_ARG;
    const int rc = launch_window_kernel(a, aligned, p, set, how.width > 0 ? how.width : F, !whole, st);
    if (rc) return rc;
    if (n_heavy > 0) {
        PeerDst pd;
        pd.n = a.n_peers; pd.row0 = a.peer_row0;
        for (int d = 0; d < 8; ++d) pd.ptr[d] = a.peers[d];
        const dim3 rgrid(n_heavy, ceil_div(16 * a.ldS / 4, 128));
        return launch_behind(k_reduce_heavy, rgrid, 128, 0, st, true, heavy, (const float*)workspace, C, F, a.ldS, p->m_rows, p->window,
                             a.out_half, a.relu, w0, w1, pd);
    }
    return TRS_OK;
}

// ----------------------------------------------------------------------------------------------
// SpMM without any allocation: partial sums in a fixed, library-owned device array
// ----------------------------------------------------------------------------------------------
// Some hosts cannot give this library scratch memory at call time: applications that hand the
// whole device memory to their own pool at start-up (a later cudaMalloc from a plug-in fails or
// fragments that pool) and latency-critical loops in which cudaMalloc / cudaFree would stall
// every stream of the device.  For them trs_spmm_run_static runs the ordinary kernels
// (k_window_spmm_warp + k_reduce_heavy), whose scratch need is small and known from the plan, with the partial sums of split windows kept in the array below instead of a
// caller-provided workspace.  Every GPU that loads the library holds these bytes until exit.
//
// In host code the array's name is only a stand-in for the symbol; the device address is asked
// for once per device (cudaGetSymbolAddress with that device current) and cached.
static __device__ __align__(256) unsigned char g_static_scratch[TRS_STATIC_SCRATCH_BYTES];

namespace {
constexpr int kMaxDevices = 64;
void* g_static_scratch_ptr[kMaxDevices] = {};
bool g_static_scratch_ready[kMaxDevices] = {};
std::mutex g_static_scratch_mutex;
}  // namespace

extern "C" int trs_spmm_run_static(const trs_spmm_plan* p, const trs_half* B, void* C, int F, int out_dtype,
                                   void* stream) {
    if (!p || !B || !C || F <= 0) return TRS_E_ARG;
    if (set_scratch_bytes(items_for(p, F, TRS_STATIC_SCRATCH_BYTES), F) > (size_t)TRS_STATIC_SCRATCH_BYTES) return TRS_E_LIMIT;
    int dev = -1;
    TRS_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return TRS_E_LIMIT;
    void* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
        if (!g_static_scratch_ready[dev]) {  // first call on this device: look the symbol up
            void* ptr = nullptr;
            TRS_CUDA(cudaGetSymbolAddress(&ptr, g_static_scratch));
            g_static_scratch_ptr[dev] = ptr;
            g_static_scratch_ready[dev] = true;
        }
        scratch = g_static_scratch_ptr[dev];
    }
    // Nothing in the array has to start at zero: every slot a call reads is first written in
    // full by that call's window kernel.
    return run_impl(p, B, C, F, out_dtype, 0, scratch, (size_t)TRS_STATIC_SCRATCH_BYTES, stream);
}
