// vdf_segreduce.cu -- sort-based group-by: segment boundaries + segmented
// count / sum / min / max / mean over rows already in key order.
//
// The reference group-by is hash based (transform_group_by_onecol_mt.hpp:
// 182-337 with AddLookupOneCol / OccLookupOneCol, onecol_functions.inl:4-86:
// one ankerl map probe per row, per-thread maps merged serially,
// merge_functions.inl:3-36; output via CreateValueCol, create_value_col.inl:
// 36-61).  On the GPU the rows are first sorted, so each group is a contiguous
// segment and the whole aggregation is one streaming pass ("reduce by key"):
//
//   * a row is a segment head when any key differs from the previous row;
//   * each thread folds its ITEMS rows into an aggregate
//       (heads, open-segment partial {count, per column sum/min/max}),
//     combined with the associative reduce-by-key operator
//       A (+) B = (A.heads + B.heads, B.heads ? B.partial : A.partial (+) B.partial);
//   * k_seg_tiles reduces every tile of rows to one aggregate (all tiles in
//     parallel, no waiting on other tiles);
//   * k_seg_scan (one CTA) turns the tile aggregates into exclusive tile
//     prefixes: the number of groups before each tile and the partial of the
//     segment that runs into it;
//   * k_seg_emit re-reads the rows, lists the segments that start in a CTA's
//     tiles, and folds and writes each (keys, count, sum, min, max, mean) by
//     one thread, eight lanes or a warp, depending on its length; rows
//     without a segment head (known from the prefixes) are skipped.
// Nothing spins on another CTA, so there is no look-back latency chain: the
// price is one extra sequential read of the key and value columns (of the
// tiles that hold a head).
//
// Exactness: integer sums are 128-bit (lo, hi words); float sums are carried
// as (sum, compensation) with an error-free TwoSum at every combine, so a
// group's f64 sum is accurate to about one rounding of the exact value,
// independent of how the rows were split over threads and tiles.
//
// All columns are read in sorted row order (the fused sort + group-by call
// gathers them first with the high-occupancy gather kernel: a random read
// costs a full DRAM access of 64 bytes, so each gathered value is read
// randomly exactly once and everything here is sequential).
#include <algorithm>

#include "vdf_agg.cuh"
#include "vdf_common.cuh"
#include "vdf_internal.h"

namespace vdf {

namespace {

// Raw bits of a key / emitted element (zero-extended).
__device__ __forceinline__ uint64_t load_raw(const void* src, int w, uint64_t i) {
    return w == 4 ? (uint64_t)__ldg(static_cast<const uint32_t*>(src) + i)
                  : (uint64_t)__ldg(static_cast<const unsigned long long*>(src) + i);
}
// Rows row0 .. row0+ITEMS-1 of a column into arr[j][c] (raw bits, zero-
// extended), with 16-byte vector loads when the rows are in bounds and
// aligned (row0 is a multiple of ITEMS; tile starts are multiples of it).
template <int ITEMS, int W>
__device__ __forceinline__ void load_rows(const void* src, int w, uint64_t row0, uint64_t n, uint64_t (&arr)[ITEMS][W],
                                          int c) {
    const bool full = row0 + ITEMS <= n;
    if (w == 8) {
        const unsigned long long* p = static_cast<const unsigned long long*>(src) + row0;
        if (full && ITEMS % 2 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < ITEMS; j += 2) {
                const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(p + j));
                arr[j][c] = v.x;
                arr[j + 1][c] = v.y;
            }
            return;
        }
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) arr[j][c] = row0 + j < n ? __ldg(p + j) : 0ull;
    } else {
        const uint32_t* p = static_cast<const uint32_t*>(src) + row0;
        if (full && ITEMS % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < ITEMS; j += 4) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(p + j));
                arr[j][c] = v.x;
                arr[j + 1][c] = v.y;
                arr[j + 2][c] = v.z;
                arr[j + 3][c] = v.w;
            }
            return;
        }
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) arr[j][c] = row0 + j < n ? (uint64_t)__ldg(p + j) : 0ull;
    }
}

// Canonical images (see load_val) of rows row0 .. row0+ITEMS-1.
template <int ITEMS, int W>
__device__ __forceinline__ void load_vals(const void* src, int dt, uint64_t row0, uint64_t n, uint64_t (&arr)[ITEMS][W],
                                          int c) {
    load_rows<ITEMS>(src, dtype_width(dt), row0, n, arr, c);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint64_t x = arr[j][c];
        if (dt == I32) arr[j][c] = (uint64_t)(int64_t)(int32_t)(uint32_t)x;
        else if (dt == F32) arr[j][c] = as_b((double)__uint_as_float((uint32_t)x));
    }
}

template <int NV>
struct Agg {
    uint32_t heads;  // segment heads in the covered rows
    uint32_t cnt;    // rows of the open (last) segment inside the covered rows
    uint64_t w[NV > 0 ? NV : 1][4];
};

template <int NV>
__device__ __forceinline__ Agg<NV> agg_identity() {
    Agg<NV> r;
    r.heads = 0;
    r.cnt = 0;
#pragma unroll
    for (int v = 0; v < (NV > 0 ? NV : 1); ++v)
#pragma unroll
        for (int q = 0; q < 4; ++q) r.w[v][q] = 0;
    return r;
}

// A is earlier in row order than B.
template <int NV>
__device__ __forceinline__ Agg<NV> agg_combine(const Agg<NV>& A, const Agg<NV>& B, const int* vc) {
    Agg<NV> r;
    r.heads = A.heads + B.heads;
    if (B.heads > 0 || A.cnt == 0) {
        r.cnt = B.cnt;
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
            for (int q = 0; q < 4; ++q) r.w[v][q] = B.w[v][q];
    } else if (B.cnt == 0) {
        r.cnt = A.cnt;
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
            for (int q = 0; q < 4; ++q) r.w[v][q] = A.w[v][q];
    } else {
        r.cnt = A.cnt + B.cnt;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
#pragma unroll
            for (int q = 0; q < 4; ++q) r.w[v][q] = A.w[v][q];
            col_merge(r.w[v], B.w[v], vc[v]);
        }
    }
    if (NV == 0) r.w[0][0] = 0;
    return r;
}

template <int NV>
__device__ __forceinline__ Agg<NV> agg_shfl_up(const Agg<NV>& a, int d) {
    Agg<NV> r;
    r.heads = __shfl_up_sync(0xffffffffu, a.heads, d);
    r.cnt = __shfl_up_sync(0xffffffffu, a.cnt, d);
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int q = 0; q < 4; ++q) r.w[v][q] = __shfl_up_sync(0xffffffffu, a.w[v][q], d);
    return r;
}
template <int NV>
__device__ __forceinline__ Agg<NV> agg_shfl_down(const Agg<NV>& a, int d) {
    Agg<NV> r;
    r.heads = __shfl_down_sync(0xffffffffu, a.heads, d);
    r.cnt = __shfl_down_sync(0xffffffffu, a.cnt, d);
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
        for (int q = 0; q < 4; ++q) r.w[v][q] = __shfl_down_sync(0xffffffffu, a.w[v][q], d);
    return r;
}
constexpr int kSegThreads = 256;
constexpr int kSegTile = 512;  // rows per tile

// Value-class patterns fixed at compile time (VCP): 0 = read from the column
// dtypes at run time; 1 = two columns, float then signed integer (the
// aggregation every workload here runs).  With the pattern fixed, the
// per-row merges carry no branches on the class.
template <int NV, int VCP>
__device__ __forceinline__ void fix_classes(int* vc) {
    if constexpr (VCP == 1 && NV == 2) {
        vc[0] = VC_FLOAT;
        vc[1] = VC_SINT;
    }
}
// Key-width patterns fixed at compile time (KWP): 0 = run time; otherwise
// key k is (KWP >> 4k) & 15 bytes wide (two keys: 0x48 = 8 then 4 bytes).
template <int NK, int KWP>
__device__ __forceinline__ void fix_widths(int* kw) {
    if constexpr (KWP != 0) {
#pragma unroll
        for (int k = 0; k < NK; ++k) kw[k] = (KWP >> (4 * k)) & 15;
    }
}
inline int key_width_pattern(const SegArgs& a) {
    int p = 0;
    for (int k = 0; k < a.nkeys; ++k) p |= (dtype_width(a.key[k].dtype) & 15) << (4 * k);
    return p;
}
inline int value_class_pattern(const SegArgs& a) {
    auto cls = [](int dt) { return (dt == F64 || dt == F32) ? 0 : (dt == I32 || dt == I64) ? 1 : 2; };
    return (a.nvals == 2 && cls(a.val[0].dtype) == 0 && cls(a.val[1].dtype) == 1) ? 1 : 0;
}

template <int NK, int NV>
__device__ __forceinline__ void seg_setup(const SegArgs& a, int* vc, int* kw) {
#pragma unroll
    for (int v = 0; v < NV; ++v) vc[v] = vclass(a.val[v].dtype);
#pragma unroll
    for (int k = 0; k < NK; ++k) kw[k] = dtype_width(a.key[k].dtype);
}

// ---- phase 1: one aggregate per tile ----------------------------------------
// A tile's aggregate is its head count plus the aggregate of its trailing
// open segment (the rows from its last head, or all its rows if it has none).
// So the keys are read to find the heads and the last head, and only the
// threads whose rows lie in the trailing segment read values and fold them;
// only warps overlapping it reduce.  With many groups (one per few rows)
// almost no values are read here.
// Eight rows per thread: one CTA covers kSubTiles consecutive 512-row tiles
// (two warps each).
constexpr int kWideItems = 8;
constexpr int kSubTiles = kSegThreads * kWideItems / kSegTile;  // 4
constexpr int kWarpsPerSub = kSegThreads / 32 / kSubTiles;      // 2

template <int NK, int NV, int VCP = 0, int KWP = 0>
__global__ void __launch_bounds__(kSegThreads) k_seg_tiles_wide(SegArgs a, Agg<NV>* tile_agg, uint32_t tiles,
                                                                uint32_t* done) {
    wait_for_launch_before();
    if (blockIdx.x == 0 && threadIdx.x == 0) *done = 0;  // for k_seg_scan
    constexpr int ITEMS = kWideItems, WARPS = kSegThreads / 32;
    __shared__ Agg<NV> s_warp[WARPS];
    __shared__ uint32_t s_heads[WARPS];
    __shared__ int s_last[WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = warp / kWarpsPerSub;                    // sub-tile of this warp
    const uint32_t tile = blockIdx.x * kSubTiles + sub;     // global tile index
    const int sub_tid = tid - sub * kWarpsPerSub * 32;      // thread within the sub-tile
    const uint64_t n = a.n;
    const uint64_t row0 = (uint64_t)tile * kSegTile + (uint64_t)sub_tid * ITEMS;
    int vc[NV > 0 ? NV : 1], kw[NK];
    seg_setup<NK, NV>(a, vc, kw);
    fix_classes<NV, VCP>(vc);
    fix_widths<NK, KWP>(kw);

    uint64_t key[ITEMS][NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) load_rows<ITEMS>(a.key[k].src, kw[k], row0, n, key, k);
    uint64_t prev[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k) prev[k] = __shfl_up_sync(0xffffffffu, key[ITEMS - 1][k], 1);
    if (lane == 0 && row0 > 0 && row0 < n) {
#pragma unroll
        for (int k = 0; k < NK; ++k) prev[k] = load_raw(a.key[k].src, kw[k], row0 - 1);
    }
    uint32_t hmask = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint64_t r = row0 + j;
        bool h = (r == 0);
#pragma unroll
        for (int k = 0; k < NK; ++k) h |= (j == 0 ? prev[k] : key[j - 1][k]) != key[j][k];
        if (r < n && h) hmask |= 1u << j;
    }
    uint32_t heads = __popc(hmask);
    int last = hmask ? sub_tid * ITEMS + (31 - __clz(hmask)) : -1;
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        heads += __shfl_down_sync(0xffffffffu, heads, d);
        last = max(last, __shfl_down_sync(0xffffffffu, last, d));
    }
    if (lane == 0) {
        s_heads[warp] = heads;
        s_last[warp] = last;
    }
    __syncthreads();
    uint32_t tile_heads = 0;
    int tile_last = -1;
#pragma unroll
    for (int w = 0; w < kWarpsPerSub; ++w) {
        tile_heads += s_heads[sub * kWarpsPerSub + w];
        tile_last = max(tile_last, s_last[sub * kWarpsPerSub + w]);
    }
    const int from = tile_last >= 0 ? tile_last : 0;

    Agg<NV> t = agg_identity<NV>();
    if (sub_tid * ITEMS + ITEMS - 1 >= from && row0 < n) {
        uint64_t val[ITEMS][NV > 0 ? NV : 1];
#pragma unroll
        for (int v = 0; v < NV; ++v) load_vals<ITEMS>(a.val[v].src, a.val[v].dtype, row0, n, val, v);
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (row0 + j >= n || sub_tid * ITEMS + j < from) continue;
            if (t.cnt == 0) {
#pragma unroll
                for (int v = 0; v < NV; ++v) col_init(t.w[v], val[j][v], vc[v]);
            } else {
#pragma unroll
                for (int v = 0; v < NV; ++v) {
                    uint64_t one[4];
                    col_init(one, val[j][v], vc[v]);
                    col_merge(t.w[v], one, vc[v]);
                }
            }
            t.cnt++;
        }
    }
    const int wsub = warp - sub * kWarpsPerSub;  // warp within the sub-tile
    const bool active = (wsub + 1) * 32 * ITEMS - 1 >= from;
    if (active) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const Agg<NV> o = agg_shfl_down(t, d);
            if (lane + d < 32) t = agg_combine(t, o, vc);
        }
        if (lane == 0) s_warp[warp] = t;
    }
    __syncthreads();
    if (sub_tid == 0 && tile < tiles) {
        Agg<NV> r = agg_identity<NV>();
        for (int w = 0; w < kWarpsPerSub; ++w)
            if ((w + 1) * 32 * ITEMS - 1 >= from) r = agg_combine(r, s_warp[sub * kWarpsPerSub + w], vc);
        r.heads = tile_heads;
        tile_agg[tile] = r;
    }
}

// ---- phase 2: exclusive prefixes of the tile aggregates ----------------------
// Each CTA scans kScanTiles consecutive tile aggregates in place (exclusive,
// within the CTA) and writes the CTA total; the CTA that finishes last (a
// counter the tile pass clears) turns the totals into exclusive prefixes.  The
// emit pass combines the two levels.  Latency bound: as a launch of its own
// the second level cost 3 us and a launch gap per group-by, whatever the size.
constexpr int kScanTiles = 256;

template <int NV>
__device__ __forceinline__ Agg<NV> block_exclusive_scan(Agg<NV> x, Agg<NV>* s_warp, const int* vc, Agg<NV>& total) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    Agg<NV> incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Agg<NV> o = agg_shfl_up(incl, d);
        if (lane >= d) incl = agg_combine(o, incl, vc);
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    Agg<NV> pre = agg_identity<NV>();
    for (int w = 0; w < warp; ++w) pre = agg_combine(pre, s_warp[w], vc);
    Agg<NV> lx = agg_shfl_up(incl, 1);
    if (lane == 0) lx = agg_identity<NV>();
    total = agg_identity<NV>();
    for (int w = 0; w < (int)(blockDim.x / 32); ++w) total = agg_combine(total, s_warp[w], vc);
    return agg_combine(pre, lx, vc);
}

template <int NV>
__global__ void __launch_bounds__(kScanTiles) k_seg_scan(const SegArgs a, Agg<NV>* tile_agg, Agg<NV>* block_tot,
                                                         uint32_t tiles, uint32_t* done) {
    __shared__ Agg<NV> s_warp[kScanTiles / 32];
    __shared__ bool s_last;
    wait_for_launch_before();
    int vc[NV > 0 ? NV : 1];
#pragma unroll
    for (int v = 0; v < NV; ++v) vc[v] = vclass(a.val[v].dtype);
    const uint32_t t = blockIdx.x * kScanTiles + threadIdx.x, blocks = gridDim.x;
    const Agg<NV> x = t < tiles ? tile_agg[t] : agg_identity<NV>();
    Agg<NV> total;
    const Agg<NV> ex = block_exclusive_scan(x, s_warp, vc, total);
    if (t < tiles) tile_agg[t] = ex;
    if (blocks == 1) {
        if (threadIdx.x == 0) block_tot[0] = agg_identity<NV>();
        return;
    }
    if (threadIdx.x == 0) {
        block_tot[blockIdx.x] = total;
        __threadfence();
        s_last = atomicAdd(done, 1u) == blocks - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t per = (blocks + kScanTiles - 1) / kScanTiles;
    const uint32_t b0 = min(blocks, threadIdx.x * per), b1 = min(blocks, b0 + per);
    Agg<NV> acc = agg_identity<NV>();
    for (uint32_t b = b0; b < b1; ++b) acc = agg_combine(acc, block_tot[b], vc);
    Agg<NV> run = block_exclusive_scan(acc, s_warp, vc, total);
    for (uint32_t b = b0; b < b1; ++b) {
        const Agg<NV> cur = block_tot[b];
        block_tot[b] = run;
        run = agg_combine(run, cur, vc);
    }
}

// ---- phase 3: emit the groups of each CTA's rows ------------------------------
// Heads before tile t are the exclusive prefix of the tile pass's head counts,
// so a CTA knows the heads in its rows before it reads them (all but the last
// CTA: the prefix past the last tile is not stored).
//   * None: it writes nothing unless rows' groups are wanted (row_group) and
//     returns -- a CTA writes the group that ends before each head in its
//     rows, with the new group's key and first row; a group running through
//     head-less rows is written where the next head is.  With few groups over
//     many rows nearly every CTA returns, and its rows are not read a second
//     time.
//   * As many as rows (most keys distinct): row r is group H + r, written
//     straight from its loads.
// The CTA holding the last row writes the last group and the group count.

// The aggregate of some rows of one group: lanes or threads build it row by
// row, a warp merges its lanes'.
template <int NV>
struct Fold {
    uint32_t cnt = 0;
    uint64_t w[NV > 0 ? NV : 1][4];
    __device__ __forceinline__ void row(const uint64_t* vals, uint32_t stride, const int* vc) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const uint64_t x = vals[v * stride];
            if (cnt == 0) {
                col_init(w[v], x, vc[v]);
            } else {
                uint64_t one[4];
                col_init(one, x, vc[v]);
                col_merge(w[v], one, vc[v]);
            }
        }
        ++cnt;
    }
    __device__ __forceinline__ void merge(const Fold& o, const int* vc) {
        if (o.cnt == 0) return;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            if (cnt == 0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) w[v][q] = o.w[v][q];
            } else {
                col_merge(w[v], o.w[v], vc[v]);
            }
        }
        cnt += o.cnt;
    }
    // afterwards each of `lanes` (a power of two) neighbouring lanes holds the sum of theirs
    __device__ __forceinline__ void team(int lanes, const int* vc) {
#pragma unroll 1
        for (int d = 1; d < lanes; d <<= 1) {
            Fold o;
            o.cnt = __shfl_xor_sync(0xffffffffu, cnt, d);
#pragma unroll
            for (int v = 0; v < NV; ++v)
#pragma unroll
                for (int q = 0; q < 4; ++q) o.w[v][q] = __shfl_xor_sync(0xffffffffu, w[v][q], d);
            merge(o, vc);
        }
    }
};

constexpr int kEmitRows = kSubTiles * kSegTile;        // rows of a CTA
constexpr int kEmitPer = kEmitRows / kSegThreads;      // rows per thread
constexpr int kEmitWords = kEmitRows / 32;             // head-mask words
constexpr uint32_t kThreadRows = 32, kTeamRows = 256;  // longest group one thread and eight lanes fold
static_assert(kEmitWords == 64 && kEmitRows <= 65536, "two words per lane of a warp; rows in 16 bits");

extern __shared__ __align__(16) unsigned char seg_smem[];
template <int NV>
constexpr size_t emit_smem_bytes() { return (size_t)NV * kEmitRows * 8; }

// A CTA takes four tiles: its rows' values go into shared memory, the heads
// become a list of group starts, and then one thread folds and writes each
// group of up to kThreadRows rows -- consecutive threads consecutive groups,
// so every output column is written by full warps -- eight lanes each longer
// group, and one warp each group past kTeamRows and the one running in from
// earlier rows (whose part before the CTA is the tile prefix).  Where nearly every row starts a group (from
// striped_min_heads of 512 rows) the threads go by rows instead of by groups.
//
// What bounds it: instructions.  A thread per eight rows that scanned
// aggregates of 18 words across the warp and wrote each group where its rows
// ended (a quarter of the lanes storing at a time) took 341 instructions per
// row of a batch of short groups.  Per launch on one B200, that kernel ->
// this one: 200M rows of 50M keys 4.76 -> 2.42 ms, 9M rows in groups of two
// 0.32 -> 0.25 ms, 100M one-row groups of two keys 2.09 -> 1.80 ms (12.2 GB:
// HBM-bound), a batch of 4,096 queries 1.26 -> 1.07 ms, 1M rows in groups of
// 100 22.9 -> 15.1 us.
template <int NK, int NV, int VCP = 0, int KWP = 0>
__global__ void __launch_bounds__(kSegThreads, (NV >= 3 ? 2 : 4))
    k_seg_emit(SegArgs a, const Agg<NV>* tile_prefix, const Agg<NV>* block_prefix, uint32_t tiles) {
    constexpr int R = kEmitPer, B = 4;  // rows per thread, loaded B at a time
    uint64_t* vals = reinterpret_cast<uint64_t*>(seg_smem);  // [NV][kEmitRows]
    __shared__ uint32_t s_word[kEmitWords], s_pre[kEmitWords + 1];
    __shared__ uint16_t s_pos[kEmitRows + 1];  // first row of each group that starts here
    __shared__ uint16_t s_long[kEmitRows / (kThreadRows + 1) + 1];  // the longer groups
    __shared__ uint32_t s_nlong;
    const uint32_t t0 = blockIdx.x * kSubTiles, t1 = t0 + kSubTiles;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t n = a.n, base = (uint64_t)t0 * kSegTile;
    const uint32_t rows = (uint32_t)min((uint64_t)kEmitRows, n - base);
    const bool table_end = base + rows == n;
    int vc[NV > 0 ? NV : 1], kw[NK];
    seg_setup<NK, NV>(a, vc, kw);
    fix_classes<NV, VCP>(vc);
    fix_widths<NK, KWP>(kw);
    wait_for_launch_before();
    // groups that start before the CTA's rows, and in them where that is known
    const uint32_t H = block_prefix[t0 / kScanTiles].heads + tile_prefix[t0].heads;
    const uint32_t known = t1 < tiles ? block_prefix[t1 / kScanTiles].heads + tile_prefix[t1].heads - H : ~0u;
    if (known == 0 && !a.row_group) return;  // the same for the whole CTA
    // the group running in from earlier rows ends at the CTA's row e, the first
    // head: one warp adds the rows from e's own tile on to that tile's prefix
    auto carried = [&](uint32_t e) {
        const uint32_t sub = (e ? e - 1 : 0u) / kSegTile;
        Fold<NV> f;
#pragma unroll 1
        for (uint32_t r = sub * kSegTile + lane; r < e; r += 32) f.row(vals + r, kEmitRows, vc);
        if (e) f.team(32, vc);
        if (lane == 0) {
            const Agg<NV> P = agg_combine(block_prefix[(t0 + sub) / kScanTiles], tile_prefix[t0 + sub], vc);
            Fold<NV> c;
            c.cnt = P.cnt;
#pragma unroll
            for (int v = 0; v < NV; ++v)
#pragma unroll
                for (int q = 0; q < 4; ++q) c.w[v][q] = P.w[v][q];
            c.merge(f, vc);
            emit_group<NV>(a, H - 1, c.cnt, c.w, vc);
        }
    };
    if (known == (uint32_t)kEmitRows) {
        if (warp == 0 && H > 0) carried(0);
#pragma unroll
        for (int j0 = 0; j0 < R; j0 += B) {
            // every load of the batch before its first store (outputs may not
            // be assumed apart from inputs, so the compiler would not reorder them)
            uint64_t key[B][NK], x[B][NV > 0 ? NV : 1];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const uint64_t r = base + (uint32_t)(j0 + j) * kSegThreads + tid;
#pragma unroll
                for (int k = 0; k < NK; ++k) key[j][k] = load_raw(a.key[k].src, kw[k], r);
#pragma unroll
                for (int v = 0; v < NV; ++v) x[j][v] = load_val(a.val[v].src, a.val[v].dtype, r);
            }
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const uint32_t o = (uint32_t)(j0 + j) * kSegThreads + tid, g = H + o;
#pragma unroll
                for (int k = 0; k < NK; ++k)
                    if (a.key_out[k]) store_raw(a.key_out[k], kw[k], g, key[j][k]);
                if (a.group_start) a.group_start[g] = (uint32_t)(base + o);
                if (a.row_group) a.row_group[base + o] = g;
                if (o + 1 == (uint32_t)kEmitRows) break;  // may go on: left to the next CTA (never the table's last row)
                uint64_t w[NV > 0 ? NV : 1][4];
#pragma unroll
                for (int v = 0; v < NV; ++v) col_init(w[v], x[j][v], vc[v]);
                emit_group<NV>(a, g, 1, w, vc);
            }
        }
        return;
    }

    if (tid == 0) s_nlong = 0;
    uint32_t mine = 0;  // bit j: row j * kSegThreads + tid starts a group
#pragma unroll
    for (int j0 = 0; j0 < R; j0 += B) {
        uint64_t key[B][NK], before[B][NK], x[B][NV > 0 ? NV : 1];
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const uint32_t r = (uint32_t)(j0 + j) * kSegThreads + tid;
            const bool ok = r < rows;
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                key[j][k] = ok ? load_raw(a.key[k].src, kw[k], base + r) : 0ull;
                before[j][k] = ok && lane == 0 && base + r > 0 ? load_raw(a.key[k].src, kw[k], base + r - 1) : 0ull;
            }
#pragma unroll
            for (int v = 0; v < NV; ++v) x[j][v] = ok ? load_val(a.val[v].src, a.val[v].dtype, base + r) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < B; ++j) {
            const uint32_t r = (uint32_t)(j0 + j) * kSegThreads + tid;
            bool h = base + r == 0;
#pragma unroll
            for (int k = 0; k < NK; ++k) {
                const uint64_t up = __shfl_up_sync(0xffffffffu, key[j][k], 1);
                h |= (lane ? up : before[j][k]) != key[j][k];
            }
            h = h && r < rows;
            const uint32_t word = __ballot_sync(0xffffffffu, h);
            if (lane == 0) s_word[(j0 + j) * (kSegThreads / 32) + warp] = word;
            mine |= h ? 1u << (j0 + j) : 0u;
#pragma unroll
            for (int v = 0; v < NV; ++v) vals[v * kEmitRows + r] = x[j][v];
        }
    }
    __syncthreads();
    if (warp == 0) {  // heads before each word
        const uint32_t c0 = __popc(s_word[2 * lane]), c1 = __popc(s_word[2 * lane + 1]);
        uint32_t incl = c0 + c1;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += t;
        }
        s_pre[2 * lane] = incl - c0 - c1;
        s_pre[2 * lane + 1] = incl - c1;
        if (lane == 31) s_pre[kEmitWords] = incl;
    }
    __syncthreads();
    const uint32_t heads = s_pre[kEmitWords];
    const uint32_t lt = lanemask_lt();
    auto index_of = [&](int j) -> uint32_t {  // groups that start here before row j * kSegThreads + tid
        const int w = j * (kSegThreads / 32) + warp;
        return s_pre[w] + __popc(s_word[w] & lt);
    };
    if (a.row_group) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint32_t r = (uint32_t)j * kSegThreads + tid;
            if (r < rows) a.row_group[base + r] = H + index_of(j) + ((mine >> j) & 1u) - 1u;
        }
    }
    if (table_end && tid == 0 && a.n_groups) *a.n_groups = H + heads;
#pragma unroll
    for (int j = 0; j < R; ++j)
        if ((mine >> j) & 1u) s_pos[index_of(j)] = (uint16_t)(j * kSegThreads + tid);
    if (tid == 0) s_pos[heads] = (uint16_t)rows;
    __syncthreads();
    // the last group that starts here is complete only at the table's end
    const uint32_t whole = table_end ? heads : (heads ? heads - 1 : 0);
    auto group = [&](uint32_t k) {
        const uint32_t b = s_pos[k], e = s_pos[k + 1];
#pragma unroll
        for (int q = 0; q < NK; ++q)
            if (a.key_out[q]) store_raw(a.key_out[q], kw[q], H + k, load_raw(a.key[q].src, kw[q], base + b));
        if (a.group_start) a.group_start[H + k] = (uint32_t)(base + b);
        if (k >= whole) return;
        if (e - b > kThreadRows) {  // left to a team below
            s_long[atomicAdd(&s_nlong, 1u)] = (uint16_t)k;
            return;
        }
        Fold<NV> f;
#pragma unroll 1
        for (uint32_t r = b; r < e; ++r) f.row(vals + r, kEmitRows, vc);
        emit_group<NV>(a, H + k, f.cnt, f.w, vc);
    };
    const uint32_t min_heads = a.striped_min_heads ? a.striped_min_heads : kStripedMinHeads;
    if (heads >= min_heads * (uint32_t)kSubTiles) {
#pragma unroll 1
        for (int j = 0; j < R; ++j)
            if ((mine >> j) & 1u) group(index_of(j));
    } else {
#pragma unroll 1
        for (uint32_t k = tid; k < heads; k += kSegThreads) group(k);
    }
    // groups past one thread's rows, if there can be one: eight lanes or a warp each
    if (rows - heads >= kThreadRows) {
        __syncthreads();
        const uint32_t nlong = s_nlong;
#pragma unroll 1
        for (uint32_t i0 = warp * 4; i0 < nlong; i0 += kSegThreads / 8) {
            const uint32_t i = i0 + (lane >> 3);
            const uint32_t k = i < nlong ? s_long[i] : 0;
            const uint32_t b = s_pos[k], e = s_pos[k + 1];
            const bool here = i < nlong && e - b <= kTeamRows;
            Fold<NV> f;
            if (here) {
#pragma unroll 1
                for (uint32_t r = b + (lane & 7); r < e; r += 8) f.row(vals + r, kEmitRows, vc);
            }
            f.team(8, vc);
            if (here && (lane & 7) == 0) emit_group<NV>(a, H + k, f.cnt, f.w, vc);
        }
#pragma unroll 1
        for (uint32_t i = warp; i < nlong; i += kSegThreads / 32) {
            const uint32_t k = s_long[i], b = s_pos[k], e = s_pos[k + 1];
            if (e - b <= kTeamRows) continue;
            Fold<NV> f;
#pragma unroll 1
            for (uint32_t r = b + lane; r < e; r += 32) f.row(vals + r, kEmitRows, vc);
            f.team(32, vc);
            if (lane == 0) emit_group<NV>(a, H + k, f.cnt, f.w, vc);
        }
    }
    if (warp == kSegThreads / 32 - 1 && H > 0 && (heads > 0 || table_end)) carried(s_pos[0]);  // (no head: rows)
}

template <int NK, int NV>
cudaError_t seg_run(const SegArgs& a, unsigned char* ws, uint32_t tiles, cudaStream_t s, Profiler* prof) {
    uint32_t* done = reinterpret_cast<uint32_t*>(ws);
    Agg<NV>* ta = reinterpret_cast<Agg<NV>*>(ws + 256);
    const uint32_t blocks = (tiles + kScanTiles - 1) / kScanTiles;
    Agg<NV>* bt = ta + tiles;
    if (prof) prof->begin(KC_SEGREDUCE, s);
    // the float + signed-integer value pair with two keys of fixed widths
    // (8+4, 4+8, 4+4 bytes) gets fully specialised kernels
    const bool fixed = NV == 2 && value_class_pattern(a) == 1;
    const int kwp = (fixed && NK == 2) ? key_width_pattern(a) : 0;
    const uint32_t wide_grid = (tiles + kSubTiles - 1) / kSubTiles;
    bool launched_tiles = false;
    if constexpr (NK == 2 && NV == 2) {
        launched_tiles = true;
        if (kwp == 0x48)
            k_seg_tiles_wide<NK, NV, 1, 0x48><<<wide_grid, kSegThreads, 0, s>>>(a, ta, tiles, done);
        else if (kwp == 0x84)
            k_seg_tiles_wide<NK, NV, 1, 0x84><<<wide_grid, kSegThreads, 0, s>>>(a, ta, tiles, done);
        else if (kwp == 0x44)
            k_seg_tiles_wide<NK, NV, 1, 0x44><<<wide_grid, kSegThreads, 0, s>>>(a, ta, tiles, done);
        else
            launched_tiles = false;
    }
    if (!launched_tiles) {
        if constexpr (NV == 2) {
            if (fixed) k_seg_tiles_wide<NK, NV, 1><<<wide_grid, kSegThreads, 0, s>>>(a, ta, tiles, done);
            else k_seg_tiles_wide<NK, NV, 0><<<wide_grid, kSegThreads, 0, s>>>(a, ta, tiles, done);
        } else {
            k_seg_tiles_wide<NK, NV, 0><<<wide_grid, kSegThreads, 0, s>>>(a, ta, tiles, done);
        }
    }
    if (prof) prof->end(KC_SEGREDUCE, s);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (prof) prof->begin(KC_SEGSCAN, s);
    e = launch_after(k_seg_scan<NV>, blocks, kScanTiles, 0, s, a, ta, bt, tiles, done);
    if (prof) prof->end(KC_SEGSCAN, s);
    if (e != cudaSuccess) return e;
    if (prof) prof->begin(KC_SEGEMIT, s);
    constexpr size_t smem = emit_smem_bytes<NV>();
    auto emit = k_seg_emit<NK, NV, 0>;
    if constexpr (NV == 2) {
        if (fixed) emit = k_seg_emit<NK, NV, 1>;
    }
    if constexpr (NK == 2 && NV == 2) {
        if (kwp == 0x48) emit = k_seg_emit<NK, NV, 1, 0x48>;
        else if (kwp == 0x84) emit = k_seg_emit<NK, NV, 1, 0x84>;
        else if (kwp == 0x44) emit = k_seg_emit<NK, NV, 1, 0x44>;
    }
    e = launch_after(emit, wide_grid, kSegThreads, smem, s, a, ta, bt, tiles);
    if (prof) prof->end(KC_SEGEMIT, s);
    return e;
}

// Only three and four value columns need more than 48 KB (none of the
// specialised instances does).
template <int NK, int NV>
cudaError_t seg_attr() {
    return cudaFuncSetAttribute(k_seg_emit<NK, NV, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)emit_smem_bytes<NV>());
}

template <int NK>
cudaError_t seg_attrs() {
    cudaError_t e;
    if ((e = seg_attr<NK, 0>()) != cudaSuccess) return e;
    if ((e = seg_attr<NK, 1>()) != cudaSuccess) return e;
    if ((e = seg_attr<NK, 2>()) != cudaSuccess) return e;
    if ((e = seg_attr<NK, 3>()) != cudaSuccess) return e;
    return seg_attr<NK, 4>();
}

template <int NK>
cudaError_t seg_run_nv(const SegArgs& a, unsigned char* ws, uint32_t tiles, cudaStream_t s, Profiler* prof) {
    switch (a.nvals) {
    case 0: return seg_run<NK, 0>(a, ws, tiles, s, prof);
    case 1: return seg_run<NK, 1>(a, ws, tiles, s, prof);
    case 2: return seg_run<NK, 2>(a, ws, tiles, s, prof);
    case 3: return seg_run<NK, 3>(a, ws, tiles, s, prof);
    default: return seg_run<NK, 4>(a, ws, tiles, s, prof);
    }
}

size_t agg_bytes(int nvals) {
    switch (nvals) {
    case 0: return sizeof(Agg<0>);
    case 1: return sizeof(Agg<1>);
    case 2: return sizeof(Agg<2>);
    case 3: return sizeof(Agg<3>);
    default: return sizeof(Agg<4>);
    }
}

uint32_t seg_tiles(uint64_t n) { return (uint32_t)((n + kSegTile - 1) / kSegTile); }

}  // namespace

cudaError_t prepare_segreduce_kernels() {
    cudaError_t e;
    if ((e = seg_attrs<1>()) != cudaSuccess) return e;
    if ((e = seg_attrs<2>()) != cudaSuccess) return e;
    if ((e = seg_attrs<3>()) != cudaSuccess) return e;
    return seg_attrs<4>();
}

// [256 B: the scan's counter][tile aggregates][CTA totals of the scan]
size_t segreduce_workspace_bytes(uint64_t n, int nvals) {
    const size_t tiles = seg_tiles(n);
    return 256 + (tiles + (tiles + kScanTiles - 1) / kScanTiles) * agg_bytes(nvals);
}

cudaError_t run_segreduce(SegArgs a, unsigned char* ws, cudaStream_t s, Profiler* prof, int* launches) {
    if (a.n == 0) {
        if (a.n_groups) return cudaMemsetAsync(a.n_groups, 0, sizeof(uint64_t), s);
        return cudaSuccess;
    }
    const uint32_t tiles = seg_tiles(a.n);
    cudaError_t e;
    switch (a.nkeys) {
    case 1: e = seg_run_nv<1>(a, ws, tiles, s, prof); break;
    case 2: e = seg_run_nv<2>(a, ws, tiles, s, prof); break;
    case 3: e = seg_run_nv<3>(a, ws, tiles, s, prof); break;
    default: e = seg_run_nv<4>(a, ws, tiles, s, prof); break;
    }
    if (launches) *launches += 3;
    return e;
}

}  // namespace vdf
