// vdf_dictagg.cu -- group-by by one key of at most kDictMax distinct values
// without a sort, for calls that ask only for the group table.
//
// The reference's group-by is one hash probe per row into per-thread maps
// merged serially (transform_group_by_onecol_mt.hpp:182-337,
// merge_functions.inl:3-36).  With few distinct keys the same shape fits the
// GPU's shared memory: every row is read once and folded into its group's
// accumulators there, instead of being sorted, gathered and reduced as a
// segment.
//   1. k_dict_seen    the key's distinct values from a sample of the rows (one
//                     in 32) or, when the sample missed one, from every row:
//                     rows already in the CTA's table cost one lookup, new
//                     values take the insertion path;
//   2. k_dict_rank    (vdf_dict.cu) ranks them: rank = group
//   3. k_dict_agg     one CTA per SM; each row's rank is looked up and the
//                     row added to accumulators in shared memory; per CTA one
//                     partial per group goes to HBM; a key that was not
//                     collected sets `missed`
//   4. k_dict_finish  one warp per group merges the CTAs' partials in CTA
//                     order and writes the group.
// Sums are carried as in the segmented reduction (vdf_agg.cuh): 128-bit
// integers, compensated f64.  Nothing is read back between the launches; the
// words that tell whether the groups were written are read with the group
// count.
#include <algorithm>
#include <type_traits>

#include "vdf_agg.cuh"
#include "vdf_common.cuh"
#include "vdf_dict.cuh"
#include "vdf_internal.h"

namespace vdf {
namespace {

constexpr int kAggThreads = 1024, kAggWarps = kAggThreads / 32;
constexpr size_t kAggSmem = 220 * 1024;
constexpr size_t kAggTables = 8192;  // lookup table
constexpr uint32_t kSampleStep = 32;
constexpr int kSeenRows = 4;  // rows per lane of a warp's piece: when collecting values
// ... and when aggregating (two sets of rows are held in 64 registers)
template <typename K>
constexpr int kAggRows = sizeof(K) == 8 ? 3 : 4;

// Partial of one group in one CTA: rows, and four words per value column.
struct AggPart {
    uint64_t cnt;
    uint64_t w[kMaxVals][4];
};

// ---------------------------------------------------------------------------
// 1. the key's values
// ---------------------------------------------------------------------------
// Rows come in pieces of 32 * kSeenRows consecutive ones, a warp per piece;
// every `step`-th piece is looked at.
template <typename K>
__global__ void __launch_bounds__(512) k_dict_seen(DictArgs a, uint64_t step) {
    __shared__ unsigned long long skey[kDictCtaSlots];
    __shared__ uint32_t scnt[kDictCtaSlots], sst[kDictCtaSlots];
    __shared__ uint32_t sdist, sover;
    for (uint32_t i = threadIdx.x; i < kDictCtaSlots; i += blockDim.x) {
        scnt[i] = 0;
        sst[i] = 0;
    }
    if (threadIdx.x == 0) {
        sdist = 0;
        sover = 0;
    }
    __syncthreads();
    const uint32_t limit = a.spin_limit ? a.spin_limit : kSpinLimit;
    const K* src = static_cast<const K*>(a.keys);
    const int lane = threadIdx.x & 31;
    constexpr uint64_t PIECE = 32 * kSeenRows;
    const uint64_t pieces = (a.n + PIECE - 1) / PIECE;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x / 32);
    uint32_t round = 0;
    for (uint64_t q = ((uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32) * step; q < pieces;
         q += warps * step, ++round) {
        // exits are decided for the whole warp (see k_dict_collect)
        if (__any_sync(0xffffffffu, ld_volatile(&sover) != 0)) break;
        if ((round & 7) == 7 && __any_sync(0xffffffffu, ld_volatile(a.overflow) != 0)) break;
        const uint64_t i0 = q * PIECE + lane;
        K k[kSeenRows];
#pragma unroll
        for (int r = 0; r < kSeenRows; ++r) k[r] = i0 + 32 * r < a.n ? ldg_stream(src + i0 + 32 * r) : K(0);
#pragma unroll
        for (int r = 0; r < kSeenRows; ++r) {
            const bool valid = i0 + 32 * r < a.n;
            const unsigned long long x = (unsigned long long)KeyOps<K>::order(k[r], a.dtype, a.invert != 0);
            const uint32_t h0 = dict_hash(x) & (kDictCtaSlots - 1), h1 = (h0 + 1) & (kDictCtaSlots - 1);
            const uint32_t st0 = ld_volatile(&sst[h0]);
            bool seen = st0 == 2 && ld_volatile(&skey[h0]) == x;
            if (!seen && st0 != 0) seen = ld_volatile(&sst[h1]) == 2 && ld_volatile(&skey[h1]) == x;
            const uint32_t want = __ballot_sync(0xffffffffu, valid && !seen);
            if (want) {  // new values (or ones placed further on): one lane each
                const uint32_t peers = __match_any_sync(0xffffffffu, x) & want;
                if (valid && !seen && lane == __ffs(peers) - 1)
                    dict_add(skey, scnt, sst, kDictCtaSlots - 1, x, 0, limit, &sdist, &sover, a.err);
                __syncwarp();
            }
        }
    }
    __syncthreads();
    if (sover) {
        if (threadIdx.x == 0) atomicOr(a.overflow, 1u);
        return;
    }
    if (ld_volatile(a.overflow)) return;
    dict_merge(skey, scnt, sst, a, limit);
}

// ---------------------------------------------------------------------------
// 3. the aggregation
// ---------------------------------------------------------------------------
struct AggArgs {
    SegArgs seg;
    int invert, order;
    const unsigned long long* sorted;  // the values' order images by rank
    DictAggWords* words;
    unsigned char* parts;  // [CTA][kDictMax] AggPart
    uint32_t nparts;
    uint32_t* taken;
};

// Streaming loads that stay where they are written (the next rows' loads must
// be issued before the current rows are added).
__device__ __forceinline__ uint32_t ld_ahead(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.cs.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long ld_ahead(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.global.cs.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

// Column kinds fixed at compile time (CK_ANY: the dtype at run time; CK_NONE:
// rows are only counted).
enum ColKind : int { CK_ANY = 0, CK_F64 = 1, CK_I64 = 2, CK_NONE = 3 };
template <int CK>
__device__ __forceinline__ uint64_t canonical(uint64_t x, int dt) {
    if (CK != CK_ANY) return x;
    if (dt == I32) return (uint64_t)(int64_t)(int32_t)(uint32_t)x;
    if (dt == F32) return as_b((double)__uint_as_float((uint32_t)x));
    return x;
}

// Minimum and maximum of a group, shared by the CTA, as canonical values.
// Before any row: the largest value and the smallest (for floats +-infinity;
// both still in place at the end mean that every value was NaN).
__device__ __forceinline__ ulonglong2 minmax_start(int vc) {
    if (vc == VC_FLOAT) return make_ulonglong2(0x7ff0000000000000ull, 0xfff0000000000000ull);
    if (vc == VC_SINT) return make_ulonglong2(0x7fffffffffffffffull, 0x8000000000000000ull);
    return make_ulonglong2(~0ull, 0ull);
}
__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2* shared) {
    ulonglong2 v;
    asm volatile("ld.volatile.shared.v2.u64 {%0,%1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(smem_u32(shared)));
    return v;
}
// x is at or beyond the group's minimum or maximum as last read: rarely true.
__device__ __forceinline__ bool minmax_hit(uint64_t x, ulonglong2 m, int vc) {
    if (vc == VC_FLOAT) return (as_f(x) <= as_f(m.x)) | (as_f(x) >= as_f(m.y));  // never for NaN
    if (vc == VC_SINT) return ((int64_t)x < (int64_t)m.x) | ((int64_t)x > (int64_t)m.y);
    return (x < m.x) | (x > m.y);
}
// By the order of the bits' images, so that -0 comes before +0.
__device__ __noinline__ void minmax_update(unsigned long long* m, uint64_t x, int vc) {
    auto image = [vc](uint64_t v) -> uint64_t {
        if (vc == VC_FLOAT) return v ^ ((0ull - (v >> 63)) | 0x8000000000000000ull);
        return vc == VC_SINT ? v ^ 0x8000000000000000ull : v;
    };
    const uint64_t o = image(x);
#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
        unsigned long long cur = ld_volatile(m + side);
        while (side == 0 ? o < image(cur) : o > image(cur)) {
            const unsigned long long was = atomicCAS(m + side, cur, (unsigned long long)x);
            if (was == cur) break;
            cur = was;  // moved on by another row: closer to x with every round
        }
    }
}

// One value into an accumulator: (sum, compensation), or the 128-bit sum.
__device__ __forceinline__ void add_value(ulonglong2* p, uint64_t x, int cls) {
    ulonglong2 t = *p;
    if (cls == VC_FLOAT) {
        const double u = as_f(t.x), y = as_f(x);
        const double sum = __dadd_rn(u, y), bp = __dsub_rn(sum, u);
        const double e = __dadd_rn(__dsub_rn(u, __dsub_rn(sum, bp)), __dsub_rn(y, bp));  // TwoSum error
        t.x = as_b(sum);
        t.y = as_b(__dadd_rn(as_f(t.y), e));
    } else {
        const uint64_t hi = cls == VC_SINT ? (uint64_t)((int64_t)x >> 63) : 0ull;
        asm("add.cc.u64 %0, %0, %2;\n addc.u64 %1, %1, %3;" : "+l"(t.x), "+l"(t.y) : "l"(x), "l"(hi));
    }
    *p = t;
}
// The CTA's lookup table: raw key and rank side by side, one load per row.
template <typename K> struct RankEntry;
template <> struct RankEntry<uint32_t> {
    using E = uint2;
    static constexpr uint32_t SLOTS = 1024;
    static __device__ __forceinline__ uint32_t hash(uint32_t k) { return (k * 0x9e3779b1u) >> 22; }
};
template <> struct RankEntry<uint64_t> {
    using E = ulonglong2;
    static constexpr uint32_t SLOTS = 512;
    static __device__ __forceinline__ uint32_t hash(uint64_t k) {
        return (((uint32_t)k ^ (uint32_t)(k >> 32) * 0x85ebca6bu) * 0x9e3779b1u) >> 23;
    }
};

// A warp's share of the rows of one value column.  tab: lookup table, mm: the
// groups' minimum and maximum (nv pairs per group, this column's at mm), acc:
// this column's accumulators [group][slots], cnt: row counts (first column
// only).  Returns the largest rank met, d for a key without one.
template <typename K, int CK>
__device__ __forceinline__ uint32_t agg_column(const K* keys, const void* vals, int dt, uint64_t n, uint32_t d,
                                               const typename RankEntry<K>::E* tab, ulonglong2* mm, uint32_t nv,
                                               ulonglong2* acc, uint32_t* cnt, uint32_t slots, uint32_t mine,
                                               uint32_t copies, uint64_t first, uint64_t stride) {
    using RE = RankEntry<K>;
    using Entry = typename RE::E;
    constexpr int R = kAggRows<K>;
    constexpr uint64_t PIECE = 32 * R;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = lanemask_lt();
    const int cls = CK == CK_F64 ? VC_FLOAT : CK == CK_I64 ? VC_SINT : vclass(dt);
    const bool wide = CK != CK_ANY || dtype_width(dt) == 8;
    uint32_t worst = 0;
    K k[R], kn[R];
    uint64_t x[R], xn[R];
    auto load = [&](uint64_t i0) {  // i0 may lie past the end
        using L = typename std::conditional<sizeof(K) == 8, unsigned long long, uint32_t>::type;
        const L* kp = reinterpret_cast<const L*>(keys) + i0;
        const bool whole = i0 - lane + PIECE <= n;  // the same for the whole warp
        if (whole) {
#pragma unroll
            for (int r = 0; r < R; ++r) kn[r] = ld_ahead(kp + 32 * r);
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) kn[r] = i0 + 32 * r < n ? ld_ahead(kp + 32 * r) : 0;
        }
        if constexpr (CK != CK_NONE) {
            if (wide) {
                const unsigned long long* p = static_cast<const unsigned long long*>(vals) + i0;
                if (whole) {
#pragma unroll
                    for (int r = 0; r < R; ++r) xn[r] = ld_ahead(p + 32 * r);
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) xn[r] = i0 + 32 * r < n ? ld_ahead(p + 32 * r) : 0ull;
                }
            } else {
                const uint32_t* p = static_cast<const uint32_t*>(vals) + i0;
#pragma unroll
                for (int r = 0; r < R; ++r) xn[r] = i0 + 32 * r < n ? ld_ahead(p + 32 * r) : 0u;
            }
        }
    };
    load(first + lane);
    for (uint64_t p0 = first; p0 < n; p0 += stride) {
        const uint64_t i0 = p0 + lane;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            k[r] = kn[r];
            if constexpr (CK != CK_NONE) x[r] = xn[r];
        }
        load(i0 + stride);
        uint32_t rk[R];
        bool found = true;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const Entry e = tab[RE::hash(k[r])];
            rk[r] = (uint32_t)e.y;
            found &= e.x == k[r];
        }
        if (!found) {  // some row's key is not in its first slot
#pragma unroll
            for (int r = 0; r < R; ++r) {
                uint32_t h = RE::hash(k[r]);
                Entry e = tab[h];
                // (at most a lap of the table)
                for (uint32_t probe = 1; e.x != k[r] && (uint32_t)e.y != d && probe < RE::SLOTS; ++probe) {
                    h = (h + 1) & (RE::SLOTS - 1);
                    e = tab[h];
                }
                rk[r] = e.x == k[r] ? (uint32_t)e.y : d;
            }
        }
        if (p0 + PIECE <= n) {
#pragma unroll
            for (int r = 0; r < R; ++r) worst = max(worst, rk[r]);
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (i0 + 32 * r < n) worst = max(worst, rk[r]);
                else rk[r] = d;
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t s = rk[r] * slots + mine;
            const uint64_t xv = CK == CK_NONE ? 0ull : canonical<CK>(x[r], dt);
            auto add = [&]() {
                if (cnt) cnt[s] += 1;
                if constexpr (CK != CK_NONE) add_value(acc + s, xv, cls);
            };
            if (copies == 32) {
                add();
            } else {
                // lanes of one copy with the same group: one after another
                const uint32_t peers = __match_any_sync(0xffffffffu, rk[r] * 32 + (lane & (copies - 1)));
                const uint32_t turn = __popc(peers & lt);
                const uint32_t turns = __reduce_max_sync(0xffffffffu, turn);
                for (uint32_t q = 0; q <= turns; ++q) {
                    if (turn == q) add();
                    __syncwarp();
                }
            }
            if constexpr (CK != CK_NONE) {
                ulonglong2* m = mm + rk[r] * nv;
                if (minmax_hit(xv, ld_pair(m), cls)) minmax_update(reinterpret_cast<unsigned long long*>(m), xv, cls);
            }
        }
    }
    return worst;
}

// What bounds it: 20 bytes per row (a 4-byte key, two 8-byte values) at the
// copy rate leave an SM about 0.9 cycles per row, so instructions per row and
// the warps in flight count.  Accumulators sit in shared memory, private to a
// lane where they fit: `copies` of each group's accumulators per warp (32
// when the groups are few, fewer with more groups), lane l using copy
// l % copies; lanes of one copy that hold the same group take turns.  With
// many groups such clashes are rare, with few groups every lane has its own
// copy, so a row costs about one read-modify-write of 16 bytes per column
// either way.  Each warp takes one value column (the first column's warps
// count the rows): a lane then holds one column's accumulators, so twice the
// warps fit for two columns, which is worth more than looking every key up
// once per column costs.  Minimum and maximum are shared by the CTA: compared
// on every row, changed rarely.  The next rows are loaded while the current
// ones are added.  200M rows of 16 int32 keys (two hot ones), f64 + int64
// values, one B200: 1.58 ms (137 instructions per row, 46 % of issue slots)
// where collection, sort pass, pack, gather and reduction took 6.2 ms; with
// both columns in one warp 1.95 ms, with atomic row counts 7.6 ms.
template <typename K>
__global__ void __launch_bounds__(kAggThreads, 1) k_dict_agg(const __grid_constant__ AggArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    using RE = RankEntry<K>;
    using Entry = typename RE::E;
    if (a.words->state != 2) return;  // written by an earlier launch
    const uint32_t d = a.words->ndist;
    const uint32_t nv = (uint32_t)a.seg.nvals, cols = max(nv, 1u);
    Entry* tab = reinterpret_cast<Entry*>(smem);
    ulonglong2* mm = reinterpret_cast<ulonglong2*>(smem + kAggTables);  // [d + 1][nv] minimum, maximum
    // layout: the most copies that leave 16 warps, then as many warps as fit
    // (group d takes the rows that belong to none)
    const uint32_t room = (uint32_t)(kAggSmem - kAggTables) - (d + 1) * nv * 16;
    const uint32_t per = (d + 1) * (16 * nv + 4);
    uint32_t copies = 32, warps;  // warps: of one column
    for (;; copies >>= 1) {
        warps = min((uint32_t)kAggWarps / cols, room / (per * copies));
        if (warps * cols >= 16 || copies == 1) break;
    }
    const uint32_t slots = warps * copies;  // accumulators of one group and column
    ulonglong2* acc = mm + (d + 1) * nv;    // [nv][d + 1][slots]
    uint32_t* cnt = reinterpret_cast<uint32_t*>(acc + nv * (d + 1) * slots);  // [d + 1][slots]
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t warp = tid >> 5;
    for (uint32_t i = tid; i < RE::SLOTS; i += kAggThreads) tab[i].y = d;
    for (uint32_t i = tid; i < (d + 1) * nv; i += kAggThreads) mm[i] = minmax_start(vclass(a.seg.val[i % nv].dtype));
    for (uint32_t i = tid; i < nv * (d + 1) * slots; i += kAggThreads) acc[i] = make_ulonglong2(0ull, 0ull);
    for (uint32_t i = tid; i < (d + 1) * slots; i += kAggThreads) cnt[i] = 0;
    __syncthreads();
    for (uint32_t g = tid; g < d; g += kAggThreads) {
        const K k = KeyOps<K>::unorder((K)a.sorted[g], a.seg.key[0].dtype, a.invert != 0);
        uint32_t h = RE::hash(k);
        // more slots than groups: a free one is always found
        while (atomicCAS(&tab[h].y, (decltype(tab[h].y))d, (decltype(tab[h].y))g) != d) h = (h + 1) & (RE::SLOTS - 1);
        tab[h].x = k;
    }
    __syncthreads();

    const K* keys = static_cast<const K*>(a.seg.key[0].src);
    uint32_t worst = 0;
    const uint32_t v = warp % cols, wi = warp / cols;
    if (wi < warps) {
        const void* vals = nv ? a.seg.val[v].src : nullptr;
        const int dt = nv ? a.seg.val[v].dtype : 0;
        constexpr uint64_t PIECE = 32 * kAggRows<K>;
        const uint64_t first = ((uint64_t)blockIdx.x * warps + wi) * PIECE, stride = (uint64_t)gridDim.x * warps * PIECE;
        const uint32_t mine = wi * copies + (lane & (copies - 1));
        ulonglong2* vacc = acc + v * (d + 1) * slots;
        uint32_t* vcnt = v == 0 ? cnt : nullptr;
        if (nv == 0)
            worst = agg_column<K, CK_NONE>(keys, vals, dt, a.seg.n, d, tab, mm, nv, vacc, vcnt, slots, mine, copies,
                                           first, stride);
        else if (dt == F64)
            worst = agg_column<K, CK_F64>(keys, vals, dt, a.seg.n, d, tab, mm + v, nv, vacc, vcnt, slots, mine, copies,
                                          first, stride);
        else if (dt == I64)
            worst = agg_column<K, CK_I64>(keys, vals, dt, a.seg.n, d, tab, mm + v, nv, vacc, vcnt, slots, mine, copies,
                                          first, stride);
        else
            worst = agg_column<K, CK_ANY>(keys, vals, dt, a.seg.n, d, tab, mm + v, nv, vacc, vcnt, slots, mine, copies,
                                          first, stride);
    }
    if (__syncthreads_or(worst >= d) && tid == 0) atomicOr(&a.words->missed, 1u);

    // ---- one partial per group and column: a warp merges the accumulators.
    //      The rows of a slot's column-0 accumulator are counted there; the
    //      other columns' slots covered the same rows (the same warp index,
    //      lane and pieces), so the counts hold for every column.
    AggPart* part = reinterpret_cast<AggPart*>(a.parts) + (size_t)blockIdx.x * kDictMax;
    for (uint32_t i = warp; i < d * cols; i += kAggWarps) {
        const uint32_t g = i / cols, c = i % cols;
        const int vc = nv ? vclass(a.seg.val[c].dtype) : VC_UINT;
        uint32_t rows = 0;
        uint64_t w[4] = {0, 0, 0, 0};
        auto merge = [&](uint32_t r, const uint64_t (&o)[4]) {
            if (r == 0) return;
            if (rows == 0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) w[q] = o[q];
            } else {
                col_merge(w, o, vc);
            }
            rows += r;
        };
        for (uint32_t s = lane; s < slots; s += 32) {
            const uint32_t r = cnt[g * slots + s];
            uint64_t o[4] = {0, 0, 0, 0};
            if (nv) {
                const ulonglong2 t = acc[(c * (d + 1) + g) * slots + s];
                o[0] = t.x;
                // one row's sum is the row (an infinity left a NaN behind)
                o[1] = vc == VC_FLOAT && r == 1 ? 0ull : t.y;
                o[2] = o[3] = t.x;  // replaced by the CTA's below
            }
            merge(r, o);
        }
#pragma unroll 1
        for (int sh = 1; sh < 32; sh <<= 1) {
            const uint32_t r = __shfl_xor_sync(0xffffffffu, rows, sh);
            uint64_t o[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) o[q] = __shfl_xor_sync(0xffffffffu, w[q], sh);
            merge(r, o);
        }
        if (lane == 0) {
            if (c == 0) part[g].cnt = rows;
            if (nv) {
                const ulonglong2 m = mm[g * nv + c];
                const ulonglong2 none = minmax_start(vc);
                const bool nan = vc == VC_FLOAT && m.x == none.x && m.y == none.y;
                part[g].w[c][0] = w[0];
                part[g].w[c][1] = w[1];
                part[g].w[c][2] = nan ? 0x7fffffffffffffffull : m.x;
                part[g].w[c][3] = nan ? 0x7fffffffffffffffull : m.y;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// 4. merge of the partials, one warp per group
// ---------------------------------------------------------------------------
template <int NV>
__global__ void __launch_bounds__(256) k_dict_finish(const __grid_constant__ AggArgs a) {
    constexpr int NW = NV > 0 ? NV : 1;
    if (a.words->state != 2 || a.words->missed) return;  // written by earlier launches
    const uint32_t d = a.words->ndist;
    const uint32_t g = blockIdx.x * 8 + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (g >= d) return;
    int vc[NW];
#pragma unroll
    for (int v = 0; v < NV; ++v) vc[v] = vclass(a.seg.val[v].dtype);
    const AggPart* part = reinterpret_cast<const AggPart*>(a.parts) + g;
    uint32_t c = 0;
    uint64_t w[NW][4];
#pragma unroll
    for (int v = 0; v < NW; ++v)
#pragma unroll
        for (int q = 0; q < 4; ++q) w[v][q] = 0;
    auto merge = [&](uint32_t oc, const uint64_t (*o)[4]) {
        if (oc == 0) return;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            if (c == 0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) w[v][q] = o[v][q];
            } else {
                col_merge(w[v], o[v], vc[v]);
            }
        }
        c += oc;
    };
    for (uint32_t b = lane; b < a.nparts; b += 32) {
        const AggPart& p = part[(size_t)b * kDictMax];
        uint64_t o[NW][4];
#pragma unroll
        for (int v = 0; v < NV; ++v)
#pragma unroll
            for (int q = 0; q < 4; ++q) o[v][q] = p.w[v][q];
        merge((uint32_t)p.cnt, o);
    }
#pragma unroll 1
    for (int sh = 1; sh < 32; sh <<= 1) {
        const uint32_t oc = __shfl_xor_sync(0xffffffffu, c, sh);
        uint64_t o[NW][4];
#pragma unroll
        for (int v = 0; v < NW; ++v)
#pragma unroll
            for (int q = 0; q < 4; ++q) o[v][q] = __shfl_xor_sync(0xffffffffu, w[v][q], sh);
        merge(oc, o);
    }
    if (lane != 0) return;
    const uint32_t out = a.order == 2 ? d - 1 - g : g;
    const int kdt = a.seg.key[0].dtype, kw = dtype_width(kdt);
    if (a.seg.key_out[0])
        store_raw(a.seg.key_out[0], kw, out,
                  kw == 4 ? (uint64_t)unorder32((uint32_t)a.sorted[g], kdt, a.invert != 0)
                          : unorder64(a.sorted[g], kdt, a.invert != 0));
    emit_group<NV>(a.seg, out, c, w, vc);
    if (g == 0) {
        if (a.seg.n_groups) *a.seg.n_groups = d;
        if (a.taken) atomicAdd(a.taken, 1u);
    }
}

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// cleared words: DictAggWords | number of values | collection table
constexpr size_t kZeroTable = (sizeof(DictAggWords) + 4 + 15) / 16 * 16;
constexpr size_t kZeroBytes = kZeroTable + sizeof(DictSlot) * kDictSlots;
// workspace: lookup table | sorted values | partials
struct AggLayout {
    size_t lut, sorted, parts, total;
};
AggLayout agg_layout(int ctas) {
    AggLayout L{};
    size_t o = 0;
    L.lut = o; o = align_up(o + sizeof(DictLut), 256);
    L.sorted = o; o = align_up(o + 8 * kDictMax, 256);
    L.parts = o; o = align_up(o + (size_t)ctas * kDictMax * sizeof(AggPart), 256);
    L.total = o;
    return L;
}

// one copy of every accumulator, in one warp per column, always fits
static_assert(kAggTables + (size_t)(kDictMax + 1) * (kMaxVals * 16 + 16 * kMaxVals + 4) <= kAggSmem,
              "accumulators of one warp per column");
}  // namespace

size_t dict_agg_zeroed_bytes() { return kZeroBytes; }

size_t dict_agg_workspace_bytes() { return agg_layout(sm_count()).total; }

cudaError_t prepare_dict_agg_kernels() {
    cudaError_t e = cudaFuncSetAttribute(k_dict_agg<uint32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAggSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_dict_agg<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAggSmem);
    return e;
}

cudaError_t run_dict_agg(const DictAggPlan& p, bool sample, unsigned char* zeroed, unsigned char* ws, cudaStream_t s, Profiler* prof,
                         int* launches) {
    const SegArgs& g = p.seg;
    const int sms = sm_count();
    const AggLayout L = agg_layout(sms);
    const int width = dtype_width(g.key[0].dtype);
    cudaError_t e = cudaMemsetAsync(zeroed, 0, kZeroBytes, s);
    if (e != cudaSuccess) return e;
    DictAggWords* words = reinterpret_cast<DictAggWords*>(zeroed);
    DictArgs da{};
    da.keys = g.key[0].src;
    da.dtype = g.key[0].dtype;
    da.invert = p.order == 1 ? 1 : 0;
    da.width = width;
    da.n = g.n;
    da.table = reinterpret_cast<DictSlot*>(zeroed + kZeroTable);
    da.distinct = reinterpret_cast<uint32_t*>(zeroed + sizeof(DictAggWords));
    da.overflow = &words->overflow;
    da.state = &words->state;
    da.fail_state = 1;
    da.lut = reinterpret_cast<DictLut*>(ws + L.lut);
    da.spin_limit = p.spin_limit;
    da.err = g.err;
    da.counted = 0;
    da.sorted = reinterpret_cast<unsigned long long*>(ws + L.sorted);
    da.ndist = &words->ndist;
    const uint64_t step = sample ? kSampleStep : 1;
    const uint64_t per_cta = 16 * 32 * kSeenRows * step;  // rows one round of a CTA covers
    const uint32_t seen = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((g.n + per_cta - 1) / per_cta,
                                                                            (uint64_t)sms * 4));
    if (prof) prof->begin(KC_DICT, s);
    if (width == 8) k_dict_seen<uint64_t><<<seen, 512, 0, s>>>(da, step);
    else k_dict_seen<uint32_t><<<seen, 512, 0, s>>>(da, step);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = dict_rank(da, s);
    if (prof) prof->end(KC_DICT, s);
    if (e != cudaSuccess) return e;

    AggArgs a{};
    a.seg = g;
    a.invert = da.invert;
    a.order = p.order;
    a.sorted = da.sorted;
    a.words = words;
    a.parts = ws + L.parts;
    a.nparts = (uint32_t)sms;
    a.taken = p.taken;
    if (prof) prof->begin(KC_SEGREDUCE, s);
    if (width == 8) k_dict_agg<uint64_t><<<(uint32_t)sms, kAggThreads, kAggSmem, s>>>(a);
    else k_dict_agg<uint32_t><<<(uint32_t)sms, kAggThreads, kAggSmem, s>>>(a);
    if (prof) prof->end(KC_SEGREDUCE, s);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (prof) prof->begin(KC_SEGEMIT, s);
    switch (g.nvals) {
    case 0: k_dict_finish<0><<<kDictMax / 8, 256, 0, s>>>(a); break;
    case 1: k_dict_finish<1><<<kDictMax / 8, 256, 0, s>>>(a); break;
    case 2: k_dict_finish<2><<<kDictMax / 8, 256, 0, s>>>(a); break;
    case 3: k_dict_finish<3><<<kDictMax / 8, 256, 0, s>>>(a); break;
    default: k_dict_finish<4><<<kDictMax / 8, 256, 0, s>>>(a); break;
    }
    if (prof) prof->end(KC_SEGEMIT, s);
    if (launches) *launches += 4;
    return cudaGetLastError();
}

}  // namespace vdf
