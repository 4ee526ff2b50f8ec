// vdf_small.cu -- one small frame sorted, gathered and grouped by one CTA in
// one launch.
//
// The reference runs such a call (sort_by_mt.hpp:3-180, then
// transform_group_by_onecol_mt.hpp:182-337) in tens of microseconds on the
// host; on the GPU the general path's fifteen launches of a few microseconds
// each cost more than the work.  Up to kSmallRows rows fit one CTA: one
// counting pass where a single key's values are spread, else stable 8-bit LSD
// passes in shared memory over every key column (least significant first,
// digits that do not vary skipped), the payload gathered through the
// row ids, the groups' heads from one scan, and each group folded from
// staged values -- by one thread up to 32 rows, by a warp above.  Sums and
// results are those of the segmented reduction (vdf_agg.cuh).
//
// What bounds it is one SM's instruction issue and the barriers; whole calls
// with the group count read back, one B200, general path -> this kernel: 1,000
// rows of 100 int32 keys with f64 + int64 values 98 -> 38 us (13 us of them
// the kernel; with LSD passes instead of the counting pass 18 us), 4,096 rows
// of int64 keys 140 -> 52 us, 3,000 rows sorted by three keys 257 -> 60 us.
#include "vdf_agg.cuh"
#include "vdf_common.cuh"
#include "vdf_count.cuh"
#include "vdf_internal.h"

namespace vdf {
namespace {

constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kItems = (int)kSmallRows / kThreads;
constexpr int kRadix = 256;
static_assert(kWarps * kRadix * 2 + 16 >= ((int)kSmallRows + 1) * 4, "groups' first rows");
constexpr uint32_t kThreadRows = 32;  // longest group one thread folds

constexpr int kBins = kWarps * kRadix * 2 / 4;  // counting bins: the passes' counters as words
static_assert(kBins == 4 * kThreads, "four bins per thread");

// Shared memory for n rows: key images | row ids | counters (or bins, later
// the groups' first rows) | small words | positions | staged value columns.
struct Layout {
    uint32_t vals, cnt, misc, orig, cols, total;
};
__host__ __device__ inline Layout layout(uint32_t n, int nvals) {
    const uint32_t rows = (n + 31) / 32 * 32;
    Layout L{};
    L.vals = rows * 8;
    L.cnt = L.vals + rows * 4;
    L.misc = L.cnt + kWarps * kRadix * 2 + 16;  // the groups' first rows need one word more
    L.orig = L.misc + 1024;
    L.cols = L.orig + rows * 2;
    L.total = L.cols + rows * 8 * (uint32_t)nvals;
    return L;
}
static_assert(kWarps * kRadix * 2 >= ((int)kSmallRows + 1) * 4 - 512, "groups' first rows fit the counters and words");

// Exclusive scan of one value per thread over the CTA; *total: the sum.
__device__ __forceinline__ uint32_t cta_scan(uint32_t v, uint32_t* wsum, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    const uint32_t t = wsum[lane];  // kWarps = 32 totals
    const uint32_t base = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0u);
    *total = __reduce_add_sync(0xffffffffu, t);
    return base + incl - v;
}

__device__ __forceinline__ uint64_t raw_at(const void* p, int w, uint32_t i) {
    return w == 4 ? (uint64_t) static_cast<const uint32_t*>(p)[i] : static_cast<const uint64_t*>(p)[i];
}
__device__ __forceinline__ uint64_t raw_key(uint64_t image, int dt, bool invert) {
    return dtype_width(dt) == 4 ? (uint64_t)unorder32((uint32_t)image, dt, invert) : unorder64(image, dt, invert);
}

// One key: a counting pass over kBins bins of the keys' range; the histogram's
// atomics hand each row its slot in its bin, and the rows sharing a bin are
// ranked by (key, position), as in the MSD sort's finish (vdf_msd.cu).  False,
// with sk and sv unspecified, when a bin holds more than kMsdRunMax rows: the
// LSD passes take the rows then.  On success they are in sk / sv.
__device__ __forceinline__ bool count_sort(const uint64_t (&key)[kItems], const uint32_t (&val)[kItems], uint32_t n,
                                           uint32_t ia, uint64_t* sk, uint32_t* sv, uint16_t* so, uint32_t* bins,
                                           uint32_t* wsum, uint64_t* wkey, uint32_t* err) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t pos0 = (uint32_t)warp * ia * 32 + lane;
    uint64_t kmin = ~0ull, kmax = 0;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (j < (int)ia && pos0 + 32 * j < n) {
            kmin = min(kmin, key[j]);
            kmax = max(kmax, key[j]);
        }
    }
    kmin = warp_min(kmin);
    kmax = warp_max(kmax);
    if (lane == 0) {
        wkey[warp] = kmin;
        wkey[32 + warp] = kmax;
    }
    reinterpret_cast<uint4*>(bins)[tid] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    BinMap<uint64_t, kBins> bin;
    bin.set(warp_min(wkey[lane]), warp_max(wkey[32 + lane]));
    uint32_t br[kItems];  // bin | arrival index in the bin << 16
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        br[j] = 0;
        if (j < (int)ia && pos0 + 32 * j < n) {
            const uint32_t b = bin(key[j]);
            br[j] = b | (atomicAdd(&bins[b], 1u) << 16);
        }
    }
    __syncthreads();
    const uint4 c = reinterpret_cast<const uint4*>(bins)[tid];
    if (__syncthreads_or(max(max(c.x, c.y), max(c.z, c.w)) > kMsdRunMax)) return false;
    uint32_t all, run = cta_scan(c.x + c.y + c.z + c.w, wsum, &all);
    uint4 q;  // first slot | rows << 16
    q.x = run | (c.x << 16);
    q.y = (run + c.x) | (c.y << 16);
    q.z = (run + c.x + c.y) | (c.z << 16);
    q.w = (run + c.x + c.y + c.z) | (c.w << 16);
    reinterpret_cast<uint4*>(bins)[tid] = q;
    __syncthreads();
    uint32_t slot[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        slot[j] = 0;
        if (j < (int)ia && pos0 + 32 * j < n) {
            const uint32_t w = bins[br[j] & 0xffffu];
            slot[j] = (w & 0xffffu) + (br[j] >> 16);
            if (slot[j] >= n) {  // never when the counts are consistent
                atomicOr(err, ERR_BAD_INDEX);
                slot[j] = pos0 + 32 * j;
            }
            sk[slot[j]] = key[j];
            so[slot[j]] = (uint16_t)(pos0 + 32 * j);
            br[j] = w;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t rows = br[j] >> 16, b = br[j] & 0xffffu;
        if (rows <= 1) continue;
        uint32_t r = b;
#pragma unroll 1
        for (uint32_t t = b; t < b + rows; ++t) r += row_less(sk[t], so[t], key[j], pos0 + 32 * j);
        slot[j] = r;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        if (j < (int)ia && pos0 + 32 * j < n) {
            sk[slot[j]] = key[j];
            sv[slot[j]] = val[j];
        }
    }
    __syncthreads();
    return true;
}

__global__ void __launch_bounds__(kThreads, 1) k_small(const __grid_constant__ SmallArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t n = a.n;
    const Layout L = layout(n, a.seg.nvals);
    uint64_t* sk = reinterpret_cast<uint64_t*>(smem);
    uint32_t* sv = reinterpret_cast<uint32_t*>(smem + L.vals);
    uint16_t* wcnt = reinterpret_cast<uint16_t*>(smem + L.cnt);  // [kWarps][kRadix]
    uint32_t* hpos = reinterpret_cast<uint32_t*>(smem + L.cnt);  // after the sort: [groups + 1]
    uint32_t* wsum = reinterpret_cast<uint32_t*>(smem + L.misc);        // [32]
    uint32_t* wvary = reinterpret_cast<uint32_t*>(smem + L.misc + 128);  // [2][32]
    uint64_t* wkey = reinterpret_cast<uint64_t*>(smem + L.misc + 512);   // [2][32]
    uint16_t* so = reinterpret_cast<uint16_t*>(smem + L.orig);
    uint64_t* cols = reinterpret_cast<uint64_t*>(smem + L.cols);
    const uint32_t col_rows = (n + 31) / 32 * 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = lanemask_lt();
    const uint32_t ia = (n + kThreads - 1) / kThreads;  // items per thread in use
    const uint32_t pos0 = (uint32_t)warp * ia * 32 + lane;
    const bool invert = a.order == 1;

    // ---- stable LSD passes; item j of a thread sits at position pos0 + 32 j
    uint64_t key[kItems];
    uint32_t val[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t pos = pos0 + 32 * j;
        val[j] = 0;
        if (j < (int)ia && pos < n) {
            val[j] = a.perm_in ? a.perm_in[pos] : pos;
            if (val[j] >= n) {  // never for a permutation of [0, n)
                atomicOr(a.seg.err, ERR_BAD_INDEX);
                val[j] = 0;
            }
        }
    }
    for (int kc = a.seg.nkeys - 1; kc >= 0; --kc) {
        const int dt = a.seg.key[kc].dtype, kw = dtype_width(dt);
        uint64_t vary = 0;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            key[j] = 0;
            if (j < (int)ia && pos0 + 32 * j < n) {
                const uint64_t raw = raw_at(a.seg.key[kc].src, kw, val[j]);
                key[j] = kw == 4 ? (uint64_t)order32((uint32_t)raw, dt, invert) : order64(raw, dt, invert);
            }
        }
        if (a.seg.nkeys == 1 && count_sort(key, val, n, ia, sk, sv, so, reinterpret_cast<uint32_t*>(wcnt), wsum, wkey,
                                           a.seg.err))
            break;
        // the key bits that vary: against the first row's key
        __syncthreads();  // wsum, wvary, sk and sv of the previous key have been read
        if (tid == 0) sk[0] = key[0];
        __syncthreads();
        const uint64_t k0 = sk[0];
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            if (j < (int)ia && pos0 + 32 * j < n) vary |= key[j] ^ k0;
        const uint32_t vlo = __reduce_or_sync(0xffffffffu, (uint32_t)vary);
        const uint32_t vhi = __reduce_or_sync(0xffffffffu, (uint32_t)(vary >> 32));
        if (lane == 0) {
            wvary[warp] = vlo;
            wvary[32 + warp] = vhi;
        }
        __syncthreads();
        vary = (uint64_t)__reduce_or_sync(0xffffffffu, wvary[32 + lane]) << 32 |
               __reduce_or_sync(0xffffffffu, wvary[lane]);
        bool moved = false;
        for (int p = 0; p < kw; ++p) {
            const uint32_t shift = 8u * p;
            if (((vary >> shift) & 0xff) == 0) continue;
            for (int i = tid; i < kWarps * kRadix / 8; i += kThreads)
                reinterpret_cast<uint4*>(wcnt)[i] = make_uint4(0, 0, 0, 0);
            __syncthreads();
            uint16_t* my = wcnt + warp * kRadix;
            uint32_t rank[kItems];
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                rank[j] = 0;
                if (j < (int)ia) {
                    const bool ok = pos0 + 32 * j < n;
                    const uint32_t d = (uint32_t)(key[j] >> shift) & 0xffu;
                    const uint32_t peers = __match_any_sync(0xffffffffu, ok ? d : (uint32_t)kRadix);
                    const int leader = __ffs(peers) - 1;
                    uint32_t base = 0;
                    if (lane == leader && ok) {
                        base = my[d];
                        my[d] = (uint16_t)(base + __popc(peers));
                    }
                    __syncwarp();
                    base = __shfl_sync(0xffffffffu, base, leader);
                    rank[j] = base + __popc(peers & lt);
                }
            }
            __syncthreads();
            // starts in (digit, warp) order: four threads per digit, eight
            // warps' counters each
            const uint32_t bin = (uint32_t)tid >> 2, w0 = ((uint32_t)tid & 3) * 8;
            uint32_t c[8], sum = 0, all;
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                c[w] = wcnt[(w0 + w) * kRadix + bin];
                sum += c[w];
            }
            uint32_t run = cta_scan(sum, wsum, &all);
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                wcnt[(w0 + w) * kRadix + bin] = (uint16_t)run;
                run += c[w];
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                if (j < (int)ia && pos0 + 32 * j < n) {
                    uint32_t r = rank[j] + my[(uint32_t)(key[j] >> shift) & 0xffu];
                    if (r >= n) {  // never when the counts are consistent
                        atomicOr(a.seg.err, ERR_BAD_INDEX);
                        r = pos0 + 32 * j;
                    }
                    sk[r] = key[j];
                    sv[r] = val[j];
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                if (j < (int)ia && pos0 + 32 * j < n) {
                    key[j] = sk[pos0 + 32 * j];
                    val[j] = sv[pos0 + 32 * j];
                }
            }
            moved = true;
        }
        if (kc == 0 && !moved) {  // key 0 does not vary: the rows as they are
            __syncthreads();      // sk[0] has been read
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                if (j < (int)ia && pos0 + 32 * j < n) {
                    sk[pos0 + 32 * j] = key[j];
                    sv[pos0 + 32 * j] = val[j];
                }
            }
        }
    }
    __syncthreads();

    // ---- from here output row i is sorted row at(i) (order 2: mirrored)
    auto at = [&](uint32_t i) -> uint32_t { return a.order == 2 ? n - 1 - i : i; };
    uint32_t row[kItems];  // thread's output rows tid, tid + kThreads, ...
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t i = (uint32_t)j * kThreads + tid;
        row[j] = i < n ? sv[at(i)] : 0u;
    }
    uint32_t G = 0;
    if (a.groupby) {
        // heads: thread t looks at output rows [t * ia, t * ia + ia)
        const uint32_t r0 = min(n, (uint32_t)tid * ia), r1 = min(n, r0 + ia);
        uint32_t heads = 0;
        for (uint32_t i = r0; i < r1; ++i) {
            bool h = i == 0 || sk[at(i)] != sk[at(i - 1)];
            for (int k = 1; k < a.seg.nkeys && !h; ++k) {
                const int kw = dtype_width(a.seg.key[k].dtype);
                h = raw_at(a.seg.key[k].src, kw, sv[at(i)]) != raw_at(a.seg.key[k].src, kw, sv[at(i - 1)]);
            }
            heads |= h ? 1u << (i - r0) : 0u;
        }
        uint32_t g = cta_scan(__popc(heads), wsum, &G);  // (its barrier: the counters are free now)
        for (uint32_t i = r0; i < r1; ++i) {
            if ((heads >> (i - r0)) & 1u) {
                hpos[g] = i;
                for (int k = 0; k < a.seg.nkeys; ++k) {
                    if (!a.seg.key_out[k]) continue;
                    const int dt = a.seg.key[k].dtype, kw = dtype_width(dt);
                    store_raw(a.seg.key_out[k], kw, g,
                              k == 0 ? raw_key(sk[at(i)], dt, invert) : raw_at(a.seg.key[k].src, kw, sv[at(i)]));
                }
                if (a.seg.group_start) a.seg.group_start[g] = i;
                ++g;
            }
            if (a.seg.row_group) a.seg.row_group[i] = g - 1;
        }
        if (tid == 0) {
            hpos[G] = n;
            if (a.seg.n_groups) *a.seg.n_groups = G;
        }
    }
    // ---- permutation, sorted keys and payload; a column is read whole before
    //      it is written (outputs may be the inputs' own buffers)
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const uint32_t i = (uint32_t)j * kThreads + tid;
        if (i < n && a.perm_out) a.perm_out[i] = row[j];
    }
    uint64_t x[kItems];
    for (int k = 0; k < a.seg.nkeys; ++k) {
        if (!a.skey_out[k]) continue;
        const int dt = a.seg.key[k].dtype, kw = dtype_width(dt);
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const uint32_t i = (uint32_t)j * kThreads + tid;
            x[j] = 0;
            if (i < n) x[j] = k == 0 ? raw_key(sk[at(i)], dt, invert) : raw_at(a.seg.key[k].src, kw, row[j]);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const uint32_t i = (uint32_t)j * kThreads + tid;
            if (i < n) store_raw(a.skey_out[k], kw, i, x[j]);
        }
    }
    for (int p = 0; p < a.npay; ++p) {
        const int dt = a.pay_dtype[p], pw = dtype_width(dt);
        bool used = a.pay_dst[p] != nullptr;
        for (int v = 0; v < a.seg.nvals; ++v) used = used || a.val_pay[v] == p;
        if (!used) continue;
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
            const uint32_t i = (uint32_t)j * kThreads + tid;
            x[j] = i < n ? raw_at(a.pay_src[p], pw, row[j]) : 0ull;
        }
        for (int v = 0; v < a.seg.nvals; ++v) {
            if (a.val_pay[v] != p) continue;
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                const uint32_t i = (uint32_t)j * kThreads + tid;
                if (i >= n) continue;
                uint64_t y = x[j];
                if (dt == I32) y = (uint64_t)(int64_t)(int32_t)(uint32_t)y;
                else if (dt == F32) y = as_b((double)__uint_as_float((uint32_t)y));
                cols[v * col_rows + i] = y;
            }
        }
        if (a.pay_dst[p]) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                const uint32_t i = (uint32_t)j * kThreads + tid;
                if (i < n) store_raw(a.pay_dst[p], pw, i, x[j]);
            }
        }
    }
    if (!a.groupby) return;
    __syncthreads();

    // ---- groups: one thread per short group and column, a warp per long one
    if (a.seg.count_out)
        for (uint32_t g = tid; g < G; g += kThreads) a.seg.count_out[g] = (int64_t)(hpos[g + 1] - hpos[g]);
    const uint32_t tasks = G * (uint32_t)a.seg.nvals;
    for (uint32_t t = tid; t < tasks; t += kThreads) {
        const uint32_t v = t / G, g = t - v * G;
        const uint32_t b = hpos[g], e = hpos[g + 1];
        if (e - b > kThreadRows) continue;
        const int vc = vclass(a.seg.val[v].dtype);
        const uint64_t* c = cols + v * col_rows;
        uint64_t w[4];
        col_init(w, c[b], vc);
        for (uint32_t i = b + 1; i < e; ++i) {
            uint64_t one[4];
            col_init(one, c[i], vc);
            col_merge(w, one, vc);
        }
        emit_column(a.seg.agg[v], a.seg.val[v].dtype, g, e - b, w, vc);
    }
    for (uint32_t v = 0; v < (uint32_t)a.seg.nvals; ++v) {
        const int vc = vclass(a.seg.val[v].dtype);
        const uint64_t* c = cols + v * col_rows;
        for (uint32_t g = warp; g < G; g += kWarps) {
            const uint32_t b = hpos[g], e = hpos[g + 1];
            if (e - b <= kThreadRows) continue;
            uint64_t w[4];  // every lane holds a row: the group has more than 32
            col_init(w, c[b + lane], vc);
            for (uint32_t i = b + lane + 32; i < e; i += 32) {
                uint64_t one[4];
                col_init(one, c[i], vc);
                col_merge(w, one, vc);
            }
#pragma unroll 1
            for (int d = 16; d >= 1; d >>= 1) {
                uint64_t other[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) other[q] = __shfl_xor_sync(0xffffffffu, w[q], d);
                col_merge(w, other, vc);
            }
            if (lane == 0) emit_column(a.seg.agg[v], a.seg.val[v].dtype, g, e - b, w, vc);
        }
    }
}

}  // namespace

cudaError_t prepare_small_kernels() {
    return cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)layout(kSmallRows, kMaxVals).total);
}

cudaError_t run_small(const SmallArgs& a, cudaStream_t s, Profiler* prof) {
    static_assert(kItems * kThreads == (int)kSmallRows, "rows per thread");
    const Layout L = layout(a.n, a.seg.nvals);
    if (prof) prof->begin(KC_BATCH, s);
    k_small<<<1, kThreads, L.total, s>>>(a);
    if (prof) prof->end(KC_BATCH, s);
    return cudaGetLastError();
}

}  // namespace vdf
