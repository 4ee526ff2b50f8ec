// vdf_msd.cu -- most-significant-digit-first radix sort with a shared-memory
// finish, for sorts by one or two key columns.
//
// The reference sorts with LSD radix passes over every 16-bit digit of the
// key (radix_sort_uint64_mt.inl:6-166: four passes for an 8-byte key, each a
// histogram and a scatter of (key, size_t idx)), and composes a second key by
// a second sort through the in/out idx.  The LSD onesweep passes of
// vdf_radix.cu follow that shape with 8-bit digits: eight passes over HBM for
// an 8-byte key.  Here only the top P digits of key 0 go through HBM-wide
// passes, so that rows sharing the top 8P bits ("buckets") end up
// contiguous; the rest is finished per chunk of whole buckets in shared
// memory:
//
//   1. k_msd_hist    histograms of the top P digits of key 0 (one read)
//   2. k_msd_scan    their exclusive scans; a top-digit bin holding more rows
//                    than chunks could take for every bucket possible under it
//                    (bounded by the lower digits' non-empty bins) flags the
//                    MSD path as failed up front
//   3. P onesweep passes (vdf_radix.cu kernels), stable, over digits
//      W-P .. W-1 of key 0, least significant first: afterwards the rows
//      are stably sorted by their top 8P bits.  With P = 2 and 8-byte keys
//      the scan may ask for a third digit below them (keys whose top digits
//      are clustered, as those of doubles are)
//   4. k_msd_chunks  chunk c holds the whole buckets that start in
//                    [c*T, (c+1)*T); found by a two-level warp search for
//                    the first bucket boundary at or after c*T
//   5. k_msd_local   one CTA per chunk (<= kMsdCap rows): one counting pass
//                    over kMsdCap bins of the chunk's key range puts the rows
//                    of spread keys about two bins apart; the rows sharing a
//                    bin are ranked by (key 0, key 1's order image, position
//                    in the chunk) -- key 1 is read through the row id only
//                    where key 0 ties -- and the raw sorted key 0 and the
//                    permutation are written.  A chunk where a bin holds a
//                    run longer than kMsdRunMax (many equal or clustered
//                    keys) is sorted instead by stable passes over the dense
//                    bin index, or by stable 8-bit LSD passes in shared
//                    memory over the digits of key 0 above its low F bits
//                    that vary inside it, with runs of equal high bits ranked
//                    the same way (F = 32 for 8-byte keys, 0 for 4-byte keys).
//
// Every pass is stable and ties keep their row order, so the result is
// exactly the stable order over all keys.  A one-key chunk with a run longer
// than kMsdRunMax out of order is finished with more shared-memory passes.
// Where the data defeats the plan (a chunk above kMsdCap rows, or with two
// keys a long run whose key 0 ties or is out of order),
// a device flag is set and the LSD passes that follow in the same stream run
// from the raw columns instead (they return at once while the flag is
// clear); no host round trip either way.
#include "vdf_common.cuh"
#include "vdf_count.cuh"
#include "vdf_internal.h"

namespace vdf {

// ---------------------------------------------------------------------------
// 1. histograms of the top digits of key 0
// ---------------------------------------------------------------------------
template <typename K>
__global__ void __launch_bounds__(512) k_msd_hist(MsdHistArgs a) {
    // the plan word (written by an earlier launch): this plan runs only at 0
    if (a.flag && *a.flag != 0) return;
    __shared__ uint32_t h[kMsdMaxPasses * 256];
    for (int i = threadIdx.x; i < a.ndig * 256; i += blockDim.x) h[i] = 0;
    __syncthreads();
    const K* src = static_cast<const K*>(a.keys);
    const uint64_t n = a.n;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    constexpr int R = 4;  // four keys per thread per round, all loaded first
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += R * stride) {
        K k[R];
#pragma unroll
        for (int r = 0; r < R; ++r) k[r] = i0 + r * stride < n ? ldg_stream(src + i0 + r * stride) : K(0);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (i0 + r * stride >= n) break;
            const K x = KeyOps<K>::order(k[r], a.dtype, a.invert);
            for (int p = 0; p < a.ndig; ++p)
                atomicAdd(&h[p * 256 + (uint32_t)((x >> (8 * (a.first_digit + p))) & 0xff)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < a.ndig * 256; i += blockDim.x)
        if (h[i]) atomicAdd(&a.hist[i], h[i]);
}

// ---------------------------------------------------------------------------
// 2. exclusive scans (one CTA, one bin per thread) + the up-front checks
// ---------------------------------------------------------------------------
// The optional third digit serves clustered keys: 20M N(0,1) doubles sort in
// three top-digit passes and the finish, 0.95 ms, instead of eight LSD passes,
// 1.6 ms (the whole hard sort of a five-column frame 2.72 -> 1.98 ms).
//
// Also a sample of the keys (4 us), counted by their top 24 bits: where one value (or
// a cluster) holds far more rows than a chunk takes, the passes would be
// wasted (30M rows of 1,000 int64 values: 4.06 -> 3.53 ms without them).  One
// byte per slot of the count table; a slot that overflows only
// makes its neighbour look larger, when its own count has long told the same.
constexpr uint32_t kScanThreads = 1024, kSampleSlots = 8192, kSampleMax = 4096;
template <typename K>
__global__ void __launch_bounds__(kScanThreads) k_msd_scan(MsdHistArgs a, uint32_t* offs, uint32_t cap, uint32_t* flag,
                                                           uint32_t* deep) {
    __shared__ uint32_t wsum[8];
    __shared__ uint32_t nonempty[kMsdMaxPasses], largest[kMsdMaxPasses], most;
    __shared__ uint32_t seen[kSampleSlots / 4];
    if (*static_cast<volatile uint32_t*>(flag) != 0) return;  // another plan sorts (written by an earlier launch)
    const int ndig = a.ndig;
    const uint64_t n = a.n;
    const uint32_t* hist = a.hist;
    const int b = threadIdx.x, lane = b & 31, warp = b >> 5;
    if (b < kMsdMaxPasses) nonempty[b] = largest[b] = 0;
    if (b == 0) most = 0;
    for (uint32_t i = b; i < kSampleSlots / 4; i += kScanThreads) seen[i] = 0;
    // rows at equal distances (repeats in sorted data are spread like others)
    const uint32_t S = (uint32_t)min((uint64_t)kSampleMax, n / 256);
    const uint64_t step = n / kSampleMax > 256 ? n / kSampleMax : 256;
    constexpr int R = kSampleMax / kScanThreads;
    K key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t i = (uint32_t)r * kScanThreads + b;
        key[r] = i < S ? static_cast<const K*>(a.keys)[i * step] : K(0);
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if ((uint32_t)r * kScanThreads + b >= S) break;
        const uint32_t top = (uint32_t)(KeyOps<K>::order(key[r], a.dtype, a.invert) >> (8 * sizeof(K) - 24));
        const uint32_t slot = (top * 0x9e3779b1u) >> 19;
        atomicAdd(&seen[slot / 4], 1u << (8 * (slot & 3)));
    }
    for (int p = 0; p < ndig; ++p) {
        __syncthreads();  // wsum of the previous digit has been read
        const uint32_t v = b < 256 ? hist[p * 256 + b] : 0u;
        uint32_t incl = v;
        if (b < 256) {
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += t;
            }
            if (lane == 31) wsum[warp] = incl;
            const uint32_t ne = __popc(__ballot_sync(0xffffffffu, v != 0));
            const uint32_t top = __reduce_max_sync(0xffffffffu, v);
            if (lane == 0) {
                atomicAdd(&nonempty[p], ne);
                atomicMax(&largest[p], top);
            }
        }
        __syncthreads();
        if (b < 256) {
            uint32_t base = 0;
            for (int w = 0; w < warp; ++w) base += wsum[w];
            offs[p * 256 + b] = base + incl - v;
        }
    }
    uint32_t m = 0;
    for (uint32_t i = b; i < kSampleSlots / 4; i += kScanThreads) {
        const uint32_t q = seen[i];
        m = max(max(m, max(q & 0xffu, (q >> 8) & 0xffu)), max((q >> 16) & 0xffu, q >> 24));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0 && m) atomicMax(&most, m);
    __syncthreads();
    if (b != 0) return;
    // The optional lowest digit: taken where the top digit is clustered and
    // the largest bucket without it, as far as the digits' largest bins tell
    // (as if they were independent), is more than a chunk takes beside its
    // nominal rows, and fits with it.  (A few values spread over the whole
    // range have uneven bins too, but fill most of them.)
    int first = 0;
    if (deep) {
        const double f = 1.0 / (double)n;
        double est = (double)largest[ndig - 1];
        for (int p = 1; p + 1 < ndig; ++p) est *= largest[p] * f;
        const bool take = nonempty[ndig - 1] <= 128 && est > 0.5 * cap && est * largest[0] * f <= 0.5 * cap;
        *deep = take ? 1u : 0u;
        first = take ? 0 : 1;
    }
    // Rows under one top-digit value can form at most as many buckets as the
    // lower digits have distinct values (the product of their non-empty
    // bins); more rows than that many full chunks hold means some bucket
    // cannot fit a chunk.
    uint64_t under = 1;
    for (int p = first; p + 1 < ndig; ++p) under *= nonempty[p];
    if ((uint64_t)largest[ndig - 1] > (uint64_t)cap * under) atomicOr(flag, 1u);
    // Ten or more sampled rows in one slot do not come together by chance
    // (half a row per slot on average), and three chunks' rows by that count
    // are more than the count can be off.
    if (most >= 10 && (uint64_t)most * n > (uint64_t)3 * cap * S) atomicOr(flag, 1u);
}

// ---------------------------------------------------------------------------
// 4. chunk starts: one warp per chunk
// ---------------------------------------------------------------------------
template <typename K, uint32_t CAP>
__global__ void __launch_bounds__(256) k_msd_chunks(MsdChunkArgs a) {
    const int lane = threadIdx.x & 31;
    const uint32_t c = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (c > a.nchunks) return;
    const K* keys = static_cast<const K*>(a.keys);
    // chunk c starts at or after row x of rows [start, end) sorted by their
    // top bits (key >> pshift); a segmented sort gives each chunk its
    // segment's bounds, shift and failure flag
    uint64_t x = 0, start = 0, end = a.n;
    uint32_t pshift = a.pshift - (a.deep && *a.deep ? 8u : 0u);
    uint32_t* flag = a.flag;
    if (c < a.nchunks) {
        if (a.seg_chunks) {
            const MsdSegChunk d = a.seg_chunks[c];
            x = d.x;
            start = d.seg_start;
            end = min((uint64_t)d.seg_end, a.n);
            pshift = d.pshift;
            flag = a.seg_flag + d.seg;
        } else {
            x = (uint64_t)c * a.chunk_rows;
        }
    }
    uint64_t out;
    if (c == a.nchunks) {
        out = a.n;
    } else if (x <= start || x >= end) {
        // a segment's first chunk starts with it (written even when the
        // segment has failed: the chunk before it may end another segment)
        out = min(max(x, start), end);
    } else {
        uint32_t failed = 0;  // read once per warp: the ballots below need the whole warp
        if (lane == 0) failed = *static_cast<volatile uint32_t*>(flag);
        if (__shfl_sync(0xffffffffu, failed, 0)) return;
        // first i >= x whose top bits differ from row x-1's; rows are sorted
        // by their top bits, so "differs" is false up to the boundary and
        // true after it, and a probe tells on which side it lies
        const K p0 = keys[x - 1] >> pshift;
        constexpr uint32_t S = CAP / 32;  // level-1 probe spacing
        const uint64_t q = min(x + (uint64_t)(lane + 1) * S - 1, end - 1);
        const uint32_t hit = __ballot_sync(0xffffffffu, (keys[q] >> pshift) != p0);
        if (!hit) {
            // CAP rows after x still share row x-1's top bits: that bucket
            // is larger than a chunk can hold (or runs to the end)
            out = end;
            if (x + (uint64_t)32 * S - 1 < end - 1 && lane == 0) atomicOr(flag, 1u);
        } else {
            const uint32_t L = __ffs(hit) - 1;
            const uint64_t lo = x + (uint64_t)L * S;  // every row before lo shares p0
            const uint64_t hi = min(x + (uint64_t)(L + 1) * S - 1, end - 1);  // differs at hi
            out = hi;
#pragma unroll
            for (uint32_t r = 0; r < S / 32; ++r) {
                const uint64_t pos = lo + r * 32 + lane;
                const bool d = pos >= hi || (keys[pos] >> pshift) != p0;
                const uint32_t b = __ballot_sync(0xffffffffu, d);
                if (b) {
                    out = lo + r * 32 + (__ffs(b) - 1);
                    break;
                }
            }
        }
    }
    if (lane == 0) a.chunk_start[c] = (uint32_t)out;
}

// ---------------------------------------------------------------------------
// 5. shared-memory finish, one CTA per chunk
// ---------------------------------------------------------------------------
// Shared memory of a chunk of CAP rows: keys | row ids | bins (or the LSD
// passes' per-warp counters) | chunk positions | small words.  The key-1
// images of tied rows take the row ids' and bins' place: they are needed
// only between the last use of the bins and the row ids' exchange.
template <typename K, int THREADS, int ITEMS>
struct LocalCfg {
    static constexpr int WARPS = THREADS / 32;
    static constexpr int CAP = THREADS * ITEMS;
    static constexpr int NB = CAP;                  // counting bins: one per row a chunk can hold
    static constexpr int BPT = NB / THREADS;        // bins per thread of the scan
    static constexpr size_t KEYS = (size_t)CAP * sizeof(K);
    static constexpr size_t VALS = (size_t)CAP * 4;
    static constexpr size_t BINS = (size_t)NB * 4 > (size_t)WARPS * 256 * 4 ? (size_t)NB * 4 : (size_t)WARPS * 256 * 4;
    static constexpr size_t ORIG = (size_t)CAP * 2;  // chunk position of each slot's row; the dense-index table
    static constexpr size_t MISC = 16 * 4 + (size_t)WARPS * 4 + (size_t)2 * WARPS * 8;
    static constexpr size_t SMEM = KEYS + VALS + BINS + ORIG + MISC;
    static_assert(VALS + BINS >= (size_t)CAP * 8 && (KEYS % 16) == 0 && (VALS % 16) == 0, "key-1 images");
    static_assert(BPT % 4 == 0 && ORIG >= (size_t)NB * 2, "bin layout");
};

template <int THREADS>
__device__ __forceinline__ uint32_t local_excl_scan(uint32_t v, uint32_t* wsum, uint32_t* total) {
    constexpr int WARPS = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    // every warp sums the earlier warps' totals with one reduction
    static_assert(WARPS <= 32, "one lane per warp total");
    const uint32_t t = lane < WARPS ? wsum[lane] : 0u;
    const uint32_t base = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0u);
    *total = __reduce_add_sync(0xffffffffu, t);
    return base + incl - v;
}

__device__ __forceinline__ uint64_t sec_image(const void* col, int dt, uint32_t row, bool invert) {
    if (dtype_width(dt) == 8) return order64(ld_rand8(static_cast<const unsigned long long*>(col) + row), dt, invert);
    return (uint64_t)order32(ld_rand4(static_cast<const uint32_t*>(col) + row), dt, invert);
}

// One stable 8-bit LSD pass in shared memory over the digit digit(key) of
// the CTA's rows (item j of a thread at position (warp * ia + j) * 32 + lane;
// slots past the chunk hold all-ones keys, whose digit must be the largest,
// and rank last).  Afterwards the rows are in sk / sv in the new order and
// back in key / val by position.
template <typename K, int THREADS, int ITEMS, int MATCH, typename DigitF>
__device__ __forceinline__ void local_pass(K (&key)[ITEMS], uint32_t (&val)[ITEMS], DigitF digit, uint32_t ia,
                                           K* sk, uint32_t* sv, uint32_t* wcnt, uint32_t* wsum, uint32_t* err) {
    constexpr int WARPS = THREADS / 32, RADIX = 256;
    constexpr uint32_t CAP = (uint32_t)(THREADS * ITEMS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = lanemask_lt();
    uint32_t* my = wcnt + warp * RADIX;
    for (int i = tid; i < WARPS * RADIX; i += THREADS) wcnt[i] = 0;
    __syncthreads();
    uint32_t rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        rank[j] = 0;
        if (j < (int)ia) {
            const uint32_t d = digit(key[j]);
            uint32_t peers;
            if constexpr (MATCH == 1) {
                peers = __match_any_sync(0xffffffffu, d);
            } else {
                peers = 0xffffffffu;
#pragma unroll
                for (int bt = 0; bt < 8; ++bt) {
                    const uint32_t bal = __ballot_sync(0xffffffffu, (d >> bt) & 1u);
                    peers &= ((d >> bt) & 1u) ? bal : ~bal;
                }
            }
            const int leader = __ffs(peers) - 1;
            uint32_t base = 0;
            if (lane == leader) {
                base = my[d];
                my[d] = base + __popc(peers);
            }
            __syncwarp();
            base = __shfl_sync(0xffffffffu, base, leader);
            rank[j] = base + __popc(peers & lt);
        }
    }
    __syncthreads();
    // bin-major exclusive prefix over (bin, warp)
    uint32_t tot = 0;
    if (tid < RADIX) {
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const uint32_t c = wcnt[w * RADIX + tid];
            wcnt[w * RADIX + tid] = tot;
            tot += c;
        }
    }
    uint32_t all;
    const uint32_t start = local_excl_scan<THREADS>(tot, wsum, &all);
    if (tid < RADIX)
#pragma unroll
        for (int w = 0; w < WARPS; ++w) wcnt[w * RADIX + tid] += start;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (j < (int)ia) {
            const uint32_t d = digit(key[j]);
            uint32_t r = rank[j] + my[d];
            if (r >= CAP) {  // never when the counts are consistent
                atomicOr(err, ERR_BAD_INDEX);
                r = ((uint32_t)warp * ia + j) * 32 + lane;
            }
            sk[r] = key[j];
            sv[r] = val[j];
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (j < (int)ia) {
            const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
            key[j] = sk[pos];
            val[j] = sv[pos];
        }
    }
}

// The chunk's rows in one counting pass over NB bins of the chunk's key
// range (BinMap; the range is the chunk's first and last bucket, known from
// the rows' order, so no reduction over the keys is needed).  The histogram's
// atomics also hand every row its arrival index in its bin; after the scan a
// row alone in its bin is in its final position, and the few rows sharing a
// bin are ranked among themselves by (key, key 1's order image, position in
// the chunk) -- positions are the rows' stable order so far --, which
// restores the exact stable order.  Where a bin holds more than kMsdRunMax
// rows, the bins are laid out again over the keys' own range if that is less
// than half as wide (clustered keys), else (many equal keys) stable passes
// over the dense bin index order the rows.  On success the rows are in sk /
// sv by final position; false (nothing written to global memory): the caller
// sorts the chunk with LSD passes.
template <typename K, int THREADS, int ITEMS, int MATCH>
__device__ __forceinline__ bool counting_finish(K (&key)[ITEMS], uint32_t (&val)[ITEMS], uint32_t m, uint32_t ia,
                                                K lo, K hi, const MsdLocalArgs& a, K* sk, uint32_t* sv, uint16_t* so,
                                                uint32_t* bins, uint64_t* ssec, uint32_t* wsum, K* wmin, K* wmax) {
    using C = LocalCfg<K, THREADS, ITEMS>;
    constexpr int WARPS = C::WARPS, NB = C::NB, BPT = C::BPT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t pos0 = (uint32_t)warp * ia * 32 + lane;  // item j's position: pos0 + 32 j
    BinMap<K, NB> bin;
    bin.set(lo, hi);
    uint32_t br[ITEMS];  // bin | arrival index in the bin << 16
    uint32_t cnt[BPT], tsum;
    bool narrowed = false;
#pragma unroll 1
    for (;;) {  // at most twice; the bins are clear
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            br[j] = 0;
            if (j < (int)ia && pos0 + 32 * j < m) {
                const uint32_t b = bin(key[j]);
                br[j] = b | (atomicAdd(&bins[b], 1u) << 16);
            }
        }
        __syncthreads();
        uint32_t tmax = 0;
        tsum = 0;
#pragma unroll
        for (int i = 0; i < BPT; i += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(bins + tid * BPT + i);
            cnt[i] = q.x;
            cnt[i + 1] = q.y;
            cnt[i + 2] = q.z;
            cnt[i + 3] = q.w;
        }
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
            tmax = max(tmax, cnt[i]);
            tsum += cnt[i];
        }
        if (__syncthreads_or(tmax > kMsdRunMax) == 0) break;
        // A bin holds more rows than the direct ranking takes (many equal or
        // clustered keys).
        uint32_t occ = 0, total, b0 = NB, b1 = 0;  // occupied bins: how many, the first and last
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
            if (cnt[i]) {
                ++occ;
                b0 = min(b0, (uint32_t)(tid * BPT + i));
                b1 = tid * BPT + i;
            }
        }
        b0 = __reduce_min_sync(0xffffffffu, b0);
        b1 = __reduce_max_sync(0xffffffffu, b1);
        if (lane == 0) wmin[warp] = (K)((b1 << 16) | b0);
        uint32_t dn = local_excl_scan<THREADS>(occ, wsum, &total);
        b0 = lane < WARPS ? (uint32_t)wmin[lane] & 0xffffu : (uint32_t)NB;
        b1 = lane < WARPS ? (uint32_t)wmin[lane] >> 16 : 0u;
        b0 = __reduce_min_sync(0xffffffffu, b0);
        b1 = __reduce_max_sync(0xffffffffu, b1);
        if (!narrowed && b1 - b0 < NB / 2) {  // uniform over the CTA
            // the rows sit in less than half of the range: the bins again,
            // over the keys' own range
            narrowed = true;
            K kmin = ~K(0), kmax = 0;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if (j < (int)ia && pos0 + 32 * j < m) {
                    kmin = min(kmin, key[j]);
                    kmax = max(kmax, key[j]);
                }
            }
            kmin = warp_min(kmin);
            kmax = warp_max(kmax);
            __syncthreads();  // wmin has been read
            if (lane == 0) {
                wmin[warp] = kmin;
                wmax[warp] = kmax;
            }
#pragma unroll
            for (int i = 0; i < BPT; i += 4)
                *reinterpret_cast<uint4*>(bins + tid * BPT + i) = make_uint4(0, 0, 0, 0);
            __syncthreads();
            kmin = warp_min(lane < WARPS ? wmin[lane] : ~K(0));
            kmax = warp_max(lane < WARPS ? wmax[lane] : K(0));
            bin.set(kmin, kmax);
            __syncthreads();  // ... and again, before it may be written again
            continue;
        }
        // Stable passes over the dense bin index -- one when at most 256 bins
        // are occupied, else two -- keep each bin's rows in their stable
        // order, which is the final order wherever a bin holds one key value.
        uint16_t* dt = so;  // dense index of each bin
#pragma unroll
        for (int i = 0; i < BPT; ++i) {
            dt[tid * BPT + i] = (uint16_t)dn;
            dn += cnt[i] ? 1u : 0u;
        }
        __syncthreads();
        // slots past the chunk (all-ones keys) take the largest index, so they stay last
        auto dense = [&](K k) -> uint32_t { return k > bin.hi ? 0xffffu : (uint32_t)dt[bin(k)]; };
        if (total <= 256) {
            local_pass<K, THREADS, ITEMS, MATCH>(
                key, val, [&](K k) { return min(dense(k), 255u); }, ia, sk, sv, bins, wsum, a.err);
        } else {
            local_pass<K, THREADS, ITEMS, MATCH>(
                key, val, [&](K k) { return dense(k) & 0xffu; }, ia, sk, sv, bins, wsum, a.err);
            local_pass<K, THREADS, ITEMS, MATCH>(
                key, val, [&](K k) { return dense(k) >> 8; }, ia, sk, sv, bins, wsum, a.err);
        }
        // in order now unless some bin holds several key values (or, with a
        // second key, key 0 ties): then the caller's LSD passes take over
        bool bad = false;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t pos = pos0 + 32 * j;
            if (j < (int)ia && pos > 0 && pos < m) {
                const K prev = sk[pos - 1];
                bad |= a.sec ? !(prev < key[j]) : (prev > key[j]);
            }
        }
        return __syncthreads_or(bad) == 0;
    }
    // ---- bin starts (with the count, one word per bin), rows into their slots
    uint32_t all;
    uint32_t run = local_excl_scan<THREADS>(tsum, wsum, &all);
#pragma unroll
    for (int i = 0; i < BPT; i += 4) {
        uint4 q;
        q.x = run | (cnt[i] << 16);
        run += cnt[i];
        q.y = run | (cnt[i + 1] << 16);
        run += cnt[i + 1];
        q.z = run | (cnt[i + 2] << 16);
        run += cnt[i + 2];
        q.w = run | (cnt[i + 3] << 16);
        run += cnt[i + 3];
        *reinterpret_cast<uint4*>(bins + tid * BPT + i) = q;
    }
    __syncthreads();
    uint32_t fin[ITEMS];  // slot | rows in the bin << 16 (0: alone), then final position | moved << 16
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        fin[j] = 0;
        if (j < (int)ia && pos0 + 32 * j < m) {
            const uint32_t w = bins[br[j] & 0xffffu];
            uint32_t slot = (w & 0xffffu) + (br[j] >> 16);
            if (slot >= m) {  // never when the counts are consistent
                atomicOr(a.err, ERR_BAD_INDEX);
                slot = pos0 + 32 * j;
            }
            const bool shared = (w >> 16) > 1;
            fin[j] = shared ? slot | (w & 0xffff0000u) : slot;
            sk[slot] = key[j];
            if (shared) so[slot] = (uint16_t)(pos0 + 32 * j);
            br[j] = w & 0xffffu;  // the bin's first slot
        }
    }
    __syncthreads();
    // ---- rows sharing a bin: each looks at the bin's slots
    bool ties = false;  // some row's key 0 ties (two keys): key 1 decides
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t c = fin[j] >> 16;
        if (c <= 1) continue;
        const uint32_t slot = fin[j] & 0xffffu, end = br[j] + c;
        const K k = key[j];
        uint32_t r = br[j];
        bool tie = false;
        if (a.sec) {
            uint32_t t = slot;
#pragma unroll 1
            for (uint32_t i = 1; i < c; ++i) {
                if (++t == end) t = br[j];
                const K tk = sk[t];
                tie |= tk == k;
                r += tk < k ? 1u : 0u;
            }
        } else {
            const uint32_t o = pos0 + 32 * j;
#pragma unroll 1
            for (uint32_t t = br[j]; t < end; ++t) r += row_less(sk[t], so[t], k, o);
        }
        if (tie) {
            ties = true;
            uint32_t row = val[j];
            if (row >= a.n) {  // never for a permutation of [0, n)
                atomicOr(a.err, ERR_BAD_INDEX);
                row = 0;
            }
            ssec[slot] = sec_image(a.sec, a.sec_dtype, row, a.invert != 0);
            br[j] |= 0x10000u;  // ranked again below
        } else {
            fin[j] = r | (r != slot ? 0x10000u : 0u);  // bit 16: the row moves
        }
    }
    if (a.sec && __syncthreads_or(ties)) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (!(br[j] >> 16)) continue;
            const uint32_t b0 = br[j] & 0xffffu;
            const uint32_t c = fin[j] >> 16, slot = fin[j] & 0xffffu, end = b0 + c;
            const K k = key[j];
            const uint64_t sc = ssec[slot];
            uint32_t r = b0, t = slot;
#pragma unroll 1
            for (uint32_t i = 1; i < c; ++i) {
                if (++t == end) t = b0;
                const K tk = sk[t];
                bool less = tk < k;
                if (tk == k) {
                    const uint64_t tsc = ssec[t];
                    less = tsc < sc || (tsc == sc && so[t] < pos0 + 32 * j);
                }
                r += less ? 1u : 0u;
            }
            fin[j] = r | (r != slot ? 0x10000u : 0u);
        }
    }
    __syncthreads();  // every slot has been compared: rows to their final positions
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        if (j < (int)ia && pos0 + 32 * j < m) {
            const uint32_t f = fin[j] & 0xffffu;
            if (fin[j] >> 16) sk[f] = key[j];
            sv[f] = val[j];
        }
    }
    __syncthreads();
    return true;
}

// Issue-bound: what counts is instructions per row and the barriers between
// the phases.  Hence one histogram atomic per row whose result is also the
// row's slot (no second counting pass), bins scaled to the chunk's range
// without a reduction over its keys, a bin per row of capacity (half full on
// average: four rows in ten share one), ranking in registers with only the
// shared rows' compares going through shared memory, and one branch-free
// multi-word compare per slot.  100M rows of two keys, one B200: 2.80 ms
// before (506 instructions per row: two atomic passes over 8,192 bins, rows
// re-read by slot with their run bounds found by ballots), 1.33 ms now (247
// per row, 57 % of issue slots); 200M rows of 50M keys in 8,192-row chunks
// 7.1 -> 4.2 ms; 50M rows of 25M keys 1.40 -> 0.80 ms.  HBM would take the
// 24 bytes per row in 0.37 ms per 100M rows.
//
// MATCH (the stable passes): 0 = one ballot per digit bit, 1 = match.any.
template <typename K, int THREADS, int ITEMS, int MATCH>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) k_msd_local(MsdLocalArgs a) {
    using C = LocalCfg<K, THREADS, ITEMS>;
    constexpr int WARPS = C::WARPS;
    constexpr uint32_t CAP = (uint32_t)C::CAP;
    constexpr int KBITS = 8 * (int)sizeof(K);
    extern __shared__ __align__(16) unsigned char smem[];
    K* sk = reinterpret_cast<K*>(smem);
    uint32_t* sv = reinterpret_cast<uint32_t*>(smem + C::KEYS);
    uint64_t* ssec = reinterpret_cast<uint64_t*>(smem + C::KEYS);  // over the row ids and bins
    uint32_t* wcnt = reinterpret_cast<uint32_t*>(smem + C::KEYS + C::VALS);  // bins, or [WARPS][RADIX]
    uint16_t* so = reinterpret_cast<uint16_t*>(smem + C::KEYS + C::VALS + C::BINS);
    uint32_t* misc = reinterpret_cast<uint32_t*>(smem + C::KEYS + C::VALS + C::BINS + C::ORIG);  // [0]: long runs
    uint32_t* wsum = misc + 16;                                                                  // [WARPS]
    K* wor = reinterpret_cast<K*>(smem + C::KEYS + C::VALS + C::BINS + C::ORIG + 16 * 4 + WARPS * 4);
    K* wand = wor + WARPS;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the flag a failing chunk raises: the sort's, or its segment's
    uint32_t* const fail_word = a.seg_chunks ? a.seg_flag + a.seg_chunks[blockIdx.x].seg : a.flag;
    // One thread reads the flag and the chunk bounds for the whole CTA (the
    // flag may be raised by another CTA meanwhile; every thread must take
    // the same branch around the barriers below).
    if (tid == 0) {
        misc[1] = *static_cast<volatile uint32_t*>(fail_word);
        misc[2] = a.chunk_start[blockIdx.x];
        uint32_t e = a.chunk_start[blockIdx.x + 1];
        uint32_t ps = a.pshift - (a.deep && *a.deep ? 8u : 0u);
        if (a.seg_chunks) {
            e = min(e, a.seg_chunks[blockIdx.x].seg_end);  // the segment's last chunk
            ps = a.seg_chunks[blockIdx.x].pshift;
        }
        misc[3] = e;
        misc[4] = ps;
        misc[0] = 0;
    }
    __syncthreads();
    if (misc[1]) return;  // the plan failed earlier: the LSD passes take over
    const uint32_t s0 = misc[2], s1 = misc[3], pshift = misc[4];
    if (s1 <= s0) return;
    const uint32_t m = s1 - s0;
    if (m > CAP || s1 > a.n) {
        if (tid == 0) atomicOr(fail_word, 1u);
        return;
    }
    const uint32_t ia = (m + THREADS - 1) / THREADS;  // items per thread in use
#pragma unroll
    for (int i = 0; i < C::BPT; i += 4) *reinterpret_cast<uint4*>(wcnt + tid * C::BPT + i) = make_uint4(0, 0, 0, 0);

    // ---- load: item j of a thread sits at position (warp * ia + j) * 32 + lane;
    //      slots past m hold all-ones keys, which every pass ranks last
    K key[ITEMS];
    uint32_t val[ITEMS];
    const K* kin = static_cast<const K*>(a.keys) + s0;
    const uint32_t* vin = a.vals + s0;
    const uint32_t pos0 = (uint32_t)warp * ia * 32 + lane;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t pos = pos0 + 32 * j;
        key[j] = ~K(0);
        val[j] = 0;
        if (j < (int)ia && pos < m) {
            key[j] = ldg_stream(kin + pos);
            val[j] = ldg_stream(vin + pos);
        }
    }
    K carry = 0;  // the row before this warp's
    if (pos0 - lane > 0 && pos0 - lane < m) carry = kin[pos0 - lane - 1];
    const K first = kin[0], last = kin[m - 1];

    // ---- rows already in order (with one key: non-decreasing; with two:
    //      increasing, so key 1 decides nothing) stay where they are; this is
    //      the common case when each bucket holds one key value
    // (each warp's first 32 rows tell most chunks apart before the rest is looked at)
    bool in_order = true;
    auto check = [&](int j) {
        const uint32_t pos = pos0 + 32 * j;
        const K before = __shfl_sync(0xffffffffu, key[j], (lane + 31) & 31);
        const K prev = lane ? before : carry;
        carry = before;  // lane 0: lane 31's key, the row before the next item's
        if (pos > 0 && pos < m) in_order = in_order && (a.sec ? prev < key[j] : prev <= key[j]);
    };
    check(0);
    bool ordered = __syncthreads_or(!in_order) == 0;
    if (ordered && ia > 1) {
#pragma unroll
        for (int j = 1; j < ITEMS; ++j)
            if (j < (int)ia) check(j);
        ordered = __syncthreads_or(!in_order) == 0;
    }
    K* kout = static_cast<K*>(a.keys_out);
    if (ordered) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t pos = pos0 + 32 * j;
            if (j < (int)ia && pos < m) {
                uint64_t gp = (uint64_t)s0 + pos;
                if (a.reverse) gp = a.n - 1 - gp;
                stg_stream(a.perm_out + gp, val[j]);
                if (kout) stg_stream(kout + gp, KeyOps<K>::unorder(key[j], a.dtype, a.invert != 0));
            }
        }
        return;
    }

    // ---- one counting pass over the chunk's key range (whole buckets, so
    //      the first and last row's top bits bound it); where that leaves a
    //      long run (many equal or clustered keys), stable LSD passes instead
    const K below = pshift < (uint32_t)KBITS ? (K)((((K)1) << pshift) - 1) : ~K(0);
    if (counting_finish<K, THREADS, ITEMS, MATCH>(key, val, m, ia, first & ~below, last | below, a, sk, sv, so, wcnt,
                                                  ssec, wsum, wor, wand)) {
        for (uint32_t i = tid; i < m; i += THREADS) {
            uint64_t gp = (uint64_t)s0 + i;
            if (a.reverse) gp = a.n - 1 - gp;
            stg_stream(a.perm_out + gp, sv[i]);
            if (kout) stg_stream(kout + gp, KeyOps<K>::unorder(sk[i], a.dtype, a.invert != 0));
        }
        return;
    }
    uint32_t newpos[ITEMS];
    {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
            key[j] = ~K(0);
            val[j] = 0;
            if (j < (int)ia && pos < m) {
                key[j] = ldg_stream(kin + pos);
                val[j] = ldg_stream(vin + pos);
            }
        }
        // ---- which digits vary inside the chunk
        K vor = 0, vand = ~K(0);
    #pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
            if (j < (int)ia && pos < m) {
                vor |= key[j];
                vand &= key[j];
            }
        }
    #pragma unroll
        for (int d = 16; d >= 1; d >>= 1) {
            vor |= __shfl_xor_sync(0xffffffffu, vor, d);
            vand &= __shfl_xor_sync(0xffffffffu, vand, d);
        }
        if (lane == 0) {
            wor[warp] = vor;
            wand[warp] = vand;
        }
        __syncthreads();
        vor = 0;
        vand = ~K(0);
    #pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            vor |= wor[w];
            vand &= wand[w];
        }
        const K vary = vor ^ vand;

        // ---- stable 8-bit LSD passes in shared memory over the varying digits
        //      of key 0 from digit lo_bits / 8 up
        bool sorted_in_smem = false;
        for (int dg = (int)(a.lo_bits / 8); dg < KBITS / 8; ++dg) {
            const uint32_t shift = 8u * dg;
            if (((vary >> shift) & 0xff) == 0) continue;
            local_pass<K, THREADS, ITEMS, MATCH>(
                key, val, [shift](K k) { return (uint32_t)(k >> shift) & 0xffu; }, ia, sk, sv, wcnt, wsum, a.err);
            sorted_in_smem = true;
        }
        if (!sorted_in_smem) {
    #pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if (j < (int)ia) {
                    const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
                    sk[pos] = key[j];
                    sv[pos] = val[j];
                }
            }
            __syncthreads();
        }

        __syncthreads();  // the row ids' buffer has been read back: key 1's images go over it

        // ---- runs of equal high bits, ranked by (low bits, key 1, position).
        //      Key 1 is read (through the row id) only for rows whose low bits
        //      tie with another row of their run, i.e. rows whose key 0 ties.
        const bool fix = a.lo_bits > 0 || a.sec != nullptr;
        const uint32_t hs = a.lo_bits;  // high part = key >> hs
        const K lo_mask = hs ? (K)((((K)1) << hs) - 1) : K(0);
        uint32_t run[ITEMS];  // run bounds s | e << 16 (positions < 2^16); 0: not in a run
    #pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
            newpos[j] = pos;
            run[j] = 0;
            if (fix && j < (int)ia && pos < m) {
                const K h = key[j] >> hs;
                if ((pos > 0 && (sk[pos - 1] >> hs) == h) || (pos + 1 < m && (sk[pos + 1] >> hs) == h)) {
                    uint32_t s = pos, e = pos + 1;
                    while (s > 0 && pos - s < kMsdRunMax && (sk[s - 1] >> hs) == h) --s;
                    while (e < m && e - pos <= kMsdRunMax && (sk[e] >> hs) == h) ++e;
                    run[j] = s | (e << 16);
                    if (a.sec && e - s <= kMsdRunMax) {
                        const K lo = key[j] & lo_mask;
                        bool tie = false;
                        for (uint32_t t = s; t < e; ++t) tie |= (t != pos) && ((sk[t] & lo_mask) == lo);
                        if (tie) {
                            uint32_t row = val[j];
                            if (row >= a.n) {  // never for a permutation of [0, n)
                                atomicOr(a.err, ERR_BAD_INDEX);
                                row = 0;
                            }
                            ssec[pos] = sec_image(a.sec, a.sec_dtype, row, a.invert != 0);
                        }
                    }
                }
            }
        }
        if (fix) {
            __syncthreads();
    #pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if (run[j] == 0) continue;
                const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
                const uint32_t s = run[j] & 0xffffu, e = run[j] >> 16;
                const K lo = key[j] & lo_mask;
                if (e - s > kMsdRunMax) {
                    // a long run: fine if it already is in order (e.g. equal
                    // keys of a one-key sort); otherwise see below
                    if (pos > s) {
                        const K plo = sk[pos - 1] & lo_mask;
                        if (plo > lo || (plo == lo && a.sec)) misc[0] = 1;
                    }
                    continue;
                }
                uint32_t r = 0;
                bool have_sec = false;
                uint64_t sc = 0;
                for (uint32_t t = s; t < e; ++t) {
                    const K tlo = sk[t] & lo_mask;
                    bool less = tlo < lo;
                    if (tlo == lo && t != pos) {
                        if (a.sec) {
                            if (!have_sec) {
                                sc = ssec[pos];
                                have_sec = true;
                            }
                            const uint64_t tsc = ssec[t];
                            less = tsc < sc || (tsc == sc && t < pos);
                        } else {
                            less = t < pos;
                        }
                    }
                    r += less ? 1u : 0u;
                }
                newpos[j] = s + r;
            }
            __syncthreads();
            if (misc[0]) {
                // A run longer than the direct ranking handles is out of order.
                // With a second key that needs key 1 for every row: the plan
                // fails.  With one key the chunk is finished in shared memory:
                // LSD passes over the varying low digits, then the high ones
                // again (every pass is stable, so ties keep their row order).
                if (a.sec) {
                    if (tid == 0) atomicOr(fail_word, 1u);
                    return;
                }
                for (int dg = 0; dg < KBITS / 8; ++dg) {
                    const uint32_t shift = 8u * dg;
                    if (((vary >> shift) & 0xff) == 0) continue;
                    local_pass<K, THREADS, ITEMS, MATCH>(
                        key, val, [shift](K k) { return (uint32_t)(k >> shift) & 0xffu; }, ia, sk, sv, wcnt, wsum,
                        a.err);
                }
    #pragma unroll
                for (int j = 0; j < ITEMS; ++j) newpos[j] = ((uint32_t)warp * ia + j) * 32 + lane;
            }
        }
    }

    // ---- output: raw sorted key 0 and the permutation
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t pos = ((uint32_t)warp * ia + j) * 32 + lane;
        if (j < (int)ia && pos < m) {
            uint64_t gp = (uint64_t)s0 + newpos[j];
            if (a.reverse) gp = a.n - 1 - gp;
            stg_stream(a.perm_out + gp, val[j]);
            if (kout) stg_stream(kout + gp, KeyOps<K>::unorder(key[j], a.dtype, a.invert != 0));
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {
// Chunks of up to CAP rows, one CTA of CAP / 8 threads each: 4096 rows (two
// CTAs per SM) or 8192 (one).
constexpr int kLocalItems = 8;
static_assert(kMsdWideCap < (1u << 16), "run bounds are packed in 16 bits");
template <typename K, uint32_t CAP, int MATCH>
struct Local {
    static constexpr int THREADS = (int)CAP / kLocalItems;
    static constexpr size_t SMEM = LocalCfg<K, THREADS, kLocalItems>::SMEM;
    static cudaError_t prepare() {
        return cudaFuncSetAttribute(k_msd_local<K, THREADS, kLocalItems, MATCH>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    }
    static void launch(const MsdLocalArgs& a, uint32_t nchunks, cudaStream_t s) {
        k_msd_local<K, THREADS, kLocalItems, MATCH><<<nchunks, THREADS, SMEM, s>>>(a);
    }
};
template <typename K, uint32_t CAP>
cudaError_t local_prepare() {
    const cudaError_t e = Local<K, CAP, 0>::prepare();
    return e == cudaSuccess ? Local<K, CAP, 1>::prepare() : e;
}
template <typename K, uint32_t CAP>
void local_launch(const MsdLocalArgs& a, uint32_t nchunks, int match, cudaStream_t s) {
    if (match) Local<K, CAP, 1>::launch(a, nchunks, s);
    else Local<K, CAP, 0>::launch(a, nchunks, s);
}
template <typename K>
void chunks_launch(const MsdChunkArgs& a, uint32_t cap, cudaStream_t s) {
    const uint32_t grid = (a.nchunks + 1 + 7) / 8;
    if (cap == kMsdWideCap) k_msd_chunks<K, kMsdWideCap><<<grid, 256, 0, s>>>(a);
    else k_msd_chunks<K, kMsdCap><<<grid, 256, 0, s>>>(a);
}

int sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}
}  // namespace

cudaError_t prepare_msd_kernels() {
    cudaError_t e = local_prepare<uint64_t, kMsdCap>();
    if (e == cudaSuccess) e = local_prepare<uint64_t, kMsdWideCap>();
    if (e == cudaSuccess) e = local_prepare<uint32_t, kMsdCap>();
    if (e == cudaSuccess) e = local_prepare<uint32_t, kMsdWideCap>();
    return e;
}

cudaError_t msd_hist(const MsdHistArgs& a, int width, cudaStream_t s) {
    const uint64_t want = (a.n + 511) / 512;
    const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(want, (uint64_t)sm_count() * 4));
    if (width == 8) k_msd_hist<uint64_t><<<grid, 512, 0, s>>>(a);
    else k_msd_hist<uint32_t><<<grid, 512, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t msd_scan(const MsdHistArgs& a, int width, uint32_t* offs, uint32_t cap, uint32_t* flag, uint32_t* deep,
                     cudaStream_t s) {
    if (width == 8) k_msd_scan<uint64_t><<<1, kScanThreads, 0, s>>>(a, offs, cap, flag, deep);
    else k_msd_scan<uint32_t><<<1, kScanThreads, 0, s>>>(a, offs, cap, flag, deep);
    return cudaGetLastError();
}

cudaError_t msd_chunks(const MsdChunkArgs& a, int width, cudaStream_t s, uint32_t cap) {
    if (width == 8) chunks_launch<uint64_t>(a, cap, s);
    else chunks_launch<uint32_t>(a, cap, s);
    return cudaGetLastError();
}

cudaError_t msd_local(const MsdLocalArgs& a, int width, uint32_t nchunks, int match, cudaStream_t s, uint32_t cap) {
    if (nchunks == 0) return cudaSuccess;
    if (cap == kMsdWideCap) {
        if (width == 8) local_launch<uint64_t, kMsdWideCap>(a, nchunks, match, s);
        else local_launch<uint32_t, kMsdWideCap>(a, nchunks, match, s);
    } else {
        if (width == 8) local_launch<uint64_t, kMsdCap>(a, nchunks, match, s);
        else local_launch<uint32_t, kMsdCap>(a, nchunks, match, s);
    }
    return cudaGetLastError();
}

}  // namespace vdf
