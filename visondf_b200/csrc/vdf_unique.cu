// vdf_unique.cu -- de-duplication and left-join row matching.  In a stable
// ascending radix sort of the key column the rows of one key value form a run
// in row order: the run's first row is the key's first occurrence and its
// last row the last occurrence.
//   * k_unique_mark  marks those rows in a per-row keep mask (one pass over
//                    the sorted keys, a scatter through the permutation);
// The left join's First and Last need no order at all:
//   * k_join_insert  puts the right rows into a hash table of {key, row} slots,
//                    keeping each key's smallest (largest) row;
//   * k_join_find    looks each left key up in it.
// Aligned pairs the k-th occurrences of a key, which the sorted sides number:
//   * k_join_build   puts the right side's distinct sorted keys (the
//                    group-by's segment pass finds them) with their runs into
//                    a hash table;
//   * k_join_probe_aligned  looks each sorted left row's key up in it.
// Keys compare by their raw bits, so -0.0 and +0.0 are different keys and a
// NaN equals a NaN with the same bits, as with the reference's byte-wise
// hash lookups.
#include <cstdint>

#include "vdf_common.cuh"
#include "vdf_internal.h"

namespace vdf {
namespace {

uint32_t grid_size(uint64_t n) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint64_t want = (n + 255) / 256;
    const uint64_t cap = (uint64_t)sms * 8;
    return (uint32_t)(want < cap ? (want ? want : 1) : cap);
}

// Warp sum of a per-thread count, added once per warp.
__device__ __forceinline__ void add_count(unsigned long long* total, uint32_t mine) {
    const uint32_t w = __reduce_add_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(total, (unsigned long long)w);
}

// Marks go into a bit per row (atomicOr on 32-row words: the n/8-byte mask
// stays in L2 while the permutation scatters into it), then one coalesced
// pass expands the bits into the caller's byte mask.
template <typename T>
__global__ void __launch_bounds__(256) k_unique_mark(const T* __restrict__ sk, const uint32_t* __restrict__ perm,
                                                      uint64_t n, int last, uint32_t* __restrict__ bits,
                                                      unsigned long long* count, uint32_t* err) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t kept = 0;
    // every lane runs the same number of rounds (the warp sum needs them all)
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint64_t i = base + threadIdx.x;
        if (i < n) {
            const T k = sk[i];
            const bool mark = last ? (i + 1 == n || sk[i + 1] != k) : (i == 0 || sk[i - 1] != k);
            if (mark) {
                const uint32_t r = perm[i];
                if (r >= n) {
                    atomicOr(err, ERR_BAD_INDEX);
                } else {
                    atomicOr(&bits[r >> 5], 1u << (r & 31));
                    ++kept;
                }
            }
        }
    }
    add_count(count, kept);
}

// keep[r] = bit r; one 32-row word per thread, 32 bytes written per thread.
__global__ void __launch_bounds__(256) k_expand_bits(const uint32_t* __restrict__ bits, uint64_t n,
                                                      uint8_t* __restrict__ keep) {
    const uint64_t words = (n + 31) / 32;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const bool vec = (reinterpret_cast<uintptr_t>(keep) & 15) == 0;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += stride) {
        const uint32_t b = bits[w];
        uint32_t q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t nib = (b >> (4 * k)) & 0xfu;
            q[k] = (nib & 1u) | ((nib & 2u) << 7) | ((nib & 4u) << 14) | ((nib & 8u) << 21);
        }
        const uint64_t r0 = w * 32;
        if (vec && r0 + 32 <= n) {
            uint4* d = reinterpret_cast<uint4*>(keep + r0);
            d[0] = make_uint4(q[0], q[1], q[2], q[3]);
            d[1] = make_uint4(q[4], q[5], q[6], q[7]);
        } else {
            for (uint32_t j = 0; j < 32 && r0 + j < n; ++j) keep[r0 + j] = (uint8_t)((b >> j) & 1u);
        }
    }
}

// Hash table of the right side's distinct keys: 16-byte slots {raw key,
// run + 1 (0 = empty)}, open addressing with linear probing over a
// power-of-two capacity of at least twice the right side's rows.  The keys
// inserted are distinct, so a slot is claimed by a CAS of its row field and
// its key written after; the probe kernel runs after the build completes.
struct JoinSlot {
    unsigned long long key;
    uint32_t row1;
    uint32_t pad;
};

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    // 64-bit finaliser of MurmurHash3 (fmix64)
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}

// The slot holds the key's run index g.
template <typename T>
__global__ void __launch_bounds__(256) k_join_build(const T* __restrict__ ukeys, const uint64_t* n_groups,
                                                     JoinSlot* table, uint64_t mask, uint32_t* err) {
    const uint64_t G = *n_groups;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < G; g += stride) {
        const uint32_t row1 = (uint32_t)g + 1u;
        const unsigned long long key = (unsigned long long)ukeys[g];
        uint64_t s = mix64(key) & mask;
        bool placed = false;
        for (uint64_t t = 0; t <= mask; ++t) {  // at most one lap of the table
            if (atomicCAS(&table[s].row1, 0u, row1) == 0u) {
                table[s].key = key;
                placed = true;
                break;
            }
            s = (s + 1) & mask;
        }
        if (!placed) atomicOr(err, ERR_BAD_INDEX);
    }
}

// First / Last: open addressing over buckets of 32 bytes, filled slot by slot
// and bucket after bucket, so that a probe is one 32-byte load and an empty
// slot ends the search: four slots {key, row} of 4-byte keys (all ones:
// empty), or two slots {key, row + 1} of 8-byte keys (zero: empty).  A slot is
// claimed by one compare-and-swap of the whole slot
// and its key never changes; its row only moves towards the first (last) one.
// What bounds both kernels is random accesses (about 60 G per second): a
// table built from the sorted right side and probed slot by slot took 0.91 ms
// for 50M left rows against 5M right ones and 0.6 ms to sort and build; this
// one takes 0.85 ms and 0.19 ms.  Slots of a hash tag and a row, checked
// against the right rows' keys, halve the table but double the accesses (1.33
// ms).
template <typename T> struct JoinTable;
template <> struct JoinTable<uint32_t> {
    static constexpr int SLOTS = 4;  // per bucket
    static constexpr int EMPTY_BYTE = 0xff;
    static constexpr size_t SLOT_BYTES = 8;
    unsigned long long* t;
    static __device__ __forceinline__ unsigned long long pack(uint32_t key, uint32_t row) {
        return ((unsigned long long)key << 32) | row;
    }
    // Offers (key, row) to slot s: true when the slot holds the key now.
    template <bool LAST> __device__ __forceinline__ bool offer(uint64_t s, uint32_t key, uint32_t row) const {
        const unsigned long long mine = pack(key, row);
        unsigned long long cur = ld_relaxed_u64(reinterpret_cast<const uint64_t*>(t + s));
        if (cur == ~0ull) cur = atomicCAS(t + s, ~0ull, mine);
        if (cur == ~0ull) return true;
        if ((uint32_t)(cur >> 32) != key) return false;
        if (LAST ? (uint32_t)cur < row : (uint32_t)cur > row) {
            if (LAST) atomicMax(t + s, mine);
            else atomicMin(t + s, mine);
        }
        return true;
    }
    // Looks key up in a loaded bucket: its row, -1 (not here, go on) or -2 (an
    // empty slot: nowhere).
    static __device__ __forceinline__ int64_t find(const unsigned long long (&b)[4], uint32_t key) {
        int64_t r = -1;
#pragma unroll
        for (int i = 3; i >= 0; --i) {
            if (b[i] == ~0ull) r = -2;
            else if ((uint32_t)(b[i] >> 32) == key) r = (uint32_t)b[i];
        }
        return r;
    }
};
template <> struct JoinTable<unsigned long long> {
    static constexpr int SLOTS = 2;
    static constexpr int EMPTY_BYTE = 0;
    static constexpr size_t SLOT_BYTES = 16;
    unsigned long long* t;
    template <bool LAST> __device__ __forceinline__ bool offer(uint64_t s, unsigned long long key, uint32_t row) const {
        unsigned long long* slot = t + 2 * s;
        unsigned long long k, r;
        asm volatile("{\n .reg .b128 v;\n ld.relaxed.gpu.global.b128 v, [%2];\n mov.b128 {%0, %1}, v;\n}"
                     : "=l"(k), "=l"(r) : "l"(slot) : "memory");
        if (r == 0)
            asm volatile(
                "{\n .reg .b128 c, n, o;\n mov.b128 c, {%4, %4};\n mov.b128 n, {%2, %3};\n"
                " atom.relaxed.gpu.global.cas.b128 o, [%5], c, n;\n mov.b128 {%0, %1}, o;\n}"
                : "=l"(k), "=l"(r)
                : "l"(key), "l"((unsigned long long)row + 1), "l"(0ull), "l"(slot)
                : "memory");
        if (r == 0) return true;
        if (k != key) return false;
        uint32_t* row1 = reinterpret_cast<uint32_t*>(slot + 1);
        if (LAST ? (uint32_t)r < row + 1 : (uint32_t)r > row + 1) {
            if (LAST) atomicMax(row1, row + 1);
            else atomicMin(row1, row + 1);
        }
        return true;
    }
    static __device__ __forceinline__ int64_t find(const unsigned long long (&b)[4], unsigned long long key) {
        if (b[1] == 0) return -2;
        if (b[0] == key) return (int64_t)b[1] - 1;
        if (b[3] == 0) return -2;
        return b[2] == key ? (int64_t)b[3] - 1 : -1;
    }
};

template <typename T, bool LAST>
__global__ void __launch_bounds__(256) k_join_insert(const T* __restrict__ right, uint64_t n, JoinTable<T> table,
                                                      uint64_t buckets, uint32_t* err) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t cap = buckets * JoinTable<T>::SLOTS;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        // rows in the order that settles a repeated key's slot early: most
        // repeats then find the slot as it should be and write nothing
        const uint32_t row = (uint32_t)(LAST ? n - 1 - i : i);
        const T key = right[row];
        uint64_t s = __umul64hi(mix64((uint64_t)key), buckets) * JoinTable<T>::SLOTS;
        bool placed = false;
        for (uint64_t t = 0; t < cap && !placed; ++t) {  // at most one lap of the table
            placed = table.template offer<LAST>(s, key, row);
            if (++s == cap) s = 0;
        }
        if (!placed) atomicOr(err, ERR_BAD_INDEX);
    }
}

// Four left rows per thread, their buckets all loaded before the first is
// looked at.
template <typename T>
__global__ void __launch_bounds__(256) k_join_find(const T* __restrict__ left, uint64_t n_left, JoinTable<T> table,
                                                    uint64_t buckets, uint32_t* __restrict__ match,
                                                    unsigned long long* matched) {
    constexpr int R = 4;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t found = 0;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n_left; base += R * stride) {
        T x[R];
        uint64_t b[R];
        unsigned long long v[R][4];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint64_t i = base + r * stride + threadIdx.x;
            x[r] = i < n_left ? ldg_stream(left + i) : T(0);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            b[r] = __umul64hi(mix64((uint64_t)x[r]), buckets);
            ld_rand32(table.t + 4 * b[r], v[r]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint64_t i = base + r * stride + threadIdx.x;
            int64_t m = JoinTable<T>::find(v[r], x[r]);
            for (uint64_t t = 1; m == -1 && t < buckets; ++t) {  // half the slots or more are empty
                if (++b[r] == buckets) b[r] = 0;
                unsigned long long w[4];
                ld_rand32(table.t + 4 * b[r], w);
                m = JoinTable<T>::find(w, x[r]);
            }
            if (i < n_left) {
                stg_stream(match + i, m >= 0 ? (uint32_t)m : 0xffffffffu);
                found += m >= 0 ? 1u : 0u;
            }
        }
    }
    add_count(matched, found);
}

// Aligned matching over the left side's stable sort: sorted left row i is
// occurrence r = i - (start of its run) of its key; it takes the right row
// at position r of that key's run in the right side's sort, if the run is
// long enough.  Results are scattered back through the left permutation.
template <typename T>
__global__ void __launch_bounds__(256) k_join_probe_aligned(
    const T* __restrict__ sorted_l, const uint32_t* __restrict__ perm_l, const uint32_t* __restrict__ group_l,
    const uint32_t* __restrict__ gstart_l, uint64_t n_left, const JoinSlot* __restrict__ table, uint64_t mask,
    const uint32_t* __restrict__ gstart_r, const uint64_t* n_groups_r, const uint32_t* __restrict__ perm_r,
    uint64_t n_right, uint32_t* __restrict__ match, unsigned long long* matched, uint32_t* err) {
    const uint64_t Gr = *n_groups_r;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t found = 0;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n_left; base += stride) {
        const uint64_t i = base + threadIdx.x;
        if (i >= n_left) continue;
        const unsigned long long x = (unsigned long long)sorted_l[i];
        const uint32_t rank = (uint32_t)i - gstart_l[group_l[i]];
        uint64_t s = mix64(x) & mask;
        uint32_t m = 0xffffffffu;
        for (uint64_t t = 0; t <= mask; ++t) {
            const ulonglong2 v = ld_rand16(reinterpret_cast<const ulonglong2*>(table + s));
            const uint32_t g1 = (uint32_t)v.y;
            if (g1 == 0u) break;
            if (v.x == x) {
                const uint64_t g = g1 - 1u;
                const uint64_t start = g < Gr ? gstart_r[g] : n_right;
                const uint64_t end = g + 1 < Gr ? gstart_r[g + 1] : n_right;
                if (start + rank < end) {
                    m = perm_r[start + rank];
                    ++found;
                }
                break;
            }
            s = (s + 1) & mask;
        }
        const uint32_t r = perm_l[i];
        if (r >= n_left) atomicOr(err, ERR_BAD_INDEX);
        else match[r] = m;
    }
    add_count(matched, found);
}

}  // namespace

size_t unique_workspace_bytes(uint64_t n) { return ((n + 31) / 32) * 4; }

cudaError_t run_unique_mark(const void* sorted_keys, int width, const uint32_t* perm, uint64_t n, int last,
                            uint8_t* keep, unsigned long long* count, uint32_t* bits, uint32_t* err,
                            cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(bits, 0, unique_workspace_bytes(n), s);
    if (e != cudaSuccess) return e;
    const uint32_t grid = grid_size(n);
    if (width == 8)
        k_unique_mark<unsigned long long><<<grid, 256, 0, s>>>(
            static_cast<const unsigned long long*>(sorted_keys), perm, n, last, bits, count, err);
    else
        k_unique_mark<uint32_t><<<grid, 256, 0, s>>>(static_cast<const uint32_t*>(sorted_keys), perm, n, last, bits,
                                                     count, err);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_expand_bits<<<grid_size((n + 31) / 32), 256, 0, s>>>(bits, n, keep);
    return cudaGetLastError();
}

uint64_t join_table_slots(uint64_t n_right) {
    uint64_t cap = 1024;
    while (cap < 2 * n_right) cap <<= 1;
    return cap;
}
size_t join_workspace_bytes(uint64_t n_right) { return join_table_slots(n_right) * sizeof(JoinSlot); }

cudaError_t run_join_build(const void* ukeys, int width, const uint64_t* n_groups, uint64_t n_right, void* table_ws,
                           uint32_t* err, cudaStream_t s) {
    const uint64_t slots = join_table_slots(n_right);
    JoinSlot* table = static_cast<JoinSlot*>(table_ws);
    cudaError_t e = cudaMemsetAsync(table, 0, slots * sizeof(JoinSlot), s);
    if (e != cudaSuccess || n_right == 0) return e;
    if (width == 8)
        k_join_build<unsigned long long><<<grid_size(n_right), 256, 0, s>>>(
            static_cast<const unsigned long long*>(ukeys), n_groups, table, slots - 1, err);
    else
        k_join_build<uint32_t><<<grid_size(n_right), 256, 0, s>>>(static_cast<const uint32_t*>(ukeys), n_groups, table,
                                                                   slots - 1, err);
    return cudaGetLastError();
}

// Slots per right row: two of 4-byte keys and three of 8-byte keys, whose
// buckets hold half as many.  50M left rows against 5M right ones, 8-byte
// keys, insert + find: 1.30 / 1.03 / 1.05 ms at 2 / 3 / 4 slots; 30M against
// 15M, 4-byte keys: 1.04 / 1.28 / 1.39 ms.
template <typename T>
static uint64_t join_buckets(uint64_t n_right) {
    return (sizeof(T) == 8 ? 3 : 2) * n_right / JoinTable<T>::SLOTS + 2;
}
size_t join_rows_workspace_bytes(uint64_t n_right) { return join_buckets<unsigned long long>(n_right) * 32; }

template <typename T>
static cudaError_t join_rows(const T* left, uint64_t n_left, const T* right, uint64_t n_right, bool last,
                             unsigned long long* ws, uint32_t* match, unsigned long long* matched, uint32_t* err,
                             cudaStream_t s) {
    const uint64_t buckets = join_buckets<T>(n_right);
    const JoinTable<T> table{ws};
    cudaError_t e = cudaMemsetAsync(ws, JoinTable<T>::EMPTY_BYTE, buckets * 32, s);
    if (e != cudaSuccess) return e;
    if (last) k_join_insert<T, true><<<grid_size(n_right), 256, 0, s>>>(right, n_right, table, buckets, err);
    else k_join_insert<T, false><<<grid_size(n_right), 256, 0, s>>>(right, n_right, table, buckets, err);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_join_find<T><<<grid_size((n_left + 3) / 4), 256, 0, s>>>(left, n_left, table, buckets, match, matched);
    return cudaGetLastError();
}

cudaError_t run_join_rows(const void* left, uint64_t n_left, const void* right, uint64_t n_right, int width, bool last,
                          void* table_ws, uint32_t* match, unsigned long long* matched, uint32_t* err, cudaStream_t s) {
    if (n_left == 0 || n_right == 0) return cudaSuccess;
    unsigned long long* table = static_cast<unsigned long long*>(table_ws);
    if (width == 8)
        return join_rows(static_cast<const unsigned long long*>(left), n_left,
                         static_cast<const unsigned long long*>(right), n_right, last, table, match, matched, err, s);
    return join_rows(static_cast<const uint32_t*>(left), n_left, static_cast<const uint32_t*>(right), n_right, last,
                     table, match, matched, err, s);
}

cudaError_t run_join_probe_aligned(const void* sorted_left, int width, const uint32_t* perm_left,
                                   const uint32_t* group_left, const uint32_t* gstart_left, uint64_t n_left,
                                   const void* table_ws, const uint32_t* gstart_right, const uint64_t* n_groups_right,
                                   const uint32_t* perm_right, uint64_t n_right, uint32_t* match,
                                   unsigned long long* matched, uint32_t* err, cudaStream_t s) {
    if (n_left == 0) return cudaSuccess;
    const uint64_t mask = join_table_slots(n_right) - 1;
    const JoinSlot* table = static_cast<const JoinSlot*>(table_ws);
    const uint32_t grid = grid_size(n_left);
    if (width == 8)
        k_join_probe_aligned<unsigned long long><<<grid, 256, 0, s>>>(
            static_cast<const unsigned long long*>(sorted_left), perm_left, group_left, gstart_left, n_left, table,
            mask, gstart_right, n_groups_right, perm_right, n_right, match, matched, err);
    else
        k_join_probe_aligned<uint32_t><<<grid, 256, 0, s>>>(
            static_cast<const uint32_t*>(sorted_left), perm_left, group_left, gstart_left, n_left, table, mask,
            gstart_right, n_groups_right, perm_right, n_right, match, matched, err);
    return cudaGetLastError();
}

}  // namespace vdf
