// vdf_count.cuh -- pieces of the counting sort of a few thousand rows in
// shared memory (vdf_msd.cu, vdf_small.cu): warp-wide key extremes, the
// branch-free (key, position) compare, and the map from keys to bins.
#pragma once
#include "vdf_common.cuh"

namespace vdf {

// Warp-wide minimum / maximum with the 32-bit reduce instructions: 8-byte
// keys reduce their high halves first, then the low halves of the lanes that
// hold the extreme high half.
__device__ __forceinline__ uint32_t warp_min(uint32_t x) { return __reduce_min_sync(0xffffffffu, x); }
__device__ __forceinline__ uint32_t warp_max(uint32_t x) { return __reduce_max_sync(0xffffffffu, x); }
__device__ __forceinline__ uint64_t warp_min(uint64_t x) {
    const uint32_t hi = __reduce_min_sync(0xffffffffu, (uint32_t)(x >> 32));
    const uint32_t lo = __reduce_min_sync(0xffffffffu, (uint32_t)(x >> 32) == hi ? (uint32_t)x : 0xffffffffu);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ uint64_t warp_max(uint64_t x) {
    const uint32_t hi = __reduce_max_sync(0xffffffffu, (uint32_t)(x >> 32));
    const uint32_t lo = __reduce_max_sync(0xffffffffu, (uint32_t)(x >> 32) == hi ? (uint32_t)x : 0u);
    return ((uint64_t)hi << 32) | lo;
}

// 1 when (key ak, position ao) comes before (bk, bo): the borrow of one
// multi-word subtraction, four instructions with no branch.
__device__ __forceinline__ uint32_t row_less(uint64_t ak, uint32_t ao, uint64_t bk, uint32_t bo) {
    uint32_t r;
    asm("{\n .reg .u32 t;\n sub.cc.u32 t, %1, %2;\n subc.cc.u32 t, %3, %4;\n subc.cc.u32 t, %5, %6;\n"
        " subc.u32 %0, 0, 0;\n}"
        : "=r"(r)
        : "r"(ao), "r"(bo), "r"((uint32_t)ak), "r"((uint32_t)bk), "r"((uint32_t)(ak >> 32)), "r"((uint32_t)(bk >> 32)));
    return 0u - r;
}
__device__ __forceinline__ uint32_t row_less(uint32_t ak, uint32_t ao, uint32_t bk, uint32_t bo) {
    uint32_t r;
    asm("{\n .reg .u32 t;\n sub.cc.u32 t, %1, %2;\n subc.cc.u32 t, %3, %4;\n subc.u32 %0, 0, 0;\n}"
        : "=r"(r)
        : "r"(ao), "r"(bo), "r"(ak), "r"(bk));
    return 0u - r;
}

// A monotone map of the keys in [lo, hi] to bins [0, NB): a 32-bit window of
// key - lo (all of it when the range fits), scaled by NB / range with one
// high multiply, so that spread keys fill all NB bins evenly whatever the
// range.  The scale is rounded down by more than its float error, so the
// largest window stays below NB.
template <typename K, int NB>
struct BinMap {
    K lo, hi;
    uint32_t sh, mult;
    bool direct;  // fewer than NB windows: the window is the bin
    __device__ __forceinline__ void set(K l, K h) {
        lo = l;
        hi = h;
        const K range = h - l;
        uint32_t rw;
        if constexpr (sizeof(K) == 8) {
            const uint32_t top = (uint32_t)(range >> 32);
            sh = top ? 32u - __clz((int)top) : 0u;
            rw = __funnelshift_rc((uint32_t)range, top, sh);
        } else {
            sh = 0;
            rw = range;
        }
        direct = rw < (uint32_t)NB;
        mult = direct ? 0u : (uint32_t)__fdividef((float)NB * 4294967296.0f * 0.999999f, (float)rw + 1.0f);
    }
    __device__ __forceinline__ uint32_t operator()(K k) const {
        const K off = k - lo;
        uint32_t w;
        if constexpr (sizeof(K) == 8) w = __funnelshift_rc((uint32_t)off, (uint32_t)(off >> 32), sh);
        else w = off;
        // the clamp never acts on keys in [lo, hi]; it keeps the bins in
        // bounds for the rows a timed-out look-back left out of place
        return min(direct ? w : __umulhi(w, mult), (uint32_t)NB - 1u);
    }
};

}  // namespace vdf
