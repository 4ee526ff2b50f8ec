// vdf_dict.cuh -- the collection tables of the dictionary plans (vdf_dict.cu,
// vdf_dictagg.cu): insertion into a CTA's shared-memory table and the merge
// of such a table into the global one.
#pragma once
#include "vdf_common.cuh"
#include "vdf_internal.h"

namespace vdf {

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) { return *static_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ unsigned long long ld_volatile(const unsigned long long* p) {
    return *static_cast<const volatile unsigned long long*>(p);
}

// Adds `add` rows of value x to a CTA's open-addressing table in shared
// memory (keys / counts / states).  A new value takes the next index of
// *distinct; more than kDictMax of them, a full table or a wait that gives up
// set *over.  Returns false when the value was not recorded.  The fences are
// CTA-scoped: only the CTA's own threads read the table.
__device__ inline bool dict_add(unsigned long long* keys, uint32_t* cnt, uint32_t* st, uint32_t mask, unsigned long long x,
                         uint32_t add, uint32_t limit, uint32_t* distinct, uint32_t* over, uint32_t* err) {
    uint32_t s = dict_hash(x) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe) {
        // too many values already: the table is not filled further.  Checked
        // at every step, before a slot is claimed: with many distinct keys all
        // the CTA's threads insert at once, and without it they would fill
        // the table and probe it end to end after the plan has failed.
        if (ld_volatile(over)) return false;
        uint32_t state = ld_volatile(st + s);
        if (state == 0) {
            state = atomicCAS(st + s, 0u, 1u);
            if (state == 0) {  // this thread owns the slot: key, then count, then publish
                keys[s] = x;
                atomicAdd(cnt + s, add);
                __threadfence_block();
                atomicExch(st + s, 2u);
                if (atomicAdd(distinct, 1u) >= kDictMax) atomicOr(over, 1u);
                return true;
            }
        }
        uint32_t spins = 0;
        while (state != 2) {  // another thread is writing the slot's key
            if (ld_volatile(over)) return false;
            if (++spins > limit) {
                atomicOr(err, ERR_LOOKBACK_TIMEOUT);
                atomicOr(over, 1u);
                return false;
            }
            if (spins > 16) __nanosleep(32);
            state = ld_volatile(st + s);
        }
        __threadfence_block();
        if (ld_volatile(keys + s) == x) {
            atomicAdd(cnt + s, add);
            return true;
        }
        s = (s + 1) & mask;
    }
    atomicOr(over, 1u);  // never with the planned sizes: more values than slots
    return false;
}

// Merges a CTA's table (kDictCtaSlots slots) into the global one; more than
// kDictMax values in all, or a wait that gives up, set the overflow word.
// Every thread of the CTA calls it.
__device__ inline void dict_merge(const unsigned long long* skey, const uint32_t* scnt, const uint32_t* sst,
                                  const DictArgs& a, uint32_t limit) {
    for (uint32_t s = threadIdx.x; s < kDictCtaSlots; s += blockDim.x) {
        if (sst[s] != 2 || ld_volatile(a.overflow)) continue;
        DictSlot* t = a.table;
        uint32_t g = dict_hash(skey[s]) & (kDictSlots - 1);
        bool done = false;
        for (uint32_t probe = 0; probe < kDictSlots && !done; ++probe) {
            uint32_t state = ld_volatile(&t[g].state);
            if (state == 0) {
                state = atomicCAS(&t[g].state, 0u, 1u);
                if (state == 0) {
                    t[g].key = skey[s];
                    atomicAdd(&t[g].count, scnt[s]);
                    __threadfence();
                    atomicExch(&t[g].state, 2u);
                    if (atomicAdd(a.distinct, 1u) >= kDictMax) atomicOr(a.overflow, 1u);
                    done = true;
                    break;
                }
            }
            uint32_t spins = 0;
            while (state != 2) {
                if (++spins > limit) {
                    atomicOr(a.err, ERR_LOOKBACK_TIMEOUT);
                    atomicOr(a.overflow, 1u);
                    return;
                }
                if (spins > 16) __nanosleep(32);
                state = ld_volatile(&t[g].state);
            }
            __threadfence();
            if (ld_volatile(&t[g].key) == skey[s]) {
                atomicAdd(&t[g].count, scnt[s]);
                done = true;
                break;
            }
            g = (g + 1) & (kDictSlots - 1);
        }
        if (!done) atomicOr(a.overflow, 1u);
    }
}

}  // namespace vdf
