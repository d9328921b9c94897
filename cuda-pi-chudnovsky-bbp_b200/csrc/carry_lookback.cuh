// carry_lookback.cuh -- decoupled lookback over carry chunks, shared by the
// carry kernels of the 64-bit transform (ntt_carry.cu) and of the residue
// transforms (rns_carry.cu). Waits are bounded.
#pragma once
#include "b2m_internal.h"
#include "carry.cuh"

namespace b2m {

__device__ __forceinline__ u64 ld_acquire(const u64* p) {
    u64 v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
// Release store: the thread's earlier writes (the slot's threshold) are
// visible to any thread that reads this word with ld_acquire.
__device__ __forceinline__ void st_release(u64* p, u64 v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

constexpr int LOOKBACK_SPIN_LIMIT = 1 << 22;
constexpr u64 SLOT_CONST = 1, SLOT_INCL = 2, SLOT_AGG = 3;

__device__ __forceinline__ CState cs_shfl(CState f, int src) {
    return {__shfl_sync(0xFFFFFFFFu, f.h, src), __shfl_sync(0xFFFFFFFFu, f.t, src)};
}

// Warp 0 (all lanes): publish chunk `chunk`'s aggregate, then resolve its
// carry-in. Each round reads the slots of the 32 nearest unresolved
// predecessors at once (lane i: chunk base - i); the nearest slot holding a
// constant aggregate or an inclusive value ends the walk, the aggregates in
// front of it are composed onto it. A round with 32 thresholded aggregates
// composes them all and moves 32 chunks further back. Returns the carry-in
// on every lane; the inclusive value is published by the caller.
__device__ __forceinline__ u64 warp_lookback(LookbackSlot* slots, u32 chunk, CState agg, u32* err) {
    const int lane = threadIdx.x & 31;
    if (chunk == 0) {
        if (lane == 0) st_release(&slots[0].word, (cs_eval(agg, 0) << 2) | SLOT_INCL);
        return 0;
    }
    if (lane == 0) {
        if (agg.t != CS_NEVER) slots[chunk].agg_t = agg.t;
        st_release(&slots[chunk].word, (agg.h << 2) | (agg.t == CS_NEVER ? SLOT_CONST : SLOT_AGG));
    }
    CState acc{0, CS_NEVER};  // composition of the predecessors passed so far (nearest applied last)
    bool acc_id = true;
    long base = (long)chunk - 1;
    int spins = 0;
    while (true) {
        const long p = base - lane;
        u64 w = SLOT_INCL;  // before chunk 0: carry 0
        unsigned need;
        int f;
        while (true) {
            if (p >= 0) w = ld_acquire(&slots[p].word);
            const unsigned stop = __ballot_sync(0xFFFFFFFFu, (w & 3) == SLOT_CONST || (w & 3) == SLOT_INCL);
            const unsigned pub = __ballot_sync(0xFFFFFFFFu, (w & 3) != 0);
            f = stop ? __ffs(stop) - 1 : 31;  // lanes 0..f must be published
            need = f == 31 ? 0xFFFFFFFFu : ((2u << f) - 1);
            if ((pub & need) == need) break;
            if (++spins > LOOKBACK_SPIN_LIMIT) {  // gave up: report, use 0 and finish cleanly
                if (lane == 0) atomicOr(err, 1u);
                return 0;
            }
            __nanosleep(64);
        }
        CState mine{w >> 2, CS_NEVER};
        if ((w & 3) == SLOT_AGG) mine.t = *(volatile u64*)&slots[p].agg_t;
        const unsigned stop = __ballot_sync(0xFFFFFFFFu, (w & 3) != SLOT_AGG);
        if (stop & need) {
            // lane f is constant or inclusive: evaluate lanes f-1 .. 0 on its value
            u64 x = __shfl_sync(0xFFFFFFFFu, mine.h, f);
            for (int k = f - 1; k >= 0; --k) x = cs_eval(cs_shfl(mine, k), x);
            return acc_id ? x : cs_eval(acc, x);
        }
        // 32 thresholded aggregates: compose them (lane 31 applies first)
        CState blk = cs_shfl(mine, 31);
        for (int k = 30; k >= 0; --k) blk = cs_then(blk, cs_shfl(mine, k));
        acc = acc_id ? blk : cs_then(blk, acc);
        acc_id = false;
        if (acc.t == CS_NEVER) return acc.h;  // constant: earlier chunks cannot matter
        base -= 32;
    }
}

}  // namespace b2m
