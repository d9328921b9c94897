// gp_scan.cuh -- carry (or borrow) propagation of multi-limb additions as a
// parallel prefix over (generate, propagate) pairs.
//
// A group of limbs generates a carry out (g) or passes a carry in through (p);
// groups compose associatively, so a carry chain of any length is a scan.
// Used by the signed add of the Chudnovsky merge and by the big-integer
// add/subtract kernels. Reference counterpart: the sequential carry loops of
// add_mag / sub_mag (src/bignum.cpp:63-104).
#pragma once
#include "gl.cuh"

namespace b2m {

struct GP {
    u32 g, p;
};
__device__ __forceinline__ GP gp_then(GP lo, GP hi) { return {hi.g | (hi.p & lo.g), hi.p & lo.p}; }

// One limb's pair, of a + b or (sub) a - b.
__device__ __forceinline__ GP limb_gp(u32 a, u32 b, int sub) {
    if (!sub) {
        const u64 s = (u64)a + b;
        return {(u32)(s >> 32), (u32)((u32)s == 0xFFFFFFFFu)};
    }
    return {(u32)(a < b), (u32)(a == b)};
}

constexpr int ADD_LPT = 8;  // limbs per thread

// Exclusive block scan of GP (low threads first). blockDim multiple of 32.
// A warp's carry chain is an integer addition: with G the lanes that generate
// and P those that only propagate, the carries into the lanes are the carries
// of (G | P) + G, that is P ^ ((G | P) + G [+ 1 with a carry in]). The warps'
// aggregates go the same way, by every warp: one barrier, no loop over lanes
// or warps. Callers synchronise before writing `ws` again.
__device__ __forceinline__ GP block_scan_gp(GP v, GP* ws, GP* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const u32 G = __ballot_sync(0xFFFFFFFFu, v.g != 0), P = __ballot_sync(0xFFFFFFFFu, v.p && !v.g);
    const u64 s0 = (u64)(G | P) + G;
    if (lane == 0) {
        const u32 c0 = (u32)(s0 >> 32), c1 = (u32)((s0 + 1) >> 32);
        ws[warp] = {c0, c1 & ~c0};
    }
    __syncthreads();
    const GP w = lane < nw ? ws[lane] : GP{0, 0};
    const u32 WG = __ballot_sync(0xFFFFFFFFu, w.g != 0), WP = __ballot_sync(0xFFFFFFFFu, w.p != 0);
    const u64 t0 = (u64)(WG | WP) + WG, t1 = t0 + 1;
    const u32 o0 = (u32)(t0 >> nw) & 1, o1 = (u32)(t1 >> nw) & 1;
    *total = {o0, o1 & ~o0};
    // carry into this warp, then into this lane, for a block carry-in of 0 and 1
    const u32 w0 = ((WP ^ (u32)t0) >> warp) & 1, w1 = ((WP ^ (u32)t1) >> warp) & 1;
    const u32 c0 = ((P ^ (u32)(s0 + w0)) >> lane) & 1, c1 = ((P ^ (u32)(s0 + w1)) >> lane) & 1;
    return {c0, c1 & ~c0};
}

}  // namespace b2m
