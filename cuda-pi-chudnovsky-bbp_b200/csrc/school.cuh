// school.cuh -- schoolbook product of two small u32-limb numbers by one CTA.
//
// A schoolbook product costs about 4.5 instructions per limb multiply-add, so
// for the smallest products (rns_small.cu) it is cheaper than the transforms.
// Reference
// counterpart: mul_schoolbook (src/bignum.cpp:125-143), the same column
// products, here with every column sum of a thread's four-column block
// accumulated in 96 bits by one carry chain per multiply-add, and the carries
// resolved by a block scan of carry functions (carry.cuh).
#pragma once
#include "carry.cuh"

namespace b2m {

// (lo, mid, hi) += x * y as one 96-bit carry chain.
__device__ __forceinline__ void mac96(u32& lo, u32& mid, u32& hi, u32 x, u32 y) {
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, %2, 0;"
        : "+r"(lo), "+r"(mid), "+r"(hi)
        : "r"(x), "r"(y));
}

// Limits of school_cta: columns (na + nb) and threads, and its shared memory
// in words: both operands (b padded by up to seven words) and three words of
// every column sum, from each of the parts the terms are split into.
constexpr int SCHOOL_MAX_COLS = 256, SCHOOL_THREADS = 128, SCHOOL_WARPS_CTA = SCHOOL_THREADS / 32;
__host__ __device__ constexpr int school_parts(int nc) {
    return nc <= 128 ? SCHOOL_WARPS_CTA : SCHOOL_WARPS_CTA / 2;  // warps per block of 128 columns
}
constexpr int SCHOOL_SMEM_WORDS = SCHOOL_MAX_COLS + 12 + 3 * 128 * SCHOOL_WARPS_CTA;

// out[0, na + nb) = a * b and *out_len = its trimmed length (when out_len is
// not null), by the SCHOOL_THREADS threads of the block. `smem`:
// SCHOOL_SMEM_WORDS words; `st`: one CState per warp.
static __device__ __forceinline__ void school_cta(const u32* __restrict__ a, u64 na, const u32* __restrict__ b, u64 nb,
                                                  u32* __restrict__ out, unsigned long long* out_len, u32* smem,
                                                  CState* st, unsigned long long* s_top) {
    constexpr int T = SCHOOL_THREADS;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int la = (int)na, lb = (int)nb, nc = la + lb;
    const int parts = school_parts(nc), pstride = 3 * nc;
    // b is stored as four interleaved quarter arrays, b[j] at (j & 3) * qb +
    // (j >> 2), so that lanes reading b[k0 + c - i] with k0 = 4 * lane read
    // consecutive words.
    const int qb = (lb + 3) / 4 + 1;
    u32* sa = smem;
    u32* sb = sa + la;
    u32* cs = sb + 4 * qb;  // part p's column sums: cs[p * 3 nc + w * nc + column]
    for (int i = t; i < la; i += T) sa[i] = __ldg(a + i);
    for (int j = t; j < lb; j += T) sb[(j & 3) * qb + (j >> 2)] = __ldg(b + j);
    if (t == 0) *s_top = 0;
    __syncthreads();

    // Column sums. A warp takes a block of 128 consecutive columns, lane l the
    // four at k0 = K0 + 4l, and a part of the block's range of i (the parts
    // side by side on the block's warps: one warp alone stepped through up to
    // 128 dependent iterations); terms outside a lane's own range read b as
    // zero, so the loop is warp-uniform. Window w[c] = b[k0 + c - i] slides
    // down a limb a step.
    {
        const int part = warp % parts, K0 = 128 * (warp / parts);
        const int k0 = K0 + 4 * lane;
        const int lo_i = K0 - lb + 1 > 0 ? K0 - lb + 1 : 0;
        const int hi_i = K0 + 127 < la - 1 ? K0 + 127 : la - 1;
        const int cnt = hi_i >= lo_i ? hi_i - lo_i + 1 : 0, per = (cnt + parts - 1) / parts;
        const int i0 = lo_i + part * per, i1 = i0 + per - 1 < hi_i ? i0 + per - 1 : hi_i;
        u32 lo[4] = {0, 0, 0, 0}, mid[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
        u32 w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int j = k0 + c - i0;
            w[c] = (j >= 0 && j < lb) ? sb[(j & 3) * qb + (j >> 2)] : 0u;
        }
        for (int i = i0; i <= i1; ++i) {
            const u32 x = sa[i];
#pragma unroll
            for (int c = 0; c < 4; ++c) mac96(lo[c], mid[c], hi[c], x, w[c]);
            w[3] = w[2];
            w[2] = w[1];
            w[1] = w[0];
            const int j = k0 - i - 1;
            w[0] = (j >= 0 && j < lb) ? sb[(j & 3) * qb + (j >> 2)] : 0u;
        }
        u32* c0 = cs + part * pstride;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (k0 + c < nc) {
                c0[k0 + c] = lo[c];
                c0[nc + k0 + c] = mid[c];
                c0[2 * nc + k0 + c] = hi[c];
            }
        }
    }
    __syncthreads();

    // Carries: thread t owns two consecutive columns, so that a carry in
    // (< 2^45) changes a range's carry out by at most one. Its limbs with no
    // carry in and its carry function f(c) = h + [c >= th]. Only the last
    // non-empty range can be one limb long, and only empty ranges, whose
    // functions nothing uses, follow it.
    static_assert(2 * T >= SCHOOL_MAX_COLS, "two columns per thread");
    const int k_beg = 2 * t, n_own = k_beg + 2 <= nc ? 2 : (k_beg < nc ? 1 : 0);
    u32 limb[2] = {0, 0};
    u64 carry = 0;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (m < n_own) {
            const int k = k_beg + m;
            u64 s0 = 0, s1 = 0, s2 = 0;
            for (int p = 0; p < parts; ++p) {
                const u32* c0 = cs + p * pstride + k;
                s0 += c0[0];
                s1 += c0[nc];
                s2 += c0[2 * nc];
            }
            s0 += carry;  // carry < 2^45: column sums are below 2^76
            limb[m] = (u32)s0;
            carry = (s0 >> 32) + s1 + (s2 << 32);
        }
    }
    CState f{carry, CS_NEVER};
    const u64 dl = (u64)limb[0] | ((u64)limb[1] << 32);
    if (n_own == 2 && dl != 0) {
        const u64 tt = 0ull - dl;  // 2^64 less the two limbs
        if (tt < (1ull << 62)) f.t = tt;
    }
    bool has;
    CState agg;
    const CState ex = block_scan_carry(f, &has, &agg, st);
    u64 cin = has ? cs_eval(ex, 0) : 0;
    // Add the carry in and store; the carry out of the range is f(cin).
    unsigned long long top = 0;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        if (m < n_own) {
            const u64 s0 = (u64)limb[m] + (cin & 0xFFFFFFFFull);
            const u32 v = (u32)s0;
            cin = (cin >> 32) + (s0 >> 32);
            out[k_beg + m] = v;
            if (v) top = (unsigned long long)(k_beg + m) + 1;
        }
    }
    const unsigned any = __ballot_sync(0xFFFFFFFFu, top != 0);
    if (any && lane == 31 - __clz(any)) atomicMax(s_top, top);
    __syncthreads();
    if (t == 0 && out_len) *out_len = *s_top;
}

}  // namespace b2m
