// school.cuh -- schoolbook product of two small u32-limb numbers.
//
// A schoolbook product costs about 4.5 instructions per limb multiply-add, so
// for the smallest products (rns_small.cu) it is cheaper than the transforms.
// Reference counterpart: mul_schoolbook (src/bignum.cpp:125-143), the same
// column products, here with every column sum of a thread's four columns
// accumulated in 96 bits by one carry chain per multiply-add, and the carries
// resolved by a scan of carry functions (carry.cuh).
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

// Limits of school_product: columns (na + nb), and its shared memory in words
// per product: both operands (b padded by up to seven words), and from W > 1
// warps three words of every column sum of each.
constexpr int SCHOOL_MAX_COLS = 128, SCHOOL_WARPS_CTA = 4, SCHOOL_THREADS = 32 * SCHOOL_WARPS_CTA;
template <int W>
constexpr int SCHOOL_SMEM_WORDS = SCHOOL_MAX_COLS + 12 + (W > 1 ? 3 * SCHOOL_MAX_COLS * W : 0);

// Exclusive scan of carry functions over a warp (nothing valid on lane 0).
__device__ __forceinline__ CState warp_scan_carry(CState st, int lane) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const CState o = cs_shfl_up(st, off);
        if (lane >= off) st = cs_then(o, st);
    }
    return cs_shfl_up(st, 1);
}

// out[0, na + nb) = a * b by W warps (one, or the whole block); returns its
// trimmed length, on lane 0 of each warp. `smem`: SCHOOL_SMEM_WORDS<W> words
// of the product; `st`, `s_top`: one per warp, and one, of the block (W > 1).
//
// Column sums: lane l takes the four columns at 4l and warp w a W-th of the
// range of i (one product alone on one warp stepped through up to 128
// dependent iterations); terms outside a lane's own range read b as zero, so
// the loop is warp-uniform. Window w[c] = b[k0 + c - i] slides down a limb a
// step.
template <int W>
static __device__ __forceinline__ unsigned long long school_product(const u32* a, int la, const u32* b, int lb, u32* out,
                                                                    u32* smem, CState* st, unsigned long long* s_top) {
    constexpr int T = 32 * W;
    const int t = threadIdx.x % T, lane = t & 31, warp = t >> 5, nc = la + lb;
    // b is stored as four interleaved quarter arrays, b[j] at (j & 3) * qb +
    // (j >> 2), so that lanes reading b[k0 + c - i] with k0 = 4 * lane read
    // consecutive words.
    const int qb = (lb + 3) / 4 + 1;
    u32* sa = smem;
    u32* sb = sa + la;
    u32* cs = sb + 4 * qb;  // warp p's column sums: cs[(3 p + word) * nc + column]
    for (int i = t; i < la; i += T) sa[i] = a[i];
    for (int j = t; j < lb; j += T) sb[(j & 3) * qb + (j >> 2)] = b[j];
    if (W > 1 && t == 0) *s_top = 0;
    if constexpr (W > 1) __syncthreads();
    else __syncwarp();

    u32 lo[4] = {0, 0, 0, 0}, mid[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};
    {
        const int k0 = 4 * lane, per = (la + W - 1) / W;
        const int i0 = warp * per, i1 = i0 + per < la ? i0 + per : la;
        u32 w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int j = k0 + c - i0;
            w[c] = (j >= 0 && j < lb) ? sb[(j & 3) * qb + (j >> 2)] : 0u;
        }
        for (int i = i0; i < i1; ++i) {
            const u32 x = sa[i];
#pragma unroll
            for (int c = 0; c < 4; ++c) mac96(lo[c], mid[c], hi[c], x, w[c]);
            w[3] = w[2];
            w[2] = w[1];
            w[1] = w[0];
            const int j = k0 - i - 1;
            w[0] = (j >= 0 && j < lb) ? sb[(j & 3) * qb + (j >> 2)] : 0u;
        }
    }

    // Carries: a thread owns CPT >= 2 consecutive columns, so that a carry in
    // (< 2^45) changes a range's carry out by at most one; columns from nc on
    // are zero.
    constexpr int CPT = W > 1 ? 2 : 4;
    const int k_beg = CPT * t;
    u32 limb[CPT];
    u64 carry = 0;
    if constexpr (W > 1) {
        u32* c0 = cs + 3 * warp * nc + 4 * lane;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (4 * lane + c < nc) {
                c0[c] = lo[c];
                c0[nc + c] = mid[c];
                c0[2 * nc + c] = hi[c];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
        u64 s0 = 0, s1 = 0, s2 = 0;
        if constexpr (W > 1) {
            if (k_beg + c < nc)
                for (int p = 0; p < W; ++p) {
                    const u32* c0 = cs + 3 * p * nc + k_beg + c;
                    s0 += c0[0];
                    s1 += c0[nc];
                    s2 += c0[2 * nc];
                }
        } else {
            s0 = lo[c], s1 = mid[c], s2 = hi[c];
        }
        s0 += carry;  // carry < 2^45: column sums are below 2^76
        limb[c] = (u32)s0;
        carry = (s0 >> 32) + s1 + (s2 << 32);
    }
    const CState f = group_state<CPT>(limb, carry);
    bool has = lane > 0;
    CState ex;
    if constexpr (W > 1) {
        CState agg;
        ex = block_scan_carry(f, &has, &agg, st);
    } else {
        ex = warp_scan_carry(f, lane);
    }
    group_add_carry<CPT>(limb, has ? cs_eval(ex, 0) : 0);
    unsigned top = 0;
#pragma unroll
    for (int c = 0; c < CPT; ++c) {
        if (k_beg + c < nc) {
            out[k_beg + c] = limb[c];
            if (limb[c]) top = k_beg + c + 1;
        }
    }
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    if constexpr (W > 1) {
        if (lane == 0 && top) atomicMax(s_top, (unsigned long long)top);
        __syncthreads();
        return *s_top;
    }
    return top;
}

}  // namespace b2m
