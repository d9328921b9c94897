// rns_small.cu -- whole products of up to 2^12 32-bit points in one launch.
//
// A product is a cluster of three blocks, one per prime: each loads both
// operands, runs both forward transforms side by side (the twiddle loads
// serve both), the pointwise product and the inverse in its own shared
// memory, and leaves its CRT terms there; each block then reads a third of
// all terms through distributed shared memory, forms those coefficients and
// resolves their carries with a block scan and the other blocks' aggregates.
// Products of at most 128 limbs are
// schoolbook columns (school.cuh).
//
// What bounds it: latency. A 2048 x 2048-limb product by one block in the
// 64-bit field took 48 us on one SM; here three SMs share it.
//
// Reference counterpart: mul_ntt_cuda (src/ntt_cuda.cu:179-243), and
// mul_schoolbook (src/bignum.cpp:125-143).
#include <cooperative_groups.h>

#include "b2m_context.h"
#include "carry.cuh"
#include "publish.cuh"
#include "rns_crt.cuh"
#include "rns_kernels.cuh"
#include "school.cuh"

namespace b2m {

namespace cg = cooperative_groups;

// Register stages of a 2^M-point transform: radix 2^l[s], 2^LE points of each
// operand per thread.
template <int M>
struct SmallCfg;
template <>
struct SmallCfg<8> {
    static constexpr int LE = 3, NS = 3, l[3] = {3, 3, 2};
};
template <>
struct SmallCfg<9> {
    static constexpr int LE = 3, NS = 3, l[3] = {3, 3, 3};
};
template <>
struct SmallCfg<10> {
    static constexpr int LE = 4, NS = 3, l[3] = {4, 3, 3};
};
template <>
struct SmallCfg<11> {
    static constexpr int LE = 4, NS = 3, l[3] = {4, 4, 3};
};
template <>
struct SmallCfg<12> {
    static constexpr int LE = 4, NS = 3, l[3] = {4, 4, 4};
};

template <int M, int S>
struct SmallStage {
    using C = SmallCfg<M>;
    static constexpr int before() {
        int r = 0;
        for (int i = 0; i < S; ++i) r += C::l[i];
        return r;
    }
    static constexpr int L = C::l[S], LEV = before(), REST = M - LEV - L;
    static constexpr int T = 1 << (M - C::LE), TASKS = 1 << (C::LE - L);  // transforms per thread
    // Transform i of this thread: node and the position of its element 0.
    __device__ __forceinline__ static int node(int i) { return ((int)threadIdx.x + i * T) >> REST; }
    __device__ __forceinline__ static int pos(int i) {
        const int id = (int)threadIdx.x + i * T;
        return ((id >> REST) << (M - LEV)) + (id & ((1 << REST) - 1));
    }
};

// Shared-memory index of a position: one pad every 16.
__device__ __forceinline__ int small_pad(int p) { return p + (p >> 4); }

// Stage S of the forward transforms of both operands (pairs in shared
// memory); the last stage leaves the values in registers.
template <int M, int S, bool HZ>
__device__ __forceinline__ void small_fwd(u32* x, uint2* sp, const uint2* T, const RnsMod& m) {
    using G = SmallStage<M, S>;
    constexpr bool LAST = S + 1 == SmallCfg<M>::NS;
#pragma unroll
    for (int i = 0; i < G::TASKS; ++i) {
        u32* y = x + (i << (G::L + 1));
        const int p = G::pos(i);
        if constexpr (S > 0) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k) {
                const uint2 v = sp[small_pad(p + (k << G::REST))];
                y[2 * k] = v.x, y[2 * k + 1] = v.y;
            }
        }
        rns_dft_fwd<G::L, 2, S == 0, HZ && S == 0>(y, T, (u32)G::node(i), m);
        if constexpr (!LAST) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k)
                sp[small_pad(p + (k << G::REST))] = make_uint2(y[2 * k], y[2 * k + 1]);
        }
    }
    if constexpr (!LAST) {
        __syncthreads();
        small_fwd<M, S + 1, HZ>(x, sp, T, m);
    }
}

// Inverse stages S .. 0; values of the last forward stage's layout in x.
template <int M, int S>
__device__ __forceinline__ void small_inv(u32* x, u32* sx, const uint2* T, const RnsMod& m) {
    using G = SmallStage<M, S>;
    constexpr bool FIRST = S + 1 == SmallCfg<M>::NS;
#pragma unroll
    for (int i = 0; i < G::TASKS; ++i) {
        u32* y = x + (i << G::L);
        const int p = G::pos(i);
        if constexpr (!FIRST) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k) y[k] = sx[small_pad(p + (k << G::REST))];
        }
        rns_dft_inv<G::L, 1, S == 0>(y, T, (u32)G::node(i), m);
        if constexpr (S > 0) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k) sx[small_pad(p + (k << G::REST))] = y[k];
        }
    }
    if constexpr (S > 0) {
        __syncthreads();
        small_inv<M, S - 1>(x, sx, T, m);
    }
}

template <int M>
struct SmallShape {
    static constexpr int N = 1 << M, T = 1 << (M - SmallCfg<M>::LE), PAD = N + N / 16;
    // pairs, then the product, and one carry state per warp
    static constexpr int BYTES = PAD * 12 + T / 32 * 16;
    static constexpr int D = (N + 3 * T - 1) / (3 * T);  // digits per thread of the cluster
    static constexpr int MINB = T >= 256 ? 3 : (T >= 128 ? 6 : (SmallCfg<M>::LE == 4 ? 12 : (T == 64 ? 16 : 28)));
};

template <int M>
__global__ void __cluster_dims__(3, 1, 1) __launch_bounds__(SmallShape<M>::T, SmallShape<M>::MINB)
    k_rns_small(const RnsArgs a, u32* __restrict__ out, unsigned long long* out_len, const RnsCrt crt,
                const HostLen hl) {
    using G = SmallShape<M>;
    using C = SmallCfg<M>;
    constexpr int E = 1 << C::LE;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long s_top;
    __shared__ unsigned long long s_tops[3];
    __shared__ CState s_agg[2];  // of the blocks before this one
    const int pi = blockIdx.x % 3;
    pdl_enter();
    const u32 *la = a.a, *lb = a.b;
    u64 na = a.na, nb = a.nb;
    if (a.jobs) {
        const ProdJob& J = a.jobs[blockIdx.x / 3];
        la = J.a;
        lb = J.b;
        na = J.na;
        nb = J.nb;
        out = J.out;
        out_len = J.out_len;
    }
    uint2* sp = reinterpret_cast<uint2*>(smem);
    u32* sx = reinterpret_cast<u32*>(sp + G::PAD);
    CState* st_scan = reinterpret_cast<CState*>(sx + G::PAD);
    const RnsMod m(pi);
    const uint2* T = a.tw + (u64)pi * a.ent;
    const uint2* Ti = a.twi + (u64)pi * a.ent;
    const u32 np4 = 2 * m.np2;
    u32 x[2 * E];
    {
        using S0 = SmallStage<M, 0>;
        const bool hz = 2 * na <= G::N && 2 * nb <= G::N;
#pragma unroll
        for (int i = 0; i < S0::TASKS; ++i)
#pragma unroll
            for (int k = 0; k < (1 << S0::L); ++k) {
                u32 va = 0, vb = 0;
                if (!hz || k < (1 << S0::L) / 2) {
                    const u32 j = S0::pos(i) + (k << S0::REST);
                    va = j < na ? __ldg(la + j) : 0u;
                    vb = j < nb ? __ldg(lb + j) : 0u;
                }
                u32* y = x + (i << (S0::L + 1)) + 2 * k;
                y[0] = __viaddmin_u32(va, np4, va);
                y[1] = __viaddmin_u32(vb, np4, vb);
            }
        if (threadIdx.x == 0) s_top = 0;
        if (hz) small_fwd<M, 0, true>(x, sp, T, m);
        else small_fwd<M, 0, false>(x, sp, T, m);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) x[k] = rns_redc((u64)rns_red2(x[2 * k], m) * rns_red2(x[2 * k + 1], m), pi, m);
    small_inv<M, C::NS - 1>(x, sx, Ti, m);
    {
        // CRT terms, canonical
        using S0 = SmallStage<M, 0>;
        const uint2 kap = pi == 0 ? crt.kap[0] : (pi == 1 ? crt.kap[1] : crt.kap[2]);
#pragma unroll
        for (int i = 0; i < S0::TASKS; ++i)
#pragma unroll
            for (int k = 0; k < (1 << S0::L); ++k) {
                const u32 v = rns_mul(x[(i << S0::L) + k], kap, m);
                sx[small_pad(S0::pos(i) + (k << S0::REST))] = __viaddmin_u32(v, 0u - m.p, v);
            }
    }
    // The cluster's 3T threads take G::D consecutive digits each, the block of
    // rank r those from r T D on (digits past N are zero): a block scan, then
    // the aggregates of the blocks before it, pushed by them.
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const u32* y0 = cluster.map_shared_rank(sx, 0);
    const u32* y1 = cluster.map_shared_rank(sx, 1);
    const u32* y2 = cluster.map_shared_rank(sx, 2);
    const int base = (pi * G::T + (int)threadIdx.x) * G::D;
    u32 lm[G::D];
    u64 c = 0;
#pragma unroll
    for (int k = 0; k < G::D; ++k) {
        u32 y[3] = {0, 0, 0};
        if (base + k < G::N) {
            const int p = small_pad(base + k);
            y[0] = y0[p], y[1] = y1[p], y[2] = y2[p];
        }
        lm[k] = rns_crt_digit(y, crt, c);
    }
    const CState st = group_state<G::D>(lm, c);
    bool has;
    CState agg;
    CState ex = block_scan_carry(st, &has, &agg, st_scan);
    if (threadIdx.x == 0)
        for (int r = pi + 1; r < 3; ++r) cluster.map_shared_rank(s_agg, r)[pi] = agg;
    cluster.sync();
    u64 cin = 0;
    for (int r = 0; r < pi; ++r) cin = cs_eval(s_agg[r], cin);
    group_add_carry<G::D>(lm, has ? cs_eval(ex, cin) : cin);
    const u64 nout = na + nb;
    unsigned long long top = 0;
#pragma unroll
    for (int k = 0; k < G::D; ++k)
        if (base + k < nout) {
            out[base + k] = lm[k];
            if (lm[k]) top = base + k + 1;
        }
    if (top) atomicMax(&s_top, top);
    __syncthreads();
    if (threadIdx.x == 0) cluster.map_shared_rank(s_tops, 0)[pi] = s_top;
    cluster.sync();
    if (pi == 0 && threadIdx.x == 0) {
        const unsigned long long n = s_tops[2] ? s_tops[2] : (s_tops[1] ? s_tops[1] : s_tops[0]);
        if (out_len) *out_len = n;
        if (hl.host) publish(hl, n);
    }
}

// Products of at most 128 limbs in all (256 in large batches): schoolbook
// columns. (Above that the transforms win at every shape: 500 x 8 limbs 16.6 us a call against 10.4,
// 2,048 of them 97 against 56 us; 250 x 250 18.6 against 8.3.)
__global__ void __launch_bounds__(SCHOOL_THREADS) k_school(const RnsArgs a, u32* __restrict__ out,
                                                           unsigned long long* out_len, const HostLen hl) {
    __shared__ u32 smem[SCHOOL_SMEM_WORDS];
    __shared__ CState st[SCHOOL_WARPS_CTA];
    __shared__ unsigned long long s_top;
    pdl_enter();
    const u32 *la = a.a, *lb = a.b;
    u64 na = a.na, nb = a.nb;
    if (a.jobs) {
        const ProdJob& J = a.jobs[blockIdx.x];
        la = J.a;
        lb = J.b;
        na = J.na;
        nb = J.nb;
        out = J.out;
        out_len = J.out_len;
    }
    school_cta(la, na, lb, nb, out, out_len, smem, st, &s_top);
    if (threadIdx.x == 0 && hl.host) publish(hl, s_top);
}

template <int M>
static cudaError_t configure() {
    return cudaFuncSetAttribute(k_rns_small<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, SmallShape<M>::BYTES);
}
cudaError_t rns_configure_small() {
    cudaError_t e = configure<8>();
    if (e == cudaSuccess) e = configure<9>();
    if (e == cudaSuccess) e = configure<10>();
    if (e == cudaSuccess) e = configure<11>();
    if (e == cudaSuccess) e = configure<12>();
    return e;
}

template <int M>
static cudaError_t launch(unsigned njobs, cudaStream_t s, const RnsArgs& a, u32* out, unsigned long long* out_len,
                          const RnsCrt& crt, HostLen hl) {
    return launch_pdl(k_rns_small<M>, 3 * njobs, SmallShape<M>::T, SmallShape<M>::BYTES, s, a, out, out_len, crt, hl);
}

cudaError_t rns_launch_small(int m, unsigned njobs, cudaStream_t s, const RnsArgs& a, u32* out,
                             unsigned long long* out_len, const RnsCrt& crt, HostLen hl) {
    switch (m) {
        case 8:
            // one after the other the cluster is faster (128 x 128 limbs 8.5
            // against 12.4 us a call), thousands at once the schoolbook
            // (0.015 against 0.021 us each); 512 jobs fill the SMs
            if (njobs >= 512) return launch_pdl(k_school, njobs, SCHOOL_THREADS, 0, s, a, out, out_len, hl);
            return launch<8>(njobs, s, a, out, out_len, crt, hl);
        case 9: return launch<9>(njobs, s, a, out, out_len, crt, hl);
        case 10: return launch<10>(njobs, s, a, out, out_len, crt, hl);
        case 11: return launch<11>(njobs, s, a, out, out_len, crt, hl);
        case 12: return launch<12>(njobs, s, a, out, out_len, crt, hl);
        default:
            if (m > 7) return cudaErrorInvalidValue;
            return launch_pdl(k_school, njobs, SCHOOL_THREADS, 0, s, a, out, out_len, hl);
    }
}

}  // namespace b2m
