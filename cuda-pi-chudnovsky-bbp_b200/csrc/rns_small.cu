// rns_small.cu -- whole products of up to 2^12 32-bit points in one launch.
//
// For each of the three primes a group of threads loads both operands, runs
// both forward transforms side by side (the twiddle loads serve both), the
// pointwise product and the inverse in its own shared memory, and leaves its
// CRT terms there; then all threads form a share of the coefficients each and
// resolve their carries with a block scan. Products of at most 128 limbs are
// schoolbook columns (school.cuh).
//
// The three groups are one block (k_rns_small_one), or a cluster of three
// blocks that read each other's terms through distributed shared memory
// (k_rns_small), so that the longer transforms have three SMs' arithmetic.
// What bounds it: one product alone, latency (the stages are a chain of
// exchanges); thousands at once, arithmetic and the cluster's barriers, which
// cost a block's own several times over. Measured (a call among others / each
// of 4,096 products at once, us; the 64-bit transform on one block before):
//                  before         cluster        one block
//    200 x 150   14.5 / 0.018    6.9 / 0.023    6.3 / 0.014
//    500 x 500   24.7 / 0.079    8.8 / 0.039    6.7 / 0.023
//   1000 x 1000  41.0 / 0.136    9.7 / 0.063    9.9 / 0.047
//   1500 x 400   39.1 / 0.135   10.2 / 0.066   11.5 / 0.052
//   2000 x 2000  53.5 / 0.358   12.7 / 0.145   18.1 / 0.124
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
    // Transform i of thread t: node and the position of its element 0.
    __device__ __forceinline__ static int node(int t, int i) { return (t + i * T) >> REST; }
    __device__ __forceinline__ static int pos(int t, int i) {
        const int id = t + i * T;
        return ((id >> REST) << (M - LEV)) + (id & ((1 << REST) - 1));
    }
};

// Shared-memory index of a position: one pad every 16.
__device__ __forceinline__ int small_pad(int p) { return p + (p >> 4); }

// Barrier of the T threads of prime pi: the block, or (ONE) a third of it.
template <int T, bool ONE>
__device__ __forceinline__ void small_bar(int pi) {
    if constexpr (!ONE) __syncthreads();
    else if constexpr (T == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(pi + 1), "n"(T) : "memory");
}

// Stage S of the forward transforms of both operands (pairs in shared
// memory); the last stage leaves the values in registers.
template <int M, int S, bool HZ, bool ONE>
__device__ __forceinline__ void small_fwd(u32* x, uint2* sp, const uint2* T, const RnsMod& m, int t, int pi) {
    using G = SmallStage<M, S>;
    constexpr bool LAST = S + 1 == SmallCfg<M>::NS;
#pragma unroll
    for (int i = 0; i < G::TASKS; ++i) {
        u32* y = x + (i << (G::L + 1));
        const int p = G::pos(t, i);
        if constexpr (S > 0) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k) {
                const uint2 v = sp[small_pad(p + (k << G::REST))];
                y[2 * k] = v.x, y[2 * k + 1] = v.y;
            }
        }
        rns_dft_fwd<G::L, 2, S == 0, HZ && S == 0>(y, T, (u32)G::node(t, i), m);
        if constexpr (!LAST) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k)
                sp[small_pad(p + (k << G::REST))] = make_uint2(y[2 * k], y[2 * k + 1]);
        }
    }
    if constexpr (!LAST) {
        small_bar<G::T, ONE>(pi);
        small_fwd<M, S + 1, HZ, ONE>(x, sp, T, m, t, pi);
    }
}

// Inverse stages S .. 0; values of the last forward stage's layout in x.
template <int M, int S, bool ONE>
__device__ __forceinline__ void small_inv(u32* x, u32* sx, const uint2* T, const RnsMod& m, int t, int pi) {
    using G = SmallStage<M, S>;
    constexpr bool FIRST = S + 1 == SmallCfg<M>::NS;
#pragma unroll
    for (int i = 0; i < G::TASKS; ++i) {
        u32* y = x + (i << G::L);
        const int p = G::pos(t, i);
        if constexpr (!FIRST) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k) y[k] = sx[small_pad(p + (k << G::REST))];
        }
        rns_dft_inv<G::L, 1, S == 0>(y, T, (u32)G::node(t, i), m);
        if constexpr (S > 0) {
#pragma unroll
            for (int k = 0; k < (1 << G::L); ++k) sx[small_pad(p + (k << G::REST))] = y[k];
        }
    }
    if constexpr (S > 0) {
        small_bar<G::T, ONE>(pi);
        small_inv<M, S - 1, ONE>(x, sx, T, m, t, pi);
    }
}

template <int M, bool ONE>
struct SmallShape {
    static constexpr int N = 1 << M, T = 1 << (M - SmallCfg<M>::LE), PAD = N + N / 16;
    static constexpr int D = (N + 3 * T - 1) / (3 * T);  // digits per thread of the three primes
    // One prime: pairs, then its product. A block of one prime, or of three,
    // and one carry state per warp.
    static constexpr int WORDS = 3 * PAD, BLOCK = ONE ? 3 * T : T;
    static constexpr int BYTES = (ONE ? 3 : 1) * WORDS * 4 + BLOCK / 32 * 16;
    static constexpr int MINT = T >= 256 ? 3 : (T >= 128 ? 6 : (SmallCfg<M>::LE == 4 ? 12 : (T == 64 ? 16 : 28)));
    static constexpr int MINB = ONE ? MINT / 3 : MINT;
};

// One prime's share of a product by its T threads: limbs to CRT terms in sx.
template <int M, bool ONE>
__device__ __forceinline__ void small_product(const u32* la, u64 na, const u32* lb, u64 nb, const RnsArgs& a,
                                              const RnsCrt& crt, uint2* sp, u32* sx, int t, int pi) {
    using G = SmallShape<M, ONE>;
    using C = SmallCfg<M>;
    using S0 = SmallStage<M, 0>;
    constexpr int E = 1 << C::LE;
    const RnsMod m(pi);
    const uint2* T = a.tw + (u64)pi * a.ent;
    const uint2* Ti = a.twi + (u64)pi * a.ent;
    const u32 np4 = 2 * m.np2;
    u32 x[2 * E];
    const bool hz = 2 * na <= G::N && 2 * nb <= G::N;
#pragma unroll
    for (int i = 0; i < S0::TASKS; ++i)
#pragma unroll
        for (int k = 0; k < (1 << S0::L); ++k) {
            u32 va = 0, vb = 0;
            if (!hz || k < (1 << S0::L) / 2) {
                const u32 j = S0::pos(t, i) + (k << S0::REST);
                va = j < na ? la[j] : 0u;
                vb = j < nb ? lb[j] : 0u;
            }
            u32* y = x + (i << (S0::L + 1)) + 2 * k;
            y[0] = __viaddmin_u32(va, np4, va);
            y[1] = __viaddmin_u32(vb, np4, vb);
        }
    if (hz) small_fwd<M, 0, true, ONE>(x, sp, T, m, t, pi);
    else small_fwd<M, 0, false, ONE>(x, sp, T, m, t, pi);
#pragma unroll
    for (int k = 0; k < E; ++k) x[k] = rns_redc((u64)rns_red2(x[2 * k], m) * rns_red2(x[2 * k + 1], m), pi, m);
    small_inv<M, C::NS - 1, ONE>(x, sx, Ti, m, t, pi);
    // CRT terms, canonical
    const uint2 kap = pi == 0 ? crt.kap[0] : (pi == 1 ? crt.kap[1] : crt.kap[2]);
#pragma unroll
    for (int i = 0; i < S0::TASKS; ++i)
#pragma unroll
        for (int k = 0; k < (1 << S0::L); ++k) {
            const u32 v = rns_mul(x[(i << S0::L) + k], kap, m);
            sx[small_pad(S0::pos(t, i) + (k << S0::REST))] = __viaddmin_u32(v, 0u - m.p, v);
        }
}

template <int M, bool ONE>
__device__ __forceinline__ void small_kernel(const RnsArgs& a, u32* out, unsigned long long* out_len,
                                             const RnsCrt& crt, const HostLen& hl) {
    using G = SmallShape<M, ONE>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned long long s_top;
    __shared__ unsigned long long s_tops[3];
    __shared__ CState s_agg[2];  // of the blocks before this one
    const int pi = ONE ? __shfl_sync(0xFFFFFFFFu, (int)threadIdx.x / G::T, 0) : blockIdx.x % 3;
    const int t = ONE ? threadIdx.x % G::T : threadIdx.x;
    pdl_enter();
    const u32 *la = a.a, *lb = a.b;
    u64 na = a.na, nb = a.nb;
    if (a.jobs) {
        const ProdJob& J = a.jobs[ONE ? blockIdx.x : blockIdx.x / 3];
        la = J.a;
        lb = J.b;
        na = J.na;
        nb = J.nb;
        out = J.out;
        out_len = J.out_len;
    }
    u32* sw = reinterpret_cast<u32*>(smem);
    CState* st_scan = reinterpret_cast<CState*>(sw + (ONE ? 3 : 1) * G::WORDS);
    u32* mine = sw + (ONE ? pi * G::WORDS : 0);
    u32* sx = mine + 2 * G::PAD;
    if (threadIdx.x == 0) s_top = 0;
    small_product<M, ONE>(la, na, lb, nb, a, crt, reinterpret_cast<uint2*>(mine), sx, t, pi);
    // The 3T threads take G::D consecutive digits each, prime r's from r T D
    // on (digits past N are zero).
    cg::cluster_group cluster = cg::this_cluster();
    const u32 *y0, *y1, *y2;
    if constexpr (ONE) {
        __syncthreads();
        y0 = sw + 2 * G::PAD, y1 = y0 + G::WORDS, y2 = y1 + G::WORDS;
    } else {
        cluster.sync();
        y0 = cluster.map_shared_rank(sx, 0), y1 = cluster.map_shared_rank(sx, 1), y2 = cluster.map_shared_rank(sx, 2);
    }
    const int base = (pi * G::T + t) * G::D;
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
    u64 cin = 0;
    if constexpr (!ONE) {
        // a block scan, then the aggregates of the blocks before it, pushed by them
        if (threadIdx.x == 0)
            for (int r = pi + 1; r < 3; ++r) cluster.map_shared_rank(s_agg, r)[pi] = agg;
        cluster.sync();
        for (int r = 0; r < pi; ++r) cin = cs_eval(s_agg[r], cin);
    }
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
    unsigned long long n = s_top;
    if constexpr (!ONE) {
        if (threadIdx.x == 0) cluster.map_shared_rank(s_tops, 0)[pi] = n;
        cluster.sync();
        n = s_tops[2] ? s_tops[2] : (s_tops[1] ? s_tops[1] : s_tops[0]);
        if (pi != 0) return;
    }
    if (threadIdx.x == 0) {
        if (out_len) *out_len = n;
        if (hl.host) publish(hl, n);
    }
}

template <int M>
__global__ void __cluster_dims__(3, 1, 1) __launch_bounds__(SmallShape<M, false>::T, SmallShape<M, false>::MINB)
    k_rns_small(const RnsArgs a, u32* out, unsigned long long* out_len, const RnsCrt crt,
                const HostLen hl) {
    small_kernel<M, false>(a, out, out_len, crt, hl);
}

template <int M>
__global__ void __launch_bounds__(SmallShape<M, true>::BLOCK, SmallShape<M, true>::MINB)
    k_rns_small_one(const RnsArgs a, u32* out, unsigned long long* out_len, const RnsCrt crt,
                    const HostLen hl) {
    small_kernel<M, true>(a, out, out_len, crt, hl);
}

// Products of at most 128 limbs in all: schoolbook columns. (Above that the
// transforms were faster than columns on four warps at every shape; columns on
// more warps were not measured.) W warps a product, 4 / W products a block.
template <int W>
__global__ void __launch_bounds__(SCHOOL_THREADS) k_school(const RnsArgs a, unsigned njobs, u32* out,
                                                           unsigned long long* out_len, const HostLen hl) {
    constexpr int PER = SCHOOL_WARPS_CTA / W;
    __shared__ u32 smem[PER * SCHOOL_SMEM_WORDS<W>];
    __shared__ CState st[SCHOOL_WARPS_CTA];
    __shared__ unsigned long long s_top;
    pdl_enter();
    const int sl = PER > 1 ? threadIdx.x / (32 * W) : 0;
    const unsigned job = blockIdx.x * PER + sl;
    if (job >= njobs) return;  // whole warps, none of which meets a barrier of the block (PER > 1)
    const u32 *la = a.a, *lb = a.b;
    u64 na = a.na, nb = a.nb;
    if (a.jobs) {
        const ProdJob& J = a.jobs[job];
        la = J.a;
        lb = J.b;
        na = J.na;
        nb = J.nb;
        out = J.out;
        out_len = J.out_len;
    }
    if (na > nb) {  // the loop runs over the first operand
        const u32* l = la;
        la = lb, lb = l;
        const u64 n = na;
        na = nb, nb = n;
    }
    const unsigned long long n =
        school_product<W>(la, (int)na, lb, (int)nb, out, smem + sl * SCHOOL_SMEM_WORDS<W>, st, &s_top);
    if (threadIdx.x % (32 * W) == 0) {
        if (out_len) *out_len = n;
        if (hl.host) publish(hl, n);
    }
}

// Lengths whose single products run as a cluster: from 2^11 points the work
// of a prime is worth an SM of its own.
constexpr int SMALL_CLUSTER_M = 11;

template <int M>
static cudaError_t configure() {
    cudaError_t e = cudaFuncSetAttribute(k_rns_small_one<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SmallShape<M, true>::BYTES);
    if constexpr (M >= SMALL_CLUSTER_M)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_rns_small<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SmallShape<M, false>::BYTES);
    return e;
}
cudaError_t rns_configure_small() {
    cudaError_t e = configure<8>();
    if (e == cudaSuccess) e = configure<9>();
    if (e == cudaSuccess) e = configure<10>();
    if (e == cudaSuccess) e = configure<11>();
    if (e == cudaSuccess) e = configure<12>();
    return e;
}

// A cluster below `many` products, from there (the SMs are full either way)
// one block each: 64 products of 1000 x 1000 limbs 15.1 against 13.0 us, 512
// of 2000 x 2000 86 against 76 us, but 64 of those 22.6 against 22.8 and one
// 12.7 against 18.1 us.
template <int M>
static cudaError_t launch(unsigned many, unsigned njobs, cudaStream_t s, const RnsArgs& a, u32* out,
                          unsigned long long* out_len, const RnsCrt& crt, HostLen hl) {
    if constexpr (M >= SMALL_CLUSTER_M)
        if (njobs < many)
            return launch_pdl(k_rns_small<M>, 3 * njobs, SmallShape<M, false>::T, SmallShape<M, false>::BYTES, s, a,
                              out, out_len, crt, hl);
    return launch_pdl(k_rns_small_one<M>, njobs, SmallShape<M, true>::BLOCK, SmallShape<M, true>::BYTES, s, a, out,
                      out_len, crt, hl);
}

cudaError_t rns_launch_small(int m, unsigned njobs, cudaStream_t s, const RnsArgs& a, u32* out,
                             unsigned long long* out_len, const RnsCrt& crt, HostLen hl) {
    switch (m) {
        case 8: return launch<8>(0, njobs, s, a, out, out_len, crt, hl);
        case 9: return launch<9>(0, njobs, s, a, out, out_len, crt, hl);
        case 10: return launch<10>(0, njobs, s, a, out, out_len, crt, hl);
        case 11: return launch<11>(64, njobs, s, a, out, out_len, crt, hl);
        case 12: return launch<12>(256, njobs, s, a, out, out_len, crt, hl);
        default:
            if (m > 7) return cudaErrorInvalidValue;
            // Four warps split one product's terms; once a block each fills
            // the SMs a warp a product does less in all (60 x 60 limbs: 512
            // products 8.7 against 7.1 us, 4,096 23.1 against 14.8; 64 the
            // same).
            if (njobs >= 512)
                return launch_pdl(k_school<1>, (njobs + SCHOOL_WARPS_CTA - 1) / SCHOOL_WARPS_CTA, SCHOOL_THREADS, 0, s,
                                  a, njobs, out, out_len, hl);
            return launch_pdl(k_school<SCHOOL_WARPS_CTA>, njobs, SCHOOL_THREADS, 0, s, a, njobs, out, out_len, hl);
    }
}

}  // namespace b2m
