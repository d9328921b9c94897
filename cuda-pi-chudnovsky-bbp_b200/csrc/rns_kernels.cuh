// rns_kernels.cuh -- transform passes over the three 30-bit primes.
//
// A product of na x nb limbs uses 32-bit digits (one limb each) and
// N = q * 2^m >= na + nb points. Evaluating at N points means reducing the
// operand modulo x^M - c_t for q constants c_t (M = 2^m, t < q) and splitting
// each x^M - c_t down to linear factors by a binary tree:
//     x^2h - w^2 = (x^h - w)(x^h + w),
// one butterfly (a, b) -> (a + w b, a - w b) per pair of coefficients, with
// one twiddle w per tree node, the same for every position inside the node.
// Nodes are numbered 2k, 2k + 1 below k, so with T[k] = product over the set
// bits j of k of the 2^(j+2)-th root of unity, node k of every level splits
// with w = T[k]: one table serves all lengths and all levels, and there are
// no twiddles between passes. The inverse runs the tree backwards with the
// inverses. Everything stays in place; the spectrum's order never matters.
//
// Passes: pass k handles logr[k] levels. An array is B sub-problems (the
// nodes at the level where the pass starts) of R rows x S columns, row-major.
// A block takes C columns of one sub-problem; each thread holds 2^LA
// elements in registers: stage A does LA levels over rows 2^LB apart, one
// exchange through shared memory, stage B the remaining LB levels over
// adjacent rows. Loads and stores go straight between registers and global
// memory (C columns of a row are contiguous). The last pass (S = 1) keeps a
// sub-problem inside one warp, transforms both operands, multiplies, and
// runs the first inverse pass on the product without leaving the registers
// but for the exchanges, so a product of P passes is P + (P - 1) transform
// launches for both operands and all primes together.
//
// What bounds them: the multiply-add pipe (8 cycles of it per butterfly) with
// the ALU pipe close behind (rns_field.cuh), both at 50 to 65% of their peak,
// and the exchange between the stages; DRAM is at 30 to 60% of its bandwidth.
// Three blocks of 256 threads at 80 registers an SM; four of 64 registers
// gained 1%. Measured at 2^24 x 2^24 limbs (four parts of 2^23 points), ms, and
// the same passes of the 64-bit transform: first 0.45 (2 x 0.46), middle 0.29
// (2 x 0.47), fused 0.43 (0.74, and the other operand's last pass besides),
// inverse 0.15 and 0.28 with the parts put together (2 x 0.50), carry 0.16
// (0.18).
//
// Reference counterpart: the per-stage launches of src/ntt_cuda.cu:99-128;
// the product is the same integer.
#pragma once
#include "b2m_internal.h"
#include "pdl.cuh"
#include "rns_field.cuh"

namespace b2m {

__device__ __forceinline__ uint2 rns_ld(const uint2* p) { return __ldg(p); }
__device__ __forceinline__ uint4 rns_ld2(const uint2* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
// Four twiddles in one 32-byte load (32-byte aligned): a warp's lanes read
// runs of eight that lie 64 bytes apart, and every load instruction looks up
// each 128-byte line it touches.
struct Tw4 {
    uint2 w[4];
};
__device__ __forceinline__ Tw4 rns_ld4(const uint2* p) {
    Tw4 t;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(t.w[0].x), "=r"(t.w[0].y), "=r"(t.w[1].x), "=r"(t.w[1].y), "=r"(t.w[2].x), "=r"(t.w[2].y),
          "=r"(t.w[3].x), "=r"(t.w[3].y)
        : "l"(p));
    return t;
}

// L levels below node `node` on 2^L positions of V vectors side by side
// (x[i * V + v]; position i of the node's 2^L equal parts), which share every
// twiddle load. N0: the node is node 0, whose leftmost chain has w = 1. HZ
// (with N0): the upper half is zero, so the first level copies.
template <int L, int V, bool N0, bool HZ, int LEV = 0>
__device__ __forceinline__ void rns_dft_fwd(u32* x, const uint2* __restrict__ T, u32 node, const RnsMod& m) {
    constexpr int half = V << (L - 1 - LEV);
    if constexpr (LEV == 0) {
        if constexpr (N0 && HZ) {
#pragma unroll
            for (int i = 0; i < half; ++i) x[i + half] = x[i];
        } else if constexpr (N0) {
#pragma unroll
            for (int i = 0; i < half; ++i) rns_bfly_fwd1(x[i], x[i + half], m);
        } else {
            const uint2 w = rns_ld(T + node);
#pragma unroll
            for (int i = 0; i < half; ++i) rns_bfly_fwd(x[i], x[i + half], w, m);
        }
    } else {
        constexpr int W = LEV == 1 ? 2 : 4;  // twiddles per load
#pragma unroll
        for (int j0 = 0; j0 < (1 << LEV); j0 += W) {
            uint2 w[W];
            if constexpr (W == 2) {
                const uint4 v = rns_ld2(T + (node << LEV) + j0);
                w[0] = make_uint2(v.x, v.y), w[1] = make_uint2(v.z, v.w);
            } else {
                const Tw4 v = rns_ld4(T + (node << LEV) + j0);
#pragma unroll
                for (int j = 0; j < W; ++j) w[j] = v.w[j];
            }
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int i = 2 * (j0 + j) * half; i < (2 * (j0 + j) + 1) * half; ++i) {
                    if (N0 && j0 + j == 0) rns_bfly_fwd1(x[i], x[i + half], m);
                    else rns_bfly_fwd(x[i], x[i + half], w[j], m);
                }
        }
    }
    if constexpr (LEV + 1 < L) rns_dft_fwd<L, V, N0, HZ, LEV + 1>(x, T, node, m);
}

template <int L, int V, bool N0, int LEV = L - 1>
__device__ __forceinline__ void rns_dft_inv(u32* x, const uint2* __restrict__ T, u32 node, const RnsMod& m) {
    constexpr int half = V << (L - 1 - LEV);
    if constexpr (LEV == 0) {
        if constexpr (N0) {
#pragma unroll
            for (int i = 0; i < half; ++i) rns_bfly_inv1(x[i], x[i + half], m);
        } else {
            const uint2 w = rns_ld(T + node);
#pragma unroll
            for (int i = 0; i < half; ++i) rns_bfly_inv(x[i], x[i + half], w, m);
        }
    } else {
        constexpr int W = LEV == 1 ? 2 : 4;  // twiddles per load
#pragma unroll
        for (int j0 = 0; j0 < (1 << LEV); j0 += W) {
            uint2 w[W];
            if constexpr (W == 2) {
                const uint4 v = rns_ld2(T + (node << LEV) + j0);
                w[0] = make_uint2(v.x, v.y), w[1] = make_uint2(v.z, v.w);
            } else {
                const Tw4 v = rns_ld4(T + (node << LEV) + j0);
#pragma unroll
                for (int j = 0; j < W; ++j) w[j] = v.w[j];
            }
#pragma unroll
            for (int j = 0; j < W; ++j)
#pragma unroll
                for (int i = 2 * (j0 + j) * half; i < (2 * (j0 + j) + 1) * half; ++i) {
                    if (N0 && j0 + j == 0) rns_bfly_inv1(x[i], x[i + half], m);
                    else rns_bfly_inv(x[i], x[i + half], w[j], m);
                }
        }
        rns_dft_inv<L, V, N0, LEV - 1>(x, T, node, m);
    }
}

// V adjacent words.
template <int V>
__device__ __forceinline__ void rns_get(u32* x, const u32* p) {
    if constexpr (V == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        x[0] = v.x, x[1] = v.y;
    } else {
        x[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void rns_put(u32* p, const u32* x) {
    if constexpr (V == 2) *reinterpret_cast<uint2*>(p) = make_uint2(x[0], x[1]);
    else *p = x[0];
}

// ---------------------------------------------------------------------------
// Column passes. LA >= LB; a block is 256 threads: 2^LB row groups x C / V
// lanes of V adjacent columns. V = 2 halves the memory instructions, the
// address arithmetic and the twiddle loads per element (a 16-byte twiddle
// load takes the L1 four cycles even when every lane reads the same one);
// V = 1 keeps twice as many blocks for short transforms. Shared memory rows
// get one pad row every 2^LB, so that the row groups of a warp fall into
// different banks in both stages. Global addresses are a block-uniform
// 64-bit base per row plus the thread's 32-bit offset.
// ---------------------------------------------------------------------------
template <int LOGR, int V>
struct RnsCol {
    static constexpr int LA = (LOGR + 1) / 2, LB = LOGR - LA;
    static constexpr int E = 1 << LA, U = 1 << LB, R = 1 << LOGR;
    static constexpr int LP = 8 - LB, LC = LP + V - 1, C = 1 << LC;
    static constexpr int NB = 1 << (LA - LB);  // stage-B transforms per thread
    static constexpr int SMEM = (R + (R >> LB)) << LC;  // words
    static constexpr int THREADS = 256;
    static constexpr int MINB = E * V >= 32 ? 3 : 4;
    static_assert(V == 1 || V == 2, "one or two columns");
    __device__ __forceinline__ static int sa(int row, int col) { return ((row + (row >> LB)) << LC) + col; }
};

// Thread coordinates of a column pass.
template <class G, int V>
struct RnsThread {
    int u, col;
    __device__ __forceinline__ RnsThread()
        : u(threadIdx.x >> G::LP), col(((int)threadIdx.x & ((1 << G::LP) - 1)) * V) {}
};

template <int LOGR, int V>
__device__ __forceinline__ void rns_exchange_ab(u32* sm, u32* x, int u, int col) {
    using G = RnsCol<LOGR, V>;
#pragma unroll
    for (int k = 0; k < G::E; ++k) rns_put<V>(sm + G::sa(u + (k << G::LB), col), x + k * V);
    __syncthreads();
#pragma unroll
    for (int n = 0; n < G::NB; ++n)
#pragma unroll
        for (int k = 0; k < G::U; ++k)
            rns_get<V>(x + (n * G::U + k) * V, sm + G::sa(((u + (n << G::LB)) << G::LB) + k, col));
}
template <int LOGR, int V>
__device__ __forceinline__ void rns_exchange_ba(u32* sm, u32* x, int u, int col) {
    using G = RnsCol<LOGR, V>;
#pragma unroll
    for (int n = 0; n < G::NB; ++n)
#pragma unroll
        for (int k = 0; k < G::U; ++k)
            rns_put<V>(sm + G::sa(((u + (n << G::LB)) << G::LB) + k, col), x + (n * G::U + k) * V);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < G::E; ++k) rns_get<V>(x + k * V, sm + G::sa(u + (k << G::LB), col));
}

// Stage B of a column pass: NB transforms of LB levels at nodes node0 + s.
template <int LOGR, int V, bool INV>
__device__ __forceinline__ void rns_stage_b(u32* x, const uint2* T, u32 node0, int u, const RnsMod& m) {
    using G = RnsCol<LOGR, V>;
#pragma unroll
    for (int n = 0; n < G::NB; ++n) {
        u32* y = x + n * G::U * V;
        if constexpr (INV) rns_dft_inv<G::LB, V, false>(y, T, node0 + u + (n << G::LB), m);
        else rns_dft_fwd<G::LB, V, false, false>(y, T, node0 + u + (n << G::LB), m);
    }
}

// Stage-A rows u + k 2^LB and stage-B rows (u + n 2^LB) 2^LB + k of the
// thread's columns, from a block-uniform base.
template <int LOGR, int V>
__device__ __forceinline__ void rns_store_a(const u32* x, u32* base, int u, int col, int logs) {
    using G = RnsCol<LOGR, V>;
    const u32 o = ((u32)u << logs) + col;
#pragma unroll
    for (int k = 0; k < G::E; ++k) rns_put<V>(base + ((u64)k << (logs + G::LB)) + o, x + k * V);
}
template <int LOGR, int V>
__device__ __forceinline__ void rns_load_a(u32* x, const u32* base, int u, int col, int logs) {
    using G = RnsCol<LOGR, V>;
    const u32 o = ((u32)u << logs) + col;
#pragma unroll
    for (int k = 0; k < G::E; ++k) rns_get<V>(x + k * V, base + ((u64)k << (logs + G::LB)) + o);
}
template <int LOGR, int V>
__device__ __forceinline__ void rns_store_b(const u32* x, u32* base, int u, int col, int logs) {
    using G = RnsCol<LOGR, V>;
    const u32 o = ((u32)u << (logs + G::LB)) + col;
#pragma unroll
    for (int n = 0; n < G::NB; ++n)
#pragma unroll
        for (int k = 0; k < G::U; ++k)
            rns_put<V>(base + ((u64)((n << (2 * G::LB)) + k) << logs) + o, x + (n * G::U + k) * V);
}
template <int LOGR, int V>
__device__ __forceinline__ void rns_load_b(u32* x, const u32* base, int u, int col, int logs) {
    using G = RnsCol<LOGR, V>;
    const u32 o = ((u32)u << (logs + G::LB)) + col;
#pragma unroll
    for (int n = 0; n < G::NB; ++n)
#pragma unroll
        for (int k = 0; k < G::U; ++k)
            rns_get<V>(x + (n * G::U + k) * V, base + ((u64)((n << (2 * G::LB)) + k) << logs) + o);
}
// K stage-A rows of limbs (j0 + k rows of 2^LB), zero at and past n, below
// 4p (np4 = -4p). Operands are 4-byte aligned: limbs load one by one. Tiles
// below the operand's end take no per-limb check.
template <int LOGR, int V, int K>
__device__ __forceinline__ void rns_load_limbs(u32* x, const u32* limbs, u32 j0, u32 n, int logs, u32 np4) {
    using G = RnsCol<LOGR, V>;
    const int ls = logs + G::LB;
    // last position the block's K rows touch, plus one (at most 2^26)
    if (((u32)K << ls) - (1u << logs) + G::C <= n) {
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int v = 0; v < V; ++v) x[k * V + v] = limbs[((u64)k << ls) + j0 + v];
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k)
#pragma unroll
            for (int v = 0; v < V; ++v)
                x[k * V + v] = j0 + ((u32)k << ls) + v < n ? limbs[((u64)k << ls) + j0 + v] : 0u;
    }
#pragma unroll
    for (int k = 0; k < K * V; ++k) x[k] = __viaddmin_u32(x[k], np4, x[k]);
}

// Buffer of operand `op` (0: A, 1: B) of the block's job.
__device__ __forceinline__ u32* rns_buf(const RnsArgs& a, int op) {
    return op ? a.bufB + blockIdx.y * a.stride_b : a.bufA + blockIdx.y * a.stride_a;
}

// The operand of a first pass, and the zeroing of the product's carry scratch
// and length by the pass's first grid layer. JOBS: from the job table (kept apart so that
// single products address their limbs from uniform registers).
template <bool JOBS>
__device__ __forceinline__ const u32* rns_operand(const RnsArgs& a, int op, u32* n) {
    if constexpr (JOBS) {
        const ProdJob& J = a.jobs[blockIdx.y];
        if (blockIdx.z == 0 && J.slots) {  // (null: only the spectrum is wanted)
            const u32 i = blockIdx.x * 256 + threadIdx.x;
            if (i < a.nzero) reinterpret_cast<unsigned long long*>(J.slots)[i] = 0;
            if (i == 0) *J.out_len = 0;
        }
        *n = (u32)(op ? J.nb : J.na);  // at most 2^26
        return op ? J.b : J.a;
    } else {
        if (blockIdx.z == 0 && a.zero) {
            const u32 i = blockIdx.x * 256 + threadIdx.x;
            if (i < a.nzero) a.zero[i] = 0;
            if (i == 0) *a.zero_len = 0;
        }
        *n = (u32)(op ? a.nb : a.na);
        return op ? a.b : a.a;
    }
}

// First forward pass: limbs -> residues. Grid x: tiles, y: jobs, z: operand *
// 3 + prime.
template <int LOGR, int V, bool JOBS>
__global__ void __launch_bounds__(256, (RnsCol<LOGR, V>::MINB)) k_rns_first(const RnsArgs a) {
    using G = RnsCol<LOGR, V>;
    extern __shared__ __align__(16) u32 smr[];
    const int pi = blockIdx.z % 3, op = a.op0 + blockIdx.z / 3;
    const RnsMod m(pi);
    pdl_enter();
    u32 n;
    const u32* limbs = rns_operand<JOBS>(a, op, &n);
    const RnsThread<G, V> t;
    const u32 c0 = blockIdx.x << G::LC;            // first column of the tile
    const u32 j0 = ((u32)t.u << a.logs) + t.col;   // this thread's first position, less c0
    const u32 np4 = 2 * m.np2;
    u32 x[G::E * V];
    const uint2* T = a.tw + (u64)pi * a.ent;
    if (2 * (u64)n <= a.nt) {
        // the upper half of the points is zero for almost every product
        rns_load_limbs<LOGR, V, G::E / 2>(x, limbs + c0, j0, n > c0 ? n - c0 : 0u, a.logs, np4);
        rns_dft_fwd<G::LA, V, true, true>(x, T, 0, m);
    } else {
        rns_load_limbs<LOGR, V, G::E>(x, limbs + c0, j0, n > c0 ? n - c0 : 0u, a.logs, np4);
        rns_dft_fwd<G::LA, V, true, false>(x, T, 0, m);
    }
    rns_exchange_ab<LOGR, V>(smr, x, t.u, t.col);
    rns_stage_b<LOGR, V, false>(x, T, 0, t.u, m);
    rns_store_b<LOGR, V>(x, rns_buf(a, op) + ((u64)pi * a.nt + c0), t.u, t.col, a.logs);
}

// The same for a transform in q parts: the operand modulo x^M - c_t, that is
// the sum over the filled M-blocks of c_t^i x_i (highest first), then the
// part's levels. A block runs a.pper parts of its tile one after the other on
// the limbs it loaded once (the two blocks that a balanced product's operand
// fills; further ones are read again). Grid x: tiles of M, then part groups.
template <int LOGR, int V, bool JOBS>
__global__ void __launch_bounds__(256, 3) k_rns_first_parts(const RnsArgs a) {
    using G = RnsCol<LOGR, V>;
    extern __shared__ __align__(16) u32 smr[];
    const int pi = blockIdx.z % 3, op = a.op0 + blockIdx.z / 3;
    const RnsMod m(pi);
    pdl_enter();
    u32 n;
    const u32* limbs = rns_operand<JOBS>(a, op, &n);
    const RnsThread<G, V> t;
    const u32 c0 = (blockIdx.x & ((1u << (a.logs - G::LC)) - 1)) << G::LC;
    const u32 j0 = ((u32)t.u << a.logs) + t.col;
    const u32 np4 = 2 * m.np2;
    const int lm = a.logs + LOGR;
    const u32 last = n ? (n - 1) >> lm : 0u;
    u32 hi[G::E * V], lo[G::E * V];
    {
        const u32 b0 = (last << lm) + c0;
        rns_load_limbs<LOGR, V, G::E>(hi, limbs + b0, j0, n > b0 ? n - b0 : 0u, a.logs, np4);
        if (last) {  // blocks below the last are full
            rns_load_limbs<LOGR, V, G::E>(lo, limbs + (((last - 1) << lm) + c0), j0, ~0u, a.logs, np4);
#pragma unroll
            for (int k = 0; k < G::E * V; ++k) lo[k] = rns_red2(lo[k], m);
        }
    }
    const u32 t0 = (blockIdx.x >> (a.logs - G::LC)) * a.pper;
#pragma unroll 1
    for (u32 part = t0; part < t0 + a.pper; ++part) {
        const uint2 ct = a.ct[pi][part];
        u32 x[G::E * V];
        if (last == 0) {
#pragma unroll
            for (int k = 0; k < G::E * V; ++k) x[k] = hi[k];
        } else if (part == 0) {  // c_0 = 1
#pragma unroll
            for (int k = 0; k < G::E * V; ++k) x[k] = lo[k] + rns_red2(hi[k], m);
        } else {
#pragma unroll
            for (int k = 0; k < G::E * V; ++k) x[k] = lo[k] + rns_mul(hi[k], ct, m);
        }
        for (u32 i = last; i-- > 1;) {
            const u32* lp = limbs + (((i - 1) << lm) + c0);
#pragma unroll
            for (int k = 0; k < G::E * V; ++k) {
                const u32 v = lp[((u64)(k / V) << (a.logs + G::LB)) + j0 + k % V];
                x[k] = rns_red2(__viaddmin_u32(v, np4, v), m) + rns_mul(x[k], ct, m);
            }
        }
        // roots of unity as the c_t: the nodes of the common tree; otherwise
        // (weighted) each part has its own first-pass tree and leaves a
        // factor theta_t^column (theta_0 = 1)
        const uint2* T = a.wtree ? a.wtree + ((u64)(pi * a.q + part) << LOGR) : a.tw + (u64)pi * a.ent;
        const u32 n0 = a.wtree ? 1u : part;
        rns_dft_fwd<G::LA, V, false, false>(x, T, n0, m);
        rns_exchange_ab<LOGR, V>(smr + (part & 1) * G::SMEM, x, t.u, t.col);  // two buffers in turn
        rns_stage_b<LOGR, V, false>(x, T, n0 << G::LA, t.u, m);
        if (a.wtree && part) {
            const uint2* wc = a.wcol + ((u64)(pi * a.q + part) << a.logs) + c0 + t.col;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const uint2 w = rns_ld(wc + v);
#pragma unroll
                for (int k = 0; k < G::E; ++k) x[k * V + v] = rns_mul(x[k * V + v], w, m);
            }
        }
        rns_store_b<LOGR, V>(x, rns_buf(a, op) + ((u64)pi * a.nt + ((u64)part << lm) + c0), t.u, t.col, a.logs);
    }
}

// A middle forward pass, in place. Grid as above.
template <int LOGR, int V>
__global__ void __launch_bounds__(256, (RnsCol<LOGR, V>::MINB)) k_rns_mid(const RnsArgs a) {
    using G = RnsCol<LOGR, V>;
    extern __shared__ __align__(16) u32 smr[];
    const int pi = blockIdx.z % 3, op = a.op0 + blockIdx.z / 3;
    const RnsMod m(pi);
    const RnsThread<G, V> t;
    const u32 cg = blockIdx.x & ((1u << (a.logs - G::LC)) - 1), sub = blockIdx.x >> (a.logs - G::LC);
    const u32 node = sub & a.nmask;
    u32* buf = rns_buf(a, op) + ((u64)pi * a.nt + ((u64)sub << (a.logs + LOGR)) + (cg << G::LC));
    const uint2* T = a.tw + (u64)pi * a.ent;
    u32 x[G::E * V];
    pdl_enter();
    rns_load_a<LOGR, V>(x, buf, t.u, t.col, a.logs);
    rns_dft_fwd<G::LA, V, false, false>(x, T, node, m);
    rns_exchange_ab<LOGR, V>(smr, x, t.u, t.col);
    rns_stage_b<LOGR, V, false>(x, T, node << G::LA, t.u, m);
    rns_store_b<LOGR, V>(x, buf, t.u, t.col, a.logs);
}

// An inverse column pass, in place. Grid z: prime. FIRST: the tree's top
// levels (pass 0) of an undivided transform.
template <int LOGR, int V, bool FIRST>
__global__ void __launch_bounds__(256, (RnsCol<LOGR, V>::MINB)) k_rns_inv(const RnsArgs a) {
    using G = RnsCol<LOGR, V>;
    extern __shared__ __align__(16) u32 smr[];
    const int pi = blockIdx.z;
    const RnsMod m(pi);
    const RnsThread<G, V> t;
    const u32 cg = blockIdx.x & ((1u << (a.logs - G::LC)) - 1), sub = blockIdx.x >> (a.logs - G::LC);
    u32* buf = rns_buf(a, 1) + ((u64)pi * a.nt + ((u64)sub << (a.logs + LOGR)) + (cg << G::LC));
    const uint2* T = a.twi + (u64)pi * a.ent;
    const u32 node = FIRST ? 0u : sub & a.nmask;
    u32 x[G::E * V];
    pdl_enter();
    rns_load_b<LOGR, V>(x, buf, t.u, t.col, a.logs);
    rns_stage_b<LOGR, V, true>(x, T, node << G::LA, t.u, m);
    rns_exchange_ba<LOGR, V>(smr, x, t.u, t.col);
    rns_dft_inv<G::LA, V, FIRST>(x, T, node, m);
    rns_store_a<LOGR, V>(x, buf, t.u, t.col, a.logs);
}

// Inverse pass 0 of a transform in Q parts: each block runs its tile of every
// part, then puts the parts together in registers,
//     f_s[j] = sum_t V^-1[s][t] z_t[j]
// (V the Vandermonde matrix of the c_t), one wide sum and one reduction per
// value: z_t is brought below p, so Q <= 8 terms below 2^59.8 fit 64 bits. As
// a kernel of its own the last step read and wrote all residues once more
// (215 us of the 2^24-limb product, 88 us at 3 * 2^22 points).
template <int LOGR, int Q>
__global__ void __launch_bounds__(256, (RnsCol<LOGR, 1>::E * Q >= 48 ? 2 : 3))
    k_rns_inv_parts(const RnsArgs a, const RnsCombine c) {
    using G = RnsCol<LOGR, 1>;
    extern __shared__ __align__(16) u32 smr[];
    const int pi = blockIdx.z;
    const RnsMod m(pi);
    const RnsThread<G, 1> t;
    const u32 c0 = blockIdx.x << G::LC;
    const u64 M = 1ull << (a.logs + LOGR);
    u32* buf = rns_buf(a, 1) + ((u64)pi * a.nt + c0);
    u32 z[Q][G::E];
    pdl_enter();
#pragma unroll
    for (int s = 0; s < Q; ++s) {
        u32* x = z[s];
        rns_load_b<LOGR, 1>(x, buf + s * M, t.u, t.col, a.logs);
        const uint2* T = a.twi + (u64)pi * a.ent;
        u32 node = s;
        if (a.wtree) {
            T = a.wtree + ((u64)(pi * Q + s) << LOGR);
            node = 1;
            if (s) {  // theta_0 = 1
                const uint2 w = rns_ld(a.wcol + ((u64)(pi * Q + s) << a.logs) + c0 + t.col);
#pragma unroll
                for (int k = 0; k < G::E; ++k) x[k] = rns_mul(x[k], w, m);
            }
        }
        rns_stage_b<LOGR, 1, true>(x, T, node << G::LA, t.u, m);
        // two buffers in turn: a part's writes never meet the previous part's
        // reads, which end before the barrier in between
        rns_exchange_ba<LOGR, 1>(smr + (s & 1) * G::SMEM, x, t.u, t.col);
        rns_dft_inv<G::LA, 1, false>(x, T, node, m);
#pragma unroll
        for (int k = 0; k < G::E; ++k) x[k] = __viaddmin_u32(x[k], 0u - m.p, x[k]);
    }
#pragma unroll
    for (int k = 0; k < G::E; ++k) {
        u32 y[Q];
#pragma unroll
        for (int s = 0; s < Q; ++s) {
            u64 acc = 0;
#pragma unroll
            for (int i = 0; i < Q; ++i) acc += (u64)z[i][k] * c.v[pi][s][i];
            y[s] = rns_redc(acc, pi, m);
        }
#pragma unroll
        for (int s = 0; s < Q; ++s) z[s][k] = y[s];
    }
#pragma unroll
    for (int s = 0; s < Q; ++s) rns_store_a<LOGR, 1>(z[s], buf + s * M, t.u, t.col, a.logs);
}

// ---------------------------------------------------------------------------
// Last forward pass of both operands, pointwise product, first inverse pass.
// A sub-problem is R contiguous elements handled by U = 2^LB lanes of one
// warp (U * 2^LA = R), so the exchanges need no block barrier. Grid x: tiles
// of 256 * 2^LA elements, y: jobs, z: prime. bufA null: a square.
// ---------------------------------------------------------------------------
template <int LOGR>
struct RnsLast {
    static constexpr int LA = (LOGR + 1) / 2, LB = LOGR - LA;
    static constexpr int E = 1 << LA, U = 1 << LB, R = 1 << LOGR;
    static constexpr int NB = 1 << (LA - LB);
    static constexpr int THREADS = 256, SUBS = THREADS / U;
    // padded sub-problem: one word per 2^LB, and sub-problems of one warp
    // start U banks apart (mod 32), so both stages are free of conflicts
    static constexpr int RAW = R + (R >> LB);
    static constexpr int BS = LB >= 5 ? RAW : RAW + ((U - RAW % 32) + 32) % 32;
    static constexpr int SMEM = BS * SUBS;  // words
    static constexpr int MINB = E >= 32 ? 2 : 3;
    __device__ __forceinline__ static int sa(int row) { return row + (row >> LB); }
};

// The forward levels of the pass on V operands side by side (x[k * V + v]).
template <int LOGR, int V>
__device__ __forceinline__ void rns_last_fwd(u32* x, u32* sm, const uint2* T, u32 node, int u, const RnsMod& m) {
    using G = RnsLast<LOGR>;
    rns_dft_fwd<G::LA, V, false, false>(x, T, node, m);
#pragma unroll
    for (int v = 0; v < V; ++v) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < G::E; ++k) sm[G::sa(u + (k << G::LB))] = x[k * V + v];
        __syncwarp();
#pragma unroll
        for (int n = 0; n < G::NB; ++n)
#pragma unroll
            for (int k = 0; k < G::U; ++k)
                x[(n * G::U + k) * V + v] = sm[G::sa(((u + (n << G::LB)) << G::LB) + k)];
    }
#pragma unroll
    for (int n = 0; n < G::NB; ++n)
        rns_dft_fwd<G::LB, V, false, false>(x + n * G::U * V, T, (node << G::LA) + u + (n << G::LB), m);
}

template <int LOGR>
__global__ void __launch_bounds__(256, RnsLast<LOGR>::MINB) k_rns_fused(const RnsArgs a) {
    using G = RnsLast<LOGR>;
    extern __shared__ u32 smr[];
    const int pi = blockIdx.z;
    const RnsMod m(pi);
    const int u = threadIdx.x & (G::U - 1), sl = threadIdx.x >> G::LB;
    // Weighted parts read the same twiddles: blocks go round the parts, so that
    // the copies in L2 serve all of them. (A twiddle per point and direction:
    // with part after part each came from memory q times.)
    u32 sub = blockIdx.x * G::SUBS + sl;
    if (a.nmask != ~0u) sub = (blockIdx.x % a.q) * (a.nmask + 1) + (blockIdx.x / a.q) * G::SUBS + sl;
    if (((u64)sub << LOGR) >= a.nt) return;  // whole sub-problems: whole groups of U lanes
    u32* sm = smr + sl * G::BS;
    const u64 off = (u64)pi * a.nt + ((u64)sub << LOGR) + u;
    u32* bb = rns_buf(a, 1) + off;
    const uint2* T = a.tw + (u64)pi * a.ent;
    const uint2* Ti = a.twi + (u64)pi * a.ent;
    const u32 node = sub & a.nmask;
    u32 x[G::E];
    pdl_enter();
    if (!a.square) {
        const u32* ab = rns_buf(a, 0) + off;
        u32 y[2 * G::E];
#pragma unroll
        for (int k = 0; k < G::E; ++k) y[2 * k] = bb[k << G::LB], y[2 * k + 1] = ab[k << G::LB];
        rns_last_fwd<LOGR, 2>(y, sm, T, node, u, m);
#pragma unroll
        for (int k = 0; k < G::E; ++k) x[k] = rns_redc((u64)rns_red2(y[2 * k], m) * rns_red2(y[2 * k + 1], m), pi, m);
    } else {
#pragma unroll
        for (int k = 0; k < G::E; ++k) x[k] = bb[k << G::LB];
        rns_last_fwd<LOGR, 1>(x, sm, T, node, u, m);
#pragma unroll
        for (int k = 0; k < G::E; ++k) {
            const u32 v = rns_red2(x[k], m);
            x[k] = rns_redc((u64)v * v, pi, m);
        }
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < G::NB; ++n) {
        rns_dft_inv<G::LB, 1, false>(x + n * G::U, Ti, (node << G::LA) + u + (n << G::LB), m);
#pragma unroll
        for (int k = 0; k < G::U; ++k) sm[G::sa(((u + (n << G::LB)) << G::LB) + k)] = x[n * G::U + k];
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < G::E; ++k) x[k] = sm[G::sa(u + (k << G::LB))];
    rns_dft_inv<G::LA, 1, false>(x, Ti, node, m);
#pragma unroll
    for (int k = 0; k < G::E; ++k) bb[k << G::LB] = x[k];
}

}  // namespace b2m
