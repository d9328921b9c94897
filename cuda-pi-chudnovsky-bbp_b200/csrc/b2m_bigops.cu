// b2m_bigops.cu -- big-integer arithmetic on device-resident magnitudes, built
// on the NTT product: add / subtract with parallel carries, shifts, a Newton
// reciprocal, exact floor division, integer square root, and decimal
// conversion by divide and conquer with each level's divisions batched.
//
// Reference counterparts: divmod_knuth / div_fast (src/bignum_div.cpp:162-178),
// isqrt (src/bignum_div.cpp:189-204) and BigInt::to_decimal
// (src/bignum_div.cpp:239-267). Those are quadratic (schoolbook division, a
// Newton square root whose every step is a schoolbook division, repeated
// division by 10^9); these cost a few NTT products of the operand size each
// (O(M(n)) division and square root, O(M(n) log n) decimal conversion), and
// return the same integers: every result is exact, not approximate -- the
// Newton iterates only seed a quotient or root that a bounded correction loop
// then makes exact against the definition (remainder in [0, b), root with
// s^2 <= a < (s+1)^2).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstring>
#include <exception>
#include <vector>

#include "b2m.h"
#include "b2m_context.h"
#include "b2m_internal.h"
#include "carry_lookback.cuh"
#include "gp_scan.cuh"
#include "pdl.cuh"
#include "publish.cuh"
#include "school.cuh"

namespace b2m {
namespace big {

struct Err {
    b2m_status st;
};

// A device magnitude: n little-endian u32 limbs at p (n == 0 is zero).
struct DV {
    u32* p = nullptr;
    uint64_t n = 0;
};

inline void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw Err{cuda_status(e, what)};
}

// Stream-ordered memory of one API call, released when it returns: vectors
// are carved from a few growing blocks (an allocation call per vector was a
// large part of the host's time between kernels), one product workspace
// serves all products, which the stream runs one after the other.
class Scope {
public:
    Scope(Context* c, cudaStream_t s) : c_(c), s_(s), host_(c, s) {
        if (!host_.words()) {
            set_error("cannot pin host memory");
            throw Err{B2M_ERR_OUT_OF_MEMORY};
        }
        w_ = static_cast<unsigned long long*>(raw(256));
        const cudaError_t e = cudaMemsetAsync(w_, 0, 256, s);
        if (e != cudaSuccess) {
            release();
            throw Err{cuda_status(e, "cudaMemsetAsync")};
        }
    }
    ~Scope() { release(); }
    Scope(const Scope&) = delete;
    Scope& operator=(const Scope&) = delete;
    void* raw(uint64_t bytes) {
        bytes = (std::max<uint64_t>(bytes, 16) + 255) & ~255ull;
        if (bytes > left_) {
            // blocks double from 1 MiB to 64 MiB; what does not fit the
            // budget rounded up is taken as it is
            uint64_t block = std::max(bytes, next_);
            void* p = grab(block);
            if (!p && block > bytes) p = grab(block = bytes);
            if (!p) throw Err{st_};
            next_ = std::min<uint64_t>(2 * next_, 64ull << 20);
            if (block - bytes < left_) return p;  // the old block has more room left: keep carving it
            cur_ = static_cast<unsigned char*>(p);
            left_ = block;
        }
        void* p = cur_;
        cur_ += bytes;
        left_ -= bytes;
        return p;
    }
    // The workspace of products, which use it one after the other on s().
    void* workspace(uint64_t bytes) {
        if (bytes > ws_cap_) {
            ws_ = raw(bytes);
            ws_cap_ = bytes;
        }
        return ws_;
    }
    // Lookback slots of add/subtract kernels, zero between kernels.
    LookbackSlot* slots(uint64_t n) {
        if (n > slots_cap_) {
            const uint64_t cap = std::max<uint64_t>(64, 2 * n);
            slots_ = static_cast<LookbackSlot*>(raw(cap * sizeof(LookbackSlot)));
            slots_cap_ = cap;
            ck(cudaMemsetAsync(slots_, 0, cap * sizeof(LookbackSlot), s_), "cudaMemsetAsync");
        }
        return slots_;
    }
    DV vec(uint64_t n) { return {static_cast<u32*>(raw(4 * std::max<uint64_t>(n, 1))), n}; }
    DV zeros(uint64_t n) {
        DV d = vec(n);
        ck(cudaMemsetAsync(d.p, 0, 4 * std::max<uint64_t>(n, 1), s_), "cudaMemsetAsync");
        return d;
    }
    cudaStream_t s() const { return s_; }
    Context* c() const { return c_; }
    unsigned long long* word() const { return w_; }  // device scratch: words 8.. are a PubState
    HostLen publication() { return host_.next(); }
    // The words of the last publication (values from [1]).
    const u64* published() {
        ck(host_.wait(), "waiting for a kernel's result");
        return host_.words();
    }

private:
    void* grab(uint64_t bytes) {
        if (!budget_reserve(c_, bytes)) {
            set_error("HBM budget exhausted");
            st_ = B2M_ERR_OUT_OF_MEMORY;
            return nullptr;
        }
        void* p = nullptr;
        const cudaError_t e = cudaMallocAsync(&p, bytes, s_);
        if (e != cudaSuccess) {
            budget_release(c_, bytes);
            cudaGetLastError();
            st_ = cuda_status(e, "cudaMallocAsync");
            return nullptr;
        }
        v_.push_back({p, bytes});
        return p;
    }
    void release() {
        for (auto& a : v_) {
            cudaFreeAsync(a.first, s_);
            budget_release(c_, a.second);
        }
        v_.clear();
    }
    Context* c_;
    cudaStream_t s_;
    HostWords host_;
    unsigned long long* w_ = nullptr;
    std::vector<std::pair<void*, uint64_t>> v_;
    unsigned char* cur_ = nullptr;
    uint64_t left_ = 0, next_ = 1ull << 20;
    void* ws_ = nullptr;
    uint64_t ws_cap_ = 0;
    LookbackSlot* slots_ = nullptr;
    uint64_t slots_cap_ = 0;
    b2m_status st_ = B2M_OK;
};

// ---------------------------------------------------------------------------- kernels
constexpr int AS_T = 256, AS_L = ADD_LPT, AS_CH = AS_T * AS_L;  // limbs per block

// Device words of a call's publishing kernels, all zero between kernels: the
// last block of a kernel to finish zeroes them again.
struct PubState {
    unsigned long long top;
    u32 done, ticket, carry, early;
};

// All threads of the block: `top` is the thread's candidate for the trimmed
// length; (length, *word) is published, word null for none. A block whose top
// lies above `last` -- the elements from there on are its own -- has the
// length, and publishes without waiting for the others; without such a block
// (the result is short) the last one to finish does. The host launches the
// next step meanwhile, and that is ordered by the stream. Waiting for all
// blocks, a chain of three atomics and two fences, made a division of
// 400,003 / 200,001 limbs 1171 us long instead of 1135.
__device__ __forceinline__ void publish_top(unsigned long long top, u64 last, const u32* word, PubState* st,
                                            unsigned nblocks, LookbackSlot* slots, const HostLen& hl) {
    __shared__ bool s_last;
    __shared__ unsigned long long s_tops[32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, top, off);
        top = o > top ? o : top;
    }
    if ((threadIdx.x & 31) == 0) s_tops[threadIdx.x >> 5] = top;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < blockDim.x / 32; ++w) top = s_tops[w] > top ? s_tops[w] : top;
        if (top > last) {
            publish(hl, top, word ? *(volatile const u32*)word : 0);
            st->early = 1;
        } else if (top) {
            atomicMax(&st->top, top);
        }
        __threadfence();
        s_last = atomicAdd(&st->done, 1u) == nblocks - 1;
    }
    __syncthreads();
    if (!s_last) return;
    if (slots)
        for (unsigned i = threadIdx.x; i < nblocks; i += blockDim.x) slots[i].word = 0;
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned long long t = atomicMax(&st->top, 0ull);
        if (!*(volatile u32*)&st->early) publish(hl, t, word ? *(volatile const u32*)word : 0);
        st->top = 0;
        st->done = st->ticket = st->carry = st->early = 0;
    }
}

// `limb` (may be null): a limb published beside the length.
__global__ void k_top_pub(const u32* a, u64 n, const u32* limb, PubState* st, const HostLen hl) {
    pdl_enter();
    unsigned long long t = 0;
    for (u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (u64)gridDim.x * blockDim.x)
        if (a[k]) t = k + 1;
    publish_top(t, (n - 1) / blockDim.x * blockDim.x, limb, st, gridDim.x, nullptr, hl);
}

__global__ void k_limb_pub(const u32* a, u64 k, const HostLen hl) {
    pdl_enter();
    publish(hl, a[k]);
}

// a >= b over the warp's limbs (one a lane); *d = a - b. The borrows into the
// lanes by one integer addition, as in block_scan_gp.
__device__ __forceinline__ bool warp_ge_sub(u32 a, u32 b, int lane, u32* d) {
    const u32 G = __ballot_sync(0xFFFFFFFFu, a < b), P = __ballot_sync(0xFFFFFFFFu, a == b);
    const u64 s = (u64)(G | P) + G;
    *d = a - b - (((P ^ (u32)s) >> lane) & 1);
    return (s >> 32) == 0;
}

// One warp, a limb a lane: the root r = floor(sqrt(a)) of n <= 32 limbs (h =
// 0), or the seed floor((2^(64h) - 1) / r) of its reciprocal (h <= 16); the
// result's 32 limbs to out, its length published. A bit of the root, then of
// the quotient, a step (the schoolbook methods in base 2), each a compare and
// subtract of one integer addition's carries.
// What bounds it: the chain of at most 512 and 545 steps, each a few dependent
// ballots, shuffles and additions. The same by nested Newton divisions from the
// host, for the top 16 limbs, made square roots 0.6 to 0.7 ms longer.
constexpr int SEED_LIMBS = 32;
__global__ void __launch_bounds__(32) k_seed_sqrt(const u32* a, int n, int h, u32* out, const HostLen hl) {
    pdl_enter();
    const int lane = threadIdx.x;
    u32 v = lane < n ? a[lane] : 0u, res = 0, d;
    const u32 nz = __ballot_sync(0xFFFFFFFFu, v != 0);
    const int tl = nz ? 31 - __clz(nz) : 0;
    const u32 tv = __shfl_sync(0xFFFFFFFFu, v, tl);
    // res holds the bits found so far, shifted; p walks the even positions
    for (int p = nz ? (32 * tl + 31 - __clz(tv)) & ~1 : -1; p >= 0; p -= 2) {
        const u32 bit = lane == p >> 5 ? 1u << (p & 31) : 0u;
        const bool ge = warp_ge_sub(v, res | bit, lane, &d);
        const u32 up = __shfl_down_sync(0xFFFFFFFFu, res, 1);
        res = (res >> 1) | (lane < 31 ? up << 31 : 0u);
        if (ge) {
            v = d;
            res |= bit;
        }
    }
    u32 q = res;
    if (h > 0 && nz) {
        const u32 rz = __ballot_sync(0xFFFFFFFFu, res != 0);
        const int rl = 31 - __clz(rz);
        const int L = 32 * rl + 32 - __clz(__shfl_sync(0xFFFFFFFFu, res, rl));  // bits of the root
        // the first L - 1 ones of the numerator give no quotient bit
        const int ones = L - 1 - 32 * lane;
        u32 rem = ones >= 32 ? 0xFFFFFFFFu : (ones > 0 ? (1u << ones) - 1 : 0u);
        q = 0;
        for (int i = 64 * h - L; i >= 0; --i) {
            const u32 dn = __shfl_up_sync(0xFFFFFFFFu, rem, 1);
            rem = (rem << 1) | (lane > 0 ? dn >> 31 : 1u);
            if (warp_ge_sub(rem, res, lane, &d)) {
                rem = d;
                if (lane == i >> 5) q |= 1u << (i & 31);
            }
        }
    }
    out[lane] = q;
    const u32 qz = __ballot_sync(0xFFFFFFFFu, q != 0);
    if (lane == 0 && hl.host) publish(hl, 32 - __clz(qz));
}

// CTA-wide out = A +- B over n limbs (A: la limbs, B: lb limbs, or B null and
// the one-limb value bsmall), carry / borrow out returned to every thread.
// out may be A. blockDim a multiple of 32.
__device__ u32 cta_addsub(const u32* A, u64 la, const u32* B, u64 lb, u32 bsmall, u32* out, u64 n, int sub,
                          GP* ws, u32* s_carry) {
    if (threadIdx.x == 0) *s_carry = 0;
    __syncthreads();
    for (u64 c0 = 0; c0 < n; c0 += (u64)blockDim.x * ADD_LPT) {
        const u64 base = c0 + (u64)threadIdx.x * ADD_LPT;
        u32 av[ADD_LPT], bv[ADD_LPT];
        GP g{0, 1};
#pragma unroll
        for (int w = 0; w < ADD_LPT; ++w) {
            const u64 k = base + w;
            av[w] = k < n && k < la ? A[k] : 0u;
            bv[w] = k < n ? (B ? (k < lb ? B[k] : 0u) : (k == 0 ? bsmall : 0u)) : 0u;
            if (k < n) g = gp_then(g, limb_gp(av[w], bv[w], sub));
        }
        GP tot;
        const GP ex = block_scan_gp(g, ws, &tot);
        const u32 cin_chunk = *s_carry;
        u32 c = ex.g | (ex.p & cin_chunk);
#pragma unroll
        for (int w = 0; w < ADD_LPT; ++w) {
            const u64 k = base + w;
            if (k >= n) break;
            u32 r;
            if (!sub) {
                const u64 x = (u64)av[w] + bv[w] + c;
                r = (u32)x;
                c = (u32)(x >> 32);
            } else {
                const u64 x = (u64)av[w] - bv[w] - c;
                r = (u32)x;
                c = (u32)((x >> 63) & 1);
            }
            out[k] = r;
        }
        __syncthreads();
        if (threadIdx.x == 0) *s_carry = tot.g | (tot.p & cin_chunk);
        __syncthreads();
    }
    // every thread has read the carry before the next call clears it: callers
    // branch on it, and then meet barriers
    const u32 carry = *s_carry;
    __syncthreads();
    return carry;
}

// ---- Newton reciprocals of up to RECIP_MAX limbs by one block
constexpr int RECIP_MAX = 512, RECIP_BASE = 32, RECIP_W = 16, RECIP_T = 32 * RECIP_W;
struct RecipArgs {
    int nlev, h[6];                // levels' limbs, ascending; each from (h + 3) / 2 limbs, the first from the base
    int nx;                        // limbs of the base
    u32 x[RECIP_BASE + 3];
};

// out[0, la + lb) = a * b, all in shared memory, la + lb <= 2 RECIP_T, by the
// RECIP_T threads of the block: blocks of 128 columns, four a lane, each by as
// many warps as there are to a block (school.cuh has the method). cs: column
// sums, 3 * 128 * RECIP_W words.
__device__ void cta_mul(const u32* a, int la, const u32* b, int lb, u32* out, u32* cs, CState* st) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nc = la + lb;
    const int ncb = (nc + 127) / 128, parts = RECIP_W / ncb;
    if (warp < ncb * parts) {
        const int K0 = 128 * (warp % ncb), part = warp / ncb, k0 = K0 + 4 * lane;
        const int lo_i = K0 - lb + 1 > 0 ? K0 - lb + 1 : 0, hi_i = K0 + 127 < la - 1 ? K0 + 127 : la - 1;
        const int cnt = hi_i >= lo_i ? hi_i - lo_i + 1 : 0, per = (cnt + parts - 1) / parts;
        const int i0 = lo_i + part * per, i1 = i0 + per - 1 < hi_i ? i0 + per - 1 : hi_i;
        u32 lo[4] = {0, 0, 0, 0}, mid[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0}, w[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int j = k0 + c - i0;
            w[c] = j >= 0 && j < lb ? b[j] : 0u;
        }
        for (int i = i0; i <= i1; ++i) {
            const u32 x = a[i];
#pragma unroll
            for (int c = 0; c < 4; ++c) mac96(lo[c], mid[c], hi[c], x, w[c]);
            w[3] = w[2];
            w[2] = w[1];
            w[1] = w[0];
            const int j = k0 - i - 1;
            w[0] = j >= 0 && j < lb ? b[j] : 0u;
        }
        u32* c0 = cs + 3 * 128 * ncb * part + k0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            c0[c] = lo[c];
            c0[128 * ncb + c] = mid[c];
            c0[2 * 128 * ncb + c] = hi[c];
        }
    }
    __syncthreads();
    u32 limb[2];
    u64 carry = 0;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int k = 2 * t + c;
        u64 s0 = 0, s1 = 0, s2 = 0;
        if (k < nc)
            for (int p = 0; p < parts; ++p) {
                const u32* c0 = cs + 3 * 128 * ncb * p + k;
                s0 += c0[0];
                s1 += c0[128 * ncb];
                s2 += c0[2 * 128 * ncb];
            }
        s0 += carry;
        limb[c] = (u32)s0;
        carry = (s0 >> 32) + s1 + (s2 << 32);
    }
    bool has;
    CState agg;
    const CState ex = block_scan_carry(group_state<2>(limb, carry), &has, &agg, st);
    group_add_carry<2>(limb, has ? cs_eval(ex, 0) : 0);
#pragma unroll
    for (int c = 0; c < 2; ++c)
        if (2 * t + c < nc) out[2 * t + c] = limb[c];
    __syncthreads();
}

// The largest k + 1 with v[k] != 0, by the block.
__device__ int cta_top(const u32* v, int n) {
    __shared__ int s_n;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    int t = 0;
    for (int k = threadIdx.x; k < n; k += blockDim.x)
        if (v[k]) t = k + 1;
    if (t) atomicMax(&s_n, t);
    __syncthreads();
    const int r = s_n;
    __syncthreads();
    return r;
}

// st[0, e) = |2^(32e) - T| for the T < 2^(32(e + 1)) in st, whose limb e is top.
__device__ void cta_error(u32* st, int e, u32 top) {
    __shared__ int s_low;
    if (top) return;  // the low limbs are it
    if (threadIdx.x == 0) s_low = e;
    __syncthreads();
    for (int k = threadIdx.x; k < e; k += RECIP_T)
        if (st[k]) {
            atomicMin(&s_low, k);
            break;
        }
    __syncthreads();
    const int low = s_low;
    for (int k = threadIdx.x; k < e; k += RECIP_T) st[k] = k > low ? ~st[k] : 0u - st[k];
    __syncthreads();
}

// recip's steps for the top limbs y[0, h[nlev - 1]) of a divisor, one level
// after the other, the same integers as from the host: X_h = X_l 2^(32(h-l)) +
// X_l (2^(32(h+l)) - Y_h X_l) / 2^(64 l). X to out (h + 2 limbs of the last
// level); publishes its trimmed length, 0 when the iteration diverged.
// What bounds it: the products' multiply-adds on one SM, 2 x 512 x 257 of them
// at the last level. From the host a level is four launches, each waited for:
// the division of pi to 10,000 digits, 1,000 limbs, 0.48 ms, and 0.34 so.
__global__ void __launch_bounds__(RECIP_T) k_recip(const u32* y, const RecipArgs a, u32* out, const HostLen hl) {
    __shared__ u32 sy[RECIP_MAX], sx[RECIP_MAX + 2], st[RECIP_MAX + RECIP_MAX / 2 + 16], sd[2 * RECIP_T];
    __shared__ u32 cs[3 * 128 * RECIP_W];
    __shared__ CState sc[RECIP_W];
    __shared__ GP ws[33];
    __shared__ u32 s_carry;
    pdl_enter();
    const int t = threadIdx.x, H = a.h[a.nlev - 1];
    for (int k = t; k < H; k += RECIP_T) sy[k] = y[k];
    if (t < RECIP_BASE + 2) sx[t] = t < a.nx ? a.x[t] : 0u;
    __syncthreads();
    for (int lev = 0; lev < a.nlev; ++lev) {
        const int h = a.h[lev], l = (h + 3) / 2, e = h + l;
        cta_mul(sx, l + 2, sy + (H - h), h, st, cs, sc);  // Y_h X_l: e + 2 limbs
        const u32 top = st[e];
        if (top > 1 || st[e + 1]) {
            if (t == 0) publish(hl, 0);
            return;
        }
        cta_error(st, e, top);
        const int en = cta_top(st, e);
        if (en > h + 2) {
            if (t == 0) publish(hl, 0);
            return;
        }
        int cn = 0;  // limbs of X_l |E| / 2^(64 l)
        if (en) {
            cta_mul(sx, l + 2, st, en, sd, cs, sc);
            cn = l + 2 + en - 2 * l > 0 ? l + 2 + en - 2 * l : 0;
        }
        // X_h = X_l 2^(32 (h - l)) +- that, by way of st
        for (int k = t; k < h + 2; k += RECIP_T) st[k] = k >= h - l ? sx[k - (h - l)] : 0u;
        __syncthreads();
        if (cn) cta_addsub(st, h + 2, sd + 2 * l, cn, 0, sx, h + 2, top != 0, ws, &s_carry);
        else
            for (int k = t; k < h + 2; k += RECIP_T) sx[k] = st[k];
        __syncthreads();
    }
    const int n = cta_top(sx, H + 2);
    for (int k = t; k < H + 2; k += RECIP_T) out[k] = sx[k];
    if (t == 0) publish(hl, n);
}

// rsqrt_approx's steps up to RSQRT_MAX limbs for nh, the top 2 h[nlev - 1]
// limbs (n of them not zero above), from the seed of (h[0] + 3) / 2 limbs, the
// same integers as from the host: with y of l limbs,
//     U = N_h y^2, y_h = y 2^(32(h-l)) +- y |2^(32(2h+2l)) - U| / 2^(32(h+3l) + 1).
// Bounded as k_recip; from the host a level is seven launches.
constexpr int RSQRT_MAX = 224;
struct RsqrtArgs {
    int nlev, h[6];
};
__global__ void __launch_bounds__(RECIP_T) k_rsqrt(const u32* nh, int n, const u32* seed, const RsqrtArgs a,
                                                   u32* out, const HostLen hl) {
    __shared__ u32 sn[2 * RSQRT_MAX], sy[RSQRT_MAX + 2], ss[RSQRT_MAX + 16], su[2 * RECIP_T], sd[2 * RECIP_T];
    __shared__ u32 cs[3 * 128 * RECIP_W];
    __shared__ CState sc[RECIP_W];
    __shared__ GP ws[33];
    __shared__ u32 s_carry;
    pdl_enter();
    const int t = threadIdx.x, H = a.h[a.nlev - 1];
    for (int k = t; k < 2 * H; k += RECIP_T) sn[k] = k < n ? nh[k] : 0u;
    for (int k = t; k < RSQRT_MAX + 2; k += RECIP_T) sy[k] = k < SEED_LIMBS ? seed[k] : 0u;
    __syncthreads();
    for (int lev = 0; lev < a.nlev; ++lev) {
        const int h = a.h[lev], l = (h + 3) / 2, e = 2 * h + 2 * l;
        cta_mul(sy, l + 2, sy, l + 2, ss, cs, sc);
        cta_mul(ss, 2 * l + 4, sn + 2 * (H - h), 2 * h, su, cs, sc);  // e + 4 limbs
        const u32 top = su[e];
        if (top > 1 || (su[e + 1] | su[e + 2] | su[e + 3])) {
            if (t == 0) publish(hl, 0);
            return;
        }
        cta_error(su, e, top);
        const int en = cta_top(su, e), sh = h + 3 * l;
        int cn = 0;
        if (en) {
            cta_mul(sy, l + 2, su, en, sd, cs, sc);
            cn = l + 2 + en > sh ? l + 2 + en - sh : 0;
            for (int k = t; k < cn; k += RECIP_T)
                ss[k] = sd[sh + k] >> 1 | (k + 1 < cn ? sd[sh + k + 1] << 31 : 0u);
        }
        for (int k = t; k < h + 2; k += RECIP_T) su[k] = k >= h - l ? sy[k - (h - l)] : 0u;
        __syncthreads();
        if (cn) cta_addsub(su, h + 2, ss, cn, 0, sy, h + 2, top != 0, ws, &s_carry);
        else
            for (int k = t; k < h + 2; k += RECIP_T) sy[k] = su[k];
        __syncthreads();
    }
    const int m = cta_top(sy, H + 2);
    for (int k = t; k < H + 2; k += RECIP_T) out[k] = sy[k];
    if (t == 0) publish(hl, m);
}

// out = a 2^(32 a_off) +- b mod 2^(32n) in one pass, the trimmed length and
// the carry or borrow out published. out may be a (a_off = 0) or b. One block
// per 2048 limbs; the carry into a block comes by decoupled lookback, as in
// the carry kernels.
__global__ void __launch_bounds__(AS_T) k_addsub_pub(const u32* A, u64 a_off, u64 la, const u32* B, u64 lb, u64 n,
                                                     int sub, u32* out, LookbackSlot* slots, PubState* st,
                                                     const HostLen hl, u32* err) {
    __shared__ GP ws[AS_T / 32 + 1];
    __shared__ u32 s_chunk, s_cin;
    pdl_enter();
    u32 chunk = 0;
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) s_chunk = atomicAdd(&st->ticket, 1u);
        __syncthreads();
        chunk = s_chunk;
    }
    const u64 base = (u64)chunk * AS_CH + (u64)threadIdx.x * AS_L;
    u32 av[AS_L], bv[AS_L];
    GP g{0, 1};
#pragma unroll
    for (int w = 0; w < AS_L; ++w) {
        const u64 k = base + w;
        av[w] = k >= a_off && k - a_off < la && k < n ? A[k - a_off] : 0u;
        bv[w] = k < lb && k < n ? B[k] : 0u;
        if (k < n) g = gp_then(g, limb_gp(av[w], bv[w], sub));
    }
    GP tot;
    const GP ex = block_scan_gp(g, ws, &tot);
    u32 cin = 0;
    if (gridDim.x > 1) {
        if (threadIdx.x < 32) {
            // the block as a carry function: constant, or passing 0 and 1 through
            const CState agg{tot.g, tot.p && !tot.g ? 1ull : CS_NEVER};
            const u64 c = warp_lookback(slots, chunk, agg, err);
            if (threadIdx.x == 0) {
                if (agg.t != CS_NEVER) st_release(&slots[chunk].word, (cs_eval(agg, c) << 2) | SLOT_INCL);
                s_cin = (u32)c;
            }
        }
        __syncthreads();
        cin = s_cin;
    }
    u32 c = ex.g | (ex.p & cin);
    unsigned long long top = 0;
#pragma unroll
    for (int w = 0; w < AS_L; ++w) {
        const u64 k = base + w;
        if (k >= n) break;
        u32 r;
        if (!sub) {
            const u64 x = (u64)av[w] + bv[w] + c;
            r = (u32)x;
            c = (u32)(x >> 32);
        } else {
            const u64 d = (u64)av[w] - bv[w] - c;
            r = (u32)d;
            c = (u32)((d >> 63) & 1);
        }
        out[k] = r;
        if (r) top = k + 1;
    }
    if (chunk == gridDim.x - 1 && threadIdx.x == 0) st->carry = tot.g | (tot.p & cin);
    publish_top(top, (u64)(gridDim.x - 1) * AS_CH, &st->carry, st, gridDim.x, gridDim.x > 1 ? slots : nullptr, hl);
}

// out[k] = (a * 2^(32*wl + bits))[k], k < nout (bits in [0, 32)); publishes
// the trimmed length.
__global__ void k_shl(const u32* a, u64 na, int bits, u64 wl, u32* out, u64 nout, PubState* st, const HostLen hl) {
    pdl_enter();
    unsigned long long t = 0;
    for (u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x; k < nout; k += (u64)gridDim.x * blockDim.x) {
        u32 v = 0;
        if (k >= wl && k - wl < na) v = a[k - wl] << bits;
        if (bits && k >= wl + 1 && k - wl - 1 < na) v |= a[k - wl - 1] >> (32 - bits);
        out[k] = v;
        if (v) t = k + 1;
    }
    publish_top(t, (nout - 1) / blockDim.x * blockDim.x, nullptr, st, gridDim.x, nullptr, hl);
}

// out[k] = floor(a / 2^(32*wl + bits))[k], k < nout (bits in [0, 32));
// publishes the trimmed length.
__global__ void k_shr(const u32* a, u64 na, int bits, u64 wl, u32* out, u64 nout, PubState* st, const HostLen hl) {
    pdl_enter();
    unsigned long long t = 0;
    for (u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x; k < nout; k += (u64)gridDim.x * blockDim.x) {
        u32 v = 0;
        if (k + wl < na) v = a[k + wl] >> bits;
        if (bits && k + wl + 1 < na) v |= a[k + wl + 1] << (32 - bits);
        out[k] = v;
        if (v) t = k + 1;
    }
    publish_top(t, (nout - 1) / blockDim.x * blockDim.x, nullptr, st, gridDim.x, nullptr, hl);
}

inline unsigned grid_for(uint64_t n, unsigned threads = 256) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + threads - 1) / threads, 65535));
}

// ---------------------------------------------------------------------------- host ops
PubState* pub(Scope& S) { return reinterpret_cast<PubState*>(S.word() + 8); }

// Grids of publishing kernels: each block ends in an atomic on one word.
inline unsigned pub_grid(uint64_t n) { return std::min(grid_for(n), 1024u); }

uint64_t top_len(Scope& S, DV a) {
    if (a.n == 0) return 0;
    ck(launch_pdl(k_top_pub, pub_grid(a.n), 256, 0, S.s(), a.p, a.n, nullptr, pub(S), S.publication()),
       "k_top_pub");
    return S.published()[1];
}

DV trim(Scope& S, DV a) { return {a.p, top_len(S, a)}; }

// The low n limbs of a, trimmed, and limb n.
DV split_at(Scope& S, DV a, uint64_t n, u32* limb) {
    ck(launch_pdl(k_top_pub, pub_grid(n), 256, 0, S.s(), a.p, n, a.p + n, pub(S), S.publication()), "k_top_pub");
    const u64* h = S.published();
    *limb = (u32)h[2];
    return {a.p, h[1]};
}

// out = a 2^(32 a_off) +- b mod 2^(32 out.n): the carry (add) or borrow (sub)
// out, and the trimmed result.
struct Sum {
    u32 carry;
    DV v;
};
Sum addsub(Scope& S, DV a, DV b, DV out, bool sub, uint64_t a_off = 0) {
    const uint64_t n = out.n;
    if (n == 0) return {0, out};
    const uint64_t nb = (n + AS_CH - 1) / AS_CH;
    LookbackSlot* slots = nb > 1 ? S.slots(nb) : nullptr;
    ck(launch_pdl(k_addsub_pub, (unsigned)nb, AS_T, 0, S.s(), a.p, a_off, a.n, b.p, b.n, n, sub ? 1 : 0, out.p, slots,
                  pub(S), S.publication(), S.c()->d_err),
       "k_addsub_pub");
    const u64* h = S.published();
    return {(u32)h[2], {out.p, h[1]}};
}

DV upload(Scope& S, const std::vector<u32>& h) {
    DV d = S.vec(h.size());
    if (!h.empty()) ck(cudaMemcpyAsync(d.p, h.data(), 4 * h.size(), cudaMemcpyHostToDevice, S.s()), "H2D");
    ck(cudaStreamSynchronize(S.s()), "cudaStreamSynchronize");  // h may be a temporary
    return d;
}

std::vector<u32> download(Scope& S, DV d) {
    std::vector<u32> h(d.n);
    if (d.n) ck(cudaMemcpyAsync(h.data(), d.p, 4 * d.n, cudaMemcpyDeviceToHost, S.s()), "D2H");
    ck(cudaStreamSynchronize(S.s()), "cudaStreamSynchronize");
    return h;
}

u32 limb_at(Scope& S, DV d, uint64_t k) {
    ck(launch_pdl(k_limb_pub, 1, 1, 0, S.s(), d.p, k, S.publication()), "k_limb_pub");
    return (u32)S.published()[1];
}

DV copy(Scope& S, DV a, uint64_t cap) {
    DV d = S.zeros(std::max(cap, a.n));
    if (a.n) ck(cudaMemcpyAsync(d.p, a.p, 4 * a.n, cudaMemcpyDeviceToDevice, S.s()), "D2D");
    d.n = a.n;
    return d;
}

// a * 2^(32 wl + bits), trimmed.
// normalizes: bits take the top limb's leading zeros (wl = 0), so the length
// stays and is not waited for.
DV shl(Scope& S, DV a, uint64_t wl, int bits, bool normalizes = false) {
    if (a.n == 0) return a;
    const uint64_t n = a.n + wl + 1;
    DV d = S.vec(n);
    ck(launch_pdl(k_shl, pub_grid(n), 256, 0, S.s(), a.p, a.n, bits, wl, d.p, n, pub(S), S.publication()), "k_shl");
    return {d.p, normalizes ? a.n : S.published()[1]};
}

// floor(a / 2^(32 wl + bits)), trimmed.
DV shr(Scope& S, DV a, uint64_t wl, int bits) {
    if (a.n <= wl) return {a.p, 0};
    const uint64_t n = a.n - wl;
    DV d = S.vec(n);
    ck(launch_pdl(k_shr, pub_grid(n), 256, 0, S.s(), a.p, a.n, bits, wl, d.p, n, pub(S), S.publication()), "k_shr");
    return {d.p, S.published()[1]};
}

// a + delta for delta in {-1, +1} (a + 1 may grow by one limb; a - 1 needs a > 0).
DV add_one(Scope& S, DV a, bool minus) {
    static const u32 one_h = 1;
    DV one = S.vec(1);
    ck(cudaMemcpyAsync(one.p, &one_h, 4, cudaMemcpyHostToDevice, S.s()), "H2D");
    return addsub(S, a, one, S.vec(a.n + 1), minus).v;
}

// The NTT product, trimmed.
DV mul(Scope& S, DV a, DV b) {
    if (a.n == 0 || b.n == 0) return {a.p ? a.p : b.p, 0};
    int logn = 0;
    const b2m_status st = check_sizes(a.n, b.n, &logn);
    if (st != B2M_OK) throw Err{st};
    Context* c = S.c();
    Plan p = product_plan(c, a.n, b.n);
    ck(twtable_ensure(c, p, S.s()), "twiddle table");
    DV out = S.vec(a.n + b.n);
    void* ws = p.npass ? S.workspace(workspace_bytes_plan(p)) : nullptr;
    uint64_t* d_len = reinterpret_cast<uint64_t*>(S.word() + 2);
    const bool published = p.npass == 0 || p.rns;
    ck(launch_product(a.p, a.n, b.p, b.n, out.p, d_len, ws, p, c->tw, c->d_err, S.s(), nullptr, nullptr,
                      published ? S.publication() : HostLen{}),
       "product");
    if (published) {
        out.n = S.published()[1];
        return out;
    }
    unsigned long long h = 0;
    ck(cudaMemcpyAsync(&h, d_len, 8, cudaMemcpyDeviceToHost, S.s()), "D2H");
    ck(cudaStreamSynchronize(S.s()), "cudaStreamSynchronize");
    out.n = h;  // the sticky device error word is checked once, when the call ends
    return out;
}

// ---------------------------------------------------------------------------- small host arithmetic
// floor((2^(64h) - 1) / Y) for an h-limb Y whose top bit is set: schoolbook
// long division on 32-bit digits (Knuth, TAOCP vol. 2, 4.3.1, algorithm D),
// the numerator being 2h all-ones limbs. Seeds the Newton reciprocal.
std::vector<u32> recip_small(const std::vector<u32>& Y) {
    const size_t n = Y.size();
    std::vector<u32> q(n + 1, 0);
    if (n == 1) {
        const u64 v = ~0ull / Y[0];
        q[0] = (u32)v;
        q[1] = (u32)(v >> 32);
    } else {
        std::vector<u32> un(2 * n + 1, 0xFFFFFFFFu);
        un[2 * n] = 0;
        const u64 b = 1ull << 32;
        for (long j = (long)n; j >= 0; --j) {
            const u64 num = ((u64)un[j + n] << 32) | un[j + n - 1];
            u64 qhat = num / Y[n - 1], rhat = num % Y[n - 1];
            while (qhat >= b || qhat * Y[n - 2] > ((rhat << 32) | un[j + n - 2])) {
                --qhat;
                rhat += Y[n - 1];
                if (rhat >= b) break;
            }
            int64_t k = 0, t;
            for (size_t i = 0; i < n; ++i) {
                const u64 p = qhat * Y[i];
                t = (int64_t)un[i + j] - k - (int64_t)(p & 0xFFFFFFFFull);
                un[i + j] = (u32)t;
                k = (int64_t)(p >> 32) - (t >> 32);
            }
            t = (int64_t)un[j + n] - k;
            un[j + n] = (u32)t;
            if (t < 0) {
                --qhat;
                u64 c = 0;
                for (size_t i = 0; i < n; ++i) {
                    const u64 s = (u64)un[i + j] + Y[i] + c;
                    un[i + j] = (u32)s;
                    c = s >> 32;
                }
                un[j + n] += (u32)c;
            }
            q[j] = (u32)qhat;
        }
    }
    while (!q.empty() && q.back() == 0) q.pop_back();
    return q;
}
// ---------------------------------------------------------------------------- Newton reciprocal
// Top h limbs of the normalized Bn (n limbs), or Bn * 2^(32(h - n)) if h > n.
DV top_limbs(Scope& S, DV Bn, uint64_t h) {
    if (h <= Bn.n) return {Bn.p + (Bn.n - h), h};
    DV d = S.zeros(h);
    ck(cudaMemcpyAsync(d.p + (h - Bn.n), Bn.p, 4 * Bn.n, cudaMemcpyDeviceToDevice, S.s()), "D2D");
    return d;
}

// X ~ 2^(64h) / Y_h, Y_h = top_limbs(Bn, h) (top bit set), within a few units:
// X_h = X_l 2^(32(h-l)) + X_l (2^(32(h+l)) - Y_h X_l) / 2^(64 l), with the
// lower precision l = floor((h + 3) / 2) seeding each step (Newton doubles
// the correct limbs; the +3 keeps a guard limb).
DV recip(Scope& S, DV Bn, uint64_t h) {
    DV Y = top_limbs(S, Bn, h);
    if (h <= RECIP_BASE) return trim(S, upload(S, recip_small(download(S, Y))));
    if (h <= RECIP_MAX) {
        uint64_t hs[8] = {h};
        int n = 1;
        while (hs[n - 1] > RECIP_BASE) {
            hs[n] = (hs[n - 1] + 3) / 2;
            ++n;
        }
        const std::vector<u32> x = recip_small(download(S, {Y.p + (h - hs[n - 1]), hs[n - 1]}));
        RecipArgs a{};
        a.nlev = n - 1;
        for (int i = 0; i < a.nlev; ++i) a.h[i] = (int)hs[a.nlev - 1 - i];
        a.nx = (int)x.size();
        std::copy(x.begin(), x.end(), a.x);
        DV X = S.vec(h + 2);
        ck(launch_pdl(k_recip, 1, RECIP_T, 0, S.s(), Y.p, a, X.p, S.publication()), "k_recip");
        X.n = S.published()[1];
        if (X.n == 0) {
            set_error("Newton reciprocal diverged");
            throw Err{B2M_ERR_INTERNAL};
        }
        return X;
    }
    const uint64_t l = (h + 3) / 2;
    DV Xl = recip(S, Bn, l);
    DV T = mul(S, Y, Xl);
    const uint64_t e = h + l;
    DV E;
    bool neg = false;
    if (T.n <= e) {  // E = 2^(32e) - T >= 0
        E = addsub(S, DV{T.p, 0}, T, S.vec(e), true).v;
    } else {  // T = 2^(32e) + E', 0 <= E' < 2^(32e)
        u32 top = 0;
        if (T.n == e + 1) E = split_at(S, T, e, &top);
        if (top != 1) {
            set_error("Newton reciprocal diverged");
            throw Err{B2M_ERR_INTERNAL};
        }
        neg = true;
    }
    DV D = mul(S, Xl, E);
    DV corr = D.n > 2 * l ? DV{D.p + 2 * l, D.n - 2 * l} : DV{D.p, 0};
    return addsub(S, Xl, corr, S.vec(h + 2), neg, h - l).v;
}

// ---------------------------------------------------------------------------- division
constexpr int MAX_FIX = 16;  // correction steps allowed after a Newton estimate

// q = floor(a / b), r = a mod b for trimmed a, b (b > 0). The estimate
// q~ = floor(top(a') X / 2^(32 s)) from the reciprocal of the normalized
// divisor is within a few units; r = a - q~ b then moves q~ to the exact
// quotient one unit at a time.
void divmod(Scope& S, DV a, DV b, DV* q, DV* r) {
    if (b.n == 0) {
        set_error("division by zero");
        throw Err{B2M_ERR_INVALID_ARGUMENT};
    }
    if (a.n < b.n) {
        *q = {a.p, 0};
        *r = a;
        return;
    }
    const int sh = __builtin_clz(limb_at(S, b, b.n - 1));
    DV Bn = sh ? shl(S, b, 0, sh, true) : b;
    DV An = sh ? shl(S, a, 0, sh) : a;
    const uint64_t n = b.n;
    const uint64_t m = An.n - n + 1;  // quotient limbs, at most
    const uint64_t L = m + 2;
    DV X = recip(S, Bn, L);          // ~ 2^(32(L + n)) / Bn
    const uint64_t k = An.n > L + 1 ? An.n - (L + 1) : 0;
    DV P = mul(S, DV{An.p + k, An.n - k}, X);
    const uint64_t s = L + n - k;
    DV Q{P.p + std::min(s, P.n), P.n > s ? P.n - s : 0};
    DV QB = mul(S, Q, b);
    const uint64_t w = std::max(a.n, QB.n) + 1;
    DV R = S.vec(w);
    Sum rs = addsub(S, a, QB, R, true);
    bool negative = rs.carry != 0;
    int it = 0;
    while (negative) {  // two's complement R < 0: add b back
        rs = addsub(S, R, b, R, false);
        if (rs.carry) negative = false;
        Q = add_one(S, Q, true);
        if (++it > MAX_FIX) break;
    }
    while (it <= MAX_FIX) {  // R >= b: subtract it
        DV T = S.vec(w);
        const Sum ts = addsub(S, R, b, T, true);
        if (ts.carry) break;
        R = T;
        rs = ts;
        Q = add_one(S, Q, false);
        ++it;
    }
    if (it > MAX_FIX) {
        set_error("division correction did not converge");
        throw Err{B2M_ERR_INTERNAL};
    }
    *q = Q;
    *r = rs.v;
}

// ---------------------------------------------------------------------------- square root
// floor(sqrt(N)) of at most 32 limbs (h = 0), or floor((2^(64h) - 1) / that).
DV seed_sqrt(Scope& S, DV N, uint64_t h) {
    DV d = S.vec(SEED_LIMBS);
    ck(launch_pdl(k_seed_sqrt, 1, 32, 0, S.s(), N.p, (int)N.n, (int)h, d.p, S.publication()), "k_seed_sqrt");
    return {d.p, S.published()[1]};
}

// Y ~ 2^(64h) / sqrt(N_h), N_h = floor(N / 2^(32(2k - 2h))), by Newton on the
// reciprocal square root, y <- y + y (1 - N y^2) / 2: three products a step
// and no division. The seed (h <= 16) is floor((2^(64h) - 1) / isqrt(N_h))
// from the exact root; each step starts from l = floor((h + 3) / 2) limbs.
DV rsqrt_approx(Scope& S, DV N, uint64_t k, uint64_t h) {
    const uint64_t drop = 2 * k - 2 * h;
    DV Nh = N.n > drop ? DV{N.p + drop, N.n - drop} : DV{N.p, 0};
    if (2 * h <= SEED_LIMBS) return seed_sqrt(S, Nh, h);
    if (h <= RSQRT_MAX) {
        uint64_t hs[8] = {h};
        int n = 1;
        while (2 * hs[n - 1] > SEED_LIMBS) {
            hs[n] = (hs[n - 1] + 3) / 2;
            ++n;
        }
        RsqrtArgs a{};
        a.nlev = n - 1;
        for (int i = 0; i < a.nlev; ++i) a.h[i] = (int)hs[a.nlev - 1 - i];
        const uint64_t cut = 2 * k - 2 * hs[n - 1];
        DV seed = S.vec(SEED_LIMBS), Y = S.vec(h + 2);
        ck(launch_pdl(k_seed_sqrt, 1, 32, 0, S.s(), N.p + cut, (int)(N.n - cut), (int)hs[n - 1], seed.p, HostLen{}),
           "k_seed_sqrt");
        ck(launch_pdl(k_rsqrt, 1, RECIP_T, 0, S.s(), Nh.p, (int)Nh.n, seed.p, a, Y.p, S.publication()), "k_rsqrt");
        Y.n = S.published()[1];
        if (Y.n == 0) {
            set_error("Newton reciprocal square root diverged");
            throw Err{B2M_ERR_INTERNAL};
        }
        return Y;
    }
    const uint64_t l = (h + 3) / 2;
    DV Y0 = shl(S, rsqrt_approx(S, N, k, l), h - l, 0);
    DV U = mul(S, Nh, mul(S, Y0, Y0));  // ~ 2^(128h)
    const uint64_t e = 4 * h;
    DV E;
    bool neg = false;
    if (U.n <= e) {  // E = 2^(32e) - U >= 0
        E = addsub(S, DV{U.p, 0}, U, S.vec(e), true).v;
    } else {  // U = 2^(32e) + E'
        u32 top = 0;
        if (U.n == e + 1) E = split_at(S, U, e, &top);
        if (top != 1) {
            set_error("Newton reciprocal square root diverged");
            throw Err{B2M_ERR_INTERNAL};
        }
        neg = true;
    }
    DV corr = shr(S, mul(S, Y0, E), e, 1);  // Y0 |E| / 2^(32e + 1)
    return addsub(S, Y0, corr, S.vec(std::max(Y0.n, corr.n) + 1), neg).v;
}

// floor(sqrt(N)) for trimmed N: up to 32 limbs bit by bit (k_seed_sqrt), above
// that the estimate N * Y / 2^(64k) from the reciprocal square root, whose
// remainder R = N - s^2 then moves s until 0 <= R <= 2s.
DV isqrt(Scope& S, DV N) {
    if (N.n == 0) return N;
    if (N.n <= SEED_LIMBS) return seed_sqrt(S, N, 0);
    const uint64_t k = (N.n + 1) / 2;
    DV s = shr(S, mul(S, N, rsqrt_approx(S, N, k, k)), 2 * k, 0);
    DV SQ = mul(S, s, s);
    const uint64_t w = std::max(N.n, SQ.n) + 2;
    DV R = S.vec(w);
    bool negative = addsub(S, N, SQ, R, true).carry != 0;
    int it = 0;
    while (negative && it <= MAX_FIX) {  // N - (s-1)^2 = R + 2s - 1
        DV twice = shl(S, s, 0, 1);
        DV d = add_one(S, twice, true);
        if (addsub(S, R, d, R, false).carry) negative = false;
        s = add_one(S, s, true);
        ++it;
    }
    while (it <= MAX_FIX) {  // N - (s+1)^2 = R - (2s + 1)
        DV d = add_one(S, shl(S, s, 0, 1), false);
        DV T = S.vec(w);
        if (addsub(S, R, d, T, true).carry) break;
        R = T;
        s = add_one(S, s, false);
        ++it;
    }
    if (it > MAX_FIX) {
        set_error("square-root correction did not converge");
        throw Err{B2M_ERR_INTERNAL};
    }
    return s;
}

// ---------------------------------------------------------------------------- decimal conversion
// Divide and conquer with powers P_j = 10^(9 * 2^j): a node of level j holds
// a value below P_j^2; dividing it by P_j gives two nodes below P_j (quotient
// first: the more significant digits). All nodes of a level have the same
// size and divisor, so each level is two batched products (the quotient
// estimate from P_j's reciprocal, then estimate * P_j) and one kernel that
// makes every quotient and remainder exact. Nodes below 10^72 are printed by
// one thread each.

constexpr int DC_LEAF_J = 2;     // leaves: values below P_2^2 = 10^72
constexpr int DC_LEAF_LIMBS = 8;  // 10^72 < 2^240
constexpr int DC_LEAF_GROUPS = 8;

// Job i multiplies a + i*sa by b + i*sb. With `spec` (b shared, sb = 0, its
// spectrum already in spec), b becomes every job's first operand with bufA =
// spec, and the workspace holds only bufB and the carry scratch.
__global__ void k_dc_jobs(const u32* a, u64 sa, u64 na, const u32* b, u64 sb, u64 nb, u32* out, u64 so,
                          unsigned long long* lens, ProdJob* jobs, u64 njobs, unsigned char* ws, u64 wss, u64 npts,
                          u64* spec) {
    pdl_enter();
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= njobs) return;
    ProdJob J{};
    J.a = a + i * sa;
    J.na = na;
    J.b = b + i * sb;
    J.nb = nb;
    if (spec) {
        J.a = b;
        J.na = nb;
        J.b = a + i * sa;
        J.nb = na;
    }
    J.out = out + i * so;
    J.out_len = lens + i;
    if (wss) {
        const u64 n = npts;
        unsigned char* w = ws + i * wss;
        unsigned char* scratch;
        if (spec) {
            J.bufA = spec;
            J.bufB = reinterpret_cast<u64*>(w);
            scratch = w + 8 * n;
        } else {
            J.bufA = reinterpret_cast<u64*>(w);
            J.bufB = J.bufA + n;
            scratch = w + 16 * n;
        }
        J.slots = reinterpret_cast<LookbackSlot*>(scratch);
        J.ticket = reinterpret_cast<u32*>(scratch + (n / CARRY_CHUNK) * sizeof(LookbackSlot));
    }
    jobs[i] = J;
}

// The one-job table that transforms b into spec.
__global__ void k_dc_spec_job(const u32* b, u64 nb, u64* spec, ProdJob* job) {
    pdl_enter();
    ProdJob J{};
    J.a = b;
    J.na = nb;
    J.bufA = spec;
    *job = J;
}

__global__ void k_dc_zero_ws(const ProdJob* jobs, u64 njobs, u64 scratch_words) {
    pdl_enter();
    const u64 j = blockIdx.x;
    if (j >= njobs) return;
    unsigned long long* s = reinterpret_cast<unsigned long long*>(jobs[j].slots);
    for (u64 i = threadIdx.x; i < scratch_words; i += blockDim.x) s[i] = 0;
    if (threadIdx.x == 0) *jobs[j].out_len = 0;
}

// out_i = a_i * b_i for m products of na x nb limbs (strides sa, sb, so; sb = 0
// shares one b), as size-bucketed launches of the batch path. A shared b is
// transformed once and its spectrum read by every product (two transforms a
// product instead of three).
void batched_mul(Scope& S, const u32* a, uint64_t sa, uint64_t na, const u32* b, uint64_t sb, uint64_t nb, u32* out,
                 uint64_t so, uint64_t m) {
    if (m == 0) return;
    int logn = 0;
    const b2m_status st = check_sizes(na, nb, &logn);
    if (st != B2M_OK) throw Err{st};
    Context* c = S.c();
    Plan p = product_plan(c, na, nb);
    ck(twtable_ensure(c, p, S.s()), "twiddle table");
    const uint64_t npts = plan_points(p);
    u64* spec = nullptr;
    if (sb == 0 && m > 1 && p.npass > 0) {
        spec = static_cast<u64*>(S.raw(8 * npts));
        ProdJob* sj = static_cast<ProdJob*>(S.raw(sizeof(ProdJob)));
        ck(launch_pdl(k_dc_spec_job, 1, 1, 0, S.s(), b, nb, spec, sj), "spectrum job");
        ck(launch_bucket_spectrum(p, sj, 1, {spec, 0, nullptr, 0}, c->tw, S.s()), "shared spectrum");
    }
    const uint64_t wss = !p.npass ? 0
                         : spec   ? ((8 * npts + carry_scratch_bytes_n(npts) + 255) & ~255ull)
                                  : ((workspace_bytes_plan(p) + 255) & ~255ull);
    // at most 65535 jobs a launch, and at most ~1 GiB of transform workspace
    uint64_t chunk = 65535;
    if (wss) chunk = std::max<uint64_t>(1, std::min<uint64_t>(chunk, (1ull << 30) / wss));
    for (uint64_t off = 0; off < m; off += chunk) {
        const uint64_t nj = std::min(chunk, m - off);
        ProdJob* jobs = static_cast<ProdJob*>(S.raw(nj * sizeof(ProdJob)));
        unsigned long long* lens = static_cast<unsigned long long*>(S.raw(nj * 8));
        unsigned char* ws = wss ? static_cast<unsigned char*>(S.raw(nj * wss)) : nullptr;
        ck(launch_pdl(k_dc_jobs, (unsigned)((nj + 255) / 256), 256, 0, S.s(), a + off * sa, sa, na, b + off * sb, sb, nb,
                      out + off * so, so, lens, jobs, nj, ws, wss, npts, spec),
           "job tables");
        // (residue products zero their scratch and lengths themselves)
        if (wss && !p.rns)
            ck(launch_pdl(k_dc_zero_ws, (unsigned)nj, 256, 0, S.s(), jobs, nj, carry_scratch_bytes_n(npts) / 8),
               "carry scratch");
        JobBufs bufs;
        if (wss) bufs = spec ? JobBufs{spec, 0, ws, wss} : JobBufs{ws, wss, ws + 8 * npts, wss};
        ck(launch_bucket(p, jobs, (unsigned)nj, bufs, c->tw, c->d_err, S.s(), spec != nullptr), "batched product");
    }
}

// A >= B over n limbs, by the CTA: from the top, a limb a thread, until some
// limb differs (nearly always in the first round).
__device__ bool cta_ge(const u32* A, const u32* B, u64 n) {
    __shared__ u32 s_key;
    for (u64 hi = n; hi > 0; hi -= hi < blockDim.x ? hi : (u64)blockDim.x) {
        const u32 x = threadIdx.x < hi ? A[hi - 1 - threadIdx.x] : 0u, y = threadIdx.x < hi ? B[hi - 1 - threadIdx.x] : 0u;
        if (threadIdx.x == 0) s_key = 0xFFFFFFFFu;
        if (__syncthreads_or(x != y)) {
            if (x != y) atomicMin(&s_key, 2 * threadIdx.x + (x > y));
            __syncthreads();
            return s_key & 1;
        }
    }
    return true;
}

// One CTA per node i: R = V_i - U_i (U_i = q~_i P), then q~ and R move one
// unit at a time until 0 <= R < P; writes q (node 2i) and R (node 2i + 1) of
// the next level, zero-padded to its stride sout >= n. q~ is within a few
// units of the quotient, so R lies within 64 P of zero and its n limbs and
// one more, in two's complement, hold it: the upper half of V - U is not
// formed. A correction count above the bound sets bit 2 of *err (reported as
// an internal error).
// What bounds it: the chain of rounds of 8192 limbs, one CTA a node. Four
// nodes of 13,000 limbs take 25 us, and took 69 over all limbs of V - U, with
// R - P formed to see its sign and the results copied to their place.
__global__ void k_dc_fix(const u32* V, u64 sin, const u32* U, u64 su, const u32* QE, u64 sq, u64 nq, const u32* P,
                         u64 n, u32* out, u64 sout, u32* err) {
    pdl_enter();
    __shared__ GP ws[33];
    __shared__ u32 s_carry;
    const u64 i = blockIdx.x;
    V += i * sin;
    U += i * su;
    u32* Q = out + 2 * i * sout;
    u32* R = Q + sout;
    for (u64 k = threadIdx.x; k < sout; k += blockDim.x) {
        Q[k] = k < n && k < nq ? QE[i * sq + k] : 0u;
        if (k >= n) R[k] = 0;
    }
    u32 top = (n < sin ? V[n] : 0u) - (n < su ? U[n] : 0u);
    top -= cta_addsub(V, sin, U, su, 0, R, n, 1, ws, &s_carry);
    int it = 0;
    while ((int)top < 0 && it < 64) {
        top += cta_addsub(R, n, P, n, 0, R, n, 0, ws, &s_carry);
        cta_addsub(Q, n, nullptr, 0, 1, Q, n, 1, ws, &s_carry);
        ++it;
    }
    while (it < 64 && (top || cta_ge(R, P, n))) {
        top -= cta_addsub(R, n, P, n, 0, R, n, 1, ws, &s_carry);
        cta_addsub(Q, n, nullptr, 0, 1, Q, n, 0, ws, &s_carry);
        ++it;
    }
    if (it >= 64 && threadIdx.x == 0) atomicOr(err, 2u);
}

// One thread per leaf (a value below 10^72 in 8 limbs): 72 decimal digits.
__global__ void k_dc_leaf(const u32* nodes, u64 stride, u64 m, char* out) {
    pdl_enter();
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    u32 x[DC_LEAF_LIMBS];
#pragma unroll
    for (int k = 0; k < DC_LEAF_LIMBS; ++k) x[k] = (u64)k < stride ? nodes[i * stride + k] : 0u;
    char* o = out + i * (9 * DC_LEAF_GROUPS);
#pragma unroll 1
    for (int g = DC_LEAF_GROUPS - 1; g >= 0; --g) {
        u64 rem = 0;
#pragma unroll
        for (int k = DC_LEAF_LIMBS - 1; k >= 0; --k) {
            const u64 cur = (rem << 32) | x[k];
            x[k] = (u32)(cur / 1000000000u);
            rem = cur % 1000000000u;
        }
        u32 r = (u32)rem;
#pragma unroll
        for (int d = 8; d >= 0; --d) {
            o[9 * g + d] = (char)('0' + r % 10);
            r /= 10;
        }
    }
}

// The n digits without their leading zeros: publishes how many are left, and
// *err. n is a multiple of 8 and the digits are 8-byte aligned; block 0's
// first words are the leading ones, and nearly always decide.
__global__ void k_dc_count(const u64* digits, u64 n, const u32* err, PubState* st, const HostLen hl) {
    pdl_enter();
    unsigned long long t = 0;
    for (u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x; k < n / 8 && !t; k += (u64)gridDim.x * blockDim.x) {
        const u64 w = digits[k] ^ 0x3030303030303030ull;
        if (w) t = n - (8 * k + (__ffsll((long long)w) - 1) / 8);
    }
    const u64 head = 8 * (u64)blockDim.x;
    publish_top(t, n > head ? n - head : 0, err, st, gridDim.x, nullptr, hl);
}

// k_dc_fix's steps for one node as grid-wide passes driven from the host:
// for the top levels, whose few nodes have up to millions of limbs, one CTA
// a node would leave the GPU idle. R = V - U over w limbs, then R += P with
// q -= 1 while R is negative, then R -= P with q += 1 while R >= P; q and R
// go to oq / orr (n limbs, zero-padded to sout). R, T: w limbs; Q: nq + 1.
void fix_node_grid(Scope& S, const u32* V, uint64_t sin, const u32* U, uint64_t su, const u32* QE, uint64_t nq,
                   DV Pj, DV R, DV T, DV Q, DV one, u32* oq, u32* orr, uint64_t sout) {
    const uint64_t n = Pj.n;
    ck(cudaMemsetAsync(Q.p, 0, 4 * (nq + 1), S.s()), "cudaMemsetAsync");
    ck(cudaMemcpyAsync(Q.p, QE, 4 * nq, cudaMemcpyDeviceToDevice, S.s()), "D2D");
    u32 neg = addsub(S, {const_cast<u32*>(V), sin}, {const_cast<u32*>(U), su}, R, true).carry;
    int it = 0;
    while (neg && it < 64) {
        if (addsub(S, R, Pj, R, false).carry) neg = 0;
        addsub(S, Q, one, Q, true);
        ++it;
    }
    while (it < 64) {
        if (addsub(S, R, Pj, T, true).carry) break;
        std::swap(R, T);
        addsub(S, Q, one, Q, false);
        ++it;
    }
    if (it >= 64) {
        set_error("decimal conversion: a quotient correction did not converge");
        throw Err{B2M_ERR_INTERNAL};
    }
    ck(cudaMemsetAsync(oq, 0, 4 * sout, S.s()), "cudaMemsetAsync");
    ck(cudaMemsetAsync(orr, 0, 4 * sout, S.s()), "cudaMemsetAsync");
    const uint64_t k = std::min(n, sout);
    ck(cudaMemcpyAsync(oq, Q.p, 4 * std::min(k, nq + 1), cudaMemcpyDeviceToDevice, S.s()), "D2D");
    ck(cudaMemcpyAsync(orr, R.p, 4 * std::min(k, R.n), cudaMemcpyDeviceToDevice, S.s()), "D2D");
}

// Levels whose V - U has at least this many limbs per node, times the number
// of nodes, fix them with grid-wide passes (fix_node_grid), one node after the
// other, two waits of the host and eight launches and copies each; k_dc_fix
// takes all nodes of a level side by side, 25 us at 26,000 limbs of V - U and
// about 0.7 us more per 1,000.
constexpr uint64_t DC_GRID_MIN_LIMBS = 1 << 16;

// -1, 0, 1 as a <, ==, > b (trimmed).
int cmp(Scope& S, DV a, DV b) {
    if (a.n != b.n) return a.n < b.n ? -1 : 1;
    const Sum d = addsub(S, a, b, S.vec(a.n), true);
    return d.carry ? -1 : (d.v.n ? 1 : 0);
}

// Decimal digits of trimmed X, no leading zeros ("0" for zero), left on the
// device: callers copy them straight to where they are wanted (by way of
// strings on the host ten million digits took 10 ms longer).
struct Digits {
    const char* d;  // on the device
    uint64_t n;
};
Digits to_decimal(Scope& S, DV X) {
    if (X.n == 0) {
        char* z = static_cast<char*>(S.raw(1));
        ck(cudaMemsetAsync(z, '0', 1, S.s()), "cudaMemsetAsync");
        return {z, 1};
    }
    std::vector<DV> P;  // P[j] = 10^(9 2^j)
    P.push_back(upload(S, {1000000000u}));
    P[0] = trim(S, P[0]);
    while (true) {
        DV sq = mul(S, P.back(), P.back());
        if ((int)P.size() - 1 >= DC_LEAF_J && cmp(S, X, sq) < 0) {
            P.push_back(sq);
            break;
        }
        P.push_back(sq);
    }
    const int J = (int)P.size() - 2;  // X < P[J]^2 = P[J+1], J >= DC_LEAF_J
    u32* err = reinterpret_cast<u32*>(S.word() + 4);
    ck(cudaMemsetAsync(err, 0, 4, S.s()), "cudaMemsetAsync");
    // level J input: one node, X zero-padded to 2 len(P_J) limbs
    uint64_t sin = std::max<uint64_t>(2 * P[J].n, X.n);
    DV in = copy(S, X, sin);
    uint64_t m = 1;
    // Reciprocals R ~ 2^(32 E) / P_j: Newton for the top level only; below,
    // 1/P_j = P_j / P_{j+1}, so R_j = P_j * R_{j+1} (more precise than level j
    // needs), truncated to its top n + 4 limbs.
    DV R;
    uint64_t E = 0;
    for (int j = J; j > DC_LEAF_J; --j) {
        const DV Pj = P[j];
        const uint64_t n = Pj.n;
        const uint64_t L = n + 3;
        if (j == J) {
            const int sh = __builtin_clz(limb_at(S, Pj, n - 1));
            DV Pn = sh ? shl(S, Pj, 0, sh, true) : Pj;
            R = recip(S, Pn, L);  // ~ 2^(32 (L + n)) / Pn, Pn = P_j 2^sh
            if (sh) R = shl(S, R, 0, sh);
            E = L + n;
        } else {
            R = mul(S, Pj, R);
        }
        if (R.n > L + 1) {  // keep the top L + 1 limbs
            const uint64_t t = R.n - (L + 1);
            R = {R.p + t, R.n - t};
            E -= t;
        }
        // q~ = floor(V * R / 2^(32 E)) ~ floor(V / P_j), from V's top L + 1 limbs
        const uint64_t k = sin > L + 1 ? sin - (L + 1) : 0;
        if (E < k) {
            set_error("decimal conversion: reciprocal scale below the operand cut");
            throw Err{B2M_ERR_INTERNAL};
        }
        const uint64_t na = sin - k, sp = na + R.n;
        DV prod = S.vec(m * sp);
        batched_mul(S, in.p + k, sin, na, R.p, 0, R.n, prod.p, sp, m);
        // q~ are limbs [s, s + nq) of each product, read where they are
        const uint64_t s = E - k;
        if (s >= sp) {
            set_error("decimal conversion: reciprocal scale above the product");
            throw Err{B2M_ERR_INTERNAL};
        }
        const uint64_t nq = std::min(n + 1, sp - s);
        const u32* qe = prod.p + s;
        const uint64_t su = nq + n;
        DV U = S.vec(m * su);
        batched_mul(S, qe, sp, nq, Pj.p, 0, n, U.p, su, m);
        // next level: 2m nodes below P_j = P_{j-1}^2, stride 2 len(P_{j-1})
        const uint64_t sout = j - 1 > DC_LEAF_J ? 2 * P[j - 1].n : DC_LEAF_LIMBS;
        DV out = S.vec(2 * m * sout);
        const uint64_t w = std::max(sin, su) + 1;
        if (w >= DC_GRID_MIN_LIMBS * m) {
            DV R = S.vec(w), T = S.vec(w), Q = S.vec(nq + 1);
            DV one = S.vec(1);
            static const u32 one_h = 1;
            ck(cudaMemcpyAsync(one.p, &one_h, 4, cudaMemcpyHostToDevice, S.s()), "H2D");
            for (uint64_t i = 0; i < m; ++i)
                fix_node_grid(S, in.p + i * sin, sin, U.p + i * su, su, qe + i * sp, nq, Pj, R, T, Q, one,
                              out.p + (2 * i) * sout, out.p + (2 * i + 1) * sout, sout);
        } else {
            unsigned threads = 32;
            while (threads < 1024 && (uint64_t)threads * ADD_LPT < n) threads <<= 1;
            ck(launch_pdl(k_dc_fix, (unsigned)m, threads, 0, S.s(), in.p, sin, U.p, su, qe, sp, nq, Pj.p, n, out.p, sout,
                          err),
               "k_dc_fix");
        }
        in = out;
        sin = sout;
        m *= 2;
    }
    // leaves: m nodes below 10^72 in 8-limb slots
    const uint64_t digits = m * 9 * DC_LEAF_GROUPS;
    char* d_str = static_cast<char*>(S.raw(digits));
    ck(launch_pdl(k_dc_leaf, (unsigned)((m + 127) / 128), 128, 0, S.s(), in.p, sin, m, d_str), "k_dc_leaf");
    ck(launch_pdl(k_dc_count, pub_grid(digits / 8), 256, 0, S.s(), reinterpret_cast<const u64*>(d_str), digits, err,
                  pub(S), S.publication()),
       "k_dc_count");
    const u64* h = S.published();
    const uint64_t left = h[1];
    if (h[2]) {
        set_error("decimal conversion: a quotient correction did not converge");
        throw Err{B2M_ERR_INTERNAL};
    }
    const b2m_status e = take_device_error(S.c());
    if (e != B2M_OK) throw Err{e};
    if (left == 0) return {d_str, 1};  // all zeros
    return {d_str + (digits - left), left};
}

// The digits and a NUL to out (cap bytes).
void put_digits(Scope& S, Digits v, char* out, uint64_t cap, uint64_t* len) {
    if (v.n + 1 > cap) {
        set_error("decimal output buffer too small");
        throw Err{B2M_ERR_OUTPUT_TOO_SMALL};
    }
    ck(cudaMemcpyAsync(out, v.d, v.n, cudaMemcpyDeviceToHost, S.s()), "D2H");
    ck(cudaStreamSynchronize(S.s()), "cudaStreamSynchronize");
    out[v.n] = 0;
    *len = v.n;
}

// Wraps an API body: context, device, error translation.
template <class F>
b2m_status run_op(b2m_stream stream, F&& f) {
    Context* c = ctx();
    if (!c) return B2M_ERR_NOT_INITIALIZED;
    cudaSetDevice(c->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    try {
        Scope S(c, s);
        f(S);
    } catch (const Err& e) {
        cudaStreamSynchronize(s);
        return e.st;
    } catch (const std::exception& e) {
        cudaStreamSynchronize(s);
        set_error(e.what());
        return B2M_ERR_INTERNAL;
    }
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_status(e, "cudaStreamSynchronize");
    return take_device_error(c);
}

void put(Scope& S, DV v, uint32_t* dst, uint64_t cap, uint64_t* len) {
    if (v.n > cap) {
        set_error("output buffer too small");
        throw Err{B2M_ERR_OUTPUT_TOO_SMALL};
    }
    if (v.n) ck(cudaMemcpyAsync(dst, v.p, 4 * v.n, cudaMemcpyDeviceToDevice, S.s()), "D2D");
    *len = v.n;
}

}  // namespace big

}  // namespace b2m

using namespace b2m;

extern "C" {

b2m_status b2m_divmod_device(const uint32_t* d_a, uint64_t na, const uint32_t* d_b, uint64_t nb, uint32_t* d_q,
                             uint64_t q_cap, uint64_t* q_len, uint32_t* d_r, uint64_t r_cap, uint64_t* r_len,
                             b2m_stream stream) {
    if ((na && !d_a) || !d_b || !nb || (d_q && !q_len) || (d_r && !r_len)) return B2M_ERR_INVALID_ARGUMENT;
    return big::run_op(stream, [&](big::Scope& S) {
        big::DV a = big::trim(S, {const_cast<u32*>(d_a), na});
        big::DV b = big::trim(S, {const_cast<u32*>(d_b), nb});
        big::DV q, r;
        big::divmod(S, a, b, &q, &r);
        if (d_q) big::put(S, q, d_q, q_cap, q_len);
        if (d_r) big::put(S, r, d_r, r_cap, r_len);
    });
}

b2m_status b2m_isqrt_device(const uint32_t* d_a, uint64_t na, uint32_t* d_out, uint64_t cap, uint64_t* out_len,
                            b2m_stream stream) {
    if ((na && !d_a) || !d_out || !out_len) return B2M_ERR_INVALID_ARGUMENT;
    return big::run_op(stream, [&](big::Scope& S) {
        big::DV a = big::trim(S, {const_cast<u32*>(d_a), na});
        big::put(S, big::isqrt(S, a), d_out, cap, out_len);
    });
}

/* compute_pi_chudnovsky (src/chudnovsky.cpp:107-164) with every step on the
 * device: the same guard digits (16), term count, tree, floor square root of
 * 10005 * 10^(2 prec), numerator 426880 * Q * sqrtC, floor division by T and
 * decimal formatting. */
b2m_status b2m_compute_pi(uint64_t digits, char* out, uint64_t cap, uint64_t* len, b2m_pi_timings* times) {
    if (!out || !len) return B2M_ERR_INVALID_ARGUMENT;
    if (cap < digits + 3) return B2M_ERR_OUTPUT_TOO_SMALL;  // "3." + digits + NUL
    const uint64_t prec = digits + 16;
    uint64_t terms = (uint64_t)((double)prec / 14.181647462725477) + 2;  // src/chudnovsky.cpp:37,54-59
    if (terms < 2) terms = 2;
    using clk = std::chrono::steady_clock;
    auto ms = [](clk::time_point a, clk::time_point b) {
        return std::chrono::duration<double, std::milli>(b - a).count();
    };
    b2m_pi_timings tm{};
    tm.terms = terms;
    const auto t0 = clk::now();
    b2m_pqt* tree = nullptr;
    b2m_status st = b2m_chudnovsky_bs(0, terms, nullptr, &tree);
    if (st != B2M_OK) return st;
    uint64_t tl[3];
    int32_t tsign = 0;
    b2m_pqt_info(tree, tl, &tsign, nullptr, nullptr);
    const auto t1 = clk::now();
    clk::time_point t2, t3, t4;
    st = big::run_op(nullptr, [&](big::Scope& S) {
        if (tsign <= 0) {
            set_error("compute_pi: T of the tree is not positive");
            throw big::Err{B2M_ERR_INTERNAL};
        }
        big::DV Q{const_cast<u32*>(b2m_pqt_device(tree, 1)), tl[1]};
        big::DV T{const_cast<u32*>(b2m_pqt_device(tree, 2)), tl[2]};
        // one = 10^prec by square-and-multiply, as pow10_big (src/chudnovsky.cpp:42-51)
        big::DV one = big::trim(S, big::upload(S, {1u})), base = big::trim(S, big::upload(S, {10u}));
        for (uint64_t e = prec; e; e >>= 1) {
            if (e & 1) one = big::mul(S, one, base);
            if (e > 1) base = big::mul(S, base, base);
        }
        big::DV rad = big::mul(S, big::mul(S, one, one), big::trim(S, big::upload(S, {10005u})));
        big::DV sqrt_c = big::isqrt(S, rad);
        t2 = clk::now();
        big::DV num = big::mul(S, big::mul(S, Q, big::trim(S, big::upload(S, {426880u}))), sqrt_c);
        big::DV q, r;
        big::divmod(S, num, T, &q, &r);
        t3 = clk::now();
        const big::Digits d = big::to_decimal(S, q);
        // "3." and `digits` digits, or "3": the first digit moves in front of the point
        const uint64_t n = digits ? std::min(d.n, digits + 1) : 1;
        big::ck(cudaMemcpyAsync(digits ? out + 1 : out, d.d, n, cudaMemcpyDeviceToHost, S.s()), "D2H");
        big::ck(cudaStreamSynchronize(S.s()), "cudaStreamSynchronize");
        t4 = clk::now();
        if (digits) {
            out[0] = out[1];
            out[1] = '.';
        }
        *len = digits ? n + 1 : 1;
        out[*len] = 0;
    });
    b2m_pqt_free(tree);
    if (st != B2M_OK) return st;
    if (times) {
        tm.tree_ms = ms(t0, t1);
        tm.sqrt_ms = ms(t1, t2);
        tm.div_ms = ms(t2, t3);
        tm.decimal_ms = ms(t3, t4);
        tm.total_ms = ms(t0, clk::now());
        *times = tm;
    }
    return B2M_OK;
}

b2m_status b2m_to_decimal_device(const uint32_t* d_a, uint64_t na, char* out, uint64_t cap, uint64_t* len,
                                 b2m_stream stream) {
    if ((na && !d_a) || !out || !len) return B2M_ERR_INVALID_ARGUMENT;
    return big::run_op(stream, [&](big::Scope& S) {
        big::put_digits(S, big::to_decimal(S, big::trim(S, {const_cast<u32*>(d_a), na})), out, cap, len);
    });
}

// ---- host-buffer forms (the reference's BigInt magnitudes live on the host)
static big::DV host_in(big::Scope& S, const uint32_t* h, uint64_t n) {
    big::DV d = S.vec(n);
    if (n) big::ck(cudaMemcpyAsync(d.p, h, 4 * n, cudaMemcpyHostToDevice, S.s()), "H2D");
    return big::trim(S, d);  // synchronises: h may be pageable
}
static void host_out(big::Scope& S, big::DV v, uint32_t* h, uint64_t cap, uint64_t* len) {
    if (v.n > cap) {
        set_error("output buffer too small");
        throw big::Err{B2M_ERR_OUTPUT_TOO_SMALL};
    }
    if (v.n) big::ck(cudaMemcpyAsync(h, v.p, 4 * v.n, cudaMemcpyDeviceToHost, S.s()), "D2H");
    big::ck(cudaStreamSynchronize(S.s()), "cudaStreamSynchronize");
    *len = v.n;
}

b2m_status b2m_divmod_host(const uint32_t* a, uint64_t na, const uint32_t* b, uint64_t nb, uint32_t* q,
                           uint64_t q_cap, uint64_t* q_len, uint32_t* r, uint64_t r_cap, uint64_t* r_len) {
    if ((na && !a) || !b || !nb || (q && !q_len) || (r && !r_len)) return B2M_ERR_INVALID_ARGUMENT;
    return big::run_op(nullptr, [&](big::Scope& S) {
        big::DV dq, dr;
        big::divmod(S, host_in(S, a, na), host_in(S, b, nb), &dq, &dr);
        if (q) host_out(S, dq, q, q_cap, q_len);
        if (r) host_out(S, dr, r, r_cap, r_len);
    });
}

b2m_status b2m_isqrt_host(const uint32_t* a, uint64_t na, uint32_t* out, uint64_t cap, uint64_t* out_len) {
    if ((na && !a) || !out || !out_len) return B2M_ERR_INVALID_ARGUMENT;
    return big::run_op(nullptr, [&](big::Scope& S) { host_out(S, big::isqrt(S, host_in(S, a, na)), out, cap, out_len); });
}

b2m_status b2m_to_decimal_host(const uint32_t* a, uint64_t na, char* out, uint64_t cap, uint64_t* len) {
    if ((na && !a) || !out || !len) return B2M_ERR_INVALID_ARGUMENT;
    return big::run_op(nullptr, [&](big::Scope& S) {
        big::put_digits(S, big::to_decimal(S, host_in(S, a, na)), out, cap, len);
    });
}

}  // extern "C"
