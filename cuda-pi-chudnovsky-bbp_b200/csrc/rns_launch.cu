// rns_launch.cu -- products on the three-prime residue transforms: lengths,
// tables and launch sequences (kernels: rns_kernels.cuh, rns_carry.cu).
//
// A product whose 16-bit-digit length is 2^L or 3 * 2^k points takes half as
// many 32-bit digits: N = q * 2^m with q = 1 or 3 -- or 5/6 of the latter, q =
// 5, where that holds it -- as long as the roots of unity last (q * 2^m <=
// 2^23); beyond that N splits into q <= 8 parts of at
// most 2^23 points (N <= 2^26, the CRT's bound on the coefficients: at most
// 2^25 terms below 2^64 each). Parts evaluate modulo x^M - c_t. Where the
// 2^23 roots allow, c_t is the constant of tree node t and the parts are the
// first q nodes of the next power of two (a truncated tree); otherwise
// c_t = theta_t^M with theta_t a power of the generator, the first pass runs
// the tree of theta_t and its columns take a factor theta_t^column
// ("weighted"). The parts of the inverse are put together by the inverse
// Vandermonde matrix of the c_t (k_rns_inv_parts).
//
// Reference counterpart: mul_ntt_cuda (src/ntt_cuda.cu:179-243).
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <vector>

#include "b2m.h"
#include "b2m_context.h"
#include "b2m_internal.h"
#include "pdl.cuh"
#include "rns_field.cuh"

namespace b2m {

namespace {

struct RnsShape {
    int q = 0, m = 0;       // N = q * 2^m
    bool weighted = false;
    int npass = 0, logr[3] = {0, 0, 0};
    u64 points() const { return (u64)q << m; }
};

// Pass radices of a 2^m-point part, from a sweep over the splits of each
// length (us a product): 2^17 [5, 5, 7] 24.5 against 26.5 to 31.7 in two passes
// (64 at once 4.9 each against 4.7); 2^19 [6, 6, 7] 37.3 against [10, 9] 43.4;
// 2^22 [6, 8, 8] 195 against [7, 7, 8] 199.
constexpr int RNS_MIN_M = 13, RNS_MAX_M = RNS_TWO_ADICITY;
constexpr int kSplit[RNS_MAX_M - RNS_MIN_M + 1][3] = {
    {6, 0, 7},  // 2^13
    {6, 0, 8},  // 2^14
    {7, 0, 8},  // 2^15
    {8, 0, 8},  // 2^16
    {5, 5, 7},  // 2^17
    {5, 6, 7},  // 2^18
    {6, 6, 7},  // 2^19
    {6, 6, 8},  // 2^20
    {6, 7, 8},  // 2^21
    {6, 8, 8},  // 2^22
    {7, 8, 8},  // 2^23
};
// 6 and 8 parts: eight values per thread and part in the first pass (the
// inverse holds all parts of its tile in registers).
constexpr int kSplitParts23[3] = {6, 8, 9};

// Part lengths of transforms in five parts (first radix 2^6 and below: the
// inverse holds five values per row in registers). 2^15 has a first radix of
// 2^7; a split of it that would do, [6, 9], was not measured.
constexpr bool five_parts(int m) { return m >= 13 && m <= 22 && m != 15; }
constexpr int kSplitFive16[3] = {5, 5, 6};

// Launches of at least this many points (over all jobs) take two columns per
// thread, shorter ones twice as many blocks: at 2^20 points 57.6 against
// 61.4 us a product, at 2^18 31.7 against 28.5.
constexpr u64 RNS_V2_POINTS = 1ull << 19;

// Blocks that keep the SMs busy (three per SM) several times over.
constexpr u64 RNS_FULL_GRID = 148 * 6;

// The shape of a plan's length, q = 0 when these transforms do not take it.
RnsShape rns_shape(const Plan& p) {
    RnsShape r;
    if (p.npass < 2) {  // one launch
        r.q = 1;
        r.m = p.logn - 1;
        return r;
    }
    int m = p.logn - 1, q = p.three ? 3 : 1;  // 32-bit digits
    while (m > RNS_MAX_M) {
        --m;
        q *= 2;
    }
    if (m < RNS_MIN_M || q > 8) return r;
    if (p.three && q == 3 && p.need && p.need <= 5ull << (m - 1) && five_parts(m - 1)) {
        q = 5;
        --m;
    }
    int lq = 0;
    while ((1 << lq) < q) ++lq;
    r.q = q;
    r.m = m;
    r.weighted = q > 1 && m + lq > RNS_TWO_ADICITY;
    const int* s = q > 5 ? kSplitParts23 : (q == 5 && m == 16 ? kSplitFive16 : kSplit[m - RNS_MIN_M]);
    for (int k = 0; k < 3; ++k)
        if (s[k]) r.logr[r.npass++] = s[k];
    return r;
}

// ---- tables -------------------------------------------------------------------
// T[k] = prod over set bits j of k of root_(2^(j+2)), root[] given per prime
// (forward, or the inverses).
struct RootSet {
    u32 w[3][22];
};

__device__ __forceinline__ u32 dmulmod(u32 a, u32 b, u32 p) { return (u32)((u64)a * b % p); }

// T[k] = T[k mod 2^11] * T[(k div 2^11) 2^11], from the two short tables.
constexpr int RNS_BUILD_LOG = 11;

__global__ void __launch_bounds__(1 << RNS_BUILD_LOG >> 1) k_rns_build(uint2* __restrict__ t, u32 ent,
                                                                      const RootSet fwd, const RootSet inv) {
    __shared__ u32 lo[1 << RNS_BUILD_LOG];
    const int i = blockIdx.y % 3;
    const u32 p = rns_prime(i);
    const RootSet& r = blockIdx.y < 3 ? fwd : inv;
    uint2* dst = t + (u64)blockIdx.y * ent;
    for (u32 k = threadIdx.x; k < (1u << RNS_BUILD_LOG); k += blockDim.x) {
        u32 v = 1;
        for (u32 b = k; b; b &= b - 1) v = dmulmod(v, r.w[i][__ffs(b) - 1], p);
        lo[k] = v;
    }
    __syncthreads();
    for (u32 h = blockIdx.x; (h << RNS_BUILD_LOG) < ent; h += gridDim.x) {
        u32 w = 1;
        for (u32 b = h; b; b &= b - 1) w = dmulmod(w, r.w[i][RNS_BUILD_LOG + __ffs(b) - 1], p);
        for (u32 k = threadIdx.x; k < (1u << RNS_BUILD_LOG); k += blockDim.x) {
            const u32 v = dmulmod(w, lo[k], p);
            dst[((u64)h << RNS_BUILD_LOG) + k] = make_uint2(v, (u32)(((u64)v << 32) / p));
        }
    }
}

// Weighted parts: w^column (column < 2^logs) of a per-part base w, and the
// first-pass tree: entry 2^lev + k = (theta^(M / 2^(lev+1))) T[k].
struct WeightSet {
    u32 col[3][8];          // theta_t (or its inverse)
    u32 lev[3][8][10];      // theta_t^(M / 2^(lev+1))
};

__device__ __forceinline__ u32 dpowmod(u32 a, u32 e, u32 p) {
    u32 r = 1;
    for (; e; e >>= 1, a = dmulmod(a, a, p))
        if (e & 1) r = dmulmod(r, a, p);
    return r;
}

__global__ void k_rns_build_weights(uint2* __restrict__ tree, uint2* __restrict__ col, int q, int logr, int logs,
                                    const uint2* __restrict__ T, u32 ent, const WeightSet w) {
    const int i = blockIdx.y / q, t = blockIdx.y % q;
    const u32 p = rns_prime(i);
    const u32 n1 = 1u << logr, n2 = 1u << logs;
    for (u32 x = blockIdx.x * blockDim.x + threadIdx.x; x < n1 + n2; x += gridDim.x * blockDim.x) {
        if (x < n1) {
            u32 v = 1;
            if (x) {
                const int lev = 31 - __clz(x);
                v = dmulmod(w.lev[i][t][lev], T[(u64)i * ent + (x - (1u << lev))].x, p);
            }
            tree[((u64)(i * q + t) << logr) + x] = make_uint2(v, (u32)(((u64)v << 32) / p));
        } else {
            const u32 v = dpowmod(w.col[i][t], x - n1, p);
            col[((u64)(i * q + t) << logs) + (x - n1)] = make_uint2(v, (u32)(((u64)v << 32) / p));
        }
    }
}

RootSet root_set(bool inverse) {
    RootSet r;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 22; ++j) {
            const u32 w = j + 2 <= RNS_TWO_ADICITY ? rns_root(i, j + 2) : 1u;
            r.w[i][j] = inverse ? rns_invmod(w, rns_prime(i)) : w;
        }
    return r;
}

// T[k] on the host, for small k.
u32 node_root(int i, u32 k) {
    u32 v = 1;
    for (int j = 0; j < 22; ++j)
        if ((k >> j) & 1) v = rns_mulmod(v, rns_root(i, j + 2), rns_prime(i));
    return v;
}

u32 theta(int i, int t) { return rns_powmod(rns_generator(i), t, rns_prime(i)); }

// c_t of part t.
u32 part_constant(const RnsShape& sh, int i, int t) {
    const u32 p = rns_prime(i);
    if (sh.q == 1) return 1;
    if (sh.weighted) return rns_powmod(theta(i, t), 1ull << sh.m, p);
    const u32 w = node_root(i, t / 2);  // x^2M - w^2 = (x^M - w)(x^M + w)
    return (t & 1) ? p - w : w;
}

// Host constants of a shape, computed once.
struct RnsConst {
    uint2 ct[3][8];
    RnsCombine comb;
    RnsCrt crt;
};

RnsConst make_const(const RnsShape& sh) {
    RnsConst k{};
    const int q = sh.q;
    for (int i = 0; i < 3; ++i) {
        const u32 p = rns_prime(i);
        u32 c[8];
        for (int t = 0; t < q; ++t) {
            c[t] = part_constant(sh, i, t);
            k.ct[i][t] = rns_pair(c[t], p);
        }
        // inverse of V[t][s] = c_t^s by Gauss-Jordan
        u32 a[8][16];
        for (int t = 0; t < q; ++t) {
            u32 x = 1;
            for (int s = 0; s < q; ++s, x = rns_mulmod(x, c[t], p)) {
                a[t][s] = x;
                a[t][q + s] = s == t;
            }
        }
        for (int col = 0; col < q; ++col) {
            int piv = col;
            while (!a[piv][col]) ++piv;
            for (int s = 0; s < 2 * q; ++s) std::swap(a[piv][s], a[col][s]);
            const u32 inv = rns_invmod(a[col][col], p);
            for (int s = 0; s < 2 * q; ++s) a[col][s] = rns_mulmod(a[col][s], inv, p);
            for (int r = 0; r < q; ++r) {
                if (r == col || !a[r][col]) continue;
                const u32 f = p - a[r][col];
                for (int s = 0; s < 2 * q; ++s) a[r][s] = (u32)((a[r][s] + (u64)f * a[col][s]) % p);
            }
        }
        for (int s = 0; s < q; ++s)
            for (int t = 0; t < q; ++t) k.comb.v[i][s][t] = a[s][q + t];
        // residues arrive as c * 2^m * 2^-32 (Montgomery pointwise product),
        // times 2^-32 again where parts were put together
        u32 scale = rns_invmod(rns_powmod(2, 32, p), p);
        if (q > 1) scale = rns_mulmod(scale, scale, p);
        scale = rns_mulmod(scale, rns_powmod(2, sh.m, p), p);
        const u64 qi = i == 0 ? (u64)RNS_P1 * RNS_P2 : (i == 1 ? (u64)RNS_P0 * RNS_P2 : (u64)RNS_P0 * RNS_P1);
        k.crt.kap[i] = rns_pair(rns_invmod(rns_mulmod(scale, (u32)(qi % p), p), p), p);
        k.crt.qlo[i] = (u32)qi;
        k.crt.qhi[i] = (u32)(qi >> 32);
    }
    return k;
}

const RnsConst& shape_const(const RnsShape& sh) {
    static std::mutex mu;
    static std::map<std::pair<int, int>, RnsConst> cache;  // at most a few dozen shapes
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find({sh.q, sh.m});
    if (it == cache.end()) it = cache.emplace(std::make_pair(sh.q, sh.m), make_const(sh)).first;
    return it->second;
}

// ---- context tables --------------------------------------------------------------
constexpr int RNS_BASE_LOG = 18, RNS_FULL_LOG = RNS_TWO_ADICITY - 1;  // log2 entries per prime and direction

uint64_t table_bytes(int log_ent) { return 6ull * sizeof(uint2) << log_ent; }

cudaError_t build_tables(uint2** out, int log_ent, cudaStream_t s) {
    const u64 bytes = table_bytes(log_ent);
    cudaError_t e = cudaMalloc(out, bytes);
    if (e != cudaSuccess) return e;
    const u32 ent = 1u << log_ent;
    k_rns_build<<<dim3(std::min<u32>(148, ent >> RNS_BUILD_LOG), 6), 1 << RNS_BUILD_LOG >> 1, 0, s>>>(
        *out, ent, root_set(false), root_set(true));
    if ((e = cudaGetLastError()) == cudaSuccess) e = cudaStreamSynchronize(s);  // complete before anyone sees it
    if (e != cudaSuccess) {
        cudaFree(*out);
        *out = nullptr;
    }
    return e;
}

int need_log_ent(const RnsShape& sh) {
    int lq = 0;
    if (!sh.weighted)
        while ((1 << lq) < sh.q) ++lq;
    return sh.m + lq - 1;
}

// Caller holds c->twt_mu.
const Context::RnsWeights* find_weights(Context* c, const RnsShape& sh) {
    for (const Context::RnsWeights& w : c->rns_weights)
        if (w.q == sh.q && w.m == sh.m) return &w;
    return nullptr;
}

cudaError_t build_weights(Context* c, const RnsShape& sh, Context::RnsWeights* w, cudaStream_t s) {
    const int logr = sh.logr[0], logs = sh.m - logr;
    const u64 tree = 3ull * sh.q << logr, col = 3ull * sh.q << logs;
    cudaError_t e = cudaMalloc(&w->mem, 2 * (tree + col) * sizeof(uint2));
    if (e != cudaSuccess) return e;
    for (int dir = 0; dir < 2 && e == cudaSuccess; ++dir) {
        WeightSet ws{};
        for (int i = 0; i < 3; ++i)
            for (int t = 0; t < sh.q; ++t) {
                u32 th = theta(i, t);
                if (dir) th = rns_invmod(th, rns_prime(i));
                ws.col[i][t] = th;
                for (int l = 0; l < logr; ++l) ws.lev[i][t][l] = rns_powmod(th, 1ull << (sh.m - l - 1), rns_prime(i));
            }
        uint2* base = w->mem + dir * (tree + col);
        k_rns_build_weights<<<dim3(64, 3 * sh.q), 256, 0, s>>>(base, base + tree, sh.q, logr, logs,
                                                              c->rns_t + (dir ? 3ull << c->rns_log : 0),
                                                              1u << c->rns_log, ws);
        e = cudaGetLastError();
        w->tree[dir] = base;
        w->col[dir] = base + tree;
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        cudaFree(w->mem);
        w->mem = nullptr;
    }
    return e;
}

}  // namespace

cudaError_t rns_init_tables(Context* c) {
    cudaError_t e = build_tables(&c->rns_t, RNS_BASE_LOG, 0);
    if (e != cudaSuccess) return e;
    c->rns_base = c->rns_t;
    c->rns_log = RNS_BASE_LOG;
    return cudaSuccess;
}

void rns_free_tables(Context* c) {
    std::lock_guard<std::mutex> lk(c->twt_mu);
    for (auto& g : c->rns_grown) {
        cudaFree(g.first);
        budget_release(c, g.second);
    }
    c->rns_grown.clear();
    if (c->rns_base) cudaFree(c->rns_base);
    c->rns_t = c->rns_base = nullptr;
    for (Context::RnsWeights& w : c->rns_weights) {
        cudaFree(w.mem);
        budget_release(c, w.bytes);
    }
    c->rns_weights.clear();
}

// Only default plans run here: a plan fixed by b2m_set_plan or kept by an
// autotuner names passes of the 64-bit transform and gets them.
static bool is_default_plan(const Plan& p) {
    for (int three = 0; three < 2; ++three) {
        const Plan d = make_plan(p.logn, three);
        bool same = d.npass == p.npass;
        for (int k = 0; same && k < p.npass; ++k) same = d.logr[k] == p.logr[k] && d.logc[k] == p.logc[k];
        if (same) return true;
    }
    return false;
}

static uint64_t weight_bytes(const RnsShape& sh) {
    return 2 * 3ull * sh.q * sizeof(uint2) * ((1ull << sh.logr[0]) + (1ull << (sh.m - sh.logr[0])));
}

// log2 entries of the tables that plan p's product runs on: the present ones,
// or those to build, full ones if they fit and else what the length needs. -1
// where none fit: then the 64-bit transforms run. Caller holds c->twt_mu.
//
// What a plan lacks is built, all or none, where it takes at most a quarter of
// what the budget has left and leaves the product its workspace. Tables are
// kept, so they must not cost a call the memory that it asks for after them (a
// tree level's other products). The 64-bit transforms keep 24 bytes of tables
// a point of each length: a call that finds room beside those needs 0.4 (one
// product, 16 bytes a point) to 0.67 (3 * 2^k points) of what is left, a tree
// level about 0.55.
static int tables_for(Context* c, const Plan& p, const RnsShape& sh) {
    const int need = need_log_ent(sh);
    const uint64_t weights = sh.weighted && !find_weights(c, sh) ? weight_bytes(sh) : 0;
    if (need <= c->rns_log && !weights) return c->rns_log;
    const uint64_t used = c->in_use.load(), left = c->budget > used ? c->budget - used : 0;
    for (int log : {RNS_FULL_LOG, need}) {
        if (need <= c->rns_log) log = c->rns_log;
        const uint64_t bytes = (log > c->rns_log ? table_bytes(log) : 0) + weights;
        if (bytes <= left / 4 && bytes + workspace_bytes_plan(p) <= left) return log;
    }
    return -1;
}

bool rns_expected(Context* c, const Plan& p) {
    const RnsShape sh = rns_shape(p);
    if (p.npass < 2 || sh.q == 0 || !is_default_plan(p)) return false;
    if (!c) return true;
    std::lock_guard<std::mutex> lk(c->twt_mu);
    return tables_for(c, p, sh) >= 0;
}

cudaError_t rns_resolve(Context* c, Plan& p, cudaStream_t s, bool build) {
    p.rns = 0;
    const RnsShape sh = rns_shape(p);
    if (!c || !c->rns_t || sh.q == 0 || !is_default_plan(p)) return cudaSuccess;
    if (build) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) build = false;
    }
    std::lock_guard<std::mutex> lk(c->twt_mu);
    if (!build && (need_log_ent(sh) > c->rns_log || (sh.weighted && !find_weights(c, sh)))) return cudaSuccess;
    const int log = tables_for(c, p, sh);
    if (log < 0) return cudaSuccess;
    if (log > c->rns_log) {
        const uint64_t bytes = table_bytes(log);
        if (!budget_reserve(c, bytes)) return cudaSuccess;
        uint2* t = nullptr;
        const cudaError_t e = build_tables(&t, log, s);
        if (e != cudaSuccess) {
            budget_release(c, bytes);
            if (e != cudaErrorMemoryAllocation) return e;
            cudaGetLastError();
            return cudaSuccess;
        }
        c->rns_grown.push_back({t, bytes});  // the earlier ones stay: launches in flight and captured graphs read them
        c->rns_t = t;
        c->rns_log = log;
    }
    if (sh.weighted && !find_weights(c, sh)) {
        Context::RnsWeights w{};
        w.q = sh.q;
        w.m = sh.m;
        w.bytes = weight_bytes(sh);
        if (!budget_reserve(c, w.bytes)) return cudaSuccess;
        const cudaError_t e = build_weights(c, sh, &w, s);
        if (e != cudaSuccess) {
            budget_release(c, w.bytes);
            if (e != cudaErrorMemoryAllocation) return e;
            cudaGetLastError();
            return cudaSuccess;
        }
        c->rns_weights.push_back(w);
    }
    p.rns = 1;
    return cudaSuccess;
}

int rns_launches(const Plan& p) {
    const RnsShape sh = rns_shape(p);
    if (sh.npass == 0) return 1;
    return 2 * sh.npass - 1 + 1;
}

namespace {

struct RnsRun {
    RnsShape sh;
    RnsArgs a{};
    unsigned njobs = 1;
    const uint2 *wtree[2] = {nullptr, nullptr}, *wcol[2] = {nullptr, nullptr};
    cudaStream_t s;
    Tracer* tr = nullptr;

    bool small;  // one launch (rns_small.cu)

    RnsRun(const Plan& p, cudaStream_t st) : sh(rns_shape(p)), s(st), small(sh.q == 1 && sh.npass == 0) {
        Context* c = ctx();
        std::lock_guard<std::mutex> lk(c->twt_mu);
        a.nt = sh.points();
        a.nzero = (u32)(carry_scratch_bytes_n(plan_points(p)) / 8);
        a.tw = c->rns_t;
        a.ent = 1u << c->rns_log;
        a.twi = a.tw + 3ull * a.ent;
        a.q = sh.q;
        if (sh.weighted) {
            const Context::RnsWeights* w = find_weights(c, sh);
            for (int d = 0; d < 2; ++d) {
                wtree[d] = w->tree[d];
                wcol[d] = w->col[d];
            }
        }
        const RnsConst& k = shape_const(sh);
        for (int i = 0; i < 3; ++i)
            for (int t = 0; t < 8; ++t) a.ct[i][t] = k.ct[i][t];
    }
    void batch(const ProdJob* jobs, unsigned n, const JobBufs& bufs) {
        a.jobs = jobs;
        njobs = n;
        a.bufA = static_cast<u32*>(bufs.a);
        a.bufB = static_cast<u32*>(bufs.b);
        a.stride_a = bufs.stride_a / sizeof(u32);
        a.stride_b = bufs.stride_b / sizeof(u32);
    }
    // Pass k's stride and node mask.
    void pass(int k) {
        int before = 0;
        for (int i = 0; i < k; ++i) before += sh.logr[i];
        a.logs = sh.m - before - sh.logr[k];
        a.nmask = sh.weighted ? (1u << before) - 1 : ~0u;
    }
    void weights(int dir, bool on) {
        a.wtree = on ? wtree[dir] : nullptr;
        a.wcol = on ? wcol[dir] : nullptr;
    }
    // Columns per thread of pass k, and its tiles: blocks of 256 threads with
    // V 2^LA elements each. First passes in parts have 16 elements.
    // (two columns: 2^(9 - LB) columns a tile, which must fit the stride S).
    int cols(int k) const {
        int logs = sh.m;
        for (int i = 0; i <= k; ++i) logs -= sh.logr[i];
        return a.nt * njobs >= RNS_V2_POINTS && logs >= 9 - sh.logr[k] / 2 ? 2 : 1;
    }
    unsigned tiles(int k) const { return (unsigned)(a.nt >> (7 + cols(k) + (sh.logr[k] + 1) / 2)); }
    unsigned part_tiles() const { return (unsigned)((1ull << sh.m) >> 12); }
    // Forward passes but the last, operands op0 .. op0 + nops - 1.
    cudaError_t forward(int op0, int nops) {
        cudaError_t e = cudaSuccess;
        a.op0 = op0;
        for (int k = 0; k + 1 < sh.npass && e == cudaSuccess; ++k) {
            pass(k);
            dim3 grid(tiles(k), njobs, 3 * nops);
            if (k == 0 && sh.q > 1) {
                // all parts in one block where that leaves enough blocks
                a.pper = (u64)part_tiles() * njobs * 3 * nops >= RNS_FULL_GRID ? sh.q : 1;
                grid.x = part_tiles() * (sh.q / a.pper);
            }
            if (tr) tr->mark(s, k == 0 ? B2M_K_FWD_FIRST : B2M_K_FWD_MID, sh.logr[k]);
            weights(0, k == 0);
            e = k == 0 ? rns_launch_first(sh.logr[k], cols(k), grid, s, a)
                       : rns_launch_mid(sh.logr[k], cols(k), grid, s, a);
        }
        weights(0, false);
        return e;
    }
    // Last forward pass of both operands, product, inverse passes, parts.
    cudaError_t finish() {
        const int last = sh.npass - 1;
        pass(last);
        if (tr) tr->mark(s, B2M_K_FUSED_LAST, sh.logr[last]);
        cudaError_t e = rns_launch_fused(sh.logr[last], dim3(1, njobs, 3), s, a);
        for (int k = last - 1; k >= 0 && e == cudaSuccess; --k) {
            pass(k);
            if (tr) tr->mark(s, B2M_K_INV_MID, sh.logr[k]);
            weights(1, k == 0);
            if (k == 0 && sh.q > 1)
                e = rns_launch_inv_parts(sh.logr[0], dim3((unsigned)((1ull << sh.m) >> (8 + (sh.logr[0] + 1) / 2)), njobs, 3), s, a, shape_const(sh).comb);
            else
                e = rns_launch_inv(sh.logr[k], cols(k), k == 0, dim3(tiles(k), njobs, 3), s, a);
        }
        weights(1, false);
        return e;
    }
    cudaError_t carry(u32* out, u64 nout, LookbackSlot* slots, u32* ticket, unsigned long long* out_len, u32* err,
                      HostLen hl = {}) {
        if (tr) tr->mark(s, B2M_K_CARRY, 0);
        return rns_launch_carry(s, a.bufB, a.nt, out, nout, slots, ticket,
                                out_len, err, a.jobs, njobs, shape_const(sh).crt, hl);
    }
};

}  // namespace

cudaError_t rns_launch_product(const u32* a, uint64_t na, const u32* b, uint64_t nb, u32* out, u64 nout, u32* bufA,
                               u32* bufB, LookbackSlot* slots, u32* ticket, unsigned long long* out_len,
                               const Plan& p, u32* err, cudaStream_t s, Tracer* tr, cudaEvent_t b_ready,
                               HostLen hl) {
    RnsRun r(p, s);
    r.tr = tr;
    r.a.a = a;
    r.a.b = b;
    r.a.na = na;
    r.a.nb = nb;
    r.a.bufA = bufA;
    r.a.bufB = bufB;
    r.a.square = a == b && na == nb;
    cudaError_t e = cudaSuccess;
    if (r.small) {
        if (b_ready && (e = cudaStreamWaitEvent(s, b_ready, 0)) != cudaSuccess) return e;
        if (tr) tr->mark(s, B2M_K_SMALL, p.logn);
        e = rns_launch_small(r.sh.m, 1, s, r.a, out, out_len, shape_const(r.sh).crt, hl);
        if (tr) tr->end(s);
        return e;
    }
    // lookback slots, then the ticket: one word per 1024 points and a few
    r.a.zero = reinterpret_cast<unsigned long long*>(slots);
    r.a.zero_len = out_len;
    if (r.a.square || !b_ready) {
        if (b_ready) e = cudaStreamWaitEvent(s, b_ready, 0);
        if (e == cudaSuccess) e = r.forward(r.a.square ? 1 : 0, r.a.square ? 1 : 2);
    } else {
        // operand B may still be on its way: A's passes go first
        e = r.forward(0, 1);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(s, b_ready, 0);
        r.a.zero = nullptr;
        if (e == cudaSuccess) e = r.forward(1, 1);
    }
    if (e == cudaSuccess) e = r.finish();
    if (e == cudaSuccess) e = r.carry(out, nout, slots, ticket, out_len, err, hl);
    if (tr) tr->end(s);
    return e;
}

// Operand a of each job up to the last forward pass, which the fused pass
// repeats for every product that shares it.
cudaError_t rns_launch_spectrum(const Plan& p, const ProdJob* jobs, unsigned njobs, const JobBufs& bufs,
                                cudaStream_t s) {
    RnsRun r(p, s);
    if (r.small) return cudaSuccess;  // transforms both operands itself
    r.batch(jobs, njobs, bufs);
    return r.forward(0, 1);
}

cudaError_t rns_launch_bucket(const Plan& p, const ProdJob* jobs, unsigned njobs, const JobBufs& bufs, u32* err,
                              cudaStream_t s, bool a_ready) {
    RnsRun r(p, s);
    r.batch(jobs, njobs, bufs);
    if (r.small) return rns_launch_small(r.sh.m, njobs, s, r.a, nullptr, nullptr, shape_const(r.sh).crt);
    cudaError_t e = a_ready ? r.forward(1, 1) : r.forward(0, 2);
    if (e == cudaSuccess) e = r.finish();
    return e == cudaSuccess ? r.carry(nullptr, 0, nullptr, nullptr, nullptr, err) : e;
}

}  // namespace b2m
