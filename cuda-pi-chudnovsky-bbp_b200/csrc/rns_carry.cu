// rns_carry.cu -- CRT and carry: residues of the coefficients modulo three
// 30-bit primes -> u32 limbs.
//
// Same decoupled-lookback scan as ntt_carry.cu (one CTA of 256 threads per
// 2048 limbs, eight consecutive digits per thread), reading 12 bytes of
// residues per digit instead of two 8-byte coefficients, with the CRT
// (rns_crt.cuh) in front of it.
//
// What bounds it: the CRT's multiplies and the latency of its serial part
// (ticket, loads, lookback), FMA heavy 35%, ALU 41%, DRAM 37% of their peaks at
// 2^24 digits, 82 us. Four digits a thread took 65 against 47 us at 2^23, blocks
// in index order without a ticket the same as with one.
//
// Reference counterpart: carry_propagate (include/ntt.h:70-91).
#include <cuda_runtime.h>

#include "b2m_internal.h"
#include "carry.cuh"
#include "carry_lookback.cuh"
#include "pdl.cuh"
#include "publish.cuh"
#include "rns_crt.cuh"

namespace b2m {

constexpr int CHUNK = CARRY_CHUNK / 2;  // limbs per block
constexpr int RCARRY_G = 8;  // digits per thread: CARRY_CHUNK / 2 limbs per CTA, as ntt_carry.cu
static_assert(CARRY_THREADS * RCARRY_G == CHUNK, "one lookback slot per 2048 limbs");

// One digit from its residues: c + carry -> limb and the new carry.
__device__ __forceinline__ u32 rns_digit(const u32* r, const RnsCrt& k, u64& carry) {
    u32 y[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const u32 v = r[i] * k.kap[i].x - __umulhi(r[i], k.kap[i].y) * rns_prime(i);  // [0, 2p)
        y[i] = __viaddmin_u32(v, 0u - rns_prime(i), v);                               // [0, p)
    }
    return rns_crt_digit(y, k, carry);
}

__global__ void __launch_bounds__(CARRY_THREADS, 6)
    k_rns_carry(const u32* coef, u64 nt, u32* out, u64 nout,
                LookbackSlot* slots, u32* ticket, unsigned long long* out_len, u32* err,
                const ProdJob* jobs, const RnsCrt crt, const HostLen hl) {
    pdl_enter();
    if (jobs) {
        const ProdJob& J = jobs[blockIdx.y];
        coef = reinterpret_cast<const u32*>(J.bufB);
        out = J.out;
        nout = J.na + J.nb;
        slots = J.slots;
        ticket = J.ticket;
        out_len = J.out_len;
    }
    __shared__ u32 s_chunk;
    __shared__ u64 s_cin;
    __shared__ unsigned long long s_top[CARRY_THREADS / 32];
    __shared__ u64 s_lasth[CARRY_THREADS / 32];
    __shared__ CState s_ws[CARRY_THREADS / 32 + 1];
    if (threadIdx.x == 0) s_chunk = atomicAdd(ticket, 1u);
    __syncthreads();
    const u32 chunk = s_chunk;
    // digits from na + nb on are zero: no block for them alone
    const u32 nchunks = (u32)((nout + CHUNK - 1) / CHUNK);
    if (chunk >= nchunks) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u64 base = ((u64)chunk * CARRY_THREADS + threadIdx.x) * RCARRY_G;

    u32 lm[RCARRY_G];
    CState st;
    {
        uint4 r[3][RCARRY_G / 4];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < RCARRY_G / 4; ++k)
                r[i][k] = reinterpret_cast<const uint4*>(coef + (u64)i * nt + base)[k];
        u64 c = 0;
#pragma unroll
        for (int k = 0; k < RCARRY_G / 4; ++k) {
            const u32 d0[3] = {r[0][k].x, r[1][k].x, r[2][k].x}, d1[3] = {r[0][k].y, r[1][k].y, r[2][k].y},
                      d2[3] = {r[0][k].z, r[1][k].z, r[2][k].z}, d3[3] = {r[0][k].w, r[1][k].w, r[2][k].w};
            lm[4 * k] = rns_digit(d0, crt, c);
            lm[4 * k + 1] = rns_digit(d1, crt, c);
            lm[4 * k + 2] = rns_digit(d2, crt, c);
            lm[4 * k + 3] = rns_digit(d3, crt, c);
        }
        st = group_state<RCARRY_G>(lm, c);
    }
    const u64 h_before = __shfl_up_sync(0xFFFFFFFFu, st.h, 1);
    if (lane == 31) s_lasth[warp] = st.h;
    u64 cin;
    if (!__syncthreads_or(st.t != CS_NEVER)) {
        // no group's carry-out depends on its carry-in (the usual case)
        const CState agg{s_lasth[CARRY_THREADS / 32 - 1], CS_NEVER};
        cin = lane > 0 ? h_before : (warp > 0 ? s_lasth[warp - 1] : 0);
        if (warp == 0) {
            const u64 c = warp_lookback(slots, chunk, agg, err);
            if (lane == 0) cin = c;
        }
    } else {
        bool has_ex;
        CState agg;
        const CState ex = block_scan_carry(st, &has_ex, &agg, s_ws);
        if (warp == 0) {
            const u64 c = warp_lookback(slots, chunk, agg, err);
            if (threadIdx.x == 0) s_cin = c;
        }
        __syncthreads();
        const u64 cin_chunk = s_cin;
        if (threadIdx.x == 0) st_release(&slots[chunk].word, (cs_eval(agg, cin_chunk) << 2) | SLOT_INCL);
        cin = has_ex ? cs_eval(ex, cin_chunk) : cin_chunk;
    }
    group_add_carry<RCARRY_G>(lm, cin);

    unsigned long long top = 0;
#pragma unroll
    for (int i = 0; i < RCARRY_G; ++i)
        if (lm[i] && base + i < nout) top = base + i + 1;
    if (base + RCARRY_G <= nout && ((reinterpret_cast<uintptr_t>(out + base) & 15) == 0)) {
        uint4* dst = reinterpret_cast<uint4*>(out + base);
#pragma unroll
        for (int i = 0; i < RCARRY_G / 4; ++i)
            dst[i] = make_uint4(lm[4 * i], lm[4 * i + 1], lm[4 * i + 2], lm[4 * i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < RCARRY_G; ++i)
            if (base + i < nout) out[base + i] = lm[i];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        unsigned long long o = __shfl_xor_sync(0xFFFFFFFFu, top, off);
        top = o > top ? o : top;
    }
    if (lane == 0) s_top[warp] = top;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 0; w < CARRY_THREADS / 32; ++w) top = s_top[w] > top ? s_top[w] : top;
        if (top) atomicMax(out_len, top);
        // A single product: the block of the last limbs publishes the length
        // (and the host launches what follows, in stream order) unless those
        // are zero; then the last block to finish does.
        if (hl.host && top > (u64)(nchunks - 1) * CHUNK) {
            publish(hl, top);
        } else if (hl.host) {
            __threadfence();
            if (atomicAdd(ticket + 1, 1u) == nchunks - 1) publish(hl, atomicMax(out_len, 0ull));
        }
    }
}

cudaError_t rns_launch_carry(cudaStream_t s, const u32* coef, u64 nt, u32* out, u64 nout,
                             LookbackSlot* slots, u32* ticket, unsigned long long* out_len, u32* err,
                             const ProdJob* jobs, unsigned njobs, const RnsCrt& crt, HostLen hl) {
    const u64 n = jobs ? nt : nout;
    if (n == 0 || njobs == 0) return cudaSuccess;
    return launch_pdl(k_rns_carry, dim3((unsigned)((n + CHUNK - 1) / CHUNK), njobs), CARRY_THREADS, 0, s, coef, nt, out,
                      nout, slots, ticket, out_len, err, jobs, crt, hl);
}

}  // namespace b2m
