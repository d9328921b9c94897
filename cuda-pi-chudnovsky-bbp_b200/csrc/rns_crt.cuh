// rns_crt.cuh -- coefficients from their residues modulo the three primes.
//
// With y_i = r_i (scale P / p_i)^-1 mod p_i,
//     c = sum y_i P / p_i - t P,   t = floor(sum y_i / p_i) in {0, 1, 2}.
// t comes from the top 16 bits of each y_i: the estimate of the sum is low by
// less than 2^-11.7, and c / P <= 2^89 / P = 0.79 leaves room for the 2^-11
// added back.
#pragma once
#include "b2m_internal.h"
#include "rns_field.cuh"

namespace b2m {

constexpr u64 RNS_P01 = (u64)RNS_P0 * RNS_P1;
constexpr u32 RNS_PLO = (u32)((u64)(u32)RNS_P01 * RNS_P2);                                // P mod 2^32
constexpr u64 RNS_PHI = (RNS_P01 >> 32) * RNS_P2 + (((u64)(u32)RNS_P01 * RNS_P2) >> 32);  // P >> 32
__host__ __device__ constexpr u32 rns_kt(int i) { return (u32)((1ull << 44) / rns_prime(i)); }

// One digit from canonical y: c + carry -> limb and the new carry. The carry
// in and out is below 2^59.
__device__ __forceinline__ u32 rns_crt_digit(const u32* y, const RnsCrt& k, u64& carry) {
    u32 s = 1u << 19;  // 2^30 * 2^-11
#pragma unroll
    for (int i = 0; i < 3; ++i) s += (y[i] >> 14) * rns_kt(i);
    const u32 t = s >> 30;
    u64 lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        lo += (u64)y[i] * k.qlo[i];  // three terms below 2^62
        hi += (u64)y[i] * k.qhi[i];
    }
    // (hi : lo) - t P + carry, in words w0 and v
    const u64 tl = (u64)t * RNS_PLO;
    u64 v = hi + (lo >> 32) - (u64)t * RNS_PHI - (tl >> 32) + (carry >> 32);
    u32 w = (u32)lo;
    v -= w < (u32)tl;
    w -= (u32)tl;
    w += (u32)carry;
    v += w < (u32)carry;
    carry = v;
    return w;
}

}  // namespace b2m
