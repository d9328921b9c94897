// rns_field.cuh -- the three 30-bit primes of the residue transforms.
//
// A product's coefficients (32-bit digits, at most 2^25 terms) stay below
// 2^89, less than p0 p1 p2 = 2^89.35, so three word-sized transforms and a
// CRT replace one transform over a 64-bit field of 16-bit digits. Each prime
// is c * 2^23 + 1 below 2^30: lazily reduced values in [0, 4p) fit a 32-bit
// word, and a product by a known factor w is Shoup's
//   q = floor(a w' / 2^32), w' = floor(2^32 w / p), r = a w - q p in [0, 2p)
// for any a < 2^32: one high and two low multiplies.
//
// Why this field: a butterfly of the 64-bit field Goldilocks needs eight
// instructions on the integer ALU pipe, which bounded every pass; three
// 30-bit butterflies on half as many digits need 4.5 on the ALU pipe and as
// many on the multiply-add pipe beside it. Measured on a B200, cycles per
// warp instruction per scheduler: multiply low 2.1, multiply high 4.1, wide
// multiply-add 5, three-input add 2.1, add-then-min 2.1, and a whole
// butterfly below 9.8 with Shoup's product, 13.9 with Montgomery's.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "gl.cuh"

namespace b2m {

constexpr int RNS_TWO_ADICITY = 23;  // each p - 1 is divisible by 2^23
constexpr u32 RNS_P0 = 998244353u, RNS_P1 = 897581057u, RNS_P2 = 880803841u;

__host__ __device__ constexpr u32 rns_prime(int i) { return i == 0 ? RNS_P0 : (i == 1 ? RNS_P1 : RNS_P2); }
// -p^-1 mod 2^32: p = c 2^23 + 1, so p^-1 = 1 - c 2^23 + c^2 2^46 - ... = 2 - p mod 2^46.
__host__ __device__ constexpr u32 rns_npinv(int i) { return rns_prime(i) - 2u; }

// Host arithmetic (tables and constants).
inline u32 rns_mulmod(u32 a, u32 b, u32 p) { return (u32)((u64)a * b % p); }
inline u32 rns_powmod(u32 a, u64 e, u32 p) {
    u32 r = 1;
    for (; e; e >>= 1, a = rns_mulmod(a, a, p))
        if (e & 1) r = rns_mulmod(r, a, p);
    return r;
}
inline u32 rns_invmod(u32 a, u32 p) { return rns_powmod(a, p - 2, p); }
inline uint2 rns_pair(u32 w, u32 p) { return make_uint2(w, (u32)(((u64)w << 32) / p)); }
// A generator of the multiplicative group: not a square, ..., checked against
// the prime factors of p - 1 (2 and those of 119 = 7*17, 107 and 105 = 3*5*7).
inline u32 rns_generator(int i) {
    const u32 p = rns_prime(i);
    const u32 f[3][4] = {{2, 7, 17, 0}, {2, 107, 0, 0}, {2, 3, 5, 7}};
    for (u32 g = 2;; ++g) {
        bool ok = true;
        for (int k = 0; k < 4; ++k)
            if (f[i][k] && rns_powmod(g, (p - 1) / f[i][k], p) == 1) ok = false;
        if (ok) return g;
    }
}
// Primitive 2^l-th root of unity, one chain of squares for l <= 23.
inline u32 rns_root(int i, int l) {
    const u32 p = rns_prime(i);
    return rns_powmod(rns_generator(i), (u64)(p - 1) >> l, p);
}

#if defined(__CUDACC__)
// The prime a block works on, in registers.
struct RnsMod {
    u32 p, np2;  // p and -2p mod 2^32
    __device__ __forceinline__ explicit RnsMod(int i) : p(rns_prime(i)), np2(0u - 2u * rns_prime(i)) {}
};

// a mod 2p in [0, 2p) for a < 4p: the wrapped a - 2p is the larger one when a < 2p.
__device__ __forceinline__ u32 rns_red2(u32 a, const RnsMod& m) { return __viaddmin_u32(a, m.np2, a); }
// a * w mod p in [0, 2p) for any a.
__device__ __forceinline__ u32 rns_mul(u32 a, uint2 w, const RnsMod& m) { return a * w.x - __umulhi(a, w.y) * m.p; }
// t * 2^-32 mod p for t < 2^64 - 2^32 p; below t / 2^32 + p.
__device__ __forceinline__ u32 rns_redc(u64 t, int i, const RnsMod& m) {
    return (u32)(((u64)((u32)t * rns_npinv(i)) * m.p + t) >> 32);
}
// Forward butterfly (a, b) -> (a + w b, a - w b), all values in [0, 4p).
__device__ __forceinline__ void rns_bfly_fwd(u32& a, u32& b, uint2 w, const RnsMod& m) {
    const u32 x = rns_red2(a, m), t = rns_mul(b, w, m);
    a = x + t;
    b = x - t - m.np2;
}
// The same for w = 1.
__device__ __forceinline__ void rns_bfly_fwd1(u32& a, u32& b, const RnsMod& m) {
    const u32 x = rns_red2(a, m), t = rns_red2(b, m);
    a = x + t;
    b = x - t - m.np2;
}
// Inverse butterfly (a, b) -> (a + b, (a - b) w), all values in [0, 2p).
__device__ __forceinline__ void rns_bfly_inv(u32& a, u32& b, uint2 w, const RnsMod& m) {
    const u32 s = a + b, d = a - b - m.np2;
    a = rns_red2(s, m);
    b = rns_mul(d, w, m);
}
__device__ __forceinline__ void rns_bfly_inv1(u32& a, u32& b, const RnsMod& m) {
    const u32 s = a + b, d = a - b - m.np2;
    a = rns_red2(s, m);
    b = rns_red2(d, m);
}
#endif

}  // namespace b2m
