// nz_wide.cuh -- exact 192- and 256-bit unsigned integers for run-reductions.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace nz {

typedef unsigned __int128 u128;

// Unsigned 256-bit helpers (4 little-endian 64-bit limbs).
struct U256 { uint64_t w[4]; };

__device__ __forceinline__ void u256_add(U256 &a, const U256 &b) {
    uint64_t c = 0;
    for (int i = 0; i < 4; ++i) {
        const uint64_t s = a.w[i] + b.w[i];
        const uint64_t c1 = s < a.w[i];
        const uint64_t s2 = s + c;
        const uint64_t c2 = s2 < s;
        a.w[i] = s2;
        c = c1 | c2;
    }
}
__device__ __forceinline__ U256 u256_from_u128(u128 x) {
    U256 r = {{(uint64_t)x, (uint64_t)(x >> 64), 0, 0}};
    return r;
}
// a (< 2^128) squared
__device__ __forceinline__ U256 u128_sq(u128 a) {
    const uint64_t lo = (uint64_t)a, hi = (uint64_t)(a >> 64);
    const u128 ll = (u128)lo * lo, lh = (u128)lo * hi, hh = (u128)hi * hi;
    U256 r = u256_from_u128(ll);
    U256 mid = {{0, (uint64_t)lh, (uint64_t)(lh >> 64), 0}};
    u256_add(r, mid);
    u256_add(r, mid);
    U256 top = {{0, 0, (uint64_t)hh, (uint64_t)(hh >> 64)}};
    u256_add(r, top);
    return r;
}
// a * k for k < 2^64
__device__ __forceinline__ U256 u256_mul64(const U256 &a, uint64_t k) {
    U256 r = {{0, 0, 0, 0}};
    u128 carry = 0;
    for (int i = 0; i < 4; ++i) {
        const u128 p = (u128)a.w[i] * k + carry;
        r.w[i] = (uint64_t)p;
        carry = p >> 64;
    }
    return r;
}
// a - b (a >= b)
__device__ __forceinline__ U256 u256_sub(const U256 &a, const U256 &b) {
    U256 r;
    uint64_t borrow = 0;
    for (int i = 0; i < 4; ++i) {
        const uint64_t d = a.w[i] - b.w[i];
        const uint64_t b1 = a.w[i] < b.w[i];
        const uint64_t d2 = d - borrow;
        const uint64_t b2 = d < borrow;
        r.w[i] = d2;
        borrow = b1 | b2;
    }
    return r;
}
__device__ __forceinline__ double u256_to_f64(const U256 &a) {
    const double t64 = 18446744073709551616.0;
    return ((a.w[3] * t64 + (double)a.w[2]) * t64 + (double)a.w[1]) * t64 + (double)a.w[0];
}

// running sum of 128-bit terms
struct U192 {
    uint64_t w0, w1, w2;
    __device__ __forceinline__ void add(u128 x) {
        const u128 s = (((u128)w1 << 64) | w0) + x;
        w2 += s < x ? 1u : 0u;
        w0 = (uint64_t)s;
        w1 = (uint64_t)(s >> 64);
    }
    __device__ __forceinline__ void add(const U192 &o) {
        add(((u128)o.w1 << 64) | o.w0);
        w2 += o.w2;
    }
    __device__ __forceinline__ U256 wide() const { return U256{{w0, w1, w2, 0}}; }
};

}  // namespace nz
