// nz_conv.cuh -- accumulators of the canonical convolutions.
#pragma once

#include <cstdint>

#include "nz_common.cuh"

namespace nz {

constexpr int kConvChunk = 128;  // rows summed in FP32 before they are added into the running sum

// Window accumulator of one canonical value: the FP32 partial sums of the row
// chunks are added into an FP32 (sum, compensation) pair by an error-free
// addition -- as accurate as an FP64 sum of them, without the FP64 pipe, which
// runs at 1/64 of the FP32 rate on this chip.
struct ConvAcc {
    float s = 0.0f, c = 0.0f;
    // chunk sums and the running sum are >= 0: Fast2Sum on the operands
    // ordered by size is exact (3 additions and a max / min, not TwoSum's 6)
    __device__ __forceinline__ void add(float x) {
        const float a = fmaxf(s, x), b = fminf(s, x);
        const float t = __fadd_rn(a, b);
        c = __fadd_rn(c, __fsub_rn(b, __fsub_rn(t, a)));
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// ---------------------------------------------------------------------
// m2 with compensated FP32 arithmetic
// ---------------------------------------------------------------------
// sum' s^2 / N is the susceptibility curve: up to ~2e4 at L = 1024, and its
// canonical value must come within 1e-6 absolute of the FP64 convolution,
// i.e. ~5e-11 relative per run.  Plain FP32 sums of 128 products carry
// ~1e-7, and FP32 weights alone ~2e-9.  So every term is computed from exact
// two-part operands and summed with its rounding errors kept, after Dot2 of
// Ogita, Rump & Oishi (2005, "Accurate sum and dot product"):
//   w = wh + wl        (wh = FP32(w64), wl = FP32(w64 - wh): ~2^-48 relative)
//   q = qh + ql        (qh = q rounded toward zero to 24 bits, ql = q - qh,
//                       both exact in FP32 for q < 2^48)
//   ph = wh qh, eh = fma(wh, qh, -ph)     (TwoProduct: ph + eh = wh qh exactly)
//   (s, e) = Fast2Sum(max(s, ph), min(s, ph))  (s + e = old s + ph exactly)
//   c += e + eh + wh ql + wl qh           (wl ql, ~2^-48 of the term, dropped)
// The run's value is s + c (FP64), about 2^-44 relative; the statistic's
// curve then inherits FP64-level accuracy from the FP64 run reduction.
// Only the band's core -- the rows whose weight is >= e^-8 of the mode, +-4
// standard deviations -- needs this: the tails hold < 1e-4 of the weight,
// and plain FP32 products summed per chunk keep their error near 1e-11 of
// the value.  Chunks of rows outside every core of a tile (about a third of
// a tile's rows) take the plain path.
struct Dot2Acc {
    float s = 0.0f, c = 0.0f, tail = 0.0f;
    // a compensated term.  Every term and the running sum are >= 0, so
    // ordering the two operands by size (max / min, on the integer pipe)
    // makes Dekker's Fast2Sum exact: 3 additions instead of TwoSum's 6.
    __device__ __forceinline__ void add(float wh, float wl, float qh, float ql) {
        const float ph = __fmul_rn(wh, qh);
        const float eh = __fmaf_rn(wh, qh, -ph);
        const float a = fmaxf(s, ph), b = fminf(s, ph);
        const float t = __fadd_rn(a, b);
        const float e = __fsub_rn(b, __fsub_rn(t, a));
        s = t;
        c = __fadd_rn(c, __fadd_rn(e, eh));
        c = __fmaf_rn(wh, ql, c);
        c = __fmaf_rn(wl, qh, c);
    }
    // a term of a chunk outside every core: plain FP32 product and sum,
    // added into the running sum once per chunk by Fast2Sum (so the
    // compensation stays of the size of the rounding errors it collects)
    __device__ __forceinline__ void add_tail(float wh, float q) { tail = __fmaf_rn(wh, q, tail); }
    __device__ __forceinline__ void flush_tail() {
        const float a = fmaxf(s, tail), b = fminf(s, tail);
        const float t = __fadd_rn(a, b);
        c = __fadd_rn(c, __fsub_rn(b, __fsub_rn(t, a)));
        s = t;
        tail = 0.0f;
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

// q (< 2^48) as qh + ql, both exact in FP32
__device__ __forceinline__ void split_u64(uint64_t q, float &qh, float &ql) {
    qh = __ull2float_rz(q);
    ql = (float)(int64_t)(q - (uint64_t)qh);
}
__device__ __forceinline__ void split_u32(uint32_t q, float &qh, float &ql) {
    qh = __uint2float_rz(q);
    ql = (float)(int32_t)(q - (uint32_t)qh);
}

}  // namespace nz
