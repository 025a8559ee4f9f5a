// Values of one statistic of the per-step records, as the canonical
// convolutions read them.
#pragma once
#include <cstdint>

#include "nz_common.cuh"

namespace nz {

// Statistic S of the record at `off` (S = 0 spanning, 1 max, 2 m0, 3 m1,
// 4 m2, 5 m3, 6 m4; 7 = m4 of records without the m4_hi plane, whose high
// word is zero; 8 = m0 and 9 = m2 of narrow records, stored as uint16 and
// uint32).  The FP32 loader splits 64-bit words into 32-bit halves so
// that every conversion stays on the FP32 pipe.
template <int S>
__device__ __forceinline__ double record_value(const NzRecords &rec, size_t off, uint32_t N) {
    if (S == 0) return (rec.max_span[off] & kSpanBit) ? 1.0 : 0.0;
    if (S == 1) return (double)(rec.max_span[off] & ~kSpanBit);
    if (S == 2) return (double)rec.m0[off];
    if (S == 3) return (double)(N - (rec.max_span[off] & ~kSpanBit));
    if (S == 4) return (double)rec.m2[off];
    if (S == 5) return (double)rec.m3[off];
    if (S == 7) return (double)rec.m4_lo[off];
    if (S == 8) return (double)reinterpret_cast<const uint16_t *>(rec.m0)[off];
    if (S == 9) return (double)reinterpret_cast<const uint32_t *>(rec.m2)[off];
    return fma((double)rec.m4_hi[off], 18446744073709551616.0, (double)rec.m4_lo[off]);
}

__device__ __forceinline__ float u64_to_f32(uint64_t x) {
    return fmaf((float)(uint32_t)(x >> 32), 4294967296.0f, (float)(uint32_t)x);
}

// m0 and m2 of a record in either layout (narrow: uint16 / uint32)
__device__ __forceinline__ uint32_t record_m0(const NzRecords &rec, size_t off) {
    return rec.narrow ? (uint32_t)reinterpret_cast<const uint16_t *>(rec.m0)[off] : rec.m0[off];
}
__device__ __forceinline__ uint64_t record_m2(const NzRecords &rec, size_t off) {
    return rec.narrow ? (uint64_t)reinterpret_cast<const uint32_t *>(rec.m2)[off] : rec.m2[off];
}

// Where row i of run r lies in a tiled plane of BYTES-wide values: 32 rows of a
// run next to each other (a line of 64, 128 or 256 bytes), which is what a block
// working on one run writes and a thread summing over a run's rows reads; the
// lines of a tile's runs follow each other, so that the rows of many runs are
// one contiguous copy.  Within its line a 16-byte piece is moved by the run's
// number, so that 8 runs' equal rows, once in shared memory, lie in different
// banks.
template <int BYTES>
__device__ __forceinline__ size_t tile_off(int64_t run_stride, uint32_t i, int32_t r) {
    constexpr uint32_t kPer = 16 / BYTES;  // rows per 16 bytes
    const uint32_t turn = BYTES == 2 ? (uint32_t)(r >> 1) & 3u : (uint32_t)r & 7u;
    const size_t line = ((size_t)(i >> 5) * run_stride + r) * 32;
    return line + (((((i & 31u) / kPer) ^ turn) * kPer) | (i & (kPer - 1u)));
}

// The raw words of rows i .. i + 7 (i a multiple of 8) of one run in a tiled
// plane, in 16-byte loads.
template <class T>
__device__ __forceinline__ void load_rows8(const T *plane, int64_t run_stride, uint32_t i, int32_t r, T (&q)[8]) {
    constexpr int kPer = 16 / (int)sizeof(T);
#pragma unroll
    for (int k = 0; k < 8; k += kPer) {
        const uint4 v = *reinterpret_cast<const uint4 *>(plane + tile_off<sizeof(T)>(run_stride, i + k, r));
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int b = 0; b < kPer; ++b) {
            if constexpr (sizeof(T) == 2) q[k + b] = (T)(w[b / 2] >> (16 * (b & 1)));
            else if constexpr (sizeof(T) == 4) q[k + b] = (T)w[b];
            else q[k + b] = (T)(((uint64_t)w[2 * b + 1] << 32) | w[2 * b]);
        }
    }
}

// writes m0 and m2 of a record in either layout
__device__ __forceinline__ void put_m0_m2(const NzRecords &rec, size_t off, uint32_t m0, uint64_t m2) {
    if (rec.narrow) {
        if (rec.m0) reinterpret_cast<uint16_t *>(rec.m0)[off] = (uint16_t)m0;
        if (rec.m2) reinterpret_cast<uint32_t *>(rec.m2)[off] = (uint32_t)m2;
    } else {
        if (rec.m0) rec.m0[off] = m0;
        if (rec.m2) rec.m2[off] = m2;
    }
}

}  // namespace nz
