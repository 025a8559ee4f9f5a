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

template <int S>
__device__ __forceinline__ float record_value_f(const NzRecords &rec, size_t off, uint32_t N) {
    if (S == 0) return (rec.max_span[off] & kSpanBit) ? 1.0f : 0.0f;
    if (S == 1) return (float)(rec.max_span[off] & ~kSpanBit);
    if (S == 2) return (float)rec.m0[off];
    if (S == 3) return (float)(N - (rec.max_span[off] & ~kSpanBit));
    if (S == 4) return u64_to_f32(rec.m2[off]);
    if (S == 5) return u64_to_f32(rec.m3[off]);
    if (S == 7) return u64_to_f32(rec.m4_lo[off]);
    if (S == 8) return (float)reinterpret_cast<const uint16_t *>(rec.m0)[off];
    if (S == 9) return (float)reinterpret_cast<const uint32_t *>(rec.m2)[off];
    return fmaf((float)rec.m4_hi[off], 18446744073709551616.0f, u64_to_f32(rec.m4_lo[off]));
}

// m0 and m2 of a record in either layout (narrow: uint16 / uint32)
__device__ __forceinline__ uint32_t record_m0(const NzRecords &rec, size_t off) {
    return rec.narrow ? (uint32_t)reinterpret_cast<const uint16_t *>(rec.m0)[off] : rec.m0[off];
}
__device__ __forceinline__ uint64_t record_m2(const NzRecords &rec, size_t off) {
    return rec.narrow ? (uint64_t)reinterpret_cast<const uint32_t *>(rec.m2)[off] : rec.m2[off];
}

// Where row i of run r lies in a window's planes.  n-major: runs next to each
// other.  Tiled (bond ensembles): 32 rows of a run next to each other, which is
// what a block working on one run writes and a thread summing over a run's
// rows reads.
__device__ __forceinline__ size_t record_off(const NzRecords &rec, bool tiled, uint32_t i, int32_t r) {
    return tiled ? ((size_t)(i >> 5) * rec.run_stride + r) * 32 + (i & 31u) : (size_t)i * rec.run_stride + r;
}

// The raw words of 8 consecutive rows of one run in a tiled plane (off: the
// first row's place, a multiple of 8 rows), in 16-byte loads.
__device__ __forceinline__ void load_rows8(const uint32_t *plane, size_t off, uint32_t (&q)[8]) {
    const uint4 *v = reinterpret_cast<const uint4 *>(plane + off);
    const uint4 a = v[0], b = v[1];
    q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
    q[4] = b.x; q[5] = b.y; q[6] = b.z; q[7] = b.w;
}
__device__ __forceinline__ void load_rows8(const uint64_t *plane, size_t off, uint64_t (&q)[8]) {
    const ulonglong2 *v = reinterpret_cast<const ulonglong2 *>(plane + off);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const ulonglong2 a = v[k];
        q[2 * k] = a.x;
        q[2 * k + 1] = a.y;
    }
}
__device__ __forceinline__ void load_rows8(const uint16_t *plane, size_t off, uint16_t (&q)[8]) {
    const uint4 a = *reinterpret_cast<const uint4 *>(plane + off);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q[2 * k] = (uint16_t)w[k];
        q[2 * k + 1] = (uint16_t)(w[k] >> 16);
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
