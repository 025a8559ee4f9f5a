// nz_group_rows.cuh -- per-step records, one run per thread block (nz_group.cuh):
// the kernel and its launch shapes, for nz_ufg.cu (bonds) and nz_lattice.cu
// (sites).
#pragma once
#include <cstdint>

#include "nz_common.cuh"
#include "nz_group.cuh"
#include "nz_internal.cuh"
#include "nz_records.cuh"

namespace nz {
namespace group {

// Bonds: rows i0, i0 + 1 of run r (window rows; i0 is even), in tiles or
// n-major.  Both rows lie in one 16-byte piece of a tile, and the planes hold
// whole tiles.  Sites: row i0.
template <bool NARROW, int E>
__device__ __forceinline__ void put_rows(const NzRecords &rec, bool tiled, uint32_t i0, uint32_t rows, int32_t r,
                                         const uint32_t (&ms)[E], const uint32_t (&m0)[E],
                                         const Sums<NARROW> (&m)[E], const uint32_t (&e)[E]) {
    if (i0 >= rows) return;
    if (E == 2 && tiled) {
        const size_t o4 = tile_off<4>(rec.run_stride, i0, r), o8 = tile_off<8>(rec.run_stride, i0, r);
        *reinterpret_cast<uint2 *>(rec.max_span + o4) = make_uint2(ms[0], ms[E - 1]);
        if (rec.narrow) {
            const size_t o2 = tile_off<2>(rec.run_stride, i0, r);
            *reinterpret_cast<uint32_t *>(reinterpret_cast<uint16_t *>(rec.m0) + o2) = m0[0] | (m0[E - 1] << 16);
            *reinterpret_cast<uint2 *>(reinterpret_cast<uint32_t *>(rec.m2) + o4) =
                make_uint2((uint32_t)m[0].m2(), (uint32_t)m[E - 1].m2());
        } else {
            *reinterpret_cast<uint2 *>(rec.m0 + o4) = make_uint2(m0[0], m0[E - 1]);
            *reinterpret_cast<ulonglong2 *>(rec.m2 + o8) = make_ulonglong2(m[0].m2(), m[E - 1].m2());
        }
        *reinterpret_cast<ulonglong2 *>(rec.m3 + o8) = make_ulonglong2(m[0].u3, m[E - 1].u3);
        *reinterpret_cast<ulonglong2 *>(rec.m4_lo + o8) = make_ulonglong2(m[0].u4, m[E - 1].u4);
        if (rec.m4_hi) *reinterpret_cast<uint2 *>(rec.m4_hi + o4) = make_uint2(m[0].m4_hi(), m[E - 1].m4_hi());
        return;
    }
    if (tiled) {
        const size_t o4 = tile_off<4>(rec.run_stride, i0, r), o8 = tile_off<8>(rec.run_stride, i0, r);
        rec.max_span[o4] = ms[0];
        if (rec.narrow) {
            reinterpret_cast<uint16_t *>(rec.m0)[tile_off<2>(rec.run_stride, i0, r)] = (uint16_t)m0[0];
            reinterpret_cast<uint32_t *>(rec.m2)[o4] = (uint32_t)m[0].m2();
        } else {
            rec.m0[o4] = m0[0];
            rec.m2[o8] = m[0].m2();
        }
        rec.m3[o8] = m[0].u3;
        rec.m4_lo[o8] = m[0].u4;
        if (rec.m4_hi) rec.m4_hi[o4] = m[0].m4_hi();
        return;
    }
#pragma unroll
    for (int k = 0; k < E; ++k) {
        if (i0 + k >= rows) break;
        const size_t off = (size_t)(i0 + k) * rec.run_stride + r;
        if (rec.max_span) rec.max_span[off] = ms[k];
        put_m0_m2(rec, off, m0[k], m[k].m2());
        if (rec.m3) rec.m3[off] = m[k].u3;
        if (rec.m4_lo) rec.m4_lo[off] = m[k].u4;
        if (rec.m4_hi) rec.m4_hi[off] = m[k].m4_hi();
        if (rec.edge) rec.edge[off] = e[k];
    }
}

struct RowSink {
    NzRecords rec;
    bool tiled;
    int32_t r;
    uint32_t rows;
    __device__ __forceinline__ bool wants(uint32_t, uint32_t) const { return true; }
    template <bool NARROW, int E>
    __device__ __forceinline__ void put(uint32_t i0, const uint32_t (&ms)[E], const uint32_t (&m0)[E],
                                        const Sums<NARROW> (&m)[E], const uint32_t (&e)[E]) const {
        put_rows<NARROW, E>(rec, tiled, i0, rows, r, ms, m0, m, e);
    }
};

// Block r adds the bonds (sites) of rows [n_begin, n_end) of run r.
template <int W, bool SHARED, bool TORUS, bool SITE>
__global__ void __launch_bounds__(32 * W, 24 / W) uf_group_kernel(UfParams p, uint32_t claim_count, bool given, bool spanning) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ GroupShared<W, SHARED> sh;
    const int32_t r = blockIdx.x;
    Claims<W> claims;
    claims.init(reinterpret_cast<uint32_t *>(smem), claim_count);
    Run run;
    run.perm = given ? p.perms + (size_t)r * p.g.M : nullptr;
    run.key = p.key;
    run.id = p.run0 + (uint64_t)r;
    run.home = p.nodes + (size_t)r * p.g.slots;
    run.state = p.state + r;
    run.n_begin = p.n_begin;
    run.n_end = p.n_end;
    run.spanning = spanning;
    run.init_both = p.init_flag && *p.init_flag;
    RowSink sink{p.rec, p.tiled, r, p.n_end - p.n_begin};
    const bool bad = group_run<W, SHARED, TORUS, SITE>(p.g, run, sh, claims, smem + (size_t)claim_count * 4u, sink);
    if (bad && p.errors && threadIdx.x == 0) atomicAdd(p.errors, 1u);
}

// Runs that an SM has room and work for at a time: as many as fit with some 1,100
// words of claims each, spread evenly over the waves that takes (3,000 chains of
// 6,000, 20 to an SM: 9, 9 and 2 at a time 0.86 ms, 7, 7 and 6 0.72).
inline int runs_per_sm(const UfParams &p) {
    const uint32_t N = p.g.N;
    const bool torus = p.g.kind == NZ_GRAPH_TORUS2D;
    const int runs = (p.n_runs + 151) / 152;
    if (N > (torus ? kSharedTorus : kSharedNodes)) return runs < 2 ? runs : 2;
    const int fit = (int)(226u * 1024u / ((torus ? node_bytes<true>(N) : node_bytes<false>(N)) + 6144u));
    const int waves = (runs + fit - 1) / fit;
    return (runs + waves - 1) / waves;
}

template <int W, bool SHARED, bool TORUS, bool SITE>
cudaError_t launch_group(const UfParams &p, bool given, bool span, cudaStream_t s) {
    const uint32_t nodes = SHARED ? node_bytes<TORUS>(p.g.N) : 0u;
    const int blocks = min(24 / W, runs_per_sm(p));
    const uint32_t claims = claim_words<W, SHARED>(node_count<SHARED, TORUS>(p.g), nodes, (uint32_t)blocks);
    const size_t smem = (size_t)claims * 4u + nodes;
    return launch_kernel(uf_group_kernel<W, SHARED, TORUS, SITE>, dim3(p.n_runs), 32 * W, smem, most_shared<W, SHARED>(), s, p,
                         claims, given, span);
}

// Warps per run.  In shared memory: kWarpsPerSm warps on every SM (80 registers
// a thread) with the runs that are there and that fit, and batches of at most
// an eighth of a run.  More warps per SM beat smaller batches until there are
// about 24 (ms by warps per run 1, 2, 4, 8: 4,000 runs of 97 x 97, 6 to an SM,
// 6.5, 4.1, 3.3, 3.6 with 4,096 words of claims; 20,000 runs of 32 x 32, 24 to an SM, 1.1, 1.4, 1.9, 3.0).
// In global memory: 12 warps, two runs to an SM, so that the nodes of the
// resident runs stay near L2's size (200 runs of 512 x 512: 18.6, 11.1, 9.3,
// 10.7 ms with 4, 8, 12, 24), 24 where there are no more runs than SMs.  Sites
// alike (300 runs of 400 x 400: 8.7, 7.0, 8.3 ms with 8, 12, 24; 100 of 300 x
// 300: 3.7 and 2.5 with 8 and 24).
constexpr int kWarpsPerSm = 24;
constexpr int kWarpChoices[8] = {1, 2, 3, 4, 6, 8, 12, 24};
inline int group_warps(const UfParams &p, bool site) {
    const uint32_t N = p.g.N;
    if (N > (p.g.kind == NZ_GRAPH_TORUS2D ? kSharedTorus : kSharedNodes)) return p.n_runs <= 152 ? 24 : 12;
    const int runs = runs_per_sm(p);
    int w = 1;
    for (int c : kWarpChoices)
        if (c * runs <= kWarpsPerSm && (site ? 32u : 64u) * c * 8u <= p.g.M) w = c;
    return w;
}

template <bool TORUS, bool SITE>
cudaError_t launch_groups(const UfParams &p, bool given, bool span, cudaStream_t s) {
    const int warps = group_warps(p, SITE);
    if (p.g.N <= (TORUS ? kSharedTorus : kSharedNodes)) {
        switch (warps) {
            case 1: return launch_group<1, true, TORUS, SITE>(p, given, span, s);
            case 2: return launch_group<2, true, TORUS, SITE>(p, given, span, s);
            case 3: return launch_group<3, true, TORUS, SITE>(p, given, span, s);
            case 4: return launch_group<4, true, TORUS, SITE>(p, given, span, s);
            case 6: return launch_group<6, true, TORUS, SITE>(p, given, span, s);
            case 8: return launch_group<8, true, TORUS, SITE>(p, given, span, s);
            case 12: return launch_group<12, true, TORUS, SITE>(p, given, span, s);
            default: return launch_group<24, true, TORUS, SITE>(p, given, span, s);
        }
    }
    if (warps == 12) return launch_group<12, false, TORUS, SITE>(p, given, span, s);
    return launch_group<24, false, TORUS, SITE>(p, given, span, s);
}

}  // namespace group
}  // namespace nz
