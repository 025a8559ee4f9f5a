// nz_thread.cuh -- Newman-Ziff steps of one run in one thread: its totals, and the
// union of two clusters whose node words lie in global memory.
//
// Per step the exact totals T_k = sum over all clusters of s^k are updated by
// (a + b)^k - a^k - b^k where sizes a and b merge, and the largest size S is kept;
// the reference's moments are T_k - S^k.  Spanning (percolate/hpc.py:224-274): a
// root carries the sides its cluster touches, and the run's flag is set at the
// first union that produces a root touching both sides (or at the first union at
// all where some node touches both).
#pragma once

#include <cstdint>

#include "nz_common.cuh"

namespace nz {
namespace thread {

constexpr uint32_t kEmpty = kRoot;  // make_root(0, 0): an unoccupied site
constexpr int kMaxHops = 64;        // union by size: log2(N) <= 21; guards against corrupted words only

__device__ __forceinline__ void add128(uint64_t &lo, uint64_t &hi, uint64_t blo, uint64_t bhi) {
    const uint64_t nlo = lo + blo;
    hi += bhi + (nlo < lo ? 1ull : 0ull);
    lo = nlo;
}

// Totals of a run.
struct Tally {
    RunState st;

    // a new cluster of one site
    __device__ __forceinline__ void add_single() {
        st.t0 += 1u;
        st.t2 += 1u;
        st.t3 += 1u;
        add128(st.t4_lo, st.t4_hi, 1u, 0u);
        st.max = max(st.max, 1u);
    }
    // clusters of sizes a and b become one
    __device__ __forceinline__ void merge(uint32_t a, uint32_t b) {
        const uint32_t s = a + b;
        st.t0 -= 1u;
        const uint64_t ab = (uint64_t)a * b;
        st.t2 += 2ull * ab;
        st.t3 += 3ull * ab * s;
        const uint64_t q = 4ull * a * a + 6ull * ab + 4ull * b * b;
        add128(st.t4_lo, st.t4_hi, ab * q, __umul64hi(ab, q));
        st.max = max(st.max, s);
    }
};

// Joins the clusters of u and v, whose words are wu and wv (interleaved finds
// with path splitting, union by size).
__device__ __forceinline__ void link(uint32_t *node, uint32_t xu, uint32_t xv, uint32_t wu, uint32_t wv, bool span,
                                     Tally &t) {
    for (int hops = 0; !(is_root(wu) && is_root(wv)); ++hops) {
        if (hops >= kMaxHops) { t.st.flags |= kFlagCorrupt; return; }
        if (!is_root(wu)) {
            const uint32_t nu = node[wu];
            if (!is_root(nu)) node[xu] = nu;
            xu = wu; wu = nu;
        }
        if (!is_root(wv)) {
            const uint32_t nv = node[wv];
            if (!is_root(nv)) node[xv] = nv;
            xv = wv; wv = nv;
        }
    }
    if (xu == xv) return;
    const uint32_t a = root_size(wu), b = root_size(wv);
    const uint32_t sides = root_sides(wu) | root_sides(wv);
    node[a < b ? xu : xv] = a < b ? xv : xu;
    node[a < b ? xv : xu] = make_root(a + b, sides);
    t.merge(a, b);
    if (span && (sides == 3u || (t.st.flags & kFlagInitBoth))) t.st.flags |= kFlagSpan;
}

}  // namespace thread
}  // namespace nz
