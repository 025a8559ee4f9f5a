// nz_mix.cu -- batched uneven ensembles: one launch per range of sizes.
//
// n_runs independent runs whose substrate is drawn per run: with probability
// chain_share a spanning_1d_chain(l), l log-uniform in [chain_min, chain_max],
// otherwise a spanning_2d_grid(L), L log-uniform in [grid_min, grid_max]
// (percolate/percolate.py:899-965).  The draw and the bond permutation of
// run r both come from Philox-4x32-10 keyed by `key` at counter r.
//
// Pipeline (all on the caller's stream, no host synchronisation):
//   1. mix_class_kernel   : class of every run (threshold tables, no libm),
//                           histogram of classes;
//   2. mix_offsets_kernel : classes ordered by node words S descending
//                           (longest-first scheduling) -> segment offsets;
//                           S = l for a chain, grid_slots(L) >= L^2 for a
//                           grid, whose sites sit in 4 x 2 blocks per sector;
//   3. mix_scatter_kernel : run ids bucketed into a queue sorted by S desc;
//   4. mix_segments_kernel: where in the queue the lattices stop needing more
//      than 65,536, 16,384, 4,096 and 1,024 node words;
//   5. mix_group_kernel   : the union-find, one launch per segment of the queue,
//      a run per thread block (nz_group.cuh) with as many warps as fill the SMs
//      with the blocks that fit there: node words in global memory above
//      65,536, in shared memory below.  The blocks stay and claim runs with an
//      atomic counter, the largest lattices first.  (Very many runs of lattices of
//      at most 4,096 words with the fused reduction: mix_thread_kernel, a run per
//      thread.)
//      At F evenly spaced occupation checkpoints
//      n_j = floor(j M / (F - 1)) each run either writes its exact
//      statistics (records) or, with the fused reduction, adds them and
//      their squares into its class's cell j itself (integer atomics of
//      32-bit limbs: exact, and independent of the order the runs finish in);
//   6. mix_reduce_kernel  : per (class, checkpoint) exact integer sums of x
//      and x^2 (up to 192 bits) over the class's records -> mean and M2
//      (percolate/percolate.py:450-705 semantics at those n); or
//      mix_finalize_kernel: the same sums and M2 from the fused cells.
//   Both reductions give identical results; which is faster depends on the
//   mix of lattices (many runs per lattice favour the fused one).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "nz_common.cuh"
#include "nz_group.cuh"
#include "nz_internal.cuh"
#include "nz_thread.cuh"
#include "nz_wide.cuh"

namespace nz {

constexpr uint32_t kSizeTag = 0x53495A45u;  // "SIZE"


__device__ __forceinline__ uint32_t class_of_run(const MixDev &m, uint64_t key, uint64_t r) {
    uint32_t c[4] = {(uint32_t)r, (uint32_t)(r >> 32), 0u, kSizeTag};
    philox4x32_10(c, (uint32_t)key, (uint32_t)(key >> 32));
    const bool chain = c[0] < m.chain_share;
    const uint32_t *thr = chain ? m.thr_chain : m.thr_grid;
    const uint32_t n = chain ? m.n_chain : m.n_grid;
    // largest i with thr[i] <= u (thr[0] == 0)
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (thr[mid] <= c[1]) lo = mid; else hi = mid;
    }
    return chain ? m.n_grid + lo : lo;
}

__device__ __forceinline__ void class_graph(const MixDev &m, uint32_t cls, uint32_t &kind, uint32_t &L,
                                            uint32_t &N, uint32_t &M) {
    if (cls < m.n_grid) {
        kind = NZ_GRAPH_GRID2D; L = m.grid_min + cls; N = L * L; M = 2u * L * (L - 1u);
    } else {
        kind = NZ_GRAPH_CHAIN1D; L = m.chain_min + (cls - m.n_grid); N = L; M = L - 1u;
    }
}

// node words a run of class cls needs: grid_slots(L) (the tiled layout) or l
__device__ __forceinline__ uint32_t class_slots(const MixDev &m, uint32_t cls) {
    return cls < m.n_grid ? grid_slots(m.grid_min + cls) : m.chain_min + (cls - m.n_grid);
}

// the rest of the GraphDev of class cls, whose L, N and M are set
__device__ __forceinline__ void set_class_graph(const MixDev &m, uint32_t cls, uint32_t kind, GraphDev &g) {
    g.kind = (int32_t)kind; g.site = 0; g.wrap = 0;
    g.slots = class_slots(m, cls);
    g.tile_cols = kind == NZ_GRAPH_GRID2D ? (g.L + 3u) >> 2 : 0u;
    g.two_l_m1 = kind == NZ_GRAPH_GRID2D ? 2u * g.L - 1u : 1u;
    g.row_edges = kind == NZ_GRAPH_GRID2D ? (g.L - 1u) * g.two_l_m1 : 0u;
    g.inv_two_l_m1 = 1.0f / (float)g.two_l_m1;
    g.eu = g.ev = nullptr; g.side = nullptr;
}

__global__ void mix_class_kernel(MixDev m, uint32_t *cls, uint32_t *counts) {
    const uint64_t key = *m.key_ptr;
    for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < m.n_runs; r += gridDim.x * blockDim.x) {
        const uint32_t c = class_of_run(m, key, (uint64_t)r);
        cls[r] = c;
        atomicAdd(&counts[c], 1u);
    }
}

// Position of every class in the order "node words S descending, grids
// before chains on equal S" (grid S = grid_slots(L) and chain S = l are
// non-decreasing in the length).  Ordering by the words a run needs -- not
// by M -- makes the queue's segments (lattices that need at most so many
// words) contiguous.
__global__ void mix_order_kernel(MixDev m, uint32_t *order) {
    const uint32_t n_classes = m.n_grid + m.n_chain;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n_classes; c += gridDim.x * blockDim.x) {
        uint32_t rank;
        if (c < m.n_grid) {
            const uint64_t Nc = grid_slots(m.grid_min + c);
            // chains with more words: l >= Nc + 1
            const uint64_t lo = Nc + 1u;
            const uint32_t more = lo > m.chain_max ? 0u
                                : (uint32_t)(m.chain_max - (lo > m.chain_min ? lo : (uint64_t)m.chain_min) + 1u);
            rank = (m.n_grid - 1u - c) + more;
        } else {
            const uint32_t k = c - m.n_grid;
            const uint64_t Nk = (uint64_t)m.chain_min + k;
            // grids with at least as many words: smallest L in range with
            // grid_slots(L) >= Nk
            uint32_t a = m.grid_min, b = m.grid_max + 1u;
            while (a < b) {
                const uint32_t mid = (a + b) >> 1;
                if ((uint64_t)grid_slots(mid) >= Nk) b = mid; else a = mid + 1u;
            }
            rank = (m.n_chain - 1u - k) + (m.grid_max + 1u - a);
        }
        order[rank] = c;
    }
}

// Single block: exclusive scan of counts taken in the order `order` (classes
// by N descending) -> offsets[c]; also the cursor copy used by the scatter.
__global__ void mix_offsets_kernel(const uint32_t *counts, const uint32_t *order, uint32_t n_classes,
                                   uint32_t *offsets, uint32_t *cursor) {
    __shared__ uint32_t s[1024];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n_classes; base += 1024) {
        const uint32_t i = base + threadIdx.x;
        const uint32_t v = i < n_classes ? counts[order[i]] : 0u;
        s[threadIdx.x] = v;
        __syncthreads();
        for (int off = 1; off < 1024; off <<= 1) {
            const uint32_t y = threadIdx.x >= (unsigned)off ? s[threadIdx.x - off] : 0u;
            __syncthreads();
            s[threadIdx.x] += y;
            __syncthreads();
        }
        if (i < n_classes) {
            const uint32_t ex = carry + s[threadIdx.x] - v;
            offsets[order[i]] = ex;
            cursor[order[i]] = ex;
        }
        __syncthreads();
        if (threadIdx.x == 1023) carry += s[1023];
        __syncthreads();
    }
}

__global__ void mix_scatter_kernel(int32_t n_runs, const uint32_t *cls, uint32_t *cursor, uint32_t *queue) {
    for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_runs; r += gridDim.x * blockDim.x)
        queue[atomicAdd(&cursor[cls[r]], 1u)] = (uint32_t)r;
}

// Segment k of the queue: runs whose lattices need at most segment_words(k - 1)
// node words (any, for k = 0) but more than segment_words(k).
constexpr int kSegments = kMixSegments;
__host__ __device__ constexpr uint32_t segment_words(int k) {
    return k == 0 ? group::kSharedNodes : k == 1 ? 16384u : k == 2 ? 4096u : k == 3 ? 1024u : 0u;
}

// begin[k] and head[k] = the first queue position of segment k, begin[kSegments]
// = n_runs: class order[k] starts segment j if it is the first class in the
// order with at most segment_words(j - 1) words.
__global__ void mix_segments_kernel(MixDev m, const uint32_t *order, const uint32_t *offsets, uint32_t *begin,
                                    uint32_t *head) {
    const uint32_t n_classes = m.n_grid + m.n_chain;
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k == 0) {
        begin[0] = head[0] = 0;
        begin[kSegments] = (uint32_t)m.n_runs;
    }
    if (k > n_classes) return;
    // position n_classes stands for "no class left"
    const uint32_t at = k < n_classes ? offsets[order[k]] : (uint32_t)m.n_runs;
    const uint32_t words = k < n_classes ? class_slots(m, order[k]) : 0u;
    const uint32_t above = k > 0 ? class_slots(m, order[k - 1]) : 0xffffffffu;
    for (int j = 1; j < kSegments; ++j)
        if (words <= segment_words(j - 1) && above > segment_words(j - 1)) begin[j] = head[j] = at;
}

// ------------------------------------------------------- fused reduction
// Cell words.  Each word sums one 32-bit limb over the class's runs: at most
// NZ_MAX_RUNS = 2^24 limbs < 2^32, so no word can overflow.  With N <= 2^21:
// max, m0 < 2^21, m2 < 2^42, m3 < 2^63, m4 < 2^84.
//   0 runs with a spanning cluster
//   sums of x:   1 max, 2 m0, 3-4 m2, 5-6 m3, 7-9 m4
//   sums of x^2: 10-11 max, 12-13 m0, 14-16 m2, 17-20 m3, 21-26 m4
// (m1 = N - max follows from the max sums.)
constexpr int kCellSpan = 0, kSxMax = 1, kSxM0 = 2, kSxM2 = 3, kSxM3 = 5, kSxM4 = 7;
constexpr int kSqMax = 10, kSqM0 = 12, kSqM2 = 14, kSqM3 = 17, kSqM4 = 21;
static_assert(kSqM4 + 6 == kMixCellWords, "cell layout");

// Adds 32-bit limbs into the words of one cell.  When every active lane of
// the warp adds into the same cell (with a thread per run, neighbours in the queue
// being runs of one lattice), the lanes' limbs are summed first (redux.sync on
// 16-bit halves, so 32 lanes' sums fit 32 bits) and one lane issues the
// atomic: 27 atomics per warp and checkpoint instead of up to 27 x 32.
struct CellAdder {
    uint64_t *cell;
    unsigned mask;
    bool warp, leader;
    __device__ __forceinline__ explicit CellAdder(uint64_t *c) : cell(c) {
        mask = __activemask();
        warp = __match_any_sync(mask, (unsigned long long)(uintptr_t)c) == mask;
        leader = (threadIdx.x & 31u) == (unsigned)(__ffs(mask) - 1);
    }
    __device__ __forceinline__ void limb(int k, uint32_t v) const {
        if (warp) {
            const uint32_t lo = __reduce_add_sync(mask, v & 0xffffu);
            const uint32_t hi = __reduce_add_sync(mask, v >> 16);
            const uint64_t sum = (uint64_t)lo + ((uint64_t)hi << 16);
            if (leader && sum) atomicAdd(reinterpret_cast<unsigned long long *>(cell + k), (unsigned long long)sum);
        } else if (v) {
            atomicAdd(reinterpret_cast<unsigned long long *>(cell + k), (unsigned long long)v);
        }
    }
    __device__ __forceinline__ void u64(int k, uint64_t v) const {
        limb(k, (uint32_t)v);
        limb(k + 1, (uint32_t)(v >> 32));
    }
    template <int LIMBS>
    __device__ __forceinline__ void wide(int k, u128 v) const {
#pragma unroll
        for (int i = 0; i < LIMBS; ++i) limb(k + i, (uint32_t)(v >> (32 * i)));
    }
};

// One run's statistics at one checkpoint into its class's cell.
__device__ __forceinline__ void mix_checkpoint(uint64_t *cell, uint32_t mx, bool span, uint32_t m0, uint64_t m2,
                                               uint64_t m3, uint64_t m4lo, uint32_t m4hi) {
    const CellAdder a(cell);
    a.limb(kCellSpan, span ? 1u : 0u);
    a.limb(kSxMax, mx);
    a.limb(kSxM0, m0);
    a.u64(kSxM2, m2);
    a.u64(kSxM3, m3);
    a.u64(kSxM4, m4lo);
    a.limb(kSxM4 + 2, m4hi);
    a.u64(kSqMax, (uint64_t)mx * mx);
    a.u64(kSqM0, (uint64_t)m0 * m0);
    a.wide<3>(kSqM2, (u128)m2 * m2);
    a.wide<4>(kSqM3, (u128)m3 * m3);
    // m4^2 = lo^2 + 2 lo hi 2^64 + hi^2 2^128 (< 2^168) as three 64-bit words
    const u128 ll = (u128)m4lo * m4lo;
    const u128 mid = ((u128)m4lo * m4hi) << 1;  // < 2^85
    const u128 t = (ll >> 64) + (uint64_t)mid;  // < 2^65
    a.u64(kSqM4, (uint64_t)ll);
    a.u64(kSqM4 + 2, (uint64_t)t);
    a.u64(kSqM4 + 4, (uint64_t)(t >> 64) + (uint64_t)(mid >> 64) + (uint64_t)m4hi * m4hi);
}

// Where a run's checkpoints go: its records (queue position `pos`, F
// entries) or its class's F cells.
template <bool FUSED>
struct MixSink {
    MixRec rec;
    size_t rec_base;
    uint64_t *cells;
    uint32_t F, M;
    uint32_t base, batch;  // rows of the current batch
    uint32_t j, target;    // next checkpoint and its row
    bool dense;            // a checkpoint every 8 rows or more often

    __device__ __forceinline__ uint32_t row_of(uint32_t jj) const {
        return (uint32_t)(((uint64_t)jj * M) / (F - 1u));
    }
    __device__ __forceinline__ void start() {
        j = target = 0;
        dense = (uint64_t)(F - 1u) * 8u >= M;
    }
    __device__ __forceinline__ bool wants(uint32_t first, uint32_t rows) {
        base = first;
        batch = rows;
        return dense || (j < F && target < first + rows);
    }
    __device__ __forceinline__ void write(uint32_t jj, uint32_t ms, uint32_t m0, uint64_t m2, uint64_t m3,
                                          uint64_t m4lo, uint32_t m4hi) const {
        if (FUSED) {
            mix_checkpoint(cells + (size_t)jj * kMixCellWords, ms & ~kSpanBit, (ms & kSpanBit) != 0, m0, m2, m3, m4lo,
                           m4hi);
        } else {
            const size_t off = rec_base + jj;
            rec.max_span[off] = ms;
            rec.m0[off] = m0;
            rec.m2[off] = m2;
            rec.m3[off] = m3;
            rec.m4_lo[off] = m4lo;
            rec.m4_hi[off] = m4hi;
        }
    }
    template <bool NARROW>
    __device__ __forceinline__ void put(uint32_t i0, const uint32_t (&ms)[group::kE], const uint32_t (&m0)[group::kE],
                                        const group::Sums<NARROW> (&m)[group::kE], const uint32_t (&)[group::kE]) {
        if (dense) {
            // every thread looks up the checkpoints of its rows (several
            // share a row when F - 1 > M)
#pragma unroll
            for (int k = 0; k < group::kE; ++k) {
                const uint32_t n = i0 + k;
                if (n > M) break;
                uint32_t jj = M > 0 ? (uint32_t)(((uint64_t)n * (F - 1u) + M - 1u) / M) : 0u;
                for (; jj < F && row_of(jj) == n; ++jj)
                    write(jj, ms[k], m0[k], m[k].m2(), m[k].u3, m[k].u4, m[k].m4_hi());
            }
            return;
        }
        // the block walks the batch's checkpoints; the row's thread writes
        while (j < F && target < base + batch) {
#pragma unroll
            for (int k = 0; k < group::kE; ++k)
                if (i0 + k == target) write(j, ms[k], m0[k], m[k].m2(), m[k].u3, m[k].u4, m[k].m4_hi());
            ++j;
            if (j < F) target = row_of(j);
        }
    }
};

template <int W, bool SHARED, bool FUSED>
__global__ void __launch_bounds__(32 * W, 24 / W) mix_group_kernel(MixLaunch p, int segment, uint32_t claim_count,
                                                                   uint64_t home_words) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ group::GroupShared<W, SHARED> sh;
    __shared__ GraphDev g;
    __shared__ uint32_t s_pos;
    group::Claims<W> claims;
    claims.init(reinterpret_cast<uint32_t *>(smem), claim_count);
    const uint32_t end = p.begin[segment + 1];
    group::Run run;
    run.perm = nullptr;
    run.key = *p.m.key_ptr;
    run.home = SHARED ? nullptr : p.nodes + (size_t)blockIdx.x * home_words;
    run.state = nullptr;
    run.n_begin = 0;
    run.spanning = true;
    run.init_both = false;
    for (;;) {
        if (threadIdx.x == 0) s_pos = atomicAdd(p.head + segment, 1u);
        __syncthreads();
        const uint32_t pos = s_pos;
        if (pos >= end) break;
        const uint32_t id = p.queue[pos], cls = p.cls[id];
        uint32_t kind, L, N, M;
        class_graph(p.m, cls, kind, L, N, M);
        if (threadIdx.x == 0) {
            g.L = L; g.N = N; g.M = M;
            set_class_graph(p.m, cls, kind, g);
        }
        __syncthreads();
        run.id = id;
        run.n_end = M + 1u;
        MixSink<FUSED> sink;
        sink.rec = p.rec;
        sink.rec_base = (size_t)pos * (uint32_t)p.m.F;
        sink.cells = FUSED ? p.cells + (size_t)cls * (uint32_t)p.m.F * kMixCellWords : nullptr;
        sink.F = (uint32_t)p.m.F;
        sink.M = M;
        sink.start();
        const bool bad = group::group_run<W, SHARED, false, false>(g, run, sh, claims, smem + (size_t)claim_count * 4u, sink);
        if (bad && threadIdx.x == 0) atomicAdd(p.acc.errors, 1u);
        __syncthreads();
    }
}

// The fused reduction of small lattices: a thread per run.  Runs of one lattice
// are neighbours in the queue, so a warp's lanes mostly reach their checkpoints
// together and add their limbs up before one of them adds to the cell (27 atomics
// a warp and checkpoint).  Blocks of a run each would issue these per run.
// `node`: this thread's slot, as many words as the segment's largest lattice has.
template <int KIND>
__device__ __forceinline__ void mix_thread_run(const MixDev &m, uint64_t key, uint32_t id, const GraphDev &g,
                                               uint32_t *node, uint64_t *cells, uint32_t *errors) {
    for (uint32_t j = 0; j < g.slots; ++j) {
        uint32_t i = j;
        if (KIND == NZ_GRAPH_GRID2D && kGridTiled) {
            const uint32_t tile = j >> 3, w = j & 7u, tr = tile / g.tile_cols, tc = tile - tr * g.tile_cols;
            const uint32_t row = 2u * tr + (w >> 2), col = 4u * tc + (w & 3u);
            if (row >= g.L || col >= g.L) continue;  // a padding slot, never read
            i = row * g.L + col;
        }
        node[j] = make_root(1u, node_sides<KIND>(g, i));
    }
    FeistelPerm fp;
    fp.init(key, id, g.M);
    thread::Tally t;
    t.st.t2 = t.st.t3 = t.st.t4_lo = t.st.t0 = g.N;
    t.st.t4_hi = 0;
    t.st.max = 1;
    t.st.flags = 0;
    const uint32_t F = (uint32_t)m.F;
    auto row_of = [&](uint32_t j) { return (uint32_t)(((uint64_t)j * g.M) / (F - 1u)); };
    uint32_t j = 0, target = 0;
    for (uint32_t n = 0; n <= g.M; ++n) {
        if (n > 0) {
            uint32_t u, v;
            decode_edge_slots<KIND>(g, fp.at(n - 1u), u, v);
            thread::link(node, u, v, node[u], node[v], true, t);
        }
        if (n != target) continue;
        const RunState &st = t.st;
        const uint64_t mx = st.max, mx2 = mx * mx, mx3 = mx2 * mx, mx4_lo = mx3 * mx;
        const uint32_t m4_hi = (uint32_t)(st.t4_hi - __umul64hi(mx3, mx) - (st.t4_lo < mx4_lo ? 1u : 0u));
        while (j < F && n == target) {  // several checkpoints share row n where F - 1 > M
            mix_checkpoint(cells + (size_t)j * kMixCellWords, st.max, (st.flags & kFlagSpan) != 0, st.t0 - 1u,
                           st.t2 - mx2, st.t3 - mx3, st.t4_lo - mx4_lo, m4_hi);
            ++j;
            if (j < F) target = row_of(j);
        }
    }
    if (t.st.flags & kFlagCorrupt) atomicAdd(errors, 1u);
}

// (80 registers: 6 blocks on an SM)
constexpr int kMixThreads = 128;
__global__ void __launch_bounds__(kMixThreads, 6) mix_thread_kernel(MixLaunch p, int segment, uint32_t threads,
                                                                    uint32_t slot_words) {
    const uint32_t t = blockIdx.x * kMixThreads + threadIdx.x;
    if (t >= threads) return;
    const uint64_t key = *p.m.key_ptr;
    const uint32_t end = p.begin[segment + 1];
    uint32_t *node = p.nodes + (size_t)t * slot_words;
    for (uint32_t pos = atomicAdd(p.head + segment, 1u); pos < end; pos = atomicAdd(p.head + segment, 1u)) {
        const uint32_t id = p.queue[pos], cls = p.cls[id];
        uint32_t kind;
        GraphDev g;
        class_graph(p.m, cls, kind, g.L, g.N, g.M);
        set_class_graph(p.m, cls, kind, g);
        uint64_t *cells = p.cells + (size_t)cls * (uint32_t)p.m.F * kMixCellWords;
        if (kind == NZ_GRAPH_GRID2D) mix_thread_run<NZ_GRAPH_GRID2D>(p.m, key, id, g, node, cells, p.acc.errors);
        else mix_thread_run<NZ_GRAPH_CHAIN1D>(p.m, key, id, g, node, cells, p.acc.errors);
    }
}

// ---------------------------------------------------------------- reduction
// grid (classes, ceil(F / 32)); thread = checkpoint j; loop over the class's runs.
__global__ void mix_reduce_kernel(MixDev m, const uint32_t *counts, const uint32_t *offsets, MixRec rec,
                                  MixAccum acc, uint32_t n_classes) {
    const uint32_t c = blockIdx.x;
    const uint32_t j = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= n_classes || j >= (uint32_t)m.F) return;
    const uint32_t cnt = counts[c], off = offsets[c];
    uint32_t kind, L, N, M;
    class_graph(m, c, kind, L, N, M);
    (void)kind; (void)L; (void)M;
    uint32_t span = 0;
    u128 sx[6] = {0, 0, 0, 0, 0, 0};
    U256 sq[6];
    for (int k = 0; k < 6; ++k) sq[k] = U256{{0, 0, 0, 0}};
    for (uint32_t i = 0; i < cnt; ++i) {
        const size_t o = (size_t)(off + i) * (uint32_t)m.F + j;
        const uint32_t ms = rec.max_span[o];
        const uint32_t mxv = ms & ~kSpanBit;
        span += ms >> 31;
        const u128 x[6] = {mxv, rec.m0[o], (u128)(N - mxv), rec.m2[o], rec.m3[o],
                           ((u128)rec.m4_hi[o] << 64) | rec.m4_lo[o]};
        for (int k = 0; k < 6; ++k) {
            sx[k] += x[k];
            u256_add(sq[k], u128_sq(x[k]));
        }
    }
    const size_t cj = (size_t)c * (uint32_t)m.F + j;
    const size_t plane = (size_t)n_classes * (uint32_t)m.F;
    if (j == 0) acc.count[c] = cnt;
    acc.span[cj] = span;
    for (int k = 0; k < 6; ++k) {
        acc.sum_lo[k * plane + cj] = (uint64_t)sx[k];
        acc.sum_hi[k * plane + cj] = (uint64_t)(sx[k] >> 64);
        // M2 = (cnt * sum x^2 - (sum x)^2) / cnt, numerator exact in 256 bits
        double m2 = 0.0;
        if (cnt > 0) {
            const U256 num = u256_sub(u256_mul64(sq[k], cnt), u128_sq(sx[k]));
            m2 = u256_to_f64(num) / (double)cnt;
        }
        acc.m2[k * plane + cj] = m2;
    }
}

// a + (w << (32 k)) for a cell word w < 2^64
__device__ __forceinline__ void u256_add_limb(U256 &a, uint64_t w, int k) {
    U256 t = {{0, 0, 0, 0}};
    const int q = k >> 1;
    if (k & 1) {
        t.w[q] = w << 32;
        if (q + 1 < 4) t.w[q + 1] = w >> 32;
    } else {
        t.w[q] = w;
    }
    u256_add(a, t);
}
__device__ __forceinline__ U256 cell_sum(const uint64_t *w, int limbs) {
    U256 r = {{0, 0, 0, 0}};
    for (int k = 0; k < limbs; ++k) u256_add_limb(r, w[k], k);
    return r;
}

// thread = cell (class c, checkpoint j): the fused limb sums -> exact sums
// of x and M2 = (cnt * sum x^2 - (sum x)^2) / cnt from the exact 256-bit
// numerator, as mix_reduce_kernel computes them from the records.
__global__ void mix_finalize_kernel(MixDev m, const uint32_t *counts, const uint64_t *cells, MixAccum acc,
                                    uint32_t n_classes) {
    const size_t plane = (size_t)n_classes * (uint32_t)m.F;
    const size_t cj = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (cj >= plane) return;
    const uint32_t c = (uint32_t)(cj / (uint32_t)m.F), j = (uint32_t)(cj % (uint32_t)m.F);
    const uint32_t cnt = counts[c];
    uint32_t kind, L, N, M;
    class_graph(m, c, kind, L, N, M);
    (void)kind; (void)L; (void)M;
    const uint64_t *w = cells + cj * kMixCellWords;
    const u128 sx_max = cell_sum(w + kSxMax, 1).w[0];
    const U256 sq_max = cell_sum(w + kSqMax, 2);
    // m1 = N - max: sum (N - x) = cnt N - sum x; sum (N - x)^2 = cnt N^2 - 2 N sum x + sum x^2 (< 2^67)
    const u128 sq_max128 = ((u128)sq_max.w[1] << 64) | sq_max.w[0];
    const u128 sx_m1 = (u128)cnt * N - sx_max;
    const u128 sq_m1 = (u128)cnt * N * N + sq_max128 - (u128)(2ull * N) * sx_max;
    U256 sx[6], sq[6];
    sx[0] = cell_sum(w + kSxMax, 1);  sq[0] = sq_max;
    sx[1] = cell_sum(w + kSxM0, 1);   sq[1] = cell_sum(w + kSqM0, 2);
    sx[2] = u256_from_u128(sx_m1);    sq[2] = u256_from_u128(sq_m1);
    sx[3] = cell_sum(w + kSxM2, 2);   sq[3] = cell_sum(w + kSqM2, 3);
    sx[4] = cell_sum(w + kSxM3, 2);   sq[4] = cell_sum(w + kSqM3, 4);
    sx[5] = cell_sum(w + kSxM4, 3);   sq[5] = cell_sum(w + kSqM4, 6);
    if (j == 0) acc.count[c] = cnt;
    acc.span[cj] = (uint32_t)w[kCellSpan];
    for (int k = 0; k < 6; ++k) {
        const u128 sum = ((u128)sx[k].w[1] << 64) | sx[k].w[0];  // < 2^108
        acc.sum_lo[k * plane + cj] = (uint64_t)sum;
        acc.sum_hi[k * plane + cj] = (uint64_t)(sum >> 64);
        double m2 = 0.0;
        if (cnt > 0) {
            const U256 num = u256_sub(u256_mul64(sq[k], cnt), u128_sq(sum));
            m2 = u256_to_f64(num) / (double)cnt;
        }
        acc.m2[k * plane + cj] = m2;
    }
}

// ---------------------------------------------------------------- launchers

// Segment `segment` with W warps per run; `words`: the most node words one of
// its runs needs; per_sm: blocks that fit on an SM.
template <int W, bool SHARED, bool FUSED>
static int launch_segment(const MixLaunch &p, int segment, uint32_t words, int per_sm, cudaStream_t s) {
    const uint32_t nodes = SHARED ? group::val_bytes(words) + group::flag_bytes(words) : 0u;
    const uint32_t claims = group::claim_words<W, SHARED>(words, nodes, (uint32_t)per_sm);
    const size_t smem = (size_t)claims * 4u + nodes;
    int blocks = 152 * per_sm;
    if (blocks > p.m.n_runs) blocks = p.m.n_runs;
    if (!SHARED) blocks = (int)std::min<uint64_t>(blocks, p.node_words / p.home_words);  // one node array each
    return launch_kernel(mix_group_kernel<W, SHARED, FUSED>, dim3(blocks), 32 * W, smem, group::most_shared<W, SHARED>(), s, p,
                         segment, claims, p.home_words) == cudaSuccess
               ? NZ_OK
               : NZ_ERR_CUDA;
}

constexpr uint64_t kMostThreads = 152ull * 6 * kMixThreads;  // 6 blocks to an SM
constexpr uint64_t kMostHomes = 152ull * 2;                   // blocks of the largest lattices
constexpr int32_t kFewestThreads = 20000;                     // runs for which there are no threads below

// A place for each resident run beyond shared memory, or a slot for each thread of
// the fused reduction (a size for both reductions); the segments run one after
// another.
uint64_t mix_node_words(uint64_t home_words, int32_t n_runs, int32_t T) {
    const uint64_t runs = (uint64_t)n_runs;
    const uint64_t homes = home_words > segment_words(0) ? std::min(kMostHomes, runs) * home_words : 0;
    const uint64_t threads =
        n_runs >= kFewestThreads ? std::min(kMostThreads, runs) * std::min<uint64_t>(segment_words(2), home_words) : 0;
    return std::min((uint64_t)T * home_words, std::max(homes, threads));
}

// Node words that the slots of segment k's threads have, and their number, as far as
// the slots reach.
static uint32_t thread_words(const MixLaunch &p, int k) {
    return (uint32_t)std::min<uint64_t>(segment_words(k - 1), p.home_words);
}
static uint32_t thread_count(const MixLaunch &p, int k) {
    return (uint32_t)std::min<uint64_t>({kMostThreads, p.node_words / thread_words(p, k), (uint64_t)p.m.n_runs});
}

// Runs that segment k can expect, its lengths being log-uniform.
static double expected_runs(const MixLaunch &p, int k) {
    auto part = [](uint32_t lo, uint32_t hi, uint32_t a, uint32_t b) {  // lengths a .. b - 1 of lo .. hi
        if (a >= b) return 0.0;
        if (lo == hi) return 1.0;
        return std::min(1.0, (log(b - 0.5) - log(a - 0.5)) / log((double)hi / lo));
    };
    uint32_t a = p.m.grid_min, b = p.m.grid_max + 1u;
    while (a < b && grid_slots(a) <= segment_words(k)) ++a;
    while (a < b && grid_slots(b - 1u) > segment_words(k - 1)) --b;
    const double grids = part(p.m.grid_min, p.m.grid_max, a, b);
    const double chains = part(p.m.chain_min, p.m.chain_max, std::max(p.m.chain_min, segment_words(k) + 1u),
                               std::min(p.m.chain_max, segment_words(k - 1)) + 1u);
    const double share = p.m.chain_share / 4294967296.0;
    return p.m.n_runs * ((1.0 - share) * grids + share * chains);
}

// Is a thread per run the better one for the fused reduction of segment k (3 or 4)?
// A thread's steps take some 2.9 us each, so the largest lattice's are the least time;
// a block of a run adds all its checkpoints' limbs itself.  ms by blocks and by threads,
// 256 checkpoints: 10^6 runs of grids 2-16 and chains 2-64 67 and 8.5, 10^5 7.5 and 3.4,
// 10^4 1.6 and 3; of grids 8-31 and chains 64-1000 55 and 26, 5.5 and 6.9; 3 10^5 of grids
// 33-64 and chains 2000-4096 171 and 83, 10^5 57 and 37, 3 10^4 17.6 and 27.
static bool mix_threads(const MixLaunch &p, int k) {
    const double runs = expected_runs(p, k);
    return thread_count(p, k) >= std::min(runs, 65536.0) && runs >= (k == 4 ? kFewestThreads + 100.0 * thread_words(p, k) : 50000.0);
}

static int launch_threads(const MixLaunch &p, int k, cudaStream_t s) {
    const uint32_t threads = thread_count(p, k);
    return launch_kernel(mix_thread_kernel, dim3((threads + kMixThreads - 1) / kMixThreads), kMixThreads, 0, 0, s, p, k, threads,
                         thread_words(p, k)) == cudaSuccess
               ? NZ_OK
               : NZ_ERR_CUDA;
}

template <bool FUSED>
static int launch_segments(const MixLaunch &p, cudaStream_t s) {
    const uint64_t most = std::max<uint64_t>(grid_slots(p.m.grid_max), p.m.chain_max);
    const uint64_t least = std::min<uint64_t>(grid_slots(p.m.grid_min), p.m.chain_min);
    int st = NZ_OK;
    // a segment that no lattice of the ranges can fall into is not launched
    auto used = [&](int k) {
        return (k == 0 || least <= segment_words(k - 1)) && most > segment_words(k);
    };
    if (used(0)) st = launch_segment<12, false, FUSED>(p, 0, (uint32_t)most, 2, s);
    if (st == NZ_OK && used(1)) st = launch_segment<24, true, FUSED>(p, 1, segment_words(0), 1, s);
    if (st == NZ_OK && used(2)) st = launch_segment<8, true, FUSED>(p, 2, segment_words(1), 3, s);
    if constexpr (FUSED) {
        if (st == NZ_OK && used(3)) st = mix_threads(p, 3) ? launch_threads(p, 3, s) : launch_segment<2, true, true>(p, 3, segment_words(2), 11, s);
        if (st == NZ_OK && used(4)) st = mix_threads(p, 4) ? launch_threads(p, 4, s) : launch_segment<1, true, true>(p, 4, segment_words(3), 24, s);
        return st;
    }
    if (st == NZ_OK && used(3)) st = launch_segment<2, true, FUSED>(p, 3, segment_words(2), 11, s);
    if (st == NZ_OK && used(4)) st = launch_segment<1, true, FUSED>(p, 4, segment_words(3), 24, s);
    return st;
}

int launch_mix(const MixLaunch &p, cudaStream_t s) {
    const uint32_t n_classes = p.m.n_grid + p.m.n_chain;
    if (cudaMemsetAsync(p.counts, 0, sizeof(uint32_t) * n_classes, s) != cudaSuccess) return NZ_ERR_CUDA;
    if (cudaMemsetAsync(p.acc.errors, 0, sizeof(uint32_t), s) != cudaSuccess) return NZ_ERR_CUDA;
    int blocks = (p.m.n_runs + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    mix_class_kernel<<<blocks, 256, 0, s>>>(p.m, p.cls, p.counts);
    mix_order_kernel<<<(n_classes + 255) / 256, 256, 0, s>>>(p.m, p.order);
    mix_offsets_kernel<<<1, 1024, 0, s>>>(p.counts, p.order, n_classes, p.offsets, p.cursor);
    mix_scatter_kernel<<<blocks, 256, 0, s>>>(p.m.n_runs, p.cls, p.cursor, p.queue);
    mix_segments_kernel<<<(n_classes + 256) / 256, 256, 0, s>>>(p.m, p.order, p.offsets, p.begin, p.head);
    if (p.fused) {
        const size_t cells = (size_t)n_classes * (uint32_t)p.m.F;
        if (cudaMemsetAsync(p.cells, 0, cells * kMixCellWords * sizeof(uint64_t), s) != cudaSuccess)
            return NZ_ERR_CUDA;
        const int st = launch_segments<true>(p, s);
        if (st != NZ_OK) return st;
        mix_finalize_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(p.m, p.counts, p.cells, p.acc,
                                                                            n_classes);
    } else {
        const int st = launch_segments<false>(p, s);
        if (st != NZ_OK) return st;
        dim3 rg(n_classes, (p.m.F + 31) / 32);
        mix_reduce_kernel<<<rg, 32, 0, s>>>(p.m, p.counts, p.offsets, p.rec, p.acc, n_classes);
    }
    return cudaGetLastError() == cudaSuccess ? NZ_OK : NZ_ERR_CUDA;
}

}  // namespace nz
