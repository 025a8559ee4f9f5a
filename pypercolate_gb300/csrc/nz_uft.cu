// nz_uft.cu -- Newman-Ziff percolation, one run per thread.
//
// The same records as those of nz_group.cuh, for launches of very many runs: a
// thread adds its run's bonds (percolate/hpc.py:249-307) or sites one at a time.
// One instruction of a warp serves 32 runs that way, and there are no rounds and no
// prefix sums; but a run's steps are a chain of dependent accesses, some 1 us a step
// in shared memory and 2 to 3.5 in global memory, which only very many threads hide.
// So it is the better one (run_per_thread below has the sizes)
//   * for small lattices in an ensemble, on which a group is mostly set-up, with
//     the node words of 128 runs in a block's shared memory (tiny_thread_kernel);
//   * for n-major records of many runs, since the threads of a warp write one row
//     of neighbouring runs, and a group each row of its run to another line.
//
// Torus (Newman & Ziff, Phys. Rev. E 64, 016706 (2001), Sec. III.B): a node has
// its displacement (dx, dy) from its parent beside its word; a step from u to v =
// u + delta inside one cluster closes a loop, which winds around the torus where
// pos(u) + delta != pos(v).
//
// Sites: the joins with the four neighbours are a loop with one copy of the union.
// (With four inlined copies the kernel of the torus lost joins where a warp's lanes
// took different ways; the sources' plain reading, and the same code on the host,
// do not.  Its shared words are volatile for the same reason.)
#include <cstdint>

#include "nz_common.cuh"
#include "nz_internal.cuh"
#include "nz_records.cuh"
#include "nz_thread.cuh"

namespace nz {
namespace {

using namespace thread;

constexpr int kThreads = 128;
constexpr uint32_t kTinyNodes = 256, kTinyTorus = 121;  // largest N in shared memory

// Where a run's rows go (n-major), in increasing order.
struct Rows {
    const NzRecords &rec;
    size_t off;

    __device__ __forceinline__ Rows(const NzRecords &records, int32_t r) : rec(records), off((size_t)r) {}
    // the powers of the largest size are formed per row (a few multiplies)
    // rather than kept: registers are worth more
    __device__ __forceinline__ void put(const RunState &st, bool flag, uint32_t step) {
        const uint64_t mx = st.max, mx2 = mx * mx, mx3 = mx2 * mx, mx4_lo = mx3 * mx;
        if (rec.max_span) rec.max_span[off] = st.max | (flag ? kSpanBit : 0u);
        put_m0_m2(rec, off, st.t0 - (st.t0 ? 1u : 0u), st.t2 - mx2);
        if (rec.m3) rec.m3[off] = st.t3 - mx3;
        if (rec.m4_lo) rec.m4_lo[off] = st.t4_lo - mx4_lo;
        if (rec.m4_hi) rec.m4_hi[off] = (uint32_t)(st.t4_hi - __umul64hi(mx3, mx) - (st.t4_lo < mx4_lo ? 1ull : 0ull));
        if (rec.edge) rec.edge[off] = step;
        off += (size_t)rec.run_stride;
    }
};

// A run before its first step: N clusters of one node (bonds) or none (sites).
__device__ __forceinline__ RunState first_state(const UfParams &p) {
    RunState s;
    s.t2 = s.t3 = s.t4_lo = p.g.site ? 0u : p.g.N;
    s.t4_hi = 0;
    s.t0 = p.g.site ? 0u : p.g.N;
    s.max = p.g.site ? 0u : 1u;
    s.flags = p.init_flag ? *p.init_flag : 0u;
    s.pad = 0;
    return s;
}

// The order of a run's steps.
template <bool GIVEN>
struct Order {
    FeistelPerm fp;
    const uint32_t *perm;
    __device__ __forceinline__ Order(const UfParams &p, int32_t r) {
        if (GIVEN) perm = p.perms + (size_t)r * p.g.M;
        else fp.init(p.key, p.run0 + (uint64_t)r, p.g.M);
    }
    __device__ __forceinline__ uint32_t at(uint32_t idx) const { return GIVEN ? __ldg(perm + idx) : fp.at(idx); }
};

// ------------------------------------------------------ grid, chain, edges
// 9 CTAs of 128 threads per SM (56 registers): the more threads, the more
// accesses are in flight (1,491 ms per 100,000 runs of 256 x 256 beside their
// consumers, 1,636 at 70 registers).  The next step's index is computed while
// this one's first loads are in flight.
template <int KIND, bool GIVEN>
__global__ void __launch_bounds__(kThreads, 9) bond_thread_kernel(UfParams p, bool span) {
    const int32_t r = blockIdx.x * kThreads + threadIdx.x;
    if (r >= p.n_runs) return;
    const GraphDev &g = p.g;
    uint32_t *node = p.nodes + (size_t)r * g.slots;
    Tally t{first_state(p)};
    const Order<GIVEN> order(p, r);
    Rows rows(p.rec, r);
    uint32_t next = g.M > 0 ? order.at(0) : 0u;
    for (uint32_t n = 0; n <= g.M; ++n) {
        uint32_t e = 0;
        if (n > 0) {
            e = next;
            uint32_t u, v;
            if (GIVEN && e >= g.M) {
                u = v = 0;  // caller-supplied index out of range: no bond added
            } else {
                decode_edge_slots<KIND>(g, e, u, v);
                if (KIND == NZ_GRAPH_EDGES && (u >= g.N || v >= g.N)) u = v = 0;  // invalid edge list
            }
            const uint32_t wu = node[u], wv = node[v];
            if (n < g.M) next = order.at(n);
            link(node, u, v, wu, wv, span, t);
        }
        rows.put(t.st, span && (t.st.flags & kFlagSpan), e);
    }
}

// Sites of the grid and the chain.
template <int KIND, bool GIVEN>
__global__ void __launch_bounds__(kThreads, 9) site_thread_kernel(UfParams p, bool span) {
    const int32_t r = blockIdx.x * kThreads + threadIdx.x;
    if (r >= p.n_runs) return;
    const GraphDev &g = p.g;
    uint32_t *node = p.nodes + (size_t)r * g.slots;
    Tally t{first_state(p)};
    const Order<GIVEN> order(p, r);
    Rows rows(p.rec, r);
    const uint32_t width = KIND == NZ_GRAPH_GRID2D ? g.L : g.N, height = KIND == NZ_GRAPH_GRID2D ? g.L : 1u;
    auto slot = [&](uint32_t row, uint32_t col) {
        if (KIND == NZ_GRAPH_GRID2D && kGridTiled) return grid_slot(g.tile_cols, row, col);
        return row * width + col;
    };
    uint32_t next = g.M > 0 ? order.at(0) : 0u;
    for (uint32_t n = 0; n <= g.M; ++n) {
        uint32_t i = 0;
        if (n > 0) {
            i = next;
            // a caller-supplied index out of range or repeated occupies nothing
            const bool in = !GIVEN || i < g.N;
            const uint32_t row = in && height > 1u ? i / width : 0u, col = in ? i - row * width : 0u;
            const uint32_t x = slot(row, col), wx = node[x];
            if (n < g.M) next = order.at(n);
            if (in && wx == kEmpty) {
                const uint32_t sides = node_sides<KIND>(g, i);
                node[x] = make_root(1u, sides);
                t.add_single();
                if (span && sides == 3u) t.st.flags |= kFlagSpan;
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {  // left, right, above, below
                    const bool along = c < 2, forth = (c & 1) != 0;
                    const uint32_t here = along ? col : row, size = along ? width : height;
                    if (forth ? here + 1u == size : here == 0) continue;
                    const uint32_t there = forth ? here + 1u : here - 1u;
                    const uint32_t y = along ? slot(row, there) : slot(there, col), wy = node[y];
                    if (wy != kEmpty) link(node, x, y, node[x], wy, span, t);
                }
            }
        }
        rows.put(t.st, span && (t.st.flags & kFlagSpan), i);
    }
}

// ------------------------------------------------------ torus with wrapping
// cell: x = node word, y = dx, z = dy (two's complement), w unused
__device__ __forceinline__ bool torus_flag(uint32_t flags, uint32_t crit) {
    const bool x = (flags & kFlagWrapX) != 0, y = (flags & kFlagWrapY) != 0;
    return crit == 0 ? (x || y) : crit == 1 ? x : crit == 2 ? y : (x && y);
}

// Joins u and v = u + (ddx, ddy), whose cells are cu and cv.
__device__ __forceinline__ void link_torus(uint4 *cell, uint32_t xu, uint32_t xv, uint4 cu, uint4 cv, int32_t ddx,
                                           int32_t ddy, Tally &t) {
    int32_t pux = 0, puy = 0, pvx = 0, pvy = 0;  // positions relative to the current node
    for (int hops = 0; !(is_root(cu.x) && is_root(cv.x)); ++hops) {
        if (hops >= kMaxHops) { t.st.flags |= kFlagCorrupt; return; }
        if (!is_root(cu.x)) {
            const uint32_t par = cu.x;
            const uint4 cp = cell[par];
            pux += (int32_t)cu.y;
            puy += (int32_t)cu.z;
            if (!is_root(cp.x)) cell[xu] = make_uint4(cp.x, cu.y + cp.y, cu.z + cp.z, 0u);
            xu = par;
            cu = cp;
        }
        if (!is_root(cv.x)) {
            const uint32_t par = cv.x;
            const uint4 cp = cell[par];
            pvx += (int32_t)cv.y;
            pvy += (int32_t)cv.z;
            if (!is_root(cp.x)) cell[xv] = make_uint4(cp.x, cv.y + cp.y, cv.z + cp.z, 0u);
            xv = par;
            cv = cp;
        }
    }
    // position of v's root as seen from u's root, were v at pos(u) + delta
    const int32_t ox = pux + ddx - pvx, oy = puy + ddy - pvy;
    if (xu == xv) {
        if (ox != 0) t.st.flags |= kFlagWrapX;
        if (oy != 0) t.st.flags |= kFlagWrapY;
        return;
    }
    const uint32_t a = root_size(cu.x), b = root_size(cv.x);
    if (a >= b) {
        cell[xv] = make_uint4(xu, (uint32_t)ox, (uint32_t)oy, 0u);
        cell[xu] = make_uint4(make_root(a + b, 0u), 0u, 0u, 0u);
    } else {
        cell[xu] = make_uint4(xv, (uint32_t)(-ox), (uint32_t)(-oy), 0u);
        cell[xv] = make_uint4(make_root(a + b, 0u), 0u, 0u, 0u);
    }
    t.merge(a, b);
}

template <bool SITE, bool GIVEN>
__global__ void __launch_bounds__(kThreads) torus_thread_kernel(UfParams p, bool span) {
    const int32_t r = blockIdx.x * kThreads + threadIdx.x;
    if (r >= p.n_runs) return;
    const GraphDev &g = p.g;
    uint4 *cell = reinterpret_cast<uint4 *>(p.nodes + (size_t)r * g.slots);
    Tally t{first_state(p)};
    const Order<GIVEN> order(p, r);
    Rows rows(p.rec, r);
    const uint32_t L = g.L;
    // bonds: the next index while this step's loads are in flight (7.3e9 against
    // 7.0e9 additions/s at L = 256); sites are 2 % slower that way
    uint32_t next = !SITE && g.M > 0 ? order.at(0) : 0u;
    for (uint32_t n = 0; n <= g.M; ++n) {
        uint32_t e = 0;
        if (n > 0) {
            e = SITE ? order.at(n - 1u) : next;
            const uint32_t u = SITE || e < g.N ? e : e - g.N, row = u / L, col = u - row * L;
            const uint32_t right = row * L + (col + 1u == L ? 0u : col + 1u);
            const uint32_t down = (row + 1u == L ? 0u : row + 1u) * L + col;
            if (SITE) {
                if ((!GIVEN || e < g.N) && cell[e].x == kEmpty) {
                    cell[e] = make_uint4(make_root(1u, 0u), 0u, 0u, 0u);
                    t.add_single();
                    // this site's cell is read again for every link: an earlier
                    // link may have hung it below another root
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {  // right, left, below, above
                        const uint32_t y = c == 0   ? right
                                           : c == 1 ? row * L + (col == 0u ? L - 1u : col - 1u)
                                           : c == 2 ? down
                                                    : (row == 0u ? L - 1u : row - 1u) * L + col;
                        const uint4 cy = cell[y];
                        const int32_t one = (c & 1) ? -1 : 1;
                        if (cy.x != kEmpty) link_torus(cell, e, y, cell[e], cy, c < 2 ? one : 0, c < 2 ? 0 : one, t);
                    }
                }
            } else {
                const bool in = !GIVEN || e < g.M, vertical = e >= g.N;
                const uint32_t a = in ? u : 0u, b = in ? (vertical ? down : right) : 0u;
                const uint4 ca = cell[a], cb = cell[b];
                if (n < g.M) next = order.at(n);
                if (in) link_torus(cell, a, b, ca, cb, vertical ? 0 : 1, vertical ? 1 : 0, t);
            }
        }
        rows.put(t.st, span && torus_flag(t.st.flags, g.wrap), e);
    }
}

// ------------------------------------------------- small lattices, in tiles
// A thread's node words lie in shared memory, 16 bits each (root: bit 15, sides
// 13..14, size; else the parent; word x of thread t at x * kThreads + t), on the
// torus with the displacement from the parent as one integer dx 2^16 + dy.
// Totals are kept modulo 2^32, which all moments are below (sum' s^4 <= max s^3 (N -
// s) < N^4 / 9).  Four rows of a run are written at a time, in the tiles' 16-byte
// pieces.  10^6 runs of 8 x 8: 2.3 ms;
// with node words in global memory 6.0, and 14.3 with rows written value by value,
// a warp's 32 lanes in 32 lines.
constexpr uint32_t kTinyRoot = 0x8000u;
static_assert((uint64_t)kTinyNodes * kTinyNodes * kTinyNodes * kTinyNodes / 9 < 1ull << 32, "moments in 32 bits");

struct TinyRows {
    uint32_t ms[4][kThreads], m2[4][kThreads], m3[4][kThreads], m4[4][kThreads];
    uint16_t m0[4][kThreads];
};

template <bool TORUS>
constexpr uint32_t tiny_bytes(uint32_t N) { return N * kThreads * (TORUS ? 6u : 2u); }

template <int KIND, bool SITE>
__global__ void __launch_bounds__(kThreads) tiny_thread_kernel(UfParams p, bool span) {
    constexpr bool kTorus = KIND == NZ_GRAPH_TORUS2D;
    extern __shared__ __align__(16) uint8_t tiny_smem[];
    __shared__ TinyRows four;
    const uint32_t t = threadIdx.x;
    const int32_t r = blockIdx.x * kThreads + t;
    if (r >= p.n_runs) return;
    const GraphDev &g = p.g;
    volatile int32_t *disp = reinterpret_cast<int32_t *>(tiny_smem) + t;
    volatile uint16_t *word = reinterpret_cast<uint16_t *>(tiny_smem + (kTorus ? g.N * kThreads * 4u : 0u)) + t;
    uint32_t *home = p.nodes + (size_t)r * g.slots;

    uint32_t t0, t2, t3, t4, mx, flags;
    if (p.n_begin == 0) {
        t0 = t2 = t3 = t4 = SITE ? 0u : g.N;
        mx = SITE ? 0u : 1u;
        flags = 0;
        for (uint32_t x = 0; x < g.N; ++x)
            word[x * kThreads] = (uint16_t)(SITE ? kTinyRoot : kTinyRoot | (kTorus ? 0u : node_sides<kTorus ? NZ_GRAPH_GRID2D : KIND>(g, x)) << 13 | 1u);
    } else {
        const RunState st = p.state[r];
        t0 = st.t0; t2 = (uint32_t)st.t2; t3 = (uint32_t)st.t3; t4 = (uint32_t)st.t4_lo;
        mx = st.max;
        flags = st.flags;
        for (uint32_t x = 0; x < g.N; ++x) {
            word[x * kThreads] = (uint16_t)home[x];
            if (kTorus) disp[x * kThreads] = (int32_t)home[g.N + x];
        }
    }
    // joins the clusters of u and v, v at u's position + d (union by size, and no
    // path is ever longer than log2(N))
    auto link = [&](uint32_t xu, uint32_t xv, int32_t d) {
        uint32_t wu = word[xu * kThreads], wv = word[xv * kThreads];
        for (int hops = 0; !(wu & wv & kTinyRoot); ++hops) {
            if (hops >= kMaxHops) { flags |= kFlagCorrupt; return; }
            if (!(wu & kTinyRoot)) {
                if (kTorus) d += disp[xu * kThreads];
                xu = wu;
                wu = word[xu * kThreads];
            }
            if (!(wv & kTinyRoot)) {
                if (kTorus) d -= disp[xv * kThreads];
                xv = wv;
                wv = word[xv * kThreads];
            }
        }
        if (xu == xv) {
            if (kTorus && d != 0) {
                const int32_t dy = (int16_t)(d & 0xffff);
                flags |= (d != dy ? kFlagWrapX : 0u) | (dy != 0 ? kFlagWrapY : 0u);
            }
            return;
        }
        const uint32_t a = wu & 0x1fffu, b = wv & 0x1fffu, s = a + b, ab = a * b, sides = (wu | wv) & 0x6000u;
        const uint32_t big = a < b ? xv : xu, small = a < b ? xu : xv;
        word[small * kThreads] = (uint16_t)big;
        if (kTorus) disp[small * kThreads] = a < b ? -d : d;
        word[big * kThreads] = (uint16_t)(kTinyRoot | sides | s);
        t0 -= 1u;
        t2 += 2u * ab;
        t3 += 3u * ab * s;
        t4 += ab * (4u * s * s - 2u * ab);
        mx = max(mx, s);
        if (!kTorus && sides == 0x6000u) flags |= kFlagSpan;
    };

    FeistelPerm fp;
    fp.init(p.key, p.run0 + (uint64_t)r, g.M);
    const uint32_t rows = p.n_end - p.n_begin;
    const uint32_t turn = (uint32_t)r & 7u, turn2 = (uint32_t)(r >> 1) & 3u;
    size_t line = (size_t)r * 32;  // of 32 rows of the run
    for (uint32_t i = 0; i < rows; ++i) {
        const uint32_t n = p.n_begin + i;
        if (n > 0) {
            const uint32_t e = fp.at(n - 1u);
            if (!SITE) {
                uint32_t u, v;
                int32_t d = 0;
                if (kTorus) {
                    const bool down = e >= g.N;
                    u = down ? e - g.N : e;
                    const uint32_t row = u / g.L, col = u - row * g.L;
                    v = down ? (row + 1u == g.L ? 0u : row + 1u) * g.L + col : row * g.L + (col + 1u == g.L ? 0u : col + 1u);
                    d = down ? 1 : 1 << 16;
                } else {
                    decode_edge<kTorus ? NZ_GRAPH_GRID2D : KIND>(g, e, u, v);
                }
                link(u, v, d);
            } else {
                const uint32_t width = KIND == NZ_GRAPH_CHAIN1D ? g.N : g.L, height = KIND == NZ_GRAPH_CHAIN1D ? 1u : g.L;
                const uint32_t row = KIND == NZ_GRAPH_CHAIN1D ? 0u : e / width, col = e - row * width;
                const uint32_t sides = kTorus ? 0u : node_sides<kTorus ? NZ_GRAPH_GRID2D : KIND>(g, e);
                word[e * kThreads] = (uint16_t)(kTinyRoot | sides << 13 | 1u);
                t0 += 1u; t2 += 1u; t3 += 1u; t4 += 1u;
                mx = max(mx, 1u);
                if (sides == 3u) flags |= kFlagSpan;
                const uint32_t at = row * width;
#pragma unroll 1
                for (int c = 0; c < 4; ++c) {  // right, left, below, above
                    const bool along = c < 2, forth = (c & 1) == 0;
                    const uint32_t here = along ? col : row, size = along ? width : height;
                    if (!kTorus && (forth ? here + 1u == size : here == 0)) continue;
                    const uint32_t there = forth ? (here + 1u == size ? 0u : here + 1u) : (here == 0 ? size - 1u : here - 1u);
                    const uint32_t y = along ? at + there : there * width + col;
                    if (word[y * kThreads] != kTinyRoot) link(e, y, (forth ? 1 : -1) * (along ? 1 << 16 : 1));
                }
            }
        }
        const uint32_t mx2 = mx * mx, mx3 = mx2 * mx, k = i & 3u;
        const bool flag = span && (kTorus ? torus_flag(flags, g.wrap) : (flags & kFlagSpan) != 0);
        four.ms[k][t] = mx | (flag ? kSpanBit : 0u);
        four.m0[k][t] = (uint16_t)(t0 - (t0 ? 1u : 0u));
        four.m2[k][t] = t2 - mx2;
        four.m3[k][t] = t3 - mx3;
        four.m4[k][t] = t4 - mx3 * mx;
        if (k == 3u || i + 1u == rows) {
            // as tile_off; rows past the window's end get what was there before
            const uint32_t q = i & 28u;
            const size_t o4 = line + (((q >> 2) ^ turn) << 2), o2 = line + ((((q >> 3) ^ turn2) << 3) | (q & 4u));
            const size_t o8 = line + (((q >> 1) ^ turn) << 1), o8b = line + ((((q >> 1) + 1u) ^ turn) << 1);
            auto put4 = [&](uint32_t *plane, const uint32_t (&v)[4][kThreads]) {
                *reinterpret_cast<uint4 *>(plane + o4) = make_uint4(v[0][t], v[1][t], v[2][t], v[3][t]);
            };
            auto put8 = [&](uint64_t *plane, const uint32_t (&v)[4][kThreads]) {
                *reinterpret_cast<uint4 *>(plane + o8) = make_uint4(v[0][t], 0u, v[1][t], 0u);
                *reinterpret_cast<uint4 *>(plane + o8b) = make_uint4(v[2][t], 0u, v[3][t], 0u);
            };
            put4(p.rec.max_span, four.ms);
            *reinterpret_cast<uint2 *>(reinterpret_cast<uint16_t *>(p.rec.m0) + o2) =
                make_uint2(four.m0[0][t] | (uint32_t)four.m0[1][t] << 16, four.m0[2][t] | (uint32_t)four.m0[3][t] << 16);
            put4(reinterpret_cast<uint32_t *>(p.rec.m2), four.m2);
            put8(p.rec.m3, four.m3);
            put8(p.rec.m4_lo, four.m4);
            if (q == 28u) line += (size_t)p.rec.run_stride * 32;
        }
    }
    if (p.n_end == g.M + 1u) {
        if (p.errors && (flags & kFlagCorrupt)) atomicAdd(p.errors, 1u);
        return;
    }
    RunState st;
    st.t0 = t0; st.t2 = t2; st.t3 = t3; st.t4_lo = t4; st.t4_hi = 0;
    st.max = mx;
    st.flags = flags;
    st.pad = 0;
    p.state[r] = st;
    for (uint32_t x = 0; x < g.N; ++x) {
        home[x] = word[x * kThreads];
        if (kTorus) home[g.N + x] = (uint32_t)disp[x * kThreads];
    }
}

template <int KIND, bool SITE>
cudaError_t launch_tiny(const UfParams &p, bool span, cudaStream_t s) {
    constexpr bool kTorus = KIND == NZ_GRAPH_TORUS2D;
    return launch_kernel(tiny_thread_kernel<KIND, SITE>, dim3((p.n_runs + kThreads - 1) / kThreads), kThreads,
                         tiny_bytes<kTorus>(p.g.N), tiny_bytes<kTorus>(kTorus ? kTinyTorus : kTinyNodes), s, p, span);
}

// ------------------------------------------------------------ set-up, launch
// Block b: chunk b % chunks (kInitChunk slots) of run b / chunks.  Slots are
// written in order; padding slots of the grid's layout (never read) get 0.
constexpr uint32_t kInitChunk = 4096;
template <int KIND>
__global__ void thread_nodes_kernel(GraphDev g, uint64_t blocks, uint32_t chunks, uint32_t *nodes) {
    for (uint64_t b = blockIdx.x; b < blocks; b += gridDim.x) {
        const uint64_t r = b / chunks;
        const uint32_t ch = (uint32_t)(b - r * chunks);
        uint32_t *row = nodes + r * g.slots;
        const uint32_t count = KIND == NZ_GRAPH_TORUS2D ? g.N : g.slots;
        const uint32_t j1 = min(count, (ch + 1u) * kInitChunk);
        for (uint32_t j = ch * kInitChunk + threadIdx.x; j < j1; j += blockDim.x) {
            if (KIND == NZ_GRAPH_TORUS2D) {
                reinterpret_cast<uint4 *>(row)[j] = make_uint4(g.site ? kEmpty : make_root(1u, 0u), 0u, 0u, 0u);
                continue;
            }
            uint32_t i = j;
            bool pad = j >= g.N;
            if (KIND == NZ_GRAPH_GRID2D && kGridTiled) {
                const uint32_t tile = j >> 3, w = j & 7u;
                const uint32_t tr = tile / g.tile_cols, tc = tile - tr * g.tile_cols;
                const uint32_t rr = 2u * tr + (w >> 2), c = 4u * tc + (w & 3u);
                pad = rr >= g.L || c >= g.L;
                i = rr * g.L + c;
            }
            row[j] = pad ? 0u : g.site ? kEmpty : make_root(1u, node_sides<KIND == NZ_GRAPH_TORUS2D ? NZ_GRAPH_CHAIN1D : KIND>(g, i));
        }
    }
}

template <int KIND>
void init_nodes(const UfParams &p, cudaStream_t s) {
    const uint32_t count = KIND == NZ_GRAPH_TORUS2D ? p.g.N : p.g.slots;
    const uint32_t chunks = (count + kInitChunk - 1) / kInitChunk;
    const uint64_t blocks = (uint64_t)p.n_runs * chunks;
    thread_nodes_kernel<KIND><<<(unsigned)(blocks < 152ull * 256 ? blocks : 152ull * 256), count < 256 ? 64 : 256, 0, s>>>(
        p.g, blocks, chunks, p.nodes);
}

template <int KIND, bool GIVEN>
cudaError_t launch_threads(const UfParams &p, bool span, cudaStream_t s) {
    init_nodes<KIND>(p, s);
    constexpr bool kTorus = KIND == NZ_GRAPH_TORUS2D;
    const dim3 grid((p.n_runs + kThreads - 1) / kThreads);
    if constexpr (kTorus) {
        return launch_kernel(p.g.site ? torus_thread_kernel<true, GIVEN> : torus_thread_kernel<false, GIVEN>, grid, kThreads,
                             0, 0, s, p, span);
    } else if constexpr (KIND == NZ_GRAPH_EDGES) {
        return launch_kernel(bond_thread_kernel<KIND, GIVEN>, grid, kThreads, 0, 0, s, p, span);
    } else {
        return launch_kernel(p.g.site ? site_thread_kernel<KIND, GIVEN> : bond_thread_kernel<KIND, GIVEN>, grid, kThreads, 0,
                             0, s, p, span);
    }
}

template <int KIND>
cudaError_t launch_kind(const UfParams &p, bool given, bool span, cudaStream_t s) {
    if constexpr (KIND != NZ_GRAPH_EDGES) {
        if (p.tiled) return p.g.site ? launch_tiny<KIND, true>(p, span, s) : launch_tiny<KIND, false>(p, span, s);
    }
    return given ? launch_threads<KIND, true>(p, span, s) : launch_threads<KIND, false>(p, span, s);
}

}  // namespace

// Where a thread per run is the better one, each line where both take the same
// time.  Union-find in ms, a group per run and a thread per run:
//   ensembles, 10^6 runs: 8 x 8 7.6 and 2.3, 12 x 12 14.0 and 6.4, chains of 200
//   10.5 and 3.6, sites of 8 x 8 8.2 and 1.3, 5 10^5 of 16 x 16 8.7 and 4.1, sites 9.6 and
//   4.6; 33,000 runs of 8 x 8 0.30 and 0.12, of 16 x 16 0.64 and 0.45; 20,000 of 8 x 8 0.17
//   and 0.11, of chains of 200 0.24 each.  The torus needs three times the memory, so that only
//   one block fits an SM beyond 121 nodes (10^6 / 2 runs of 11 x 11 6.5 and 3.0, 12 x
//   12 8.4 and 10.4).
//   n-major, bonds: 10^5 runs of 16 x 16 3.2 and 2.1, of 64 x 64 79 and 53, 50,000 of
//   128 x 128 226 and 147, 30,000 of 256 x 256 604 and 515, 20,000 chains of 10^5 348
//   and 305; 30,000 of 32 x 32 4.7 and 6.3, 20,000 of 128 x 128 89 and 118, 15,000 of
//   256 x 256 309 and 465.  Torus: 20,000 of 256 x 256 677 and 530, 3 10^5 of 16 x 16
//   14.4 and 12.3, 10^5 of 64 x 64 62 and 65.  Sites: 5 10^5 of 16 x 16 12.1 and 9.5, 10^5
//   of 64 x 64 32 and 46.
bool run_per_thread(const UfParams &p) {
    const uint32_t N = p.g.N;
    const bool torus = p.g.kind == NZ_GRAPH_TORUS2D;
    if (p.tiled) return N <= (torus ? kTinyTorus : kTinyNodes) && p.n_runs >= 32768;
    if (p.g.site) return !torus && N <= 1024 && p.n_runs >= 200000;
    if (torus) return N > 16384 ? p.n_runs >= 16000 : N <= 1024 && p.n_runs >= 200000;
    return p.n_runs >= (N <= 16384 ? 40000 : N <= 65536 ? 24000 : 16000);
}

cudaError_t launch_uf_threads(const UfParams &p, bool given, bool span, cudaStream_t s) {
    if (p.n_runs <= 0) return cudaSuccess;
    switch (p.g.kind) {
        case NZ_GRAPH_GRID2D: return launch_kind<NZ_GRAPH_GRID2D>(p, given, span, s);
        case NZ_GRAPH_CHAIN1D: return launch_kind<NZ_GRAPH_CHAIN1D>(p, given, span, s);
        case NZ_GRAPH_TORUS2D: return launch_kind<NZ_GRAPH_TORUS2D>(p, given, span, s);
        default: return launch_kind<NZ_GRAPH_EDGES>(p, given, span, s);
    }
}

}  // namespace nz
