// nz_group.cuh -- Newman-Ziff percolation, one run per thread block.
//
// Replaces the hot loop of percolate/hpc.py:249-307 (bond_sample_states).
// The bonds of a run are added in batches of B = 64 W (W warps, two
// consecutive bonds per thread) instead of one at a time, with the statistics
// after every single bond unchanged:
//
//   1. every thread finds the roots of its bonds' ends as they stand at the
//      start of the round (read-only, so the order of the threads does not
//      matter) and points the start nodes at their root;
//   2. a bond inside one cluster is done: it stays inside one cluster.  Every
//      other bond claims its two roots for its position in the batch (an
//      atomicMin into a hash table).  A bond that holds both claims shares no
//      root with an earlier unfinished bond, so its two clusters are exactly
//      what they are when its turn comes: it joins them and notes their sizes.
//      The others go into the next round.  The earliest unfinished bond always
//      succeeds, so a batch ends;
//   3. the largest cluster G is not claimed: below it the bonds of a batch
//      would queue up for it.  A bond (G, c) joins c to G and notes |c| alone;
//      G's size at each bond is G's size at the batch start plus a prefix sum.
//   4. the totals after each bond are prefix sums over the batch of what each
//      bond noted.  They run over U_k = sum of s^k over all clusters but G, in
//      which a join with G is a mere -|c|^k; T_k = U_k + |G|^k, and the
//      reference's moments are T_k - (largest)^k.
//
// Integers are exact throughout, so the records equal those of adding one
// bond at a time, whatever the shape of the trees.
//
// Site percolation (SITE) is the same with a site per thread (B = 32 W): the
// batch's sites are marked with their positions in it, so that each thread links
// its site to those neighbours that are occupied before it.  A site claims its
// own node, at which later neighbours of the batch wait, and its neighbours'
// roots; once it holds them all, it and the up to four clusters become one.
// There is no G until a first cluster has formed.  (One thread per run took 6 to
// 170 times as long: 4,000 runs of 256 x 256, 508 ms for the whole ensemble
// against 39; 300 of 400 x 400, 1,186 against 11.)
//
// A run needs few rounds (CPU count of this scheme at L = 256: 1.8 rounds per
// batch of 64, 2.6 per 256, 4.7 per 1024), so one run keeps a whole block
// busy, and a block's node words fit where one thread's 10^5 runs never could:
// up to N = 65,536 nodes in shared memory, as 16 bits (parent, or size - 1 of
// a root) and 8 bits (root, sides) per node; beyond, as the 32-bit words of
// nz_common.cuh in global memory, of which the resident blocks' ones stay
// near L2's size.
//
// What bounds it: dependent integer instructions and barriers (some 750 warp
// instructions per 32 bonds at L = 64, 1,000 at L = 256, a warp's next one 7 and 11
// cycles after the last), so warps per SM are worth more than anything; memory is
// idle.  Very many runs of small lattices, and n-major records of very many runs, are
// nz_uft.cu's.
#pragma once

#include <cstdint>
#include <type_traits>

#include "nz_common.cuh"

namespace nz {
namespace group {

constexpr int kE = 2;                         // bonds per thread and batch
constexpr uint32_t kSharedNodes = 65536;      // largest N whose nodes live in shared memory
constexpr uint32_t kSharedTorus = 16384;      // the same on the torus
constexpr int kMaxHops = 4096;                // guards against corrupted node words only
constexpr uint32_t kTagBits = 11;             // position in the batch (B <= 2048)
constexpr uint32_t kStampTop = (1u << (32 - kTagBits)) - 2u;

// Site percolation: the word of a site that the current batch occupies has this
// bit, and its position in the batch in the low 16 bits.
constexpr uint32_t kNewSite = 1u << 28;
__device__ __forceinline__ bool is_new(uint32_t w) { return (w & (kRoot | kNewSite)) == (kRoot | kNewSite); }
__device__ __forceinline__ uint32_t new_at(uint32_t w) { return w & 0xffffu; }

// Node words of one run.  load() gives the word format of nz_common.cuh
// (root: bit 31, sides 29..30, size; else the parent), sizes less one in
// shared memory.
template <bool SHARED, bool TORUS>
struct Nodes;

template <>
struct Nodes<true, false> {
    // volatile: other threads of the block shorten paths meanwhile (any parent read
    // is an ancestor), so no access may be repeated or kept (1 % of the time)
    volatile uint16_t *val;
    volatile uint8_t *flag;
    __device__ __forceinline__ uint32_t load(uint32_t x) const { return ((uint32_t)flag[x] << 24) | val[x]; }
    __device__ __forceinline__ void shorten(uint32_t x, uint32_t parent) const { val[x] = (uint16_t)parent; }
    __device__ __forceinline__ void link(uint32_t x, uint32_t parent) const {
        val[x] = (uint16_t)parent;
        flag[x] = 0;
    }
    __device__ __forceinline__ void set_root(uint32_t x, uint32_t size, uint32_t sides) const {
        val[x] = (uint16_t)(size - 1u);
        flag[x] = (uint8_t)(0x80u | (sides << 5));
    }
    static __device__ __forceinline__ uint32_t size(uint32_t w) { return (w & kSizeMask) + 1u; }
    // site percolation: an unoccupied site, and one that the batch occupies
    __device__ __forceinline__ void set_empty(uint32_t x) const {
        val[x] = 0;
        flag[x] = 0x88u;
    }
    static __device__ __forceinline__ bool is_empty(uint32_t w) { return (w & 0x08000000u) != 0; }
    __device__ __forceinline__ void set_new(uint32_t x, uint32_t at, uint32_t sides) const {
        val[x] = (uint16_t)at;
        flag[x] = (uint8_t)(0x90u | (sides << 5));
    }
};

template <>
struct Nodes<false, false> {
    uint32_t *w;
    // weak accesses that the compiler neither repeats nor caches: other
    // threads of the block shorten paths meanwhile (any word read is an ancestor)
    __device__ __forceinline__ uint32_t load(uint32_t x) const {
        uint32_t v;
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(w + x));
        return v;
    }
    __device__ __forceinline__ void put(uint32_t x, uint32_t v) const {
        asm volatile("st.global.u32 [%0], %1;" ::"l"(w + x), "r"(v));
    }
    __device__ __forceinline__ void shorten(uint32_t x, uint32_t parent) const { put(x, parent); }
    __device__ __forceinline__ void link(uint32_t x, uint32_t parent) const { put(x, parent); }
    __device__ __forceinline__ void set_root(uint32_t x, uint32_t size, uint32_t sides) const {
        put(x, make_root(size, sides));
    }
    static __device__ __forceinline__ uint32_t size(uint32_t w) { return root_size(w); }
    __device__ __forceinline__ void set_empty(uint32_t x) const { put(x, kRoot); }
    static __device__ __forceinline__ bool is_empty(uint32_t w) { return w == kRoot; }
    __device__ __forceinline__ void set_new(uint32_t x, uint32_t at, uint32_t sides) const {
        put(x, kRoot | (sides << kSideShift) | kNewSite | at);
    }
};

// Sum of a 64-bit value over the warp: its low 64 bits, and what carries over.
__device__ __forceinline__ uint64_t warp_sum(uint64_t v, uint32_t &over) {
    const uint32_t s0 = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0xffffu);
    const uint32_t s1 = __reduce_add_sync(0xffffffffu, (uint32_t)v >> 16);
    const uint32_t s2 = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 32) & 0xffffu);
    const uint32_t s3 = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 48));
    const uint64_t lo = s0 + ((uint64_t)s1 << 16), hi = s2 + ((uint64_t)s3 << 16) + (lo >> 32);
    over = (uint32_t)(hi >> 32);
    return (hi << 32) | (uint32_t)lo;
}

// On the torus every node but a root also has its displacement (dx, dy) from its
// parent, as one integer dx S + dy, which adds and compares like the pair: S =
// 2^16 in 32 bits in shared memory (up to N = 16,384 nodes, where every
// difference that is formed, of at most 2 N - 1 steps, fits 16 bits), S = 2^32
// in 64 bits beyond.  Parent and displacement are two words, so a start node is
// only pointed at its root while no thread climbs.
template <>
struct Nodes<true, true> : Nodes<true, false> {
    typedef int32_t Disp;
    static constexpr int kShift = 16;
    Disp *off;
    __device__ __forceinline__ Disp disp(uint32_t x) const { return off[x]; }
    __device__ __forceinline__ void set_disp(uint32_t x, Disp d) const { off[x] = d; }
    static __device__ __forceinline__ int32_t dy(Disp d) { return (int16_t)(d & 0xffff); }
    static __device__ __forceinline__ int32_t dx(Disp d) { return (d - dy(d)) >> kShift; }
};

template <>
struct Nodes<false, true> {
    typedef int64_t Disp;
    static constexpr int kShift = 32;
    uint4 *cell;  // x: node word; z, w: displacement
    __device__ __forceinline__ uint32_t load(uint32_t x) const {
        uint32_t v;
        asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(&cell[x].x));
        return v;
    }
    __device__ __forceinline__ void put(uint32_t x, uint32_t v) const {
        asm volatile("st.global.u32 [%0], %1;" ::"l"(&cell[x].x), "r"(v));
    }
    __device__ __forceinline__ void shorten(uint32_t x, uint32_t parent) const { put(x, parent); }
    __device__ __forceinline__ void link(uint32_t x, uint32_t parent) const { put(x, parent); }
    __device__ __forceinline__ void set_root(uint32_t x, uint32_t size, uint32_t sides) const {
        put(x, make_root(size, sides));
    }
    static __device__ __forceinline__ uint32_t size(uint32_t w) { return root_size(w); }
    __device__ __forceinline__ void set_empty(uint32_t x) const { put(x, kRoot); }
    static __device__ __forceinline__ bool is_empty(uint32_t w) { return w == kRoot; }
    __device__ __forceinline__ void set_new(uint32_t x, uint32_t at, uint32_t sides) const {
        put(x, kRoot | (sides << kSideShift) | kNewSite | at);
    }
    __device__ __forceinline__ Disp disp(uint32_t x) const {
        Disp v;
        asm volatile("ld.global.s64 %0, [%1];" : "=l"(v) : "l"(&cell[x].z));
        return v;
    }
    __device__ __forceinline__ void set_disp(uint32_t x, Disp d) const {
        asm volatile("st.global.s64 [%0], %1;" ::"l"(&cell[x].z), "l"(d));
    }
    static __device__ __forceinline__ int32_t dy(Disp d) { return (int32_t)(d & 0xffffffffll); }
    static __device__ __forceinline__ int32_t dx(Disp d) { return (int32_t)((d - dy(d)) >> kShift); }
};

// What a stretch of bonds adds to the totals.  Up to N = 65,536, sum s^2 is
// needed modulo 2^32 (sum' s^2 <= N^2 / 4) and sum s^4 modulo 2^64 (sum' s^4
// < 2^64); beyond, modulo 2^64 and 2^96.
template <bool NARROW>
struct Sums;

template <>
struct Sums<true> {
    uint32_t g, u2;  // |G|, sum s^2 without G
    uint64_t u3, u4;
    __device__ __forceinline__ void zero() { g = u2 = 0; u3 = u4 = 0; }
    __device__ __forceinline__ void add(const Sums &o) { g += o.g; u2 += o.u2; u3 += o.u3; u4 += o.u4; }
    __device__ __forceinline__ Sums up(int d) const {
        Sums r;
        r.g = __shfl_up_sync(0xffffffffu, g, d);
        r.u2 = __shfl_up_sync(0xffffffffu, u2, d);
        r.u3 = __shfl_up_sync(0xffffffffu, u3, d);
        r.u4 = __shfl_up_sync(0xffffffffu, u4, d);
        return r;
    }
    __device__ __forceinline__ Sums over_warp() const {
        Sums r;
        uint32_t over;
        r.g = __reduce_add_sync(0xffffffffu, g);
        r.u2 = __reduce_add_sync(0xffffffffu, u2);
        r.u3 = warp_sum(u3, over);
        r.u4 = warp_sum(u4, over);
        return r;
    }
    // clusters a and b, neither of them G, become one
    __device__ __forceinline__ void join(uint32_t a, uint32_t b) {
        const uint32_t s = a + b, ab = a * b;  // a + b <= 2^16: ab < 2^31
        g = 0;
        u2 = 2u * ab;
        u3 = 3ull * ((uint64_t)ab * s);
        u4 = (uint64_t)ab * (4ull * ((uint64_t)s * s) - 2u * ab);
    }
    // cluster b becomes part of G
    __device__ __forceinline__ void absorb(uint32_t b) {
        const uint64_t b2 = (uint64_t)b * b;
        g = b;
        u2 = 0u - (uint32_t)b2;
        u3 = 0ull - b2 * b;
        u4 = 0ull - b2 * b2;
    }
    // += s^k
    __device__ __forceinline__ void plus_powers(uint32_t s) {
        const uint64_t s2 = (uint64_t)s * s;
        u2 += (uint32_t)s2;
        u3 += s2 * s;
        u4 += s2 * s2;
    }
    __device__ __forceinline__ void minus_powers(uint32_t s) {
        const uint64_t s2 = (uint64_t)s * s;
        u2 -= (uint32_t)s2;
        u3 -= s2 * s;
        u4 -= s2 * s2;
    }
    __device__ __forceinline__ void load(const RunState &st) {
        u2 = (uint32_t)st.t2;
        u3 = st.t3;
        u4 = st.t4_lo;
    }
    __device__ __forceinline__ void store(RunState &st) const {
        st.t2 = u2;
        st.t3 = u3;
        st.t4_lo = u4;
        st.t4_hi = 0;
    }
    __device__ __forceinline__ uint64_t m2() const { return u2; }
    __device__ __forceinline__ uint32_t m4_hi() const { return 0u; }
};

template <>
struct Sums<false> {
    uint32_t g, u4x;  // |G|; bits 64..95 of sum s^4
    uint64_t u2, u3, u4;
    __device__ __forceinline__ void zero() { g = u4x = 0; u2 = u3 = u4 = 0; }
    __device__ __forceinline__ void add4(uint64_t lo, uint32_t hi) {
        const uint64_t n = u4 + lo;
        u4x += hi + (n < lo ? 1u : 0u);
        u4 = n;
    }
    __device__ __forceinline__ void sub4(uint64_t lo, uint32_t hi) {
        const uint64_t n = u4 - lo;
        u4x -= hi + (u4 < lo ? 1u : 0u);
        u4 = n;
    }
    __device__ __forceinline__ void add(const Sums &o) {
        g += o.g;
        u2 += o.u2;
        u3 += o.u3;
        add4(o.u4, o.u4x);
    }
    __device__ __forceinline__ Sums up(int d) const {
        Sums r;
        r.g = __shfl_up_sync(0xffffffffu, g, d);
        r.u4x = __shfl_up_sync(0xffffffffu, u4x, d);
        r.u2 = __shfl_up_sync(0xffffffffu, u2, d);
        r.u3 = __shfl_up_sync(0xffffffffu, u3, d);
        r.u4 = __shfl_up_sync(0xffffffffu, u4, d);
        return r;
    }
    __device__ __forceinline__ Sums over_warp() const {
        Sums r;
        uint32_t over;
        r.g = __reduce_add_sync(0xffffffffu, g);
        r.u2 = warp_sum(u2, over);
        r.u3 = warp_sum(u3, over);
        r.u4 = warp_sum(u4, over);
        r.u4x = __reduce_add_sync(0xffffffffu, u4x) + over;
        return r;
    }
    __device__ __forceinline__ void join(uint32_t a, uint32_t b) {
        const uint64_t s = (uint64_t)a + b, ab = (uint64_t)a * b, q = 4ull * s * s - 2ull * ab;
        g = 0;
        u2 = 2ull * ab;
        u3 = 3ull * ab * s;
        u4 = ab * q;
        u4x = (uint32_t)__umul64hi(ab, q);
    }
    __device__ __forceinline__ void absorb(uint32_t b) {
        zero();
        g = b;
        minus_powers(b);
    }
    __device__ __forceinline__ void plus_powers(uint32_t s) {
        const uint64_t s2 = (uint64_t)s * s;
        u2 += s2;
        u3 += s2 * s;
        add4(s2 * s2, (uint32_t)__umul64hi(s2, s2));
    }
    __device__ __forceinline__ void minus_powers(uint32_t s) {
        const uint64_t s2 = (uint64_t)s * s;
        u2 -= s2;
        u3 -= s2 * s;
        sub4(s2 * s2, (uint32_t)__umul64hi(s2, s2));
    }
    __device__ __forceinline__ void load(const RunState &st) {
        u2 = st.t2;
        u3 = st.t3;
        u4 = st.t4_lo;
        u4x = (uint32_t)st.t4_hi;
    }
    __device__ __forceinline__ void store(RunState &st) const {
        st.t2 = u2;
        st.t3 = u3;
        st.t4_lo = u4;
        st.t4_hi = u4x;
    }
    __device__ __forceinline__ uint64_t m2() const { return u2; }
    __device__ __forceinline__ uint32_t m4_hi() const { return u4x; }
};

__device__ __forceinline__ void decode_any(const GraphDev &g, bool shared, uint32_t e, uint32_t &u, uint32_t &v) {
    if (g.kind == NZ_GRAPH_GRID2D) {
        // shared memory: row-major node ids; global memory: the tiled slots
        if (shared) decode_edge<NZ_GRAPH_GRID2D>(g, e, u, v);
        else decode_edge_slots<NZ_GRAPH_GRID2D>(g, e, u, v);
    } else if (g.kind == NZ_GRAPH_CHAIN1D) {
        decode_edge<NZ_GRAPH_CHAIN1D>(g, e, u, v);
    } else {
        decode_edge<NZ_GRAPH_EDGES>(g, e, u, v);
        if (u >= g.N || v >= g.N) u = v = 0;  // invalid edge list: no bond
    }
}

// Bonds of the torus: e < N to the right neighbour, else to the one below;
// `down` says which.
__device__ __forceinline__ void decode_torus(const GraphDev &g, uint32_t e, uint32_t &u, uint32_t &v, bool &down) {
    down = e >= g.N;
    u = down ? e - g.N : e;
    const uint32_t row = u / g.L, col = u - row * g.L;
    v = down ? (row + 1u == g.L ? 0u : row + 1u) * g.L + col : row * g.L + (col + 1u == g.L ? 0u : col + 1u);
}

__device__ __forceinline__ uint32_t sides_any(const GraphDev &g, uint32_t i) {
    if (g.kind == NZ_GRAPH_GRID2D) return node_sides<NZ_GRAPH_GRID2D>(g, i);
    if (g.kind == NZ_GRAPH_CHAIN1D) return node_sides<NZ_GRAPH_CHAIN1D>(g, i);
    if (g.kind == NZ_GRAPH_TORUS2D) return 0u;
    return node_sides<NZ_GRAPH_EDGES>(g, i);
}

template <bool SHARED, bool TORUS>
struct DispOf {
    typedef typename std::conditional<SHARED, int32_t, int64_t>::type type;
};

template <int W, bool NARROW>
struct GroupShared {
    Sums<NARROW> carry[2];  // totals after the last finished batch, double-buffered
    Sums<NARROW> warp[W];   // what each warp's bonds add
    uint32_t clusters[2];
    uint32_t joins[W], top[W], sides[W];
    uint32_t first[4];  // span search: first bond that joins both sides / adds side 0 / side 1 to G / joins at all
    uint32_t wrap[2];       // torus: first window row at which a cluster wraps along x / y
    uint32_t winner, g_root, g_sides;
    FeistelPerm fp;         // the run's keyed permutation: its registers are needed elsewhere
};

// bytes of a run's nodes in shared memory (and of the copy kept in its node
// words between windows): the 16-bit values, then the flags, each padded to
// a word
__host__ __device__ __forceinline__ uint32_t val_bytes(uint32_t N) { return (2u * N + 3u) & ~3u; }
__host__ __device__ __forceinline__ uint32_t flag_bytes(uint32_t N) { return (N + 3u) & ~3u; }
template <bool TORUS>
__host__ __device__ __forceinline__ uint32_t node_bytes(uint32_t N) {
    return val_bytes(N) + flag_bytes(N) + (TORUS ? 4u * N : 0u);
}
// numbers that node ids run up to
template <bool SHARED, bool TORUS>
__host__ __device__ __forceinline__ uint32_t node_count(const GraphDev &g) {
    return SHARED || TORUS ? g.N : g.slots;
}

// Claims: one word per node where that is few, else enough that bonds of one
// batch seldom share a word (a bond that loses a word to a stranger waits a round
// for nothing), as far as they fit beside `nodes` bytes of a run with `blocks`
// blocks to an SM (228 KB, of which 1 KB is each block's own and 256 B are left
// for the caller).  Filling the SM beats 4,096 words whatever the nodes, which
// kept a block out where they were too many and gave up room where they were
// few: 1,000 runs of 97 x 97 1.07 -> 0.95 ms, 3,000 of 150 x 150 6.95 -> 5.77,
// 1,000 of 256 x 256 7.02 -> 6.57, of chains of 6,000 0.37 -> 0.27, of the torus
// 120 3.10 -> 1.83.  Powers of two need a cheaper hash (2 % less at L = 97), but
// leave up to half of the room (7 % more at L = 128, 18 % on the torus 120).
template <int W, bool SHARED>
__host__ __device__ __forceinline__ uint32_t claim_words(uint32_t slots, uint32_t nodes, uint32_t blocks) {
    constexpr uint32_t kMost = 16384u, kAsked = 32u * W * kE * 16u;
    constexpr uint32_t kEnough = SHARED && kAsked < kMost ? kAsked : kMost;
    const uint32_t left = 228u * 1024u / blocks - 1280u - (uint32_t)sizeof(GroupShared<W, SHARED>);
    const uint32_t room = nodes + 1024u < left ? (left - nodes) / 4u & ~31u : 256u;
    const uint32_t all = (slots + 31u) & ~31u;
    const uint32_t claims = room < kEnough ? room : kEnough;
    return claims < all ? claims : all;
}

// The most shared memory that a block's claims and nodes take: one block to an SM.
template <int W, bool SHARED>
constexpr size_t most_shared() { return 228u * 1024u - 1280u - sizeof(GroupShared<W, SHARED>); }

// The claims of a block, for all the runs it takes, at the start of its dynamic
// shared memory (a multiple of 32 words).
template <int W>
struct Claims {
    uint32_t *at;
    uint32_t count;
    uint32_t stamp;  // counts the rounds down: a new round's claims beat all older ones
    __device__ __forceinline__ void init(uint32_t *words, uint32_t n) {
        at = words;
        count = n;
        clear();
    }
    __device__ __forceinline__ void clear() {
        for (uint32_t i = threadIdx.x; i < count; i += 32u * W) at[i] = 0xffffffffu;
        stamp = kStampTop;
    }
};

// A run's node words from or to its place in global memory, with the whole block.
// 64 bytes per thread in flight where the place is at a 16-byte boundary (a word each
// left the union-find of 100,000 site runs of 256 x 256, seven windows, at 850 ms;
// now 829).
template <int W>
__device__ __forceinline__ void copy_words(uint32_t *dst, const uint32_t *src, uint32_t words) {
    uint32_t done = 0;
    if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) == 0) {
        const uint4 *from = reinterpret_cast<const uint4 *>(src);
        uint4 *to = reinterpret_cast<uint4 *>(dst);
        const uint32_t pieces = words / 4u;
        for (uint32_t i = threadIdx.x; i < pieces; i += 4u * 32u * W) {
            uint4 v[4];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (i + k * 32u * W < pieces) v[k] = from[i + k * 32u * W];
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                if (i + k * 32u * W < pieces) to[i + k * 32u * W] = v[k];
        }
        done = pieces * 4u;
    }
    for (uint32_t i = done + threadIdx.x; i < words; i += 32u * W) dst[i] = src[i];
}

// The run to be done: rows [n_begin, n_end) of it.
struct Run {
    const uint32_t *perm;  // the order of its bonds, or null: the keyed permutation of
    uint64_t key, id;      // this key and run id
    uint32_t *home;        // its node words in global memory (between windows, or all along)
    RunState *state;       // its state between windows (null: one window)
    uint32_t n_begin, n_end;
    bool spanning, init_both;
};

// Does the rows of `run` (SITE: of site percolation) with the whole block of W warps, handing batches of
// rows to `sink`: wants(base, B) says (for the whole block alike) whether rows
// base .. base + B - 1 of the window are wanted, put(i0, ...) takes this
// thread's rows i0 .. i0 + E - 1 (rows past the window's end among them).
// `nodes`: shared memory for node_bytes of the run (SHARED only).  TORUS: the
// flag of a row says that a cluster wraps (g.wrap); other lattices: that one
// spans.
// Every thread of the block calls it and may call it again at once.  Returns
// whether the run is finished and was found corrupt.
template <int W, bool SHARED, bool TORUS, bool SITE, class Sink>
__device__ __forceinline__ bool group_run(const GraphDev &g, const Run &run, GroupShared<W, SHARED> &sh,
                                          Claims<W> &claims, uint8_t *nodes, Sink &sink) {
    constexpr bool NARROW = SHARED;
    constexpr int E = SITE ? 1 : kE;  // steps per thread and batch
    constexpr int C = 4;              // finds: both ends of two bonds, or a site's neighbours
    constexpr uint32_t B = 32u * W * E;
    constexpr uint32_t kNone = 0xffffffffu;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    typedef Nodes<SHARED, TORUS> NodesT;
    NodesT nd;
    if constexpr (SHARED) {
        nd.val = reinterpret_cast<volatile uint16_t *>(nodes);
        nd.flag = nodes + val_bytes(g.N);
        if constexpr (TORUS) nd.off = reinterpret_cast<int32_t *>(nodes + val_bytes(g.N) + flag_bytes(g.N));
    } else if constexpr (TORUS) {
        nd.cell = reinterpret_cast<uint4 *>(run.home);
    } else {
        nd.w = run.home;
    }

    // ---- state at the start of the window
    bool span = false, init_both = false, corrupt = false;
    if (run.n_begin == 0) {
        if constexpr (SHARED) {
            for (uint32_t i = t; i < g.N; i += 32u * W) {
                if (SITE) nd.set_empty(i);
                else nd.set_root(i, 1u, sides_any(g, i));
            }
        } else {
            for (uint32_t j = t; j < node_count<SHARED, TORUS>(g); j += 32u * W) {
                uint32_t i = j;
                if (g.kind == NZ_GRAPH_GRID2D && kGridTiled) {
                    const uint32_t tile = j >> 3, w = j & 7u;
                    const uint32_t tr = tile / g.tile_cols, tc = tile - tr * g.tile_cols;
                    const uint32_t row = 2u * tr + (w >> 2), col = 4u * tc + (w & 3u);
                    if (row >= g.L || col >= g.L) continue;  // a padding slot, never read
                    i = row * g.L + col;
                }
                if (SITE) nd.set_empty(j);
                else nd.set_root(j, 1u, sides_any(g, i));
            }
        }
        init_both = !SITE && run.init_both;
        if (t < 2) sh.wrap[t] = 0xffffffffu;
        if (t == 0) {
            sh.g_root = SITE ? kNone : 0u;
            sh.g_sides = SITE ? 0u : sides_any(g, 0);
            Sums<NARROW> c;  // bonds: N clusters of one node, one of them G; sites: none
            c.zero();
            RunState all;
            all.t2 = all.t3 = all.t4_lo = g.N;
            all.t4_hi = 0;
            if (!SITE) {
                c.load(all);
                c.minus_powers(1u);
                c.g = 1;
            }
            sh.carry[0] = c;
            sh.clusters[0] = SITE ? 0u : g.N;
        }
    } else {
        const RunState st = *run.state;
        span = (st.flags & kFlagSpan) != 0;
        init_both = (st.flags & kFlagInitBoth) != 0;
        corrupt = (st.flags & kFlagCorrupt) != 0;
        if (t < 2) sh.wrap[t] = (st.flags & (t == 0 ? kFlagWrapX : kFlagWrapY)) ? 0u : 0xffffffffu;
        if constexpr (SHARED) {
            copy_words<W>(reinterpret_cast<uint32_t *>(nodes), run.home, node_bytes<TORUS>(g.N) / 4u);
        }
        if (t == 0) {
            Sums<NARROW> c;
            c.load(st);
            c.minus_powers(st.max);
            c.g = st.max;
            sh.carry[0] = c;
            sh.clusters[0] = st.t0;
            sh.g_root = st.pad;
            sh.g_sides = (st.flags >> 8) & 3u;
        }
    }
    if (t < 4) sh.first[t] = 0xffffffffu;
    if (t == 0) {
        sh.winner = 0xffffffffu;
        if (!run.perm) sh.fp.init(run.key, run.id, g.M);
    }
    __syncthreads();
    uint32_t G = sh.g_root, g_size = sh.carry[0].g, g_sides = sh.g_sides;
    uint32_t cur = 0;  // sh.carry buffer in use

    const bool given = run.perm != nullptr;
    const uint32_t rows = run.n_end - run.n_begin;
    uint32_t ahead[E];  // keyed bonds of the next batch
    bool have_ahead = false;
    // M well below its power of two: cycle walks are common (the domain is
    // 1.8 M at L = 97, within 1.01 M at L = 2^k)
    const bool walks = !given && (sh.fp.maskR + 1ull) * (sh.fp.maskL + 1ull) > g.M + g.M / 8ull;

    // torus: (dx, dy) of a bond (0 to the right, 1 downwards), or from a site to
    // its neighbour 0 right, 1 left, 2 below, 3 above
    typedef typename DispOf<SHARED, TORUS>::type Disp;
    auto step = [](int dir) {
        constexpr Disp kDx = (Disp)1 << (SHARED ? 16 : 32);
        if (SITE) return dir == 0 ? kDx : dir == 1 ? -kDx : dir == 2 ? (Disp)1 : (Disp)-1;
        return dir ? (Disp)1 : kDx;
    };
    // a loop closed at window row `row` winds around the torus where the two
    // ways around it differ by d
    auto close_loop = [&](Disp d, uint32_t row) {
        if constexpr (TORUS) {
            if (d == 0) return;
            if (NodesT::dx(d) != 0 && row < sh.wrap[0]) atomicMin(&sh.wrap[0], row);
            if (NodesT::dy(d) != 0 && row < sh.wrap[1]) atomicMin(&sh.wrap[1], row);
        }
    };
    (void)step;
    (void)close_loop;

    for (uint32_t base = 0; base < rows; base += B) {
        const uint32_t i0 = base + t * E;
        // ---- 1. the bonds of rows i0, i0 + 1 (the site of row i0) and the roots of
        // their ends (of its neighbours)
        uint32_t edge[E];
#pragma unroll
        for (int k = 0; k < E; ++k) edge[k] = 0;
        if (!given && g.M > 0) {
            auto from = [&](uint32_t j) {
                const uint32_t idx = run.n_begin + i0 + j % E + (j / E) * B - 1u;
                return idx < g.M ? idx : 0u;
            };
            if (!walks) {
                const FeistelPerm fp = sh.fp;
#pragma unroll
                for (int k = 0; k < E; ++k) edge[k] = fp.at(from(k));
            } else if (have_ahead) {
#pragma unroll
                for (int k = 0; k < E; ++k) edge[k] = ahead[k];
                have_ahead = false;
            } else {
                // this batch's bonds and the next one's in one loop: a lane
                // goes on to its next bond when the cycle walk of one ends, so
                // the warp waits for the longest sum of 2 E walks, not 2 E
                // times for the longest walk
                const FeistelPerm fp = sh.fp;
                uint32_t j = 0, y = from(0);
                while (j < 2 * E) {
                    y = fp.encrypt(y);
                    if (y < g.M) {
#pragma unroll
                        for (int k = 0; k < E; ++k) {
                            if (j == (uint32_t)k) edge[k] = y;
                            if (j == (uint32_t)(E + k)) ahead[k] = y;
                        }
                        ++j;
                        y = from(j);
                    }
                }
                have_ahead = true;
            }
        }
        uint32_t start[C], x[C], w[C], first_w[C];
        bool open[E], down[E] = {}, linked[C] = {};
        uint32_t self = 0, self_sides = 0;  // the site's own node
        typename DispOf<SHARED, TORUS>::type pos[C] = {};  // displacement of each start node from x
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const uint32_t n = run.n_begin + i0 + k;
            open[k] = i0 + k < rows && n > 0;
            if (open[k] && given) edge[k] = __ldg(run.perm + (n - 1u));
            if (!open[k]) edge[k] = 0;
            if (given && edge[k] >= g.M) open[k] = false;  // caller-supplied index out of range: nothing happens
        }
        if constexpr (!SITE) {
#pragma unroll
            for (int k = 0; k < E; ++k) {
                start[2 * k] = start[2 * k + 1] = 0;
                if (open[k]) {
                    if constexpr (TORUS) decode_torus(g, edge[k], start[2 * k], start[2 * k + 1], down[k]);
                    else decode_any(g, SHARED, edge[k], start[2 * k], start[2 * k + 1]);
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                x[c] = start[c];
                w[c] = nd.load(x[c]);
                first_w[c] = w[c];
            }
        } else {
            // occupy the batch's sites: until its turn a new site's node says
            // at which position of the batch it comes
            const uint32_t site = edge[0];
            const bool chain = !TORUS && g.kind == NZ_GRAPH_CHAIN1D;
            const uint32_t width = chain ? g.N : g.L, height = chain ? 1u : g.L;
            const uint32_t row = chain ? 0u : site / width, col = site - row * width;
            auto slot = [&](uint32_t rr, uint32_t cc) {
                if (!SHARED && !TORUS && g.kind == NZ_GRAPH_GRID2D && kGridTiled) return grid_slot(g.tile_cols, rr, cc);
                return rr * width + cc;
            };
            self = slot(row, col);
            if (open[0]) open[0] = nd.is_empty(nd.load(self));
            self_sides = sides_any(g, site);
            __syncthreads();
            if (open[0]) nd.set_new(self, t, self_sides);
            __syncthreads();
            if (given) {
                // a caller's order may name a site twice in a batch: its first
                // time counts (each turn lowers some site's position)
                for (;;) {
                    const bool earlier = open[0] && new_at(nd.load(self)) > t;
                    if (!__syncthreads_or(earlier)) break;
                    if (earlier) nd.set_new(self, t, self_sides);
                    __syncthreads();
                }
                open[0] = open[0] && new_at(nd.load(self)) == t;
            }
            // neighbours that are occupied by now: right, left, below, above
#pragma unroll
            for (int c = 0; c < C; ++c) {
                bool there = open[0];
                uint32_t rr = row, cc = col;
                if constexpr (TORUS) {
                    if (c == 0) cc = col + 1u == width ? 0u : col + 1u;
                    if (c == 1) cc = col == 0 ? width - 1u : col - 1u;
                    if (c == 2) rr = row + 1u == height ? 0u : row + 1u;
                    if (c == 3) rr = row == 0 ? height - 1u : row - 1u;
                } else {
                    if (c == 0) { there = there && col + 1u < width; cc = col + 1u; }
                    if (c == 1) { there = there && col > 0; cc = col - 1u; }
                    if (c == 2) { there = there && row + 1u < height; rr = row + 1u; }
                    if (c == 3) { there = there && row > 0; rr = row - 1u; }
                }
                start[c] = x[c] = there ? slot(rr, cc) : self;
                w[c] = kRoot;
                if (there) {
                    const uint32_t v = nd.load(x[c]);
                    linked[c] = !nd.is_empty(v) && !(is_new(v) && new_at(v) > t);
                    if (linked[c]) w[c] = v;
                }
                first_w[c] = w[c];
            }
        }
        auto climb = [&]() {
            for (int hops = 0; hops < kMaxHops; ++hops) {
                bool more = false;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    if (!is_root(w[c])) {
                        if constexpr (TORUS) pos[c] += nd.disp(x[c]);
                        x[c] = w[c];
                        w[c] = nd.load(x[c]);
                        more |= !is_root(w[c]);
                    }
                }
                if (!more) return;
            }
            corrupt = true;
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (!is_root(w[c])) {  // what cannot be placed joins nothing
                    if (SITE) linked[c] = false;
                    else x[c & ~1] = x[c | 1];
                }
        };
        climb();
        if constexpr (!TORUS) {
#pragma unroll
            for (int c = 0; c < C; ++c)
                if (!is_root(first_w[c]) && first_w[c] != x[c]) nd.shorten(start[c], x[c]);
        }

        // ---- 2., 3. rounds of joins
        Sums<NARROW> d[E];
        uint32_t formed[E], sd[E], kind[E];  // kind: 0 nothing, 1 a cluster other than G formed, 2 joined to G
        uint32_t fewer[E];                   // clusters lost by the step (modulo 2^32)
#pragma unroll
        for (int k = 0; k < E; ++k) {
            d[k].zero();
            formed[k] = sd[k] = kind[k] = fewer[k] = 0;
        }
        bool any_join = false;
        for (uint32_t round = 0; round <= B; ++round) {
            const uint32_t tag = (claims.stamp << kTagBits) | (t * E);
            bool wants = false;
            uint32_t h[C], h_self = 0;
            auto hash = [&](uint32_t at) {
                return node_count<SHARED, TORUS>(g) <= claims.count ? at : __umulhi(at * 0x9E3779B1u, claims.count);
            };
#pragma unroll
            for (int c = 0; c < C; ++c) h[c] = hash(x[c]);
            if constexpr (SITE) {
                // a site claims its own node too: its later neighbours wait
                h_self = hash(self);
                if (open[0]) {
                    wants = true;
                    atomicMin(claims.at + h_self, tag);
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        if (linked[c] && x[c] != G) atomicMin(claims.at + h[c], tag);
                }
            } else {
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    if constexpr (TORUS) {
                        // a bond inside one cluster closes a loop
                        if (open[k] && x[2 * k] == x[2 * k + 1])
                            close_loop(pos[2 * k] + step(down[k]) - pos[2 * k + 1], i0 + k);
                    }
                    open[k] = open[k] && x[2 * k] != x[2 * k + 1];
                    if (!open[k]) continue;
                    wants = true;
                    if (x[2 * k] != G) atomicMin(claims.at + h[2 * k], tag + k);
                    if (x[2 * k + 1] != G) atomicMin(claims.at + h[2 * k + 1], tag + k);
                }
            }
            if (!__syncthreads_or(wants)) break;
            any_join = true;
            const bool wanted = wants;
            wants = false;
            if constexpr (TORUS) {
                if (round == 0) {
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        if (!is_root(first_w[c]) && first_w[c] != x[c]) {
                            nd.shorten(start[c], x[c]);
                            nd.set_disp(start[c], pos[c]);
                        }
                }
            }
            if constexpr (SITE) {
                if (open[0]) {
                    bool lost = claims.at[h_self] != tag;
#pragma unroll
                    for (int c = 0; c < C; ++c) lost |= linked[c] && x[c] != G && claims.at[h[c]] != tag;
                    wants = lost;
                    if (!lost) {
                        open[0] = false;
                        // the site (one node, so far in no total) and the
                        // distinct clusters around it become one
                        bool first_of[C], with_g = false;
                        uint32_t total = 1, most = 1, big = self, held = 0;
                        sd[0] = self_sides;
                        typename DispOf<SHARED, TORUS>::type at_big = 0;  // the site's position in big's cluster
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            first_of[c] = linked[c] && x[c] != self;
                            if constexpr (TORUS) {
                                pos[c] -= step(c);  // the site's position in x's cluster
                                if (linked[c] && x[c] == self) close_loop(pos[c], i0);
                            }
#pragma unroll
                            for (int q = 0; q < c; ++q)
                                if (linked[c] && linked[q] && x[q] == x[c]) {
                                    if constexpr (TORUS) {
                                        if (first_of[q]) close_loop(pos[c] - pos[q], i0);
                                    }
                                    first_of[c] = false;
                                }
                            if (!first_of[c]) continue;
                            ++held;
                            if (x[c] == G) {
                                with_g = true;
                                if constexpr (TORUS) at_big = pos[c];
                                continue;
                            }
                            const uint32_t size = nd.size(w[c]);
                            total += size;
                            d[0].minus_powers(size);
                            sd[0] |= root_sides(w[c]);
                        }
                        if (with_g) {
                            big = G;
                        } else {
#pragma unroll
                            for (int c = 0; c < C; ++c) {
                                const uint32_t size = nd.size(w[c]);
                                if (first_of[c] && (size > most || big == self)) {
                                    most = size;
                                    big = x[c];
                                    if constexpr (TORUS) at_big = pos[c];
                                }
                            }
                        }
#pragma unroll
                        for (int c = 0; c < C; ++c) {
                            if (!first_of[c] || x[c] == big) continue;
                            nd.link(x[c], big);
                            if constexpr (TORUS) nd.set_disp(x[c], at_big - pos[c]);
                        }
                        if (self != big) {
                            nd.link(self, big);
                            if constexpr (TORUS) nd.set_disp(self, at_big);
                        }
                        kind[0] = with_g ? 2 : 1;
                        fewer[0] = held - 1u;
                        if (with_g) {
                            d[0].g = total;
                        } else {
                            nd.set_root(big, total, sd[0]);
                            d[0].plus_powers(total);
                            formed[0] = total;
                        }
                    }
                }
            } else {
                // (a warp with no bond left does without, but in shared memory the
                // code is faster without the branch)
                if (SHARED || __any_sync(0xffffffffu, wanted))
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    if (!open[k]) continue;
                    const uint32_t xu = x[2 * k], xv = x[2 * k + 1];
                    const bool gu = xu == G, gv = xv == G;
                    if ((!gu && claims.at[h[2 * k]] != tag + k) || (!gv && claims.at[h[2 * k + 1]] != tag + k)) {
                        wants = true;
                        continue;
                    }
                    open[k] = false;
                    fewer[k] = 1;
                    const uint32_t a = nd.size(w[2 * k]), b = nd.size(w[2 * k + 1]);
                    if constexpr (TORUS) {
                        // position of v's root as seen from u's
                        const auto d = pos[2 * k] + step(down[k]) - pos[2 * k + 1];
                        const bool under_u = gu || (!gv && a >= b);
                        nd.set_disp(under_u ? xv : xu, under_u ? d : -d);
                    }
                    if (gu || gv) {
                        const uint32_t c = gu ? xv : xu, wc = gu ? w[2 * k + 1] : w[2 * k];
                        nd.link(c, G);
                        kind[k] = 2;
                        d[k].absorb(gu ? b : a);
                        sd[k] = root_sides(wc);
                    } else {
                        const bool keep_u = a >= b;
                        kind[k] = 1;
                        sd[k] = root_sides(w[2 * k]) | root_sides(w[2 * k + 1]);
                        nd.link(keep_u ? xv : xu, keep_u ? xu : xv);
                        nd.set_root(keep_u ? xu : xv, a + b, sd[k]);
                        d[k].join(a, b);
                        formed[k] = a + b;
                    }
                }
            }
            if (--claims.stamp == 0) {  // stamps used up: start over with a clean table
                __syncthreads();
                claims.clear();
            }
            if (!__syncthreads_or(wants)) break;
            // the roots of unfinished bonds may have been joined to others (of
            // many warps, one with none goes straight on to the next barrier)
            if ((SHARED && W <= 4) || __any_sync(0xffffffffu, wants)) {
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (SITE ? open[0] && linked[c] : open[(c >> 1) % E]) w[c] = nd.load(x[c]);
                climb();
            }
        }

        // ---- 4. totals after every bond
        const bool want = sink.wants(base, B);
        // torus: first window row whose flag is set (a later row of another
        // thread's next batch may be in already; it does not reach these rows)
        uint32_t wrap_row = 0xffffffffu;
        if constexpr (TORUS) {
            if (run.spanning) {
                const uint32_t rx = sh.wrap[0], ry = sh.wrap[1];
                wrap_row = g.wrap == 0 ? min(rx, ry) : g.wrap == 1 ? rx : g.wrap == 2 ? ry : max(rx, ry);
            }
        }
        uint32_t ms[E], m0[E];
        Sums<NARROW> m[E];
        if (!any_join) {
            const Sums<NARROW> c = sh.carry[cur];
            const uint32_t cl = sh.clusters[cur] - (SITE && sh.clusters[cur] == 0 ? 0u : 1u);
#pragma unroll
            for (int k = 0; k < E; ++k) {
                m[k] = c;
                m0[k] = cl;
                ms[k] = g_size | (span || i0 + k >= wrap_row ? kSpanBit : 0u);
            }
        } else {
            // prefix sums over the thread's bonds, then over the warp
            uint32_t top[E];
            top[0] = formed[0];
#pragma unroll
            for (int k = 1; k < E; ++k) {
                top[k] = formed[k];
                d[k].add(d[k - 1]);
                top[k] = max(top[k], top[k - 1]);
            }
            Sums<NARROW> inc = d[E - 1];
            uint32_t tmax = top[E - 1], joins = 0;
#pragma unroll
            for (int k = 0; k < E; ++k) joins += fewer[k];
            uint32_t njoin = joins;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const Sums<NARROW> y = inc.up(o);
                const uint32_t ym = __shfl_up_sync(0xffffffffu, tmax, o), yj = __shfl_up_sync(0xffffffffu, njoin, o);
                if (lane >= (uint32_t)o) {
                    inc.add(y);
                    tmax = max(tmax, ym);
                    njoin += yj;
                }
            }
            uint32_t sall = 0;
#pragma unroll
            for (int k = 0; k < E; ++k) sall |= sd[k];
            sall = __reduce_or_sync(0xffffffffu, sall);
            if (lane == 31) {
                sh.warp[warp] = inc;
                sh.top[warp] = tmax;
                sh.joins[warp] = njoin;
                sh.sides[warp] = sall;
            }
            __syncthreads();
            // before this thread's bonds: the carry, the earlier warps, the
            // earlier lanes.  Of the whole batch: the largest cluster formed
            // other than G, the sides touched, what G gained
            Sums<NARROW> pre = sh.carry[cur];
            uint32_t ptop = 0, pj = 0, top_all = 0, sides_all = g_sides, grown = g_size;
            if constexpr (W <= 4) {
#pragma unroll
                for (uint32_t q = 0; q < (uint32_t)W; ++q) {
                    if (q < warp) {
                        pre.add(sh.warp[q]);
                        ptop = max(ptop, sh.top[q]);
                        pj += sh.joins[q];
                    }
                    top_all = max(top_all, sh.top[q]);
                    sides_all |= sh.sides[q];
                    grown += sh.warp[q].g;
                }
            } else {
                // lane q takes warp q, and the warp sums over its lanes
                Sums<NARROW> of;
                of.zero();
                uint32_t qtop = 0, qside = 0, qj = 0, qg = 0;
                if (lane < (uint32_t)W) {
                    of = sh.warp[lane];
                    qtop = sh.top[lane];
                    qside = sh.sides[lane];
                    qj = sh.joins[lane];
                    qg = of.g;
                }
                top_all = __reduce_max_sync(0xffffffffu, qtop);
                sides_all |= __reduce_or_sync(0xffffffffu, qside);
                grown += __reduce_add_sync(0xffffffffu, qg);
                if (lane >= warp) {
                    of.zero();
                    qtop = qj = 0;
                }
                ptop = __reduce_max_sync(0xffffffffu, qtop);
                pj = __reduce_add_sync(0xffffffffu, qj);
                pre.add(of.over_warp());
            }
            {
                const Sums<NARROW> y = inc.up(1);
                const uint32_t ym = __shfl_up_sync(0xffffffffu, tmax, 1);
                if (lane > 0) {
                    pre.add(y);
                    ptop = max(ptop, ym);
                }
                pj += njoin - joins;
            }
            const uint32_t cl = sh.clusters[cur];
            // first row (of the batch) at which a cluster spans
            uint32_t span_row = span ? 0u : 0xffffffffu;
            if (!TORUS && run.spanning && !span && (sides_all == 3u || init_both)) {
#pragma unroll
                for (int k = 0; k < E; ++k) {
                    if (kind[k] == 0) continue;
                    const uint32_t row = t * E + k;
                    if (init_both) atomicMin(&sh.first[3], row);
                    if (kind[k] == 1) {
                        if (sd[k] == 3u) atomicMin(&sh.first[0], row);
                    } else {
                        if (sd[k] & 1u) atomicMin(&sh.first[1], row);
                        if (sd[k] & 2u) atomicMin(&sh.first[2], row);
                    }
                }
                __syncthreads();
                // a node that touches both sides: the first join of all; else G
                // spans from the join that brings it its missing side
                const uint32_t f1 = (g_sides & 1u) ? 0u : sh.first[1], f2 = (g_sides & 2u) ? 0u : sh.first[2];
                span_row = init_both ? sh.first[3] : min(sh.first[0], max(f1, f2));
                __syncthreads();
                if (t < 4) sh.first[t] = 0xffffffffu;
            }
#pragma unroll
            for (int k = 0; k < E; ++k) {
                pj += fewer[k];
                if (!want) continue;
                m[k] = pre;
                m[k].add(d[k]);
                m0[k] = cl - pj - (SITE && cl == pj ? 0u : 1u);
                const uint32_t gs = m[k].g, largest = max(gs, max(ptop, top[k]));
                if (largest != gs) {  // moments leave out the largest cluster, which is not G here
                    m[k].plus_powers(gs);
                    m[k].minus_powers(largest);
                }
                ms[k] = largest | (t * E + k >= span_row || i0 + k >= wrap_row ? kSpanBit : 0u);
            }
            if (t == 32u * W - 1u) {
                Sums<NARROW> c = pre;
                c.add(d[E - 1]);
                sh.carry[cur ^ 1u] = c;
                sh.clusters[cur ^ 1u] = cl - pj;
            }
            span = span || span_row != 0xffffffffu;
            // sides that G has now: those of the clusters it took in
            uint32_t gsd = 0;
#pragma unroll
            for (int k = 0; k < E; ++k) gsd |= kind[k] == 2 ? sd[k] : 0u;
            g_size = grown;
            cur ^= 1u;
            if (sides_all != g_sides) {
                const bool s1 = __syncthreads_or(gsd & 1u), s2 = __syncthreads_or(gsd & 2u);
                g_sides |= (s1 ? 1u : 0u) | (s2 ? 2u : 0u);
            }
            if (top_all > g_size) {
                // another cluster is the largest now: it becomes G
#pragma unroll
                for (int k = 0; k < E; ++k)
                    if (formed[k] == top_all) atomicMin(&sh.winner, t * E + k);
                __syncthreads();
                const uint32_t win = sh.winner;
                if (win / E == t) {
                    uint32_t root = SITE ? self : x[0];
#pragma unroll
                    for (int k = 1; k < E; ++k)
                        if (win % E == (uint32_t)k) root = x[2 * k];
                    uint32_t wr = nd.load(root);
                    for (int hops = 0; hops < kMaxHops && !is_root(wr); ++hops) {
                        root = wr;
                        wr = nd.load(root);
                    }
                    if (!SITE || G != kNone) nd.set_root(G, g_size, g_sides);
                    sh.g_root = root;
                    sh.g_sides = root_sides(wr);
                    Sums<NARROW> c = sh.carry[cur];
                    c.plus_powers(g_size);
                    c.minus_powers(top_all);
                    c.g = top_all;
                    sh.carry[cur] = c;
                }
                __syncthreads();
                if (t == 0) sh.winner = 0xffffffffu;
                G = sh.g_root;
                g_sides = sh.g_sides;
                g_size = top_all;
            }
        }
        if (want) sink.put(i0, ms, m0, m, edge);
    }

    // ---- state at the end of the window
    const bool last = run.n_end == g.M + 1u;
    __syncthreads();
    if (!last) {
        if (t == 0 && (!SITE || G != kNone)) nd.set_root(G, g_size, g_sides);
        __syncthreads();
        if constexpr (SHARED) {
            copy_words<W>(run.home, reinterpret_cast<const uint32_t *>(nodes), node_bytes<TORUS>(g.N) / 4u);
        }
    }
    const bool bad = __syncthreads_or(corrupt);
    if (t == 0 && run.state) {
        RunState st;
        Sums<NARROW> c = sh.carry[cur];
        c.plus_powers(g_size);
        c.store(st);
        st.t0 = sh.clusters[cur];
        st.max = g_size;
        st.flags = (span ? kFlagSpan : 0u) | (init_both ? kFlagInitBoth : 0u) | (bad ? kFlagCorrupt : 0u) |
                   (g_sides << 8);
        if (TORUS)
            st.flags |= (sh.wrap[0] != 0xffffffffu ? kFlagWrapX : 0u) | (sh.wrap[1] != 0xffffffffu ? kFlagWrapY : 0u);
        st.pad = G;
        *run.state = st;
    }
    return bad && last;
}

}  // namespace group
}  // namespace nz
