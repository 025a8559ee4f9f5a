// nz_uf.cu -- permutations, reference rows and the union-find's dispatch.
//
// Bond percolation (percolate/hpc.py:249-307, bond_sample_states) runs in
// nz_ufg.cu, site percolation and the torus in nz_lattice.cu; all of them
// write the per-step records that the consumers share.
#include <cstdint>

#include "nz_common.cuh"
#include "nz_internal.cuh"
#include "nz_records.cuh"

namespace nz {

__global__ void any_both_sides_kernel(GraphDev g, uint32_t *flag) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < g.N; i += gridDim.x * blockDim.x)
        if (g.side && (g.side[i] & 3u) == 3u) *flag = kFlagInitBoth;
}

// ------------------------------------------------------- permutation kernels
__global__ void philox_perm_kernel(uint32_t M, int32_t n_runs, uint64_t key, uint64_t run0,
                                   uint32_t *out) {
    const uint64_t total = (uint64_t)n_runs * M;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t r = (uint32_t)(i / M), n = (uint32_t)(i % M);
        FeistelPerm fp;
        fp.init(key, run0 + r, M);
        out[i] = fp.at(n);
    }
}

// MT19937 (Matsumoto & Nishimura 1998) with the authors' init_genrand and
// init_by_array seeding; then the Fisher-Yates shuffle with masked rejection
// that numpy's legacy RandomState.permutation(M) performs.  One thread per
// run; the 624-word state lives in local memory.
struct Mt19937 {
    uint32_t mt[624];
    int mti;

    __device__ void init_genrand(uint32_t seed) {
        mt[0] = seed;
        for (int i = 1; i < 624; ++i) mt[i] = 1812433253u * (mt[i - 1] ^ (mt[i - 1] >> 30)) + (uint32_t)i;
        mti = 624;
    }
    __device__ void init_by_array(const uint32_t *key, int len) {
        init_genrand(19650218u);
        int i = 1, j = 0;
        for (int k = (624 > len ? 624 : len); k; --k) {
            mt[i] = (mt[i] ^ ((mt[i - 1] ^ (mt[i - 1] >> 30)) * 1664525u)) + key[j] + (uint32_t)j;
            ++i; ++j;
            if (i >= 624) { mt[0] = mt[623]; i = 1; }
            if (j >= len) j = 0;
        }
        for (int k = 623; k; --k) {
            mt[i] = (mt[i] ^ ((mt[i - 1] ^ (mt[i - 1] >> 30)) * 1566083941u)) - (uint32_t)i;
            ++i;
            if (i >= 624) { mt[0] = mt[623]; i = 1; }
        }
        mt[0] = 0x80000000u;
        mti = 624;
    }
    __device__ uint32_t next() {
        if (mti >= 624) {
            for (int kk = 0; kk < 624; ++kk) {
                uint32_t y = (mt[kk] & 0x80000000u) | (mt[kk + 1 < 624 ? kk + 1 : 0] & 0x7fffffffu);
                int src = kk + 397 < 624 ? kk + 397 : kk + 397 - 624;
                mt[kk] = mt[src] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
            }
            mti = 0;
        }
        uint32_t y = mt[mti++];
        y ^= (y >> 11);
        y ^= (y << 7) & 0x9d2c5680u;
        y ^= (y << 15) & 0xefc60000u;
        y ^= (y >> 18);
        return y;
    }
};

__global__ void mt_perm_kernel(uint32_t M, int32_t n_runs, const uint32_t *seed_words,
                               const int32_t *seed_len, int32_t stride, uint32_t *out) {
    const int32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_runs) return;
    Mt19937 g;
    const int len = seed_len[r];
    const uint32_t *w = seed_words + (size_t)r * stride;
    if (len == 0) g.init_genrand(w[0]);
    else g.init_by_array(w, len);
    uint32_t *o = out + (size_t)r * M;
    for (uint32_t i = 0; i < M; ++i) o[i] = i;
    for (int64_t i = (int64_t)M - 1; i >= 1; --i) {
        uint32_t mx = (uint32_t)i, mask = mx;
        mask |= mask >> 1; mask |= mask >> 2; mask |= mask >> 4; mask |= mask >> 8; mask |= mask >> 16;
        uint32_t j;
        do { j = g.next() & mask; } while (j > mx);
        uint32_t t = o[i]; o[i] = o[j]; o[j] = t;
    }
}

// Continuation of one MT19937 stream (numpy's global RandomState): the state
// (624 words + position) is loaded, n_runs permutations of range(M) are drawn
// one after another exactly as np.random.permutation(M) would draw them
// (percolate/percolate.py:270, once per run in run order), and the advanced
// state is stored back.  One thread: the stream is sequential by nature.
__global__ void mt_stream_perm_kernel(const uint32_t *state_in, uint32_t M, int32_t n_runs, uint32_t *out,
                                      uint32_t *state_out) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    Mt19937 g;
    for (int i = 0; i < 624; ++i) g.mt[i] = state_in[i];
    g.mti = (int)state_in[624];
    for (int32_t r = 0; r < n_runs; ++r) {
        uint32_t *o = out + (size_t)r * M;
        for (uint32_t i = 0; i < M; ++i) o[i] = i;
        for (int64_t i = (int64_t)M - 1; i >= 1; --i) {
            uint32_t mx = (uint32_t)i, mask = mx;
            mask |= mask >> 1; mask |= mask >> 2; mask |= mask >> 4; mask |= mask >> 8; mask |= mask >> 16;
            uint32_t j;
            do { j = g.next() & mask; } while (j > mx);
            uint32_t t = o[i]; o[i] = o[j]; o[j] = t;
        }
    }
    for (int i = 0; i < 624; ++i) state_out[i] = g.mt[i];
    state_out[624] = (uint32_t)g.mti;
}

void launch_mt_stream_perms(const uint32_t *state_in, uint32_t M, int32_t n_runs, uint32_t *out,
                            uint32_t *state_out, cudaStream_t s) {
    mt_stream_perm_kernel<<<1, 1, 0, s>>>(state_in, M, n_runs, out, state_out);
}

// ---------------------------------------------------------------- packing
// Reference row layout (packed little-endian), percolate/hpc.py:34-70:
//   n u32 | edge u32 | [has_spanning_cluster u8] | max_cluster_size u32 | moments 5 x u64
__device__ __forceinline__ void put_bytes(uint8_t *dst, uint64_t v, int nbytes) {
    for (int i = 0; i < nbytes; ++i) dst[i] = (uint8_t)(v >> (8 * i));
}

__global__ void pack_rows_kernel(NzRecords rec, int32_t run, uint32_t N, uint32_t M, int32_t spanning,
                                 uint8_t *rows) {
    const uint32_t row_bytes = spanning ? 53u : 52u;
    for (uint32_t n = blockIdx.x * blockDim.x + threadIdx.x; n <= M; n += gridDim.x * blockDim.x) {
        const size_t off = (size_t)n * rec.run_stride + run;
        uint8_t *d = rows + (size_t)n * row_bytes;
        const uint32_t ms = rec.max_span[off];
        const uint32_t mx = ms & ~kSpanBit;
        put_bytes(d, n, 4);
        put_bytes(d + 4, rec.edge ? rec.edge[off] : 0u, 4);
        int o = 8;
        if (spanning) { d[8] = (ms & kSpanBit) ? 1 : 0; o = 9; }
        put_bytes(d + o, mx, 4);
        put_bytes(d + o + 4, record_m0(rec, off), 8);
        put_bytes(d + o + 12, (uint64_t)((rec.site ? n : N) - mx), 8);
        put_bytes(d + o + 20, record_m2(rec, off), 8);
        put_bytes(d + o + 28, rec.m3[off], 8);
        put_bytes(d + o + 36, rec.m4_lo[off], 8);
    }
}

// ------------------------------------------------------------ launchers
const uint32_t *launch_init_runs(const GraphDev &g, int32_t n_runs, uint32_t *nodes, RunState *state,
                                 uint32_t *flag_scratch, cudaStream_t s) {
    if (lattice_extension(g)) {
        launch_init_lattice_runs(g, n_runs, nodes, state, s);
        return nullptr;
    }
    // bond percolation: the union-find kernel initialises its runs itself
    if (g.kind != NZ_GRAPH_EDGES) return nullptr;
    cudaMemsetAsync(flag_scratch, 0, sizeof(uint32_t), s);
    any_both_sides_kernel<<<(g.N + 255) / 256 < 1024 ? (g.N + 255) / 256 : 1024, 256, 0, s>>>(g, flag_scratch);
    return flag_scratch;
}

void launch_uf_window(const UfParams &p, int perm_mode, bool span, int block, cudaStream_t s) {
    if (lattice_extension(p.g)) launch_lattice_window(p, perm_mode, span, block, s);
    else launch_uf_groups(p, perm_mode != NZ_PERM_PHILOX, span, s);
}

void launch_philox_perms(uint32_t M, int32_t n_runs, uint64_t key, uint64_t run0, uint32_t *out,
                         cudaStream_t s) {
    uint64_t total = (uint64_t)n_runs * M;
    uint64_t blocks = (total + 255) / 256;
    if (blocks > 152ull * 64) blocks = 152ull * 64;
    if (blocks == 0) return;
    philox_perm_kernel<<<(unsigned)blocks, 256, 0, s>>>(M, n_runs, key, run0, out);
}

void launch_mt_perms(uint32_t M, int32_t n_runs, const uint32_t *seed_words, const int32_t *seed_len,
                     int32_t stride, uint32_t *out, cudaStream_t s) {
    if (n_runs <= 0) return;
    mt_perm_kernel<<<(n_runs + 63) / 64, 64, 0, s>>>(M, n_runs, seed_words, seed_len, stride, out);
}

void launch_pack_rows(const NzRecords &rec, int32_t run, uint32_t N, uint32_t M, int32_t spanning,
                      uint8_t *rows, cudaStream_t s) {
    uint32_t blocks = (M + 1 + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    pack_rows_kernel<<<blocks, 256, 0, s>>>(rec, run, N, M, spanning, rows);
}

}  // namespace nz
