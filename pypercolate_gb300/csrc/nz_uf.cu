// nz_uf.cu -- permutations, reference rows and the union-find's dispatch.
//
// Bond percolation (percolate/hpc.py:249-307, bond_sample_states) is launched by
// nz_ufg.cu, site percolation by nz_lattice.cu, very many runs by nz_uft.cu; all
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
const uint32_t *launch_init_flag(const GraphDev &g, uint32_t *flag_scratch, cudaStream_t s) {
    if (g.kind != NZ_GRAPH_EDGES) return nullptr;
    cudaMemsetAsync(flag_scratch, 0, sizeof(uint32_t), s);
    any_both_sides_kernel<<<(g.N + 255) / 256 < 1024 ? (g.N + 255) / 256 : 1024, 256, 0, s>>>(g, flag_scratch);
    return flag_scratch;
}

cudaError_t launch_uf_window(const UfParams &p, int perm_mode, bool span, cudaStream_t s) {
    const bool given = perm_mode != NZ_PERM_PHILOX;
    if (run_per_thread(p)) return launch_uf_threads(p, given, span, s);
    return p.g.site ? launch_site_groups(p, given, span, s) : launch_uf_groups(p, given, span, s);
}

void launch_philox_perms(uint32_t M, int32_t n_runs, uint64_t key, uint64_t run0, uint32_t *out,
                         cudaStream_t s) {
    uint64_t total = (uint64_t)n_runs * M;
    uint64_t blocks = (total + 255) / 256;
    if (blocks > 152ull * 64) blocks = 152ull * 64;
    if (blocks == 0) return;
    philox_perm_kernel<<<(unsigned)blocks, 256, 0, s>>>(M, n_runs, key, run0, out);
}

void launch_pack_rows(const NzRecords &rec, int32_t run, uint32_t N, uint32_t M, int32_t spanning,
                      uint8_t *rows, cudaStream_t s) {
    uint32_t blocks = (M + 1 + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    pack_rows_kernel<<<blocks, 256, 0, s>>>(rec, run, N, M, spanning, rows);
}

}  // namespace nz
