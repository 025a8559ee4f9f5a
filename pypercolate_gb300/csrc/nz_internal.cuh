// nz_internal.cuh -- kernel parameter blocks and launcher declarations shared
// between the translation units of libnzgb300.so (not part of the C ABI).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "nz_common.cuh"

namespace nz {

// Launches with `smem` bytes of dynamic shared memory.  How much a kernel may be
// given is a property of the kernel, for all host threads of the context alike: it
// is set to `most`, the most that any call gives it, and so never taken from under
// another thread's launch.  A failure is the returned status alone: it is not left
// as the context's last error, which the next call's checks, here or in the caller's
// program, would take for their own.
template <class... P, class... A>
cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, size_t most, cudaStream_t s,
                          A... args) {
    cudaError_t e = cudaSuccess;
    if (most > 40 * 1024)  // (with the static shared memory, beyond what is given unasked)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = grid;
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    }
    if (e != cudaSuccess) (void)cudaGetLastError();
    return e;
}

struct UfParams {
    GraphDev g;
    int32_t n_runs;
    uint32_t *nodes;        // [n_runs][g.slots]
    RunState *state;        // [n_runs]
    uint32_t n_begin;       // rows emitted: [n_begin, n_end)
    uint32_t n_end;
    uint64_t key, run0;     // NZ_PERM_PHILOX
    const uint32_t *perms;  // [n_runs][M] otherwise
    NzRecords rec;          // row n of run r at plane[(n - n_begin) * run_stride + r]
    uint32_t *errors;       // if set: +1 per run whose state is corrupt after its last row
    const uint32_t *init_flag;  // explicit edge lists: nonzero if a node touches both sides (or null)
    bool tiled;             // rec is tiled (tile_off in nz_records.cuh)
};

// nz_uf.cu
// explicit edge lists: UfParams::init_flag, in the caller's word (other graphs: null)
const uint32_t *launch_init_flag(const GraphDev &g, uint32_t *flag_scratch, cudaStream_t s);
cudaError_t launch_uf_window(const UfParams &p, int perm_mode, bool span, cudaStream_t s);
void launch_philox_perms(uint32_t M, int32_t n_runs, uint64_t key, uint64_t run0, uint32_t *out,
                         cudaStream_t s);
void launch_pack_rows(const NzRecords &rec, int32_t run, uint32_t N, uint32_t M, int32_t spanning,
                      uint8_t *rows, cudaStream_t s);

// nz_mt.cu: numpy's permutations
cudaError_t launch_mt_perms(uint32_t M, int32_t n_runs, const uint32_t *seed_words, const int32_t *seed_len,
                            int32_t stride, uint32_t *out, cudaStream_t s);
cudaError_t launch_mt_stream_perms(const uint32_t *state_in, uint32_t M, int32_t n_runs, uint32_t *out,
                                   uint32_t *state_out, cudaStream_t s);

// nz_ufg.cu: bond percolation with a thread block per run (which initialises
// the run in the window that begins at row 0)
cudaError_t launch_uf_groups(const UfParams &p, bool given, bool span, cudaStream_t s);

// nz_uft.cu: bonds and sites with a thread per run, and where that is the better one
bool run_per_thread(const UfParams &p);
cudaError_t launch_uf_threads(const UfParams &p, bool given, bool span, cudaStream_t s);

// nz_lattice.cu: a thread block per run for site percolation
cudaError_t launch_site_groups(const UfParams &p, bool given, bool span, cudaStream_t s);

// nz_canonical.cu
void launch_binomial_weights(uint32_t M, const double *ps, int32_t P, double cutoff, int32_t cap,
                             uint32_t *band_lo, uint32_t *band_len, double *w, int32_t *overflow,
                             cudaStream_t s);
void launch_binomial_pmf(uint32_t M, const double *ps, int32_t P, double cutoff, double *out, cudaStream_t s);
// out[i * cols + c] = sum over the band of p_i of w[i][j] V[(lo_i + j) * cols + c] (FP64)
void launch_band_dot(const uint32_t *band_lo, const uint32_t *band_len, const double *w, int32_t cap, int32_t P,
                     const double *V, uint32_t rows, int32_t cols, double *out, cudaStream_t s);
void launch_canonical_rows(const uint8_t *rows, uint32_t M, int32_t spanning, const double *factors,
                           int32_t n_sets, double *out, cudaStream_t s);

struct ConvParams {
    NzRecords rec;           // window records, row n at (n - n_begin)
    bool tiled;              // as UfParams::tiled
    uint32_t n_begin, n_end; // window rows
    uint32_t N;
    int32_t n_runs;
    int32_t spanning;
    int32_t P, cap;
    const uint32_t *band_lo, *band_len;  // rows of w64, or of w32 on the FP32 path
    const double *w64;       // [P][cap]
    const float *w32;        // [P][cap] (FP32 path, its own narrower bands)
    const float *w32lo;      // [P][cap] w64 - w32 as FP32 (the compensated m2 products)
    const uint32_t *core_lo, *core_len;  // rows whose weight is >= e^-8 of the mode (m2 compensated)
    double *acc;             // [n_runs][P][7], accumulated (+=)
    uint32_t *errors;        // tensor-core path: counts CTAs whose waits gave up (or null)
};
bool conv_grid_fits(int32_t n_runs, int32_t P);  // grid of launch_conv_window within CUDA's limits
cudaError_t launch_conv_window(const ConvParams &p, int precision, cudaStream_t s);
// 3xTF32 tensor-core convolution (tcgen05) of the FP32 bands; 0 or -1 (launch error)
bool conv_tc_grid_fits(int32_t n_runs, int32_t P);
int launch_conv_window_tc(const ConvParams &p, cudaStream_t s);
// FP32 weights of the rows where each band's weight is >= rel x its largest,
// re-based at lo32 (the convolution's FP32 band)
// (and their FP32 remainders w64 - w32 in w32lo), and the core rows whose
// weight is >= rel_core x the largest
void launch_narrow_weights_f32(const double *w64, const uint32_t *band_lo, const uint32_t *band_len, int32_t P,
                               int32_t cap, double rel, double rel_core, float *w32, float *w32lo, uint32_t *lo32,
                               uint32_t *len32, uint32_t *core_lo, uint32_t *core_len, cudaStream_t s);
// nz_conv_tiles.cu: the FP32 convolution of tiled records (all statistics, or m2 alone)
cudaError_t launch_conv_tiles(const ConvParams &p, cudaStream_t s);
cudaError_t launch_conv_tiles_m2(const ConvParams &p, cudaStream_t s);
// part: scratch [slices][P*7][3] doubles
void launch_reduce_runs(const double *stats, int32_t n_runs, int32_t P, uint64_t *acc_count,
                        double *acc_mean, double *acc_m2, double *part, int32_t slices, cudaStream_t s);

struct MicroParams {
    NzRecords rec;
    bool tiled;  // as UfParams::tiled
    void *part;  // tiled: micro_part_bytes() of scratch
    uint32_t n_begin, n_end;
    uint32_t N;
    int32_t n_runs;
    NzMicroAccum acc;
    uint32_t M;
    const uint64_t *count_before;  // device: runs already in acc
};
size_t micro_part_bytes();
void launch_micro_window(const MicroParams &p, cudaStream_t s);
void launch_micro_count(uint64_t *count, int32_t n_runs, cudaStream_t s);
void launch_canonical_merge(uint64_t *dst_count, double *dst_mean, double *dst_m2, const uint64_t *src_count,
                            const double *src_mean, const double *src_m2, int32_t cols, cudaStream_t s);
void launch_micro_merge(const NzMicroAccum &dst, const NzMicroAccum &src, uint32_t rows, cudaStream_t s);

void launch_init_avg(const uint8_t *canon_rows, int32_t P, int32_t spanning, uint8_t *out, cudaStream_t s);
void launch_bond_reduce(const uint8_t *a, const uint8_t *b, int32_t P, int32_t spanning, uint8_t *out,
                        cudaStream_t s);
void launch_finalize(const uint8_t *avg, int32_t P, int32_t spanning, double N, const double *ps,
                     double alpha, uint8_t *out, cudaStream_t s);
void launch_micro_finalize(const NzMicroAccum &acc, uint32_t N, uint32_t M, int32_t spanning, double alpha,
                           int32_t normalize, double *out, cudaStream_t s);
void launch_t_quantile(const double *q, const double *df, int32_t count, double *out, cudaStream_t s);

// nz_mix.cu (batched uneven ensembles)
struct MixDev {
    const uint64_t *key_ptr;
    int32_t n_runs;
    uint32_t chain_share;
    uint32_t grid_min, grid_max, chain_min, chain_max;
    uint32_t n_grid, n_chain;
    const uint32_t *thr_grid;
    const uint32_t *thr_chain;
    int32_t F;
};
struct MixRec {
    uint32_t *max_span;
    uint32_t *m0;
    uint64_t *m2, *m3, *m4_lo;
    uint32_t *m4_hi;
};
// Fused reduction: exact per-(class, checkpoint) sums that the union-find
// threads accumulate themselves, kMixCellWords uint64 words per cell, each
// the sum of one 32-bit limb of a statistic (or of its square) over the
// class's runs.
constexpr int kMixCellWords = 27;
struct MixAccum {
    uint32_t *count;
    uint32_t *span;
    uint64_t *sum_lo;
    uint64_t *sum_hi;
    double *m2;
    uint32_t *errors;
};
constexpr int kMixSegments = 5;  // parts of the queue by lattice size
struct MixLaunch {
    MixDev m;
    uint32_t *cls, *counts, *order, *offsets, *cursor, *queue;
    uint32_t *begin, *head;  // [kMixSegments + 1], [kMixSegments]
    uint32_t *nodes;         // [node_words]
    uint64_t node_words;
    uint64_t home_words;     // of the largest lattice
    bool fused;       // NZ_MIX_REDUCE_FUSED: cells, else records + mix_reduce_kernel
    MixRec rec;       // [n_runs][F] per plane (records only)
    uint64_t *cells;  // [classes][F][kMixCellWords] (fused only)
    MixAccum acc;
};
// node words in global memory that launch_mix uses, of at most T slots of home_words
uint64_t mix_node_words(uint64_t home_words, int32_t n_runs, int32_t T);
int launch_mix(const MixLaunch &p, cudaStream_t s);

}  // namespace nz
