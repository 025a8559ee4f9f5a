// nz_conv_tiles.cu -- FP32 convolution of tiled record windows.
//
// The products and sums of bond_canonical_statistics (percolate/hpc.py:443-515),
// C[run][p] += sum_n w[p][n] Q[n][run], for the records of an ensemble
// (nz_records.cuh, tiled), every sum in one order: rows upwards, in chunks of 128
// from the first row that a tile of 8 probabilities shares with the window.
//
// One CTA takes 128 runs (thread = run) and Q of the tile's 8 probabilities.  32 rows of the 128
// runs are one contiguous piece of a tiled plane, so one thread fetches them with
// one bulk copy per plane (cp.async.bulk), two pieces in flight, and the threads
// read their run's rows from shared memory in 16-byte loads without bank
// conflicts.  The weights of a chunk lie in shared memory as well; the next
// chunk's are loaded while this one is summed.  FP32 products go two to an
// instruction (fma.rn.f32x2, each half rounded like a single one).
//
// 4,000 runs at L = 97, 501 p: 0.39 ms for max, 0.19 for m0, 0.31 each for m3
// and m4, 0.86 for m2.  Reading the rows of one run straight from global memory,
// 16 bytes per thread and 128 bytes apart, kept the load pipe busy 80 % of the
// time and took 0.48, 2.0 (m0, m3 and m4) and 0.92 ms; 16 probabilities per CTA
// in two groups of threads 0.54, 0.27, 0.32 and 1.06.  What bounds it now (4,000 runs
// at L = 64, profiled): the issue slots, 78 % used by m2 (FMA pipe 49 %), 62 % by max
// (ALU pipe 51 %, FMA 25 %); 43 % by m3 and m4, of which three CTAs fit an SM.
#include <cstdint>
#include <type_traits>

#include "nz_common.cuh"
#include "nz_conv.cuh"
#include "nz_internal.cuh"
#include "nz_records.cuh"
#include "nz_tc.cuh"

namespace nz {
namespace {

constexpr int kRuns = 128;    // runs per CTA
constexpr int kPT = 8;        // probabilities per tile
constexpr int kRows = 32;     // rows per tile
constexpr int kWRows = kConvChunk + 8;  // weights staged: a chunk, from the 8-row group of its first row

// S: 1 the max_span plane (statistics 0, 1 and 3), 2 / 8 m0 (uint32 / uint16),
// 4 / 9 m2 (uint64 / uint32), 5 m3, 6 / 7 m4 with / without its high words
template <int S>
using raw_t = typename std::conditional<
    S == 8, uint16_t, typename std::conditional<S == 1 || S == 2 || S == 9, uint32_t, uint64_t>::type>::type;

template <int S>
__device__ __forceinline__ const raw_t<S> *plane_of(const NzRecords &rec) {
    if constexpr (S == 1) return rec.max_span;
    else if constexpr (S == 2) return rec.m0;
    else if constexpr (S == 8) return reinterpret_cast<const uint16_t *>(rec.m0);
    else if constexpr (S == 4) return rec.m2;
    else if constexpr (S == 9) return reinterpret_cast<const uint32_t *>(rec.m2);
    else if constexpr (S == 5) return rec.m3;
    else return rec.m4_lo;
}

template <int S, int Q>
struct TileShared {
    static constexpr bool kM2 = S == 4 || S == 9;
    raw_t<S> q[2][kRuns * kRows];
    uint32_t hi[S == 6 ? 2 : 1][S == 6 ? kRuns * kRows : 4];
    float w[kM2 ? 2 : 1][kWRows][Q];  // [hi, lo]
    uint64_t full[2];
    uint32_t lo[kPT], len[kPT], clo[kPT], clen[kPT];
    uint32_t range[4];  // window rows of the CTA; of the tile's probabilities
};

__device__ __forceinline__ uint64_t pair(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair(uint64_t v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t w, uint64_t q) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w), "l"(q));
}

// rows i .. i + N - 1 of this thread's run in a staged tile
template <int N, class T>
__device__ __forceinline__ void read_rows(const T *tile, int run, int i, T (&q)[N]) {
    constexpr int kPer = 16 / (int)sizeof(T);
#pragma unroll
    for (int k = 0; k < N; k += kPer) {
        const uint4 v = *reinterpret_cast<const uint4 *>(tile + tile_off<sizeof(T)>(0, i + k, run & 7) +
                                                         (run & ~7) * kRows);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int b = 0; b < kPer; ++b) {
            if constexpr (sizeof(T) == 2) q[k + b] = (T)(w[b / 2] >> (16 * (b & 1)));
            else if constexpr (sizeof(T) == 4) q[k + b] = (T)w[b];
            else q[k + b] = (T)(((uint64_t)w[2 * b + 1] << 32) | w[2 * b]);
        }
    }
}

// CTAs per SM that the registers are cut for: 4 for max (72 accumulators), 5 for
// m0 and m2, 3 for m3 and m4 (their 64 KB of stages)
template <int S>
constexpr int kPerSm = S == 1 ? 4 : sizeof(raw_t<S>) == 8 ? 3 : 5;

// SITE (S = 1 only): records of site percolation, m1 = n - max instead of N - max
template <int S, int Q, bool SITE>
__global__ void __launch_bounds__(kRuns, kPerSm<S>) conv_tiles_kernel(ConvParams p) {
    constexpr bool kMax = S == 1, kM2 = TileShared<S, Q>::kM2;
    // rows in straight-line code: more of m2's would not fit the instruction cache
    constexpr int kStep = kM2 ? 4 : 8;
    constexpr int kSets = kMax ? 3 : 1, kOut = S == 8 ? 2 : S == 9 ? 4 : S == 7 ? 6 : S;
    extern __shared__ __align__(128) uint8_t smem[];
    TileShared<S, Q> &sh = *reinterpret_cast<TileShared<S, Q> *>(smem);
    constexpr int kWPer = (kWRows * Q + kRuns - 1) / kRuns;
    // the tile's first probability, and which of its kPT are this CTA's
    const int run = threadIdx.x, r = blockIdx.x * kRuns + run, p0 = (int)blockIdx.y / (kPT / Q) * kPT;
    const int q0 = Q == kPT ? 0 : (int)blockIdx.y % (kPT / Q) * Q;
    if (run < kPT) {
        const bool in = p0 + run < p.P;
        sh.lo[run] = in ? p.band_lo[p0 + run] : 0u;
        sh.len[run] = in ? p.band_len[p0 + run] : 0u;
        sh.clo[run] = in && kM2 ? p.core_lo[p0 + run] : 0u;
        sh.clen[run] = in && kM2 ? p.core_len[p0 + run] : 0u;
    }
    if (threadIdx.x == 0) {
        tc::mbar_init(tc::smem_u32(&sh.full[0]));
        tc::mbar_init(tc::smem_u32(&sh.full[1]));
        tc::mbar_init_fence();
    }
    __syncthreads();
    if (run < 2) {  // the CTA's probabilities; all of the tile's
        uint32_t lo = 0xffffffffu, hi = 0;
        for (int j = run == 0 ? q0 : 0; j < (run == 0 ? q0 + Q : kPT); ++j)
            if (sh.len[j]) {
                lo = min(lo, sh.lo[j]);
                hi = max(hi, sh.lo[j] + sh.len[j]);
            }
        lo = max(lo, p.n_begin);
        hi = min(hi, p.n_end);
        sh.range[2 * run] = lo < hi ? lo - p.n_begin : 0u;
        sh.range[2 * run + 1] = lo < hi ? hi - p.n_begin : 0u;
    }
    __syncthreads();
    const uint32_t a = sh.range[0], b = sh.range[1];  // window rows
    if (a >= b) return;
    // chunks are counted from the tile's first row, whichever probabilities are
    // the CTA's, so that their sums do not depend on Q
    const uint32_t a8 = Q == kPT ? a : sh.range[2], b8 = Q == kPT ? b : sh.range[3];
    const uint32_t tile0 = a / kRows, tiles = (b + kRows - 1) / kRows - tile0;
    const int runs = min(kRuns, p.n_runs - (int)blockIdx.x * kRuns);
    auto fetch = [&](uint32_t k) {  // one thread: tile tile0 + k into stage k % 2
        const uint32_t bar = tc::smem_u32(&sh.full[k & 1]);
        const uint32_t bytes = (uint32_t)runs * kRows * (uint32_t)sizeof(raw_t<S>);
        const size_t line = ((size_t)(tile0 + k) * p.rec.run_stride + (size_t)blockIdx.x * kRuns) * kRows;
        tc::expect_bytes(bar, bytes + (S == 6 ? (uint32_t)runs * kRows * 4u : 0u));
        tc::bulk_load(tc::smem_u32(sh.q[k & 1]), plane_of<S>(p.rec) + line, bytes, bar);
        if constexpr (S == 6)
            tc::bulk_load(tc::smem_u32(sh.hi[k & 1]), p.rec.m4_hi + line, (uint32_t)runs * kRows * 4u, bar);
    };
    if (threadIdx.x == 0) {
        fetch(0);
        if (tiles > 1) fetch(1);
    }

    // the chunk [ca, cb) of the rows
    uint32_t ca = a8 + (a - a8) / kConvChunk * kConvChunk, cb = min(ca + (uint32_t)kConvChunk, b8);
    // weights of the chunk that begins at row c, zero outside it
    float wreg[kWPer], wreg_lo[kM2 ? kWPer : 1];
    auto load_weights = [&](uint32_t c) {
        const uint32_t base = c & ~7u, end = min(c + (uint32_t)kConvChunk, b);
#pragma unroll
        for (int q = 0; q < kWPer; ++q) {
            const int i = run + q * kRuns, j = i / kWRows;
            const uint32_t row = base + (uint32_t)(i % kWRows), n = p.n_begin + row;
            float v = 0.0f, vl = 0.0f;
            if (j < Q && row >= c && row < end && n >= sh.lo[q0 + j] && n < sh.lo[q0 + j] + sh.len[q0 + j]) {
                const size_t at = (size_t)(p0 + q0 + j) * p.cap + (n - sh.lo[q0 + j]);
                v = p.w32[at];
                if (kM2) vl = p.w32lo[at];
            }
            wreg[q] = v;
            if (kM2) wreg_lo[q] = vl;
        }
    };
    auto store_weights = [&]() {
#pragma unroll
        for (int q = 0; q < kWPer; ++q) {
            const int i = run + q * kRuns, j = i / kWRows, row = i % kWRows;
            if (j < Q) {
                sh.w[0][row][j] = wreg[q];
                if (kM2) sh.w[kM2 ? 1 : 0][row][j] = wreg_lo[q];
            }
        }
    };
    // does the chunk meet a core?  (uniform over the CTA; m2 only)
    auto meets_core = [&]() {
        bool core = false;
#pragma unroll
        for (int j = 0; j < kPT; ++j) {
            const uint32_t lo = sh.clo[j], len = sh.clen[j];
            core |= len && lo < p.n_begin + cb && p.n_begin + ca < lo + len;
        }
        return core;
    };
    load_weights(ca);
    store_weights();
    __syncthreads();
    if (cb < b) load_weights(cb);
    bool core = kM2 && meets_core();

    ConvAcc acc[kM2 ? 1 : kSets][kM2 ? 1 : Q];
    uint64_t part[kM2 ? 1 : kSets][kM2 ? 1 : Q / 2];
    Dot2Acc dot[kM2 ? Q : 1];
    auto clear = [&]() {
        if constexpr (!kM2) {
#pragma unroll
            for (int s = 0; s < kSets; ++s)
#pragma unroll
                for (int j = 0; j < Q / 2; ++j) part[s][j] = 0;
        }
    };
    auto flush = [&]() {
        if constexpr (kM2) {
            if (!core) {
#pragma unroll
                for (int j = 0; j < Q; ++j) dot[j].flush_tail();
            }
        } else {
#pragma unroll
            for (int s = 0; s < kSets; ++s)
#pragma unroll
                for (int j = 0; j < Q / 2; ++j) {
                    float x, y;
                    unpair(part[s][j], x, y);
                    acc[s][2 * j].add(x);
                    acc[s][2 * j + 1].add(y);
                }
        }
        clear();
    };
    clear();

    bool bad = false;
    for (uint32_t k = 0; k < tiles; ++k) {
        // every thread is done with tile k - 1, whose stage takes tile k + 1
        bad = __syncthreads_or(!tc::mbar_wait(tc::smem_u32(&sh.full[k & 1]), (k >> 1) & 1));
        if (bad) {
            // (the one other copy that can be in flight lands first)
            if (k == 0 && tiles > 1) tc::mbar_wait(tc::smem_u32(&sh.full[1]), 0);
            break;
        }
        if (threadIdx.x == 0 && k > 0 && k + 1 < tiles) fetch(k + 1);
        const raw_t<S> *tile = sh.q[k & 1];
        for (int g = 0; g < kRows / 8; ++g) {
            const uint32_t row = (tile0 + k) * kRows + 8u * g;
            if (row + 8u <= a || row >= b) continue;
            // once for every chunk that has rows among these 8
            for (;;) {
                const int w0 = (int)(row - (ca & ~7u));
#pragma unroll 1
                for (int i0 = 0; i0 < 8; i0 += kStep) {
                    raw_t<S> q[kStep];
                    uint32_t hi[S == 6 ? kStep : 1];
                    read_rows<kStep>(tile, run, 8 * g + i0, q);
                    if constexpr (S == 6) read_rows<kStep>(sh.hi[k & 1], run, 8 * g + i0, hi);
#pragma unroll
                    for (int i = 0; i < kStep; ++i) {
                        const float *w = sh.w[0][w0 + i0 + i];
                        if constexpr (kM2) {
                            float qh, ql;
                            if constexpr (S == 9) split_u32(q[i], qh, ql);
                            else split_u64(q[i], qh, ql);
                            if (core) {
                                const float *wl = sh.w[1][w0 + i0 + i];
#pragma unroll
                                for (int j = 0; j < Q; ++j) dot[j].add(w[j], wl[j], qh, ql);
                            } else {
                                const float v = __fadd_rn(qh, ql);
#pragma unroll
                                for (int j = 0; j < Q; ++j) dot[j].add_tail(w[j], v);
                            }
                        } else {
                            uint64_t ww[Q / 2];
                            if constexpr (Q == 2) {
                                ww[0] = *reinterpret_cast<const uint64_t *>(w);
                            } else {
#pragma unroll
                                for (int j = 0; j < Q / 4; ++j) {
                                    const ulonglong2 two = reinterpret_cast<const ulonglong2 *>(w)[j];
                                    ww[2 * j] = two.x;
                                    ww[2 * j + 1] = two.y;
                                }
                            }
                            auto products = [&](int s, float v) {
                                const uint64_t vv = pair(v, v);
#pragma unroll
                                for (int j = 0; j < Q / 2; ++j) fma2(part[s][j], ww[j], vv);
                            };
                            if constexpr (kMax) {
                                const uint32_t mx = q[i] & ~kSpanBit;
                                products(0, (q[i] & kSpanBit) ? 1.0f : 0.0f);
                                products(1, (float)mx);
                                products(2, (float)((SITE ? p.n_begin + row + (uint32_t)(i0 + i) : p.N) - mx));
                            } else if constexpr (S == 6) {
                                products(0, fmaf((float)hi[i], 18446744073709551616.0f, u64_to_f32(q[i])));
                            } else if constexpr (sizeof(raw_t<S>) == 8) {
                                products(0, u64_to_f32(q[i]));
                            } else {
                                products(0, (float)q[i]);
                            }
                        }
                    }
                }
                if (cb > row + 8u || cb >= b) break;
                // the chunk ends among (or with) these rows
                flush();
                const bool again = cb < row + 8u;
                __syncthreads();
                store_weights();
                ca = cb;
                cb = min(ca + (uint32_t)kConvChunk, b8);
                __syncthreads();
                if (cb < b) load_weights(cb);
                if (kM2) core = meets_core();
                if (!again) break;
            }
        }
    }
    if (bad) {  // a copy did not arrive (the same for every thread)
        if (threadIdx.x == 0 && p.errors) atomicAdd(p.errors, 1u);
        return;
    }
    flush();
    if (r < p.n_runs) {
#pragma unroll
        for (int j = 0; j < Q; ++j) {
            if (p0 + q0 + j >= p.P) continue;
            double *o = p.acc + ((size_t)r * p.P + p0 + q0 + j) * 7;
            if constexpr (kM2) {
                o[4] += dot[j].value();
            } else if constexpr (kMax) {
                if (p.spanning) o[0] += acc[0][j].value();
                o[1] += acc[1][j].value();
                o[3] += acc[2][j].value();
            } else {
                o[kOut] += acc[0][j].value();
            }
        }
    }
}

template <int S, int Q, bool SITE>
cudaError_t launch_q(const ConvParams &p, cudaStream_t s) {
    dim3 grid((p.n_runs + kRuns - 1) / kRuns, (p.P + kPT - 1) / kPT * (kPT / Q));
    constexpr size_t kSmem = sizeof(TileShared<S, Q>);
    return launch_kernel(conv_tiles_kernel<S, Q, SITE>, grid, kRuns, kSmem, kSmem, s, p);
}

// Probabilities per CTA.  Fewer make more CTAs, whose rows are fewer where the
// bands lie apart, but load the records more often: 2 where a tile of 8 each
// would leave SMs idle (1,000 runs of 300 x 300 at 50 p, 56 tiles: 9.8 ms with
// 8, 4.1 with 4, 2.2 with 2), else 4 for max and m0 (11,000 us of all kernels at
// L = 256 are 250 less), for m2 up to 8 tiles per SM (2,000 runs of 200 x 200 at
// 301 p, 608 tiles: 911 us with 8, 755 with 4; 4,000 of 97 x 97, 2,016 tiles:
// 853 and 891), and for m3 and m4 up to 2 (1,000 of 64 x 64, 304 tiles: 44 and
// 45; 1,000 of 32 x 32, 208 tiles: 22 and 18).
template <int S, bool SITE = false>
cudaError_t launch(const ConvParams &p, cudaStream_t s) {
    constexpr bool kWide = S == 5 || S == 6 || S == 7;
    const int64_t p_tiles = (p.P + kPT - 1) / kPT, tiles = (int64_t)((p.n_runs + kRuns - 1) / kRuns) * p_tiles;
    if (tiles < 152) return launch_q<S, 2, SITE>(p, s);
    // (the grid's y, of p_tiles kPT / Q, has 16 bits: conv_grid_fits admits kPT
    // to a block)
    if (p_tiles * (kPT / 4) > 65535) return launch_q<S, kPT, SITE>(p, s);
    if constexpr (kWide || TileShared<S, kPT>::kM2) {
        if (tiles >= (kWide ? 2 : 8) * 152) return launch_q<S, kPT, SITE>(p, s);
    }
    return launch_q<S, 4, SITE>(p, s);
}

}  // namespace

cudaError_t launch_conv_tiles_m2(const ConvParams &p, cudaStream_t s) {
    return p.rec.narrow ? launch<9>(p, s) : launch<4>(p, s);
}

cudaError_t launch_conv_tiles(const ConvParams &p, cudaStream_t s) {
    cudaError_t e = p.rec.site ? launch<1, true>(p, s) : launch<1>(p, s);
    if (e == cudaSuccess) e = p.rec.narrow ? launch<8>(p, s) : launch<2>(p, s);
    if (e == cudaSuccess) e = launch<5>(p, s);
    if (e == cudaSuccess) e = p.rec.m4_hi ? launch<6>(p, s) : launch<7>(p, s);
    return e == cudaSuccess ? launch_conv_tiles_m2(p, s) : e;
}

}  // namespace nz
