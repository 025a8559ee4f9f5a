// nz_canonical.cu -- canonical (binomial-convolution) stage, averages and
// confidence intervals.
//
// Replaces percolate/percolate.py:1067-1109 (_binomial_pmf),
// percolate/hpc.py:443-515 (bond_canonical_statistics), :561-635
// (bond_initialize_canonical_averages), :638-702 (bond_reduce) and :752-834
// (finalize_canonical_averages), plus the microcanonical run-reductions whose
// semantics are percolate/percolate.py:450-705.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "nz_common.cuh"
#include "nz_conv.cuh"
#include "nz_internal.cuh"
#include "nz_math.cuh"
#include "nz_records.cuh"
#include "nz_wide.cuh"

namespace nz {

// =====================================================================
// Binomial weights
// =====================================================================
// Log B(M, n, p) up to an n-independent constant, from lgamma; used only to
// locate the band edges (its absolute error does not reach the weights).
__device__ __forceinline__ double log_binom_shape(uint32_t M, uint32_t n, double lp, double lq) {
    return -lgamma((double)n + 1.0) - lgamma((double)(M - n) + 1.0) + (double)n * lp + (double)(M - n) * lq;
}

// One CTA per p.  Band = {n : log B(n) >= log B(mode) - cutoff}, found by
// bisection on each side of the mode (log B is concave in n).  The weights
// are then built from the ratio recursion of Newman & Ziff Eq. (10),
//   log B(n) - log B(n-1) = log(M - n + 1) - log(n) + log(p) - log(1 - p),
// summed by a block-wide prefix scan from the band's low edge, shifted by the
// maximum, exponentiated and normalised by their FP64 sum (as the reference
// normalises by ret.sum()).  Writes wp[0, cap) and returns (lo, len) to all
// threads of the block.
template <int BLOCK>
__device__ void band_weights_block(uint32_t M, double p, double cutoff, int32_t cap, double *wp, uint32_t &lo_out,
                                   uint32_t &len_out, bool &overflow) {
    __shared__ double s_scan[2][BLOCK];
    __shared__ double s_red[BLOCK];
    __shared__ uint32_t s_lo, s_hi;
    if (threadIdx.x == 0) {
        uint32_t lo, hi;
        if (!(p > 0.0)) { lo = hi = 0; }
        else if (!(p < 1.0)) { lo = hi = M; }
        else {
            const double lp = log(p), lq = log1p(-p);
            uint32_t mode = (uint32_t)floor((double)(M + 1) * p);
            if (mode > M) mode = M;
            const double lm = log_binom_shape(M, mode, lp, lq) - cutoff;
            // smallest n <= mode with shape(n) >= lm
            uint32_t a = 0, b = mode;
            if (log_binom_shape(M, 0, lp, lq) >= lm) b = 0;
            else while (b - a > 1) { uint32_t c = a + (b - a) / 2; if (log_binom_shape(M, c, lp, lq) >= lm) b = c; else a = c; }
            lo = b;
            // largest n >= mode with shape(n) >= lm
            a = mode; b = M;
            if (log_binom_shape(M, M, lp, lq) >= lm) a = M;
            else while (b - a > 1) { uint32_t c = a + (b - a) / 2; if (log_binom_shape(M, c, lp, lq) >= lm) a = c; else b = c; }
            hi = a;
        }
        s_lo = lo; s_hi = hi;
    }
    __syncthreads();
    const uint32_t lo = s_lo;
    uint32_t len = s_hi - s_lo + 1;
    overflow = len > (uint32_t)cap;
    if (overflow) len = cap;
    lo_out = lo;
    len_out = len;
    if (len == 1) {
        for (int j = threadIdx.x; j < cap; j += BLOCK) wp[j] = (j == 0) ? 1.0 : 0.0;
        __syncthreads();
        return;
    }
    const double lpq = log(p) - log1p(-p);
    // pass 1: log weights relative to the low edge (prefix scan of log ratios, in
    // two buffers by turns: a barrier a step)
    double carry = 0.0;
    double vmax = -INFINITY;
    int buf = 0;
    for (uint32_t base = 0; base < len; base += BLOCK) {
        const uint32_t j = base + threadIdx.x;
        double x = 0.0;
        if (j > 0 && j < len) {
            const double n = (double)(lo + j);
            x = log((double)M - n + 1.0) - log(n) + lpq;
        }
        for (int off = 1; off < BLOCK; off <<= 1) {  // Hillis-Steele inclusive scan
            s_scan[buf][threadIdx.x] = x;
            __syncthreads();
            if (threadIdx.x >= (unsigned)off) x += s_scan[buf][threadIdx.x - off];
            buf ^= 1;
        }
        s_scan[buf][threadIdx.x] = x;
        __syncthreads();
        const double lv = carry + x;
        if (j < len) { wp[j] = lv; vmax = fmax(vmax, lv); }
        carry += s_scan[buf][BLOCK - 1];
        buf ^= 1;
    }
    s_red[threadIdx.x] = vmax;
    __syncthreads();
    for (int off = BLOCK / 2; off > 0; off >>= 1) {
        if (threadIdx.x < (unsigned)off) s_red[threadIdx.x] = fmax(s_red[threadIdx.x], s_red[threadIdx.x + off]);
        __syncthreads();
    }
    vmax = s_red[0];
    __syncthreads();
    // pass 2: exponentiate and sum
    double sum = 0.0;
    for (uint32_t j = threadIdx.x; j < len; j += BLOCK) {
        const double e = exp(wp[j] - vmax);
        wp[j] = e;
        sum += e;
    }
    s_red[threadIdx.x] = sum;
    __syncthreads();
    for (int off = BLOCK / 2; off > 0; off >>= 1) {
        if (threadIdx.x < (unsigned)off) s_red[threadIdx.x] += s_red[threadIdx.x + off];
        __syncthreads();
    }
    const double inv = 1.0 / s_red[0];
    for (uint32_t j = threadIdx.x; j < (uint32_t)cap; j += BLOCK) wp[j] = (j < len) ? wp[j] * inv : 0.0;
    __syncthreads();
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) binomial_weights_kernel(uint32_t M, const double *ps, double cutoff,
                                                                 int32_t cap, uint32_t *band_lo,
                                                                 uint32_t *band_len, double *w,
                                                                 int32_t *overflow) {
    const int pi = blockIdx.x;
    uint32_t lo, len;
    bool ovf;
    band_weights_block<BLOCK>(M, ps[pi], cutoff, cap, w + (size_t)pi * cap, lo, len, ovf);
    if (threadIdx.x == 0) {
        band_lo[pi] = lo;
        band_len[pi] = len;
        if (ovf && overflow) atomicExch(overflow, 1);
    }
}

// Full-length pmf rows out[pi][0..M]: band weights computed at the row start,
// then shifted in place to their offset and the rest zeroed.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) binomial_pmf_kernel(uint32_t M, const double *ps, double cutoff,
                                                             double *out) {
    const int pi = blockIdx.x;
    double *row = out + (size_t)pi * (M + 1);
    uint32_t lo, len;
    bool ovf;
    band_weights_block<BLOCK>(M, ps[pi], cutoff, (int32_t)(M + 1), row, lo, len, ovf);
    if (lo > 0) {
        // move [0, len) to [lo, lo + len), highest block first
        for (int64_t top = (int64_t)len; top > 0; top -= BLOCK) {
            const int64_t j = top - BLOCK + threadIdx.x;
            double v = 0.0;
            if (j >= 0) v = row[j];
            __syncthreads();
            if (j >= 0) row[j + lo] = v;
            __syncthreads();
        }
        for (uint32_t j = threadIdx.x; j < lo; j += BLOCK) row[j] = 0.0;
    }
}

void launch_binomial_weights(uint32_t M, const double *ps, int32_t P, double cutoff, int32_t cap,
                             uint32_t *band_lo, uint32_t *band_len, double *w, int32_t *overflow,
                             cudaStream_t s) {
    if (P <= 0) return;
    binomial_weights_kernel<256><<<P, 256, 0, s>>>(M, ps, cutoff, cap, band_lo, band_len, w, overflow);
}

void launch_binomial_pmf(uint32_t M, const double *ps, int32_t P, double cutoff, double *out, cudaStream_t s) {
    if (P <= 0) return;
    binomial_pmf_kernel<256><<<P, 256, 0, s>>>(M, ps, cutoff, out);
}

// =====================================================================
// bond_canonical_statistics on the reference's packed rows (FP64)
// =====================================================================
__device__ __forceinline__ uint64_t ld_bytes(const uint8_t *p, int n) {
    uint64_t v = 0;
    for (int i = 0; i < n; ++i) v |= (uint64_t)p[i] << (8 * i);
    return v;
}

// grid: (factor set); each CTA reduces over the M+1 rows.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) canonical_rows_kernel(const uint8_t *rows, uint32_t M, int32_t spanning,
                                                               const double *factors, double *out) {
    const int set = blockIdx.x;
    const double *f = factors + (size_t)set * (M + 1);
    const uint32_t rb = spanning ? 53u : 52u;
    const int o = spanning ? 9 : 8;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    for (uint32_t n = threadIdx.x; n <= M; n += BLOCK) {
        const uint8_t *r = rows + (size_t)n * rb;
        const double fn = f[n];
        if (spanning) acc[0] += fn * (double)(r[8] != 0);
        acc[1] += fn * (double)(uint32_t)ld_bytes(r + o, 4);
#pragma unroll
        for (int k = 0; k < 5; ++k) acc[2 + k] += fn * (double)ld_bytes(r + o + 4 + 8 * k, 8);
    }
    __shared__ double s_red[7][BLOCK];
#pragma unroll
    for (int k = 0; k < 7; ++k) s_red[k][threadIdx.x] = acc[k];
    __syncthreads();
    for (int off = BLOCK / 2; off > 0; off >>= 1) {
        if (threadIdx.x < (unsigned)off)
#pragma unroll
            for (int k = 0; k < 7; ++k) s_red[k][threadIdx.x] += s_red[k][threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x < 7) out[(size_t)set * 7 + threadIdx.x] = (threadIdx.x == 0 && !spanning) ? 0.0 : s_red[threadIdx.x][0];
}

void launch_canonical_rows(const uint8_t *rows, uint32_t M, int32_t spanning, const double *factors,
                           int32_t n_sets, double *out, cudaStream_t s) {
    if (n_sets <= 0) return;
    canonical_rows_kernel<256><<<n_sets, 256, 0, s>>>(rows, M, spanning, factors, out);
}

// =====================================================================
// Classic canonical averages: binomial weights times microcanonical arrays
// =====================================================================
// out[i][c] = sum_j w[i][j] V[lo_i + j][c] for the band of p_i (FP64): the
// sums percolate/percolate.py:1171-1221 (canonical_averages) forms with the
// full-length pmf, over the rows where the pmf does not underflow.  One CTA
// per (p, group of 32 columns): lane c of every warp owns column c (a row
// of V is one coalesced load per warp), warps stride over the band's rows,
// and the warps' partial sums are added in a fixed order (deterministic).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) band_dot_kernel(const uint32_t *band_lo, const uint32_t *band_len,
                                                         const double *w, int32_t cap, const double *V,
                                                         uint32_t rows, int32_t cols, double *out) {
    __shared__ double part[BLOCK / 32][32];
    const int pi = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = blockIdx.y * 32 + lane;
    const uint32_t lo = band_lo[pi];
    uint32_t len = min(band_len[pi], (uint32_t)cap);
    if (lo >= rows) len = 0;
    else len = min(len, rows - lo);
    const double *wp = w + (size_t)pi * cap;
    double acc = 0.0;
    if (c < cols)
        for (uint32_t j = warp; j < len; j += BLOCK / 32) acc = fma(wp[j], V[(size_t)(lo + j) * cols + c], acc);
    part[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && c < cols) {
        double t = 0.0;
        for (int k = 0; k < BLOCK / 32; ++k) t += part[k][lane];
        out[(size_t)pi * cols + c] = t;
    }
}

void launch_band_dot(const uint32_t *band_lo, const uint32_t *band_len, const double *w, int32_t cap, int32_t P,
                     const double *V, uint32_t rows, int32_t cols, double *out, cudaStream_t s) {
    if (P <= 0 || cols <= 0) return;
    dim3 g(P, (cols + 31) / 32);
    band_dot_kernel<256><<<g, 256, 0, s>>>(band_lo, band_len, w, cap, V, rows, cols, out);
}

// =====================================================================
// Banded convolution of record windows (ensemble path)
// =====================================================================
// FP64 (the FP32 convolution of an ensemble's tiled records: nz_conv_tiles.cu)
constexpr int kConvRuns = 128;  // runs per CTA (one per thread)
constexpr int kConvPT = 8;      // most probabilities per CTA
constexpr int kConvBatch = 16;  // record loads in flight per thread

// grid: (run tiles, p tiles, 7 statistics).  Each thread accumulates the
// PT canonical values of its run for one statistic over the window's
// rows, with the tile's weights staged in shared memory (zero outside each
// p's band), with FP64 products and sums.
template <int S, bool SITE, int PT>
__device__ __forceinline__ void conv_rows(const ConvParams &p, uint32_t c0, uint32_t cn, int r,
                                          const double (*s_w)[PT],
                                          double *acc) {
    double part[PT];
#pragma unroll
    for (int j = 0; j < PT; ++j) part[j] = 0;
    const size_t base = (size_t)(c0 - p.n_begin) * p.rec.run_stride + r;
    // m1 = (sites in clusters) - max: N for bond records, n for site records
    auto value = [&](uint32_t i) -> double {
        const size_t off = base + (size_t)i * p.rec.run_stride;
        const uint32_t held = (S == 3 && SITE) ? c0 + i : p.N;
        return (double)record_value<S>(p.rec, off, held);
    };
    // the records of kConvBatch rows are loaded before their products so that
    // that many loads are in flight per thread; each accumulator still adds
    // the rows in increasing order
    uint32_t i = 0;
    for (; i + kConvBatch <= cn; i += kConvBatch) {
        double q[kConvBatch];
#pragma unroll
        for (int b = 0; b < kConvBatch; ++b) q[b] = value(i + b);
#pragma unroll
        for (int b = 0; b < kConvBatch; ++b)
#pragma unroll
            for (int j = 0; j < PT; ++j) part[j] = fma(s_w[i + b][j], q[b], part[j]);
    }
    for (; i < cn; ++i) {
        const double q = value(i);
#pragma unroll
        for (int j = 0; j < PT; ++j) part[j] = fma(s_w[i][j], q, part[j]);
    }
#pragma unroll
    for (int j = 0; j < PT; ++j) acc[j] += part[j];
}

// Statistics 0 (spanning), 1 (max) and 3 (m1 = held - max) all come from the
// max_span plane: one pass loads each word once and feeds the three sets of
// products (each accumulator adds the same values in the same order as a
// pass per statistic would).
template <bool SITE, int PT>
__device__ __forceinline__ void conv_rows_max(const ConvParams &p, uint32_t c0, uint32_t cn, int r,
                                              const double (*s_w)[PT],
                                              double *acc0, double *acc1,
                                              double *acc3) {
    double p0[PT], p1[PT], p3[PT];
#pragma unroll
    for (int j = 0; j < PT; ++j) p0[j] = p1[j] = p3[j] = 0;
    const size_t base = (size_t)(c0 - p.n_begin) * p.rec.run_stride + r;
    auto step = [&](uint32_t i, uint32_t ms) {
        const uint32_t held = SITE ? c0 + i : p.N;
        const uint32_t mx = ms & ~kSpanBit;
        const double q0 = (ms & kSpanBit) ? (double)1 : (double)0;
        const double q1 = (double)mx, q3 = (double)(held - mx);
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const double w = s_w[i][j];
            p0[j] = fma(w, q0, p0[j]);  // (dropped at the end without a spanning statistic)
            p1[j] = fma(w, q1, p1[j]);
            p3[j] = fma(w, q3, p3[j]);
        }
    };
    uint32_t i = 0;
    for (; i + kConvBatch <= cn; i += kConvBatch) {
        uint32_t ms[kConvBatch];
#pragma unroll
        for (int b = 0; b < kConvBatch; ++b) ms[b] = p.rec.max_span[base + (size_t)(i + b) * p.rec.run_stride];
#pragma unroll
        for (int b = 0; b < kConvBatch; ++b) step(i + b, ms[b]);
    }
    for (; i < cn; ++i) step(i, p.rec.max_span[base + (size_t)i * p.rec.run_stride]);
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        acc0[j] += p0[j];
        acc1[j] += p1[j];
        acc3[j] += p3[j];
    }
}

// ---- the same sums over tiled records.  A chunk's rows are read in groups of
// 8 (16-byte loads of one run's consecutive rows) from the group that holds its
// first row; s_w row 0 is that group's first row and rows outside the chunk have
// zero weights, which leave every partial sum as it is.  Rows are added in
// increasing order, chunk by chunk, as above.
//
// What bounds it: the FP64 pipe (two results per clock and SM).  So products
// that are zero are left out where a whole group's are: of a probability whose
// band does not meet the group (a sixth to a third of a tile of 8), and of the
// spanning flag where no row has it.  Ensembles of 2,000 chains of 6,000, 201 p,
// 6.93 -> 5.28 ms; 1,000 grids of 128 x 128 12.4 -> 8.7.  One group ahead: three
// took 255 registers and 18 % more time, none 2 % more.
template <int S>
using tile_raw = typename std::conditional<S == 8, uint16_t,
                                           typename std::conditional<S == 4 || S == 5 || S == 6 || S == 7, uint64_t,
                                                                     uint32_t>::type>::type;
template <int S>
__device__ __forceinline__ const tile_raw<S> *tile_plane(const NzRecords &rec) {
    if constexpr (S == 0 || S == 1 || S == 3) return rec.max_span;
    else if constexpr (S == 2) return rec.m0;
    else if constexpr (S == 4) return rec.m2;
    else if constexpr (S == 5) return rec.m3;
    else if constexpr (S == 8) return reinterpret_cast<const uint16_t *>(rec.m0);
    else if constexpr (S == 9) return reinterpret_cast<const uint32_t *>(rec.m2);
    else return rec.m4_lo;
}
template <int S>
__device__ __forceinline__ double tile_value(tile_raw<S> q, uint32_t hi) {
    if constexpr (S == 6) return fma((double)hi, 18446744073709551616.0, (double)q);
    else return (double)q;
}

// calls step(row group index k, loaded group) for the 8-row groups of
// [first, first + 8 * groups) of run r, the next one's loads in flight
template <typename Raw, typename Load, typename Step>
__device__ __forceinline__ void for_groups(uint32_t groups, Load load, Step step) {
    Raw q;
    if (groups > 0) load(0, q);
    for (uint32_t k = 0; k < groups; ++k) {
        const Raw cur = q;
        if (k + 1 < groups) load(k + 1, q);
        step(k, cur);
    }
}

// part[j] += the products of 8 rows, for the probabilities whose bands meet them
// (bit j of `in`, the same for the whole block)
template <int PT>
__device__ __forceinline__ void add_group(const double (*w)[PT], uint32_t in, const double (&v)[8],
                                          double (&part)[PT]) {
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        if (!(in >> j & 1u)) continue;
#pragma unroll
        for (int b = 0; b < 8; ++b) part[j] = fma(w[b][j], v[b], part[j]);
    }
}

template <int S, int PT>
__device__ __forceinline__ void conv_rows_tiled(const ConvParams &p, uint32_t first, uint32_t groups, int r,
                                                const double (*s_w)[PT], const uint32_t *s_in,
                                                double *acc) {
    struct Raw {
        tile_raw<S> q[8];
        uint32_t hi[S == 6 ? 8 : 1];
    };
    double part[PT];
#pragma unroll
    for (int j = 0; j < PT; ++j) part[j] = 0;
    for_groups<Raw>(
        groups,
        [&](uint32_t k, Raw &q) {
            load_rows8(tile_plane<S>(p.rec), p.rec.run_stride, first + 8 * k, r, q.q);
            if constexpr (S == 6) load_rows8(p.rec.m4_hi, p.rec.run_stride, first + 8 * k, r, q.hi);
        },
        [&](uint32_t k, const Raw &q) {
            double v[8];
#pragma unroll
            for (int b = 0; b < 8; ++b) v[b] = tile_value<S>(q.q[b], S == 6 ? q.hi[S == 6 ? b : 0] : 0u);
            add_group<PT>(s_w + 8 * k, s_in[k], v, part);
        });
#pragma unroll
    for (int j = 0; j < PT; ++j) acc[j] += part[j];
}

template <bool SITE, int PT>
__device__ __forceinline__ void conv_rows_max_tiled(const ConvParams &p, uint32_t first, uint32_t groups, int r,
                                                    const double (*s_w)[PT], const uint32_t *s_in,
                                                    double *acc0, double *acc1,
                                                    double *acc3) {
    struct Raw {
        uint32_t q[8];
    };
    double p0[PT], p1[PT], p3[PT];
#pragma unroll
    for (int j = 0; j < PT; ++j) p0[j] = p1[j] = p3[j] = 0;
    for_groups<Raw>(
        groups, [&](uint32_t k, Raw &q) { load_rows8(p.rec.max_span, p.rec.run_stride, first + 8 * k, r, q.q); },
        [&](uint32_t k, const Raw &q) {
            double v[8];
            uint32_t flags = 0;
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                flags |= q.q[b];
                v[b] = (double)(q.q[b] & ~kSpanBit);
            }
            add_group<PT>(s_w + 8 * k, s_in[k], v, p1);
#pragma unroll
            for (int b = 0; b < 8; ++b)
                v[b] = (double)((SITE ? p.n_begin + first + 8 * k + b : p.N) - (q.q[b] & ~kSpanBit));
            add_group<PT>(s_w + 8 * k, s_in[k], v, p3);
            // spanning: rows without it add nothing (a third of the work below
            // the threshold)
            if (!p.spanning || !(flags & kSpanBit)) return;
#pragma unroll
            for (int b = 0; b < 8; ++b) v[b] = (q.q[b] & kSpanBit) ? 1.0 : 0.0;
            add_group<PT>(s_w + 8 * k, s_in[k], v, p0);
        });
#pragma unroll
    for (int j = 0; j < PT; ++j) {
        acc0[j] += p0[j];
        acc1[j] += p1[j];
        acc3[j] += p3[j];
    }
}

// Each thread accumulates the PT canonical values of its run over the
// window's rows, with the tile's weights staged in shared memory (zero
// outside each p's band), in FP64.
// MAXSET: grid (run tiles, p tiles, 1), statistics 0, 1 and 3 from the
// max_span plane in one pass; otherwise grid (run tiles, p tiles, 4),
// statistics 2, 4, 5, 6 (one per z).
enum class Layout { kBond, kSite, kTiled, kTiledSite };  // records of bonds or sites, n-major or tiled

template <Layout LAYOUT, bool MAXSET, int PT>
__global__ void __launch_bounds__(kConvRuns) conv_window_kernel(ConvParams p) {
    constexpr bool SITE = LAYOUT == Layout::kSite || LAYOUT == Layout::kTiledSite;
    constexpr bool TILED = LAYOUT == Layout::kTiled || LAYOUT == Layout::kTiledSite;
    __shared__ double s_w[kConvChunk + (TILED ? 8 : 0)][PT];
    __shared__ uint32_t s_lo[PT], s_len[PT];
    __shared__ uint32_t s_range[2];
    __shared__ uint32_t s_in[TILED ? kConvChunk / 8 + 1 : 1];  // probabilities whose bands meet the 8-row group
    const int r = blockIdx.x * kConvRuns + threadIdx.x;
    const int p0 = blockIdx.y * PT;
    constexpr int kOther[4] = {2, 4, 5, 6};
    const int s = MAXSET ? 1 : kOther[blockIdx.z];
    if (threadIdx.x < PT) {
        const int pi = p0 + threadIdx.x;
        s_lo[threadIdx.x] = pi < p.P ? p.band_lo[pi] : 0u;
        s_len[threadIdx.x] = pi < p.P ? p.band_len[pi] : 0u;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t a = 0xffffffffu, b = 0;
        for (int j = 0; j < PT; ++j)
            if (s_len[j]) { a = min(a, s_lo[j]); b = max(b, s_lo[j] + s_len[j]); }
        a = max(a, p.n_begin);
        b = min(b, p.n_end);
        // chunks are counted from the first row of kConvPT probabilities, so
        // that the sums do not depend on PT
        if (PT < kConvPT && a < b) {
            uint32_t first = a;
            for (int pi = p0 / kConvPT * kConvPT; pi < min(p.P, p0 / kConvPT * kConvPT + kConvPT); ++pi)
                if (p.band_len[pi]) first = min(first, p.band_lo[pi]);
            first = max(first, p.n_begin);
            a = first + (a - first) / kConvChunk * kConvChunk;
        }
        s_range[0] = a; s_range[1] = b;
    }
    __syncthreads();
    const uint32_t nlo = s_range[0], nhi = s_range[1];
    if (nlo >= nhi) return;
    double acc[PT] = {}, acc0[MAXSET ? PT : 1] = {}, acc3[MAXSET ? PT : 1] = {};
    for (uint32_t c0 = nlo; c0 < nhi; c0 += kConvChunk) {
        const uint32_t cn = min((uint32_t)kConvChunk, nhi - c0);
        // tiled: rows of the 8-row group that holds c0 come first
        const uint32_t lead = TILED ? (c0 - p.n_begin) & 7u : 0u;
        __syncthreads();
        for (int i = threadIdx.x; i < (kConvChunk + (TILED ? 8 : 0)) * PT; i += kConvRuns) {
            const int row = i / PT, j = i % PT;
            const uint32_t n = c0 + row - lead;
            double v = 0;
            if ((uint32_t)row - lead < cn && n >= s_lo[j] && n < s_lo[j] + s_len[j]) {
                const size_t widx = (size_t)(p0 + j) * p.cap + (n - s_lo[j]);
                v = p.w64[widx];
            }
            s_w[row][j] = v;
        }
        if (TILED && threadIdx.x <= kConvChunk / 8) {
            // window rows and chunk rows of the group, then of each band
            const uint32_t a = max(c0, c0 - lead + 8u * threadIdx.x), b = min(c0 + cn, c0 - lead + 8u * threadIdx.x + 8u);
            uint32_t in = 0;
            for (int j = 0; j < PT; ++j)
                if (s_len[j] && a < b && s_lo[j] < b && a < s_lo[j] + s_len[j]) in |= 1u << j;
            s_in[threadIdx.x] = in;
        }
        __syncthreads();
        if constexpr (TILED) {
            if (r < p.n_runs) {
                const uint32_t first = c0 - p.n_begin - lead, groups = (lead + cn + 7u) / 8u;
                if (MAXSET) {
                    conv_rows_max_tiled<SITE, PT>(p, first, groups, r, s_w, s_in, acc0, acc, acc3);
                } else if (s == 2) {
                    if (p.rec.narrow) conv_rows_tiled<8, PT>(p, first, groups, r, s_w, s_in, acc);
                    else conv_rows_tiled<2, PT>(p, first, groups, r, s_w, s_in, acc);
                } else if (s == 4) {
                    if (p.rec.narrow) conv_rows_tiled<9, PT>(p, first, groups, r, s_w, s_in, acc);
                    else conv_rows_tiled<4, PT>(p, first, groups, r, s_w, s_in, acc);
                } else if (s == 5) {
                    conv_rows_tiled<5, PT>(p, first, groups, r, s_w, s_in, acc);
                } else {
                    if (p.rec.m4_hi) conv_rows_tiled<6, PT>(p, first, groups, r, s_w, s_in, acc);
                    else conv_rows_tiled<7, PT>(p, first, groups, r, s_w, s_in, acc);
                }
            }
        } else if (r < p.n_runs) {
            if (MAXSET) {
                conv_rows_max<SITE, PT>(p, c0, cn, r, s_w, acc0, acc, acc3);
            } else {
                switch (s) {
                    case 2:
                        if (p.rec.narrow) conv_rows<8, SITE, PT>(p, c0, cn, r, s_w, acc);
                        else conv_rows<2, SITE, PT>(p, c0, cn, r, s_w, acc);
                        break;
                    case 4:
                        if (p.rec.narrow) conv_rows<9, SITE, PT>(p, c0, cn, r, s_w, acc);
                        else conv_rows<4, SITE, PT>(p, c0, cn, r, s_w, acc);
                        break;
                    case 5: conv_rows<5, SITE, PT>(p, c0, cn, r, s_w, acc); break;
                    default:
                        if (p.rec.m4_hi) conv_rows<6, SITE, PT>(p, c0, cn, r, s_w, acc);
                        else conv_rows<7, SITE, PT>(p, c0, cn, r, s_w, acc);
                        break;
                }
            }
        }
    }
    if (r < p.n_runs) {
#pragma unroll
        for (int j = 0; j < PT; ++j) {
            const int pi = p0 + j;
            if (pi >= p.P) continue;
            double *o = p.acc + ((size_t)r * p.P + pi) * 7;
            o[s] += acc[j];
            if (MAXSET) {
                if (p.spanning) o[0] += acc0[j];
                o[3] += acc3[j];
            }
        }
    }
}

bool conv_grid_fits(int32_t n_runs, int32_t P) {
    // grid.y (p tiles) is limited to 65535
    return n_runs > 0 && P > 0 && (P + kConvPT - 1) / kConvPT <= 65535;
}

template <int PT>
static cudaError_t launch_conv_fp64(const ConvParams &p, cudaStream_t s) {
    // (run tiles, p tiles, statistics); launching the p tiles of one run tile
    // back to back (for L2 reuse of its records) measured slower
    dim3 gmax((p.n_runs + kConvRuns - 1) / kConvRuns, (p.P + PT - 1) / PT, 1);
    dim3 gother(gmax.x, gmax.y, 4);
    // the record model is a template parameter: a run-time test in the row
    // loop cost 17 % of the kernel's time
    auto launch = [&](auto max_set, auto others) {
        const cudaError_t e = launch_kernel(max_set, gmax, kConvRuns, 0, 0, s, p);
        return e == cudaSuccess ? launch_kernel(others, gother, kConvRuns, 0, 0, s, p) : e;
    };
    if (p.tiled && p.rec.site)
        return launch(conv_window_kernel<Layout::kTiledSite, true, PT>, conv_window_kernel<Layout::kTiledSite, false, PT>);
    if (p.tiled) return launch(conv_window_kernel<Layout::kTiled, true, PT>, conv_window_kernel<Layout::kTiled, false, PT>);
    if (p.rec.site) return launch(conv_window_kernel<Layout::kSite, true, PT>, conv_window_kernel<Layout::kSite, false, PT>);
    return launch(conv_window_kernel<Layout::kBond, true, PT>, conv_window_kernel<Layout::kBond, false, PT>);
}

cudaError_t launch_conv_window(const ConvParams &p, int precision, cudaStream_t s) {
    if (p.n_runs <= 0 || p.P <= 0) return cudaSuccess;
    if (precision != 0) return launch_conv_tiles(p, s);  // ensembles only: tiled records
    // Fewer probabilities per CTA, so more CTAs, where tiles of 8 leave SMs idle
    // (whole ensembles in ms with 8, 4, 2: 200 runs of 200 x 200 at 100 p, 26
    // tiles, 8.4, 5.5, 4.2; 1,000 toruses of 64 x 64 at 101 p, 104 tiles, 3.0,
    // 2.6, 2.6; 1,000 grids of 128 x 128 at 201 p, 208 tiles, 8.6, 8.5, 8.8).
    const int64_t tiles = (int64_t)((p.n_runs + kConvRuns - 1) / kConvRuns) * ((p.P + kConvPT - 1) / kConvPT);
    return tiles < 64 ? launch_conv_fp64<2>(p, s) : tiles < 152 ? launch_conv_fp64<4>(p, s) : launch_conv_fp64<kConvPT>(p, s);
}

// Weights of the FP32 convolution: the part of each p's band whose weights
// are at least `rel` times the band's largest, converted to FP32 and re-based
// at its own low edge (w32[i * cap + j] is the weight of row lo32[i] + j).
// The band of the FP64 path reaches weights e^-80 below its mode; at rel =
// e^-30 (7.7 standard deviations from the mode) the weights left out sum to
// less than 1e-13, far below the FP32 rounding of the sums, and the rows each
// p reads shrink by 40 %.  Band weights are unimodal, so the kept part is one
// run of rows.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) narrow_weights_f32_kernel(const double *w64, const uint32_t *band_lo,
                                                                   const uint32_t *band_len, int32_t cap, double rel,
                                                                   double rel_core, float *w32, float *w32lo,
                                                                   uint32_t *lo32, uint32_t *len32,
                                                                   uint32_t *core_lo, uint32_t *core_len) {
    __shared__ double s_max[BLOCK / 32];
    __shared__ uint32_t s_a[BLOCK / 32], s_b[BLOCK / 32], s_ca[BLOCK / 32], s_cb[BLOCK / 32];
    const int pi = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *w = w64 + (size_t)pi * cap;
    const uint32_t len = min(band_len[pi], (uint32_t)cap);
    double m = 0.0;
    for (uint32_t j = threadIdx.x; j < len; j += BLOCK) m = fmax(m, w[j]);
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) s_max[warp] = m;
    __syncthreads();
    m = s_max[0];
    for (int k = 1; k < BLOCK / 32; ++k) m = fmax(m, s_max[k]);
    const double thr = m * rel, thr_core = m * rel_core;
    uint32_t a = 0xffffffffu, b = 0, ca = 0xffffffffu, cb = 0;
    for (uint32_t j = threadIdx.x; j < len; j += BLOCK) {
        if (w[j] >= thr) { a = min(a, j); b = max(b, j + 1); }
        if (w[j] >= thr_core) { ca = min(ca, j); cb = max(cb, j + 1); }
    }
    for (int o = 16; o > 0; o >>= 1) {
        a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
        b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
        ca = min(ca, __shfl_xor_sync(0xffffffffu, ca, o));
        cb = max(cb, __shfl_xor_sync(0xffffffffu, cb, o));
    }
    if (lane == 0) { s_a[warp] = a; s_b[warp] = b; s_ca[warp] = ca; s_cb[warp] = cb; }
    __syncthreads();
    a = s_a[0]; b = s_b[0]; ca = s_ca[0]; cb = s_cb[0];
    for (int k = 1; k < BLOCK / 32; ++k) {
        a = min(a, s_a[k]); b = max(b, s_b[k]);
        ca = min(ca, s_ca[k]); cb = max(cb, s_cb[k]);
    }
    if (b <= a) a = b = 0;  // an empty band stays empty
    if (cb <= ca) ca = cb = 0;
    if (threadIdx.x == 0) {
        lo32[pi] = band_lo[pi] + a;
        len32[pi] = b - a;
        core_lo[pi] = band_lo[pi] + ca;
        core_len[pi] = cb - ca;
    }
    float *o = w32 + (size_t)pi * cap;
    float *ol = w32lo + (size_t)pi * cap;
    for (uint32_t j = threadIdx.x; j < (uint32_t)cap; j += BLOCK) {
        const double v = j < b - a ? w[a + j] : 0.0;
        const float hi = (float)v;
        o[j] = hi;
        ol[j] = (float)(v - (double)hi);  // exact difference; its FP32 rounding is 2^-24 of 2^-24 w
    }
}

void launch_narrow_weights_f32(const double *w64, const uint32_t *band_lo, const uint32_t *band_len, int32_t P,
                               int32_t cap, double rel, double rel_core, float *w32, float *w32lo, uint32_t *lo32,
                               uint32_t *len32, uint32_t *core_lo, uint32_t *core_len, cudaStream_t s) {
    if (P <= 0) return;
    narrow_weights_f32_kernel<256><<<P, 256, 0, s>>>(w64, band_lo, band_len, cap, rel, rel_core, w32, w32lo, lo32,
                                                     len32, core_lo, core_len);
}

// =====================================================================
// Pairwise (n, mean, M2) reduction over runs
// =====================================================================
// Chan, Golub & LeVeque (1979) pairwise update, the formula simoa's
// online_variance applies in bond_reduce (percolate/hpc.py:674-692).
__device__ __forceinline__ void chan_merge(double &na, double &ma, double &sa, double nb, double mb, double sb) {
    if (nb == 0.0) return;
    if (na == 0.0) { na = nb; ma = mb; sa = sb; return; }
    const double n = na + nb;
    const double d = mb - ma;
    ma += d * nb / n;
    sa += sb + d * d * na * nb / n;
    na = n;
}

// stats [n_runs][P*7]: one thread per column, looping over a slice of runs;
// partial (n, mean, M2) go to `part` [slices][cols][3].
__global__ void reduce_runs_partial_kernel(const double *stats, int32_t n_runs, int32_t cols, int32_t slice,
                                           double *part) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int sl = blockIdx.y;
    if (c >= cols) return;
    const int r0 = sl * slice, r1 = min(n_runs, r0 + slice);
    // sums of the deviations from the slice's first value, x0: mean = x0 +
    // S1 / n, M2 = S2 - S1^2 / n (the shift keeps the difference free of
    // cancellation).  Welford's update needs an FP64 division per value, and
    // FP64 runs at 1/64 of the FP32 rate on this chip.
    double x0 = 0.0, s1 = 0.0, s2 = 0.0;
    if (r0 < r1) x0 = stats[(size_t)r0 * cols + c];
    int r = r0 + 1;
    for (; r + 8 <= r1; r += 8) {  // 8 loads in flight
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = stats[(size_t)(r + k) * cols + c];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const double d = v[k] - x0;
            s1 += d;
            s2 = fma(d, d, s2);
        }
    }
    for (; r < r1; ++r) {
        const double d = stats[(size_t)r * cols + c] - x0;
        s1 += d;
        s2 = fma(d, d, s2);
    }
    const double n = (double)max(r1 - r0, 0);
    double *o = part + ((size_t)sl * cols + c) * 3;
    o[0] = n;
    o[1] = n > 0 ? x0 + s1 / n : 0.0;
    o[2] = n > 0 ? fmax(s2 - s1 * s1 / n, 0.0) : 0.0;
}

__global__ void reduce_runs_final_kernel(const double *part, int32_t cols, int32_t slices, const uint64_t *acc_count,
                                         double *acc_mean, double *acc_m2) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    double n = 0, mean = 0, m2 = 0;
    for (int sl = 0; sl < slices; ++sl) {
        const double *o = part + ((size_t)sl * cols + c) * 3;
        chan_merge(n, mean, m2, o[0], o[1], o[2]);
    }
    double na = (double)*acc_count, ma = acc_mean[c], sa = acc_m2[c];
    chan_merge(na, ma, sa, n, mean, m2);
    acc_mean[c] = ma;
    acc_m2[c] = sa;
}

__global__ void add_count_kernel(uint64_t *count, int32_t n) { *count += (uint64_t)n; }

void launch_reduce_runs(const double *stats, int32_t n_runs, int32_t P, uint64_t *acc_count, double *acc_mean,
                           double *acc_m2, double *part, int32_t slices, cudaStream_t s) {
    const int cols = P * 7;
    const int slice = (n_runs + slices - 1) / slices;
    dim3 grid((cols + 127) / 128, slices);
    reduce_runs_partial_kernel<<<grid, 128, 0, s>>>(stats, n_runs, cols, slice, part);
    reduce_runs_final_kernel<<<(cols + 127) / 128, 128, 0, s>>>(part, cols, slices, acc_count, acc_mean, acc_m2);
    add_count_kernel<<<1, 1, 0, s>>>(acc_count, n_runs);
}

// =====================================================================
// Microcanonical run-reductions (fused over a window of records)
// =====================================================================
// Per (row n, statistic): exact integer sum over runs and the sum of squared
// deviations, merged into the accumulators with the pairwise formula.
// Statistics: 0 max, 1 m0, 2 m1 (= N - max), 3 m2, 4 m3, 5 m4; block 6
// counts the spanning runs.  Deviations are taken from run 0's value x0:
//   max, m0, m1 (< 2^21) and m2 (< 2^42): d = x - x0 as int64, d^2 summed
//     exactly (u64 / u128), and M2 = (R * sum d^2 - (sum d)^2) / R from the
//     exact 128-bit numerator;
//   m3, m4: d exact as a 128-bit integer; |d| 2^-e as two FP32 parts (its
//     top 48 bits, 2^-47 relative), squared with an exact FP32 product and
//     summed as an FP32 (sum, compensation) pair per thread, then in FP64
//     across threads (the shift keeps the sum free of cancellation; the
//     power-of-two scale 2^-e, e from N, keeps squares and sums inside FP32's
//     range).  FP64 runs at 1/64 of the FP32 rate on this chip, and the FP64
//     squares were most of this kernel's time.
typedef __int128 i128;

__device__ __forceinline__ u128 shfl_down_u128(u128 v, int off) {
    uint64_t lo = (uint64_t)v, hi = (uint64_t)(v >> 64);
    lo = __shfl_down_sync(0xffffffffu, lo, off);
    hi = __shfl_down_sync(0xffffffffu, hi, off);
    return ((u128)hi << 64) | lo;
}

template <int BLOCK>
__device__ __forceinline__ u128 block_sum_u128(u128 v, u128 *s_tmp) {
    for (int off = 16; off > 0; off >>= 1) v += shfl_down_u128(v, off);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) s_tmp[warp] = v;
    __syncthreads();
    u128 t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < BLOCK / 32; ++w) t += s_tmp[w];
    return t;  // valid in thread 0
}

template <int BLOCK>
__device__ __forceinline__ double block_sum_f64(double v, double *s_tmp) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) s_tmp[warp] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < BLOCK / 32; ++w) t += s_tmp[w];
    return t;
}

__device__ __forceinline__ double u128_to_f64(u128 x) {
    return fma((double)(uint64_t)(x >> 64), 18446744073709551616.0, (double)(uint64_t)x);
}

__device__ __forceinline__ double i128_to_f64(i128 x) {
    return x < 0 ? -u128_to_f64((u128)(-x)) : u128_to_f64((u128)x);
}

// Per-thread partial sums of one row: for every statistic the exact sum of
// x, the exact sum of d = x - x0 and the sum of d^2 (exact integers for
// max, m0, m2; FP64 for m3, m4), plus the spanning count.
struct MicroPart {
    uint64_t sx_max, sx_m0, sx_m2;  // max, m0 < 2^21; m2 < 2^42 (per-thread sums fit)
    u128 sx_m3, sx_m4;
    int64_t sd_max, sd_m0, sd_m2;
    i128 sd_m3, sd_m4;
    uint64_t sq_max, sq_m0;
    u128 sq_m2;
    float fs_m3, fc_m3, fs_m4, fc_m4;  // scaled sum of d^2 and its compensation
    uint32_t span;
};

__device__ __forceinline__ float exp2i(int k) { return __int_as_float((127 + k) << 23); }  // -126 <= k <= 127

// x (< 2^96, as 64-bit halves) times 2^-e as yh + yl: yh = x's top 24
// significant bits, yl = the next 24 (both exact in FP32; the bits below are
// truncated: 2^-47 relative), so yh^2 carries the square and yl only small
// corrections.
__device__ __forceinline__ void scaled_split(uint64_t lo, uint64_t hi, int e, float &yh, float &yl) {
    const int nb = hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
    const int s2 = nb > 48 ? nb - 48 : 0;  // y = x >> s2 keeps min(nb, 48) bits
    uint64_t y;
    if (s2 == 0) y = lo;
    else if (s2 < 64) y = (lo >> s2) | (hi << (64 - s2));
    else y = hi >> (s2 - 64);
    const int sh = nb > 24 ? nb - s2 - 24 : 0;  // y's top 24 bits sit above bit sh
    const uint64_t top = y >> sh;
    const int k = s2 - e;
    yh = (float)(uint32_t)top * exp2i(sh + k);
    yl = (float)(uint32_t)(y - (top << sh)) * exp2i(k);
}

// (s, c) += (yh + yl)^2: the exact product yh^2 (TwoProd by FMA), TwoSum of
// the running sum, the cross and low terms into the compensation.
__device__ __forceinline__ void add_square(float &s, float &c, float yh, float yl) {
    const float p = __fmul_rn(yh, yh);
    const float pe = fmaf(yh, yh, -p);
    const float cross = fmaf(2.0f * yh, yl, __fmul_rn(yl, yl));
    const float t = __fadd_rn(s, p);
    const float bp = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(p, bp));
    s = t;
    c = __fadd_rn(c, __fadd_rn(err, __fadd_rn(pe, cross)));
}

template <int BLOCK>
__device__ __forceinline__ uint64_t bsum_u64(uint64_t v, uint64_t *s_tmp) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_tmp[threadIdx.x >> 5] = v;
    __syncthreads();
    uint64_t t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < BLOCK / 32; ++w) t += s_tmp[w];
    return t;
}

// 3 resident blocks of 256 threads per SM (at most 80 registers, a few
// hundred bytes of spills): beside the union-find of the next window this
// measured 1364 against 1394 ms per 100,000-run L = 256 step at 100
// registers.
#ifndef NZ_MICRO_MIN_BLOCKS
#define NZ_MICRO_MIN_BLOCKS 3
#endif
// records in flight per thread: 2 against 1 took the kernel from 400 to
// 179 ms per 100,000-run L = 256 step inside the pipeline; 4 (with a few
// hundred bytes of spills at the 80-register cap) gave the same step time
// (1076.2 against 1076.0 ms, same box)
#ifndef NZ_MICRO_INFLIGHT
#define NZ_MICRO_INFLIGHT 2
#endif
constexpr int kMicroInflight = NZ_MICRO_INFLIGHT;
#define NZ_MICRO_BOUNDS __launch_bounds__(BLOCK, NZ_MICRO_MIN_BLOCKS)

// One block per row n: reduces all statistics of that row over the runs and
// merges them into the accumulators (pairwise formula for M2).
template <int BLOCK>
__global__ void NZ_MICRO_BOUNDS micro_window_kernel(MicroParams p) {
    const uint32_t n = p.n_begin + blockIdx.x;
    const size_t row = (size_t)(n - p.n_begin) * p.rec.run_stride;
    const NzRecords &rec = p.rec;
    __shared__ u128 s_u[BLOCK / 32];
    __shared__ double s_f[BLOCK / 32];
    __shared__ uint64_t s_w[BLOCK / 32];
    const uint32_t x0_max = rec.max_span[row] & ~kSpanBit;
    const uint32_t x0_m0 = record_m0(rec, row);
    const uint64_t x0_m2 = record_m2(rec, row), x0_m3 = rec.m3[row];
    const bool has_hi = rec.m4_hi != nullptr;  // without the plane the high words are zero
    const u128 x0_m4 = ((u128)(has_hi ? rec.m4_hi[row] : 0u) << 64) | rec.m4_lo[row];
    // scales: m3 < N^3 and m4 < N^4 (< 2^96); |d| 2^-e <= 2^40, so squares
    // stay below 2^80 and sums below 2^111, and |d| >= 1 keeps its square
    // above 2^-88 (FP32 normal)
    const int nbits = 32 - __clz((int)p.N);
    const int e3 = max(0, 3 * nbits - 40), e4 = max(0, min(4 * nbits, 96) - 40);
    MicroPart a = {};
    struct Rec {
        uint32_t ms, m0, m4_hi;
        uint64_t m2, m3, m4_lo;
    };
    auto load = [&](int r) -> Rec {
        const size_t off = row + r;
        return Rec{rec.max_span[off], record_m0(rec, off), has_hi ? rec.m4_hi[off] : 0u,
                   record_m2(rec, off), rec.m3[off],     rec.m4_lo[off]};
    };
    auto add = [&](const Rec &q) {
        const uint32_t mx = q.ms & ~kSpanBit;
        const u128 m4 = ((u128)q.m4_hi << 64) | q.m4_lo;
        a.span += q.ms >> 31;
        a.sx_max += mx;
        a.sx_m0 += q.m0;
        a.sx_m2 += q.m2;
        a.sx_m3 += q.m3;
        a.sx_m4 += m4;
        const int64_t dmax = (int64_t)mx - (int64_t)x0_max;
        const int64_t dm0 = (int64_t)q.m0 - (int64_t)x0_m0;
        const int64_t dm2 = (int64_t)q.m2 - (int64_t)x0_m2;
        const int64_t dm3 = (int64_t)(q.m3 - x0_m3);  // |m3 - x0| < 2^63
        const i128 dm4 = (i128)(m4 - x0_m4);
        a.sd_max += dmax;
        a.sd_m0 += dm0;
        a.sd_m2 += dm2;
        a.sd_m3 += dm3;
        a.sd_m4 += dm4;
        a.sq_max += (uint64_t)(dmax * dmax);
        a.sq_m0 += (uint64_t)(dm0 * dm0);
        const uint64_t ad2 = (uint64_t)(dm2 < 0 ? -dm2 : dm2);
        a.sq_m2 += (u128)ad2 * ad2;
        float yh, yl;
        scaled_split((uint64_t)(dm3 < 0 ? -dm3 : dm3), 0, e3, yh, yl);
        add_square(a.fs_m3, a.fc_m3, yh, yl);
        const u128 ad4 = (u128)(dm4 < 0 ? -dm4 : dm4);
        scaled_split((uint64_t)ad4, (uint64_t)(ad4 >> 64), e4, yh, yl);
        add_square(a.fs_m4, a.fc_m4, yh, yl);
    };
    // the records of NZ_MICRO_INFLIGHT runs are loaded before any is added,
    // so each thread keeps that many records' loads in flight
    int r = threadIdx.x;
    for (; r + (kMicroInflight - 1) * BLOCK < p.n_runs; r += kMicroInflight * BLOCK) {
        Rec q[kMicroInflight];
#pragma unroll
        for (int k = 0; k < kMicroInflight; ++k) q[k] = load(r + k * BLOCK);
#pragma unroll
        for (int k = 0; k < kMicroInflight; ++k) add(q[k]);
    }
    for (; r < p.n_runs; r += BLOCK) add(load(r));
    // block sums (results valid in thread 0)
    const uint64_t span = bsum_u64<BLOCK>(a.span, s_w);
    const uint64_t sx_max = bsum_u64<BLOCK>(a.sx_max, s_w);
    const uint64_t sx_m0 = bsum_u64<BLOCK>(a.sx_m0, s_w);
    const u128 sx_m2 = block_sum_u128<BLOCK>(a.sx_m2, s_u);
    const u128 sx_m3 = block_sum_u128<BLOCK>(a.sx_m3, s_u);
    const u128 sx_m4 = block_sum_u128<BLOCK>(a.sx_m4, s_u);
    const i128 sd_max = (i128)block_sum_u128<BLOCK>((u128)(i128)a.sd_max, s_u);
    const i128 sd_m0 = (i128)block_sum_u128<BLOCK>((u128)(i128)a.sd_m0, s_u);
    const i128 sd_m2 = (i128)block_sum_u128<BLOCK>((u128)(i128)a.sd_m2, s_u);
    const i128 sd_m3 = (i128)block_sum_u128<BLOCK>((u128)a.sd_m3, s_u);
    const i128 sd_m4 = (i128)block_sum_u128<BLOCK>((u128)a.sd_m4, s_u);
    const u128 sq_max = block_sum_u128<BLOCK>(a.sq_max, s_u);
    const u128 sq_m0 = block_sum_u128<BLOCK>(a.sq_m0, s_u);
    const u128 sq_m2 = block_sum_u128<BLOCK>(a.sq_m2, s_u);
    const double fq_m3 = ldexp(block_sum_f64<BLOCK>((double)a.fs_m3 + (double)a.fc_m3, s_f), 2 * e3);
    const double fq_m4 = ldexp(block_sum_f64<BLOCK>((double)a.fs_m4 + (double)a.fc_m4, s_f), 2 * e4);
    if (threadIdx.x != 0) return;
    const double R = (double)p.n_runs;
    const uint64_t Rn = (uint64_t)p.n_runs;
    // exact M2 numerator R * sum d^2 - (sum d)^2 when it fits in 128 bits
    auto m2_exact = [&](u128 sq, i128 sd) -> double {
        const u128 ad = (u128)(sd < 0 ? -sd : sd);
        if ((sq >> 103) == 0 && (ad >> 63) == 0) return u128_to_f64(Rn * sq - ad * ad) / R;
        const double f = u128_to_f64(ad);
        const double v = u128_to_f64(sq) - f * f / R;
        return v > 0.0 ? v : 0.0;
    };
    auto m2_float = [&](double fq, i128 sd) -> double {
        const double f = i128_to_f64(sd);
        const double v = fq - f * f / R;
        return v > 0.0 ? v : 0.0;
    };
    // statistic order 0 max, 1 m0, 2 m1 (= N - max: same M2 as max), 3 m2, 4 m3, 5 m4
    const u128 held = rec.site ? n : p.N;  // sites in clusters: all N (bond) or the n occupied (site)
    const u128 sx[6] = {sx_max, sx_m0, (u128)Rn * held - sx_max, sx_m2, sx_m3, sx_m4};
    const double m2b_max = m2_exact(sq_max, sd_max);
    const double m2b[6] = {m2b_max, m2_exact(sq_m0, sd_m0), m2b_max, m2_exact(sq_m2, sd_m2),
                           m2_float(fq_m3, sd_m3), m2_float(fq_m4, sd_m4)};
    const double na = (double)*p.count_before;
    for (int k = 0; k < 6; ++k) {
        const size_t idx = (size_t)k * (p.M + 1) + n;
        const u128 acc = ((u128)p.acc.sum_hi[idx] << 64) | p.acc.sum_lo[idx];
        const double mean_a = na > 0 ? u128_to_f64(acc) / na : 0.0;
        double nn = na, mm = mean_a, ss = p.acc.m2[idx];
        chan_merge(nn, mm, ss, R, u128_to_f64(sx[k]) / R, m2b[k]);
        const u128 t = acc + sx[k];
        p.acc.sum_lo[idx] = (uint64_t)t;
        p.acc.sum_hi[idx] = (uint64_t)(t >> 64);
        p.acc.m2[idx] = ss;
    }
    p.acc.span_count[n] += span;
}

// The same reductions over tiled records: a block takes 32 rows, lane = row,
// and its warps share out the runs, so nothing is summed across lanes.  Sums
// of x and of x^2 are exact integers (x^2 of up to 168 bits), and the
// numerator R sum x^2 - (sum x)^2 of M2 is formed in 256 bits.
//
// What bounds it: reading the records once (60 % of DRAM's rate at 4,000 runs of 64 x
// 64: two blocks of 16 warps to an SM wait for loads 16 of 21 cycles).
constexpr int kMicroWarps = 16;

template <bool NARROW>
struct MicroSums {
    uint32_t span;
    uint64_t s_max, s_m0;  // < 2^21, of at most 2^24 runs
    u128 s_m2, s_m3, s_m4;  // (m2 < 2^42: 2^66)
    u128 q_max, q_m0, q_m2;
    typename std::conditional<NARROW, u128, U192>::type q_m3;  // m3 < 2^48 (narrow) or 2^63
    U192 q_m4;                                                 // m4 < 2^64 (narrow) or 2^84

    static __device__ __forceinline__ void accumulate(u128 &a, u128 x) { a += x; }
    static __device__ __forceinline__ void accumulate(U192 &a, u128 x) { a.add(x); }
    __device__ __forceinline__ void add(const MicroSums &o) {
        span += o.span;
        s_max += o.s_max;
        s_m0 += o.s_m0;
        s_m2 += o.s_m2;
        s_m3 += o.s_m3;
        s_m4 += o.s_m4;
        q_max += o.q_max;
        q_m0 += o.q_m0;
        q_m2 += o.q_m2;
        if constexpr (NARROW) q_m3 += o.q_m3;
        else q_m3.add(o.q_m3);
        q_m4.add(o.q_m4);
    }
    __device__ __forceinline__ U256 wide_m3() const {
        if constexpr (NARROW) return u256_from_u128(q_m3);
        else return q_m3.wide();
    }
};

// Adds up the sums `a` that the block's warps have of its 32 rows (in s_sum).
template <bool NARROW>
__device__ __forceinline__ void micro_combine(const MicroSums<NARROW> &a, MicroSums<NARROW> *s_sum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t w = 0; w < (uint32_t)kMicroWarps; ++w) {
        if (warp == w) {
            if (w == 0) s_sum[lane] = a;
            else s_sum[lane].add(a);
        }
        __syncthreads();
    }
}

// Merges the sums of all runs into the accumulators; the six statistics of the
// block's rows are shared out over its warps.
template <bool NARROW>
__device__ __forceinline__ void micro_accumulate(const MicroParams &p, const MicroSums<NARROW> *s_sum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t n = p.n_begin + blockIdx.x * 32u + lane;
    const NzRecords &rec = p.rec;
    if (n >= p.n_end || warp >= 7) return;
    const MicroSums<NARROW> &t = s_sum[lane];
    if (warp == 6) {
        p.acc.span_count[n] += t.span;
        return;
    }
    const uint64_t R = (uint64_t)p.n_runs;
    const u128 held = (u128)(rec.site ? n : p.N) * R;  // sites in clusters: all N (bond) or the n occupied (site)
    u128 sum = 0;
    U256 sq = {{0, 0, 0, 0}};
    switch (warp) {  // 0 max, 1 m0, 2 m1 (= N - max: same M2 as max), 3 m2, 4 m3, 5 m4
        case 1: sum = t.s_m0; sq = u256_from_u128(t.q_m0); break;
        case 3: sum = t.s_m2; sq = u256_from_u128(t.q_m2); break;
        case 4: sum = t.s_m3; sq = t.wide_m3(); break;
        case 5: sum = t.s_m4; sq = t.q_m4.wide(); break;
        default: sum = t.s_max; sq = u256_from_u128(t.q_max); break;
    }
    const double m2b = u256_to_f64(u256_sub(u256_mul64(sq, R), u128_sq(sum))) / (double)R;
    if (warp == 2) sum = held - sum;
    const double na = (double)*p.count_before;
    const size_t idx = (size_t)warp * (p.M + 1) + n;
    const u128 acc = ((u128)p.acc.sum_hi[idx] << 64) | p.acc.sum_lo[idx];
    double nn = na, mm = na > 0 ? u128_to_f64(acc) / na : 0.0, ss = p.acc.m2[idx];
    chan_merge(nn, mm, ss, (double)R, u128_to_f64(sum) / (double)R, m2b);
    const u128 total = acc + sum;
    p.acc.sum_lo[idx] = (uint64_t)total;
    p.acc.sum_hi[idx] = (uint64_t)(total >> 64);
    p.acc.m2[idx] = ss;
}

// SLICED: slice blockIdx.y of the runs, whose sums go to p.part.
template <bool NARROW, bool SLICED>
__global__ void __launch_bounds__(32 * kMicroWarps, 2) micro_tiled_kernel(MicroParams p, int slice) {
    __shared__ MicroSums<NARROW> s_sum[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * 32u + lane;
    const int r0 = SLICED ? (int)blockIdx.y * slice : 0, r1 = SLICED ? min(r0 + slice, p.n_runs) : p.n_runs;
    const NzRecords &rec = p.rec;
    MicroSums<NARROW> a = {};
    uint64_t q_max = 0, q_m0 = 0, s_m2 = 0;  // per thread: at most 2^20 runs' values < 2^42
    struct Rec {
        uint32_t ms, m0, m4_hi;
        uint64_t m2, m3, m4;
    };
    auto load = [&](int r) -> Rec {
        const size_t o4 = tile_off<4>(rec.run_stride, i, r), o8 = tile_off<8>(rec.run_stride, i, r);
        Rec q;
        q.ms = rec.max_span[o4];
        q.m0 = NARROW ? (uint32_t)reinterpret_cast<const uint16_t *>(rec.m0)[tile_off<2>(rec.run_stride, i, r)]
                      : rec.m0[o4];
        q.m2 = NARROW ? (uint64_t)reinterpret_cast<const uint32_t *>(rec.m2)[o4] : rec.m2[o8];
        q.m3 = rec.m3[o8];
        q.m4 = rec.m4_lo[o8];
        q.m4_hi = (!NARROW && rec.m4_hi) ? rec.m4_hi[o4] : 0u;
        return q;
    };
    auto add = [&](const Rec &q) {
        const uint32_t mx = q.ms & ~kSpanBit;
        a.span += q.ms >> 31;
        a.s_max += mx;
        a.s_m0 += q.m0;
        s_m2 += q.m2;
        a.s_m3 += q.m3;
        a.s_m4 += ((u128)q.m4_hi << 64) | q.m4;
        q_max += (uint64_t)mx * mx;
        q_m0 += (uint64_t)q.m0 * q.m0;
        a.q_m2 += NARROW ? (u128)(q.m2 * q.m2) : (u128)q.m2 * q.m2;
        MicroSums<NARROW>::accumulate(a.q_m3, (u128)q.m3 * q.m3);
        a.q_m4.add((u128)q.m4 * q.m4);
        if (!NARROW) {  // (hi 2^64 + lo)^2 = lo^2 + 2 lo hi 2^64 + hi^2 2^128, hi < 2^20
            const u128 mid = ((u128)q.m4 * q.m4_hi) << 1;  // < 2^85
            a.q_m4.add(mid << 64);
            a.q_m4.w2 += (uint64_t)(mid >> 64) + (uint64_t)q.m4_hi * q.m4_hi;
        }
    };
    constexpr int kAhead = 4;  // runs whose records are in flight per thread
    int r = r0 + (int)warp;
    for (; r + (kAhead - 1) * kMicroWarps < r1; r += kAhead * kMicroWarps) {
        Rec q[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) q[k] = load(r + k * kMicroWarps);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) add(q[k]);
    }
    for (; r < r1; r += kMicroWarps) add(load(r));
    a.s_m2 = s_m2;
    a.q_max = q_max;
    a.q_m0 = q_m0;
    micro_combine<NARROW>(a, s_sum);
    if constexpr (!SLICED) {
        micro_accumulate<NARROW>(p, s_sum);
    } else if (warp == 0) {
        reinterpret_cast<MicroSums<NARROW> *>(p.part)[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 32 + lane] =
            s_sum[lane];
    }
}

// The slices' sums, in order.
template <bool NARROW>
__global__ void __launch_bounds__(32 * kMicroWarps) micro_slices_kernel(MicroParams p, int slices) {
    __shared__ MicroSums<NARROW> s_sum[32];
    const uint32_t lane = threadIdx.x & 31u;
    const MicroSums<NARROW> *part = reinterpret_cast<const MicroSums<NARROW> *>(p.part);
    MicroSums<NARROW> a = {};
    for (int y = threadIdx.x >> 5; y < slices; y += kMicroWarps)
        a.add(part[((size_t)y * gridDim.x + blockIdx.x) * 32 + lane]);
    micro_combine<NARROW>(a, s_sum);
    micro_accumulate<NARROW>(p, s_sum);
}

// Few rows are few blocks: then the runs are cut into slices, of 2,048 at least,
// until there are two blocks to an SM (10^5 runs of 8 x 8, 4 blocks of 32 rows:
// 3.46 -> 0.13 ms; of 32 x 32 3.38 -> 1.31).  The sums are exact, so the results
// do not depend on it.
constexpr int kMicroBlocks = 304, kMicroSliceRuns = 2048;

template <bool NARROW>
static void launch_micro_tiled(const MicroParams &p, uint32_t rows, cudaStream_t s) {
    const int blocks = (int)((rows + 31) / 32);
    const int slices = std::max(1, std::min(kMicroBlocks / blocks, p.n_runs / kMicroSliceRuns));
    const int slice = (p.n_runs + slices - 1) / slices;
    if (slices == 1) {
        micro_tiled_kernel<NARROW, false><<<blocks, 32 * kMicroWarps, 0, s>>>(p, p.n_runs);
        return;
    }
    micro_tiled_kernel<NARROW, true><<<dim3(blocks, slices), 32 * kMicroWarps, 0, s>>>(p, slice);
    micro_slices_kernel<NARROW><<<blocks, 32 * kMicroWarps, 0, s>>>(p, slices);
}

size_t micro_part_bytes() { return sizeof(MicroSums<false>) * 32 * kMicroBlocks; }

void launch_micro_window(const MicroParams &p, cudaStream_t s) {
    const uint32_t rows = p.n_end - p.n_begin;
    if (rows == 0 || p.n_runs <= 0) return;
    if (p.tiled) {
        if (p.rec.narrow) launch_micro_tiled<true>(p, rows, s);
        else launch_micro_tiled<false>(p, rows, s);
        return;
    }
    micro_window_kernel<256><<<rows, 256, 0, s>>>(p);
}

void launch_micro_count(uint64_t *count, int32_t n_runs, cudaStream_t s) {
    add_count_kernel<<<1, 1, 0, s>>>(count, n_runs);
}

// ------------------------------------------------ merging two accumulators
// dst <- dst (+) src for running (count, mean, M2) columns sharing one count
// each side: the pairwise update of percolate/hpc.py:638-702.
__global__ void canonical_merge_kernel(const uint64_t *dst_count, double *dst_mean, double *dst_m2,
                                       const uint64_t *src_count, const double *src_mean,
                                       const double *src_m2, int32_t cols) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    double na = (double)*dst_count, ma = dst_mean[c], sa = dst_m2[c];
    chan_merge(na, ma, sa, (double)*src_count, src_mean[c], src_m2[c]);
    dst_mean[c] = ma;
    dst_m2[c] = sa;
}

// Microcanonical accumulators of rows = M + 1 rows: exact 128-bit sums and
// spanning counts add; M2 merges pairwise with the means taken from the
// exact sums, as micro_window_kernel merges a batch.
__global__ void micro_merge_kernel(NzMicroAccum dst, NzMicroAccum src, uint32_t rows) {
    const size_t total = (size_t)6 * rows;
    const double na = (double)*dst.count, nb = (double)*src.count;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total + rows;
         i += (size_t)gridDim.x * blockDim.x) {
        if (i >= total) {
            dst.span_count[i - total] += src.span_count[i - total];
            continue;
        }
        const u128 a = ((u128)dst.sum_hi[i] << 64) | dst.sum_lo[i];
        const u128 b = ((u128)src.sum_hi[i] << 64) | src.sum_lo[i];
        double nn = na, mm = na > 0 ? u128_to_f64(a) / na : 0.0, ss = dst.m2[i];
        chan_merge(nn, mm, ss, nb, nb > 0 ? u128_to_f64(b) / nb : 0.0, src.m2[i]);
        const u128 t = a + b;
        dst.sum_lo[i] = (uint64_t)t;
        dst.sum_hi[i] = (uint64_t)(t >> 64);
        dst.m2[i] = ss;
    }
}

__global__ void add_counts_kernel(uint64_t *dst, const uint64_t *src) { *dst += *src; }

// the counts are read by the merge kernels, so they are added afterwards
void launch_canonical_merge(uint64_t *dst_count, double *dst_mean, double *dst_m2, const uint64_t *src_count,
                            const double *src_mean, const double *src_m2, int32_t cols, cudaStream_t s) {
    if (cols > 0)
        canonical_merge_kernel<<<(cols + 255) / 256, 256, 0, s>>>(dst_count, dst_mean, dst_m2, src_count,
                                                                  src_mean, src_m2, cols);
    add_counts_kernel<<<1, 1, 0, s>>>(dst_count, src_count);
}

void launch_micro_merge(const NzMicroAccum &dst, const NzMicroAccum &src, uint32_t rows, cudaStream_t s) {
    const size_t work = (size_t)7 * rows;
    const unsigned grid = (unsigned)((work + 255) / 256 < 4096 ? (work + 255) / 256 : 4096);
    micro_merge_kernel<<<grid, 256, 0, s>>>(dst, src, rows);
    add_counts_kernel<<<1, 1, 0, s>>>(dst.count, src.count);
}

// =====================================================================
// Row-format kernels: initialize / reduce / finalize
// =====================================================================
// Packed structured rows with 4-byte alignment: doubles are moved as two words.
__device__ __forceinline__ double ld_f64(const uint8_t *p) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(p);
    return __hiloint2double((int)w[1], (int)w[0]);
}
__device__ __forceinline__ void st_f64(uint8_t *p, double v) {
    uint32_t *w = reinterpret_cast<uint32_t *>(p);
    w[0] = (uint32_t)__double2loint(v);
    w[1] = (uint32_t)__double2hiint(v);
}

// canonical_statistics_dtype (hpc.py:407-440): [pp f8] max f8 moments 5*f8
// canonical_averages_dtype  (hpc.py:518-558): n u4 [pp_mean pp_m2] max_mean max_m2
//                                             moments_mean 5*f8 moments_m2 5*f8
__global__ void init_avg_kernel(const uint8_t *canon, int32_t P, int32_t spanning, uint8_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const int nst = spanning ? 7 : 6;
    const uint8_t *c = canon + (size_t)i * nst * 8;
    uint8_t *o = out + (size_t)i * (4 + nst * 16);
    *reinterpret_cast<uint32_t *>(o) = 1u;
    int k = 0;
    if (spanning) { st_f64(o + 4, ld_f64(c)); st_f64(o + 12, 0.0); k = 1; }
    const int base = 4 + k * 16;
    st_f64(o + base, ld_f64(c + k * 8));
    st_f64(o + base + 8, 0.0);
    for (int m = 0; m < 5; ++m) {
        st_f64(o + base + 16 + 8 * m, ld_f64(c + (k + 1 + m) * 8));
        st_f64(o + base + 56 + 8 * m, 0.0);
    }
}

void launch_init_avg(const uint8_t *canon_rows, int32_t P, int32_t spanning, uint8_t *out, cudaStream_t s) {
    if (P > 0) init_avg_kernel<<<(P + 127) / 128, 128, 0, s>>>(canon_rows, P, spanning, out);
}

__global__ void bond_reduce_kernel(const uint8_t *a, const uint8_t *b, int32_t P, int32_t spanning, uint8_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P) return;
    const int nst = spanning ? 7 : 6;
    const size_t rb = 4 + nst * 16;
    const uint8_t *ra = a + i * rb, *rbp = b + i * rb;
    uint8_t *o = out + i * rb;
    const uint32_t na = *reinterpret_cast<const uint32_t *>(ra);
    const uint32_t nb = *reinterpret_cast<const uint32_t *>(rbp);
    // (mean offset, m2 offset) pairs
    int mo[7], so[7], cnt = 0;
    int off = 4;
    if (spanning) { mo[cnt] = off; so[cnt] = off + 8; ++cnt; off += 16; }
    mo[cnt] = off; so[cnt] = off + 8; ++cnt; off += 16;
    for (int m = 0; m < 5; ++m) { mo[cnt] = off + 8 * m; so[cnt] = off + 40 + 8 * m; ++cnt; }
    for (int k = 0; k < cnt; ++k) {
        double n1 = (double)na, m1 = ld_f64(ra + mo[k]), s1 = ld_f64(ra + so[k]);
        const double n2 = (double)nb, m2 = ld_f64(rbp + mo[k]), s2 = ld_f64(rbp + so[k]);
        const double n = n1 + n2;
        const double d = m2 - m1;
        const double mean = m1 + d * n2 / n;
        const double ss = s1 + s2 + d * d * n1 * n2 / n;
        st_f64(o + mo[k], mean);
        st_f64(o + so[k], ss);
    }
    *reinterpret_cast<uint32_t *>(o) = na + nb;
}

void launch_bond_reduce(const uint8_t *a, const uint8_t *b, int32_t P, int32_t spanning, uint8_t *out,
                        cudaStream_t s) {
    if (P > 0) bond_reduce_kernel<<<(P + 127) / 128, 128, 0, s>>>(a, b, P, spanning, out);
}

// finalized_canonical_averages_dtype (hpc.py:705-749):
//   n u4, p f8, alpha f8, [pp_mean, pp_std, pp_ci 2*f8], strength_mean, strength_std,
//   strength_ci 2*f8, moments_mean 5*f8, moments_std 5*f8, moments_ci 5*2*f8
// Student-t quantiles ppf((1 - conf)/2, df) and ppf((1 + conf)/2, df) for
// the rows of a block: threads 0 and 1 evaluate them once for df0 (the df of
// the block's first row) and share them; a row with another df evaluates its
// own.  Every thread of the block must call this (it synchronises).
struct TPair { double lo, hi; };

__device__ TPair t_pair_block(double conf, double df0, double df, bool active) {
    __shared__ double s_q[2];
    if (threadIdx.x < 2)
        s_q[threadIdx.x] = student_t_quantile(threadIdx.x == 0 ? (1.0 - conf) / 2.0 : (1.0 + conf) / 2.0, df0);
    __syncthreads();
    TPair r;
    if (df == df0) { r.lo = s_q[0]; r.hi = s_q[1]; }
    else if (active) {
        r.lo = student_t_quantile((1.0 - conf) / 2.0, df);
        r.hi = student_t_quantile((1.0 + conf) / 2.0, df);
    } else { r.lo = r.hi = NAN; }
    return r;
}

__device__ void t_interval(const TPair &q, double df, double loc, double scale, double &lo, double &hi) {
    // scipy.stats.t.interval: loc + scale * ppf((1 -+ conf)/2); NaN unless
    // scale > 0 and df > 0.
    if (!(scale > 0.0) || !(df > 0.0) || isnan(loc)) { lo = NAN; hi = NAN; return; }
    lo = loc + scale * q.lo;
    hi = loc + scale * q.hi;
}

__global__ void finalize_kernel(const uint8_t *avg, int32_t P, int32_t spanning, double N, const double *ps,
                                double alpha, uint8_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int nst = spanning ? 7 : 6;
    const size_t in_row = 4 + nst * 16;
    const double conf = 1.0 - alpha;
    // numpy uint32 arithmetic: n - 1 wraps for n = 0
    const uint32_t nu0 = *reinterpret_cast<const uint32_t *>(avg + (size_t)blockIdx.x * blockDim.x * in_row);
    const uint32_t nu_i = i < P ? *reinterpret_cast<const uint32_t *>(avg + (size_t)i * in_row) : nu0;
    const TPair tq = t_pair_block(conf, (double)(uint32_t)(nu0 - 1u), (double)(uint32_t)(nu_i - 1u), i < P);
    if (i >= P) return;
    const uint8_t *a = avg + (size_t)i * in_row;
    uint8_t *o = out + (size_t)i * (spanning ? 244 : 212);
    const uint32_t nu = nu_i;
    const double n = (double)nu;
    const double nm1 = (double)(uint32_t)(nu - 1u);
    const double sqrt_n = sqrt(n);
    *reinterpret_cast<uint32_t *>(o) = nu;
    st_f64(o + 4, ps[i]);
    st_f64(o + 12, alpha);
    int ai = 4, oi = 20;
    auto transform = [&](double mean, double m2, bool normalize, uint8_t *pm, uint8_t *pstd, uint8_t *pci) {
        double mu = mean, sd = sqrt(m2 / nm1);
        if (normalize) { mu /= N; sd /= N; }
        st_f64(pm, mu);
        st_f64(pstd, sd);
        double lo, hi;
        t_interval(tq, nm1, mu, sd / sqrt_n, lo, hi);
        st_f64(pci, lo);
        st_f64(pci + 8, hi);
    };
    if (spanning) {
        transform(ld_f64(a + ai), ld_f64(a + ai + 8), false, o + oi, o + oi + 8, o + oi + 16);
        ai += 16; oi += 32;
    }
    transform(ld_f64(a + ai), ld_f64(a + ai + 8), true, o + oi, o + oi + 8, o + oi + 16);
    ai += 16; oi += 32;
    for (int m = 0; m < 5; ++m)
        transform(ld_f64(a + ai + 8 * m), ld_f64(a + ai + 40 + 8 * m), true, o + oi + 8 * m, o + oi + 40 + 8 * m,
                  o + oi + 80 + 16 * m);
}

void launch_finalize(const uint8_t *avg, int32_t P, int32_t spanning, double N, const double *ps, double alpha,
                     uint8_t *out, cudaStream_t s) {
    if (P > 0) finalize_kernel<<<(P + 63) / 64, 64, 0, s>>>(avg, P, spanning, N, ps, alpha, out);
}

// Microcanonical averages from the run-reduction accumulators, per row n
// (percolate/percolate.py:450-705 and :968-1064): spanning -> Bayesian
// posterior mean (k+1)/(R+2) with Beta(k+1, R-k+1) quantiles at alpha/2 and
// 1 - alpha/2; max and moments -> mean and Student-t interval with scale
// std/sqrt(R), std with ddof 1, (mean, mean) where std == 0; max and moments
// divided by N as microcanonical_averages_arrays returns them.
// out[n * 21 + ...]: span (mean, lo, hi), max (mean, lo, hi), m0..m4 (mean, lo, hi).
// Two threads per row n: half 0 the spanning mean, the lower Beta bound and
// statistics max, m0, m1; half 1 the upper Beta bound and m2, m3, m4 -- the
// Beta quantiles (iterative, FP64) are most of the work, and rows where some
// but not all runs span are contiguous, so splitting them doubles the
// threads working on those rows.
// Of each warp LANES threads have one of these, the others none.
template <int LANES>
__global__ void micro_finalize_kernel(NzMicroAccum acc, uint32_t N, uint32_t M, int32_t spanning, double alpha,
                                      int32_t normalize, double *out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) / 32u * LANES + lane;
    const uint32_t n = lane < (uint32_t)LANES ? t >> 1 : M + 1u, half = t & 1u;
    const double R = (double)*acc.count;
    // every row has R runs: one pair of t quantiles per block
    const TPair tq = t_pair_block(1.0 - alpha, R - 1.0, R - 1.0, n <= M);
    if (n > M) return;
    // value j of row n: out[n * 21 + j], out[j * (M + 1) + n] field-major, or in
    // its array: j / 3 is the statistic, j % 3 its mean, lower or upper bound
    const bool fields = (normalize & NZ_MICRO_FIELD_MAJOR) != 0, arrays = (normalize & NZ_MICRO_ARRAYS) != 0;
    const size_t rows = (size_t)M + 1;
    auto put = [&](int j, double v) {
        size_t at = fields ? j * rows + n : (size_t)n * 21 + j;
        if (arrays) {
            const int f = j / 3, c = j % 3;
            at = f < 2 ? (c == 0 ? 3 * f * rows + n : (3 * f + 1) * rows + 2 * (size_t)n + c - 1)
                       : (c == 0 ? (4 + f) * rows + n : (11 + 2 * (f - 2)) * rows + 2 * (size_t)n + c - 1);
        }
        out[at] = v;
    };
    if (spanning) {
        const double k = (double)acc.span_count[n];
        if (half == 0) {
            put(0, (k + 1.0) / (R + 2.0));
            put(1, beta_quantile(alpha / 2.0, k + 1.0, R - k + 1.0));
        } else {
            put(2, beta_quantile(1.0 - alpha / 2.0, k + 1.0, R - k + 1.0));
        }
    } else if (half == 0) {
        put(0, NAN); put(1, NAN); put(2, NAN);
    }
    const int map[6] = {0, 1, 2, 3, 4, 5};  // max, m0, m1, m2, m3, m4
    for (int j = 3 * (int)half; j < 3 * (int)half + 3; ++j) {
        const size_t idx = (size_t)map[j] * (M + 1) + n;
        const double mean = fma((double)acc.sum_hi[idx], 18446744073709551616.0, (double)acc.sum_lo[idx]) / R;
        const double m2 = acc.m2[idx];
        const double sd = R > 1.0 ? sqrt(m2 / (R - 1.0)) : NAN;
        double lo = mean, hi = mean;
        if (sd > 0.0) {
            const double sc = sd / sqrt(R);
            lo = mean + sc * tq.lo;
            hi = mean + sc * tq.hi;
        }
        const double scale = (normalize & 1) ? (double)N : 1.0;
        put(3 + 3 * j, mean / scale);
        put(4 + 3 * j, lo / scale);
        put(5 + 3 * j, hi / scale);
    }
}

void launch_micro_finalize(const NzMicroAccum &acc, uint32_t N, uint32_t M, int32_t spanning, double alpha,
                           int32_t normalize, double *out, cudaStream_t s) {
    // blocks of one warp while that is few blocks: the rows with iterated
    // quantiles are neighbours, and several of their warps on one SM queue for
    // its FP64 unit (the rows of 128 threads on one SM: 1.5 against 0.63 ms for
    // 10^5 runs of 32 x 32, with the binomial sums of nz_math.cuh in the second
    // figure).  Every block works out its own t quantiles, which the 32,700
    // one-warp blocks of a 512 x 512 grid pay for (4.5 against 1.7 ms).
    const uint64_t threads = 2ull * ((uint64_t)M + 1);
    // Where warps of 8 rows' halves still find a quarter of an SM each, they
    // are shorter than full ones, in which the slowest of 32 quantiles counts
    // (10^4 runs of 32 x 32 346 -> 256 us, 6 10^4 556 -> 384; 1,000 of 48 x 48,
    // beyond, 203 and 219).
    if (threads <= 8u * 4u * 152u) {
        micro_finalize_kernel<8><<<(unsigned)((threads + 7) / 8), 32, 0, s>>>(acc, N, M, spanning, alpha, normalize, out);
        return;
    }
    const unsigned block = threads <= 80000 ? 32 : 128;
    micro_finalize_kernel<32><<<(unsigned)((threads + block - 1) / block), block, 0, s>>>(acc, N, M, spanning, alpha,
                                                                                         normalize, out);
}

__global__ void t_quantile_kernel(const double *q, const double *df, int32_t count, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) out[i] = student_t_quantile(q[i], df[i]);
}

void launch_t_quantile(const double *q, const double *df, int32_t count, double *out, cudaStream_t s) {
    if (count > 0) t_quantile_kernel<<<(count + 127) / 128, 128, 0, s>>>(q, df, count, out);
}

}  // namespace nz
