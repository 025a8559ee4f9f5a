// nz_mlp.cu -- MLP surrogate of the canonical curves: forward, backward, Adam.
//
// A fully connected network with GELU hidden activations (erf form) and a
// linear output layer.  Every GEMM takes BF16 operands -- activations and
// gradients are rounded to BF16 (round-to-nearest-even) where they enter a
// product -- and accumulates in FP32; biases, activations, the loss and the
// optimizer state are FP32.  (The surrogate has no counterpart in the
// reference; it serves the p-grid placement and the choice of the next
// lattice size, with the Monte Carlo estimate as its fallback and judge.)
//
// Parameter layout (one flat FP32 buffer, mirrored as BF16 for products):
// for layer l = 0..n_layers-1: W_l [in_l][out_l] row-major, then b_l [out_l].
#include <algorithm>
#include <cstdint>
#include <cuda_bf16.h>

#include "nz_common.cuh"
#include "nz_internal.cuh"
#include "nz_tc.cuh"

namespace nz {

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// The kernels of a step run one after the other, each for a few microseconds.
// Each lets the next one start at once (its blocks take their places, set up
// their barriers and TMEM) and waits itself, before its first access to global
// memory, until the one before it is complete (programmatic dependent launch).
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
static void launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute overlap;
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &overlap;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// ---------------------------------------------------------------------
// GEMM on the tensor cores: tcgen05.mma kind::f16 with BF16 operands and an
// FP32 accumulator in TMEM
// ---------------------------------------------------------------------
// C[m][n] = sum_k A(m, k) B(k, n), with the epilogues of GemmOut; A(m, k) =
// A[m * sam + k * sak] (FP32, rounded to BF16 as it is staged), B(k, n) =
// B[k * sbk + n * sbn] (BF16, or FP32 rounded to BF16).
//
// One CTA of 256 threads per 128 x ntile tile of C (ntile 16, 32 or 64): the
// threads stage 64-deep K chunks of A (128 rows) and B (ntile rows) into shared
// memory as BF16 in the canonical no-swizzle K-major layout (8-row x 16-byte
// core matrices, K-adjacent ones 128 bytes apart, 8-row groups 1 KB apart),
// double-buffered; one thread issues four 128 x ntile x 16 MMAs per chunk and
// commits them to the chunk's mbarrier; thread t reads row t % 128 of the
// accumulator out of TMEM (tcgen05.ld) for the epilogue, threads 128 .. 255 the
// upper half of the columns.  Every mbarrier wait gives up after 1 s: the tile
// is then written as NaN and counted in g_mlp_errors (nz_mlp_take_errors).
//
// These GEMMs are tiny (batch 4096 x 128 x 128); the staging bounds them.  A
// thread stages 8 consecutive K of one row at a time: two 16-byte loads where K
// is contiguous in memory, else 8 loads that are coalesced over the rows, and
// one 16-byte shared-memory store whose 8-lane phases cover 128 bytes; all loads
// of a chunk, and of the epilogue, are issued before the first is used.  A
// launch by itself, from cold caches, takes 10 to 17 us; one element at a time, with
// two divisions each and 2-byte stores, it took 38.  A step of 22 launches takes 176
// us, 210 when each waits for the one before to drain.  64-column tiles put 64 CTAs on a batch of 4096.
constexpr int kGM = 128;   // rows of C per CTA (TMEM lanes)
constexpr int kGK = 64;    // K per staged chunk: 4 MMAs of K = 16
constexpr int kGN = 64;    // largest column tile
constexpr int kGThreads = 256;
constexpr uint32_t kGSbo = (kGK / 8) * tc::kCoreBytes;

struct GemmSmem {
    __nv_bfloat16 a[2][kGM * kGK];
    __nv_bfloat16 b[2][kGN * kGK];
    float2 part[kGThreads];
    float bias[kGN];
    uint64_t mbar[2];
    uint32_t tmem;
};

// A running FP32 sum and its rounding errors.
struct ColSum {
    float s = 0.0f, c = 0.0f;
    __device__ __forceinline__ void add(float x) {
        const float t = s + x, b = t - s;  // TwoSum
        c += (s - (t - b)) + (x - b);
        s = t;
    }
    __device__ __forceinline__ void add8(const float (&v)[8]) {
        add(((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
    }
    // (of a sum with an infinity the errors are no numbers, and the sum is what it is)
    __device__ __forceinline__ float value() const { return isfinite(c) ? s + c : s; }
};

__device__ uint32_t g_mlp_errors;  // tiles whose mbarrier waits gave up

// Where the product goes.  kPlain: C = acc (+ bias), and Z too if given.  kGelu:
// Z = acc + bias, C = GELU(Z).  kBack: C = acc * GELU'(Z) (the gradient of the
// layer's pre-activations from that of its activations).
enum class Epi { kPlain, kGelu, kBack };
struct GemmOut {
    Epi epi;
    const float *bias;
    float *Z;
    float *C;
    int ldc;
    int64_t slice;   // floats from one K slice's C to the next
    float *colsum;   // sums over K of B's FP32 values (the bias gradient), at slice * `slice`; or null
};

// Instruction descriptor of kind::f16: D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bits
// 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t bf16_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kGM >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// The 8 values (row, k0 .. k0 + 7) of an operand, zero outside rows x K, as
// BF16 bits or FP32.  WIDE: K contiguous, every row and k0 at a 16-byte
// boundary, K a multiple of 8.  Branch-free, so that a thread's loads overlap.
template <bool WIDE, class T>
__device__ __forceinline__ void load8(const T *src, int64_t s_row, int64_t s_k, int row, int rows, int k0, int K,
                                      float (&v)[8]) {
    const bool in = row < rows && k0 < K;
    const T *p = src + (in ? row * s_row + k0 * s_k : 0);
    if constexpr (WIDE && sizeof(T) == 4) {
        const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float4 a = in ? reinterpret_cast<const float4 *>(p)[0] : zero;
        const float4 b = in ? reinterpret_cast<const float4 *>(p)[1] : zero;
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else if constexpr (WIDE) {
        const uint4 a = in ? *reinterpret_cast<const uint4 *>(p) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[2 * i] = __uint_as_float(w[i] << 16);
            v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = in && k0 + i < K ? (float)p[i * s_k] : 0.0f;
    }
}

// One K chunk of an operand (`rows` of its source's rows from row0 on, `tile`
// <= TILE of them staged) into core matrices, all its loads before the first
// store.  colsum: += this thread's values of row t % tile.
template <int TILE, bool WIDE, bool COLSUM, class T>
__device__ __forceinline__ void stage_operand(__nv_bfloat16 *dst, const T *src, int64_t s_row, int64_t s_k, int row0,
                                              int rows, int tile, int k0, int K, ColSum &colsum) {
    const bool k_fast = s_k == 1 && !COLSUM;
    // items: (row, group of 8 k).  K contiguous: 8 rows x 4 groups per warp
    // (128 contiguous bytes of each row); else 32 rows per warp
    constexpr int kItems = TILE * (kGK / 8) / kGThreads;
    float v[kItems][8];
    int at[kItems];
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        const int i = threadIdx.x + q * kGThreads;
        const int row = k_fast ? (i & 7) + ((i >> 6) << 3) : i % tile;
        const int kc = k_fast ? (i >> 3) & 7 : i / tile;
        at[q] = i < tile * (kGK / 8) ? (row >> 3) * (int)(kGSbo / 2) + kc * 64 + (row & 7) * 8 : -1;
        load8<WIDE>(src, s_row, s_k, row0 + row, at[q] >= 0 ? rows : 0, k0 + kc * 8, K, v[q]);
    }
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        if (COLSUM) colsum.add8(v[q]);
        if (at[q] >= 0)
            *reinterpret_cast<uint4 *>(dst + at[q]) =
                make_uint4(pack_bf16(v[q][0], v[q][1]), pack_bf16(v[q][2], v[q][3]), pack_bf16(v[q][4], v[q][5]),
                           pack_bf16(v[q][6], v[q][7]));
    }
}

template <class T>
struct GemmIn {
    const float *A;
    int sam, sak;
    const T *B;
    int sbk, sbn;
};

// A_WIDE, B_WIDE: operands with K contiguous, in 16-byte loads; B of type T
template <bool A_WIDE, bool B_WIDE, class T>
__global__ void __launch_bounds__(kGThreads) mlp_gemm_kernel(int M, int N, int K, GemmIn<T> in, GemmOut out, int ntile,
                                                             int k_split) {
    extern __shared__ __align__(1024) uint8_t gemm_smem[];
    GemmSmem &sh = *reinterpret_cast<GemmSmem *>(gemm_smem);
    const int t = threadIdx.x, warp = t >> 5;
    const int m0 = blockIdx.y * kGM, n0 = blockIdx.x * ntile;
    // split-K: this CTA's K range [kb, kb + k_split); its tile goes to slice
    // blockIdx.z of C
    const int kb = blockIdx.z * k_split;
    K = min(K - kb, k_split);
    float *C = out.C + blockIdx.z * out.slice;
    const float *A = in.A + (int64_t)kb * in.sak;
    constexpr bool kSums = sizeof(T) == 4;  // FP32 B: the gradient of the pre-activations
    // TMEM: a power of two >= 32.  The weight gradients (long sums over the batch, in
    // FP32 that the tensor cores round toward zero) have two accumulators, of half a
    // slice's chunks each: 16 slices are as accurate as 32 were (positive values,
    // 8,192 samples: 2.6e-8 of the sum on average, 2.3e-7 with one accumulator)
    const uint32_t acc_cols = ntile <= 32 ? 32u : 64u, cols = kSums ? 2u * acc_cols : acc_cols;
    start_next();
    // rows t % 128 of C; threads 128 .. 255 take columns 32 .. 63
    const int m = m0 + (t & 127), j0 = (t >> 7) * 32;
    const int64_t row = (int64_t)m * out.ldc + n0 + j0;
    const bool whole = ((reinterpret_cast<uintptr_t>(C) | reinterpret_cast<uintptr_t>(out.Z)) & 15u) == 0 &&
                       n0 + j0 + 32 <= N && ntile >= 32 && (out.ldc & 3) == 0;
    if (warp == 0) tc::tmem_alloc(tc::smem_u32(&sh.tmem), cols);
    if (t == 0) {
        tc::mbar_init(tc::smem_u32(&sh.mbar[0]));
        tc::mbar_init(tc::smem_u32(&sh.mbar[1]));
        tc::mbar_init_fence();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sh.tmem;
    wait_previous();
    if (t < ntile) sh.bias[t] = out.bias && n0 + t < N ? out.bias[n0 + t] : 0.0f;
    const int nch = (K + kGK - 1) / kGK, half = kSums ? (nch + 1) / 2 : nch;  // chunks of the first accumulator
    ColSum colsum, none;
    const bool sums = kSums && out.colsum && blockIdx.y == 0;
    const T *B = in.B + (int64_t)kb * in.sbk;
    auto stage = [&](int c, int buf) {
        stage_operand<kGM, A_WIDE, false>(sh.a[buf], A, in.sam, in.sak, m0, M, kGM, c * kGK, K, none);
        stage_operand<kGN, B_WIDE, kSums>(sh.b[buf], B, in.sbn, in.sbk, n0, N, ntile, c * kGK, K, colsum);
    };
    stage(0, 0);
    bool bad = false;
    int c = 0;
    for (; c < nch; ++c) {
        const int buf = c & 1;
        tc::fence_async_smem();
        tc::fence_before();
        if (__syncthreads_or(bad)) break;  // a wait below gave up
        if (t == 0) {
            tc::fence_after();
            const uint32_t a0 = tc::smem_u32(sh.a[buf]), b0 = tc::smem_u32(sh.b[buf]);
#pragma unroll
            for (int ks = 0; ks < kGK / 16; ++ks) {
                const uint32_t o = (uint32_t)ks * 2 * tc::kCoreBytes;  // K = 16: two core matrices
                mma_bf16(c < half ? tmem : tmem + acc_cols, tc::smem_desc(a0 + o, tc::kCoreBytes, kGSbo),
                         tc::smem_desc(b0 + o, tc::kCoreBytes, kGSbo), bf16_idesc(ntile),
                         ((c > 0 && c != half) || ks > 0) ? 1u : 0u);
            }
            tc::mma_commit(tc::smem_u32(&sh.mbar[buf]));
        }
        if (c + 1 < nch) {
            // the other buffer is free once the MMAs of chunk c - 1 are done
            if (c >= 1) bad = !tc::mbar_wait(tc::smem_u32(&sh.mbar[(c - 1) & 1]), ((c - 1) >> 1) & 1);
            if (!bad) stage(c + 1, (c + 1) & 1);
        }
    }
    // MMAs complete in order: the last chunk issued covers them all
    if (c > 0 && !tc::mbar_wait(tc::smem_u32(&sh.mbar[(c - 1) & 1]), ((c - 1) >> 1) & 1)) bad = true;
    sh.part[t] = make_float2(colsum.s, colsum.c);
    tc::fence_before();
    const bool any_bad = __syncthreads_or(bad) || c < nch;
    tc::fence_after();
    if (j0 < ntile) {
        float v[32], z[32];
        // all loads of the epilogue before its first store
        if (out.epi == Epi::kBack && m < M) {
            if (whole) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 q = *reinterpret_cast<const float4 *>(out.Z + row + j);
                    z[j] = q.x; z[j + 1] = q.y; z[j + 2] = q.z; z[j + 3] = q.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) z[j] = j0 + j < ntile && n0 + j0 + j < N ? out.Z[row + j] : 0.0f;
            }
        }
        if (any_bad) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __int_as_float(0x7fc00000);
            if (t == 0) atomicAdd(&g_mlp_errors, 1u);
        } else {
            const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)j0;
            tc::tmem_ld32(at, v);
            if constexpr (kSums) {
                if (half < nch) {
                    tc::tmem_ld32(at + acc_cols, z);
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] += z[j];
                }
            }
        }
        if (m < M) {
            const bool store_z = out.Z && out.epi != Epi::kBack;
            if (out.epi == Epi::kBack) {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] *= gelu_grad(z[j]);
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) z[j] = v[j] + (j0 + j < ntile ? sh.bias[j0 + j] : 0.0f);
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = out.epi == Epi::kGelu ? gelu(z[j]) : z[j];
            }
            if (whole) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    *reinterpret_cast<float4 *>(C + row + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                    if (store_z)
                        *reinterpret_cast<float4 *>(out.Z + row + j) = make_float4(z[j], z[j + 1], z[j + 2], z[j + 3]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (j0 + j >= ntile || n0 + j0 + j >= N) continue;
                    C[row + j] = v[j];
                    if (store_z) out.Z[row + j] = z[j];
                }
            }
        }
    }
    // column sums: the threads that staged one column, in order
    if (sums && t < ntile && n0 + t < N) {
        ColSum x;
        for (int q = t; q < kGThreads; q += ntile) {
            x.add(sh.part[q].x);
            x.c += sh.part[q].y;
        }
        out.colsum[blockIdx.z * out.slice + n0 + t] = any_bad ? __int_as_float(0x7fc00000) : x.value();
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        tc::tmem_dealloc(tmem, cols);
    }
}

// slices of `count` values, `stride` floats apart, summed in order into out
// (deterministic split-K): the weight gradient and, after it, the bias gradient
__global__ void splitk_sum_kernel(const float *slices, int splits, int64_t stride, int64_t count, float *out) {
    start_next();
    wait_previous();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        ColSum acc;
#pragma unroll 8
        for (int z = 0; z < splits; ++z) acc.add(slices[z * stride + i]);
        out[i] = acc.value();
    }
}

// Launches the product; `splits` K slices of k_split (1 slice: k_split = K).
template <class T>
static void gemm(int M, int N, int K, const GemmIn<T> &in, const GemmOut &out, int splits, int k_split,
                 cudaStream_t s) {
    if (M <= 0 || N <= 0) return;
    const int ntile = N > 32 ? kGN : (N > 16 ? 32 : 16);
    auto aligned = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    // slices begin at multiples of kGK, so every 8-k group does at one of 8
    const bool a_wide = in.sak == 1 && (in.sam & 3) == 0 && (K & 7) == 0 && aligned(in.A);
    const bool b_wide = sizeof(T) == 2 && in.sbk == 1 && (K & 7) == 0 && (in.sbn & 7) == 0 && aligned(in.B);
    auto launch = [&](auto *kernel) {
        // above 48 KB of dynamic shared memory the launch needs the attribute,
        // which belongs to the function in the current device's context
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GemmSmem));
        dim3 grid((N + ntile - 1) / ntile, (M + kGM - 1) / kGM, splits);
        launch_chained(kernel, grid, kGThreads, sizeof(GemmSmem), s, M, N, K, in, out, ntile, k_split);
    };
    if constexpr (sizeof(T) == 2) {
        if (a_wide && b_wide) launch(mlp_gemm_kernel<true, true, T>);
        else if (a_wide) launch(mlp_gemm_kernel<true, false, T>);
        else launch(mlp_gemm_kernel<false, false, T>);
    } else {
        launch(mlp_gemm_kernel<false, false, T>);
    }
}

__global__ void to_bf16_kernel(const float *a, __nv_bfloat16 *b, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = __float2bfloat16_rn(a[i]);
}

// Weighted squared error: loss = sum_{b,o} w[b][o] (y - t)^2 / B ; dY = 2 w (y - t) / B
__global__ void mse_kernel(const float *Y, const float *T, const float *Wt, int B, int N, float *dY,
                           float *loss_parts) {
    start_next();
    wait_previous();
    float s = 0.0f;
    const int64_t n = (int64_t)B * N;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float w = Wt ? Wt[i] : 1.0f;
        const float d = Y[i] - T[i];
        s += w * d * d;
        dY[i] = 2.0f * w * d / (float)B;
    }
    __shared__ float red[256];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (threadIdx.x < (unsigned)off) red[threadIdx.x] += red[threadIdx.x + off];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss_parts[blockIdx.x] = red[0] / (float)B;
}

__global__ void adam_kernel(float *p, const float *g, float *m, float *v, __nv_bfloat16 *pb, int64_t n, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
    start_next();
    wait_previous();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        pb[i] = __float2bfloat16_rn(pi);
    }
}

}  // namespace nz

using namespace nz;

namespace {
int param_offsets(const int32_t *widths, int32_t n_layers, int64_t *w_off, int64_t *b_off) {
    int64_t o = 0;
    for (int l = 0; l < n_layers; ++l) {
        if (widths[l] <= 0 || widths[l + 1] <= 0 || widths[l] > 4096 || widths[l + 1] > 4096) return NZ_ERR_INVALID;
        w_off[l] = o;
        o += (int64_t)widths[l] * widths[l + 1];
        b_off[l] = o;
        o += widths[l + 1];
    }
    return NZ_OK;
}
constexpr int kMaxLayers = 16;
inline int blocks_for(int64_t n) { int64_t b = (n + 255) / 256; return (int)(b > 4096 ? 4096 : (b < 1 ? 1 : b)); }
}  // namespace

extern "C" {

int64_t nz_mlp_param_count(const int32_t *widths, int32_t n_layers) {
    if (!widths || n_layers <= 0 || n_layers > kMaxLayers) return -1;
    int64_t w[kMaxLayers], b[kMaxLayers];
    if (param_offsets(widths, n_layers, w, b) != NZ_OK) return -1;
    return b[n_layers - 1] + widths[n_layers];
}

int64_t nz_mlp_activation_count(const int32_t *widths, int32_t n_layers, int32_t batch) {
    if (!widths || n_layers <= 0 || n_layers > kMaxLayers || batch <= 0) return -1;
    int64_t s = 0;
    for (int l = 1; l <= n_layers; ++l) s += (int64_t)batch * widths[l];
    return s;
}

int nz_mlp_params_to_bf16(const float *params, int64_t count, void *params_bf16, void *stream) {
    if (!params || !params_bf16 || count <= 0) return NZ_ERR_INVALID;
    to_bf16_kernel<<<blocks_for(count), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        params, reinterpret_cast<__nv_bfloat16 *>(params_bf16), count);
    return cudaGetLastError() == cudaSuccess ? NZ_OK : NZ_ERR_CUDA;
}

int nz_mlp_forward(const int32_t *widths, int32_t n_layers, int32_t batch, const float *x, const float *params,
                   const void *params_bf16, float *z, float *h, float *y, void *stream) {
    if (!widths || n_layers <= 0 || n_layers > kMaxLayers || batch <= 0 || !x || !params || !params_bf16 || !z ||
        !h || !y)
        return NZ_ERR_INVALID;
    int64_t wo[kMaxLayers], bo[kMaxLayers];
    if (param_offsets(widths, n_layers, wo, bo) != NZ_OK) return NZ_ERR_INVALID;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const __nv_bfloat16 *pb = reinterpret_cast<const __nv_bfloat16 *>(params_bf16);
    const float *in = x;
    int64_t act = 0;
    for (int l = 0; l < n_layers; ++l) {
        const int K = widths[l], N = widths[l + 1];
        const bool last = l == n_layers - 1;
        float *zl = z + act, *hl = last ? y : h + act;
        const GemmIn<__nv_bfloat16> g{in, K, 1, pb + wo[l], N, 1};
        gemm(batch, N, K, g, GemmOut{last ? Epi::kPlain : Epi::kGelu, params + bo[l], zl, hl, N, 0, nullptr}, 1, K, s);
        in = hl;
        act += (int64_t)batch * N;
    }
    return cudaGetLastError() == cudaSuccess ? NZ_OK : NZ_ERR_CUDA;
}

int nz_mlp_loss(const float *y, const float *target, const float *weight, int32_t batch, int32_t n_out,
                float *dy, float *loss_parts, int32_t n_parts, void *stream) {
    if (!y || !target || !dy || !loss_parts || batch <= 0 || n_out <= 0 || n_parts <= 0) return NZ_ERR_INVALID;
    launch_chained(mse_kernel, dim3(n_parts), 256, 0, reinterpret_cast<cudaStream_t>(stream), y, target, weight, batch,
                   n_out, dy, loss_parts);
    return cudaGetLastError() == cudaSuccess ? NZ_OK : NZ_ERR_CUDA;
}

// dy: gradient of the loss w.r.t. the output [batch][n_out]; z, h from the
// forward pass; grads: flat FP32 gradient (same layout as params);
// scratch: 2 * batch * max(width) floats.
int nz_mlp_backward(const int32_t *widths, int32_t n_layers, int32_t batch, const float *x, const void *params_bf16,
                    const float *z, const float *h, const float *dy, float *grads, float *scratch, void *stream) {
    if (!widths || n_layers <= 0 || n_layers > kMaxLayers || batch <= 0 || !x || !params_bf16 || !z || !h ||
        !dy || !grads || !scratch)
        return NZ_ERR_INVALID;
    int64_t wo[kMaxLayers], bo[kMaxLayers];
    if (param_offsets(widths, n_layers, wo, bo) != NZ_OK) return NZ_ERR_INVALID;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const __nv_bfloat16 *pb = reinterpret_cast<const __nv_bfloat16 *>(params_bf16);
    int wmax = 0;
    for (int l = 0; l <= n_layers; ++l) wmax = widths[l] > wmax ? widths[l] : wmax;
    int64_t act_off[kMaxLayers];
    int64_t a = 0;
    for (int l = 0; l < n_layers; ++l) { act_off[l] = a; a += (int64_t)batch * widths[l + 1]; }
    // dZ of the last (linear) layer = dy; the other layers' in turn in the two
    // halves of the scratch, whose other half holds the weight gradient's slices
    const int64_t half = (int64_t)batch * wmax;
    const float *dZ = dy;
    int other = 0;  // the half that dZ is not in
    for (int l = n_layers - 1; l >= 0; --l) {
        const int K = widths[l], N = widths[l + 1];
        float *spare = scratch + other * half;
        // dW[K][N] = A^T dZ and db[N] = column sums of dZ: the reduction over
        // the batch is split into up to 16 slices (dW, then db), summed in
        // order; 32 slices would not leave room for db at K = N = wmax
        const int64_t per_slice = (int64_t)K * N + N;
        int splits = (int)std::min<int64_t>(16, half / per_slice);
        int k_split = batch;
        if (splits > 1) {
            k_split = ((batch + splits - 1) / splits + kGK - 1) / kGK * kGK;
            splits = (batch + k_split - 1) / k_split;
        }
        if (splits < 2) { splits = 1; k_split = batch; }
        float *dst = splits > 1 ? spare : grads + wo[l];
        const GemmIn<float> g{l == 0 ? x : h + act_off[l - 1], 1, K, dZ, N, 1};
        gemm(K, N, batch, g, GemmOut{Epi::kPlain, nullptr, nullptr, dst, N, per_slice, dst + (int64_t)K * N}, splits,
             k_split, s);
        if (splits > 1)
            launch_chained(splitk_sum_kernel, dim3(blocks_for(per_slice)), 256, 0, s, spare, splits, per_slice,
                           per_slice, grads + wo[l]);
        if (l == 0) break;
        // dZ of layer l - 1 = (dZ W^T) * GELU'(z)  (W[K][N]: B(k=n, n=k) = W[k][n])
        const GemmIn<__nv_bfloat16> b{dZ, N, 1, pb + wo[l], 1, N};
        gemm(batch, K, N, b, GemmOut{Epi::kBack, nullptr, const_cast<float *>(z) + act_off[l - 1], spare, K, 0, nullptr},
             1, N, s);
        dZ = spare;
        other ^= 1;
    }
    return cudaGetLastError() == cudaSuccess ? NZ_OK : NZ_ERR_CUDA;
}

int nz_mlp_take_errors(uint32_t *count) {
    if (!count) return NZ_ERR_INVALID;
    const uint32_t zero = 0;
    if (cudaMemcpyFromSymbol(count, g_mlp_errors, sizeof(uint32_t)) != cudaSuccess ||
        cudaMemcpyToSymbol(g_mlp_errors, &zero, sizeof(uint32_t)) != cudaSuccess)
        return NZ_ERR_CUDA;
    return NZ_OK;
}

int nz_mlp_adam(float *params, const float *grads, float *m, float *v, void *params_bf16, int64_t count,
                float lr, float beta1, float beta2, float eps, int32_t step, void *stream) {
    if (!params || !grads || !m || !v || !params_bf16 || count <= 0 || step <= 0) return NZ_ERR_INVALID;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    launch_chained(adam_kernel, dim3(blocks_for(count)), 256, 0, reinterpret_cast<cudaStream_t>(stream), params, grads, m,
                   v, reinterpret_cast<__nv_bfloat16 *>(params_bf16), count, lr, beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? NZ_OK : NZ_ERR_CUDA;
}

}  // extern "C"
