// nz_mt.cu -- the permutations numpy's legacy RandomState draws.
//
// MT19937 (Matsumoto & Nishimura 1998) with the authors' init_genrand and
// init_by_array seeding, and the Fisher-Yates shuffle with masked rejection
// of RandomState.permutation(M): for i = M - 1 .. 1 the next outputs, masked
// to i's bits, until one is <= i, then a swap of o[i] with o[that].
//
// One block of 8 warps per stream.  The stream is sequential, but its parts
// run as a pipeline of one step per 624 outputs:
//   warps 2..7  the next 624 state words (three dependent thirds) and their
//               tempered outputs;
//   warp 0      which of the current outputs are drawn: 32 at a time, lane k's
//               bound i - (draws before it) from a ballot that is repeated
//               until it agrees with itself (lane k is right after k + 1
//               ballots at the latest, mostly after 2), up to the place where
//               i's mask changes; the drawn ones go into a ring;
//   warp 1      the swaps, 32 at a time as far as none depends on an earlier
//               one (same partner, or an earlier partner's place).
// o is 16 bits per element in shared memory up to M = 65,536, else the output
// array itself.  The dependent steps of warps 0 and 1 bound it.  M = 65,160
// (one run of a 181 x 181 grid): 0.66 ms; 40 permutations of 3,120 from one
// stream: 1.74 ms.  One thread per stream, its state in local memory and its
// swaps in global memory, took 17.8 and 21.5 ms.
#include <cstdint>

#include "nz_common.cuh"
#include "nz_internal.cuh"

namespace nz {
namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kTwisters = kThreads - 64;  // threads of warps 2..7
constexpr uint32_t kRing = 2048;               // draws between warps 0 and 1 (>= 2 x 624)
constexpr uint32_t kSmallM = 65536;

__device__ __forceinline__ uint32_t temper(uint32_t y) {
    y ^= (y >> 11);
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= (y >> 18);
    return y;
}

struct MtShared {
    uint32_t mt[2][624];   // state words: the block being drawn from, and the next
    uint32_t out[2][624];  // their tempered outputs
    uint32_t ring[kRing];
    uint32_t head, tail;   // draws pushed, swaps done, both since the start
    uint32_t pos;          // outputs of the current block used up
    uint32_t runs_drawn;
    uint32_t i_draw, i_swap;
    uint32_t run_ready;    // all swaps of the current run are done
};

__device__ void init_genrand(uint32_t *mt, uint32_t seed) {
    uint32_t x = seed;
    mt[0] = x;
    for (int i = 1; i < 624; ++i) mt[i] = x = 1812433253u * (x ^ (x >> 30)) + (uint32_t)i;
}

__device__ void init_by_array(uint32_t *mt, const uint32_t *key, int len) {
    init_genrand(mt, 19650218u);
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
}

// Warps 2..7 (thread t of kTwisters): the state words and outputs after `cur`.
__device__ __forceinline__ void next_block(const uint32_t *cur, uint32_t *next, uint32_t *out, uint32_t t) {
    auto word = [&](uint32_t kk, uint32_t src, uint32_t after) {
        const uint32_t y = (cur[kk] & 0x80000000u) | (after & 0x7fffffffu);
        const uint32_t v = src ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
        next[kk] = v;
        out[kk] = temper(v);
    };
    for (uint32_t kk = t; kk < 227; kk += kTwisters) word(kk, cur[kk + 397], cur[kk + 1]);
    asm volatile("bar.sync 1, %0;" ::"n"(kTwisters) : "memory");
    for (uint32_t kk = 227 + t; kk < 454; kk += kTwisters) word(kk, next[kk - 227], cur[kk + 1]);
    asm volatile("bar.sync 1, %0;" ::"n"(kTwisters) : "memory");
    for (uint32_t kk = 454 + t; kk < 624; kk += kTwisters) word(kk, next[kk - 227], kk == 623 ? next[0] : cur[kk + 1]);
}

// Warp 0: draws from the rest of the current block of outputs.
__device__ __forceinline__ void draw(MtShared &sh, const uint32_t *out, uint32_t M, uint32_t runs, uint32_t lane) {
    uint32_t pos = sh.pos, head = sh.head, i = sh.i_draw, drawn = sh.runs_drawn;
    const uint32_t before = (1u << lane) - 1u;
    while (pos < 624 && drawn < runs) {
        const uint32_t mask = 0xffffffffu >> __clz(i), low = (mask >> 1) + 1u;  // low <= i <= mask
        const int32_t v = pos + lane < 624 ? (int32_t)(out[pos + lane] & mask) : 0x7fffffff;
        uint32_t a = __ballot_sync(0xffffffffu, v <= (int32_t)i);
        for (int k = 0; k < 32; ++k) {
            const uint32_t b = __ballot_sync(0xffffffffu, v <= (int32_t)i - (int32_t)__popc(a & before));
            if (b == a) break;
            a = b;
        }
        uint32_t used = min(32u, 624u - pos), count = __popc(a);
        const uint32_t room = i - low + 1u;  // draws until the mask changes
        if (count >= room) {
            const bool makes_last = ((a >> lane) & 1u) && __popc(a & before) == room - 1u;
            const uint32_t last = __ffs(__ballot_sync(0xffffffffu, makes_last)) - 1;
            a &= 0xffffffffu >> (31u - last);
            count = room;
            used = last + 1u;
        }
        if ((a >> lane) & 1u) sh.ring[(head + __popc(a & before)) % kRing] = (uint32_t)v;
        head += count;
        i -= count;
        pos += used;
        if (i == 0) {
            ++drawn;
            i = M - 1u;
        }
    }
    if (lane == 0) {
        sh.pos = pos;
        sh.head = head;
        sh.i_draw = i;
        sh.runs_drawn = drawn;
    }
}

// Warp 1: the swaps of the draws up to `head`, at most to the end of the run.
template <class T>
__device__ __forceinline__ void swaps(MtShared &sh, T *o, uint32_t head, uint32_t lane) {
    uint32_t tail = sh.tail, top = sh.i_swap;
    while (tail != head && top > 0) {
        uint32_t n = min(min(32u, head - tail), top);
        const bool on = lane < n;
        const uint32_t j = on ? sh.ring[(tail + lane) % kRing] : 0xffffffffu - lane, i = top - lane;
        // swap k depends on an earlier one that has the same partner, or
        // whose partner is its own place
        const uint32_t same = __match_any_sync(0xffffffffu, j) & ((1u << lane) - 1u);
        const uint32_t d = top - j;
        const uint32_t hit = __reduce_or_sync(0xffffffffu, on && d < 32u && d > lane ? 1u << d : 0u);
        const uint32_t dep = __ballot_sync(0xffffffffu, on && (same != 0 || ((hit >> lane) & 1u)));
        if (dep) n = min(n, (uint32_t)__ffs(dep) - 1u);
        T a = 0, b = 0;
        if (lane < n) {
            a = o[i];
            b = o[j];
        }
        __syncwarp();
        if (lane < n) {
            o[i] = b;
            o[j] = a;
        }
        __syncwarp();
        tail += n;
        top -= n;
    }
    if (lane == 0) {
        sh.tail = tail;
        sh.i_swap = top;
        sh.run_ready = top == 0;
    }
}

// Block b shuffles `runs` permutations of range(M) one after another from one
// stream into out[(b * runs + k) * M + i].  Seeded by seed_words / seed_len
// (row b; length 0: a scalar), or continuing the stream state_in (624 words
// and the position) and storing it in state_out where numpy would leave it.
template <bool SMALL>
__global__ void __launch_bounds__(kThreads) mt_perm_kernel(uint32_t M, uint32_t runs, const uint32_t *seed_words,
                                                           const int32_t *seed_len, int32_t stride,
                                                           const uint32_t *state_in, uint32_t *state_out,
                                                           uint32_t *out) {
    extern __shared__ __align__(16) uint16_t s_o[];
    __shared__ MtShared sh;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t top = M > 1 ? M - 1u : 0u;  // no draws for one element or none
    uint32_t *dst = out + (size_t)blockIdx.x * runs * M;
    if (state_in) {
        for (uint32_t k = t; k < 624; k += kThreads) sh.mt[0][k] = state_in[k];
    } else if (t == 0) {
        const int len = seed_len[blockIdx.x];
        const uint32_t *w = seed_words + (size_t)blockIdx.x * stride;
        if (len == 0) init_genrand(sh.mt[0], w[0]);
        else init_by_array(sh.mt[0], w, len);
    }
    if (t == 0) {
        sh.head = sh.tail = 0;
        sh.pos = state_in ? min(state_in[624], 624u) : 624u;
        sh.runs_drawn = top > 0 ? 0 : runs;
        sh.i_draw = sh.i_swap = top;
        sh.run_ready = 0;
    }
    auto identity = [&](uint32_t *o) {
        for (uint32_t i = t; i < M; i += kThreads) {
            if (SMALL) s_o[i] = (uint16_t)i;
            else o[i] = i;
        }
    };
    identity(dst);
    __syncthreads();
    for (uint32_t k = t; k < 624; k += kThreads) sh.out[0][k] = temper(sh.mt[0][k]);
    uint32_t cur = 0, done = 0;
    bool next_ready = false;
    while (done < runs) {
        __syncthreads();
        // what this step works on, read by every thread before any warp moves it
        const uint32_t head = sh.head, fill = head - sh.tail, pos = sh.pos;
        const bool wanted = sh.runs_drawn < runs;
        __syncthreads();
        if (pos >= 624 && next_ready && wanted) {  // on to the next block of outputs
            if (t == 0) sh.pos = 0;
            cur ^= 1u;
            next_ready = false;
            continue;
        }
        if (warp == 0) {
            if (pos < 624 && kRing - fill >= 624) draw(sh, sh.out[cur], M, runs, lane);
        } else if (warp == 1) {
            if (SMALL) swaps(sh, s_o, head, lane);
            else swaps(sh, dst + (size_t)done * M, head, lane);
        } else if (!next_ready) {
            next_block(sh.mt[cur], sh.mt[cur ^ 1u], sh.out[cur ^ 1u], t - 64u);
        }
        next_ready = true;
        __syncthreads();
        if (sh.run_ready) {
            uint32_t *o = dst + (size_t)done * M;
            if (SMALL)
                for (uint32_t i = t; i < M; i += kThreads) o[i] = s_o[i];
            ++done;
            __syncthreads();
            if (done < runs) identity(dst + (size_t)done * M);
            if (t == 0) {
                sh.run_ready = 0;
                sh.i_swap = top;
            }
        }
    }
    if (state_out) {
        for (uint32_t k = t; k < 624; k += kThreads) state_out[k] = sh.mt[cur][k];
        if (t == 0) state_out[624] = sh.pos;
    }
}

// One stream and permutation per thread, the state words in local memory: for
// very many short permutations, of which a block is mostly seeding.
constexpr int kStreams = 64;  // threads per block
__global__ void __launch_bounds__(kStreams) mt_short_kernel(uint32_t M, uint32_t runs, const uint32_t *seed_words,
                                                            const int32_t *seed_len, int32_t stride, uint32_t *out) {
    const uint32_t r = blockIdx.x * kStreams + threadIdx.x;
    if (r >= runs) return;
    uint32_t mt[624];
    const int len = seed_len[r];
    const uint32_t *w = seed_words + (size_t)r * stride;
    if (len == 0) init_genrand(mt, w[0]);
    else init_by_array(mt, w, len);
    uint32_t *o = out + (size_t)r * M;
    for (uint32_t i = 0; i < M; ++i) o[i] = i;
    uint32_t pos = 624;
    for (uint32_t i = M - 1u; i >= 1; --i) {
        const uint32_t mask = 0xffffffffu >> __clz(i);
        uint32_t j;
        do {
            if (pos == 624) {
                for (uint32_t k = 0; k < 624; ++k) {
                    const uint32_t y = (mt[k] & 0x80000000u) | (mt[k + 1 < 624 ? k + 1 : 0] & 0x7fffffffu);
                    mt[k] = mt[k + 397 < 624 ? k + 397 : k - 227] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
                }
                pos = 0;
            }
            j = temper(mt[pos++]) & mask;
        } while (j > i);
        const uint32_t a = o[i];
        o[i] = o[j];
        o[j] = a;
    }
}

cudaError_t launch(uint32_t M, uint32_t blocks, uint32_t runs, const uint32_t *seed_words, const int32_t *seed_len,
                   int32_t stride, const uint32_t *state_in, uint32_t *state_out, uint32_t *out, cudaStream_t s) {
    const bool small = M <= kSmallM;
    return launch_kernel(small ? mt_perm_kernel<true> : mt_perm_kernel<false>, dim3(blocks), kThreads,
                         small ? (2 * (size_t)M + 15) & ~(size_t)15 : 0, small ? 2 * (size_t)kSmallM : 0, s, M, runs,
                         seed_words, seed_len, stride, state_in, state_out, out);
}

}  // namespace

cudaError_t launch_mt_perms(uint32_t M, int32_t n_runs, const uint32_t *seed_words, const int32_t *seed_len,
                            int32_t stride, uint32_t *out, cudaStream_t s) {
    if (n_runs <= 0 || M == 0) return cudaSuccess;
    // A thread each for 10^6 permutations of 2, 16, 100, 200, 350, 480: 1.8, 1.9, 4.4, 9.5,
    // 21.6, 59.7 ms, a block each 8.4, 10.3, 14.2, 17.0, 20.3, 22.3 (from some 400 draws on a
    // thread makes its 624 outputs twice); for 10^5 of 200 0.91 and 1.72; for 10^4 of 16
    // and 200 0.10 and 0.34 against 0.13 and 0.20.
    if (M <= 256 && n_runs >= 32768)
        return launch_kernel(mt_short_kernel, dim3((n_runs + kStreams - 1) / kStreams), kStreams, 0, 0, s, M,
                             (uint32_t)n_runs, seed_words, seed_len, stride, out);
    return launch(M, (uint32_t)n_runs, 1u, seed_words, seed_len, stride, nullptr, nullptr, out, s);
}

// Continuation of one MT19937 stream (numpy's global RandomState): n_runs
// permutations of range(M) are drawn one after another exactly as
// np.random.permutation(M) would draw them (percolate/percolate.py:270, once
// per run in run order), and the advanced state is stored.
cudaError_t launch_mt_stream_perms(const uint32_t *state_in, uint32_t M, int32_t n_runs, uint32_t *out,
                                   uint32_t *state_out, cudaStream_t s) {
    return launch(M, 1u, (uint32_t)n_runs, nullptr, nullptr, 0, state_in, state_out, out, s);
}

}  // namespace nz
