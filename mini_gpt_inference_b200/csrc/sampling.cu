// Sampling from 32-bit logits: greedy (argmax) here; the stochastic sampler follows below.
#include <cooperative_groups.h>
#include <float.h>
#include <math.h>

#include "common.cuh"

namespace {

constexpr int ARGMAX_THREADS = 256;

// Largest value of a row; among equal values the lowest index wins.  NaN never wins.
__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_kernel(const float* __restrict__ logits, int* __restrict__ out, int vocab, int limit) {
    __shared__ float best_v[ARGMAX_THREADS / 32];
    __shared__ int best_i[ARGMAX_THREADS / 32];
    const float* row = logits + (size_t)blockIdx.x * vocab;
    float v = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = threadIdx.x; i < limit; i += blockDim.x) {
        const float x = row[i];
        if (x > v || (x == v && i < idx)) { v = x; idx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { best_v[warp] = v; best_i[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        v = lane < ARGMAX_THREADS / 32 ? best_v[lane] : -INFINITY;
        idx = lane < ARGMAX_THREADS / 32 ? best_i[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
        }
        if (lane == 0) out[blockIdx.x] = idx == 0x7fffffff ? 0 : idx;
    }
}

// Stage 1 of the wide argmax: block (row, part) scans its slice of the row.
__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_part_kernel(const float* __restrict__ logits, float* __restrict__ part_v, int* __restrict__ part_i,
                   int vocab, int limit, int parts, int slice) {
    __shared__ float best_v[ARGMAX_THREADS / 32];
    __shared__ int best_i[ARGMAX_THREADS / 32];
    pdl_trigger();
    pdl_wait();                                        // the logits come from the kernel in front
    const float* row = logits + (size_t)blockIdx.x * vocab;
    const int begin = blockIdx.y * slice, end = min(limit, begin + slice);
    float v = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const float x = row[i];
        if (x > v || (x == v && i < idx)) { v = x; idx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { best_v[warp] = v; best_i[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        v = lane < ARGMAX_THREADS / 32 ? best_v[lane] : -INFINITY;
        idx = lane < ARGMAX_THREADS / 32 ? best_i[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
        }
        if (lane == 0) {
            part_v[(size_t)blockIdx.x * parts + blockIdx.y] = v;
            part_i[(size_t)blockIdx.x * parts + blockIdx.y] = idx;
        }
    }
}

// Stage 2: one warp per row merges the parts.
__global__ void argmax_merge_kernel(const float* __restrict__ part_v, const int* __restrict__ part_i,
                                    int* __restrict__ out, int parts) {
    float v = -INFINITY;
    int idx = 0x7fffffff;
    pdl_trigger();
    pdl_wait();
    for (int k = threadIdx.x; k < parts; k += 32) {
        const float x = part_v[(size_t)blockIdx.x * parts + k];
        const int i = part_i[(size_t)blockIdx.x * parts + k];
        if (x > v || (x == v && i < idx)) { v = x; idx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    if (threadIdx.x == 0) out[blockIdx.x] = idx == 0x7fffffff ? 0 : idx;
}

// Stage 2 for many parts (hundreds, as the head projection leaves them): a block per row.
__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_merge_block_kernel(const float* __restrict__ part_v, const int* __restrict__ part_i, int* __restrict__ out,
                          int parts) {
    __shared__ float best_v[ARGMAX_THREADS / 32];
    __shared__ int best_i[ARGMAX_THREADS / 32];
    float v = -INFINITY;
    int idx = 0x7fffffff;
    pdl_trigger();
    pdl_wait();
    for (int k = threadIdx.x; k < parts; k += ARGMAX_THREADS) {
        const float x = part_v[(size_t)blockIdx.x * parts + k];
        const int i = part_i[(size_t)blockIdx.x * parts + k];
        if (x > v || (x == v && i < idx)) { v = x; idx = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { best_v[warp] = v; best_i[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        v = lane < ARGMAX_THREADS / 32 ? best_v[lane] : -INFINITY;
        idx = lane < ARGMAX_THREADS / 32 ? best_i[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
        }
        if (lane == 0) out[blockIdx.x] = idx == 0x7fffffff ? 0 : idx;
    }
}

constexpr int ARGMAX_SLICE = 2048;

}  // namespace

// Parts a row is cut into by mg_argmax_wide; its scratch holds rows * parts floats and as many ints.
MG_API int mg_argmax_parts(int vocab) { return (vocab + ARGMAX_SLICE - 1) / ARGMAX_SLICE; }

// logits: [rows, vocab] 32-bit; ids >= limit are never chosen (limit <= 0: the whole vocabulary).
MG_API int mg_argmax(const float* logits, int* out, int rows, int vocab, int limit, void* stream) {
    if (rows == 0) return MG_OK;
    MG_REQUIRE(rows > 0 && vocab > 0, "argmax: bad sizes");
    if (limit <= 0 || limit > vocab) limit = vocab;
    argmax_kernel<<<rows, ARGMAX_THREADS, 0, (cudaStream_t)stream>>>(logits, out, vocab, limit);
    MG_CHECK_LAUNCH("argmax");
    return MG_OK;
}

// The same result with many blocks per row, for wide vocabularies and few rows: a row is cut
// into slices of 2048 ids, each scanned by a block; a second kernel merges.  The lowest index
// among equal maxima wins, as in mg_argmax.  scratch_v / scratch_i: rows * mg_argmax_parts(vocab).
MG_API int mg_argmax_wide(const float* logits, int* out, float* scratch_v, int* scratch_i, int rows, int vocab,
                          int limit, void* stream) {
    if (rows == 0) return MG_OK;
    MG_REQUIRE(rows > 0 && vocab > 0 && scratch_v && scratch_i, "argmax: bad arguments");
    if (limit <= 0 || limit > vocab) limit = vocab;
    const int parts = mg_argmax_parts(vocab);
    MG_REQUIRE(parts <= 65535, "argmax: vocabulary too wide");
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t le = mg_launch(argmax_part_kernel, dim3(rows, parts), dim3(ARGMAX_THREADS), 0, s, true, logits, scratch_v,
                               scratch_i, vocab, limit, parts, ARGMAX_SLICE);
    if (le != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "argmax (parts): %s", cudaGetErrorString(le));
    MG_CHECK_LAUNCH("argmax (parts)");
    le = mg_launch(argmax_merge_kernel, dim3(rows), dim3(32), 0, s, true, (const float*)scratch_v, (const int*)scratch_i, out,
                   parts);
    if (le != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "argmax (merge): %s", cudaGetErrorString(le));
    MG_CHECK_LAUNCH("argmax (merge)");
    return MG_OK;
}

// The second stage alone: part_v / part_i hold `parts` candidates per row (value and index, as
// the head projection leaves them when it takes the greedy choice on its way).
MG_API int mg_argmax_merge(const float* part_v, const int* part_i, int* out, int rows, int parts, void* stream) {
    if (rows == 0) return MG_OK;
    MG_REQUIRE(rows > 0 && parts > 0 && part_v && part_i && out, "argmax (merge): bad arguments");
    const cudaError_t le =
        parts > 64 ? mg_launch(argmax_merge_block_kernel, dim3(rows), dim3(ARGMAX_THREADS), 0, (cudaStream_t)stream, true,
                               part_v, part_i, out, parts)
                   : mg_launch(argmax_merge_kernel, dim3(rows), dim3(32), 0, (cudaStream_t)stream, true, part_v, part_i, out,
                               parts);
    if (le != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "argmax (merge): %s", cudaGetErrorString(le));
    MG_CHECK_LAUNCH("argmax (merge)");
    return MG_OK;
}

// ---- stochastic sampling -------------------------------------------------------------------------
// One block per row.  The order is the reference's (src/minigpt_infer/sampling.py:116-137):
// logits / max(temperature, 1e-6), top-k (values below the k-th largest dropped, ties pass),
// top-p (sorted descending, a token is dropped if the probability mass strictly before it
// exceeds p; the largest always stays), softmax, one draw.  A row with temperature <= 0 is
// greedy.  Instead of sorting the row, both cut-offs are found by a radix descent over the
// order-preserving bit pattern of the scaled logits: 4 passes of 8 bits with a histogram of
// counts (top-k) or of probability mass (top-p) in shared memory.  Mass is accumulated as
// 64-bit fixed point with integer atomics, so the result does not depend on the order of the
// additions.  The draw is an inverse-CDF walk in index order with a Philox4x32-10 number keyed
// by (seed, counter): the same request at the same token draws the same number whatever else
// is in the batch (the reference shares one generator across the batch,
// src/minigpt_infer/engine/engine.py:13-17).
namespace {

constexpr int SAMPLE_THREADS = 512;
constexpr float FIXED_ONE = 1099511627776.0f;   // 2^40: e in [0, 1] -> fixed point

__device__ __forceinline__ uint32_t order_key(float x) {
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }

// Philox4x32-10 (Salmon et al., "Parallel random numbers: as easy as 1, 2, 3"); first word.
__device__ uint32_t philox_first(uint32_t k0, uint32_t k1, uint32_t c0, uint32_t c1) {
    uint32_t c[4] = {c0, c1, 0u, 0u};
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t hi0 = mulhi32(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
        const uint32_t hi1 = mulhi32(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
        const uint32_t n0 = hi1 ^ c[1] ^ k0, n1 = lo1, n2 = hi0 ^ c[3] ^ k1, n3 = lo0;
        c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c[0];
}

// A row's draw from [0, 1).
__device__ __forceinline__ float uniform(uint32_t seed_lo, uint32_t seed_hi, uint32_t counter) {
    return (float)(philox_first(seed_lo, seed_hi, counter, 0u) >> 8) * (1.0f / 16777216.0f);
}

__device__ float block_reduce_max(float v, float* scratch) {
    v = warp_max(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = lane < SAMPLE_THREADS / 32 ? scratch[lane] : -INFINITY;
        v = warp_max(v);
        if (lane == 0) scratch[0] = v;
    }
    __syncthreads();
    return scratch[0];
}

__device__ float block_reduce_sum(float v, float* scratch) {
    v = warp_sum(v);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        v = lane < SAMPLE_THREADS / 32 ? scratch[lane] : 0.f;
        v = warp_sum(v);
        if (lane == 0) scratch[0] = v;
    }
    __syncthreads();
    return scratch[0];
}

// The lowest index among a row's largest values, by one CTA.
__device__ __forceinline__ void greedy_row(const float* lr, int limit, int* out, float* scratch, int* found) {
    float v = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = threadIdx.x; i < limit; i += SAMPLE_THREADS) {
        const float x = lr[i];
        if (x > v || (x == v && i < idx)) { v = x; idx = i; }
    }
    const float best = block_reduce_max(v, scratch);
    if (threadIdx.x == 0) *found = 0x7fffffff;
    __syncthreads();
    if (v == best && idx != 0x7fffffff) atomicMin(found, idx);
    __syncthreads();
    if (threadIdx.x == 0) *out = *found == 0x7fffffff ? 0 : *found;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const uint32_t* __restrict__ seed_lo, const uint32_t* __restrict__ seed_hi,
              const uint32_t* __restrict__ counter, int* __restrict__ out, int vocab, int limit) {
    __shared__ float scratch[SAMPLE_THREADS / 32];
    __shared__ unsigned long long hist[256];
    __shared__ uint32_t sh_prefix;
    __shared__ unsigned long long sh_acc;
    __shared__ int sh_found;
    const int row = blockIdx.x, tid = threadIdx.x;
    const float* lr = logits + (size_t)row * vocab;
    const float temp = temperature[row];

    if (temp <= 0.f) {   // greedy row: lowest index among the largest
        greedy_row(lr, limit, out + row, scratch, &sh_found);
        return;
    }

    const float safe_t = fmaxf(temp, 1e-6f);
    float mx = -INFINITY;
    for (int i = tid; i < limit; i += SAMPLE_THREADS) mx = fmaxf(mx, lr[i] / safe_t);
    mx = block_reduce_max(mx, scratch);

    // top-k: key of the k-th largest scaled logit
    uint32_t thr_key = 0u;
    const int k = top_k ? top_k[row] : 0;
    if (k > 0 && k < limit) {
        uint32_t prefix = 0u, mask = 0u;
        unsigned long long remaining = (unsigned long long)k;
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = 24 - 8 * pass;
            if (tid < 256) hist[tid] = 0ull;
            __syncthreads();
            for (int i = tid; i < limit; i += SAMPLE_THREADS) {
                const uint32_t key = order_key(lr[i] / safe_t);
                if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1ull);
            }
            __syncthreads();
            if (tid == 0) {
                unsigned long long cum = 0ull;
                int digit = 0;
                for (int b = 255; b >= 0; --b) {
                    if (cum + hist[b] >= remaining) { digit = b; break; }
                    cum += hist[b];
                }
                sh_prefix = prefix | ((uint32_t)digit << shift);
                sh_acc = remaining - cum;
            }
            __syncthreads();
            prefix = sh_prefix;
            remaining = sh_acc;
            mask |= 255u << shift;
            __syncthreads();
        }
        thr_key = prefix;
    }

    // top-p: lowest key whose mass of strictly larger keys is <= p * (mass kept by top-k)
    const float p = top_p ? top_p[row] : 1.f;
    if (p < 1.f) {
        float part = 0.f;
        for (int i = tid; i < limit; i += SAMPLE_THREADS) {
            const float x = lr[i] / safe_t;
            if (order_key(x) >= thr_key) part += expf(x - mx);
        }
        const float z_k = block_reduce_sum(part, scratch);
        const unsigned long long target = (unsigned long long)((double)p * (double)z_k * (double)FIXED_ONE);
        uint32_t prefix = 0u, mask = 0u;
        unsigned long long acc = 0ull;
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = 24 - 8 * pass;
            if (tid < 256) hist[tid] = 0ull;
            __syncthreads();
            for (int i = tid; i < limit; i += SAMPLE_THREADS) {
                const float x = lr[i] / safe_t;
                const uint32_t key = order_key(x);
                if (key >= thr_key && (key & mask) == prefix) {
                    // + 1 so that a token whose probability underflows still marks its bin
                    const unsigned long long e = (unsigned long long)(expf(x - mx) * FIXED_ONE) + 1ull;
                    atomicAdd(&hist[(key >> shift) & 255u], e);
                }
            }
            __syncthreads();
            if (tid == 0) {
                unsigned long long run = acc, chosen_acc = acc;
                int digit = -1;
                for (int b = 255; b >= 0; --b) {
                    if (hist[b] == 0ull) continue;
                    if (run > target && digit >= 0) break;
                    if (run <= target || digit < 0) { digit = b; chosen_acc = run; }
                    run += hist[b];
                }
                sh_prefix = prefix | ((uint32_t)(digit < 0 ? 0 : digit) << shift);
                sh_acc = chosen_acc;
            }
            __syncthreads();
            prefix = sh_prefix;
            acc = sh_acc;
            mask |= 255u << shift;
            __syncthreads();
        }
        if (prefix > thr_key) thr_key = prefix;
    }

    // normaliser of what is kept, then the inverse-CDF walk in index order
    float part = 0.f;
    for (int i = tid; i < limit; i += SAMPLE_THREADS) {
        const float x = lr[i] / safe_t;
        if (order_key(x) >= thr_key) part += expf(x - mx);
    }
    const float z = block_reduce_sum(part, scratch);
    const uint32_t rnd = philox_first(seed_lo[row], seed_hi[row], counter[row], 0u);
    const float u = (float)(rnd >> 8) * (1.0f / 16777216.0f);      // [0, 1)
    const float target = u * z;

    if (tid == 0) sh_found = 0x7fffffff;
    __syncthreads();
    float base = 0.f;
    int last_kept = -1;
    const int warp = tid >> 5, lane = tid & 31;
    for (int t0 = 0; t0 < limit; t0 += SAMPLE_THREADS) {
        const int i = t0 + tid;
        float e = 0.f;
        if (i < limit) {
            const float x = lr[i] / safe_t;
            if (order_key(x) >= thr_key) { e = expf(x - mx); if (e > 0.f) last_kept = i; }
        }
        float incl = e;                                            // inclusive scan in the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        __syncthreads();
        if (lane == 31) scratch[warp] = incl;
        __syncthreads();
        float before = 0.f, total = 0.f;
        for (int w = 0; w < SAMPLE_THREADS / 32; ++w) {
            const float s = scratch[w];
            if (w < warp) before += s;
            total += s;
        }
        const float cum = base + before + incl;
        if (e > 0.f && cum > target) atomicMin(&sh_found, i);
        __syncthreads();
        if (sh_found != 0x7fffffff) break;
        base += total;
    }
    if (sh_found == 0x7fffffff) {                                  // rounding left the target just above the sum
        __syncthreads();
        if (tid == 0) sh_found = -1;
        __syncthreads();
        if (last_kept >= 0) atomicMax(&sh_found, last_kept);
        __syncthreads();
    }
    if (tid == 0) out[row] = sh_found < 0 ? 0 : sh_found;
}

// ---- the same with a cluster of CTAs per row, for up to 131,072 ids ---------------------------------
// What bounds a row is a chain of passes over it: eight counting passes and three sums.  One CTA reads a row anew in every
// pass (it used to hold rows of up to 56,320 ids in shared memory, 98 values a thread at 50,304), one thread looks through a
// pass's 256 bins, and its 64-bit sums of probability mass meet in a few bins, lane after lane.  Here a row's values stay in the registers
// of a cluster's CTAs (16 a thread), lanes that meet in one bin of mass add up among themselves first, a warp picks the
// digit, and a pass ends in one cluster barrier behind which every CTA sums all histograms itself.
// 50,304 ids, one CTA and a cluster: 24 rows with top-k 50 and top-p 0.8, 572 -> 45 us (20 where few are left, see below); with
// top-p 0.9 alone, 526 -> 69; plain draws, 70 -> 17; 256 rows, plain draws, 123 -> 96.

// Descending over 256 bins: the digit and the sum in front of it.  `by_count`: the first bin whose inclusive sum reaches
// `goal`; otherwise the last non-empty bin in front of which at most `goal` lies (the first non-empty one if none is).
// One warp, 8 bins a lane.
__device__ __forceinline__ void pick_digit(const unsigned long long* total, unsigned long long start, unsigned long long goal,
                                           bool by_count, uint32_t* digit, unsigned long long* before, int* reached) {
    const int lane = threadIdx.x & 31;
    unsigned long long bin[8], sum = 0ull;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        bin[j] = total[255 - 8 * lane - j];
        sum += bin[j];
    }
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    unsigned long long run = start + incl - sum, first_run = run, hit_run = run;
    int first = -1, hit = -1;                                   // bins of this lane, counted from 255 down
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (bin[j] != 0ull && first < 0) { first = j; first_run = run; }
        if (by_count ? (hit < 0 && bin[j] != 0ull && run + bin[j] >= goal) : (bin[j] != 0ull && run <= goal)) { hit = j; hit_run = run; }
        run += bin[j];
    }
    const uint32_t hits = __ballot_sync(0xffffffffu, hit >= 0), any = __ballot_sync(0xffffffffu, first >= 0);
    const int chosen = hits ? (by_count ? __ffs(hits) - 1 : 31 - __clz(hits)) : any ? __ffs(any) - 1 : 0;
    if (lane == chosen) {
        const int j = hits ? hit : first;
        *digit = j < 0 ? 0u : (uint32_t)(255 - 8 * lane - j);
        *before = hits ? hit_run : first_run;
        *reached = hits != 0u;                                  // there is such a bin
    }
}

// ---- a row of which top-k leaves few ----
// The k-th largest of the threads' largest values bounds the row's k-th largest from below, so one counting pass over one value
// a thread tells which values can be kept at all: some 60 for k = 50.  They go to the first CTA, which compares each with each
// and draws: four cluster barriers instead of a dozen.  24 rows with top-k 50 and top-p 0.8, passes over all values and
// this: 50,304 ids 40.5 -> 20.3 us, 1,000 ids 22.2 -> 10.6, 131,072 ids 91 -> 41; 256 rows of 50,304 ids 335 -> 135.
constexpr int KEPT = SAMPLE_THREADS;                            // most of them: one a thread

// Bins of the distance to the row's largest value, eight to each power of two from 2^-12 on; rising with the distance.
__device__ __forceinline__ int gap_bin(float gap) { return max(0, (int)(__float_as_uint(gap) >> 20) - ((127 - 12) << 3)); }

// One CTA draws among `n` values, in index order, that hold all that top-k keeps.  scaled, key, mass: KEPT places each.
__device__ __forceinline__ void draw_among(int n, const float* scaled, const int* index, uint32_t* key, unsigned long long* mass,
                                           float mx, int k, float p, float u, float* scratch, int* found, int* last, int* out) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool in = tid < n;
    const float x = in ? scaled[tid] : 0.f;
    const uint32_t mine = in ? order_key(x) : 0u;
    if (in) key[tid] = mine;
    __syncthreads();
    int larger = 0;
    for (int j = 0; j < n; ++j) larger += key[j] > mine ? 1 : 0;
    bool keep = in && larger < k;
    const float weight = keep ? expf(x - mx) : 0.f;
    if (p < 1.f) {
        const float kept = block_reduce_sum(weight, scratch);
        const unsigned long long target = (unsigned long long)((double)p * (double)kept * (double)FIXED_ONE);
        if (in) mass[tid] = keep ? (unsigned long long)(weight * FIXED_ONE) + 1ull : 0ull;
        __syncthreads();
        unsigned long long before = 0ull;
        for (int j = 0; j < n; ++j) before += key[j] > mine ? mass[j] : 0ull;
        keep = keep && before <= target;
    }
    const float w = keep ? weight : 0.f;
    float incl = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();
    if (lane == 31) scratch[warp] = incl;
    __syncthreads();
    float before = 0.f, z = 0.f;
    for (int i = 0; i < SAMPLE_THREADS / 32; ++i) {
        if (i == warp) before = z;
        z += scratch[i];
    }
    if (w > 0.f) {
        atomicMax(last, index[tid]);
        if (before + incl > u * z) atomicMin(found, index[tid]);
    }
    __syncthreads();
    if (tid == 0) *out = *found != 0x7fffffff ? *found : max(0, *last);
}

template <int ROW_CTAS, int NV>
__global__ void __cluster_dims__(ROW_CTAS, 1, 1) __launch_bounds__(SAMPLE_THREADS, NV > 16 ? 1 : 2)
sample_cluster_kernel(const float* __restrict__ logits, const float* __restrict__ temperature,
                      const int* __restrict__ top_k, const float* __restrict__ top_p,
                      const uint32_t* __restrict__ seed_lo, const uint32_t* __restrict__ seed_hi,
                      const uint32_t* __restrict__ counter, int* __restrict__ out, int vocab, int limit, int chunk) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float scratch[SAMPLE_THREADS / 32];
    __shared__ unsigned long long hist[2][256];                 // two in turn: a pass clears the other one
    __shared__ unsigned long long total[256];
    __shared__ float sh_max, sh_kept, sh_mass;                  // this CTA's share of a cluster-wide reduction, one each
    __shared__ int sh_index, sh_last;
    __shared__ uint32_t sh_digit;
    __shared__ unsigned long long sh_before;
    __shared__ int sh_odd, sh_reached, sh_few;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = blockIdx.x / ROW_CTAS, rank = (int)cluster.block_rank();
    const float* lr = logits + (size_t)row * vocab;
    const int begin = rank * chunk, end = min(limit, begin + chunk);      // this CTA's ids; thread t has begin + t, + 512, ...
    const float temp = temperature[row];
    if (temp <= 0.f) {   // greedy row: the lowest index among the largest
        // Where all CTAs are on the GPU at once, those of the row share it (24 rows of 50,304 ids 8.9 -> 6.1 us); where they are
        // not, the others leave it to the first (256 rows 23 us, shared 42; 24 rows of 131,072 ids 13.8 and 18.7).
        if (ROW_CTAS == 1 || gridDim.x > 148 * (NV > 16 ? 1 : 2)) {
            if (rank == 0) greedy_row(lr, limit, out + row, scratch, &sh_index);
            return;
        }
        float best = -INFINITY;
        int at = 0x7fffffff;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int i = begin + v * SAMPLE_THREADS + tid;
            const float y = i < end ? lr[i] : NAN;              // (what is no number never wins)
            if (y > best || (y == best && i < at)) { best = y; at = i; }
        }
        const float most = block_reduce_max(best, scratch);
        if (tid == 0) { sh_max = most; sh_index = 0x7fffffff; }
        __syncthreads();
        if (best == most && at != 0x7fffffff) atomicMin(&sh_index, at);
        cluster.sync();
        if (rank == 0 && tid == 0) {
            best = -INFINITY;
            at = 0x7fffffff;
            for (int r = 0; r < ROW_CTAS; ++r) {                // (in index order: the first of equals is the lowest)
                const float y = *cluster.map_shared_rank(&sh_max, r);
                const int i = *cluster.map_shared_rank(&sh_index, r);
                if (i != 0x7fffffff && (y > best || at == 0x7fffffff)) { best = y; at = i; }
            }
            out[row] = at == 0x7fffffff ? 0 : at;
        }
        cluster.sync();                                         // rank 0 has read the others' shared memory
        return;
    }
    const float safe_t = fmaxf(temp, 1e-6f);

    float x[NV];
    float mx = -INFINITY;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = begin + v * SAMPLE_THREADS + tid;
        x[v] = i < end ? lr[i] / safe_t : -INFINITY;
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) mx = fmaxf(mx, x[v]);
    const float block_max = block_reduce_max(mx, scratch);
    bool nan = false;
#pragma unroll
    for (int v = 0; v < NV; ++v) nan = nan || x[v] != x[v];
    const bool any_nan = __syncthreads_or(nan);
    if (tid == 0) { sh_max = block_max; sh_index = 0x7fffffff; sh_last = -1; sh_odd = any_nan; }
    if (tid < 256) hist[0][tid] = 0ull;
    cluster.sync();
    mx = -INFINITY;
    bool odd = false;                                           // a value that is no number, or a largest that is infinite
    for (int r = 0; r < ROW_CTAS; ++r) {
        mx = fmaxf(mx, *cluster.map_shared_rank(&sh_max, r));
        odd = odd || *cluster.map_shared_rank(&sh_odd, r) != 0;
    }
    odd = odd || !(fabsf(mx) < INFINITY);

    uint32_t thr_key = 0u;
    int turn = 0;
    // One pass: the CTAs' histograms of 8 bits meet, and the digit is picked from their sum.
    auto next_digit = [&](unsigned long long start, unsigned long long goal, bool by_count) {
        cluster.sync();
        if (tid < 256) {
            unsigned long long sum = 0ull;
#pragma unroll
            for (int r = 0; r < ROW_CTAS; ++r) sum += *cluster.map_shared_rank(&hist[turn][tid], r);
            total[tid] = sum;
            hist[turn ^ 1][tid] = 0ull;                         // read by the others before this barrier, written after it
        }
        __syncthreads();
        if (warp == 0) pick_digit(total, start, goal, by_count, &sh_digit, &sh_before, &sh_reached);
        __syncthreads();
        turn ^= 1;
    };

    const int k = top_k ? top_k[row] : 0;
    const float p = top_p ? top_p[row] : 1.f;
    if (k > 0 && k < limit && k <= KEPT && !odd) {
        __shared__ float few_x[2][KEPT];                            // this CTA's; those of all, in the first CTA
        __shared__ int few_i[2][KEPT], few_at[NV * (SAMPLE_THREADS / 32)];
        float mine = -INFINITY;                                     // this thread's largest
#pragma unroll
        for (int v = 0; v < NV; ++v) mine = fmaxf(mine, x[v]);
        const int own_bin = gap_bin(mx - mine);
        if (own_bin < 256) atomicAdd(reinterpret_cast<uint32_t*>(hist[turn]) + 2 * (255 - own_bin), 1u);
        next_digit(0ull, (unsigned long long)k, true);
        if (sh_reached) {
            const int bin = 255 - (int)sh_digit;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const bool in = begin + v * SAMPLE_THREADS + tid < end && gap_bin(mx - x[v]) <= bin;
                const uint32_t who = __ballot_sync(0xffffffffu, in);
                if (lane == 0) few_at[v * (SAMPLE_THREADS / 32) + warp] = __popc(who);
            }
            __syncthreads();
            if (warp == 0) {                                        // the counts, in index order, become first places
                constexpr int PER = NV * (SAMPLE_THREADS / 32) / 32;
                int count[PER], sum = 0;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    count[j] = few_at[lane * PER + j];
                    sum += count[j];
                }
                int incl = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                int at = incl - sum;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    few_at[lane * PER + j] = at;
                    at += count[j];
                }
                if (lane == 31) sh_few = incl;
            }
            __syncthreads();
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const int i = begin + v * SAMPLE_THREADS + tid;
                const bool in = i < end && gap_bin(mx - x[v]) <= bin;
                const uint32_t who = __ballot_sync(0xffffffffu, in);
                const int at = few_at[v * (SAMPLE_THREADS / 32) + warp] + __popc(who & ((1u << lane) - 1u));
                if (in && at < KEPT) {
                    few_x[0][at] = x[v];
                    few_i[0][at] = i;
                }
            }
            cluster.sync();
            int n = 0;
            for (int r = 0; r < ROW_CTAS; ++r) n += *cluster.map_shared_rank(&sh_few, r);
            if (n <= KEPT) {
                if (rank == 0) {
                    int at = 0;
                    for (int r = 0; r < ROW_CTAS; ++r) {
                        const int count = *cluster.map_shared_rank(&sh_few, r);
                        if (tid < count) {
                            few_x[1][at + tid] = *cluster.map_shared_rank(&few_x[0][tid], r);
                            few_i[1][at + tid] = *cluster.map_shared_rank(&few_i[0][tid], r);
                        }
                        at += count;
                    }
                }
                cluster.sync();                                     // the others' shared memory is not read from here on
                if (rank == 0)
                    draw_among(n, few_x[1], few_i[1], reinterpret_cast<uint32_t*>(few_x[0]), &hist[0][0], mx, k, p,
                               uniform(seed_lo[row], seed_hi[row], counter[row]), scratch, &sh_index, &sh_last, out + row);
                return;
            }
        }
    }

    // top-k: key of the k-th largest scaled logit
    if (k > 0 && k < limit) {
        uint32_t prefix = 0u, mask = 0u;
        unsigned long long remaining = (unsigned long long)k;
        for (int shift = 24; shift >= 0; shift -= 8) {
            uint32_t* counts = reinterpret_cast<uint32_t*>(hist[turn]);       // the low words of the bins
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const uint32_t key = order_key(x[v]);
                if (begin + v * SAMPLE_THREADS + tid < end && (key & mask) == prefix) atomicAdd(counts + 2 * ((key >> shift) & 255u), 1u);
            }
            next_digit(0ull, remaining, true);
            prefix |= sh_digit << shift;
            remaining -= sh_before;
            mask |= 255u << shift;
        }
        thr_key = prefix;
    }

    // top-p: lowest key whose mass of strictly larger keys is <= p * (mass kept by top-k)
    if (p < 1.f) {
        float part = 0.f;
#pragma unroll
        for (int v = 0; v < NV; ++v)
            if (begin + v * SAMPLE_THREADS + tid < end && order_key(x[v]) >= thr_key) part += expf(x[v] - mx);
        part = block_reduce_sum(part, scratch);
        if (tid == 0) sh_kept = part;
        cluster.sync();
        float z_k = 0.f;
        for (int r = 0; r < ROW_CTAS; ++r) z_k += *cluster.map_shared_rank(&sh_kept, r);
        const unsigned long long target = (unsigned long long)((double)p * (double)z_k * (double)FIXED_ONE);
        uint32_t prefix = 0u, mask = 0u;
        unsigned long long acc = 0ull;
        for (int shift = 24; shift >= 0; shift -= 8) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const uint32_t key = order_key(x[v]);
                const bool in = begin + v * SAMPLE_THREADS + tid < end && key >= thr_key && (key & mask) == prefix;
                if (!in) continue;
                // + 1 so that a token whose probability underflows still marks its bin
                const unsigned long long e = (unsigned long long)(expf(x[v] - mx) * FIXED_ONE) + 1ull;
                const uint32_t bin = (key >> shift) & 255u;
                if (e >> 56) {                                  // not a number
                    atomicAdd(&hist[turn][bin], e);
                    continue;
                }
                const uint32_t peers = __match_any_sync(__activemask(), bin);
                // 32 numbers of up to 2^40 + 1: their low 24 and high bits add up in 32 bits each
                const uint32_t low = __reduce_add_sync(peers, (uint32_t)e & 0xffffffu);
                const uint32_t high = __reduce_add_sync(peers, (uint32_t)(e >> 24));
                if (lane == __ffs(peers) - 1) atomicAdd(&hist[turn][bin], ((unsigned long long)high << 24) + low);
            }
            next_digit(acc, target, false);
            prefix |= sh_digit << shift;
            acc = sh_before;
            mask |= 255u << shift;
        }
        if (prefix > thr_key) thr_key = prefix;
    }

    // normaliser of what is kept, CTA by CTA in index order
    float part = 0.f;
    int last_kept = -1;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        const int i = begin + v * SAMPLE_THREADS + tid;
        x[v] = i < end && order_key(x[v]) >= thr_key ? expf(x[v] - mx) : 0.f;       // from here on: the weights
        part += x[v];
        if (x[v] > 0.f) last_kept = i;
    }
    part = block_reduce_sum(part, scratch);
    if (last_kept >= 0) atomicMax(&sh_last, last_kept);
    if (tid == 0) sh_mass = part;
    cluster.sync();
    float mass[ROW_CTAS], z = 0.f;
    int last = -1;
    for (int r = 0; r < ROW_CTAS; ++r) {
        mass[r] = *cluster.map_shared_rank(&sh_mass, r);
        z += mass[r];
        last = max(last, *cluster.map_shared_rank(&sh_last, r));
    }
    cluster.sync();                                             // the others' shared memory is not read from here on
    const float target = uniform(seed_lo[row], seed_hi[row], counter[row]) * z;
    float base = 0.f;
    int owner = -1;                                             // the CTA in whose ids the sum passes the target
    for (int r = 0; r < ROW_CTAS; ++r) {
        if (base + mass[r] > target) { owner = r; break; }
        base += mass[r];
    }
    if (owner < 0) {                                            // rounding left the target just above the sum
        if (rank == 0 && tid == 0) out[row] = last < 0 ? 0 : last;
        return;
    }
    if (owner != rank) return;
    // the inverse-CDF walk in index order through this CTA's weights
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        if (v * SAMPLE_THREADS >= chunk) break;
        float incl = x[v];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += n;
        }
        __syncthreads();
        if (lane == 31) scratch[warp] = incl;
        __syncthreads();
        float before = 0.f, sum = 0.f;
        for (int w = 0; w < SAMPLE_THREADS / 32; ++w) {
            const float s = scratch[w];
            if (w < warp) before += s;
            sum += s;
        }
        if (x[v] > 0.f && base + before + incl > target) atomicMin(&sh_index, begin + v * SAMPLE_THREADS + tid);
        __syncthreads();
        if (sh_index != 0x7fffffff) break;
        base += sum;
    }
    if (tid == 0) out[row] = sh_index != 0x7fffffff ? sh_index : max(0, sh_last);
}

}  // namespace

// temperature: [rows]; top_k: [rows] int (<= 0: off) or null; top_p: [rows] (>= 1: off) or null;
// seed_lo/seed_hi/counter: [rows] 32-bit words of each row's seed and of its draw number.
MG_API int mg_sample(const float* logits, const float* temperature, const int* top_k, const float* top_p,
                     const uint32_t* seed_lo, const uint32_t* seed_hi, const uint32_t* counter, int* out,
                     int rows, int vocab, int limit, void* stream) {
    if (rows == 0) return MG_OK;
    MG_REQUIRE(rows > 0 && vocab > 0, "sample: bad sizes");
    MG_REQUIRE(temperature && seed_lo && seed_hi && counter, "sample: missing per-row parameters");
    if (limit <= 0 || limit > vocab) limit = vocab;
    // As many CTAs a row as hold it with 16 values a thread (two such CTAs share an SM), with 32 beyond 65,536 ids (24 rows
    // of 131,072 with both cuts: 1,802 -> 91 us); wider rows, which eight CTAs do not hold, keep to the kernel of one CTA.
    if (limit <= 32 * 8 * SAMPLE_THREADS) {
        const int held = 16 * SAMPLE_THREADS, ctas = limit <= held ? 1 : limit <= 2 * held ? 2 : limit <= 4 * held ? 4 : 8;
        auto kernel = ctas == 1 ? sample_cluster_kernel<1, 16> : ctas == 2 ? sample_cluster_kernel<2, 16> :
                      ctas == 4 ? sample_cluster_kernel<4, 16> : limit <= 8 * held ? sample_cluster_kernel<8, 16> :
                                                                                     sample_cluster_kernel<8, 32>;
        kernel<<<rows * ctas, SAMPLE_THREADS, 0, (cudaStream_t)stream>>>(logits, temperature, top_k, top_p, seed_lo, seed_hi,
                                                                         counter, out, vocab, limit, ceil_div(limit, ctas));
        MG_CHECK_LAUNCH("sample (cluster)");
        return MG_OK;
    }
    sample_kernel<<<rows, SAMPLE_THREADS, 0, (cudaStream_t)stream>>>(logits, temperature, top_k, top_p, seed_lo, seed_hi, counter,
                                                                     out, vocab, limit);
    MG_CHECK_LAUNCH("sample");
    return MG_OK;
}
