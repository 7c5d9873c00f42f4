// out[m, n] = sum_k a[m, k] * w[n, k] (+ bias[n]) with an epilogue, on the CUDA cores.
//
// This is the true 32-bit matrix product of the engine (plain FMA, no tensor-core mode of
// reduced precision) and the fallback for bfloat16 sizes the tensor-core kernels refuse.
// Every output element sums its k terms in one fixed order, whatever the number of rows or the kernel and
// tile it falls in, so a token's result does not depend on what else is in the batch: K is cut into slices
// of 64, a slice's terms are summed one after the other (fused multiply-adds from 0), and the slices' sums
// are added one after the other.  The slices are what lets a few rows use the whole GPU: warps sum
// different slices at the same time.  All sizes are accepted; tiles are predicated at the edges.
//
// Two kernels:
//   gemm_fma_kernel   tiles of 128 x 128, 64 x 128 or 64 x 64 by 256 threads, 8 x 8 to 4 x 4 results a thread, operands
//                     through a ring of shared-memory stages; bound by the FMA pipes and by what they read from shared memory.
//   gemm_few_kernel   up to 16 rows: a CTA takes 16 rows of w, each of its eight warps every eighth slice; w and a
//                     arrive by cp.async in a ring of the warp's own, the first round of w before the wait for the kernel
//                     in front.  Bound by reading w (and, below a few MB, by the latency of a launch and a slice).
// 8 rows, 1,536 x 512: 79 us in 64 x 64 tiles of 64 rows (24 CTAs, eight of the 64 rows in use), now 5; 2,048 rows: 204 -> 101 us.
#include <type_traits>

#include "common.cuh"

#define EPI_STORE 0      // out = acc + bias                (TOut)
#define EPI_GELU 1       // out = gelu_tanh(acc + bias)     (TOut)
#define EPI_RESIDUAL 2   // residual += acc + bias          (32-bit, in place)
#define EPI_RELU_SQ 3    // out = max(acc + bias, 0)^2      (TOut)

namespace {

constexpr int SLICE = 64;            // terms summed in one go
constexpr int BK = 16;               // columns of K per shared-memory stage of the tiles
constexpr int PITCH = BK + 4;        // words between rows there
constexpr int FMA_STAGES = 4;
static_assert(SLICE % BK == 0, "a slice is a whole number of stages");

// Four neighbouring elements of row `row` from column k on; zeros outside [rows, K].
template <typename TIn>
__device__ __forceinline__ float4 load4(const TIn* p, int row, int rows, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= rows) return v;
    const TIn* at = p + (size_t)row * K + k;
    if (k < K) v.x = to_float(at[0]);
    if (k + 1 < K) v.y = to_float(at[1]);
    if (k + 2 < K) v.z = to_float(at[2]);
    if (k + 3 < K) v.w = to_float(at[3]);
    return v;
}

// What becomes of a finished sum (both kernels).
template <typename TOut, int EPI>
__device__ __forceinline__ void finish(float sum, int m, int n, const float* bias, TOut* out, float* residual, int N) {
    float v = sum + (bias ? bias[n] : 0.f);
    const size_t idx = (size_t)m * N + n;
    if (EPI == EPI_GELU) v = gelu_tanh(v);
    if (EPI == EPI_RELU_SQ) v = relu_sq(v);
    if (EPI == EPI_RESIDUAL) residual[idx] += v;
    else out[idx] = from_float<TOut>(v);
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool there) {
    const uint32_t bytes = there ? 16u : 0u;                 // (0: sixteen zero bytes are written)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// TM x TN results a thread; a thread's rows (and columns) lie 16 apart.  Operands lie row by row in shared memory, 16 columns
// and 4 words of space a row: 16-byte reads along K by 8 neighbouring rows meet no bank twice, and a row's 64 bytes come by
// four neighbouring lanes' cp.async (with a lane to a row, the loads alone took as long as the products).
template <typename TIn, typename TOut, int EPI, int TM, int TN>
__global__ void __launch_bounds__(256)
gemm_fma_kernel(const TIn* __restrict__ a, const TIn* __restrict__ w, const float* __restrict__ bias,
                TOut* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int vec) {
    constexpr int BM = 16 * TM, BN = 16 * TN, ROWS = BM + BN;
    constexpr int LOADS = ROWS * BK / 4 / 256;               // four-element loads a thread makes per stage
    static_assert(LOADS * 256 * 4 == ROWS * BK && BM % 64 == 0, "whole loads, each of one operand");
    extern __shared__ __align__(16) float fma_smem[];        // [FMA_STAGES][ROWS][PITCH]: rows of a, then of w
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tr = tid / 16, tc = tid % 16;
    float total[TM][TN], acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) total[i][j] = acc[i][j] = 0.f;

    pdl_trigger();
    pdl_wait();
    const int blocks = (K + BK - 1) / BK;
    auto fetch = [&](int b) {
        float* stage = fma_smem + (b % FMA_STAGES) * ROWS * PITCH;
        const int k = b * BK + (tid & 3) * 4;
#pragma unroll
        for (int i = 0; i < LOADS; ++i) {
            const int e = (tid >> 2) + 64 * i;
            const bool of_a = e < BM;
            const int row = of_a ? m0 + e : n0 + e - BM, rows = of_a ? M : N;
            const TIn* from = of_a ? a : w;
            float* to = stage + e * PITCH + (tid & 3) * 4;
            if constexpr (std::is_same_v<TIn, float>) {
                if (vec) {                                   // K is a multiple of 4 and the matrices are aligned
                    const bool there = row < rows && k < K;
                    cp_async16(to, there ? from + (size_t)row * K + k : from, there);
                    continue;
                }
            }
            *reinterpret_cast<float4*>(to) = load4(from, row, rows, k, K);
        }
    };
#pragma unroll
    for (int b = 0; b < FMA_STAGES - 1; ++b) {
        if (b < blocks) fetch(b);
        cp_async_commit();
    }
    for (int b = 0; b < blocks; ++b) {
        cp_async_wait<FMA_STAGES - 2>();
        __syncthreads();                                     // the block is there for all, and the block before is done with
        if (b + FMA_STAGES - 1 < blocks) fetch(b + FMA_STAGES - 1);
        cp_async_commit();
        const float* as = fma_smem + (b % FMA_STAGES) * ROWS * PITCH + tr * PITCH;
        const float* ws = fma_smem + (b % FMA_STAGES) * ROWS * PITCH + (BM + tc) * PITCH;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 av[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = *reinterpret_cast<const float4*>(as + 16 * i * PITCH + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 wv = *reinterpret_cast<const float4*>(ws + 16 * j * PITCH + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].x, wv.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].y, wv.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].z, wv.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(av[i].w, wv.w, acc[i][j]);
            }
        }
        if ((b + 1) % (SLICE / BK) == 0 || b + 1 == blocks) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    total[i][j] += acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + tr + 16 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tc + 16 * j;
            if (n < N) finish<TOut, EPI>(total[i][j], m, n, bias, out, residual, N);
        }
    }
}

template <typename TIn, typename TOut, int EPI, int TM, int TN>
cudaError_t launch_tiles(const TIn* a, const TIn* w, const float* bias, TOut* out, float* residual, int M, int N, int K, bool vec,
                         cudaStream_t s) {
    constexpr int smem = FMA_STAGES * 16 * (TM + TN) * PITCH * (int)sizeof(float);
    const cudaError_t configured = mg_raise_shared(gemm_fma_kernel<TIn, TOut, EPI, TM, TN>, smem);
    if (configured != cudaSuccess) return configured;
    return mg_launch(gemm_fma_kernel<TIn, TOut, EPI, TM, TN>, dim3(ceil_div(N, 16 * TN), ceil_div(M, 16 * TM)), dim3(256), smem, s, true,
                     a, w, bias, out, residual, M, N, K, (int)vec);
}

constexpr int FEW_WARPS = 8, FEW_STAGES = 2, FEW_N = 16;    // rows of w per CTA
constexpr int LINE = SLICE + 4;                              // words between rows in shared memory: 16-byte reads of 8 rows meet no bank twice

// MT rows of a (8 or 16).  Wants K % 4 == 0 and 16-byte aligned matrices.
template <int EPI, int MT>
__global__ void __launch_bounds__(32 * FEW_WARPS)
gemm_few_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                float* __restrict__ out, float* __restrict__ residual, int M, int N, int K, int stages) {
    constexpr int NR = FEW_N, STAGE = (NR + MT) * LINE;      // words of a warp's stage: w's slice, then a's
    constexpr int NB = NR / 8, MB = MT / 4;                  // results a lane: NB x MB
    extern __shared__ __align__(16) float few_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* ring = few_smem + warp * stages * STAGE;
    float* parts = few_smem + FEW_WARPS * stages * STAGE;    // [2][warp][MT][NR]
    const int n0 = blockIdx.x * NR;
    const int slices = (K + SLICE - 1) / SLICE, rounds = (slices + FEW_WARPS - 1) / FEW_WARPS;

    auto ask_w = [&](int r) {
        float* dst = ring + (r & (stages - 1)) * STAGE;
        const int k0 = (r * FEW_WARPS + warp) * SLICE;
#pragma unroll
        for (int i = 0; i < NR / 2; ++i) {
            const int row = 2 * i + (lane >> 4), c = (lane & 15) * 4;
            const bool there = n0 + row < N && k0 + c < K;
            cp_async16(dst + row * LINE + c, there ? w + (size_t)(n0 + row) * K + k0 + c : w, there);
        }
    };
    auto ask_a = [&](int r) {
        float* dst = ring + (r & (stages - 1)) * STAGE + NR * LINE;
        const int k0 = (r * FEW_WARPS + warp) * SLICE;
#pragma unroll
        for (int i = 0; i < MT / 2; ++i) {
            const int row = 2 * i + (lane >> 4), c = (lane & 15) * 4;
            const bool there = row < M && k0 + c < K;
            cp_async16(dst + row * LINE + c, there ? a + (size_t)row * K + k0 + c : a, there);
        }
    };
    pdl_trigger();
    for (int r = 0; r < stages && r < rounds; ++r) ask_w(r);                // the weights depend on no kernel before
    pdl_wait();
    for (int r = 0; r < FEW_STAGES; ++r) {
        if (r < stages && r < rounds) ask_a(r);
        cp_async_commit();
    }
    const int nl = lane & 7, mg = lane >> 3;
    float total = 0.f;                                                      // of row tid / NR, column n0 + tid % NR
    for (int r = 0; r < rounds; ++r) {
        cp_async_wait<FEW_STAGES - 1>();
        __syncwarp();
        const float* ws = ring + (r & (stages - 1)) * STAGE + nl * LINE;
        const float* as = ring + (r & (stages - 1)) * STAGE + (NR + mg) * LINE;
        float acc[MB][NB];
#pragma unroll
        for (int i = 0; i < MB; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j) acc[i][j] = 0.f;
#pragma unroll 4
        for (int k = 0; k < SLICE; k += 4) {
            float4 wv[NB], av[MB];
#pragma unroll
            for (int j = 0; j < NB; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + 8 * j * LINE + k);
#pragma unroll
            for (int i = 0; i < MB; ++i) av[i] = *reinterpret_cast<const float4*>(as + 4 * i * LINE + k);
#pragma unroll
            for (int i = 0; i < MB; ++i)
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    acc[i][j] = fmaf(av[i].x, wv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(av[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(av[i].z, wv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(av[i].w, wv[j].w, acc[i][j]);
                }
        }
        __syncwarp();
        if (r + stages < rounds) {
            ask_w(r + stages);
            ask_a(r + stages);
        }
        cp_async_commit();
        float* part = parts + (r & 1) * FEW_WARPS * MT * NR;
#pragma unroll
        for (int i = 0; i < MB; ++i)
#pragma unroll
            for (int j = 0; j < NB; ++j) part[(warp * MT + mg + 4 * i) * NR + nl + 8 * j] = acc[i][j];
        // (one barrier a round: the half written two rounds later was read before the barrier in between)
        __syncthreads();
        const int here = min(FEW_WARPS, slices - r * FEW_WARPS);
        if (tid < MT * NR)
            for (int s = 0; s < here; ++s) total += part[s * MT * NR + tid];
    }
    cp_async_wait<0>();
    const int m = tid / NR, n = n0 + tid % NR;
    if (tid < MT * NR && m < M && n < N) finish<float, EPI>(total, m, n, bias, out, residual, N);
}

template <int EPI, int MT>
cudaError_t launch_few(const float* a, const float* w, const float* bias, float* out, float* residual, int M, int N, int K,
                       cudaStream_t s) {
    static_assert(MT * FEW_N <= 32 * FEW_WARPS, "a thread per result");
    // one round of slices needs one stage: more CTAs fit an SM, and one's copies run beside another's sums (a head of 50,304
    // ids at K = 512: 45 -> 33 us; 32 rows of w a CTA measured the same)
    const int stages = K <= FEW_WARPS * SLICE ? 1 : FEW_STAGES;
    auto bytes = [](int st) { return (int)((FEW_WARPS * st * (FEW_N + MT) * LINE + 2 * FEW_WARPS * MT * FEW_N) * sizeof(float)); };
    const cudaError_t configured = mg_raise_shared(gemm_few_kernel<EPI, MT>, bytes(FEW_STAGES));
    if (configured != cudaSuccess) return configured;
    return mg_launch(gemm_few_kernel<EPI, MT>, dim3(ceil_div(N, FEW_N)), dim3(32 * FEW_WARPS), bytes(stages), s, true, a, w, bias,
                     out, residual, M, N, K, stages);
}

template <typename TIn, typename TOut, int EPI>
cudaError_t launch_epilogue(const TIn* a, const TIn* w, const float* bias, TOut* out, float* residual, int M, int N, int K,
                            cudaStream_t s) {
    const bool vec = K % 4 == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)w & 15) == 0;
    if constexpr (std::is_same_v<TIn, float> && std::is_same_v<TOut, float>) {
        if (vec && M <= 8) return launch_few<EPI, 8>(a, w, bias, out, residual, M, N, K, s);
        if (vec && M <= 16) return launch_few<EPI, 16>(a, w, bias, out, residual, M, N, K, s);
    }
    auto ctas = [&](int bm, int bn) { return (long long)ceil_div(N, bn) * ceil_div(M, bm); };
    // The largest tile (the fewest shared-memory reads a product) of which there are enough for the SMs: 2,048 x 2,048 x 512 in
    // 256 tiles of 128 x 128 121 us, of 64 x 128 130; 2,048 x 1,536 x 512 (192 and 384 tiles) 121 and 101; 2,048 x 512 x 2,048
    // in 64 x 128 144, in 64 x 64 150; 500 x 512 x 2,048 144 and 99.
    if (ctas(128, 128) >= 240) return launch_tiles<TIn, TOut, EPI, 8, 8>(a, w, bias, out, residual, M, N, K, vec, s);
    if (ctas(64, 128) >= 120) return launch_tiles<TIn, TOut, EPI, 4, 8>(a, w, bias, out, residual, M, N, K, vec, s);
    return launch_tiles<TIn, TOut, EPI, 4, 4>(a, w, bias, out, residual, M, N, K, vec, s);
}

template <typename TIn, typename TOut>
int launch(const void* a, const void* w, const float* bias, void* out, float* residual, int M, int N,
           int K, int epilogue, cudaStream_t s) {
    const TIn* ap = (const TIn*)a;
    const TIn* wp = (const TIn*)w;
    TOut* op = (TOut*)out;
    cudaError_t e;
    switch (epilogue) {
        case EPI_STORE: e = launch_epilogue<TIn, TOut, EPI_STORE>(ap, wp, bias, op, residual, M, N, K, s); break;
        case EPI_GELU: e = launch_epilogue<TIn, TOut, EPI_GELU>(ap, wp, bias, op, residual, M, N, K, s); break;
        case EPI_RELU_SQ: e = launch_epilogue<TIn, TOut, EPI_RELU_SQ>(ap, wp, bias, op, residual, M, N, K, s); break;
        case EPI_RESIDUAL: e = launch_epilogue<TIn, TOut, EPI_RESIDUAL>(ap, wp, bias, op, residual, M, N, K, s); break;
        default: return mg_set_error(MG_ERR_ARG, "linear: unknown epilogue %d", epilogue);
    }
    if (e != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "gemm_simt: %s", cudaGetErrorString(e));
    MG_CHECK_LAUNCH("gemm_simt");
    return MG_OK;
}

}  // namespace

// a: [M, K] and w: [N, K], both row-major and of the same type (32-bit, or bfloat16 if in_bf16).
// epilogue 0/1 write `out` [M, N] (bfloat16 if out_bf16 else 32-bit); epilogue 2 adds into the
// 32-bit `residual` [M, N].  bias may be null.
MG_API int mg_linear_simt(const void* a, const void* w, const float* bias, void* out, float* residual,
                          int M, int N, int K, int epilogue, int in_bf16, int out_bf16, void* stream) {
    if (M == 0) return MG_OK;
    MG_REQUIRE(M > 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    MG_REQUIRE(ceil_div(M, 64) <= 65535, "linear: too many rows for one launch (%d)", M);
    MG_REQUIRE(epilogue == EPI_RESIDUAL ? residual != nullptr : out != nullptr, "linear: missing output");
    cudaStream_t s = (cudaStream_t)stream;
    if (in_bf16 && out_bf16) return launch<bf16, bf16>(a, w, bias, out, residual, M, N, K, epilogue, s);
    if (in_bf16) return launch<bf16, float>(a, w, bias, out, residual, M, N, K, epilogue, s);
    MG_REQUIRE(!out_bf16, "linear: 32-bit inputs with bfloat16 output is not a path of this engine");
    return launch<float, float>(a, w, bias, out, residual, M, N, K, epilogue, s);
}
