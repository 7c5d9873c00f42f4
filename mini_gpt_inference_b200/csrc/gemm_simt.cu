// out[m, n] = sum_k a[m, k] * w[n, k] (+ bias[n]) with an epilogue, on the CUDA cores.
//
// What the tensor-core kernels refuse: 32-bit or bfloat16 matrices whose rows are no multiples of 16 bytes (gemm_split.cu, gemm_tc.cu).
// Every output element sums its k terms in one fixed order, whatever the number of rows or the tile it falls in, so a
// token's result does not depend on what else is in the batch: K is cut into slices of 64, a slice's terms are summed
// one after the other (fused multiply-adds from 0), and the slices' sums are added one after the other.  All sizes are accepted;
// tiles of 128 x 128, 64 x 128 or 64 x 64 by 256 threads, 8 x 8 to 4 x 4 results a thread, operands through a ring of shared-memory
// stages, are predicated at the edges.  Bound by the FMA pipes and by what they read from shared memory.
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

// What becomes of a finished sum.
template <typename TOut, int EPI>
__device__ __forceinline__ void finish(float sum, int m, int n, const float* bias, TOut* out, float* residual, int N) {
    float v = sum + (bias ? bias[n] : 0.f);
    const size_t idx = (size_t)m * N + n;
    if (EPI == EPI_GELU) v = gelu_tanh(v);
    if (EPI == EPI_RELU_SQ) v = relu_sq(v);
    if (EPI == EPI_RESIDUAL) residual[idx] += v;
    else out[idx] = from_float<TOut>(v);
}

// TM x TN results a thread; a thread's rows (and columns) lie 16 apart.  Operands lie row by row in shared memory, 16 columns
// and 4 words of space a row: 16-byte reads along K by 8 neighbouring rows meet no bank twice.
template <typename TIn, typename TOut, int EPI, int TM, int TN>
__global__ void __launch_bounds__(256)
gemm_fma_kernel(const TIn* __restrict__ a, const TIn* __restrict__ w, const float* __restrict__ bias,
                TOut* __restrict__ out, float* __restrict__ residual, int M, int N, int K) {
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
            *reinterpret_cast<float4*>(to) = load4(from, row, rows, k, K);
        }
    };
#pragma unroll
    for (int b = 0; b < FMA_STAGES - 1; ++b) {
        if (b < blocks) fetch(b);
    }
    for (int b = 0; b < blocks; ++b) {
        __syncthreads();                                     // the block is there for all, and the block before is done with
        if (b + FMA_STAGES - 1 < blocks) fetch(b + FMA_STAGES - 1);
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
cudaError_t launch_tiles(const TIn* a, const TIn* w, const float* bias, TOut* out, float* residual, int M, int N, int K,
                         cudaStream_t s) {
    constexpr int smem = FMA_STAGES * 16 * (TM + TN) * PITCH * (int)sizeof(float);
    const cudaError_t configured = mg_raise_shared(gemm_fma_kernel<TIn, TOut, EPI, TM, TN>, smem);
    if (configured != cudaSuccess) return configured;
    return mg_launch(gemm_fma_kernel<TIn, TOut, EPI, TM, TN>, dim3(ceil_div(N, 16 * TN), ceil_div(M, 16 * TM)), dim3(256), smem, s, true,
                     a, w, bias, out, residual, M, N, K);
}

template <typename TIn, typename TOut, int EPI>
cudaError_t launch_epilogue(const TIn* a, const TIn* w, const float* bias, TOut* out, float* residual, int M, int N, int K,
                            cudaStream_t s) {
    auto ctas = [&](int bm, int bn) { return (long long)ceil_div(N, bn) * ceil_div(M, bm); };
    // The largest tile (the fewest shared-memory reads a product) of which there are enough for the SMs.
    if (ctas(128, 128) >= 240) return launch_tiles<TIn, TOut, EPI, 8, 8>(a, w, bias, out, residual, M, N, K, s);
    if (ctas(64, 128) >= 120) return launch_tiles<TIn, TOut, EPI, 4, 8>(a, w, bias, out, residual, M, N, K, s);
    return launch_tiles<TIn, TOut, EPI, 4, 4>(a, w, bias, out, residual, M, N, K, s);
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
