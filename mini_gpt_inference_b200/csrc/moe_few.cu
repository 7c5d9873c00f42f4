// The experts' two matrix products for steps of up to 16 tokens (decoding), bfloat16.
//
// Such a step reads every chosen expert's matrices once and does next to nothing with them, so what counts is how many of
// their bytes are asked for at once.  A CTA takes 16 outputs of one expert (16 matrix rows, 32 for a gated unit); its eight
// warps share K, 128 columns at a time, and load their share of the rows straight into the registers of mma.sync's A
// operand: a lane's 16 bytes of a row are eight neighbouring k, which serve as the k of two m16n8k16 products in an order of
// their own (a sum over k does not mind, as long as the tokens' operand is read the same way).  No shared memory, no ring:
// a whole CTA's 32 KB are in flight together.  The tokens are the product's 8 (or 16) columns; the warps' sums meet in
// shared memory and are added in warp order.
//
// The entries (token, k) of an expert are found by each warp from the ids themselves, so no grouping kernel runs in front:
// results lie by entry, and entry_slot is the identity (-1 for padding rows).
//
// The second product (form 0) reads the same ids as the first, which runs right in front of it, and its matrices come from no
// kernel: so its CTAs, as far as they find room beside the first product's, look up their entries and have their rows under way
// before the first product is done.  (Registers for a CTA's first 1,024 columns across that wait: four CTAs an SM, not five.)
//
// 4 tokens, 8 experts of 1,024 x 1,024 and one that every token uses (19 MB a product): 12.7 and 14.0 us, and 3.4 for the
// grouping, with the tiles of moe.cu; 8.3 and 7.9 here, 3 less for the two since the second starts early (16 decode steps of four
// such layers 7,041 -> 6,845 us).
#include "common.cuh"
#include "moe_units.cuh"

MG_GUARD_DECLARE(moe_few)

namespace {

constexpr int WARPS = 8;
constexpr int ROWS = 16;                 // outputs per CTA
constexpr int MAX_TOKENS = 16;

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// What becomes of an entry's finished sums (u: the up feature of a gated unit).
template <int FORM>
__device__ __forceinline__ void finish(float v, float u, int entry, int n, int N, const float* scale, int act, float limit, void* out) {
    const float s = scale ? scale[entry] : 1.f;
    const size_t to = (size_t)entry * N + n;
    if constexpr (FORM == 1) reinterpret_cast<bf16*>(out)[to] = __float2bfloat16_rn(gated_value(act, limit, v * s, u * s));
    else if constexpr (FORM == 2) reinterpret_cast<bf16*>(out)[to] = __float2bfloat16_rn(plain_value(act, v * s));
    else reinterpret_cast<float*>(out)[to] = v * s;
}

// The entries of an expert behind its first 16: tokens named it several times (a router does so for a row whose scores are not
// numbers).  One after the other, a warp to an output.  Rare, and a function of its own, so that the kernel keeps its registers.
template <int FORM>
__device__ __noinline__ void the_rest(const bf16* x, int ldx, const bf16* we, const int* ids, int n_entries, int top, const float* scale,
                                      void* out, int e, int n0, int N, int K, int x_rows, int act, float limit) {
    constexpr int MI = FORM == 1 ? 2 : 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i0 = 0, before = 0; i0 < n_entries; i0 += 32) {
        unsigned mine = __ballot_sync(0xffffffffu, i0 + lane < n_entries && ids[i0 + lane] == e);
        for (; mine != 0; mine &= mine - 1, ++before) {
            if (before < MAX_TOKENS) continue;
            const int entry = i0 + __ffs(mine) - 1, row = FORM != 0 ? entry / top : entry;
            const bool there = MG_GUARDED(moe_few, MG_GUARD_ROW, row, x_rows);
            for (int n = n0 + warp; n < min(n0 + ROWS, N); n += WARPS) {
                float v[2] = {0.f, 0.f};
                for (int k = lane; there && k < K; k += 32)
#pragma unroll
                    for (int i = 0; i < MI; ++i) v[i] = fmaf(to_float(x[(size_t)row * ldx + k]), to_float(we[(size_t)(i * N + n) * K + k]), v[i]);
#pragma unroll
                for (int i = 0; i < MI; ++i) v[i] = warp_sum(v[i]);
                if (lane == 0) finish<FORM>(v[0], v[MI - 1], entry, n, N, scale, act, limit, out);
            }
        }
    }
}

// Forms as mg_moe_gemm: 1 gated, 2 plain, 0 out.
template <int FORM>
__global__ void __launch_bounds__(32 * WARPS, FORM == 1 ? 0 : FORM == 0 ? 4 : 5)
moe_few_kernel(const bf16* __restrict__ x, int ldx, const bf16* __restrict__ w, long long w_expert_stride,
               const int* __restrict__ ids, int n_entries, int top, const float* __restrict__ scale, void* __restrict__ out,
               int* __restrict__ entry_slot, int n_experts, int N, int K, int x_rows, int act, float limit) {
    constexpr int MI = FORM == 1 ? 2 : 1;                  // m16 tiles: a gated unit's gate rows, then its up rows
    __shared__ int lists[WARPS][MAX_TOKENS];
    __shared__ float sums[WARPS][MI * ROWS][MAX_TOKENS + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int e = blockIdx.y, n0 = blockIdx.x * ROWS;
    // The second product's kernel (form 0) may start once all of the first's are behind their wait: the ids are there then, written
    // by a kernel that has ended, and its rows of the matrices can be under way while the first product is worked out.
    if (FORM == 0) {
        pdl_trigger();
    } else {
        pdl_wait();
        pdl_trigger();
    }
    // the expert's entries, in order; every warp finds them for itself
    int count = 0;
    for (int i0 = 0; i0 < n_entries; i0 += 32) {
        const int i = i0 + lane, id = i < n_entries ? __ldcg(ids + i) : -1;
        const unsigned mine = __ballot_sync(0xffffffffu, id == e);
        const int rank = count + __popc(mine & ((1u << lane) - 1u));
        if (id == e && rank < MAX_TOKENS) lists[warp][rank] = i;
        count += __popc(mine);
    }
    if (FORM == 0 && e == 0 && blockIdx.x == 0 && warp == 0) {
        pdl_wait();                                        // (nothing is written before it)
        for (int i = lane; i < n_entries; i += 32) entry_slot[i] = ids[i] >= 0 && ids[i] < n_experts ? i : -1;
    }
    if (count == 0) {
        if (FORM == 0) pdl_wait();                         // the kernel ends behind the one in front
        return;
    }
    const int entries = count;
    count = min(count, MAX_TOKENS);
    __syncwarp();
    const bf16* we = w + (size_t)e * w_expert_stride;
    const bf16* w_row[MI][2];                              // this lane's two rows of each tile
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + g + 8 * h;
            w_row[i][h] = n < N ? we + (size_t)(i * N + n) * K + 8 * t : nullptr;
        }
    uint4 a[MI][2][4];
    auto load_w = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {                      // 32 columns each: four lanes' 64 bytes of a row
            const int k = k0 + 32 * q;
            const bool in = k + 8 * t < K;
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    a[i][h][q] = w_row[i][h] != nullptr && in ? __ldcs(reinterpret_cast<const uint4*>(w_row[i][h] + k)) : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    if (FORM == 0) {
        load_w(warp * 128);
        pdl_wait();
    }
    const bf16* x_row[2] = {nullptr, nullptr};             // its tokens (columns g and g + 8)
#pragma unroll
    for (int c = 0; c < 2; ++c)
        if (g + 8 * c < count) {
            const int entry = lists[warp][g + 8 * c], row = FORM != 0 ? entry / top : entry;
            if (MG_GUARDED(moe_few, MG_GUARD_ROW, row, x_rows)) x_row[c] = x + (size_t)row * ldx + 8 * t;
        }
    float acc[MI][2][4];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c) acc[i][c][0] = acc[i][c][1] = acc[i][c][2] = acc[i][c][3] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const bool second = count > 8;                         // the same in all lanes
    for (int k0 = warp * 128; k0 < K; k0 += WARPS * 128) {
        uint4 b[2][4];
        if (FORM != 0 || k0 != warp * 128) load_w(k0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + 32 * q;
            const bool in = k + 8 * t < K;
            b[0][q] = x_row[0] != nullptr && in ? *reinterpret_cast<const uint4*>(x_row[0] + k) : zero;
            b[1][q] = second && x_row[1] != nullptr && in ? *reinterpret_cast<const uint4*>(x_row[1] + k) : zero;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < MI; ++i) {
                const uint4 lo = a[i][0][q], hi = a[i][1][q];
                mma_16816(acc[i][0], lo.x, hi.x, lo.y, hi.y, b[0][q].x, b[0][q].y);
                mma_16816(acc[i][0], lo.z, hi.z, lo.w, hi.w, b[0][q].z, b[0][q].w);
                if (second) {
                    mma_16816(acc[i][1], lo.x, hi.x, lo.y, hi.y, b[1][q].x, b[1][q].y);
                    mma_16816(acc[i][1], lo.z, hi.z, lo.w, hi.w, b[1][q].z, b[1][q].w);
                }
            }
    }
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int r = 0; r < 4; ++r) sums[warp][i * ROWS + g + 8 * (r >> 1)][8 * c + 2 * t + (r & 1)] = acc[i][c][r];
    __syncthreads();
    for (int o = tid; o < ROWS * count; o += 32 * WARPS) {
        const int row = o % ROWS, c = o / ROWS, n = n0 + row;
        if (n >= N) continue;
        float v[MI];
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            v[i] = 0.f;
#pragma unroll
            for (int k = 0; k < WARPS; ++k) v[i] += sums[k][i * ROWS + row][c];
        }
        finish<FORM>(v[0], v[MI - 1], lists[warp][c], n, N, scale, act, limit, out);
    }
    if (entries > MAX_TOKENS) the_rest<FORM>(x, ldx, we, ids, n_entries, top, scale, out, e, n0, N, K, x_rows, act, limit);
}

}  // namespace

// One of the two products for every entry of a step of up to 16 tokens.  ids: [n_tokens * top] chosen experts (-1: none; a token
// may name an expert several times); scale: [entries] or null; x: [x_rows, ldx], rows by token (forms 1 and 2) or by entry (form 0);
// out: [entries, N], bfloat16 (forms 1 and 2) or 32-bit; entry_slot: [entries], written by form 0: the entry itself, or -1.  Form 0 is
// launched right behind form 1 or 2 on the same ids: it reads them before that kernel has ended.
// Returns MG_ERR_UNSUPPORTED (and launches nothing) for sizes and alignments it does not take.
MG_API int mg_moe_few(const void* x, int ldx, const void* w, const int* ids, int n_tokens, int top, const float* scale, void* out,
                      int* entry_slot, int n_experts, int N, int K, int x_rows, int form, int act, float limit, void* stream) {
    if (n_tokens == 0) return MG_OK;
    MG_REQUIRE(n_tokens > 0 && n_experts > 0 && N > 0 && K > 0 && ldx >= K && top > 0 && form >= 0 && form <= 2, "moe (few tokens): bad sizes");
    if (n_tokens > MAX_TOKENS || K % 8 != 0 || ldx % 8 != 0 || n_experts > 65535 || (uintptr_t)x % 16 != 0 || (uintptr_t)w % 16 != 0)
        return mg_set_error(MG_ERR_UNSUPPORTED, "moe (few tokens): %d tokens, K=%d", n_tokens, K);
    MG_REQUIRE(form != 0 || entry_slot != nullptr, "moe (few tokens): no room for the entries' places");
    const long long stride = (long long)(form == 1 ? 2 : 1) * N * K;
    auto kernel = form == 1 ? moe_few_kernel<1> : form == 2 ? moe_few_kernel<2> : moe_few_kernel<0>;
    const cudaError_t e = mg_launch(kernel, dim3(ceil_div(N, ROWS), n_experts), dim3(32 * WARPS), 0, (cudaStream_t)stream, true,
                                    (const bf16*)x, ldx, (const bf16*)w, stride, ids, n_tokens * top, top, scale, out, entry_slot,
                                    n_experts, N, K, x_rows, act, limit);
    if (e != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "moe (few tokens): %s", cudaGetErrorString(e));
    return MG_OK;
}
