// Causal attention over the paged cache in 32-bit, for heads of 32, 64 or 128 features (keys and values alike), on the
// CUDA cores; the general kernel (attention_generic.cu) has every other size, mask and bias.
//
// A (token, head) pair's result is the same in whichever step and batch it is computed, whichever of the two kernels below
// computes it: keys are visited in blocks of 64 anchored at absolute multiples of 64; a block's scores (each one chain of
// fused multiply-adds over the features), its maximum m, its weights exp(s - m), their sum l and the weighted sum of the
// values (chains over the keys in order) depend on the block alone; and the blocks' (m, l, sum) are merged one after the
// other (merge_block).  A block in which a token sees no key changes nothing.
//
//   attention_fp32_split    steps of single tokens: a CTA per (token, kv head, key block) leaves (m, l, sum) in scratch, and
//                           attention_fp32_merge merges a (token, head)'s blocks in order.  Bound by latency, and by reading
//                           the keys and values once where there are many.
//   attention_fp32_tiles    portions of prompts: a CTA takes 64 tokens of one request and one head, 4 x 4 scores and 4 x
//                           (head / 16) outputs a thread, operands in shared memory; bound by shared-memory reads and FMA.
//
// 2,048 tokens of 8 prompts of 509, 8 heads of 64: the general kernel (a warp per token and head, a lane per key) 1,285 us a
// layer, the tiles 95; 8 single tokens behind such prompts 214 us and 12.
#include <math.h>

#include <type_traits>

#include "common.cuh"

MG_GUARD_DECLARE(attention_fp32)

namespace {

constexpr int TK = 64;               // keys per block
constexpr int TQ = 64;               // tokens per tile
constexpr int MAX_GROUP = 16;        // most query heads per kv head

struct Args {
    const float* q;                  // rows of q_stride, the first n_head * D are the queries
    const float* k_pages;            // [page][kv head][token in page][D]
    const float* v_pages;
    const int* block_table;
    const int* token_request;
    const int* positions;
    const int* req_q_start;
    const int* req_q_len;
    float* out;                      // [tokens][n_head * D]
    float* scratch;                  // [token][head][block of the pass][D + 2], then [token][head][D + 2]: merged so far
    const float* gate;
    const float* sinks;
    int q_stride, gate_stride, n_tokens, n_requests, n_head, n_kv_head, page_tokens, max_pages, num_pages, window;
    int blocks, first_block, last_pass;     // key blocks of this pass (single tokens), the first one, whether none come after
    float scale;
};

// One block's (m, l, acc) into what has been merged so far.  (A block in which a token sees no key has l = 0; one whose scores are
// all no numbers has m = -inf too, maxima pass them over, but l is no number, and neither is the token's result.)
template <int N>
__device__ __forceinline__ void merge_block(float& M, float& L, float (&A)[N], float m, float l, const float (&acc)[N]) {
    if (m == -INFINITY && l == 0.f) return;
    const float top = fmaxf(M, m);
    const float ca = M == -INFINITY ? 0.f : expf(M - top), cb = expf(m - top);
    L = fmaf(l, cb, __fmul_rn(L, ca));
#pragma unroll
    for (int i = 0; i < N; ++i) A[i] = fmaf(acc[i], cb, __fmul_rn(A[i], ca));
    M = top;
}

// The factor of the merged sums, with the head's sink (one more term in the softmax's sum) if there is one; *corr is what the
// sums are multiplied by first.
__device__ __forceinline__ float finish_row(float M, float L, const float* sinks, int head, float* corr) {
    *corr = 1.f;
    if (sinks) {
        const float top = fmaxf(M, sinks[head]);
        *corr = expf(M - top);
        L = __fadd_rn(__fmul_rn(L, *corr), expf(sinks[head] - top));
    }
    return 1.0f / L;                                         // (a token sees itself: only scores of -inf alone leave 0, and 0 / 0)
}

__device__ __forceinline__ float gated(float o, const float* gate) {
    return gate ? o * (1.0f / (1.0f + expf(-*gate))) : o;
}

__device__ __forceinline__ int first_key(int p, int window) { return window > 0 && p - window + 1 > 0 ? p - window + 1 : 0; }

// Row of key j in the page storage.
__device__ __forceinline__ long long key_row(const Args& a, const int* table, int kv_head, int j) {
    int page = table[j / a.page_tokens];
    if (!MG_GUARDED(attention_fp32, MG_GUARD_PAGE, page, a.num_pages)) page = 0;
    return ((long long)page * a.n_kv_head + kv_head) * a.page_tokens + j % a.page_tokens;
}

template <int D>
__global__ void __launch_bounds__(128)
attention_fp32_split(const Args a) {
    constexpr int LINE = D + 4;                              // words between rows: 16-byte reads of eight rows meet no bank twice
    extern __shared__ __align__(16) float smem[];
    const int group = a.n_head / a.n_kv_head;
    float* ks = smem;                                        // [TK][LINE]
    float* vs = ks + TK * LINE;
    float* qs = vs + TK * LINE;                              // [group][D]
    float* ps = qs + group * D;                              // [group][TK]: scores, then weights
    float* ms = ps + group * TK;                             // [group]
    __shared__ long long rows[TK];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int token = blockIdx.x, kv_head = blockIdx.y, z = blockIdx.z;
    pdl_trigger();
    pdl_wait();
    int p = a.positions[token];
    if (p < 0) return;                                       // padding row of a fixed-size batch
    if (!MG_GUARDED(attention_fp32, MG_GUARD_POSITION, p, (long long)a.max_pages * a.page_tokens)) p = 0;
    const int lo = first_key(p, a.window), block = lo / TK + a.first_block + z;
    if (block * TK > p) return;
    int request = a.token_request[token];
    if (!MG_GUARDED(attention_fp32, MG_GUARD_REQUEST, request, a.n_requests)) request = 0;
    const int* table = a.block_table + (size_t)request * a.max_pages;
    if (tid < TK) {
        const int j = block * TK + tid;
        rows[tid] = j >= lo && j <= p ? key_row(a, table, kv_head, j) : -1;
    }
    const float* qrow = a.q + (size_t)token * a.q_stride + (size_t)kv_head * group * D;
    for (int e = tid; e < group * D; e += 128) qs[e] = qrow[e] * a.scale;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TK * D / 4 / 128; ++i) {
        const int e = tid + 128 * i, r = e / (D / 4), c = e % (D / 4) * 4;
        const long long row = rows[r];
        float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
        if (row >= 0) {
            kv = *reinterpret_cast<const float4*>(a.k_pages + row * D + c);
            vv = *reinterpret_cast<const float4*>(a.v_pages + row * D + c);
        }
        *reinterpret_cast<float4*>(ks + r * LINE + c) = kv;
        *reinterpret_cast<float4*>(vs + r * LINE + c) = vv;
    }
    __syncthreads();
    const int key = tid & (TK - 1);
    for (int g = tid / TK; g < group; g += 2) {
        float dot = 0.f;
#pragma unroll
        for (int d = 0; d < D; d += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(ks + key * LINE + d), qv = *reinterpret_cast<const float4*>(qs + g * D + d);
            dot = fmaf(qv.x, kv.x, dot);
            dot = fmaf(qv.y, kv.y, dot);
            dot = fmaf(qv.z, kv.z, dot);
            dot = fmaf(qv.w, kv.w, dot);
        }
        ps[g * TK + key] = rows[key] >= 0 ? dot : -INFINITY;
    }
    __syncthreads();
    for (int g = warp; g < group; g += 4) {
        const float s0 = ps[g * TK + lane], s1 = ps[g * TK + lane + 32];
        const float m = warp_max(fmaxf(s0, s1));
        ps[g * TK + lane] = s0 == -INFINITY ? 0.f : expf(s0 - m);
        ps[g * TK + lane + 32] = s1 == -INFINITY ? 0.f : expf(s1 - m);
        if (lane == 0) ms[g] = m;
    }
    __syncthreads();
    for (int e = tid; e < group * D; e += 128) {
        const int g = e / D, d = e % D;
        float acc = 0.f, l = 0.f;
#pragma unroll 16
        for (int j = 0; j < TK; ++j) {
            const float pj = ps[g * TK + j];
            acc = fmaf(pj, vs[j * LINE + d], acc);
            l += pj;
        }
        float* dst = a.scratch + (((size_t)token * a.n_head + kv_head * group + g) * a.blocks + z) * (D + 2);
        dst[d] = acc;
        if (d == 0) {
            dst[D] = ms[g];
            dst[D + 1] = l;
        }
    }
}

template <int D>
__global__ void __launch_bounds__(D)
attention_fp32_merge(const Args a) {
    const int token = blockIdx.x, head = blockIdx.y, d = threadIdx.x;
    pdl_trigger();
    pdl_wait();
    float* out = a.out + ((size_t)token * a.n_head + head) * D + d;
    int p = a.positions[token];
    if (p < 0) {                                             // padding row of a fixed-size batch
        *out = 0.f;
        return;
    }
    if (!MG_GUARDED(attention_fp32, MG_GUARD_POSITION, p, (long long)a.max_pages * a.page_tokens)) p = 0;
    const int n = min(p / TK - first_key(p, a.window) / TK + 1 - a.first_block, a.blocks);
    const float* src = a.scratch + ((size_t)token * a.n_head + head) * a.blocks * (D + 2);
    float* so_far = a.scratch + ((size_t)a.n_tokens * a.n_head * a.blocks + (size_t)token * a.n_head + head) * (D + 2);
    float M = -INFINITY, L = 0.f, A[1] = {0.f};
    if (a.first_block > 0) {
        A[0] = so_far[d];
        M = so_far[D];
        L = so_far[D + 1];
    }
    for (int z0 = 0; z0 < n; z0 += 8) {
        float m[8], l[8], acc[8][1];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float* s = src + (size_t)min(z0 + i, n - 1) * (D + 2);
            acc[i][0] = s[d];
            m[i] = s[D];
            l[i] = s[D + 1];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (z0 + i < n) merge_block(M, L, A, m[i], l[i], acc[i]);
    }
    if (!a.last_pass) {
        __syncthreads();                                     // everybody has read what is replaced
        so_far[d] = A[0];
        if (d == 0) {
            so_far[D] = M;
            so_far[D + 1] = L;
        }
        return;
    }
    float corr;
    const float inv = finish_row(M, L, a.sinks, head, &corr);
    *out = gated(__fmul_rn(__fmul_rn(A[0], corr), inv), a.gate ? a.gate + (size_t)token * a.gate_stride + (size_t)head * D + d : nullptr);
}

template <int D>
__global__ void __launch_bounds__(256, 2)
attention_fp32_tiles(const Args a) {
    constexpr int LINE = TQ + 4;
    constexpr int NC = D / 16, VEC = NC < 4 ? NC : 4;        // output features a thread, in groups of VEC that lie 16 * VEC apart
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                        // [D][LINE]: queries, feature by feature
    float* ks = qs + D * LINE;                               // [D][LINE]
    float* vs = ks + D * LINE;                               // [TK][D]
    float* ps = vs + TK * D;                                 // [TK][LINE]: weights, key by key
    __shared__ long long rows[TK];
    const int tid = threadIdx.x, tr = tid / 16, tc = tid % 16, head = blockIdx.y;
    const int kv_head = head / (a.n_head / a.n_kv_head);
    pdl_trigger();
    pdl_wait();
    // the tile: the last ones first (a request's later tokens see more keys)
    int tile = (int)gridDim.x - 1 - (int)blockIdx.x, request = 0, len = 0;
    for (; request < a.n_requests; ++request) {
        len = a.req_q_len[request];
        const int tiles = (len + TQ - 1) / TQ;
        if (tile < tiles) break;
        tile -= tiles;
    }
    if (request >= a.n_requests) return;                     // (the host counted the same tiles)
    const int row0 = a.req_q_start[request] + tile * TQ, n_rows = min(TQ, len - tile * TQ);
    const int* table = a.block_table + (size_t)request * a.max_pages;
    int pos0 = a.positions[row0];
    if (!MG_GUARDED(attention_fp32, MG_GUARD_POSITION, pos0 + n_rows - 1, (long long)a.max_pages * a.page_tokens)) pos0 = 0;
    const int last = pos0 + n_rows - 1;
    for (int e = tid; e < TQ * (D / 4); e += 256) {
        const int r = e % TQ, d = e / TQ * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < n_rows) v = *reinterpret_cast<const float4*>(a.q + (size_t)(row0 + r) * a.q_stride + (size_t)head * D + d);
        qs[d * LINE + r] = v.x * a.scale;
        qs[(d + 1) * LINE + r] = v.y * a.scale;
        qs[(d + 2) * LINE + r] = v.z * a.scale;
        qs[(d + 3) * LINE + r] = v.w * a.scale;
    }
    float M[4], L[4], A[4][NC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        M[i] = -INFINITY;
        L[i] = 0.f;
#pragma unroll
        for (int c = 0; c < NC; ++c) A[i][c] = 0.f;
    }
    const int lo_first = first_key(pos0, a.window);
    for (int block = lo_first / TK; block <= last / TK; ++block) {
        const int key0 = block * TK;
        __syncthreads();                                     // the block before is through with keys, values and weights
        if (tid < TK) {
            const int j = key0 + tid;
            rows[tid] = j >= lo_first && j <= last ? key_row(a, table, kv_head, j) : -1;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TK * D / 4 / 256; ++i) {
            const int e = tid + 256 * i;
            {
                const int r = e % TK, d = e / TK * 4;        // neighbouring threads, neighbouring keys: no bank twice
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (rows[r] >= 0) v = *reinterpret_cast<const float4*>(a.k_pages + rows[r] * D + d);
                ks[d * LINE + r] = v.x;
                ks[(d + 1) * LINE + r] = v.y;
                ks[(d + 2) * LINE + r] = v.z;
                ks[(d + 3) * LINE + r] = v.w;
            }
            {
                const int r = e / (D / 4), d = e % (D / 4) * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (rows[r] >= 0) v = *reinterpret_cast<const float4*>(a.v_pages + rows[r] * D + d);
                *reinterpret_cast<float4*>(vs + r * D + d) = v;
            }
        }
        __syncthreads();
        float s[4][4];                                       // [token][key]
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 8
        for (int d = 0; d < D; ++d) {
            const float4 q4 = *reinterpret_cast<const float4*>(qs + d * LINE + 4 * tr), k4 = *reinterpret_cast<const float4*>(ks + d * LINE + 4 * tc);
            const float qv[4] = {q4.x, q4.y, q4.z, q4.w}, kv[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = fmaf(qv[i], kv[j], s[i][j]);
        }
        // every row of the tile sees every key of the block: no mask
        const bool whole = n_rows == TQ && key0 + TK - 1 <= pos0 && key0 >= first_key(last, a.window);
        float m[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int p = pos0 + 4 * tr + i, lo = first_key(p, a.window);
            if (!whole) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = key0 + 4 * tc + j;
                    if (4 * tr + i >= n_rows || key > p || key < lo) s[i][j] = -INFINITY;
                }
            }
            m[i] = fmaxf(fmaxf(s[i][0], s[i][1]), fmaxf(s[i][2], s[i][3]));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], o));
        }
        // the weights; -1 marks a key that the token does not see (its value is not touched: it may be no number)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = s[i][j] == -INFINITY ? (whole ? 0.f : -1.f) : expf(s[i][j] - m[i]);
            *reinterpret_cast<float4*>(ps + (4 * tc + j) * LINE + 4 * tr) = make_float4(w[0], w[1], w[2], w[3]);
        }
        __syncthreads();
        float acc[4][NC], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            l[i] = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) acc[i][c] = 0.f;
        }
        auto add_keys = [&](auto masked) {
#pragma unroll 4
            for (int j = 0; j < TK; ++j) {
                const float4 p4 = *reinterpret_cast<const float4*>(ps + j * LINE + 4 * tr);
                const float pj[4] = {p4.x, p4.y, p4.z, p4.w};
                float v[NC];
                const float* vrow = vs + j * D + VEC * tc;
                if constexpr (VEC == 4) {
#pragma unroll
                    for (int c = 0; c < NC; c += 4) *reinterpret_cast<float4*>(v + c) = *reinterpret_cast<const float4*>(vrow + 16 * c);
                } else {
                    *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(vrow);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (decltype(masked)::value && pj[i] < 0.f) continue;
#pragma unroll
                    for (int c = 0; c < NC; ++c) acc[i][c] = fmaf(pj[i], v[c], acc[i][c]);
                    l[i] += pj[i];
                }
            }
        };
        if (whole) add_keys(std::false_type());
        else add_keys(std::true_type());
#pragma unroll
        for (int i = 0; i < 4; ++i) merge_block(M[i], L[i], A[i], m[i], l[i], acc[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * tr + i;
        if (r >= n_rows) continue;
        float corr;
        const float inv = finish_row(M[i], L[i], a.sinks, head, &corr);
        float* dst = a.out + ((size_t)(row0 + r) * a.n_head + head) * D;
        const float* grow = a.gate ? a.gate + (size_t)(row0 + r) * a.gate_stride + (size_t)head * D : nullptr;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = VEC * tc + 16 * (c / VEC * VEC) + c % VEC;
            dst[d] = gated(__fmul_rn(__fmul_rn(A[i][c], corr), inv), grow ? grow + d : nullptr);
        }
    }
}

template <int D>
cudaError_t launch(const Args& a, int tiles, int all_blocks, cudaStream_t s) {
    const int group = a.n_head / a.n_kv_head;
    if (tiles > 0) {
        constexpr int smem = (2 * D * (TQ + 4) + TK * D + TK * (TQ + 4)) * (int)sizeof(float);
        const cudaError_t configured = mg_raise_shared(attention_fp32_tiles<D>, smem);
        if (configured != cudaSuccess) return configured;
        return mg_launch(attention_fp32_tiles<D>, dim3(tiles, a.n_head), dim3(256), smem, s, true, a);
    }
    constexpr int most = (2 * TK * (D + 4) + MAX_GROUP * (D + TK + 1)) * (int)sizeof(float);
    const cudaError_t configured = mg_raise_shared(attention_fp32_split<D>, most);
    if (configured != cudaSuccess) return configured;
    const int smem = (2 * TK * (D + 4) + group * (D + TK + 1)) * (int)sizeof(float);
    Args pass = a;
    for (pass.first_block = 0; pass.first_block < all_blocks; pass.first_block += a.blocks) {
        pass.last_pass = pass.first_block + a.blocks >= all_blocks;
        cudaError_t e = mg_launch(attention_fp32_split<D>, dim3(a.n_tokens, a.n_kv_head, a.blocks), dim3(128), smem, s, true, pass);
        if (e == cudaSuccess) e = mg_launch(attention_fp32_merge<D>, dim3(a.n_tokens, a.n_head), dim3(D), 0, s, true, pass);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

// Key blocks that a single token with a context of up to max_context keys can touch.
MG_API int mg_attention_fp32_blocks(int max_context, int window) {
    const int all = ceil_div(max_context, TK);
    return window > 0 && ceil_div(window, TK) + 1 < all ? ceil_div(window, TK) + 1 : all;
}
// ... of which this many are done in one pass: as many as 64 MB of scratch hold.
MG_API int mg_attention_fp32_pass_blocks(int n_tokens, int n_head, int head_dim, int blocks) {
    const long long fit = (64ll << 20) / ((long long)n_tokens * n_head * (head_dim + 2) * (long long)sizeof(float));
    return (int)(fit < 1 ? 1 : fit > blocks ? blocks : fit > 65535 ? 65535 : fit);
}
MG_API int mg_attention_fp32_tiles(int q_len) { return ceil_div(q_len, TQ); }

// Whether the kernels have these sizes (which hang on the model alone).
MG_API int mg_attention_fp32_takes(int n_head, int n_kv_head, int head_dim) {
    return (head_dim == 32 || head_dim == 64 || head_dim == 128) && n_kv_head > 0 && n_head % n_kv_head == 0 &&
           n_head / n_kv_head <= MAX_GROUP && n_head <= 65535;
}

// Arguments as mg_paged_attention_general, head_dim features in keys and values alike.  Portions of prompts: `tiles` is the
// sum of mg_attention_fp32_tiles over the requests and req_q_start / req_q_len say where each request's rows lie.  Single
// tokens: tiles = 0, `blocks` and `pass_blocks` as above, scratch of n_tokens * n_head * (pass_blocks + 1) * (head_dim + 2) numbers.
// Returns MG_ERR_UNSUPPORTED (and launches nothing) for sizes and alignments that the kernels do not have.
MG_API int mg_attention_fp32(const float* q, int q_stride, const float* k_pages, const float* v_pages, const int* block_table,
                             const int* token_request, const int* positions, const int* req_q_start, const int* req_q_len,
                             const float* gate, int gate_stride, float* out, float* scratch, int n_tokens, int n_requests,
                             int n_head, int n_kv_head, int head_dim, int page_tokens, int max_pages, int window, float scale,
                             int num_pages, int tiles, int blocks, int pass_blocks, const float* sinks, void* stream) {
    if (n_tokens == 0) return MG_OK;
    MG_REQUIRE(n_tokens > 0 && n_head > 0 && n_kv_head > 0 && n_head % n_kv_head == 0 && page_tokens > 0 && max_pages > 0 && n_requests > 0,
               "attention: bad sizes");
    if (!mg_attention_fp32_takes(n_head, n_kv_head, head_dim) || q_stride % 4 != 0 || ((uintptr_t)q & 15) || ((uintptr_t)k_pages & 15) ||
        ((uintptr_t)v_pages & 15))
        return mg_set_error(MG_ERR_UNSUPPORTED, "attention: no 32-bit tiles for heads of %d", head_dim);
    MG_REQUIRE(q_stride >= n_head * head_dim && (gate == nullptr || gate_stride >= n_head * head_dim), "attention: rows shorter than their heads");
    MG_REQUIRE(tiles > 0 ? req_q_start && req_q_len : scratch && blocks > 0 && pass_blocks > 0 && pass_blocks <= 65535,
               "attention: nothing to cut the step by");
    const Args a = {q, k_pages, v_pages, block_table, token_request, positions, req_q_start, req_q_len, out, scratch, gate, sinks,
                    q_stride, gate_stride, n_tokens, n_requests, n_head, n_kv_head, page_tokens, max_pages, num_pages, window,
                    pass_blocks, 0, 1, scale};
    cudaStream_t s = (cudaStream_t)stream;
    const cudaError_t e = head_dim == 32   ? launch<32>(a, tiles, blocks, s)
                          : head_dim == 64 ? launch<64>(a, tiles, blocks, s)
                                           : launch<128>(a, tiles, blocks, s);
    if (e != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "attention (32-bit): %s", cudaGetErrorString(e));
    MG_CHECK_LAUNCH("attention_fp32");
    return MG_OK;
}
