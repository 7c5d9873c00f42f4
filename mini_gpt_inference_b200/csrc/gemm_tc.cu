// bfloat16 matrix product on the 5th-generation tensor cores: TMA -> shared memory -> tcgen05.mma -> TMEM ->
// shared memory -> TMA.
//
//   D[m, n] = sum_k A[m, k] * B[n, k]        A: [M, K] activations, B: [N, K] weights, both K-major bf16
//
// A CTA, or a pair of CTAs (CG = 2, a cluster of two on neighbouring SMs whose tensor cores work on one product), computes
// tiles of 128 * CG x BN of D, one after the other.  Ten warps: eight for the epilogue, one with a thread that loads (64 or 128
// columns of K at a time into a ring of stages, 128-byte swizzle), one with a thread that issues the products.  In a pair
// each CTA loads its own 128 rows of A and its half of the BN rows of B; the CTA of rank 0 issues for both.  The accumulator
// lies in TMEM, twice if a CTA has more than one tile: the epilogue of a tile then runs beside the products of the next.
//
// Epilogue: two warps to each 32 TMEM lanes (rows), which take boxes of 128 bytes a row in turn.  A warp reads its lanes 32
// columns at a time, applies bias and activation, and lays the values into one of its two boxes of 4 KB in shared memory, in the
// swizzled order that the copy engine wants; one thread stores the box, or adds it to the 32-bit residual stream (every
// element has one summand, so the sum is that of a load, an add and a store).  Keys and values of the QKV projection are
// copied from the same box to their cache rows, eight lanes to 128 bytes.  Rows of D that are no multiple of 16 bytes are
// written from there with plain stores, 32 neighbouring columns at a time.
//
// What bounds it: reading the tiles from L2.  A tile of 128 x 128 asks 32 KB for every 64 columns of K, 256 clocks of
// tensor-core work; an SM takes in some 50 to 60 bytes a clock, so such a tile cannot run above half the tensor cores'
// rate.  A pair with BN = 256 asks 32 KB a CTA for 512 clocks.  (The earlier epilogue, a thread to a row, stored and read
// 16 bytes from each of 32 lines an instruction: 4 to 8 us of the 13 that a product of 2,048 x 512 x 512 took.)
//
// Edges need no special case on the load side: TMA fills what lies outside the matrices with zeros (also a K that is no
// multiple of 64), and its stores leave out what lies outside.
//
// Every wait on an mbarrier is bounded.  If one runs out, the kernel records a code in `status`, stores no tile whose products are
// not complete (a pair's CTAs learn of it by their own waits running out), waits a moment for copies in flight, frees its TMEM and
// returns; the host reads `status` later.  No multicast loads: each CTA loads its own tiles.
#include <cuda.h>

#include "blackwell.cuh"
#include "moe_units.cuh"
#include "tensor_map.cuh"

MG_STAMP_DECLARE(gemm)
MG_GUARD_DECLARE(linear_tc)

#define EPI_STORE 0
#define EPI_GELU 1
#define EPI_RELU_SQ 3
#define EPI_RESIDUAL 2

namespace {

constexpr int TILE_M = 128;         // rows of A per CTA
constexpr int BLOCK_K = 64;         // bf16 elements per k block = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int MAX_STAGES = 8;
constexpr int MAX_BN = 256;
constexpr int A_TILE_BYTES = TILE_M * BLOCK_K * 2;
constexpr int EPI_WARPS = 8;                                 // two to each 32 lanes of TMEM
constexpr int BOX_BYTES = 32 * 128;                          // 32 rows of 128 bytes: what a warp stores at a time
constexpr int BOXES = 2;                                     // ... of which it has two that take turns
constexpr int THREADS = 32 * (EPI_WARPS + 2);
constexpr int SMS = 148;

struct __align__(16) Control {
    uint64_t full[MAX_STAGES];
    uint64_t empty[MAX_STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint32_t tmem_base;
    uint32_t failed;
};

// Where the QKV projection also leaves the key and value features of each token: its row of
// the paged cache.  k_pages null: no such copy.
struct KvSink {
    bf16* k_pages;
    bf16* v_pages;
    const int* slots;                // [tokens] flat cache row, < 0: skip
    int q_width, n_kv_head, head_dim, page_tokens;
    int num_pages;                   // pages of the pool (what a cache row is held against in guarded builds)
};

// What the products are of.
constexpr int PLAIN = 0;             // one matrix
constexpr int HEADS = 1;             // a small matrix per head: columns a_off + h * a_head .. of A give columns o_off + h * o_head .. of D
constexpr int EXPERTS = 2;           // a matrix per expert: rows offsets[e] .. offsets[e + 1] of A (and D) belong to expert e
constexpr int HEADS_IN = 3;          // HEADS with matrices whose rows are inputs (their columns the results)
constexpr int MAX_EXPERTS = 256;

struct GemmArgs {
    const float* bias;
    void* out;                       // [M, N] bf16 or 32-bit; the residual stream for EPI_RESIDUAL
    int M, N, K, bn, stages;
    int a_rows;                      // rows of A that a load brings: TILE_M, or fewer where A has no more
    int epilogue, out_bf16;
    int boxes;                       // rows of the output are multiples of 16 bytes: stored by TMA
    KvSink sink;
    int* status;
    int ld_out;                      // elements between rows of D
    int heads, a_off, a_head, o_off, o_head;               // HEADS, HEADS_IN; N and K are a head's
    // EXPERTS: form 0 (32-bit results), 1 (gated: a matrix has N gate rows, then N up rows), 2 (activation), as in moe.cu;
    // scale: factor on the sums of row r's entry, slot_entry[r] (null: none)
    const int* offsets;
    const int* slot_entry;
    const float* scale;
    int n_experts, form, act;
    float limit;
};

// A tile's place: first row of this CTA's part of A (and D), columns of A, rows of B, columns of a head's or matrix's results
// and of D, and the row of D behind its last.
struct Place {
    int row, a_col, b_row, n0, out_col, rows_end;
};

// EXACT: GELU results that become bfloat16 are right to their last place (up to 128 rows, decoding); otherwise their whole groups of
// 32 columns take the hardware's tanh (prompts: 0.7 us less of 10 at 2,048 x 2,048 x 512).
template <int CG, int SUB, int MODE, bool EXACT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_out, const GemmArgs g) {
    extern __shared__ uint8_t smem_raw[];
    // 128-byte swizzle wants tiles aligned to 1024 bytes
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bn = g.bn, stages = g.stages;
    const int b_rows = bn / CG;
    constexpr uint32_t B_OFFSET = SUB * A_TILE_BYTES;        // a stage: SUB tiles of A, then as many of B
    const uint32_t b_tile_bytes = b_rows * BLOCK_K * 2, stage_bytes = B_OFFSET + SUB * b_tile_bytes;
    const uint32_t loaded = CG * SUB * (g.a_rows * BLOCK_K * 2 + b_tile_bytes);      // bytes that a stage's loads bring
    uint8_t* boxes = smem + (size_t)stages * stage_bytes;
    Control* ctl = (Control*)(boxes + EPI_WARPS * BOXES * BOX_BYTES);

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (the same register value in all lanes)
    const int rank = CG == 2 ? (int)cluster_rank() : 0;
    constexpr bool BY_HEAD = MODE == HEADS || MODE == HEADS_IN;
    const bool glu = MODE == EXPERTS && g.form == 1;         // bn / 2 gate columns, then the up columns of the same results
    const int bn_out = glu ? bn / 2 : bn;                    // results a tile has
    int m_tiles = (g.M + CG * TILE_M - 1) / (CG * TILE_M);
    const int n_tiles = (g.N + bn_out - 1) / bn_out;
    int tiles = m_tiles * n_tiles * (BY_HEAD ? g.heads : 1);
    const int first_tile = (int)blockIdx.x / CG, tile_step = (int)gridDim.x / CG;
    __shared__ int expert_row[MODE == EXPERTS ? MAX_EXPERTS + 1 : 1], expert_tile[MODE == EXPERTS ? MAX_EXPERTS + 1 : 1];
    const int num_kb = (g.K + SUB * BLOCK_K - 1) / (SUB * BLOCK_K);     // stages' worth of K
    const bool twice = MODE == EXPERTS || tiles > tile_step;                    // some CTA has several tiles: two accumulators
    uint32_t tmem_cols = 32;
    while (tmem_cols < (uint32_t)(twice ? 2 * bn : bn)) tmem_cols *= 2;

    auto place_of = [&](int tile) {
        Place p;
        if (MODE == EXPERTS) {
            const int mt = tile % m_tiles, nt = tile / m_tiles;
            int e = 0;
            for (int half = MAX_EXPERTS; half > 0; half >>= 1)             // the last expert whose tiles begin at or before mt
                if (e + half < g.n_experts && expert_tile[e + half] <= mt) e += half;
            p.row = expert_row[e] + (mt - expert_tile[e]) * TILE_M;
            p.rows_end = expert_row[e + 1];
            p.a_col = 0;
            p.n0 = p.out_col = nt * bn_out;
            p.b_row = e * (glu ? 2 : 1) * g.N + p.n0;
            return p;
        }
        int nt = tile / m_tiles;
        const int h = BY_HEAD ? nt / n_tiles : 0;
        nt -= h * n_tiles;
        p.row = (tile % m_tiles) * CG * TILE_M + rank * TILE_M;
        p.rows_end = g.M;
        p.n0 = nt * bn;
        p.a_col = BY_HEAD ? g.a_off + h * g.a_head : 0;
        p.b_row = MODE == HEADS_IN ? h * g.K : (MODE == HEADS ? h * g.N : 0) + p.n0 + rank * b_rows;
        p.out_col = (BY_HEAD ? g.o_off + h * g.o_head : 0) + p.n0;
        return p;
    };

    // HEADS_IN: k block kb of B, 64 inputs by 64 results at a time
    auto load_inputs = [&](uint32_t tile_b, uint32_t full, int kb, int b_row, int n0) {
        for (int n = 0; n < bn; n += 64) tma_load_2d_group<CG>(tile_b + n * BLOCK_K * 2, &map_b, full, n0 + n, b_row + kb * BLOCK_K);
    };

    MG_STAMP(gemm, 0);
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(&ctl->acc_full[a]), 1);
            mbar_init(smem_u32(&ctl->acc_empty[a]), CG * EPI_WARPS);
        }
        ctl->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == EPI_WARPS + 1) tmem_alloc_group<CG>(smem_u32(&ctl->tmem_base), tmem_cols);
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_barrier();                          // the pair's barriers and both halves of TMEM are there
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    const uint32_t full0 = smem_u32(&ctl->full[0]), loads_on = CG == 2 ? leader_address(full0) : full0;   // a pair's loads count on rank 0's
    // Barriers and tensor memory are set up while the kernel in front drains; its results (the activations, the residual
    // stream) are touched only behind the wait.  The weights do not come from the kernel in front: their tiles of the
    // first round of stages are asked for before it.
    MG_STAMP(gemm, 2);
    pdl_trigger();
    // (Which experts have rows is the kernel in front's to say: nothing of theirs is asked for before it.)
    const int early = MODE == EXPERTS ? 0 : num_kb < stages ? num_kb : stages;
    const bool loads = warp == EPI_WARPS, issues = warp == EPI_WARPS + 1;
    if (MODE != EXPERTS && loads && elect_one()) {
        const Place p = place_of(first_tile);
        const int n0 = p.b_row;
        for (int kb = 0; kb < early; ++kb) {
            const uint32_t full = loads_on + kb * 8, tile_b = smem_u32(smem) + kb * stage_bytes + B_OFFSET;
            if (rank == 0) mbar_expect_tx(full0 + kb * 8, loaded);
            if constexpr (MODE == HEADS_IN) load_inputs(tile_b, full, kb, n0, p.n0);
            else
#pragma unroll
                for (int i = 0; i < SUB; ++i) tma_load_2d_group<CG>(tile_b + i * b_tile_bytes, &map_b, full, (kb * SUB + i) * BLOCK_K, n0);
        }
    }
    pdl_wait();
    MG_STAMP(gemm, 3);
    if (MODE == EXPERTS) {
        for (int e = tid; e <= g.n_experts; e += THREADS) expert_row[e] = g.offsets[e];
        __syncthreads();
        if (warp == 0) {                                     // each expert's first tile: sums over 32 experts at a time
            int before = 0;
            for (int e0 = 0; e0 < g.n_experts; e0 += 32) {
                const int e = e0 + lane;
                int sum = e < g.n_experts ? (expert_row[e + 1] - expert_row[e] + TILE_M - 1) / TILE_M : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int n = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += n;
                }
                if (e < g.n_experts) expert_tile[e + 1] = before + sum;
                before += __shfl_sync(0xffffffffu, sum, 31);
            }
            if (lane == 0) expert_tile[0] = 0;
        }
        __syncthreads();
        m_tiles = expert_tile[g.n_experts];
        tiles = m_tiles * n_tiles;
    }

    // A single thread runs each of the next two loops, and the chain of its instructions is what bounds small tiles: some
    // 300 clocks a stage, whatever its size.  So the ring's place and parity are carried along (the two divisions that found
    // them took as long as the rest), the thread is chosen by elect.sync (behind a comparison with threadIdx the compiler
    // wraps each load and product in a loop over the lanes: 560 clocks a stage), and small tiles take two k blocks a stage.
    if (loads) {
        // ---- loads into the ring of stages ----
        if (elect_one()) {
            int s = 0, ahead = early;                        // stages whose weights are on their way already
            uint32_t parity = 1;
            bool ok = true;
            for (int tile = first_tile; tile < tiles && ok; tile += tile_step) {
                const Place p = place_of(tile);
                const int m0 = p.row, n0 = p.b_row, k0 = p.a_col;
                for (int kb = 0; kb < num_kb; ++kb) {
                    const uint32_t full = loads_on + s * 8, stage = smem_u32(smem) + s * stage_bytes;
                    if (ahead > 0) {
                        --ahead;
#pragma unroll
                        for (int i = 0; i < SUB; ++i) tma_load_2d_group<CG>(stage + i * A_TILE_BYTES, &map_a, full, k0 + (kb * SUB + i) * BLOCK_K, m0);
                    } else {
                        if (!mbar_wait(smem_u32(&ctl->empty[s]), parity)) {
                            atomicExch(g.status, 1);
                            ctl->failed = 1;
                            ok = false;
                            break;
                        }
                        if (rank == 0) mbar_expect_tx(full0 + s * 8, loaded);
#pragma unroll
                        for (int i = 0; i < SUB; ++i) {
                            tma_load_2d_group<CG>(stage + i * A_TILE_BYTES, &map_a, full, k0 + (kb * SUB + i) * BLOCK_K, m0);
                            if constexpr (MODE == HEADS_IN) {
                                load_inputs(stage + B_OFFSET, full, kb, n0, p.n0);
                                continue;
                            }
                            tma_load_2d_group<CG>(stage + B_OFFSET + i * b_tile_bytes, &map_b, full, (kb * SUB + i) * BLOCK_K, n0);
                            if (glu)                         // (the map's boxes are bn / 2 rows high)
                                tma_load_2d_group<CG>(stage + B_OFFSET + i * b_tile_bytes + b_tile_bytes / 2, &map_b, full,
                                                      (kb * SUB + i) * BLOCK_K, n0 + g.N);
                        }
                    }
                    if (++s == stages) { s = 0; parity ^= 1; }
                }
            }
        }
    } else if (issues) {
        // ---- products of the stages as they arrive ----
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = MODE == HEADS_IN ? instr_desc_bf16(TILE_M, 64, true) : instr_desc_bf16(CG * TILE_M, bn);
            const uint64_t desc0 = smem_desc_sw128(smem_u32(smem));
            int s = 0, round = 0;
            uint32_t parity = 0;
            bool ok = true;
            for (int tile = first_tile; tile < tiles && ok; tile += tile_step, ++round) {
                const int a = twice ? round & 1 : 0;
                const uint32_t acc = tmem_base + a * bn;
                // (the first use of an accumulator waits for nobody)
                ok = mbar_wait(smem_u32(&ctl->acc_empty[a]), ((round >> 1) & 1) ^ 1);
                tc_fence_after();
                for (int kb = 0; kb < num_kb && ok; ++kb) {
                    if (!(ok = mbar_wait(smem_u32(&ctl->full[s]), parity))) break;
                    tc_fence_after();
                    // (shared memory ends below 2^18 bytes: the 14 bits of the address field hold address / 16 without a carry)
                    const uint64_t desc_a = desc0 + (uint64_t)((s * stage_bytes) >> 4), desc_b = desc_a + (B_OFFSET >> 4);
                    if constexpr (MODE == HEADS_IN) {        // 64 results a product; rows of B are k, 16 of them 2 KB further
                        for (int n = 0; n < bn; n += 64)
#pragma unroll
                            for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                                umma_bf16_group<CG>(acc + n, desc_a + (uint64_t)((k * UMMA_K * 2) >> 4),
                                                    desc_b + (uint64_t)((n * BLOCK_K * 2 + k * UMMA_K * 128) >> 4), idesc, (k | kb) != 0 ? 1u : 0u);
                    } else {
#pragma unroll
                        for (int i = 0; i < SUB; ++i)
#pragma unroll
                            for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
                                // 16 elements further along K: 32 bytes inside the swizzled row
                                const uint64_t step = (uint64_t)((k * UMMA_K * 2) >> 4);
                                umma_bf16_group<CG>(acc, desc_a + (uint64_t)(i * (A_TILE_BYTES >> 4)) + step,
                                                    desc_b + (uint64_t)(i * (b_tile_bytes >> 4)) + step, idesc,
                                                    (i | k) != 0 || kb != 0 ? 1u : 0u);
                            }
                    }
                    umma_commit_group<CG>(smem_u32(&ctl->empty[s]));
                    if (++s == stages) { s = 0; parity ^= 1; }
                }
                if (ok) umma_commit_group<CG>(smem_u32(&ctl->acc_full[a]));
            }
            // (an accumulator that is not whole is not handed on: the epilogues' own waits, in both CTAs of a pair, run out then)
            if (!ok) {
                atomicExch(g.status, 2);
                ctl->failed = 1;
            }
        }
    } else if (warp < EPI_WARPS) {
        // ---- epilogue: eight warps, two to each 32 lanes of TMEM ----
        const int per_box = g.out_bf16 ? 64 : 32;            // columns of a 128-byte row
        const int quarter = warp & 3, first_box = (warp >> 2) * per_box;       // this warp's lanes, and its first columns
        const bool bias_wide = ((uintptr_t)g.bias & 15) == 0;
        int used = 0, round = 0;                             // boxes filled so far, tiles done so far
        for (int tile = first_tile; tile < tiles; tile += tile_step, ++round) {
            const int a = twice ? round & 1 : 0;
            const Place p = place_of(tile);
            const int row0 = p.row + quarter * 32, n0 = p.n0, out_col = p.out_col;
            float row_scale = 1.f;
            if (MODE == EXPERTS && g.scale != nullptr && row0 + lane < p.rows_end) row_scale = g.scale[g.slot_entry[row0 + lane]];
            // asked for while the products run: the cache row of this lane's token
            long long kv_row = -1;                           // the cache row's first element for kv head 0, in head rows
            if (g.sink.k_pages != nullptr && n0 + bn > g.sink.q_width && row0 + lane < g.M) {
                const int slot = g.sink.slots[row0 + lane];
                // (guarded builds: a row beyond the pool is recorded and its keys and values are not copied)
                if (slot >= 0 && MG_GUARDED(linear_tc, MG_GUARD_CACHE_ROW, slot, (long long)g.sink.num_pages * g.sink.page_tokens)) {
                    const int page = slot / g.sink.page_tokens;
                    kv_row = (long long)page * g.sink.n_kv_head * g.sink.page_tokens + (slot - page * g.sink.page_tokens);
                }
            }
            bool good = mbar_wait(smem_u32(&ctl->acc_full[a]), twice ? (round >> 1) & 1 : 0);
            if (!good) {
                atomicExch(g.status, 3);
                ctl->failed = 1;
            }
            good = good && (*(volatile uint32_t*)&ctl->failed == 0);
            if (!__all_sync(0xffffffffu, good)) break;       // tcgen05.ld needs the whole warp
            tc_fence_after();
            MG_STAMP(gemm, 5);
            const uint32_t lane_addr = tmem_base + a * bn + ((uint32_t)(quarter * 32) << 16);
            const int columns = min(bn_out, g.N - n0);
            // all of the accumulator's columns that are this warp's are in registers: the next tile's products may overwrite them
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (CG == 2) mbar_arrive_leader(smem_u32(&ctl->acc_empty[a]));
                    else mbar_arrive(smem_u32(&ctl->acc_empty[a]));
                }
            };
            if (first_box >= columns) release();
            for (int c0 = first_box; c0 < columns; c0 += 2 * per_box, ++used) {
                uint8_t* box = boxes + (warp * BOXES + used % BOXES) * BOX_BYTES;
                // the copy engine has read what this box held before
                if (g.boxes && lane == 0) tma_store_wait_read<BOXES - 1>();
                __syncwarp();
                for (int half = 0; half < per_box; half += 32) {
                    uint32_t r[32];
                    tmem_load_32(lane_addr + (uint32_t)(c0 + half), r);
                    float v[32];                             // the bias first: all lanes read the same 16 bytes
                    const int n = n0 + c0 + half;
                    if (g.bias != nullptr && bias_wide && n + 32 <= g.N) {
#pragma unroll
                        for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(v + j) = *reinterpret_cast<const float4*>(g.bias + n + j);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = g.bias != nullptr && n + j < g.N ? g.bias[n + j] : 0.f;
                    }
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] += __uint_as_float(r[j]);
                    if (MODE == EXPERTS) {
                        if (glu) {
                            tmem_load_32(lane_addr + (uint32_t)(bn_out + c0 + half), r);
                            tmem_wait_ld();
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = gated_value(g.act, g.limit, v[j] * row_scale, __uint_as_float(r[j]) * row_scale);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = g.form == 2 ? plain_value(g.act, v[j] * row_scale) : v[j] * row_scale;
                        }
                    } else if (g.epilogue == EPI_GELU) {
                        if (EXACT && g.out_bf16) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = gelu_exp(v[j]);
                        } else if (!EXACT && g.out_bf16 && n + 32 <= g.N && g.N % 8 == 0) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = gelu_tanh_fast(v[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
                        }
                    } else if (g.epilogue == EPI_RELU_SQ) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = relu_sq(v[j]);
                    }
                    // 16-byte pieces of this lane's row, in the 128-byte swizzle's places
                    if (g.out_bf16) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            uint4 o;
                            __nv_bfloat162 h[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
                            o = *reinterpret_cast<uint4*>(h);
                            *reinterpret_cast<uint4*>(box + lane * 128 + (((half / 8 + j) ^ (lane & 7)) << 4)) = o;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            *reinterpret_cast<float4*>(box + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                                make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    }
                }
                if (c0 + 2 * per_box >= columns) release();
                // (the rows behind an expert's last are the next expert's: such a box is not stored as one)
                const bool as_box = g.boxes && (MODE != EXPERTS || row0 + 32 <= p.rows_end);
                if (as_box) async_proxy_fence();
                __syncwarp();
                if (as_box) {
                    if (lane == 0) {
                        if (row0 < g.M) {
                            if (g.epilogue == EPI_RESIDUAL) tma_add_2d(&map_out, smem_u32(box), out_col + c0, row0);
                            else tma_store_2d(&map_out, smem_u32(box), out_col + c0, row0);
                        }
                        tma_store_commit();
                    }
                } else {
                    if (g.boxes && lane == 0) tma_store_commit();            // (an empty group keeps the count of boxes in use)
                    // rows that TMA cannot address: a row's columns from neighbouring lanes
                    const int wide = min(per_box, columns - c0), high = min(32, p.rows_end - row0);
                    for (int j = lane; j < wide; j += 32) {
                        const int byte = g.out_bf16 ? 2 * j : 4 * j;
#pragma unroll 8
                        for (int i = 0; i < high; ++i) {
                            const uint8_t* from = box + i * 128 + (((byte >> 4) ^ (i & 7)) << 4) + (byte & 15);
                            const size_t to = (size_t)(row0 + i) * g.ld_out + out_col + c0 + j;
                            if (g.out_bf16) ((bf16*)g.out)[to] = *reinterpret_cast<const bf16*>(from);
                            else if (g.epilogue == EPI_RESIDUAL) atomicAdd((float*)g.out + to, *reinterpret_cast<const float*>(from));
                            else ((float*)g.out)[to] = *reinterpret_cast<const float*>(from);
                        }
                    }
                }
                if (g.sink.k_pages != nullptr && n0 + c0 + per_box > g.sink.q_width) {
                    // eight lanes to a row of 64 features, eight features (of one head: head sizes are multiples of 8) each
                    const int n = n0 + c0 + 8 * (lane & 7);
                    const bool mine = n >= g.sink.q_width && n < g.N;
                    const int kv_width = g.sink.n_kv_head * g.sink.head_dim;
                    const int f = n - g.sink.q_width, which = f >= kv_width ? 1 : 0, fi = f - which * kv_width;
                    const int h = fi / g.sink.head_dim, d = fi - h * g.sink.head_dim;
                    bf16* pages = which ? g.sink.v_pages : g.sink.k_pages;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = 4 * i + (lane >> 3);
                        const long long base = __shfl_sync(0xffffffffu, kv_row, r);
                        if (mine && base >= 0)
                            *reinterpret_cast<uint4*>(pages + (base + (long long)h * g.sink.page_tokens) * g.sink.head_dim + d) =
                                *reinterpret_cast<const uint4*>(box + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
                    }
                }
                __syncwarp();
            }
        }
        if (g.boxes && lane == 0) tma_store_wait_all();
        MG_STAMP(gemm, 6);
    }
    __syncwarp();
    // something timed out: give copies that may still be in flight a moment to land
    if (*(volatile uint32_t*)&ctl->failed != 0 && lane == 0)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    if (CG == 2) cluster_barrier();                          // nobody's products, barriers or TMEM are in use any more
    tc_fence_after();
    MG_STAMP(gemm, 7);
    if (warp == EPI_WARPS + 1) tmem_dealloc_group<CG>(tmem_base, tmem_cols);
}

// ---- host side -----------------------------------------------------------------------------------
// How a product is cut: CTAs per tile, columns of a tile, k blocks per stage.
struct Cut {
    int cg, bn, sub;
};

// Rows of A in a load.  (What a tile's other rows hold in shared memory goes into results that nobody stores.  Filling them with
// zeros cost heads of 17 rows: 50,257 x 1,600 44.4 -> 38.9 us, 6,144 x 2,048 17.7 -> 13.6.)
inline int box_rows(int M) { return M >= TILE_M ? TILE_M : (M + 31) / 32 * 32; }

// The cut with the least time by a count of what bounds a tile, in microseconds (each figure from products of 64 to 2,048
// rows by 512 to 50,304 columns at K of 512 to 8,192):
//   a k block takes 0.175 of issue (0.125 where a stage holds two), or 0.0017 (in a pair, which reads half of B per CTA,
//   0.0014) for each column of products, or its bytes at the 18.5 MB/us that all SMs together read from L2, whichever is most;
//   a tile's epilogue takes 0.005 a column, beside the next tile's products if there is one, and a next tile 0.5 besides (0.2 where
//   all tiles have the same rows of A; heads of 17 to 128 rows, 50,257 x 768 in tiles of 192 columns 25.2 to 31.4 us, of 128
//   23.5 to 28.7; 32,000 x 1,024 in tiles of 256 21.2, of 128 19.5);
//   a launch takes 2.8, that of pairs 4.5 (they wait for each other at both ends).
// So pairs win where rounds of large tiles bound the time (2,048 x 6,144 x 2,048: 37.0 us, single CTAs 42.8), and single CTAs
// below (2,048 x 1,536 x 512: 6.9 us, pairs 8.0).
inline Cut choose_cut(int M, int N, int K, bool out_bf16) {
    Cut best = {1, 64, 1};
    double least = 1e30;
    const int num_kb = ceil_div(K, BLOCK_K), grain = out_bf16 ? 64 : 32;
    for (int cg = 1; cg <= (M > TILE_M ? 2 : 1); ++cg) {
        for (int bn = grain; bn <= MAX_BN; bn = bn < 64 ? 64 : bn + 64) {
            if (bn > grain && bn >= 2 * N) break;
            const long long tiles = (long long)ceil_div(M, cg * TILE_M) * ceil_div(N, bn);
            const long long places = SMS / cg, rounds = (tiles + places - 1) / places;
            const int b_bytes = bn / cg * BLOCK_K * 2, block_bytes = box_rows(M) * BLOCK_K * 2 + b_bytes;
            const int sub = A_TILE_BYTES + b_bytes <= 24 * 1024 && num_kb > 1 ? 2 : 1;
            double block = sub == 2 ? 0.125 : 0.175;
            const double products = (cg == 2 ? 0.0014 : 0.0017) * bn, reads = (double)(tiles < places ? tiles : places) * cg * block_bytes / 18.5e6;
            if (products > block) block = products;
            if (reads > block) block = reads;
            const double tile = num_kb * block, epilogue = 0.005 * bn;
            const double t = (cg == 2 ? 4.5 : 2.8) + (double)(rounds - 1) * ((M <= TILE_M ? 0.2 : 0.5) + (tile > epilogue ? tile : epilogue)) + tile + epilogue;
            if (t < least) { least = t; best = Cut{cg, bn, sub}; }
        }
    }
    return best;
}

// Rows and columns of A, rows of B and columns of D in memory, where they are not those of one product.
struct Extent {
    int a_rows, a_cols, b_rows;
    long long tiles;                 // the most there can be
};

template <int CG, int SUB, int MODE, bool EXACT = false>
int launch(const void* a, const void* b, GemmArgs g, cudaStream_t s, const Extent* extent = nullptr) {
    const bool glu = MODE == EXPERTS && g.form == 1;
    if (MODE == PLAIN) g.ld_out = g.N;
    g.a_rows = MODE == EXPERTS ? TILE_M : box_rows(g.M);
    CUtensorMap map_a, map_b, map_out = {};
    int rc = tensor_map(a, MODE == PLAIN ? g.M : extent->a_rows, MODE == PLAIN ? g.K : extent->a_cols, g.a_rows, &map_a);
    if (rc != MG_OK) return rc;
    if (MODE == HEADS_IN) rc = tensor_map(b, extent->b_rows, g.N, BLOCK_K, &map_b);
    else rc = tensor_map(b, MODE == PLAIN ? g.N : extent->b_rows, g.K, glu ? g.bn / 2 : g.bn / CG, &map_b);
    if (rc != MG_OK) return rc;
    if (g.boxes && (rc = tensor_map_store(g.out, g.M, g.ld_out, 32, !g.out_bf16, &map_out)) != MG_OK) return rc;
    const int stage_bytes = SUB * (A_TILE_BYTES + g.bn / CG * BLOCK_K * 2);
    const int num_kb = ceil_div(g.K, SUB * BLOCK_K);
    const long long tiles = MODE == PLAIN ? (long long)ceil_div(g.M, CG * TILE_M) * ceil_div(g.N, g.bn) : extent->tiles;
    const size_t fixed = EPI_WARPS * BOXES * BOX_BYTES + sizeof(Control) + 1024 + (MODE == EXPERTS ? 2 * 4 * (MAX_EXPERTS + 1) + 64 : 64);
    constexpr size_t most = 227 * 1024;
    if (g.stages == 0) g.stages = (int)((most - fixed) / stage_bytes);
    if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
    if (tiles <= SMS / CG && g.stages > num_kb) g.stages = num_kb;
    const size_t smem = (size_t)g.stages * stage_bytes + EPI_WARPS * BOXES * BOX_BYTES + sizeof(Control) + 1024;
    constexpr size_t most_dynamic = most - (MODE == EXPERTS ? 2 * 4 * (MAX_EXPERTS + 1) + 64 : 64);
    const cudaError_t e = mg_raise_shared(gemm_tc_kernel<CG, SUB, MODE, EXACT>, most_dynamic);
    if (e != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "linear: cannot raise shared memory: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CG * (tiles < SMS / CG ? tiles : SMS / CG)));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (CG > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = CG;
        attr[n_attr].val.clusterDim.y = attr[n_attr].val.clusterDim.z = 1;
        ++n_attr;
    }
    if (mg_dependent_launch_enabled()) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, gemm_tc_kernel<CG, SUB, MODE, EXACT>, map_a, map_b, map_out, g);
    if (le != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "gemm_tc: %s", cudaGetErrorString(le));
    MG_CHECK_LAUNCH("gemm_tc");
    return MG_OK;
}

}  // namespace

// How mg_linear_tc cuts a product: CTAs a tile (1 or 2), columns a tile, k blocks a stage (1 or 2).
MG_API void mg_linear_tc_cut(int M, int N, int K, int out_bf16, int* cg, int* bn, int* sub) {
    const Cut cut = choose_cut(M, N, K, out_bf16 != 0);
    *cg = cut.cg; *bn = cut.bn; *sub = cut.sub;
}

// x: [M, K] bf16, w: [N, K] bf16 (both row-major).  Epilogues as mg_linear_simt.  `status` is a
// device int that receives a non-zero code if a wait inside the kernel ran out.
// Returns MG_ERR_UNSUPPORTED (and launches nothing) for sizes or alignments TMA cannot take:
// K not a multiple of 8, pointers not 16-byte aligned.
MG_API int mg_linear_tc(const void* x, const void* w, const float* bias, void* out, float* residual, int M,
                        int N, int K, int epilogue, int out_bf16, void* k_pages, void* v_pages, const int* slots,
                        int q_width, int n_kv_head, int head_dim, int page_tokens, int num_pages, int* status,
                        void* stream) {
    if (M == 0) return MG_OK;
    MG_REQUIRE(M > 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    MG_REQUIRE(epilogue == EPI_RESIDUAL ? residual != nullptr : out != nullptr, "linear: missing output");
    MG_REQUIRE(status != nullptr, "linear: missing status word");
    if (K % 8 != 0 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15))
        return mg_set_error(MG_ERR_UNSUPPORTED, "linear: tensor-core path needs K %% 8 == 0 and 16-byte aligned operands");
    GemmArgs g = {};
    if (k_pages != nullptr) {
        MG_REQUIRE(v_pages && slots && out_bf16 && epilogue == EPI_STORE, "linear: the key/value copy wants a bfloat16 store");
        MG_REQUIRE(head_dim > 0 && head_dim % 8 == 0 && q_width % 8 == 0 && n_kv_head > 0 && page_tokens > 0 &&
                       q_width + 2 * n_kv_head * head_dim == N,
                   "linear: key/value copy with q_width=%d n_kv_head=%d head_dim=%d N=%d", q_width, n_kv_head, head_dim, N);
        g.sink = KvSink{(bf16*)k_pages, (bf16*)v_pages, slots, q_width, n_kv_head, head_dim, page_tokens, num_pages};
    }
    g.bias = bias;
    g.epilogue = epilogue;
    g.out_bf16 = epilogue == EPI_RESIDUAL ? 0 : out_bf16;
    g.out = epilogue == EPI_RESIDUAL ? (void*)residual : out;
    g.M = M; g.N = N; g.K = K;
    g.boxes = N % (g.out_bf16 ? 8 : 4) == 0 && ((uintptr_t)g.out & 15) == 0;
    g.status = status;
    const Cut cut = choose_cut(M, N, K, g.out_bf16 != 0);
    MG_REQUIRE((long long)ceil_div(M, cut.cg * TILE_M) * ceil_div(N, cut.bn) < (1ll << 30), "linear: too many tiles");
    g.bn = cut.bn;
    cudaStream_t s = (cudaStream_t)stream;
    if (cut.cg == 2) return cut.sub == 2 ? launch<2, 2, PLAIN>(x, w, g, s) : launch<2, 1, PLAIN>(x, w, g, s);
    if (M <= TILE_M) return cut.sub == 2 ? launch<1, 2, PLAIN, true>(x, w, g, s) : launch<1, 1, PLAIN, true>(x, w, g, s);
    return cut.sub == 2 ? launch<1, 2, PLAIN>(x, w, g, s) : launch<1, 1, PLAIN>(x, w, g, s);
}

// One small product per head, bfloat16: out[m, o_off + h * o_head + n] = sum_k x[m, x_off + h * x_head + k] * w[h * N + n, k] for
// n < N, k < K, or, with rows_are_inputs, w[h * K + k, n] (read as it lies: tcgen05 takes either order of B from shared memory).
// x: rows of x_ld elements, out: rows of out_ld.  Returns MG_ERR_UNSUPPORTED (and launches nothing) unless K and N
// are multiples of 64 and the rows' parts lie on 16-byte boundaries (TMA).
MG_API int mg_head_linear_tc(const void* x, int x_ld, int x_off, int x_head, const void* w, int rows_are_inputs, void* out, int out_ld, int out_off,
                             int out_head, int M, int heads, int K, int N, int* status, void* stream) {
    if (M == 0) return MG_OK;
    MG_REQUIRE(M > 0 && heads > 0 && K > 0 && N > 0 && status != nullptr, "head_linear: bad sizes");
    MG_REQUIRE(x_off >= 0 && x_head >= K && x_off + (long long)(heads - 1) * x_head + K <= x_ld && out_off >= 0 && out_head >= N &&
                   out_off + (long long)(heads - 1) * out_head + N <= out_ld,
               "head_linear: heads outside the rows");
    if (K % 64 != 0 || N % 64 != 0 || x_ld % 8 != 0 || x_off % 8 != 0 || x_head % 8 != 0 || out_ld % 8 != 0 || out_off % 8 != 0 ||
        out_head % 8 != 0 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) || (long long)heads * (N > K ? N : K) > (1 << 30))
        return mg_set_error(MG_ERR_UNSUPPORTED, "head_linear: no tensor-core tiles for %d x %d", K, N);
    GemmArgs g = {};
    g.out = out; g.out_bf16 = 1; g.boxes = 1; g.epilogue = EPI_STORE;
    g.M = M; g.N = N; g.K = K; g.ld_out = out_ld; g.status = status;
    g.heads = heads; g.a_off = x_off; g.a_head = x_head; g.o_off = out_off; g.o_head = out_head;
    g.bn = N % 128 == 0 ? 128 : 64;
    const Extent extent = {M, x_ld, heads * (rows_are_inputs ? K : N), (long long)ceil_div(M, TILE_M) * heads * (N / g.bn)};
    MG_REQUIRE(extent.tiles < (1ll << 30), "head_linear: too many tiles");
    return rows_are_inputs ? launch<1, 1, HEADS_IN>(x, w, g, (cudaStream_t)stream, &extent)
                           : launch<1, 1, HEADS>(x, w, g, (cudaStream_t)stream, &extent);
}

// The products of mg_moe_gemm on the tensor cores, rows by slot: x [n_entries, K] bfloat16 (a token's row for each of its
// entries, gathered: mg_moe_gather), w [n_experts, N (2 N for form 1), K], out [n_entries, N] bfloat16 (forms 1 and 2) or 32-bit
// (form 0).  Returns MG_ERR_UNSUPPORTED (and launches nothing) for sizes or alignments that TMA or the kernel do not take.
MG_API int mg_moe_gemm_tc(const void* x, const void* w, const int* offsets, const int* slot_entry, const float* scale, void* out,
                          int n_entries, int n_experts, int N, int K, int form, int act, float limit, int* status, void* stream) {
    if (n_entries == 0) return MG_OK;
    MG_REQUIRE(n_entries > 0 && n_experts > 0 && N > 0 && K > 0 && form >= 0 && form <= 2 && status != nullptr, "moe gemm: bad sizes");
    const long long b_rows = (long long)n_experts * (form == 1 ? 2 : 1) * N;
    if (K % 8 != 0 || n_experts > MAX_EXPERTS || b_rows > (1 << 30) || (((uintptr_t)x | (uintptr_t)w) & 15))
        return mg_set_error(MG_ERR_UNSUPPORTED, "moe gemm: no tensor-core tiles for %d experts of %d x %d", n_experts, N, K);
    GemmArgs g = {};
    g.out = out; g.out_bf16 = form != 0; g.epilogue = EPI_STORE;
    g.M = n_entries; g.N = N; g.K = K; g.ld_out = N; g.status = status;
    g.boxes = N % (g.out_bf16 ? 8 : 4) == 0 && ((uintptr_t)out & 15) == 0;
    g.offsets = offsets; g.slot_entry = slot_entry; g.scale = scale; g.n_experts = n_experts; g.form = form; g.act = act; g.limit = limit;
    // 128 results a tile: at 6,144 slots x 1,024 x 1,024 448 tiles, three rounds
    g.bn = form == 1 ? 256 : 128;
    const int bn_out = form == 1 ? g.bn / 2 : g.bn;
    const Extent extent = {n_entries, K, (int)b_rows, ((long long)n_entries / TILE_M + n_experts) * ceil_div(N, bn_out)};
    MG_REQUIRE(extent.tiles < (1ll << 30), "moe gemm: too many tiles");
    return launch<1, 1, EXPERTS>(x, w, g, (cudaStream_t)stream, &extent);
}
