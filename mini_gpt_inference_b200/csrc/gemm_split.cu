// out[m, n] = sum_k a[m, k] * w[n, k] (+ bias[n]) with an epilogue, in 32 bits, on the tensor cores.
//
// A 32-bit number down to 2^-109 is the sum of three bfloat16 numbers, exactly: its 24 bits are rounded to 8 three times, x = h + m + l
// with |m| <= 2^-8 |h| and |l| <= 2^-17 |h|.  Products of bfloat16 numbers are exact in the tensor cores, so a product of two such
// sums is nine of theirs; l l', below 2^-33 of it, is left out.  What rounds is the accumulator: it drops what lies below its last place
// at every addition of 16 products, where an ordinary addition rounds, so sums of one sign come out too small.  So K is cut into
// slices of 64, and of a slice's h h' only two such additions follow each other: its halves have an accumulator each.  The other
// seven products, which are 2^8 and more below, have two of their own (see ACCUMULATORS).  The four meet, and a slice's sum is
// added to those before it, in ordinary rounded additions; a single product is rounded once.
// Errors against 64 bits, of the result's size and in 1e-8, chains of fused multiply-adds and this: numbers of both signs, 64 terms
// 14.4 and 5.1, 512 terms 15.5 and 7.6, 2,048 terms 17.9 and 11.8, 6,400 terms 23.2 and 19.1; of one sign 12.2 and 5.5, 6.6 and 6.4,
// 9.2 and 9.8, 13.4 and 13.9 (with all four additions of h h' in one accumulator 9.0, 9.3, 11.9 and 15.4).
//
// Every element is summed in that one order whatever the number of rows and the kernel or tile that it falls in, so a token's
// result does not depend on what else is in the batch (mma.sync and tcgen05.mma give the same bits; so do the two orders of the operands).
//
// Rows (of a or w) that hold an infinity, no number, a number of 2^126 or more or one whose last piece falls below bfloat16's least number
// (possible below 2^-109) do not split so.  And sums of pieces could pass the end of the range where the sum itself does not, or run into
// infinities of both signs: a row of a and one of w whose largest numbers make that possible over K terms.  Results
// that meet either are summed by fused multiply-adds instead, slices of 64 from 0 and their sums one after the other, again whatever
// is beside them: a CTA that has such results walks their operands a second time.
//
// Two kernels:
//   gemm_split_kernel   tiles of 128 rows x 64 columns by tcgen05.  Sixteen warps read both operands of a slice from global memory
//                       (a slice ahead, in registers), split them, and lay the pieces into shared memory in the 128-byte swizzle,
//                       the three of w's rows one behind the other.  A thread of the 17th warp issues the 18 products of a slice;
//                       the sixteen then take the sums out of TMEM and add them to the totals in their registers, beside the
//                       next slice's products.
//   gemm_split_few_kernel   up to 16 rows: a CTA takes 16 rows of w, each of its eight warps every eighth slice, operands by cp.async in
//                       a ring of the warp's own (the first round of w before the wait for the kernel in front); the fragments
//                       of mma.sync are split as they are read.  Bound by reading w and by the latency of a launch and a slice.
// 2,048 rows, FMA tiles and these: 1,536 x 512 102 and 43 us, 2,048 x 512 124 and 56, 512 x 2,048 143 and 48; 17 rows (FMA tiles of 64 rows)
// 25.5 and 13.9, 25.8 and 14.0, 93.9 and 40; 8 rows (FMA and mma.sync) 3.3 and 3.5, 4.0 and 3.9, 7.6 and 7.1, 50,304 x 512 32.6 and 32.6; 16 rows
// 4.4 and 4.0, 4.9 and 4.4, 10.7 and 9.7, 50.0 and 49.6.  (1,536 x 512 at 8 rows is the price of the same bits in both kernels.)
#include "blackwell.cuh"

#define EPI_STORE 0      // out = acc + bias
#define EPI_GELU 1       // out = gelu_tanh(acc + bias)
#define EPI_RESIDUAL 2   // residual += acc + bias (in place)
#define EPI_RELU_SQ 3    // out = max(acc + bias, 0)^2

namespace {

constexpr int SLICE = 64;            // terms summed by the tensor cores in one go: a 128-byte row of bfloat16
constexpr int PIECES = 3;
static_assert(SLICE == 64, "four steps of 16");

// The accumulators of a slice: h h' of its second half, those of its first, and for each of its four steps of 16 terms, in this order,
// h m', m h', m m', l h' in the third and h l', m l', l m' in the fourth.
constexpr int ACCUMULATORS = 4;
__device__ __forceinline__ constexpr int accumulator(int q, int v) { return 1 + (q == 0 ? v : q == 1 ? (v == 2 ? 2 : 1) : v + 1); }
__device__ __forceinline__ float slice_sum(float second, float first, float rest, float below) { return first + (second + (rest + below)); }

// The pieces of two neighbouring numbers, as pairs of bfloat16 (x in the low half).  The third's upper half is all of it, as long
// as it does not fall below bfloat16's least number: what is cut off then shows in the low half of `lost`.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t (&p)[PIECES], uint32_t& lost) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    p[0] = *reinterpret_cast<const uint32_t*>(&h);
    x -= __uint_as_float(p[0] << 16);
    y -= __uint_as_float(p[0] & 0xffff0000u);
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    p[1] = *reinterpret_cast<const uint32_t*>(&m);
    x -= __uint_as_float(p[1] << 16);
    y -= __uint_as_float(p[1] & 0xffff0000u);
    lost |= __float_as_uint(x) | __float_as_uint(y);
    p[2] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

// The bits of first pieces without their signs order as the numbers do, with infinities and no numbers on top: the largest of a
// row's, for each half of the pairs.
__device__ __forceinline__ uint32_t larger(uint32_t most, uint32_t h) { return __vmaxu2(most, h & 0x7fff7fffu); }
__device__ __forceinline__ uint32_t larger(uint32_t most, uint32_t h, uint32_t i) { return __vimax3_u16x2(most, h & 0x7fff7fffu, i & 0x7fff7fffu); }
__device__ __forceinline__ uint32_t most_of(uint32_t most, uint32_t lost) { return (lost & 0xffffu) != 0 ? 0x7fff7fffu : most; }
// What a row counts for: the exponent e (as stored) of its largest number's first piece, so that all are below 2^(e - 126); UNSPLIT
// if it does not split.
constexpr uint32_t UNSPLIT = 512;
__device__ __forceinline__ uint32_t reach(uint32_t most) {
    const uint32_t of_both = max(most & 0xffffu, most >> 16);
    return of_both >= 0x7e80u ? UNSPLIT : of_both >> 7;         // 2^126
}
__device__ __forceinline__ uint32_t eight_lanes_max(uint32_t v) {
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// K products of a row with e and one with f stay below K 2^(e + f - 252), pieces' sums below 1.02 of that.  Up to this e + f
// they stay below 2^127: no sum of theirs ends, or passes, beyond the range.
inline int highest_reach(int K) {
    int log2_k = 0;
    while ((1ll << log2_k) < K) ++log2_k;
    return 378 - log2_k;
}

__device__ __forceinline__ float dot4(float4 x, float4 y, float sum) {
    return fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, sum))));
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool there) {
    const uint32_t bytes = there ? 16u : 0u;                 // (0: sixteen zero bytes are written)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float activate(float v, int epilogue) {
    return epilogue == EPI_GELU ? gelu_tanh(v) : epilogue == EPI_RELU_SQ ? relu_sq(v) : v;
}

struct SplitArgs {
    const float* a;
    const float* w;
    const float* bias;
    float* out;                      // the residual stream for EPI_RESIDUAL
    int M, N, K, epilogue;
    int wide;                        // rows of the output lie on 16-byte boundaries
    int highest;                     // reaches of two rows that add up to more: by fused multiply-adds
    int* status;
};

// What becomes of a finished sum of column n.
__device__ __forceinline__ void finish(const SplitArgs& g, float sum, int n, float* dst) {
    const float y = activate(sum + (g.bias != nullptr ? g.bias[n] : 0.f), g.epilogue);
    if (g.epilogue == EPI_RESIDUAL) *dst += y;
    else *dst = y;
}

// ---- tiles -----------------------------------------------------------------------------------------------
// A slice takes 1.45 us, 1.1 with few rows: the operands of the next one come from L2 (48 KB) while a slice is split, and the splitting
// itself is 24 numbers a thread.  Tiles of 32 columns take the same time a slice (512 x 2,048, 128 rows: 48 and 46 us).  With a worker
// that issued the products as well, a slice took 2.05 us.  Eight products and four accumulators, in the place of six and three, cost
// 2 to 3 % (42 -> 43, 47 -> 48 us), and 4 to 5 % among a model's other kernels (43.2 -> 45.1, 60.9 -> 63.3, 49.9 -> 52.4 us): what a worker
// does for a slice counts, and how long the products take (in 30 instructions of 64 columns 9 %).  The sums are taken out four columns
// at a time: eight want more registers than there are (52 us for 48).
constexpr int TILE_M = 128, BN = 64;
constexpr int WORKERS = 512;         // threads that split and add up
constexpr int THREADS = WORKERS + 32;
constexpr int ROW_BYTES = SLICE * 2;
constexpr int SMS = 148;
constexpr int OUT_BYTES = 32 * 64;   // a warp's place for 32 rows of 16 results on their way to memory
constexpr int FLAGS = 3;             // sets of rows' marks: a set is written again two tiles' barriers after it was read

constexpr int STAGE = PIECES * (TILE_M + BN) * ROW_BYTES;    // the pieces of a slice: a's three planes, then w's
constexpr int DYNAMIC_BYTES = 1024 + 2 * STAGE + (WORKERS / 32) * OUT_BYTES;

constexpr int CW = BN / 4;           // results a worker has
constexpr int ODD_WORDS = 64;        // marks of tiles with results for the multiply-adds: a CTA's tiles from the 2,048th on share the last one

__device__ __forceinline__ void tmem_load_4(uint32_t taddr, uint32_t (&r)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}

// The results that the pieces do not serve, of the tiles that are marked, by fused multiply-adds.  All threads of the CTA, behind its last tile.
// The tile's rows, a's and then w's, pass through two buffers in turn, 32 columns of each and 4 words of space (16-byte reads of 8 rows
// meet no bank twice), and are looked over again for what they count for.  512 x 2,048, 128 rows that hold what is no number: 246 us, else 46.
constexpr int FMA_COLS = SLICE / 2, FMA_LINE = FMA_COLS + 4, FMA_ROWS = TILE_M + BN, FMA_BUFFER = FMA_ROWS * FMA_LINE;
static_assert(2 * FMA_BUFFER * (int)sizeof(float) <= 2 * STAGE, "the buffers take the stages' place");

__device__ __noinline__ void fma_tiles(const SplitArgs& g, float* buffers, uint16_t* reaches, const uint32_t* odd_tiles, int m_tiles, int my_tiles) {
    const int tid = threadIdx.x, tr = (tid >> 4) & 31, tc = tid & 15, chunks = 2 * ((g.K + SLICE - 1) / SLICE);
    for (int t = 0; t < my_tiles; ++t) {
        const int mark = min(t, 32 * ODD_WORDS - 1);
        if (((odd_tiles[mark >> 5] >> (mark & 31)) & 1u) == 0) continue;
        const int tile = (int)blockIdx.x + t * (int)gridDim.x, m0 = (tile % m_tiles) * TILE_M, n0 = (tile / m_tiles) * BN;
        auto ask = [&](int c) {
            if (c < chunks && tid < WORKERS)
#pragma unroll
                for (int u = 0; u < FMA_ROWS * (FMA_COLS / 4) / WORKERS; ++u) {
                    const int at = tid + u * WORKERS, row = at / (FMA_COLS / 4), col = (at % (FMA_COLS / 4)) * 4, k = c * FMA_COLS + col;
                    const bool of_a = row < TILE_M, there = k < g.K && (of_a ? m0 + row < g.M : n0 + row - TILE_M < g.N);
                    const float* from = of_a ? g.a + (size_t)(m0 + row) * g.K + k : g.w + (size_t)(n0 + row - TILE_M) * g.K + k;
                    cp_async16(buffers + (c & 1) * FMA_BUFFER + row * FMA_LINE + col, there ? from : g.a, there);
                }
            cp_async_commit();
        };
        float total[4][4], acc[4][4];                            // of rows tr + 32 i and columns tc + 16 j
        uint32_t most = 0, lost = 0;                             // of row tid
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) total[i][j] = acc[i][j] = 0.f;
        ask(0);
        for (int c = 0; c < chunks; ++c) {
            ask(c + 1);
            cp_async_wait<1>();
            __syncthreads();                                     // the chunk is there for all
            const float* of = buffers + (c & 1) * FMA_BUFFER;
            if (tid < FMA_ROWS)
#pragma unroll 2
                for (int k = 0; k < FMA_COLS; k += 2) {
                    const float2 x = *reinterpret_cast<const float2*>(of + tid * FMA_LINE + k);
                    uint32_t p[PIECES];
                    split_pair(x.x, x.y, p, lost);
                    most = larger(most, p[0]);
                }
            if (tid < WORKERS)
#pragma unroll 2
                for (int k = 0; k < FMA_COLS; k += 4) {
                    float4 x[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(of + (tr + 32 * i) * FMA_LINE + k);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 y = *reinterpret_cast<const float4*>(of + (TILE_M + tc + 16 * j) * FMA_LINE + k);
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[i][j] = dot4(x[i], y, acc[i][j]);
                    }
                }
            if ((c & 1) != 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        total[i][j] += acc[i][j];
                        acc[i][j] = 0.f;
                    }
            }
            __syncthreads();                                     // its buffer takes the chunk after the next
        }
        if (tid < FMA_ROWS) reaches[tid] = (uint16_t)reach(most_of(most, lost));
        __syncthreads();
        if (tid < WORKERS)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int m = m0 + tr + 32 * i, room = g.highest - reaches[tr + 32 * i];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int n = n0 + tc + 16 * j;
                    if (m < g.M && n < g.N && reaches[TILE_M + tc + 16 * j] > room) finish(g, total[i][j], n, g.out + (size_t)m * g.N + n);
                }
            }
        __syncthreads();                                         // (the next tile's rows)
    }
}

struct __align__(16) SplitControl {
    uint64_t full[2], done[2];       // the pieces of a step are there; its products are done
    uint32_t tmem_base;
    uint32_t failed, odd;            // no more waiting; a tile is marked
};

__global__ void __launch_bounds__(THREADS, 1) gemm_split_kernel(const __grid_constant__ SplitArgs g) {
    constexpr int A_PLANE = TILE_M * ROW_BYTES, W_PLANE = BN * ROW_BYTES;
    constexpr int AC = TILE_M * 8 / WORKERS, WC = BN * 8 / WORKERS;      // 8-number pieces of rows a thread splits
    constexpr int SUMS = ACCUMULATORS * BN;  // columns of TMEM for a slice's sums
    extern __shared__ uint8_t split_smem[];
    __shared__ SplitControl ctl;
    __shared__ uint32_t odd_tiles[ODD_WORDS];
    __shared__ __align__(16) uint16_t reach_a[FLAGS][TILE_M], reach_w[FLAGS][BN];
    uint8_t* smem = (uint8_t*)(((uintptr_t)split_smem + 1023) & ~(uintptr_t)1023);       // (the swizzle wants 1,024-byte boundaries)
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int m_tiles = (g.M + TILE_M - 1) / TILE_M, n_tiles = (g.N + BN - 1) / BN, tiles = m_tiles * n_tiles;
    const int slices = (g.K + SLICE - 1) / SLICE;
    const int my_tiles = ((int)blockIdx.x < tiles) ? (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const long long steps = (long long)my_tiles * slices;

    if (tid < ODD_WORDS) odd_tiles[tid] = 0;
    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&ctl.full[i]), WORKERS / 32);
            mbar_init(smem_u32(&ctl.done[i]), 1);
        }
        ctl.failed = ctl.odd = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WORKERS / 32) tmem_alloc(smem_u32(&ctl.tmem_base), 2 * SUMS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl.tmem_base;
    pdl_trigger();

    if (warp == WORKERS / 32) {
        // ---- the products of a step, once all warps have laid its pieces (which each does behind its last look at the sums
        // and the stage of the step before the last: neither needs a barrier of its own) ----
        if (elect_one()) {
            const uint64_t desc0 = smem_desc_sw128(smem_u32(smem));
            bool there = true;
            for (long long i = 0; i < steps && there; ++i) {
                const int half = (int)(i & 1);
                there = mbar_wait(smem_u32(&ctl.full[half]), (uint32_t)(i >> 1) & 1u);
                if (!there) break;
                tc_fence_after();
                const uint64_t desc_a = desc0 + (uint64_t)(half * (STAGE >> 4)), desc_w = desc_a + (uint64_t)((PIECES * A_PLANE) >> 4);
                const uint32_t d = tmem_base + half * SUMS;
                // columns 16 k .. of a's piece q, of w's piece v and the n - 1 behind it, for the accumulators from `sums` on
                auto products = [&](int k, int q, int v, int n, int sums, bool add) {
                    umma_bf16(d + sums * BN, desc_a + (uint64_t)((q * A_PLANE + k * 32) >> 4), desc_w + (uint64_t)((v * W_PLANE + k * 32) >> 4),
                              instr_desc_bf16(TILE_M, n * BN), add ? 1u : 0u);
                };
#pragma unroll
                for (int k = 0; k < SLICE / 16; ++k) {
                    if (k < SLICE / 32) {
                        products(k, 0, 0, 3, 1, k != 0);
                    } else {
                        products(k, 0, 0, 1, 0, k != SLICE / 32);
                        products(k, 0, 1, 2, 2, true);
                    }
                    products(k, 1, 0, 1, 2, true);
                    products(k, 1, 1, 2, 2, true);
                    products(k, 2, 0, 2, 2, true);
                }
                umma_commit(smem_u32(&ctl.done[half]));
            }
            if (!there) {
                atomicExch(g.status, 82);
                ctl.failed = 1;
            }
        }
    } else {
        // ---- loads, splitting, and the slices' sums ----
        const int col8 = (tid & 7) * 8, row8 = tid >> 3;         // this thread's columns of a slice, and its rows row8 + 64 i
        float4 av[AC][2], wv[WC][2];
        uint32_t most_a[AC], most_w[WC], lost_a[AC], lost_w[WC];
        auto fetch = [&](float4 (&v)[2], const float* p, int row, int rows, int k) {
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float* at = p + (size_t)row * g.K + k;
            v[0] = row < rows && k < g.K ? *reinterpret_cast<const float4*>(at) : zero;
            v[1] = row < rows && k + 4 < g.K ? *reinterpret_cast<const float4*>(at + 4) : zero;
        };
        auto fetch_a = [&](float4 (&v)[AC][2], int m0, int slice) {
#pragma unroll
            for (int i = 0; i < AC; ++i) fetch(v[i], g.a, m0 + row8 + 64 * i, g.M, slice * SLICE + col8);
        };
        auto fetch_w = [&](float4 (&v)[WC][2], int n0, int slice) {
#pragma unroll
            for (int i = 0; i < WC; ++i) fetch(v[i], g.w, n0 + row8 + 64 * i, g.N, slice * SLICE + col8);
        };
        auto lay = [&](const float4 (&v)[2], uint8_t* base, int plane, int row, uint32_t& most, uint32_t& lost) {
            uint32_t p[4][PIECES];
            split_pair(v[0].x, v[0].y, p[0], lost);
            split_pair(v[0].z, v[0].w, p[1], lost);
            split_pair(v[1].x, v[1].y, p[2], lost);
            split_pair(v[1].z, v[1].w, p[3], lost);
            most = larger(larger(most, p[0][0], p[1][0]), p[2][0], p[3][0]);
            uint8_t* at = base + row * ROW_BYTES + (((tid & 7) ^ (row & 7)) << 4);
#pragma unroll
            for (int q = 0; q < PIECES; ++q) *reinterpret_cast<uint4*>(at + q * plane) = make_uint4(p[0][q], p[1][q], p[2][q], p[3][q]);
        };
        const int quarter = warp & 3, group = warp >> 2;         // this thread's row of TMEM is 32 quarter + lane, its columns CW group + 0 .. CW
        const uint32_t sums_at = tmem_base + ((uint32_t)(quarter * 32) << 16) + group * CW;
        float total[CW];
#pragma unroll
        for (int j = 0; j < CW; ++j) total[j] = 0.f;
        bool ok = true;

        // Takes step i's sums; behind a tile's last slice the tile's results go to memory.  A warp whose wait ran out (ok) takes and
        // gives nothing any more, but goes on to every barrier: the others may have got their wait and stand there.
        auto add_up = [&](long long i, int slice, int tile, int flags) {
            const int half = (int)(i & 1);
            if (ok) ok = warp_wait(smem_u32(&ctl.done[half]), (uint32_t)(i >> 1) & 1u);
            if (ok) {
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < CW; c += 4) {
                    uint32_t r[ACCUMULATORS][4];
#pragma unroll
                    for (int q = 0; q < ACCUMULATORS; ++q) tmem_load_4(sums_at + half * SUMS + q * BN + c, r[q]);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        total[c + j] += slice_sum(__uint_as_float(r[0][j]), __uint_as_float(r[1][j]), __uint_as_float(r[2][j]), __uint_as_float(r[3][j]));
                }
                tc_fence_before();
            }
            if (slice + 1 < slices) return;
            asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");            // all rows of the tile are marked
            if (!ok) return;
            const int row0 = (tile % m_tiles) * TILE_M + quarter * 32, col0 = (tile / m_tiles) * BN + group * CW;
            uint8_t* place = smem + 2 * STAGE + warp * OUT_BYTES;
            constexpr int HALF = 16, CHUNKS = HALF / 4, ROWS = 32 / CHUNKS;   // columns at a time, 16-byte chunks of them, rows an access
#pragma unroll
            for (int h = 0; h < CW; h += HALF) {
                __syncwarp();
                if (row0 < g.M) {
#pragma unroll
                    for (int c = 0; c < CHUNKS; ++c)
                        *reinterpret_cast<float4*>(place + lane * 64 + ((c ^ ((lane >> 1) & (CHUNKS - 1))) << 4)) =
                            make_float4(total[h + 4 * c], total[h + 4 * c + 1], total[h + 4 * c + 2], total[h + 4 * c + 3]);
                }
                __syncwarp();
                const int c = lane % CHUNKS, n = col0 + h + 4 * c;
                for (int r = lane / CHUNKS; r < 32; r += ROWS) {
                    const int m = row0 + r;
                    if (m >= g.M || n >= g.N) break;
                    const float4 sums = *reinterpret_cast<const float4*>(place + r * 64 + ((c ^ ((r >> 1) & (CHUNKS - 1))) << 4));
                    float v[4] = {sums.x, sums.y, sums.z, sums.w};
                    const ushort4 of_w = *reinterpret_cast<const ushort4*>(&reach_w[flags][group * CW + h + 4 * c]);
                    const int room = g.highest - reach_a[flags][quarter * 32 + r];
                    const bool odd[4] = {of_w.x > room, of_w.y > room, of_w.z > room, of_w.w > room};
                    const bool any = odd[0] || odd[1] || odd[2] || odd[3];
                    if (any) {                                   // left for fma_tiles
                        const int at = min((tile - (int)blockIdx.x) / (int)gridDim.x, 32 * ODD_WORDS - 1);
                        ctl.odd = 1;
                        atomicOr(&odd_tiles[at >> 5], 1u << (at & 31));
                    }
                    float* dst = g.out + (size_t)m * g.N + n;
                    if (g.wide && !any) {                        // (N is a multiple of 4: all four are there)
                        if (g.bias != nullptr) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) v[j] += g.bias[n + j];
                        }
                        float4 y = make_float4(activate(v[0], g.epilogue), activate(v[1], g.epilogue), activate(v[2], g.epilogue), activate(v[3], g.epilogue));
                        if (g.epilogue == EPI_RESIDUAL) {
                            const float4 old = *reinterpret_cast<const float4*>(dst);
                            y = make_float4(old.x + y.x, old.y + y.y, old.z + y.z, old.w + y.w);
                        }
                        *reinterpret_cast<float4*>(dst) = y;
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            if (n + j < g.N && !odd[j]) finish(g, v[j], n + j, dst + j);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < CW; ++j) total[j] = 0.f;
        };

        int tile = blockIdx.x, slice = 0, flags = 0;             // of the step that is split
        int m0 = (tile % m_tiles) * TILE_M, n0 = (tile / m_tiles) * BN;
        int was_tile = 0, was_slice = 0, was_flags = 0;          // of the step in front of it
        if (steps > 0) fetch_w(wv, n0, 0);                       // the weights do not come from the kernel in front
        pdl_wait();
        if (steps > 0) fetch_a(av, m0, 0);
#pragma unroll
        for (int i = 0; i < AC; ++i) most_a[i] = lost_a[i] = 0;
#pragma unroll
        for (int i = 0; i < WC; ++i) most_w[i] = lost_w[i] = 0;
        for (long long i = 0; i < steps; ++i) {
            uint8_t* stage = smem + (int)(i & 1) * STAGE;
            if (ok) {
                // (a row behind the last keeps what the place held: it gives results that nobody takes)
#pragma unroll
                for (int j = 0; j < AC; ++j)
                    if (m0 + row8 + 64 * j < g.M) lay(av[j], stage, A_PLANE, row8 + 64 * j, most_a[j], lost_a[j]);
#pragma unroll
                for (int j = 0; j < WC; ++j)
                    if (n0 + row8 + 64 * j < g.N) lay(wv[j], stage + PIECES * A_PLANE, W_PLANE, row8 + 64 * j, most_w[j], lost_w[j]);
                async_proxy_fence();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&ctl.full[(int)(i & 1)]));
            }
            const int this_tile = tile, this_slice = slice, this_flags = flags;
            if (++slice == slices) {                             // the tile's rows are known: eight lanes have each row
#pragma unroll
                for (int j = 0; j < AC; ++j) {
                    const uint32_t all = eight_lanes_max(reach(most_of(most_a[j], lost_a[j])));
                    if ((tid & 7) == 0) reach_a[flags][row8 + 64 * j] = (uint16_t)all;
                    most_a[j] = lost_a[j] = 0;
                }
#pragma unroll
                for (int j = 0; j < WC; ++j) {
                    const uint32_t all = eight_lanes_max(reach(most_of(most_w[j], lost_w[j])));
                    if ((tid & 7) == 0) reach_w[flags][row8 + 64 * j] = (uint16_t)all;
                    most_w[j] = lost_w[j] = 0;
                }
                slice = 0;
                tile += gridDim.x;
                m0 = (tile % m_tiles) * TILE_M;
                n0 = (tile / m_tiles) * BN;
                if (++flags == FLAGS) flags = 0;
            }
            if (i + 1 < steps && ok) {
                fetch_a(av, m0, slice);
                fetch_w(wv, n0, slice);
            }
            if (i > 0) add_up(i - 1, was_slice, was_tile, was_flags);
            was_tile = this_tile; was_slice = this_slice; was_flags = this_flags;
        }
        if (steps > 0) add_up(steps - 1, was_slice, was_tile, was_flags);
        if (!ok && lane == 0) {
            atomicExch(g.status, 81);
            ctl.failed = 1;
        }
    }
    __syncwarp();
    // a wait ran out: products that may still be under way get a moment to end
    if (*(volatile uint32_t*)&ctl.failed != 0 && lane == 0)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == WORKERS / 32) tmem_dealloc(tmem_base, 2 * SUMS);
    if (ctl.failed == 0 && ctl.odd != 0) fma_tiles(g, reinterpret_cast<float*>(smem), &reach_a[0][0], odd_tiles, m_tiles, my_tiles);
}

cudaError_t launch_tiles(const SplitArgs& g, cudaStream_t s) {
    const cudaError_t configured = mg_raise_shared(gemm_split_kernel, DYNAMIC_BYTES);
    if (configured != cudaSuccess) return configured;
    const long long tiles = (long long)ceil_div(g.M, TILE_M) * ceil_div(g.N, BN);
    return mg_launch(gemm_split_kernel, dim3((unsigned)(tiles < SMS ? tiles : SMS)), dim3(THREADS), DYNAMIC_BYTES, s, true, g);
}

// ---- a few rows ---------------------------------------------------------------------------------------------
constexpr int FEW_WARPS = 8, FEW_STAGES = 2, FEW_N = 16;    // rows of w per CTA: the m of m16n8k16
constexpr int LINE = SLICE + 8;                              // words between rows in shared memory: 8-byte reads of 4 rows meet no bank twice

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// MT rows of a: 8 or 16.
template <int MT>
__global__ void __launch_bounds__(32 * FEW_WARPS, MT == 8 ? 3 : 2) gemm_split_few_kernel(const SplitArgs g, int stages) {
    constexpr int NR = FEW_N, STAGE = (NR + MT) * LINE;      // words of a warp's stage: w's slice, then a's
    constexpr int TB = MT / 8;
    extern __shared__ __align__(16) float few_smem[];
    __shared__ uint32_t reach_w[NR], reach_a[MT];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* ring = few_smem + warp * stages * STAGE;
    float* parts = few_smem + FEW_WARPS * stages * STAGE;    // [2][warp][MT][NR]
    const int n0 = blockIdx.x * NR, M = g.M, N = g.N, K = g.K;
    const int slices = (K + SLICE - 1) / SLICE, rounds = (slices + FEW_WARPS - 1) / FEW_WARPS;

    auto ask_w = [&](int r) {
        float* dst = ring + (r & (stages - 1)) * STAGE;
        const int k0 = (r * FEW_WARPS + warp) * SLICE;
#pragma unroll
        for (int i = 0; i < NR / 2; ++i) {
            const int row = 2 * i + (lane >> 4), c = (lane & 15) * 4;
            const bool there = n0 + row < N && k0 + c < K;
            cp_async16(dst + row * LINE + c, there ? g.w + (size_t)(n0 + row) * K + k0 + c : g.w, there);
        }
    };
    auto ask_a = [&](int r) {
        float* dst = ring + (r & (stages - 1)) * STAGE + NR * LINE;
        const int k0 = (r * FEW_WARPS + warp) * SLICE;
#pragma unroll
        for (int i = 0; i < MT / 2; ++i) {
            const int row = 2 * i + (lane >> 4), c = (lane & 15) * 4;
            const bool there = row < M && k0 + c < K;
            cp_async16(dst + row * LINE + c, there ? g.a + (size_t)row * K + k0 + c : g.a, there);
        }
    };
    pdl_trigger();
    for (int r = 0; r < stages && r < rounds; ++r) ask_w(r);                // the weights depend on no kernel before
    if (tid < NR) reach_w[tid] = 0;
    if (tid >= 32 && tid < 32 + MT) reach_a[tid - 32] = 0;
    __syncthreads();
    pdl_wait();
    for (int r = 0; r < FEW_STAGES; ++r) {
        if (r < stages && r < rounds) ask_a(r);
        cp_async_commit();
    }
    const int gr = lane >> 2, t2 = (lane & 3) * 2;
    uint32_t mine_w[2] = {0, 0}, lost_w[2] = {0, 0}, mine_a[TB], lost_a[TB];
#pragma unroll
    for (int b = 0; b < TB; ++b) mine_a[b] = lost_a[b] = 0;
    float total = 0.f;                                                      // of row tid / NR, column n0 + tid % NR
    for (int r = 0; r < rounds; ++r) {
        cp_async_wait<FEW_STAGES - 1>();
        __syncwarp();
        const float* ws = ring + (r & (stages - 1)) * STAGE + gr * LINE + t2;
        const float* as = ws + NR * LINE;
        float c[TB][ACCUMULATORS][4];
#pragma unroll
        for (int b = 0; b < TB; ++b)
#pragma unroll
            for (int q = 0; q < ACCUMULATORS; ++q)
#pragma unroll
                for (int e = 0; e < 4; ++e) c[b][q][e] = 0.f;
#pragma unroll
        for (int k = 0; k < SLICE / 16; ++k) {
            uint32_t wp[PIECES][4], ap[PIECES][TB][2];
#pragma unroll
            for (int e = 0; e < 4; ++e) {                                   // rows gr, gr + 8; columns 2 t, then 2 t + 8
                const float2 x = *reinterpret_cast<const float2*>(ws + (e & 1) * 8 * LINE + 16 * k + (e >> 1) * 8);
                uint32_t p[PIECES];
                split_pair(x.x, x.y, p, lost_w[e & 1]);
                mine_w[e & 1] = larger(mine_w[e & 1], p[0]);
#pragma unroll
                for (int q = 0; q < PIECES; ++q) wp[q][e] = p[q];
            }
#pragma unroll
            for (int b = 0; b < TB; ++b)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float2 x = *reinterpret_cast<const float2*>(as + b * 8 * LINE + 16 * k + e * 8);
                    uint32_t p[PIECES];
                    split_pair(x.x, x.y, p, lost_a[b]);
                    mine_a[b] = larger(mine_a[b], p[0]);
#pragma unroll
                    for (int q = 0; q < PIECES; ++q) ap[q][b][e] = p[q];
                }
#pragma unroll
            for (int q = 0; q < PIECES; ++q)                                // (a's piece, w's piece: in the order of the tiles)
#pragma unroll
                for (int v = 0; v < PIECES; ++v) {
                    if (q + v > PIECES) continue;
#pragma unroll
                    for (int b = 0; b < TB; ++b) mma_bf16(c[b][q + v == 0 && k >= SLICE / 32 ? 0 : accumulator(q, v)], wp[v], ap[q][b][0], ap[q][b][1]);
                }
        }
        __syncwarp();
        if (r + stages < rounds) {
            ask_w(r + stages);
            ask_a(r + stages);
        }
        cp_async_commit();
        float* part = parts + (r & 1) * FEW_WARPS * MT * NR + warp * MT * NR;
#pragma unroll
        for (int b = 0; b < TB; ++b)
#pragma unroll
            for (int e = 0; e < 4; ++e) part[(8 * b + t2 + (e & 1)) * NR + gr + 8 * (e >> 1)] = slice_sum(c[b][0][e], c[b][1][e], c[b][2][e], c[b][3][e]);
        if (r + 1 == rounds) {                                              // what each row counts for, over all warps
#pragma unroll
            for (int e = 0; e < 2; ++e) atomicMax(&reach_w[gr + 8 * e], reach(most_of(mine_w[e], lost_w[e])));
#pragma unroll
            for (int b = 0; b < TB; ++b) atomicMax(&reach_a[gr + 8 * b], reach(most_of(mine_a[b], lost_a[b])));
        }
        // (one barrier a round: the half written two rounds later was read before the barrier in between)
        __syncthreads();
        const int here = min(FEW_WARPS, slices - r * FEW_WARPS);
        if (tid < MT * NR)
            for (int s = 0; s < here; ++s) total += parts[(r & 1) * FEW_WARPS * MT * NR + s * MT * NR + tid];
    }
    const int m = tid / NR, n = n0 + tid % NR;
    const bool mine = tid < MT * NR && m < M && n < N;
    const bool odd = mine && (int)(reach_a[m] + reach_w[tid % NR]) > g.highest;
    if (__syncthreads_or(odd)) {                                            // the rounds once more, by fused multiply-adds
        constexpr int NB = NR / 8, MB = MT / 4;
        float sum = 0.f;
#pragma unroll 1
        for (int r = 0; r < rounds; ++r) {
            ask_w(r);
            ask_a(r);
            cp_async_commit();
            cp_async_wait<0>();
            __syncwarp();
            const float* ws = ring + (r & (stages - 1)) * STAGE + (lane & 7) * LINE;
            const float* as = ring + (r & (stages - 1)) * STAGE + (NR + (lane >> 3)) * LINE;
            float acc[MB][NB];
#pragma unroll
            for (int i = 0; i < MB; ++i)
#pragma unroll
                for (int j = 0; j < NB; ++j) acc[i][j] = 0.f;
#pragma unroll 2
            for (int k = 0; k < SLICE; k += 4) {
                float4 wv[NB];
#pragma unroll
                for (int j = 0; j < NB; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + 8 * j * LINE + k);
#pragma unroll
                for (int i = 0; i < MB; ++i) {
                    const float4 av = *reinterpret_cast<const float4*>(as + 4 * i * LINE + k);
#pragma unroll
                    for (int j = 0; j < NB; ++j) acc[i][j] = dot4(av, wv[j], acc[i][j]);
                }
            }
            __syncwarp();
            float* part = parts + (r & 1) * FEW_WARPS * MT * NR;            // (one barrier a round, as above)
#pragma unroll
            for (int i = 0; i < MB; ++i)
#pragma unroll
                for (int j = 0; j < NB; ++j) part[(warp * MT + (lane >> 3) + 4 * i) * NR + (lane & 7) + 8 * j] = acc[i][j];
            __syncthreads();
            const int here = min(FEW_WARPS, slices - r * FEW_WARPS);
            if (tid < MT * NR)
                for (int s = 0; s < here; ++s) sum += part[s * MT * NR + tid];
        }
        if (odd) total = sum;
    }
    if (!mine) return;
    finish(g, total, n, g.out + (size_t)m * N + n);
}

template <int MT>
cudaError_t launch_few(const SplitArgs& g, cudaStream_t s) {
    static_assert(MT * FEW_N <= 32 * FEW_WARPS, "a thread per result");
    // one round of slices needs one stage: more CTAs fit an SM, and one's copies run beside another's sums
    const int stages = g.K <= FEW_WARPS * SLICE ? 1 : FEW_STAGES;
    auto bytes = [](int st) { return (int)((FEW_WARPS * st * (FEW_N + MT) * LINE + 2 * FEW_WARPS * MT * FEW_N) * sizeof(float)); };
    const cudaError_t configured = mg_raise_shared(gemm_split_few_kernel<MT>, bytes(FEW_STAGES));
    if (configured != cudaSuccess) return configured;
    return mg_launch(gemm_split_few_kernel<MT>, dim3(ceil_div(g.N, FEW_N)), dim3(32 * FEW_WARPS), bytes(stages), s, true, g, stages);
}

}  // namespace

// a: [M, K], w: [N, K], out: [M, N], all 32-bit and row-major; epilogues as mg_linear_simt.  `status` is a device int that receives
// a non-zero code if a wait inside the kernel ran out.  Returns MG_ERR_UNSUPPORTED (and launches nothing) unless K is a
// multiple of 4 and a and w lie on 16-byte boundaries: which kernel computes a matrix does not hang on the number of rows.
MG_API int mg_linear_split(const float* a, const float* w, const float* bias, float* out, float* residual, int M, int N, int K,
                           int epilogue, int* status, void* stream) {
    if (M == 0) return MG_OK;
    MG_REQUIRE(M > 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    MG_REQUIRE(epilogue >= EPI_STORE && epilogue <= EPI_RELU_SQ, "linear: unknown epilogue %d", epilogue);
    MG_REQUIRE(epilogue == EPI_RESIDUAL ? residual != nullptr : out != nullptr, "linear: missing output");
    MG_REQUIRE(status != nullptr, "linear: missing status word");
    if (K % 4 != 0 || (((uintptr_t)a | (uintptr_t)w) & 15))
        return mg_set_error(MG_ERR_UNSUPPORTED, "linear: 32-bit tensor-core path needs K %% 4 == 0 and 16-byte aligned operands");
    SplitArgs g = {a, w, bias, epilogue == EPI_RESIDUAL ? residual : out, M, N, K, epilogue, 0, highest_reach(K), status};
    g.wide = N % 4 == 0 && ((uintptr_t)g.out & 15) == 0;
    MG_REQUIRE((long long)ceil_div(M, TILE_M) * ceil_div(N, BN) < (1ll << 30), "linear: too many tiles");
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e;
    if (M <= 16) {
        e = M <= 8 ? launch_few<8>(g, s) : launch_few<16>(g, s);
    } else {
        e = launch_tiles(g, s);
    }
    if (e != cudaSuccess) return mg_set_error(MG_ERR_CUDA, "gemm_split: %s", cudaGetErrorString(e));
    MG_CHECK_LAUNCH("gemm_split");
    return MG_OK;
}
