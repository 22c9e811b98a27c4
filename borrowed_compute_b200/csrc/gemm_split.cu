// The true 32-bit matrix product on the tensor cores: Y[m, n] = sum_k X[m, k] W[n, k] for float operands, every operand taken whole.
//
// A float's 24 bits are three bfloat16 numbers: h, the nearest of 8 bits, m, the nearest to what is left, and l, the rest, exactly.
// Of the nine products of two such triples all but l l are summed, which lies below 2^-33 of the
// whole product.  (Without m l and l m, 2^-22 together, sums of one or a few products were further from 64 bits than a multiply-add; with them the tensor
// core's time is still hidden, a feed-forward of 300 rows 270 us against 267.)
// The products are exact and the tensor core adds them in float, but it truncates: sums
// of h h alone (the accumulator D1) are therefore taken out of tensor memory every 64 k and added up in registers, rounded, in ascending
// order; the seven smaller products, below 2^-6 of the first, go into an accumulator of their own (D2) that stays until the end.  Their signs
// are as good as random whatever the operands': h truncated, they had those of the operands, and where all of these are positive, a long D2, truncated
// at every addition, was off by more than the first sums (K 8,192 in eight pieces, squares by absolute values 2.1e-7, 16,384 uniform numbers 1.7e-6).
// Measured against 64 bits (2-norm of the error over that of the result), here and one multiply-add after another (gemm_simt.cu): normal operands
// 130 x 2,048 x 12,416 1.3e-7 and 8.1e-7, 130 x 8,192 x 128 in eight pieces 1.2e-7 and 5.7e-7, 7 x 1,024 x 128 0.9e-7 and 4.2e-7; uniform ones of one sign
// 130 x 8,192 x 128 0.8e-7 and 1.6e-7, 20 x 16,384 x 12,416 2.2e-7 and 1.7e-6; squares by absolute values 1.3e-7 and 1.8e-7, 2.6e-7 and 2.4e-6; rows of one
// number 2.5e-8 and 2.5e-8, of two 3.4e-8 and 3.5e-8.
// What is left after h and m is l only down to bfloat16's last bit, 2^-133: floats below 2^-110 may have bits past it, and an infinity or a not-a-number has
// no parts at all, nor has a float that would round to one.  Every row in which a block meets one (the bits that l drops are collected on the way, an instruction for two floats) is remembered, and
// that block's sums of it are taken anew, one multiply-add after another from the operands themselves (split_redo): slow, but whole.
// (The collecting costs that feed-forward 275 us against 270; a row taken anew of its 300 some 50 us more, a row of a single one 1.4 to 1.8 times its time.)
//
// Two ways, the same sums in the same order and so the same bits:
//
//   rows   Every block splits its weights, into tensor memory (the MMA's A operand, so that shared memory is free for the other), and its tokens, into
//          shared memory.  What bounds it: eight tensor-core products a multiply-add (six: 32 k, a chunk, of 128 weight rows by N tokens in some 1,000 clocks of an SM
//          at N 112), and the rounds of wait, split, store and fence of its warps, 1,425 clocks a chunk.
//   few    Up to 64 rows, where weights are what there is to read: a kernel splits the tokens once, into planes of bfloat16 in scratch memory; they
//          come by TMA as they are multiplied and all sixteen warps split weights, four buffers of triples on their way.
//          With more rows the planes' six bytes instead of four a value through the L2, in every block, cost more than the splits.  Us, this way and the other:
//          4,096 x 4,096 one row 21 and 27, 64 rows 28 and 31, 80 36 and 32, 112 40 and 33; 16,384 x 2,048 34 and 48, 47 and 54, 63 and 56, 70 and 59;
//          2,048 x 8,192 36 and 50, 49 and 56, 63 and 57, 70 and 60; 512 x 1,024 11 and 13, 16 and 16, 19 and 17, 21 and 18.
//
// Times, caches cold, against gemm_simt.cu's: 300 rows of a feed-forward of 2,048 x 8,192 158 + 118 us, 544 + 303; 3 rows 32 + 37, 126 + 78;
// 2,000 x 4,096 x 4,096 481, 1,574; one row of 2 x 14,336 x 4,096 110, 260, of 4,096 x 14,336 53, 219; 5 x 64 x 2,048 11, 35.
// (Tried for many rows, none faster: sixteen warps that split and take sums out, three and four buffers of triples, two thirds of the products, 80 and 96 tokens a tile.)
//
// Every wait is bounded.
//
// An output's sum depends on its own rows and the matrix's sizes alone: the pieces of K are the matrix's (split_pieces), added in
// ascending order through the shared memory of a cluster, and every launch of a matrix that these kernels take goes here, one row or many.
#include <cooperative_groups.h>

#include "mma_tiles.cuh"
#include "tc_ptx.cuh"
#include "tma_host.cuh"

namespace cg = cooperative_groups;

#define SPL_THREADS 576
#define SPL_K 32                 // k a chunk: 128 bytes of a row of floats
#define SPL_BN 128               // tokens a tile at most
#define SPL_W_BYTES (TC_BM * SPL_K * 4)
#define SPL_STAGES 8
#define SPL_FEW 64               // rows at most that go the second way, in one tile
#define SPL_X_STAGES 4           // stages of 64 k of their planes on their way
#define SPL_D2 256               // tensor memory of the first way: D1 at 0 and 128, D2, then two buffers of the weights' triples, 16 columns a part
#define SPL_A 384

// The second way: D1 (two of bn columns), D2, then the triples' buffers, one for each four of its warps.
#define SPL_A_COLS 48
#define SPL_BUFFERS 4
static_assert(3 * SPL_FEW + SPL_BUFFERS * SPL_A_COLS <= 512, "tensor memory");

struct SplitParams {
    float* out;
    int M, N, K;
    int second_row;              // SwiGLU: the matrix row where the up rows start
    int bn, stages, piece;
    const float *X, *W;          // the operands themselves
    const int* lost;             // the second way: [row][slice], whether three parts do not hold one of that slice's floats; slices a row and a piece of K
    int row_slices, piece_slices;
    int starve;                  // test hook: the last piece's first tile expects 16 bytes that never come, so that a bounded wait runs out
    float act_a, act_b;
    int act_cols;
};

// Four floats as triples of bfloat16, two to a register.  The last 16 bits of `lost` collect what the third parts drop: zero where they are exact.
__device__ __forceinline__ void split4(const float4 v, uint32_t* h, uint32_t* m, uint32_t* l, uint32_t& lost) {
    const uint64_t minus = pack_f32x2(-1.0f, -1.0f);
    auto two = [&](float a, float b, uint32_t& h2, uint32_t& m2, uint32_t& l2) {
        float r0, r1;
        h2 = pack_bf16(a, b);
        const uint64_t rest = fma_f32x2(pack_f32x2(__uint_as_float(h2 << 16), __uint_as_float(h2 & 0xffff0000u)), minus, pack_f32x2(a, b));
        unpack_f32x2(rest, r0, r1);
        m2 = pack_bf16(r0, r1);
        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(m2 << 16), __uint_as_float(m2 & 0xffff0000u)), minus, rest), r0, r1);
        l2 = pack_bf16(r0, r1);
        lost |= __float_as_uint(r0) | __float_as_uint(r1);
    };
    two(v.x, v.y, h[0], m[0], l[0]);
    two(v.z, v.w, h[1], m[1], l[1]);
}

// This block's sums of the rows (bits of lost: four words of weight rows, four of tokens) whose floats three parts do not hold, a warp a sum.
template <int EPI>
__device__ __noinline__ void split_redo(const SplitParams& p, float* tile, const uint32_t* lost, int t0, int n0) {
    constexpr int HALF_N = TC_BM / 2;
    const float *X = p.X, *W = p.W;
    PDL_FRESH(X); PDL_FRESH(W);
    const int lane = threadIdx.x & 31, rows = min(p.bn, p.M - t0);
    const int k_begin = blockIdx.z * p.piece, k_end = min(p.K, k_begin + p.piece);
    const bool weights = lost[0] | lost[1] | lost[2] | lost[3];
    for (int r = 0; r < rows; r++) {
        const bool all = lost[4 + (r >> 5)] >> (r & 31) & 1;
        if (!all && !weights) continue;
        const float* x = X + (size_t)(t0 + r) * p.K;
        for (int c = threadIdx.x >> 5; c < TC_BM; c += SPL_THREADS / 32) {
            const int n = n0 + (EPI == EPI_SWIGLU ? c % HALF_N : c);
            if (n >= p.N || !(all || (lost[c >> 5] >> (c & 31) & 1))) continue;
            const float* w = W + ((size_t)(EPI == EPI_SWIGLU && c >= HALF_N ? p.second_row : 0) + n) * p.K;
            float sum = 0.0f;
#pragma unroll 4
            for (int k = k_begin + 4 * lane; k < k_end; k += 128) {
                const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
                sum = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
            }
            sum = warp_sum(sum);
            if (lane == 0) tile[r * TC_BM + c] = sum;
        }
    }
}

// Two tokens' sums of a weight row into the tile; `largest`: of their bits without the sign.
__device__ __forceinline__ void split_put(float* at, float s0, float s1, uint32_t& largest) {
    at[0] = s0;
    at[TC_BM] = s1;
    largest = max(largest, max(__float_as_uint(s0) << 1, __float_as_uint(s1) << 1));
}
// A sum that is not finite may be the parts' doing (first parts rounded up, their product past the largest float): its token's sums are taken anew as well.
// This thread's sums: of `tokens` tokens from token0 on.
__device__ __forceinline__ void split_overflow(const float* at, int token0, int tokens, uint32_t* lost, uint32_t largest) {
    if (largest < 0xff000000u) return;
    for (int t = 0; t < tokens; t++)
        if (!(fabsf(at[t * TC_BM]) < INFINITY)) atomicOr(&lost[4 + ((token0 + t) >> 5)], 1u << ((token0 + t) & 31));
}

// The end of both: the sums of the pieces of K, in ascending order out of the cluster's blocks, and the epilogue.
template <int EPI>
__device__ __forceinline__ void split_finish(const SplitParams& p, float* tile, uint32_t tmem, bool dealloc, int* gave_up, const uint32_t* lost, int t0, int n0) {
    constexpr int HALF_N = TC_BM / 2, OUT_COLS = EPI == EPI_SWIGLU ? HALF_N : TC_BM;
    const int S = gridDim.z;
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (dealloc) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    const uint4 of_w = *reinterpret_cast<const uint4*>(lost), of_x = *reinterpret_cast<const uint4*>(lost + 4);
    const bool failed_here = *reinterpret_cast<volatile int*>(gave_up);
    const bool redo = (of_w.x | of_w.y | of_w.z | of_w.w | of_x.x | of_x.y | of_x.z | of_x.w) && !failed_here;
    if (redo) split_redo<EPI>(p, tile, lost, t0, n0);
    if (S > 1) {
        cg::this_cluster().barrier_wait();                   // of the start: all blocks' words are there
        if (failed_here && threadIdx.x < S) *cg::this_cluster().map_shared_rank(gave_up, threadIdx.x) = 1;      // what one gives up, no other writes
        cg::this_cluster().sync();
    } else if (redo) __syncthreads();
    if (!*reinterpret_cast<volatile int*>(gave_up)) {
        const int rows = min(p.bn, p.M - t0);
        for (int e = blockIdx.z * SPL_THREADS + threadIdx.x; e < rows * OUT_COLS; e += S * SPL_THREADS) {
            const int r = e / OUT_COLS, c = e % OUT_COLS, n = n0 + c;
            if (n >= p.N) continue;
            float v = 0.0f, u = 0.0f;
            for (int z = 0; z < S; z++) {
                const float* theirs = S > 1 ? cg::this_cluster().map_shared_rank(tile, z) : tile;
                v = z ? v + theirs[r * TC_BM + c] : theirs[r * TC_BM + c];
                if (EPI == EPI_SWIGLU) u = z ? u + theirs[r * TC_BM + HALF_N + c] : theirs[r * TC_BM + HALF_N + c];
            }
            simt_emit<float, EPI>(p.out, p.out, t0 + r, n, p.N, v, u, p.act_a, p.act_b, p.act_cols);
        }
    }
    if (S > 1) cg::this_cluster().sync();      // no block leaves while a peer still reads its shared memory
}

// Warps: 0-3 split the weights, a row a thread, 4-7 the tokens; 8-15 take D1 out and write the result; 16 asks for raw tiles (TMA, 32 floats of a row, 128-byte
// swizzle); 17 issues the products.
template <int EPI>
__global__ void __launch_bounds__(SPL_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ SplitParams p) {
    constexpr int HALF_N = TC_BM / 2, OUT_COLS = EPI == EPI_SWIGLU ? HALF_N : TC_BM;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * SPL_STAGES + 4 + 4 + 2 + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ int gave_up;
    __shared__ __align__(16) uint32_t lost[8];      // rows whose floats three parts do not hold, a bit each: weight rows, tokens
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int bn = p.bn, stages = p.stages;
    const int plane = bn * 128, stage_bytes = SPL_W_BYTES + plane;      // a plane: bn rows of 64 k of one part; two stages of three planes behind the raw ring
    uint8_t* planes = smem + stages * stage_bytes;
    const int t0 = blockIdx.x * bn, n0 = blockIdx.y * OUT_COLS;
    const int k_begin = blockIdx.z * p.piece, k_end = min(p.K, k_begin + p.piece);
    const int chunks = (k_end - k_begin + SPL_K - 1) / SPL_K, periods = (chunks + 1) / 2;
    const uint32_t raw_full = smem_u32(bars), raw_empty = raw_full + 8 * SPL_STAGES, ready = raw_empty + 8 * SPL_STAGES, done = ready + 32, d1_full = done + 32,
                   d1_empty = d1_full + 16;
    if (threadIdx.x < 8) lost[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int s = 0; s < stages; s++) {
            mbar_init(raw_full + 8 * s, 1);
            mbar_init(raw_empty + 8 * s, 8);
        }
        for (int i = 0; i < 4; i++) {
            mbar_init(ready + 8 * i, 256);
            mbar_init(done + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(d1_full + 8 * i, 1);
            mbar_init(d1_empty + 8 * i, 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    if (gridDim.z > 1) cg::this_cluster().barrier_arrive();      // (split_finish waits for it)
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    float* tile = reinterpret_cast<float*>(smem);        // [bn][128]: the result, over the raw ring once that is drained
    bool ok = true;
    auto wait = [&](uint32_t bar, int phase, int code) { return ok = mbar_wait_warp(bar, phase & 1, code); };   // the whole warp
    pdl_launch_dependents();
    pdl_wait();       // the weights too: a caller's matrix may be what the kernel before has just written
    if (warp < 8) {
        // Chunk j: raw stage j % stages -> weights: tensor memory buffer j % 2, free when the products of chunk j - 2 are done; tokens: half j % 2 of plane
        // stage (j / 2) % 2, free when those of chunk j - 4 are.
        const bool weights = warp < 4;
        const int row = 32 * (warp & 3) + lane;
        const uint32_t a_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + SPL_A;
        const int back = weights ? 2 : 4;
        uint32_t dropped = 0;
        for (int j = 0, s = 0, round = 0; j < chunks; j++) {
            if (!wait(raw_full + 8 * s, round, 1)) break;
            const uint8_t* src = smem + (size_t)s * stage_bytes + (weights ? 0 : SPL_W_BYTES) + row * 128;
            uint32_t h[16], m[16], l[16];
            if (weights || row < bn) {
                float4 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) v[c] = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
#pragma unroll
                for (int c = 0; c < 8; c++) split4(v[c], h + 2 * c, m + 2 * c, l + 2 * c, dropped);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(raw_empty + 8 * s);
            if (++s == stages) s = 0, round++;
            if (j >= back && !wait(done + 8 * ((j - back) & 3), (j - back) >> 2, 2)) break;
            if (weights) {
                tc_fence_after();
                const uint32_t a = a_addr + (j & 1) * 48;
                tmem_store16(a, h);
                tmem_store16(a + 16, m);
                tmem_store16(a + 32, l);
                tmem_store_wait();
                tc_fence_before();
            } else {
                if (row < bn) {
                    uint8_t* dst = planes + ((j >> 1) & 1) * 3 * plane + row * 128;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const int at = (((j & 1) * 4 + c) ^ (row & 7)) << 4;
                        *reinterpret_cast<uint4*>(dst + at) = make_uint4(h[4 * c], h[4 * c + 1], h[4 * c + 2], h[4 * c + 3]);
                        *reinterpret_cast<uint4*>(dst + plane + at) = make_uint4(m[4 * c], m[4 * c + 1], m[4 * c + 2], m[4 * c + 3]);
                        *reinterpret_cast<uint4*>(dst + 2 * plane + at) = make_uint4(l[4 * c], l[4 * c + 1], l[4 * c + 2], l[4 * c + 3]);
                    }
                }
                fence_proxy_async();
            }
            mbar_arrive(ready + 8 * (j & 3));
        }
        const uint32_t rows = __ballot_sync(0xffffffffu, dropped & 0xffffu);
        if (lane == 0 && rows) atomicOr(&lost[warp], rows);
    } else if (warp < 16) {
        // Two warps a quarter of the lanes: every other sixteen of the token columns each.
        const int q = warp & 3, half = (warp - 8) >> 2;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16) + 16 * half;
        uint64_t acc[4][8] = {};
        for (int i = 0; i < periods; i++) {
            const int b = i & 1;
            if (!wait(d1_full + 8 * b, i >> 1, 3)) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (32 * c + 16 * half >= bn) break;
                uint32_t v[16];
                tmem_load16(lanes + 128 * b + 32 * c, v);
                tmem_load_wait();
#pragma unroll
                for (int e = 0; e < 8; e++) acc[c][e] = add_f32x2(acc[c][e], pack_f32x2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])));
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d1_empty + 8 * b);
        }
        if (ok) {
            // D1's last sums came after the last product, D2's with them.  No raw tile is on its way and none is read any more.
#pragma unroll
            for (int c = 0; c < 4; c++) {
                if (32 * c + 16 * half >= bn) break;
                float* at = tile + (32 * c + 16 * half) * TC_BM + 32 * q + lane;
                uint32_t v[16], largest = 0;
                tmem_load16(lanes + SPL_D2 + 32 * c, v);
                tmem_load_wait();
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    float a0, a1;
                    unpack_f32x2(acc[c][e], a0, a1);
                    split_put(at + 2 * e * TC_BM, a0 + __uint_as_float(v[2 * e]), a1 + __uint_as_float(v[2 * e + 1]), largest);
                }
                split_overflow(at, 32 * c + 16 * half, 16, lost, largest);
            }
        }
    } else if (warp == 16) {
        if (elect_one()) {
            const int second = EPI == EPI_SWIGLU ? p.second_row + n0 : n0 + HALF_N;
            const bool starve = p.starve && blockIdx.z + 1 == gridDim.z;
            for (int j = 0, s = 0, round = 0; j < chunks; j++) {
                const int k = k_begin + j * SPL_K;
                if (round && !(ok = mbar_wait(raw_empty + 8 * s, (round - 1) & 1, 4))) break;
                const uint32_t dst = smem_u32(smem + (size_t)s * stage_bytes), bar = raw_full + 8 * s;
                mbar_expect_tx(bar, (uint32_t)stage_bytes + (j == 0 && starve ? 16 : 0));
                tma_load_2d(dst, &map_w, bar, k, n0);
                tma_load_2d(dst + SPL_W_BYTES / 2, &map_w, bar, k, second);
                tma_load_2d(dst + SPL_W_BYTES, &map_x, bar, k, t0);
                if (++s == stages) s = 0, round++;
            }
        }
    } else {
        const uint32_t idesc = instr_desc(bn);
        const uint64_t b_desc = smem_desc(smem_u32(planes));
        const uint32_t part = (uint32_t)plane >> 4;
        for (int j = 0; j < chunks; j++) {
            const int b = (j >> 1) & 1;
            if (!(j & 1) && j >= 4 && !wait(d1_empty + 8 * b, (j >> 2) - 1, 5)) break;
            if (!wait(ready + 8 * (j & 3), j >> 2, 6)) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < SPL_K / 16; kk++) {
                    const uint32_t a = tmem + SPL_A + (j & 1) * 48 + 8 * kk;
                    const uint64_t h = b_desc + (uint64_t)(b * 3 * part + (j & 1) * 4 + 2 * kk), m = h + part, l = m + part;
                    mma_bf16_a_tmem(tmem + 128 * b, a, h, idesc, (j & 1) | kk);
                    mma_bf16_a_tmem(tmem + SPL_D2, a + 16, h, idesc, j | kk);
                    mma_bf16_a_tmem(tmem + SPL_D2, a, m, idesc, 1);
                    mma_bf16_a_tmem(tmem + SPL_D2, a + 16, m, idesc, 1);
                    mma_bf16_a_tmem(tmem + SPL_D2, a + 32, h, idesc, 1);
                    mma_bf16_a_tmem(tmem + SPL_D2, a, l, idesc, 1);
                    mma_bf16_a_tmem(tmem + SPL_D2, a + 32, m, idesc, 1);
                    mma_bf16_a_tmem(tmem + SPL_D2, a + 16, l, idesc, 1);
                }
                mma_commit(done + 8 * (j & 3));
                if ((j & 1) || j + 1 == chunks) mma_commit(d1_full + 8 * b);
            }
            __syncwarp();
        }
    }
    if (!ok) *reinterpret_cast<volatile int*>(&gave_up) = 1;
    split_finish<EPI>(p, tile, tmem, warp == 17, &gave_up, lost, t0, n0);
}

// planes[part][row][k_row] = the parts of x[row][k], four k a thread; lost[row][slice]: whether they do not hold one of the slice's floats.  Block (x, y): row y's
// slice x, of at most SPL_SLICE k of one piece.
#define SPL_SLICE 1024
__global__ void __launch_bounds__(SPL_SLICE / 4) split_rows_kernel(const float* x, bf16* __restrict__ planes, int* __restrict__ lost, int rows, int K, int k_row, int piece, int piece_slices) {
    pdl_wait();                        // before the next kernel may start: it reads its weights at once
    pdl_launch_dependents();
    PDL_FRESH(x);
    const size_t part = (size_t)rows * k_row;
    const int r = blockIdx.y, begin = blockIdx.x / piece_slices * piece, k = begin + blockIdx.x % piece_slices * SPL_SLICE + 4 * threadIdx.x;
    uint32_t dropped = 0;
    if (k < min(K, begin + piece)) {
        uint32_t h[2], m[2], l[2];
        split4(*reinterpret_cast<const float4*>(x + (size_t)r * K + k), h, m, l, dropped);
        bf16* to = planes + (size_t)r * k_row + k;
        *reinterpret_cast<uint2*>(to) = make_uint2(h[0], h[1]);
        *reinterpret_cast<uint2*>(to + part) = make_uint2(m[0], m[1]);
        *reinterpret_cast<uint2*>(to + 2 * part) = make_uint2(l[0], l[1]);
    }
    const int any = __syncthreads_or(dropped & 0xffffu);
    if (threadIdx.x == 0) lost[(size_t)r * gridDim.x + blockIdx.x] = any;
}

// Warps: 0-15 split the weights of every fourth chunk, four warps a chunk, a row a thread, and take D1 out, a share of the columns each; 16 asks for tiles; 17
// issues the products.
template <int EPI>
__global__ void __launch_bounds__(SPL_THREADS, 1)
gemm_split_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ SplitParams p) {
    constexpr int HALF_N = TC_BM / 2;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * SPL_STAGES + 2 * SPL_X_STAGES + 4 + 4 + 2 + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ int gave_up;
    __shared__ __align__(16) uint32_t lost[8];      // rows whose floats three parts do not hold, a bit each: weight rows, tokens
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int bn = p.bn, stages = p.stages;
    const int d2_at = 2 * bn, a_at = 3 * bn;
    const int plane = bn * 128;                              // bn rows of 64 k of one part; stages of three behind the ring of weights
    uint8_t* planes = smem + stages * SPL_W_BYTES;
    const int t0 = blockIdx.x * bn, n0 = blockIdx.y * (EPI == EPI_SWIGLU ? HALF_N : TC_BM);
    const int k_begin = blockIdx.z * p.piece, k_end = min(p.K, k_begin + p.piece);
    const int chunks = (k_end - k_begin + SPL_K - 1) / SPL_K, periods = (chunks + 1) / 2;
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * SPL_STAGES, x_full = w_empty + 8 * SPL_STAGES, x_empty = x_full + 8 * SPL_X_STAGES,
                   ready = x_empty + 8 * SPL_X_STAGES, done = ready + 32, d1_full = done + 32, d1_empty = d1_full + 16;
    if (threadIdx.x < 8) lost[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        gave_up = 0;
        for (int i = 0; i < SPL_STAGES; i++) {
            mbar_init(w_full + 8 * i, 1);
            mbar_init(w_empty + 8 * i, 4);
        }
        for (int i = 0; i < SPL_X_STAGES; i++) {
            mbar_init(x_full + 8 * i, 1);
            mbar_init(x_empty + 8 * i, 1);
        }
        for (int i = 0; i < 4; i++) {
            mbar_init(ready + 8 * i, 4);
            mbar_init(done + 8 * i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(d1_full + 8 * i, 1);
            mbar_init(d1_empty + 8 * i, 16);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 17) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    if (gridDim.z > 1) cg::this_cluster().barrier_arrive();      // (split_finish waits for it)
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    float* tile = reinterpret_cast<float*>(smem);        // [bn][128]: the result, over the ring of weights once that is drained
    bool ok = true;
    auto wait = [&](uint32_t bar, int phase, int code) { return ok = mbar_wait_warp(bar, phase & 1, code); };   // the whole warp
    pdl_launch_dependents();
    if (warp < 16) {
        // Chunk j is four warps' (j % 4): out of ring stage j % stages into tensor memory buffer j % 4, free when the products of chunk j - 4
        // are done.  After its chunk every warp takes its share of the stretches (two chunks each) before out of D1.
        const int q = warp & 3, part = warp >> 2;
        const int row = 32 * q + lane;
        const uint32_t lanes = tmem + ((uint32_t)(32 * q) << 16);
        uint64_t acc[8] = {};                                // token columns 16 part ..
        uint32_t dropped = 0;
        int taken = 0;
        auto take_out_before = [&](int end) {
            for (; taken < end; taken++) {
                const int b = taken & 1;
                if (!wait(d1_full + 8 * b, taken >> 1, 3)) return;
                tc_fence_after();
                if (16 * part < bn) {
                    uint32_t v[16];
                    tmem_load16(lanes + bn * b + 16 * part, v);
                    tmem_load_wait();
#pragma unroll
                    for (int e = 0; e < 8; e++) acc[e] = add_f32x2(acc[e], pack_f32x2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d1_empty + 8 * b);
            }
        };
        const uint32_t to = lanes + a_at + part * SPL_A_COLS;
        for (int j = part, s = part % stages, round = part / stages; j < chunks; j += 4) {
            if (!wait(w_full + 8 * s, round, 1)) break;
            const uint8_t* src = smem + s * SPL_W_BYTES + row * 128;
            uint32_t h[16], m[16], l[16];
            float4 v[8];
#pragma unroll
            for (int c = 0; c < 8; c++) v[c] = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
#pragma unroll
            for (int c = 0; c < 8; c++) split4(v[c], h + 2 * c, m + 2 * c, l + 2 * c, dropped);
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty + 8 * s);
            if ((s += 4) >= stages) s -= stages, round++;
            if (j >= 4 && !wait(done + 8 * part, (j >> 2) - 1, 2)) break;
            tc_fence_after();
            tmem_store16(to, h);
            tmem_store16(to + 16, m);
            tmem_store16(to + 32, l);
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * part);
            take_out_before(j / 2);       // all but the stretch under way: the products of the next one but one wait for this one's sums
            if (!ok) break;
        }
        const uint32_t rows = __ballot_sync(0xffffffffu, dropped & 0xffffu);
        if (lane == 0 && rows) atomicOr(&lost[q], rows);     // (four warps a quarter)
        if (ok) take_out_before(periods);
        if (ok) {
            // D1's last sums came after the last product, D2's with them.  No tile is on its way and none is read any more.
            if (16 * part < bn) {
                float* at = tile + 16 * part * TC_BM + 32 * q + lane;
                uint32_t v[16], largest = 0;
                tmem_load16(lanes + d2_at + 16 * part, v);
                tmem_load_wait();
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    float a0, a1;
                    unpack_f32x2(acc[e], a0, a1);
                    split_put(at + 2 * e * TC_BM, a0 + __uint_as_float(v[2 * e]), a1 + __uint_as_float(v[2 * e + 1]), largest);
                }
                split_overflow(at, 16 * part, 16, lost, largest);
            }
        }
    } else if (warp == 16) {
        if (elect_one()) {
            const int second = EPI == EPI_SWIGLU ? p.second_row + n0 : n0 + HALF_N;
            const bool starve = p.starve && blockIdx.z + 1 == gridDim.z;
            auto load_w = [&](int j, int s) {
                const uint32_t dst = smem_u32(smem + s * SPL_W_BYTES), bar = w_full + 8 * s;
                mbar_expect_tx(bar, SPL_W_BYTES + (j == 0 && starve ? 16 : 0));
                tma_load_2d(dst, &map_w, bar, k_begin + j * SPL_K, n0);
                tma_load_2d(dst + SPL_W_BYTES / 2, &map_w, bar, k_begin + j * SPL_K, second);
            };
            // The kernel before is the one that split the tokens, and it waited for all before it: the weights are there.
            const int ahead = min(stages, chunks);
            for (int j = 0; j < ahead; j++) load_w(j, j);
            pdl_wait();
            for (int j = 0, s = 0, round = 0, xs = 0, x_round = 0; j < chunks; j++) {
                if (!(j & 1)) {
                    if (x_round && !(ok = mbar_wait(x_empty + 8 * xs, (x_round - 1) & 1, 4))) break;
                    const uint32_t dst = smem_u32(planes + xs * 3 * plane), bar = x_full + 8 * xs;
                    mbar_expect_tx(bar, (uint32_t)(3 * plane));
                    for (int i = 0; i < 3; i++) tma_load_3d(dst + i * plane, &map_x, bar, k_begin + j * SPL_K, t0, i);
                    if (++xs == SPL_X_STAGES) xs = 0, x_round++;
                }
                if (round) {
                    if (!(ok = mbar_wait(w_empty + 8 * s, (round - 1) & 1, 4))) break;
                    load_w(j, s);
                }
                if (++s == stages) s = 0, round++;
            }
        }
        __syncwarp();
        // The last tiles are on their way: time to look which of the tokens' rows need their sums anew.
        pdl_wait();
        const int* flags = p.lost;
        PDL_FRESH(flags);
        for (int i = 0; 32 * i < bn; i++) {
            const int r = t0 + 32 * i + lane;
            int any = 0;
            if (r < p.M)
                for (int c = 0; c < p.piece_slices; c++) any |= flags[(size_t)r * p.row_slices + blockIdx.z * p.piece_slices + c];
            const uint32_t rows = __ballot_sync(0xffffffffu, any);
            if (lane == 0 && rows) atomicOr(&lost[4 + i], rows);
        }
    } else {
        const uint32_t idesc = instr_desc(bn);
        const uint64_t b_desc = smem_desc(smem_u32(planes));
        const uint32_t part = (uint32_t)plane >> 4;
        for (int j = 0, xs = 0, x_round = 0; j < chunks; j++) {
            const int b = (j >> 1) & 1;
            const bool last = (j & 1) || j + 1 == chunks;     // of its stretch and its stage of tokens
            if (!(j & 1)) {
                if (!wait(x_full + 8 * xs, x_round, 6)) break;
                if (j >= 4 && !wait(d1_empty + 8 * b, (j >> 2) - 1, 5)) break;
            }
            if (!wait(ready + 8 * (j & 3), j >> 2, 6)) break;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < SPL_K / 16; kk++) {
                    const uint32_t a = tmem + a_at + (j & 3) * SPL_A_COLS + 8 * kk;
                    const uint64_t h = b_desc + (uint64_t)(xs * 3 * part + (j & 1) * 4 + 2 * kk), m = h + part, l = m + part;
                    mma_bf16_a_tmem(tmem + bn * b, a, h, idesc, (j & 1) | kk);
                    mma_bf16_a_tmem(tmem + d2_at, a + 16, h, idesc, j | kk);
                    mma_bf16_a_tmem(tmem + d2_at, a, m, idesc, 1);
                    mma_bf16_a_tmem(tmem + d2_at, a + 16, m, idesc, 1);
                    mma_bf16_a_tmem(tmem + d2_at, a + 32, h, idesc, 1);
                    mma_bf16_a_tmem(tmem + d2_at, a, l, idesc, 1);
                    mma_bf16_a_tmem(tmem + d2_at, a + 32, m, idesc, 1);
                    mma_bf16_a_tmem(tmem + d2_at, a + 16, l, idesc, 1);
                }
                mma_commit(done + 8 * (j & 3));
                if (last) {
                    mma_commit(x_empty + 8 * xs);
                    mma_commit(d1_full + 8 * b);
                }
            }
            __syncwarp();
            if (last && ++xs == SPL_X_STAGES) xs = 0, x_round++;
        }
    }
    pdl_wait();       // the output may still be in use by a kernel before
    if (!ok) *reinterpret_cast<volatile int*>(&gave_up) = 1;
    split_finish<EPI>(p, tile, tmem, warp == 17, &gave_up, lost, t0, n0);
}

// -------------------------------------------------------------------------------- the host
static int float_map(CUtensorMap* map, const void* base, int rows, int K, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 4};
    cuuint32_t box[2] = {SPL_K, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    const CUresult r = bc_encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        bc_set_error("gemm_split: cuTensorMapEncodeTiled failed (%d) for a [%d, %d] matrix, box %d x %d", (int)r, rows, K, box_rows, SPL_K);
        return BC_ERR_DRIVER;
    }
    return BC_OK;
}

static int planes_map(CUtensorMap* map, const void* base, int rows, int K, int k_row, int bn) {
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 3}, strides[2] = {(cuuint64_t)k_row * 2, (cuuint64_t)k_row * 2 * rows};
    cuuint32_t box[3] = {2 * SPL_K, (cuuint32_t)bn, 1}, elem[3] = {1, 1, 1};
    const CUresult r = bc_encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        bc_set_error("gemm_split: cuTensorMapEncodeTiled failed (%d) for planes of [%d, %d], box %d x %d", (int)r, rows, K, bn, 2 * SPL_K);
        return BC_ERR_DRIVER;
    }
    return BC_OK;
}

// The pieces that a sum over K is added up in, for a product with `cols` weight rows: more than one where the tiles of few rows would
// leave SMs idle and K is long enough.
static int split_pieces(int cols, int K) {
    int s = 1;
    while ((cols + 127) / 128 * s < 96 && s < 8 && K / (2 * s) >= 512) s *= 2;
    return s;
}

// Whether this kernel takes a matrix [cols, K] and rows beside it.  By the matrix alone, so that a row's sum has the same order whoever else is in the launch.
extern "C" int bc_gemm_split_takes(const void* X, const void* W, int cols, int K) {
    return K > 512 && K % 4 == 0 && (uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0 && (long long)cols <= 65535ll * 64 && bc_encode_tiled_fn() != nullptr;
}

static int g_split_starve = 0;
extern "C" void bc_gemm_split_test_starve_next_launch() { g_split_starve = 1; }

static int split_k_row(int K) { return (K + 7) / 8 * 8; }
// Bytes of scratch: three planes of the rows that go the second way, and a word a row and slice of K (the pieces' slices, at most K / SPL_SLICE and ten more).
extern "C" long long bc_gemm_split_scratch(int M, int K) { return M <= SPL_FEW ? 6ll * M * split_k_row(K) + 4ll * M * (K / SPL_SLICE + 10) : 0; }

template <int EPI>
static int launch(const void* X, const void* W, void* out, int M, int N, int K, float a, float b, int cols, void* scratch, cudaStream_t s) {
    const int w_rows = EPI == EPI_SWIGLU ? 2 * N : N, out_cols = EPI == EPI_SWIGLU ? TC_BM / 2 : TC_BM;
    const bool few = M <= SPL_FEW;
    SplitParams p = {};
    p.out = (float*)out, p.M = M, p.N = N, p.K = K, p.second_row = N, p.act_a = a, p.act_b = b, p.act_cols = cols;
    const int t_tiles = (M + SPL_BN - 1) / SPL_BN;
    p.bn = ((M + t_tiles - 1) / t_tiles + 15) / 16 * 16;
    const int splits = split_pieces(w_rows, K);
    p.piece = ((K + splits - 1) / splits + 2 * SPL_K - 1) / (2 * SPL_K) * (2 * SPL_K);
    p.X = (const float*)X, p.W = (const float*)W;
    p.piece_slices = (p.piece + SPL_SLICE - 1) / SPL_SLICE, p.row_slices = splits * p.piece_slices;
    int* lost = few ? (int*)((char*)scratch + 6ll * M * split_k_row(K)) : nullptr;
    p.lost = lost;
    p.starve = g_split_starve;
    g_split_starve = 0;
    // A ring of chunks, both operands' raw tiles or the weights' alone, and stages of 64 k of the tokens' planes.
    const int stage = SPL_W_BYTES + (few ? 0 : p.bn * 128), planes = (few ? SPL_X_STAGES : 2) * 3 * p.bn * 128;
    p.stages = (TC_SMEM_LIMIT - 1024 - planes) / stage;
    if (p.stages > SPL_STAGES) p.stages = SPL_STAGES;
    const int smem = p.stages * stage + planes + 1024;
    CUtensorMap mw, mx;
    int st = float_map(&mw, W, w_rows, K, TC_BM / 2);
    if (st == BC_OK) st = few ? planes_map(&mx, scratch, M, K, split_k_row(K), p.bn) : float_map(&mx, X, M, K, p.bn);
    if (st != BC_OK) return st;
    cudaError_t e = few ? bc_allow_shared<gemm_split_few_kernel<EPI>>(TC_SMEM_LIMIT) : bc_allow_shared<gemm_split_kernel<EPI>>(TC_SMEM_LIMIT);
    if (e == cudaSuccess && few)
        e = bc_launch(split_rows_kernel, dim3(p.row_slices, M), dim3(SPL_SLICE / 4), 0, s, (const float*)X, (bf16*)scratch, lost, M, K, split_k_row(K), p.piece, p.piece_slices);
    // Token tiles fastest: the blocks that read the same weights run side by side.
    const dim3 grid((M + p.bn - 1) / p.bn, (N + out_cols - 1) / out_cols, splits);
    auto go = [&](auto kernel) {
        return splits > 1 ? bc_launch_clustered(kernel, grid, dim3(SPL_THREADS), (size_t)smem, s, dim3(1, 1, splits), mw, mx, p)
                          : bc_launch(kernel, grid, dim3(SPL_THREADS), (size_t)smem, s, mw, mx, p);
    };
    if (e == cudaSuccess) e = few ? go(gemm_split_few_kernel<EPI>) : go(gemm_split_kernel<EPI>);
    if (e != cudaSuccess) {
        bc_set_error("gemm_split: launch failed: %s", cudaGetErrorString(e));
        return (int)e;
    }
    BC_LAUNCH_STATUS();
}

// gemm_simt's float product for what bc_gemm_split_takes, with bc_gemm_split_scratch(M, K) bytes of scratch (on a 16-byte border).
extern "C" int bc_gemm_split_f32(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, float a, float b, int cols, void* scratch, cudaStream_t s) {
    BC_CHECK_ARG(M >= 0 && N > 0 && K > 0, "gemm_split: bad sizes M=%d N=%d K=%d", M, N, K);
    BC_CHECK_ARG(bc_gemm_split_takes(X, W, epilogue == EPI_SWIGLU ? 2 * N : N, K), "gemm_split: K=%d must be more than 512 and a multiple of four, the operands on 16-byte borders", K);
    if (M == 0) return BC_OK;
    BC_CHECK_ARG(M > SPL_FEW || (scratch != nullptr && (uintptr_t)scratch % 16 == 0), "gemm_split: %d rows take scratch on a 16-byte border", M);
    switch (epilogue) {
        case EPI_STORE: return launch<EPI_STORE>(X, W, out, M, N, K, a, b, cols, scratch, s);
        case EPI_STORE_F32: return launch<EPI_STORE_F32>(X, W, out, M, N, K, a, b, cols, scratch, s);
        case EPI_ADD_F32: return launch<EPI_ADD_F32>(X, W, out, M, N, K, a, b, cols, scratch, s);
        case EPI_SWIGLU: return launch<EPI_SWIGLU>(X, W, out, M, N, K, a, b, cols, scratch, s);
        case EPI_RELU2: return launch<EPI_RELU2>(X, W, out, M, N, K, a, b, cols, scratch, s);
        case EPI_XIELU: return launch<EPI_XIELU>(X, W, out, M, N, K, a, b, cols, scratch, s);
        case EPI_SILU_F32: return launch<EPI_SILU_F32>(X, W, out, M, N, K, a, b, cols, scratch, s);
    }
    bc_set_error("gemm_split: unknown epilogue %d", epilogue);
    return BC_ERR_ARG;
}

// This unit's status word, its wait limit and its word of host memory: bc_gemm_split_status / _set_wait_cycles / _bind_host_word.
TC_STATUS_EXPORTS(gemm_split)
