// The true 32-bit matrix product on the tensor cores: Y[m, n] = sum_k X[m, k] W[n, k] for float operands, every operand taken whole.
//
// A float's 24 bits are three bfloat16 numbers: h, its first 8 bits (truncated, so that no finite number becomes an infinity), m, the
// next, rounded, and l, what is left, exactly.  Of the nine products of two such triples six are summed: h h, h m, m h, m m, h l, l h; the
// others lie below 2^-22 of the whole product.  The products are exact and the tensor core adds them in float, but it truncates: sums
// of h h alone (the accumulator D1) are therefore taken out of tensor memory every 64 k and added up in registers, rounded, in ascending
// order; the five smaller products, at most 2^-7 of the first, go into an accumulator of their own (D2) that stays until the end.
// Measured against 64 bits (2-norm of the error over that of the result, normal operands): 300 x 8,192 x 2,048 1.7e-7, one multiply-add after another
// (gemm_simt.cu) 8.1e-7; 300 x 2,048 x 8,192 in eight pieces 1.4e-7 and 5.8e-7; 3 x 2,816 x 1,024 1.1e-7 and 4.0e-7.
// Operands below 2^-110 lose their last bits (bfloat16 ends at 2^-133).
// An operand that is infinite or not a number has no m and l: where the sum of h h is either, it is the result by itself.
//
// What bounds it: six tensor-core products a multiply-add, 32 k of 128 weight rows by N tokens in 6 N clocks of an SM, beside the
// conversions (285 clocks a warp for 32 rows of 32 k) and shared memory (B operands, raw tiles and planes).  To keep shared memory free the weights' triples
// go to tensor memory (the MMA's A operand), only the tokens' to shared memory.
// Times, caches cold, this kernel against gemm_simt.cu's: 300 rows of a feed-forward of 2,048 x 8,192 157 + 126 us against 544 + 303; 3 rows 50 + 53 against 126 + 78;
// 2,000 x 4,096 x 4,096 481 against 1,574; one row of 2 x 14,336 x 4,096 168 against 260, of 4,096 x 14,336 80 against 219; 5 x 64 x 2,048 19 against 35.
//
// Warps: 0-3 split the weights, a row a thread, into tensor memory; 4-7 the tokens, into shared memory; 8-15 take D1 out and write the
// result; 16 asks for raw tiles (TMA, 32 floats of a row, 128-byte swizzle); 17 issues the products.  Every wait is bounded.
//
// An output's sum depends on its own rows and the matrix's sizes alone: the pieces of K are the matrix's (split_pieces), added in
// ascending order through the shared memory of a cluster, and every launch of a matrix that this kernel takes goes here, one row or many.
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
#define SPL_D2 256               // tensor memory: D1 at 0 and 128, D2, then two buffers of the weights' triples, 16 columns a part
#define SPL_A 384

struct SplitParams {
    float* out;
    int M, N, K;
    int second_row;              // SwiGLU: the matrix row where the up rows start
    int bn, stages, piece;
    float act_a, act_b;
    int act_cols;
};

// Four floats as triples of bfloat16, two to a register.
__device__ __forceinline__ void split4(const float4 v, uint32_t* h, uint32_t* m, uint32_t* l) {
    const uint64_t minus = pack_f32x2(-1.0f, -1.0f);
    auto two = [&](float a, float b, uint32_t& h2, uint32_t& m2, uint32_t& l2) {
        asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(h2) : "f"(b), "f"(a));
        float r0, r1;
        const uint64_t rest = fma_f32x2(pack_f32x2(__uint_as_float(h2 << 16), __uint_as_float(h2 & 0xffff0000u)), minus, pack_f32x2(a, b));
        unpack_f32x2(rest, r0, r1);
        m2 = pack_bf16(r0, r1);
        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(m2 << 16), __uint_as_float(m2 & 0xffff0000u)), minus, rest), r0, r1);
        l2 = pack_bf16(r0, r1);
    };
    two(v.x, v.y, h[0], m[0], l[0]);
    two(v.z, v.w, h[1], m[1], l[1]);
}

template <int EPI>
__global__ void __launch_bounds__(SPL_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const SplitParams p) {
    constexpr int HALF_N = TC_BM / 2, OUT_COLS = EPI == EPI_SWIGLU ? HALF_N : TC_BM;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t bars[2 * SPL_STAGES + 4 + 4 + 2 + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ int gave_up;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int bn = p.bn, stages = p.stages;
    const int plane = bn * 128, stage_bytes = SPL_W_BYTES + plane;      // a plane: bn rows of 64 k of one part; two stages of three planes behind the raw ring
    uint8_t* planes = smem + stages * stage_bytes;
    const int t0 = blockIdx.x * bn, n0 = blockIdx.y * OUT_COLS;
    const int k_begin = blockIdx.z * p.piece, k_end = min(p.K, k_begin + p.piece);
    const int chunks = (k_end - k_begin + SPL_K - 1) / SPL_K, periods = (chunks + 1) / 2;
    const uint32_t raw_full = smem_u32(bars), raw_empty = raw_full + 8 * SPL_STAGES, ready = raw_empty + 8 * SPL_STAGES, done = ready + 32, d1_full = done + 32,
                   d1_empty = d1_full + 16;
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
        for (int j = 0, s = 0, round = 0; j < chunks; j++) {
            if (!wait(raw_full + 8 * s, round, 1)) break;
            const uint8_t* src = smem + (size_t)s * stage_bytes + (weights ? 0 : SPL_W_BYTES) + row * 128;
            uint32_t h[16], m[16], l[16];
            if (weights || row < bn) {
                float4 v[8];
#pragma unroll
                for (int c = 0; c < 8; c++) v[c] = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
#pragma unroll
                for (int c = 0; c < 8; c++) split4(v[c], h + 2 * c, m + 2 * c, l + 2 * c);
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
                uint32_t v[16];
                tmem_load16(lanes + SPL_D2 + 32 * c, v);
                tmem_load_wait();
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    float a0, a1;
                    unpack_f32x2(acc[c][e], a0, a1);
                    float* to = tile + (32 * c + 16 * half + 2 * e) * TC_BM + 32 * q + lane;
                    to[0] = fabsf(a0) < INFINITY ? a0 + __uint_as_float(v[2 * e]) : a0;
                    to[TC_BM] = fabsf(a1) < INFINITY ? a1 + __uint_as_float(v[2 * e + 1]) : a1;
                }
            }
        }
    } else if (warp == 16) {
        if (elect_one()) {
            const int second = EPI == EPI_SWIGLU ? p.second_row + n0 : n0 + HALF_N;
            for (int j = 0, s = 0, round = 0; j < chunks; j++) {
                const int k = k_begin + j * SPL_K;
                if (round && !(ok = mbar_wait(raw_empty + 8 * s, (round - 1) & 1, 4))) break;
                const uint32_t dst = smem_u32(smem + (size_t)s * stage_bytes), bar = raw_full + 8 * s;
                mbar_expect_tx(bar, (uint32_t)stage_bytes);
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
                }
                mma_commit(done + 8 * (j & 3));
                if ((j & 1) || j + 1 == chunks) mma_commit(d1_full + 8 * b);
            }
            __syncwarp();
        }
    }
    if (!ok) *reinterpret_cast<volatile int*>(&gave_up) = 1;
    const int S = gridDim.z;
    __syncwarp();
    tc_fence_before();
    if (S > 1) cg::this_cluster().sync();
    else __syncthreads();
    if (warp == 17) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (!*reinterpret_cast<volatile int*>(&gave_up)) {
        const int rows = min(bn, p.M - t0);
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

template <int EPI>
static int launch(const void* X, const void* W, void* out, int M, int N, int K, float a, float b, int cols, cudaStream_t s) {
    const int w_rows = EPI == EPI_SWIGLU ? 2 * N : N, out_cols = EPI == EPI_SWIGLU ? TC_BM / 2 : TC_BM;
    SplitParams p = {};
    p.out = (float*)out, p.M = M, p.N = N, p.K = K, p.second_row = N, p.act_a = a, p.act_b = b, p.act_cols = cols;
    const int t_tiles = (M + SPL_BN - 1) / SPL_BN;
    p.bn = ((M + t_tiles - 1) / t_tiles + 15) / 16 * 16;
    const int splits = split_pieces(w_rows, K);
    p.piece = ((K + splits - 1) / splits + SPL_K - 1) / SPL_K * SPL_K;
    const int stage = SPL_W_BYTES + p.bn * 128;
    p.stages = (TC_SMEM_LIMIT - 1024 - 6 * p.bn * 128) / stage;
    if (p.stages > SPL_STAGES) p.stages = SPL_STAGES;
    const int smem = p.stages * stage + 6 * p.bn * 128 + 1024;
    CUtensorMap mw, mx;
    int st = float_map(&mw, W, w_rows, K, TC_BM / 2);
    if (st == BC_OK) st = float_map(&mx, X, M, K, p.bn);
    if (st != BC_OK) return st;
    if (cudaError_t e = bc_allow_shared<gemm_split_kernel<EPI>>(TC_SMEM_LIMIT); e != cudaSuccess) {
        bc_set_error("gemm_split: cannot raise the shared memory limit: %s", cudaGetErrorString(e));
        return (int)e;
    }
    // Token tiles fastest: the blocks that read the same weights run side by side.
    const dim3 grid((M + p.bn - 1) / p.bn, (N + out_cols - 1) / out_cols, splits);
    const cudaError_t e = splits > 1 ? bc_launch_clustered(gemm_split_kernel<EPI>, grid, dim3(SPL_THREADS), (size_t)smem, s, dim3(1, 1, splits), mw, mx, p)
                                     : bc_launch(gemm_split_kernel<EPI>, grid, dim3(SPL_THREADS), (size_t)smem, s, mw, mx, p);
    if (e != cudaSuccess) {
        bc_set_error("gemm_split: launch failed: %s", cudaGetErrorString(e));
        return (int)e;
    }
    BC_LAUNCH_STATUS();
}

// The interface of gemm_simt's float product, for what bc_gemm_split_takes.
extern "C" int bc_gemm_split_f32(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, float a, float b, int cols, cudaStream_t s) {
    switch (epilogue) {
        case EPI_STORE: return launch<EPI_STORE>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_STORE_F32: return launch<EPI_STORE_F32>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_ADD_F32: return launch<EPI_ADD_F32>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_SWIGLU: return launch<EPI_SWIGLU>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_RELU2: return launch<EPI_RELU2>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_XIELU: return launch<EPI_XIELU>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_SILU_F32: return launch<EPI_SILU_F32>(X, W, out, M, N, K, a, b, cols, s);
    }
    bc_set_error("gemm_split: unknown epilogue %d", epilogue);
    return BC_ERR_ARG;
}

// This unit's status word, its wait limit and its word of host memory: bc_gemm_split_status / _set_wait_cycles / _bind_host_word.
TC_STATUS_EXPORTS(gemm_split)
