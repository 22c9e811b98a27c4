// Matrix product on the CUDA cores: Y[m, n] = sum_k X[m, k] * W[n, k], float accumulation
// in ascending k, one fused multiply-add a term.  This is the product of the true 32-bit
// path where K is short (at most 512) or the operands are not laid out for tensor copies (the others: gemm_split.cu, by the
// matrix alone) and the checked twin of the tensor-core kernels, for bf16 operands and for those others.  Reference: the same contraction is k_matmul,
// crates/bc-infer/src/gpu/kernels.h:204-223, one warp a weight row.  An output's sum never depends on how many other rows
// share the launch: k is walked in ascending order, in one piece or in two to eight equal ones whose sums are added in
// ascending order (simt_splits, by the matrix alone), whichever of the kernels below takes the launch.
//
// Epilogues: store in the operand type; store as float (scores); add into a float buffer
// (the residual stream); SwiGLU over a weight that stacks gate rows on up rows; the square of relu; xIELU with its two
// numbers; floats whose first columns are gated by their own sigmoid.
#include <cooperative_groups.h>

#include "epilogue.cuh"
#include "mma_tiles.cuh"

namespace cg = cooperative_groups;

#define BK 16

template <class T> struct Vec4;
template <> struct Vec4<float> {
    static __device__ __forceinline__ void load(const float* p, float* o) {
        float4 v = *reinterpret_cast<const float4*>(p);
        o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
    }
};
template <> struct Vec4<bf16> {
    static __device__ __forceinline__ void load(const bf16* p, float* o) {
        uint2 v = *reinterpret_cast<const uint2*>(p);
        o[0] = __uint_as_float(v.x << 16); o[1] = __uint_as_float(v.x & 0xffff0000u);
        o[2] = __uint_as_float(v.y << 16); o[3] = __uint_as_float(v.y & 0xffff0000u);
    }
};

// The pieces that a sum over K is added up in, for a product with `cols` weight rows: more than one where the tiles of few rows would leave
// SMs idle and K is long enough (a [2048, 8192] matrix is 16 tiles of 128 columns: in one piece 80 blocks for 300 rows).
__host__ __device__ constexpr int simt_splits(int cols, int K) {
    int s = 1;
    while ((cols + 127) / 128 * s < 96 && s < 8 && K / (2 * s) >= 512) s *= 2;
    return s;
}
// k a piece: a multiple of BK.
__host__ __device__ constexpr int simt_piece(int K, int splits) { return ((K + splits - 1) / splits + BK - 1) / BK * BK; }

// A tile of BM rows by 128 weight rows a block (SwiGLU: 64 gate rows and their 64 up rows), 128 threads, TM x TN sums each, two to an
// instruction (fma.rn.f32x2: the roundings of fmaf).  The next sixteen k are on their way to registers while these are multiplied, into the
// other of two buffers.  BM 64: 8 x 8 a thread, 64 bytes of shared memory for its 64 multiply-adds a k; BM 16 (few rows): 4 x 4, and what counts is that
// the weights stream.  With several pieces of K the blocks of a tile are one cluster and add up through one another's shared memory.
// (64 x 64 tiles, 4 x 4 a thread, one buffer: 720 + 763 us for 300 rows of a feed-forward of 2,048 x 8,192, 20 TFLOP/s; these 557 + 311 us.  Such
// float products go to gemm_split.cu now.)
#define SIMT_COLS 128
template <class T, int EPI, bool VEC, int BM>
__global__ void __launch_bounds__(128) gemm_simt_kernel(const T* X, const T* __restrict__ W, T* out_act, float* out_f32, int M, int N, int K, int piece, float act_a,
                                                        float act_b, int act_cols) {
    constexpr int TM = BM == 64 ? 8 : 4, TN = BM == 64 ? 8 : 4, TX = SIMT_COLS / TN;
    constexpr int HALF_N = SIMT_COLS / 2, A_ROW = BM + 4, B_ROW = SIMT_COLS + 4;
    constexpr int A_LOADS = BM * BK / 4 / 128 ? BM * BK / 4 / 128 : 1, B_LOADS = SIMT_COLS * BK / 4 / 128;
    __shared__ __align__(16) float tiles[2 * BK * (A_ROW + B_ROW) > BM * SIMT_COLS ? 2 * BK * (A_ROW + B_ROW) : BM * SIMT_COLS];
    float *As = tiles, *Bs = tiles + 2 * BK * A_ROW;
    pdl_launch_dependents();
    pdl_wait();
    PDL_FRESH(X); PDL_FRESH(W); PDL_FRESH(out_act); PDL_FRESH(out_f32);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * (EPI == EPI_SWIGLU ? HALF_N : SIMT_COLS);
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int k_begin = blockIdx.z * piece, k_end = min(K, k_begin + piece);
    // The weight row of the tile's column c, or -1.
    auto w_row = [&](int c) {
        if (EPI == EPI_SWIGLU) {
            const int n = n0 + (c & (HALF_N - 1));
            return n < N ? (c < HALF_N ? n : N + n) : -1;
        }
        return n0 + c < N ? n0 + c : -1;
    };
    float a_next[A_LOADS][4], b_next[B_LOADS][4];
    auto fetch4 = [&](const T* base, int row, int k, float* v) {
        v[0] = v[1] = v[2] = v[3] = 0.0f;
        if (row < 0) return;
        const T* p = base + (size_t)row * K + k;
        if (VEC && k + 3 < k_end) {
            Vec4<T>::load(p, v);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (k + j < k_end) v[j] = to_f32(p[j]);
        }
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < A_LOADS; i++) {
            const int at = threadIdx.x + 128 * i, r = at >> 2;
            if (r < BM) fetch4(X, m0 + r < M ? m0 + r : -1, k0 + (at & 3) * 4, a_next[i]);
        }
#pragma unroll
        for (int i = 0; i < B_LOADS; i++) {
            const int at = threadIdx.x + 128 * i;
            fetch4(W, w_row(at >> 2), k0 + (at & 3) * 4, b_next[i]);
        }
    };
    auto put = [&](int buffer) {
#pragma unroll
        for (int i = 0; i < A_LOADS; i++) {
            const int at = threadIdx.x + 128 * i, r = at >> 2, kq = (at & 3) * 4;
            if (r < BM)
#pragma unroll
                for (int j = 0; j < 4; j++) As[(buffer * BK + kq + j) * A_ROW + r] = a_next[i][j];
        }
#pragma unroll
        for (int i = 0; i < B_LOADS; i++) {
            const int at = threadIdx.x + 128 * i, c = at >> 2, kq = (at & 3) * 4;
#pragma unroll
            for (int j = 0; j < 4; j++) Bs[(buffer * BK + kq + j) * B_ROW + c] = b_next[i][j];
        }
    };
    uint64_t acc[TM][TN / 2] = {};
    if (k_begin < k_end) {
        fetch(k_begin);
        put(0);
    }
    __syncthreads();
    int buffer = 0;
    for (int k0 = k_begin; k0 < k_end; k0 += BK, buffer ^= 1) {
        const bool more = k0 + BK < k_end;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; k++) {
            const float *ar = As + (buffer * BK + k) * A_ROW + 4 * ty, *br = Bs + (buffer * BK + k) * B_ROW + 4 * tx;
            float a[TM];
            uint64_t b[TN / 2];
#pragma unroll
            for (int i = 0; i < TM / 4; i++) {
                const float4 v = *reinterpret_cast<const float4*>(ar + i * (BM / 2));
                a[4 * i] = v.x, a[4 * i + 1] = v.y, a[4 * i + 2] = v.z, a[4 * i + 3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < TN / 4; j++) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(br + j * HALF_N);
                b[2 * j] = v.x, b[2 * j + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < TM; i++) {
                const uint64_t aa = pack_f32x2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; j++) acc[i][j] = fma_f32x2(aa, b[j], acc[i][j]);
            }
        }
        if (more) put(buffer ^ 1);
        __syncthreads();
    }
    // Sum (i, j) of this thread: the tile's row and column.
    auto row_at = [&](int i) { return TM == 8 ? (i >> 2) * (BM / 2) + 4 * ty + (i & 3) : 4 * ty + i; };
    auto col_at = [&](int j) { return TN == 8 ? (j >> 2) * HALF_N + 4 * tx + (j & 3) : 4 * tx + j; };
    if (gridDim.z == 1 && !(EPI == EPI_SWIGLU && TN == 4)) {
#pragma unroll
        for (int i = 0; i < TM; i++) {
            const int m = m0 + row_at(i);
            float v[TN];
#pragma unroll
            for (int j = 0; j < TN / 2; j++) unpack_f32x2(acc[i][j], v[2 * j], v[2 * j + 1]);
            if (m >= M) continue;
#pragma unroll
            for (int j = 0; j < (EPI == EPI_SWIGLU ? TN / 2 : TN); j++) {
                const int n = n0 + col_at(j);
                if (n < N) simt_emit<T, EPI>(out_act, out_f32, m, n, N, v[j], EPI == EPI_SWIGLU ? v[(j + TN / 2) % TN] : 0.0f, act_a, act_b, act_cols);
            }
        }
        return;
    }
    // The tile through shared memory: several pieces of K, or gate and up sums that lie with two threads.
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++) *reinterpret_cast<uint64_t*>(tiles + row_at(i) * SIMT_COLS + col_at(2 * j)) = acc[i][j];
    const int S = gridDim.z;
    if (S > 1) cg::this_cluster().sync();
    else __syncthreads();
    constexpr int OUT_COLS = EPI == EPI_SWIGLU ? HALF_N : SIMT_COLS;
    for (int e = blockIdx.z * 128 + threadIdx.x; e < BM * OUT_COLS; e += S * 128) {
        const int r = e / OUT_COLS, c = e % OUT_COLS, m = m0 + r, n = n0 + c;
        if (m >= M || n >= N) continue;
        float v = 0.0f, u = 0.0f;
        for (int z = 0; z < S; z++) {
            const float* theirs = S > 1 ? cg::this_cluster().map_shared_rank(tiles, z) : tiles;
            v = z ? v + theirs[r * SIMT_COLS + c] : theirs[r * SIMT_COLS + c];
            if (EPI == EPI_SWIGLU) u = z ? u + theirs[r * SIMT_COLS + HALF_N + c] : theirs[r * SIMT_COLS + HALF_N + c];
        }
        simt_emit<T, EPI>(out_act, out_f32, m, n, N, v, u, act_a, act_b, act_cols);
    }
    if (S > 1) cg::this_cluster().sync();      // no block leaves while a peer still reads its shared memory
}

// Short K (at most 512) and few outputs, where a launch is all latency: a lane a weight row, a warp four rows of X.  All of the block's weights
// and rows are asked for at once, into shared memory, and summed up from there; what
// the result is added to is asked for with them.  (A whole 64 x 64 tile a block behind two barriers every sixteen k: 8 to 10 us a launch at
// K 64 to 176; straight from global memory 8; now 4.6 to 5.)
#define SHORT_K 512
template <class T, int EPI, bool VEC>
__global__ void __launch_bounds__(128) gemm_simt_short_kernel(const T* X, const T* __restrict__ W, T* out_act, float* out_f32, int M, int N, int K, int k_row, float act_a,
                                                              float act_b, int act_cols) {
    extern __shared__ __align__(16) float short_smem[];
    constexpr int MATS = EPI == EPI_SWIGLU ? 2 : 1;
    float *ws = short_smem, *xs = ws + MATS * 32 * k_row;       // [32 or 64][k_row] weights, [16][k_row] rows; k_row: K and a gap, so that 16-byte reads of eight rows meet no bank twice
    const int n0 = blockIdx.x * 32, r0 = blockIdx.y * 16, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_launch_dependents();
    auto stage = [&](float* to, const T* base, int row0, int count, int rows) {
        if (VEC) {
            const int quads = K / 4;
            for (int i = threadIdx.x; i < count * quads; i += 128) {
                const int r = i / quads, c = 4 * (i - r * quads);
                float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (row0 + r < rows) Vec4<T>::load(base + (size_t)(row0 + r) * K + c, v);
                *reinterpret_cast<float4*>(to + r * k_row + c) = make_float4(v[0], v[1], v[2], v[3]);
            }
        } else {
            for (int i = threadIdx.x; i < count * K; i += 128) {
                const int r = i / K, c = i - r * K;
                to[r * k_row + c] = row0 + r < rows ? to_f32(base[(size_t)(row0 + r) * K + c]) : 0.0f;
            }
        }
    };
    // The weights too are read behind the wait: a caller's w may be what the kernel before has just written.
    pdl_wait();
    PDL_FRESH(X); PDL_FRESH(W); PDL_FRESH(out_act); PDL_FRESH(out_f32);
    stage(ws, W, n0, 32, N);
    if (EPI == EPI_SWIGLU) stage(ws + 32 * k_row, W + (size_t)N * K, n0, 32, N);
    stage(xs, X, r0, min(16, M - r0), M);
    const int n = n0 + lane, m0 = r0 + 4 * warp;
    float old[4] = {};
    if (EPI == EPI_ADD_F32) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (n < N && m0 + i < M) old[i] = out_f32[(size_t)(m0 + i) * N + n];
    }
    __syncthreads();
    if (n >= N || m0 >= M) return;
    const float *w = ws + lane * k_row, *w2 = EPI == EPI_SWIGLU ? w + 32 * k_row : w;
    const float* x[4];
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = xs + min(4 * warp + i, M - 1 - r0) * k_row;
    float v[4] = {}, u[4] = {};
    const int k4 = K & ~3;
#pragma unroll 4
    for (int k = 0; k < k4; k += 4) {
        const float4 b = *reinterpret_cast<const float4*>(w + k), c = *reinterpret_cast<const float4*>(w2 + k);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 a = *reinterpret_cast<const float4*>(x[i] + k);
            v[i] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, v[i]))));
            if (EPI == EPI_SWIGLU) u[i] = fmaf(a.w, c.w, fmaf(a.z, c.z, fmaf(a.y, c.y, fmaf(a.x, c.x, u[i]))));
        }
    }
    for (int k = k4; k < K; k++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            v[i] = fmaf(x[i][k], w[k], v[i]);
            if (EPI == EPI_SWIGLU) u[i] = fmaf(x[i][k], w2[k], u[i]);
        }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (m0 + i >= M) break;
        if (EPI == EPI_ADD_F32) out_f32[(size_t)(m0 + i) * N + n] = old[i] + v[i];
        else simt_emit<T, EPI>(out_act, out_f32, m0 + i, n, N, v[i], u[i], act_a, act_b, act_cols);
    }
}

template <class T, int EPI, bool VEC>
static cudaError_t launch_vec(const T* X, const T* W, T* oa, float* of, int M, int N, int K, float a, float b, int cols, cudaStream_t s) {
    // Short sums of few outputs.  Up to 262,144 of them the short kernel is the quicker or as quick: 128 x 1,024 at K 512 33 against 43 us in tiles,
    // 512 x 256 at K 176 16 against 20, 2,048 x 128 at K 64 10 against 12 (caches cold); past that the tiles: 300 x 1,000 at K 256 27 against 29,
    // 1,000 x 1,000 at K 64 12 against 14.
    if (K <= SHORT_K && (long long)M * N <= 1 << 18) {
        const int k_row = (K + 7) / 8 * 8 + 4;                    // an odd number of 16-byte pieces
        const size_t smem = (size_t)((EPI == EPI_SWIGLU ? 64 : 32) + 16) * k_row * sizeof(float);      // at most 165 KB
        if (smem > 48 * 1024)
            if (cudaError_t e = bc_allow_shared<gemm_simt_short_kernel<T, EPI, VEC>>(168 * 1024); e != cudaSuccess) return e;
        return bc_launch(gemm_simt_short_kernel<T, EPI, VEC>, dim3((N + 31) / 32, (M + 15) / 16), dim3(128), smem, s, X, W, oa, of, M, N, K, k_row, a, b, cols);
    }
    const int splits = simt_splits(EPI == EPI_SWIGLU ? 2 * N : N, K), piece = simt_piece(K, splits);
    const int out_cols = EPI == EPI_SWIGLU ? SIMT_COLS / 2 : SIMT_COLS;
    // Tiles of 16 rows for few rows, and as long as these are 8/3 blocks an SM at most: 48 rows of [2048, 8192] (384 blocks) 90 us against 125 in tiles of
    // 64, 128 rows of [512, 1024] (64 blocks) 37 against 53; 96 rows of [2048, 2048] (384) 49 in either; 64 rows of [8192, 2048] (512) 110 against 92.
    const int cols_grid = (N + out_cols - 1) / out_cols;
    const int bm = M <= 32 || (long long)cols_grid * splits * ((M + 15) / 16) * 3 <= 8 * bc_sm_count() ? 16 : 64;
    const dim3 grid(cols_grid, (M + bm - 1) / bm, splits);
    auto go = [&](auto kernel) {
        return splits > 1 ? bc_launch_clustered(kernel, grid, dim3(128), 0, s, dim3(1, 1, splits), X, W, oa, of, M, N, K, piece, a, b, cols)
                          : bc_launch(kernel, grid, dim3(128), 0, s, X, W, oa, of, M, N, K, piece, a, b, cols);
    };
    return bm == 16 ? go(gemm_simt_kernel<T, EPI, VEC, 16>) : go(gemm_simt_kernel<T, EPI, VEC, 64>);
}

template <class T, int EPI>
static int launch(const void* X, const void* W, void* out, int M, int N, int K, float a, float b, int cols, cudaStream_t s) {
    const bool vec = K % 4 == 0 && ((uintptr_t)X % 16 == 0) && ((uintptr_t)W % 16 == 0);
    T* oa = (EPI == EPI_STORE || EPI == EPI_SWIGLU || EPI == EPI_RELU2 || EPI == EPI_XIELU) ? (T*)out : nullptr;
    float* of = (EPI == EPI_STORE_F32 || EPI == EPI_ADD_F32 || EPI == EPI_SILU_F32) ? (float*)out : nullptr;
    const cudaError_t e = vec ? launch_vec<T, EPI, true>((const T*)X, (const T*)W, oa, of, M, N, K, a, b, cols, s)
                              : launch_vec<T, EPI, false>((const T*)X, (const T*)W, oa, of, M, N, K, a, b, cols, s);
    if (e != cudaSuccess) {
        bc_set_error("gemm_simt: %s", cudaGetErrorString(e));
        return (int)e;
    }
    BC_LAUNCH_STATUS();
}

// X [M, K] and W [N, K] (for SwiGLU: W [2N, K], gate rows then up rows) in the operand
// type; `out` is [M, N] in the operand type (store, SwiGLU) or float (store_f32, add_f32).
template <class T>
static int dispatch(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, float a, float b, int cols, cudaStream_t s) {
    BC_CHECK_ARG(M >= 0 && N > 0 && K > 0, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
    BC_CHECK_ARG((M + 63) / 64 <= 65535, "gemm_simt: %d rows are more than 65535 tiles of 64", M);
    if (M == 0) return BC_OK;
    switch (epilogue) {
        case EPI_STORE: return launch<T, EPI_STORE>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_STORE_F32: return launch<T, EPI_STORE_F32>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_ADD_F32: return launch<T, EPI_ADD_F32>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_SWIGLU: return launch<T, EPI_SWIGLU>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_RELU2: return launch<T, EPI_RELU2>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_XIELU: return launch<T, EPI_XIELU>(X, W, out, M, N, K, a, b, cols, s);
        case EPI_SILU_F32: return launch<T, EPI_SILU_F32>(X, W, out, M, N, K, a, b, cols, s);
    }
    bc_set_error("gemm_simt: unknown epilogue %d", epilogue);
    return BC_ERR_ARG;
}

extern "C" int bc_gemm_simt_f32(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, cudaStream_t s) {
    BC_CHECK_ARG(epilogue != EPI_XIELU && epilogue != EPI_SILU_F32, "gemm_simt: epilogue %d comes with numbers of its own", epilogue);
    return dispatch<float>(X, W, out, M, N, K, epilogue, 0.0f, 0.0f, 0, s);
}
extern "C" int bc_gemm_simt_bf16(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, cudaStream_t s) {
    BC_CHECK_ARG(epilogue != EPI_XIELU && epilogue != EPI_SILU_F32, "gemm_simt: epilogue %d comes with numbers of its own", epilogue);
    return dispatch<bf16>(X, W, out, M, N, K, epilogue, 0.0f, 0.0f, 0, s);
}
// The epilogues with numbers of their own: EPI_XIELU (a, b) and EPI_SILU_F32 (cols).
extern "C" int bc_gemm_simt_act_f32(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, float a, float b, int cols, cudaStream_t s) {
    return dispatch<float>(X, W, out, M, N, K, epilogue, a, b, cols, s);
}
extern "C" int bc_gemm_simt_act_bf16(const void* X, const void* W, void* out, int M, int N, int K, int epilogue, float a, float b, int cols, cudaStream_t s) {
    return dispatch<bf16>(X, W, out, M, N, K, epilogue, a, b, cols, s);
}
