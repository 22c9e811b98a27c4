// Small kernels on the float residual stream and on scores.
//
//   softcap:  s <- cap * tanh(s / cap), in place, on float scores
//   scale:    s <- factor * s, in place, on float scores
//   add_bias: x[r] += b, on float rows (the bias of a product that adds into them)
//   reentry:  for a stretch of layers that runs several times: cat[r] = [x[r]; x0[r]] in the activation
//             type (the operand of the product that mixes the stream with the embedding's output) and
//             x[r] <- step (the vector of the pass), so that the product's epilogue adds onto it
#include "common.cuh"

__global__ void softcap_kernel(float* __restrict__ s, size_t n, float cap) {
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(s);
    const float inv = 1.0f / cap;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) s[i] = cap * tanhf(s[i] * inv);
}

extern "C" int bc_softcap_f32(float* scores, long long n, float cap, cudaStream_t s) {
    BC_CHECK_ARG(n >= 0 && cap > 0.0f, "softcap: bad sizes n=%lld cap=%g", n, (double)cap);
    if (n == 0) return BC_OK;
    const int threads = 256;
    const long long blocks = (n + threads - 1) / threads;
    bc_launch(softcap_kernel, dim3((unsigned)(blocks < 65535 * 16 ? blocks : 65535 * 16)), dim3(threads), 0, s, scores, (size_t)n, cap);
    BC_LAUNCH_STATUS();
}

__global__ void scale_kernel(float* __restrict__ s, size_t n, float factor) {
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(s);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) s[i] *= factor;
}

extern "C" int bc_scale_f32(float* scores, long long n, float factor, cudaStream_t s) {
    BC_CHECK_ARG(n >= 0, "scale: bad size n=%lld", n);
    if (n == 0) return BC_OK;
    const int threads = 256;
    const long long blocks = (n + threads - 1) / threads;
    bc_launch(scale_kernel, dim3((unsigned)(blocks < 65535 * 16 ? blocks : 65535 * 16)), dim3(threads), 0, s, scores, (size_t)n, factor);
    BC_LAUNCH_STATUS();
}

// A block's 256 threads lie `across` (a power of two) to a row's columns, V columns a thread, and take BIAS_ROWS rows each, all asked for together;
// the bias is read once.  V = 4 (sixteen bytes a move) where the rows allow it.  (An element a thread and a 64-bit remainder each: 30 us
// for 2,048 x 4,096 floats, 45 cold with the launch; now 23 so.  All 256 threads along one row, four columns each whatever the alignment, left narrow rows
// with few threads and let unaligned ones touch every line four times: with the launch 63 us for 500,000 x 16 and 33 for 2,048 x 1,023, an
// element a thread 41 and 22, now 23 and 17.)
#define BIAS_ROWS 8
template <int V>
__global__ void __launch_bounds__(256) add_bias_kernel(float* x, const float* __restrict__ b, int rows, int E, int across, int col_blocks) {
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(x); PDL_FRESH(b);
    const int down = 256 / across, ty = threadIdx.x / across;
    const unsigned row_block = blockIdx.x / col_blocks;
    const long long c = (long long)(blockIdx.x - row_block * col_blocks) * across * V + V * (threadIdx.x % across), row0 = (long long)row_block * down * BIAS_ROWS + ty;
    if (c >= E) return;
    float v[V], y[BIAS_ROWS][V];
    auto load = [](const float* from, float* to) {
        if constexpr (V == 4) {
            const float4 u = *reinterpret_cast<const float4*>(from);
            to[0] = u.x, to[1] = u.y, to[2] = u.z, to[3] = u.w;
        } else to[0] = *from;
    };
    load(b + c, v);
#pragma unroll
    for (int r = 0; r < BIAS_ROWS; r++)
        if (row0 + r * down < rows) load(x + (size_t)(row0 + r * down) * E + c, y[r]);
#pragma unroll
    for (int r = 0; r < BIAS_ROWS; r++)
        if (row0 + r * down < rows) {
            float* to = x + (size_t)(row0 + r * down) * E + c;
            if constexpr (V == 4) *reinterpret_cast<float4*>(to) = make_float4(y[r][0] + v[0], y[r][1] + v[1], y[r][2] + v[2], y[r][3] + v[3]);
            else *to = y[r][0] + v[0];
        }
}

// x: [rows, E] float; b: [E] float.
extern "C" int bc_add_bias_f32(float* x, const float* b, int rows, int E, cudaStream_t s) {
    BC_CHECK_ARG(rows >= 0 && E > 0, "add_bias: bad sizes rows=%d E=%d", rows, E);
    if (rows == 0) return BC_OK;
    const int V = E % 4 == 0 && ((uintptr_t)x | (uintptr_t)b) % 16 == 0 ? 4 : 1;
    int across = 1;
    while (across < 256 && across * V < E) across *= 2;
    const long long rows_a_block = (long long)BIAS_ROWS * (256 / across), col_blocks = ((long long)E + across * V - 1) / (across * V);
    const long long blocks = (rows + rows_a_block - 1) / rows_a_block * col_blocks;       // (a block for every 2,048 floats or so: memory ends long before a grid does)
    BC_CHECK_ARG(blocks <= 2147483647ll, "add_bias: %d rows of %d are too many", rows, E);
    bc_launch(V == 4 ? add_bias_kernel<4> : add_bias_kernel<1>, dim3((unsigned)blocks), dim3(256), 0, s, x, b, rows, E, across, (int)col_blocks);
    BC_LAUNCH_STATUS();
}

template <class T>
__global__ void reentry_kernel(float* __restrict__ x, const float* __restrict__ x0, const float* __restrict__ step, T* __restrict__ cat, int E) {
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(x); PDL_FRESH(x0);
    const int r = blockIdx.x;
    float* xr = x + (size_t)r * E;
    const float* x0r = x0 + (size_t)r * E;
    T* out = cat + (size_t)r * 2 * E;
    for (int c = threadIdx.x; c < E; c += blockDim.x) {
        out[c] = from_f32<T>(xr[c]);
        out[E + c] = from_f32<T>(x0r[c]);
        xr[c] = step[c];
    }
}

template <class T>
static int reentry(float* x, const float* x0, const float* step, void* cat, int rows, int E, cudaStream_t s) {
    BC_CHECK_ARG(rows >= 0 && E > 0, "reentry: bad sizes rows=%d E=%d", rows, E);
    if (rows == 0) return BC_OK;
    bc_launch(reentry_kernel<T>, dim3(rows), dim3(E >= 1024 ? 256 : 128), 0, s, x, x0, step, (T*)cat, E);
    BC_LAUNCH_STATUS();
}
// x, x0: [rows, E] float; step: [E] float; cat: [rows, 2 E] of the activation type.
extern "C" int bc_reentry_f32(float* x, const float* x0, const float* step, void* cat, int rows, int E, cudaStream_t s) {
    return reentry<float>(x, x0, step, cat, rows, E, s);
}
extern "C" int bc_reentry_bf16(float* x, const float* x0, const float* step, void* cat, int rows, int E, cudaStream_t s) {
    return reentry<bf16>(x, x0, step, cat, rows, E, s);
}
