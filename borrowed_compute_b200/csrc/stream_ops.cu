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

// A block takes 1,024 neighbouring columns of eight rows; four columns a thread, sixteen bytes a move, the bias read once (an element a thread
// and a 64-bit remainder each: 30 us for 2,048 x 4,096 floats, against 10 us of bytes).
#define BIAS_ROWS 8
__global__ void __launch_bounds__(256) add_bias_kernel(float* x, const float* __restrict__ b, int rows, int E) {
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(x);
    const int c = blockIdx.x * 1024 + 4 * threadIdx.x, row0 = blockIdx.y * BIAS_ROWS;
    if (c >= E) return;
    if (E % 4 == 0 && ((uintptr_t)x | (uintptr_t)b) % 16 == 0) {
        const float4 v = *reinterpret_cast<const float4*>(b + c);
        float4 y[BIAS_ROWS];
#pragma unroll
        for (int r = 0; r < BIAS_ROWS; r++)
            if (row0 + r < rows) y[r] = *reinterpret_cast<const float4*>(x + (size_t)(row0 + r) * E + c);
#pragma unroll
        for (int r = 0; r < BIAS_ROWS; r++)
            if (row0 + r < rows) *reinterpret_cast<float4*>(x + (size_t)(row0 + r) * E + c) = make_float4(y[r].x + v.x, y[r].y + v.y, y[r].z + v.z, y[r].w + v.w);
        return;
    }
    for (int r = row0; r < min(rows, row0 + BIAS_ROWS); r++)
        for (int e = 0; e < 4 && c + e < E; e++) x[(size_t)r * E + c + e] += b[c + e];
}

// x: [rows, E] float; b: [E] float.
extern "C" int bc_add_bias_f32(float* x, const float* b, int rows, int E, cudaStream_t s) {
    BC_CHECK_ARG(rows >= 0 && E > 0, "add_bias: bad sizes rows=%d E=%d", rows, E);
    // More rows than a grid's second dimension holds go in turns.
    for (int at = 0; at < rows; at += 65535 * BIAS_ROWS) {
        const int n = rows - at < 65535 * BIAS_ROWS ? rows - at : 65535 * BIAS_ROWS;
        bc_launch(add_bias_kernel, dim3((E + 1023) / 1024, (n + BIAS_ROWS - 1) / BIAS_ROWS), dim3(256), 0, s, x + (size_t)at * E, b, n, E);
    }
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
