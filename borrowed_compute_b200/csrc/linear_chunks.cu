// Gated linear attention on prompts, sixteen rows at a time (chunks.cuh):
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T        o_t = f S_t^T q_t,        a = sigmoid(z)^(1/tau), z = W_2 inner + b
//
// With A(s, t) the product of the decays of rows s + 1 .. t of a chunk: X0 = q_t A(-1, t), Z0 = k_s A(s, last), tot = A(-1, last) and
// G_ts = sum_i q_ti k_si A(s, t)_i for s <= t; f multiplies the finished sums.  No decay is ever divided by, so decays of zero are as good as any.
// Float throughout, but for the products of decays in X0, Z0 and tot: those are double and rounded once (a state that decays slowly is
// multiplied by tot again and again).
// Sequences of 400, 1,100 and 1,800 rows, 16 heads of 128 x 256: 60 + 315 us, where the decays and the scan row by row take 52 + 764.  The scan
// in chunks is bound by the longest sequence's 113 chunks, one after another.  Distance from 64-bit sums: 0.94 to 1.01 times the row scan's
// (outputs) and 0.93 to 0.99 (state); with float products of decays and one running sum 1.00 to 1.12 times.
#include "chunks.cuh"

#define GLC_PAIRS (CHUNK * (CHUNK + 1) / 2)      // 136
// The number of the pair (s, t), s <= t: all t of s = 0 first.
__host__ __device__ constexpr int glc_pair(int s, int t) { return s * CHUNK - s * (s - 1) / 2 + (t - s); }
// f(I), f(I + 1) .. f(15), each with its number as a constant: registers stay registers whatever the compiler thinks of the loop's length.
template <int I, class F> __device__ __forceinline__ void glc_each(F&& f) {
    if constexpr (I < CHUNK) {
        f(std::integral_constant<int, I>());
        glc_each<I + 1>(f);
    }
}

// A block takes the chunk at a place, of one head, a thread a key channel: decays as gla_decay_kernel works them out, then the 136 products of a
// pair of rows, each a running product of k_s with the decays after it.  The sums over channels: 32 pairs at a time are halved
// among a warp's lanes, the warps' sums meet in shared memory.
template <int D>
__global__ void __launch_bounds__(D)
gla_chunks_kernel(const ChunkSpan span, const float* proj, int stride, int q_at, int k_at, int inner_at, const float* __restrict__ w2t, const float* __restrict__ b,
                  int rank, const int* __restrict__ seq_rows, const int* __restrict__ seq_slot, float* __restrict__ pack, int H, int N, float inv_tau, int seqs,
                  int n_slots) {
    constexpr int WARPS = D / 32, PACK = chunk_pack_floats(D, false);
    extern __shared__ __align__(16) float inner[];           // [rank][16]
    __shared__ float part[WARPS][160];
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(proj);
    const int h = blockIdx.y;
    const ChunkAt at = chunk_at(span, blockIdx.x, seq_rows, seq_slot, seqs, n_slots);
    const int rows = at.rows;
    if (rows <= 0) return;
    const float* p = proj + (size_t)at.row * stride;
    for (int i = threadIdx.x; i < rank * CHUNK; i += D) {
        const int t = i / rank, j = i - t * rank;
        inner[j * CHUNK + t] = t < rows ? p[(size_t)t * stride + inner_at + j] : 0.0f;
    }
    const int n = threadIdx.x;
    const bool mine = n < N;
    const int col = h * N + (mine ? n : 0);
    float q[CHUNK], k[CHUNK], a[CHUNK];
#pragma unroll
    for (int t = 0; t < CHUNK; t++) {
        const bool ok = mine && t < rows;
        q[t] = ok ? p[(size_t)t * stride + q_at + col] : 0.0f;
        k[t] = ok ? p[(size_t)t * stride + k_at + col] : 0.0f;
        a[t] = b[col];
    }
    __syncthreads();
#pragma unroll 4
    for (int j = 0; j < rank; j++) {
        const float w = w2t[(size_t)j * H * N + col];
#pragma unroll
        for (int t = 0; t < CHUNK; t++) a[t] = fmaf(w, inner[j * CHUNK + t], a[t]);
    }
#pragma unroll
    for (int t = 0; t < CHUNK; t++) {
        const float m = -a[t];                                       // softplus(m) = max(m, 0) + log1p(exp(-|m|))
        const float sp = fmaxf(m, 0.0f) + log1pf(expf(-fabsf(m)));
        a[t] = mine && t < rows ? expf(-sp * inv_tau) : 1.0f;
    }
    float* dst = pack + ((size_t)blockIdx.x * H + h) * PACK;
    double run = 1.0;
#pragma unroll
    for (int t = 0; t < CHUNK; t++) {
        run *= a[t];
        dst[t * D + n] = (float)(q[t] * run);
    }
    dst[2 * CHUNK * D + CHUNK * CHUNK_G + n] = (float)run;
    run = 1.0;
#pragma unroll
    for (int t = CHUNK - 1; t >= 0; t--) {
        dst[(CHUNK + t) * D + n] = (float)(k[t] * run);
        run *= a[t];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float buf[32];
    // Lane L keeps the sum of pair 32 g + L.
    auto reduce = [&](int g) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < o; i++) {
                const float keep = up ? buf[i + o] : buf[i], send = up ? buf[i] : buf[i + o];
                buf[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        part[warp][32 * g + lane] = buf[0];
    };
    glc_each<0>([&](auto S) {
        constexpr int s = decltype(S)::value;
        float x = k[s];
        glc_each<s>([&](auto T) {
            constexpr int t = decltype(T)::value, number = glc_pair(s, t);
            if (t > s) x *= a[t];
            buf[number & 31] = q[t] * x;
            if ((number & 31) == 31) reduce(number / 32);
        });
    });
#pragma unroll
    for (int i = GLC_PAIRS & 31; i < 32; i++) buf[i] = 0.0f;
    reduce(GLC_PAIRS / 32);
    __syncthreads();
    for (int i = threadIdx.x; i < CHUNK * CHUNK_G; i += D) {
        const int t = i / CHUNK_G, s = i - t * CHUNK_G;
        float sum = 0.0f;
        if (s <= t) {
            const int number = glc_pair(s, t);
#pragma unroll
            for (int w = 0; w < WARPS; w++) sum += part[w][number];
        }
        dst[2 * CHUNK * D + i] = sum;
    }
}

template <int D>
static int gla_chunked(const float* proj, int stride, int q_at, int k_at, int v_at, int inner_at, const float* w2t, const float* b, int rank, float inv_tau, float f,
                       float* pack, long long pack_floats, float* state, const int* seq_rows, const int* seq_slot, float* out, int rows, int seqs, int max_new, int min_rows, int H, int N,
                       int P, int n_slots, int write_state, cudaStream_t s) {
    if (cudaError_t e = bc_allow_shared<gla_chunks_kernel<D>>(64 * 1024); e != cudaSuccess) {
        bc_set_error("gla_chunked: %s", cudaGetErrorString(e));
        return (int)e;
    }
    const cudaError_t e = chunk_step(
        pack_floats / ((long long)H * chunk_pack_floats(D, false)), rows, seqs, max_new, min_rows,
        [&](const ChunkSpan& span, long long places) {
            return bc_launch(gla_chunks_kernel<D>, dim3((unsigned)places, H), dim3(D), (size_t)rank * CHUNK * sizeof(float), s, span, proj, stride, q_at, k_at, inner_at,
                             w2t, b, rank, seq_rows, seq_slot, pack, H, N, inv_tau, seqs, n_slots);
        },
        [&](const ChunkSpan& span) {
            return chunk_scan_launch<D / 32, false>(span, pack, proj + v_at, stride, state, seq_rows, seq_slot, out, rows, max_new, seqs, H, N, P, n_slots, write_state, f, s);
        });
    if (e != cudaSuccess) {
        bc_set_error("gla_chunked: %s", cudaGetErrorString(e));
        return (int)e;
    }
    BC_LAUNCH_STATUS();
}

static int glc_width(int N) { return N <= 64 ? 64 : N <= 128 ? 128 : 256; }

// Whether gated linear attention of N key and P value channels a head runs in chunks, and the floats of scratch that `rows` rows of `seqs`
// sequences take (0: it does not), of which those of fewer than min_rows rows are left alone.
extern "C" long long bc_gla_chunked_scratch(int rows, int seqs, int min_rows, int H, int N, int P, int rank, int write_state) {
    if (N <= 0 || N > 256 || N % 4 || P <= 0 || P % 4 || rank <= 0 || rank > 1024 || H <= 0 || H > 65535 || seqs <= 0 || seqs > 65535) return 0;
    const int pack = chunk_pack_floats(glc_width(N), false);
    return chunk_capacity(rows, seqs, min_rows, H, pack, write_state) * H * pack;
}

// proj: [rows, stride] float with q and k (N values a head), v (P values a head) and the decay's inner vector (`rank` values) at columns q_at, k_at,
// v_at and inner_at; w2t: [rank, H N]; b: [H N]; pack: scratch of pack_floats floats, bc_gla_chunked_scratch of them for the fewest launches; state: [slots, H, P, N]; out: [rows, H P].  Sequence i
// owns rows seq_rows[i] .. seq_rows[i + 1], at most max_new, and lives in slot seq_slot[i] (negative, or fewer than min_rows rows: skipped, its rows
// of out untouched).
extern "C" int bc_gla_chunked(const float* proj, int stride, int q_at, int k_at, int v_at, int inner_at, const float* w2t, const float* b, int rank, float tau,
                              float f, float* pack, long long pack_floats, float* state, const int* seq_rows, const int* seq_slot, float* out, int rows, int seqs, int max_new, int min_rows, int H,
                              int N, int P, int n_slots, int write_state, cudaStream_t s) {
    BC_CHECK_ARG(rows >= 0 && seqs >= 0 && max_new >= 0 && tau > 0.0f, "gla_chunked: bad sizes rows=%d seqs=%d max_new=%d tau=%g", rows, seqs, max_new, (double)tau);
    if (rows == 0 || seqs == 0 || max_new == 0) return BC_OK;
    BC_CHECK_ARG(bc_gla_chunked_scratch(rows, seqs, min_rows, H, N, P, rank, write_state) > 0, "gla_chunked: %d heads of %d x %d channels, rank %d, are outside what the kernels take",
                 H, N, P, rank);
    BC_CHECK_ARG(stride % 4 == 0 && v_at % 4 == 0 && (uintptr_t)proj % 16 == 0 && (uintptr_t)pack % 16 == 0 && (uintptr_t)state % 16 == 0 && (uintptr_t)out % 16 == 0,
                 "gla_chunked: rows, values, state and scratch must start on 16-byte borders");
    const int D = glc_width(N);
    BC_CHECK_ARG(chunk_fits(pack_floats / ((long long)H * chunk_pack_floats(D, false)), rows, seqs, min_rows, write_state), "gla_chunked: scratch of %lld floats is too small", pack_floats);
#define GLC(DD) gla_chunked<DD>(proj, stride, q_at, k_at, v_at, inner_at, w2t, b, rank, 1.0f / tau, f, pack, pack_floats, state, seq_rows, seq_slot, out, rows, seqs, max_new, min_rows, H, N, P, n_slots, write_state, s)
    return D == 64 ? GLC(64) : D == 128 ? GLC(128) : GLC(256);
#undef GLC
}
