// The generalized delta rule on prompts, sixteen rows at a time (chunks.cuh):
//
//     S_t = diag(w_t) S_(t-1) - b_t (u_t^T S_(t-1)) + k_t v_t^T        o_t = S_t^T r_t          (b = a * u)
//
// Within a chunk let W_t be the product of its decays up to row t (W_(-1) = 1).  The removed e_t = u_t^T S_(t-1) obeys
//
//     e_t = U_t S + sum_(s<t) Bm_ts v_s - A_ts e_s,      U_t = u_t W_(t-1),  A_ts = sum_i u_t b_s W_(t-1) / W_s,  Bm_ts = the same with k_s,
//
// a unit lower triangular system whose matrix is the chunk's own: e = P S + M V with P = (1 + A)^-1 U, M = (1 + A)^-1 Bm, by forward
// substitution.  With H_ts = sum_i r_t b_s W_t / W_s and Gm_ts with k_s (s <= t), the chunk is then
//
//     X1 = P      X0 = r_t W_t - H P      G = Gm - H M      Z1 = b_s W_15 / W_s      Z0 = k_s W_15 / W_s - M^T Z1      tot = W_15.
//
// A decay is at least exp(-decay_scale), so sixteen of them are divided by safely up to a decay_scale of 4 (exp(-64)).  Operands and results are
// float; the sums over channels (A, Bm, H, Gm) and the correction of Z0 are double, and rows are decayed to a chunk's end by the products
// of the decays after them.  With all of it in float the results were 1.1 to 1.9 times as far from 64-bit sums as the row scan's; so they
// are 0.80 to 1.00 times as far (outputs) and 0.95 to 1.00 (state): 1.1e-7 and 0.9e-7 at a decay_scale of exp(-1/2), the scan 1.2e-7 and 1.0e-7.
// Three kernels: the decays of all rows, a product of its own; the chunks' packs, all side by side; the chunks in time order.  One sequence
// of 2,048 rows, 64 heads of 64, decay rank 64: 350 us with the launches, where the kernels that prepare the rows and scan them one by one take 172 + 614 without.
// The first two are bound by their instructions; the last walks 128 chunks, one warp a scheduler, each chunk's products waiting for the state of
// the one before (half warps or warps a row, four or eight value channels a warp, sums across lanes or through shared memory: all within
// 3 % of one another).
#include "chunks.cuh"

// ------------------------------------------------------------------------------------ decays
// decay[r, c] = exp(-decay_scale * sigmoid(z + w0[c])) with z = sum_j w2t[j, c] tanh(inner[r, j]): a product of 64 rows x 128 channels a block,
// eight rows by four channels a thread, 64 inner channels at a time, all asked for at once, sixteen bytes a load.
// 2,048 rows x 4,096 channels, rank 64: 38 us (32 inner channels at a time, four bytes a load: 56).
#define DLC_ROWS 64
#define DLC_COLS 128
#define DLC_K 64
#define DLC_DECAY_SMEM (DLC_K * (DLC_ROWS + 4 + DLC_COLS) * sizeof(float))
__global__ void __launch_bounds__(256)
delta_decay_kernel(const float* proj, int stride, int inner_at, const float* __restrict__ w2t, const float* __restrict__ w0, float* __restrict__ decay, int rows, int HD,
                   int inner, float decay_scale) {
    extern __shared__ __align__(16) float decay_smem[];
    float (*th)[DLC_ROWS + 4] = reinterpret_cast<float (*)[DLC_ROWS + 4]>(decay_smem);
    float (*wt)[DLC_COLS] = reinterpret_cast<float (*)[DLC_COLS]>(decay_smem + DLC_K * (DLC_ROWS + 4));
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(proj);
    const int row0 = blockIdx.y * DLC_ROWS, c0 = blockIdx.x * DLC_COLS;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;             // channels 4 tx .., rows 8 ty ..
    const bool quads = (uintptr_t)w2t % 16 == 0;      // (stride, inner_at and HD are multiples of four, proj and decay start on 16-byte borders)
    uint64_t z[8][2] = {};
    for (int j0 = 0; j0 < inner; j0 += DLC_K) {
        // Row r's values j .. j + 3, zeros where there are none.  (A channel past the last reads what the weights' place held; it is not written out.)
        auto inner_at4 = [&](int r, int j) {
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row0 + r >= rows || j >= inner) return v;
            const float* p = proj + (size_t)(row0 + r) * stride + inner_at + j;
            if (j + 4 <= inner) return *reinterpret_cast<const float4*>(p);
            v.x = p[0];
            if (j + 1 < inner) v.y = p[1];
            if (j + 2 < inner) v.z = p[2];
            return v;
        };
        if (quads) {
#pragma unroll
            for (int e = 0; e < DLC_K * DLC_COLS / 1024; e++) {
                const int i = threadIdx.x + 256 * e, j = i / (DLC_COLS / 4), c = i % (DLC_COLS / 4) * 4;
                if (j0 + j < inner && c0 + c < HD) cp_async16((uint32_t)__cvta_generic_to_shared(&wt[j][c]), w2t + (size_t)(j0 + j) * HD + c0 + c);
            }
            cp_async_commit();
        } else {
            for (int i = threadIdx.x; i < DLC_K * DLC_COLS; i += 256) {
                const int j = i / DLC_COLS, c = i % DLC_COLS;
                wt[j][c] = j0 + j < inner && c0 + c < HD ? w2t[(size_t)(j0 + j) * HD + c0 + c] : 0.0f;
            }
        }
        float4 raw[DLC_K * DLC_ROWS / 1024];
#pragma unroll
        for (int e = 0; e < DLC_K * DLC_ROWS / 1024; e++) {
            const int i = threadIdx.x + 256 * e;
            raw[e] = inner_at4(i % DLC_ROWS, j0 + i / DLC_ROWS * 4);
        }
#pragma unroll
        for (int e = 0; e < DLC_K * DLC_ROWS / 1024; e++) {
            const int i = threadIdx.x + 256 * e, r = i % DLC_ROWS, j = i / DLC_ROWS * 4;
            th[j][r] = tanhf(raw[e].x);
            th[j + 1][r] = tanhf(raw[e].y);
            th[j + 2][r] = tanhf(raw[e].z);
            th[j + 3][r] = tanhf(raw[e].w);
        }
        if (quads) cp_async_wait<0>();
        __syncthreads();
        const int most = min(DLC_K, inner - j0);
#pragma unroll 8
        for (int j = 0; j < most; j++) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&wt[j][4 * tx]);
            const float4 ta = *reinterpret_cast<const float4*>(&th[j][8 * ty]), tb = *reinterpret_cast<const float4*>(&th[j][8 * ty + 4]);
            const float t[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const uint64_t t2 = pack_f32x2(t[r], t[r]);
                z[r][0] = fma_f32x2(w.x, t2, z[r][0]);
                z[r][1] = fma_f32x2(w.y, t2, z[r][1]);
            }
        }
        __syncthreads();
    }
    const int c = c0 + 4 * tx;
    if (c >= HD) return;
    const float b[4] = {w0[c], w0[c + 1], w0[c + 2], w0[c + 3]};
#pragma unroll
    for (int r = 0; r < 8; r++) {
        const int row = row0 + 8 * ty + r;
        if (row >= rows) break;
        float v[4];
        unpack_f32x2(z[r][0], v[0], v[1]);
        unpack_f32x2(z[r][1], v[2], v[3]);
#pragma unroll
        for (int e = 0; e < 4; e++) v[e] = expf(-decay_scale * sigmoid_f(v[e] + b[e]));
        *reinterpret_cast<float4*>(decay + (size_t)row * HD + c) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// ------------------------------------------------------------------------------------- packs
#define DLC_D 64
// Where channel d's number for row t of the 32 rows [r W; u W] (and [b / W; k / W]) lies, in doubles: pairs of rows are turned about by the channel, so
// that neither the 16-byte writes of eight neighbouring channels nor the reads of four rows by four channels meet a bank twice.
__device__ __forceinline__ int dlc_at(int d, int t) { return d * 2 * CHUNK + (t ^ (4 * (d & 3)) ^ (2 * (d >> 2 & 1))); }
// c += a b: an 8 x 4 and a 4 x 8 tile of doubles, one number of each a lane (a: row lane / 4, column lane % 4; b: row lane % 4, column lane / 4;
// c: row lane / 4, columns 2 (lane % 4) and the next).
__device__ __forceinline__ void dlc_mma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
#define DLC_RUN 4             // places of chunks a block takes one after another, the next one's rows on their way

// A block takes the chunks at `run` neighbouring places, of one head: 64 threads a key channel each, and a warp whose first lanes take M's sixteen
// columns through the same substitutions.  Chains of dependent steps, so what counts is how many blocks an SM holds: one stage of rows, refilled as soon as
// they are in registers, leaves room for four (two stages: three; with them and a square root a channel instead of a row 488 us
// the whole call, now 350).
__global__ void __launch_bounds__(DLC_D + 32, 4)
delta_chunks_kernel(const ChunkSpan span, const float* proj, int stride, const float* decay, const float* __restrict__ a_bias, const int* __restrict__ seq_rows,
                    const int* __restrict__ seq_slot, float* __restrict__ pack, int H, int D, float key_eps, int seqs, int n_slots, int run, int places) {
    constexpr int PACK = chunk_pack_floats(DLC_D, true), THREADS = DLC_D + 32, ROW_SET = CHUNK * DLC_D;
    extern __shared__ __align__(16) float delta_smem[];
    float (*in)[CHUNK][DLC_D] = reinterpret_cast<float (*)[CHUNK][DLC_D]>(delta_smem);                  // a chunk's decays, r, k, a
    double *Y = reinterpret_cast<double*>(delta_smem + 4 * ROW_SET), *X = Y + DLC_D * 2 * CHUNK, *M = Y;      // (M [16][16] where Y was, once that has been used)
    float (*lower)[CHUNK][CHUNK_G] = reinterpret_cast<float (*)[CHUNK][CHUNK_G]>(X + DLC_D * 2 * CHUNK);    // A, Bm, H, Gm
    __shared__ float part[2][CHUNK];
    __shared__ float2 norm[CHUNK];            // and its reciprocal
    __shared__ ChunkAt todo[DLC_RUN];
    __shared__ int todo_place[DLC_RUN], n_todo;
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(proj); PDL_FRESH(decay);
    const int h = blockIdx.y, HD = H * D;
    const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
    if (warp == 0) {                                       // the chunks there are, one after another
        const int place = blockIdx.x * run + lane;
        const ChunkAt at = lane < run && place < places ? chunk_at(span, place, seq_rows, seq_slot, seqs, n_slots) : ChunkAt{0, 0};
        const unsigned there = __ballot_sync(0xffffffffu, at.rows > 0);
        if (at.rows > 0) {
            const int i = __popc(there & ((1u << lane) - 1u));
            todo[i] = at;
            todo_place[i] = place;
        }
        if (lane == 0) n_todo = __popc(there);
    }
    __syncthreads();
    const int n = n_todo;
    if (n == 0) return;
    const bool channel = d < DLC_D, mine = d < D;
    const float bias = mine ? a_bias[h * D + d] : 0.0f;
    // What no copy reaches (rows past the sequence, channels past the head) is never used: it may hold anything.
    auto issue = [&](int c) {
        const int rows = todo[c].rows, quads = D / 4;
        const size_t first = (size_t)todo[c].row;
        const uint32_t dst = ad_smem(&in[0][0][0]);
        for (int i = threadIdx.x; i < rows * quads; i += THREADS) {
            const int t = i / quads, at = 4 * (i - t * quads);
            const float* pr = proj + (first + t) * stride + h * D + at;
            const uint32_t to = dst + 4 * (t * DLC_D + at);
            cp_async16(to, decay + (first + t) * HD + h * D + at);
            cp_async16(to + 4 * ROW_SET, pr);
            cp_async16(to + 8 * ROW_SET, pr + HD);
            cp_async16(to + 12 * ROW_SET, pr + 4 * HD);
        }
    };
    issue(0);
    cp_async_commit();
    // What lies above the diagonals by whole tiles stays zero.
    for (int i = threadIdx.x; i < 4 * 64; i += THREADS) lower[i / 64][i / 8 % 8][8 + i % 8] = 0.0f;
    const float (*sw)[DLC_D] = in[0], (*sr)[DLC_D] = in[1], (*sk)[DLC_D] = in[2], (*sa)[DLC_D] = in[3];
    for (int c = 0; c < n; c++) {
        cp_async_wait<0>();
        __syncthreads();
        const int rows = todo[c].rows;
        if (channel) {
            // Sixteen sums over a warp's channels, halved among its lanes: lane L (of sixteen) is left with row L.
            float kk[CHUNK];
#pragma unroll
            for (int t = 0; t < CHUNK; t++) {
                const float k = mine && t < rows ? sk[t][d] : 0.0f;
                kk[t] = k * k;
                kk[t] += __shfl_xor_sync(0xffffffffu, kk[t], 16);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < o; i++) {
                    const float keep = up ? kk[i + o] : kk[i], send = up ? kk[i] : kk[i + o];
                    kk[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            if (lane < CHUNK) part[warp][lane] = kk[0];
        }
        __syncthreads();
        if (d < CHUNK) norm[d] = divisor(sqrtf(part[0][d] + part[1][d] + key_eps));      // once a row, not once a channel
        __syncthreads();
        float* dst = pack + ((size_t)todo_place[c] * H + h) * PACK;
        float U[CHUNK], own[CHUNK];               // u_t W_(t-1), then P, and r_t W_t, then X0; in the last warp columns of Bm, then M, and of Gm, then G
        float z1[CHUNK], zk[CHUNK];               // b_t and k_t, then times the decays after row t
        // (With divisions and their branches a row took 520 clocks of dependent steps, now 170; the results' distance from 64-bit sums is the same to five digits.)
        if (channel) {
            float run = 1.0f, xb_even = 0.0f, xk_even = 0.0f;
#pragma unroll
            for (int t = 0; t < CHUNK; t++) {
                const bool ok = mine && t < rows;
                const float k = ok ? sk[t][d] : 0.0f;
                const float rate = sigmoid_f((ok ? sa[t][d] : 0.0f) + bias);
                const float u = ok ? quotient(k, norm[t]) : 0.0f;      // zero in rows and channels that do not exist
                U[t] = u * run;
                run *= ok ? sw[t][d] : 1.0f;
                own[t] = (ok ? sr[t][d] : 0.0f) * run;
                const float over = reciprocal(run), xb = rate * u * over, xk = k * over;
                z1[t] = rate * u;
                zk[t] = k;
                if (t & 1) {
                    const int first = dlc_at(d, t - 1), second = dlc_at(d, CHUNK + t - 1);
                    *reinterpret_cast<double2*>(Y + first) = make_double2(own[t - 1], own[t]);
                    *reinterpret_cast<double2*>(Y + second) = make_double2(U[t - 1], U[t]);
                    *reinterpret_cast<double2*>(X + first) = make_double2(xb_even, xb);
                    *reinterpret_cast<double2*>(X + second) = make_double2(xk_even, xk);
                }
                xb_even = xb;
                xk_even = xk;
            }
            // (From the last row back, not as the quotient of two products: the latest rows, which weigh most, then have the fewest roundings.)
            run = 1.0f;
#pragma unroll
            for (int t = CHUNK - 1; t >= 0; t--) {
                z1[t] *= run;
                zk[t] *= run;
                run *= mine && t < rows ? sw[t][d] : 1.0f;
                dst[(3 * CHUNK + t) * DLC_D + d] = z1[t];
            }
            dst[4 * CHUNK * DLC_D + CHUNK * CHUNK_G + d] = run;
        }
        __syncthreads();
        if (c + 1 < n) issue(c + 1);              // these rows are in registers and in Y and X: the next ones may take their place
        cp_async_commit();
        // [r W; u W] [b / W; k / W]^T over the channels in double, 8 x 8 numbers a tile: the twelve tiles that reach below a diagonal, four a
        // warp, which share one tile of rows (the last eight rows: all four) or two.  One prompt of 2,048 rows, 64 heads: 433 -> 407 us the
        // whole call (a number at a time, sixteen a thread of two warps, the halves above the diagonals too).
        {
            const bool last = warp < 2;                     // of r W, then of u W; the third warp takes the first eight rows of both
            const int g = lane >> 2, e = lane & 3;
            double acc[4][2] = {};
            const int of_y = last ? 8 + CHUNK * warp : 0;
            auto tiles = [&](auto both) {
                constexpr bool BOTH = decltype(both)::value;
#pragma unroll 8
                for (int i = 0; i < DLC_D; i += 4) {
                    const int d0 = i + e;
                    const double y0 = Y[dlc_at(d0, of_y + g)], b0 = X[dlc_at(d0, g)], k0 = X[dlc_at(d0, CHUNK + g)];
                    if (BOTH) {
                        const double y1 = Y[dlc_at(d0, CHUNK + g)];
                        dlc_mma(acc[0], y0, b0), dlc_mma(acc[1], y0, k0), dlc_mma(acc[2], y1, b0), dlc_mma(acc[3], y1, k0);
                    } else {
                        const double b1 = X[dlc_at(d0, 8 + g)], k1 = X[dlc_at(d0, CHUNK + 8 + g)];
                        dlc_mma(acc[0], y0, b0), dlc_mma(acc[1], y0, k0), dlc_mma(acc[2], y0, b1), dlc_mma(acc[3], y0, k1);
                    }
                }
            };
            if (last) tiles(std::false_type());
            else tiles(std::true_type());
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const bool of_u = last ? warp == 1 : i >= 2;                 // A and Bm (s < t), or H and Gm (s <= t)
                    const int t = last ? 8 + g : g, s = (last && i >= 2 ? 8 : 0) + 2 * e + j, most = of_u ? t - 1 : t;
                    lower[(of_u ? 0 : 2) + (i & 1)][t][s] = s <= most ? (float)acc[i][j] : 0.0f;
                }
        }
        __syncthreads();
        // The substitutions: columns of U (a channel each) and of Bm alike, and own_t - sum_s H_ts x_s of the solved ones.
        if (!channel) {
#pragma unroll
            for (int t = 0; t < CHUNK; t++) {
                U[t] = lower[1][t][lane & 15];
                own[t] = lower[3][t][lane & 15];
            }
        }
#pragma unroll
        for (int t = 1; t < CHUNK; t++)
#pragma unroll
            for (int s = 0; s < t; s++) U[t] = fmaf(-lower[0][t][s], U[s], U[t]);
#pragma unroll
        for (int t = 0; t < CHUNK; t++)
#pragma unroll
            for (int s = 0; s <= t; s++) own[t] = fmaf(-lower[2][t][s], U[s], own[t]);
        __syncwarp();
        if (!channel) {
            if (lane < CHUNK) {
#pragma unroll
                for (int t = 0; t < CHUNK; t++) {
                    M[t * CHUNK + lane] = U[t];
                    dst[4 * CHUNK * DLC_D + t * CHUNK_G + lane] = own[t];
                }
            }
        } else {
#pragma unroll
            for (int t = 0; t < CHUNK; t++) {
                dst[t * DLC_D + d] = own[t];
                dst[(CHUNK + t) * DLC_D + d] = U[t];
            }
        }
        __syncthreads();
        if (channel) {
            double z0[CHUNK];
#pragma unroll
            for (int s = 0; s < CHUNK; s++) z0[s] = zk[s];
#pragma unroll
            for (int t = 1; t < CHUNK; t++) {
                const double z = -z1[t];
#pragma unroll
                for (int s = 0; s < t; s += 2) {
                    const double2 m = *reinterpret_cast<const double2*>(M + t * CHUNK + s);
                    z0[s] = fma(m.x, z, z0[s]);
                    if (s + 1 < t) z0[s + 1] = fma(m.y, z, z0[s + 1]);
                }
            }
#pragma unroll
            for (int s = 0; s < CHUNK; s++) dst[(2 * CHUNK + s) * DLC_D + d] = (float)z0[s];
        }
        __syncthreads();          // the next chunk writes Y, X and the triangles
    }
}
#define DLC_SMEM ((4 * CHUNK * DLC_D + 4 * CHUNK * CHUNK_G) * sizeof(float) + 4 * CHUNK * DLC_D * sizeof(double))

// Whether heads of D channels run in chunks, and the floats of scratch that `rows` rows of `seqs` sequences take (0: they do not), of which those of
// fewer than min_rows rows are left alone.
extern "C" long long bc_delta_chunked_scratch(int rows, int seqs, int min_rows, int H, int D, int inner, float decay_scale, int write_state) {
    if (D <= 0 || D > DLC_D || D % 4 || inner <= 0 || H <= 0 || H > 65535 || seqs <= 0 || seqs > 65535 || !(decay_scale >= 0.0f && decay_scale <= 4.0f)) return 0;
    const int pack = chunk_pack_floats(DLC_D, true);
    return chunk_capacity(rows, seqs, min_rows, H, pack, write_state) * H * pack;
}

// proj, w2t, w0, a_bias as for bc_delta_prepare; state, seq_rows, seq_slot, out as for bc_delta_scan; decay: scratch [rows, H D]; pack: scratch of
// pack_floats floats, bc_delta_chunked_scratch of them for the fewest launches; max_new: the most rows that a sequence brings; min_rows: sequences of
// fewer rows are left alone, their states and their rows of out.
extern "C" int bc_delta_chunked(const float* proj, int stride, const float* w2t, const float* w0, const float* a_bias, float* decay, float* pack, long long pack_floats, float* state,
                                const int* seq_rows, const int* seq_slot, float* out, int rows, int seqs, int max_new, int min_rows, int H, int D, int inner,
                                float decay_scale, float key_eps, int n_slots, int write_state, cudaStream_t s) {
    BC_CHECK_ARG(rows >= 0 && seqs >= 0 && max_new >= 0, "delta_chunked: bad sizes rows=%d seqs=%d max_new=%d", rows, seqs, max_new);
    if (rows == 0 || seqs == 0 || max_new == 0) return BC_OK;
    BC_CHECK_ARG(bc_delta_chunked_scratch(rows, seqs, min_rows, H, D, inner, decay_scale, write_state) > 0,
                 "delta_chunked: %d heads of %d, inner %d, decay_scale %g are outside what the kernels take", H, D, inner, (double)decay_scale);
    BC_CHECK_ARG(stride >= 5 * H * D + inner, "delta_chunked: a row of %d values cannot hold five projections of %d and %d more", stride, H * D, inner);
    BC_CHECK_ARG((rows + DLC_ROWS - 1) / DLC_ROWS <= 65535, "delta_chunked: %d rows are too many", rows);
    BC_CHECK_ARG(stride % 4 == 0 && (uintptr_t)proj % 16 == 0 && (uintptr_t)decay % 16 == 0 && (uintptr_t)pack % 16 == 0 && (uintptr_t)state % 16 == 0 && (uintptr_t)out % 16 == 0,
                 "delta_chunked: rows, state and scratch must start on 16-byte borders");
    const long long capacity = pack_floats / ((long long)H * chunk_pack_floats(DLC_D, true));
    BC_CHECK_ARG(chunk_fits(capacity, rows, seqs, min_rows, write_state), "delta_chunked: scratch of %lld floats is too small", pack_floats);
    if (cudaError_t e = bc_allow_shared<delta_chunks_kernel>(DLC_SMEM); e != cudaSuccess) {
        bc_set_error("delta_chunked: %s", cudaGetErrorString(e));
        return (int)e;
    }
    if (cudaError_t e = bc_allow_shared<delta_decay_kernel>(DLC_DECAY_SMEM); e != cudaSuccess) {
        bc_set_error("delta_chunked: %s", cudaGetErrorString(e));
        return (int)e;
    }
    cudaError_t e = bc_launch(delta_decay_kernel, dim3((H * D + DLC_COLS - 1) / DLC_COLS, (rows + DLC_ROWS - 1) / DLC_ROWS), dim3(256), DLC_DECAY_SMEM, s, proj, stride, 5 * H * D, w2t,
                              w0, decay, rows, H * D, inner, decay_scale);
    if (e == cudaSuccess)
        e = chunk_step(
            capacity, rows, seqs, max_new, min_rows,
            [&](const ChunkSpan& span, long long places) {
                // Four chunks a block hide the loads of the next one (128 chunks of 64 heads, all in float: 232 us one a block, 143 four); where that leaves
                // places on the SMs empty, one (with the rest of a call, 64 heads: 4 sequences of 64 rows 92 us four a block, 83 one; 8 heads: one of 64 rows 67 and 47).
                const int run = (places + DLC_RUN - 1) / DLC_RUN * H >= 3 * bc_sm_count() ? DLC_RUN : 1;
                return bc_launch(delta_chunks_kernel, dim3((unsigned)((places + run - 1) / run), H), dim3(DLC_D + 32), DLC_SMEM, s, span, proj, stride, decay, a_bias, seq_rows, seq_slot, pack, H, D,
                                 key_eps, seqs, n_slots, run, (int)places);
            },
            [&](const ChunkSpan& span) {
                return chunk_scan_launch<DLC_D / 32, true>(span, pack, proj + 2 * H * D, stride, state, seq_rows, seq_slot, out, rows, max_new, seqs, H, D, D, n_slots, write_state, 1.0f, s);
            });
    if (e != cudaSuccess) {
        bc_set_error("delta_chunked: %s", cudaGetErrorString(e));
        return (int)e;
    }
    BC_LAUNCH_STATUS();
}

// out[i] = 1 / a[i], its sigmoid, or a[i] / b[i], as the kernels above work them out.  For tests.
__global__ void delta_arithmetic_kernel(const float* a, const float* b, float* out, int what, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = what == 0 ? reciprocal(a[i]) : what == 1 ? sigmoid_f(a[i]) : quotient(a[i], divisor(b[i]));
}
extern "C" int bc_delta_arithmetic(const float* a, const float* b, float* out, int what, int n, cudaStream_t s) {
    BC_CHECK_ARG(n >= 0 && what >= 0 && what <= 2 && (what < 2 || b != nullptr), "delta_arithmetic: bad arguments n=%d what=%d", n, what);
    if (n == 0) return BC_OK;
    delta_arithmetic_kernel<<<(n + 255) / 256, 256, 0, s>>>(a, b, out, what, n);
    BC_LAUNCH_STATUS();
}
