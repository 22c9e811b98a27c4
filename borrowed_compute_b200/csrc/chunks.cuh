// Recurrences over time taken sixteen rows at a time, in float on the CUDA cores.
//
// A state S [N key channels, P value channels] that decays channel by channel and takes outer products is, over a chunk of sixteen
// rows, a linear map of what it was before: with the rows' own vectors multiplied once by the decays between them and the chunk's
// borders (a kernel over all chunks side by side), what is left in time order is
//
//     O = X0 S + G V          E = X1 S (delta rules only)          S <- tot * S + Z0^T V - Z1^T E
//
// with X0, X1, Z0, Z1 [16, N] and G [16, 16] a chunk: products over sixteen rows, where the row-by-row scan has two dot products,
// three shuffles and an update a row, each waiting for the one before.  The arithmetic is of the same order (5 N P against 4 N P
// multiply-adds a row of a delta rule); what goes is the chain.
//
// A chunk of one head is one run of floats in memory ("pack"): X0 [16][D], (X1 [16][D],) Z0 [16][D], (Z1 [16][D],) G [16][20], tot [D], D = N rounded up to 64, 128 or 256, zeros (tot: ones) past N and past a sequence's last row.
#pragma once

#include <type_traits>

#include "mma_tiles.cuh"

#define CHUNK 16              // rows
#define CHUNK_G 20            // floats a row of G: sixteen and a gap, so that the rows that eight threads read start in different banks

__host__ __device__ constexpr int chunk_pack_floats(int D, bool delta) { return (delta ? 4 : 2) * CHUNK * D + CHUNK * CHUNK_G + D; }
// A launch takes chunks [first, first + count) of every sequence of at least min_rows rows.  Where sequence `seq`, whose rows start at row0 of the
// step, keeps chunk c: with all of a step's chunks in one launch (segment 0) by its rows, so that sequences never meet and few places stay
// empty; else `segment` places a sequence.  By its rows: one place more a sequence for its last, partial chunk; or, crowded (many sequences beside
// few rows, none of the ones taken shorter than a chunk), two places every sixteen rows.
struct ChunkSpan {
    int first, count, segment, crowded, min_rows;
};
__device__ __forceinline__ int chunk_first_place(const ChunkSpan& span, int row0, int seq) { return span.crowded ? row0 / CHUNK * 2 : row0 / CHUNK + seq; }
__device__ __forceinline__ size_t chunk_place(const ChunkSpan& span, int row0, int seq, int c) {
    return span.segment ? (size_t)seq * span.segment + (c - span.first) : (size_t)(chunk_first_place(span, row0, seq) + c);
}
// The chunk at a place: its first row of the step and how many it has (0: none, or one of a sequence that is not taken).  The kernel that fills the
// packs goes by places, not by the longest sequence times all of them: a prompt beside many single rows leaves few blocks without work.
struct ChunkAt {
    int row, rows;
};
__device__ __forceinline__ ChunkAt chunk_at(const ChunkSpan& span, int place, const int* seq_rows, const int* seq_slot, int seqs, int n_slots) {
    int seq = 0, c;
    if (span.segment) {
        seq = place / span.segment;
        c = place - seq * span.segment;
        if (seq >= seqs || c >= span.count) return {0, 0};
        c += span.first;
    } else {
        int end = seqs;                        // the last sequence whose places begin here or before
        while (end - seq > 1) {
            const int mid = (seq + end) / 2;
            if (chunk_first_place(span, seq_rows[mid], mid) <= place) seq = mid;
            else end = mid;
        }
        c = place - chunk_first_place(span, seq_rows[seq], seq);
    }
    const int row0 = seq_rows[seq], n_rows = seq_rows[seq + 1] - row0, slot = seq_slot[seq];
    if (c < 0 || c * CHUNK >= n_rows || n_rows < span.min_rows || slot < 0 || slot >= n_slots) return {0, 0};
    return {row0 + c * CHUNK, min(CHUNK, n_rows - c * CHUNK)};
}
static inline bool chunk_crowded(long long rows, long long seqs, int min_rows) { return min_rows >= CHUNK && rows / CHUNK + 1 < seqs; }
static inline long long chunk_places(long long rows, long long seqs, int min_rows) {
    return chunk_crowded(rows, seqs, min_rows) ? 2 * (rows / CHUNK) + 2 : rows / CHUNK + seqs + 1;
}
// Chunks of scratch for a step: all of them, or as many as 2^28 floats hold (a gigabyte; at least one a sequence), and then the step goes
// segment by segment, which hands the state on through memory and so must be allowed to write it.  0: not taken.
static inline long long chunk_capacity(long long rows, long long seqs, int min_rows, long long H, int pack_floats, int write_state) {
    const long long total = chunk_places(rows, seqs, min_rows), most = (1ll << 28) / (H * pack_floats);
    if (total <= most) return total;
    return write_state ? (most > seqs ? most / seqs * seqs : seqs) : 0;
}

// Rows of X times the state, summed over the sixteen lanes of a half warp (lane `dg` of it holds key channels 4 dg + 64 m .. + 3): lane dg is left
// with row dg.  A lane forms its I-th partial sum for row I ^ dg, so every exchange sends a register that all lanes name alike
// (fifteen shuffles a value, no selection).  The rows come in four groups, I = i, i + 8, i + 4, i + 12 for i = 0, 2, 1, 3: a group's
// rows are loaded while the group before is worked on.
__host__ __device__ constexpr int chunk_row_of(int group, int k) { return (group == 0 ? 0 : group == 1 ? 2 : group == 2 ? 1 : 3) + (k & 1) * 8 + (k >> 1) * 4; }
template <int DT> struct ChunkRows {
    ulonglong2 x[4][DT / 4];
    __device__ __forceinline__ void load(const float* rows, int group, int dg) {
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int m = 0; m < DT / 4; m++) x[k][m] = *reinterpret_cast<const ulonglong2*>(rows + (chunk_row_of(group, k) ^ dg) * (16 * DT) + 64 * m);
    }
    // out: the group's four rows times the state, halved twice.
    template <int PT> __device__ __forceinline__ void times(const uint64_t (*S)[PT], float* out) const {
        float part[4][PT];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint64_t a[PT];
#pragma unroll
            for (int m = 0; m < DT / 4; m++)
#pragma unroll
                for (int p = 0; p < PT; p++) a[p] = fma_f32x2(x[k][m].x, S[2 * m][p], m ? a[p] : 0ull);
#pragma unroll
            for (int m = 0; m < DT / 4; m++)
#pragma unroll
                for (int p = 0; p < PT; p++) a[p] = fma_f32x2(x[k][m].y, S[2 * m + 1][p], a[p]);
#pragma unroll
            for (int p = 0; p < PT; p++) {
                float lo, hi;
                unpack_f32x2(a[p], lo, hi);
                part[k][p] = lo + hi;
            }
        }
#pragma unroll
        for (int p = 0; p < PT; p++) {
            part[0][p] += __shfl_xor_sync(0xffffffffu, part[1][p], 8);
            part[2][p] += __shfl_xor_sync(0xffffffffu, part[3][p], 8);
        }
#pragma unroll
        for (int p = 0; p < PT; p++) out[p] = part[0][p] + __shfl_xor_sync(0xffffffffu, part[2][p], 4);
    }
};
template <int PT> __device__ __forceinline__ void chunk_groups(const float (*g)[PT], float* out) {
    float a[PT], b[PT];
#pragma unroll
    for (int p = 0; p < PT; p++) {
        a[p] = g[0][p] + __shfl_xor_sync(0xffffffffu, g[1][p], 2);
        b[p] = g[2][p] + __shfl_xor_sync(0xffffffffu, g[3][p], 2);
    }
#pragma unroll
    for (int p = 0; p < PT; p++) out[p] = a[p] + __shfl_xor_sync(0xffffffffu, b[p], 1);
}

// A block takes (a slice of 32 value channels, head, sequence): a half warp holds the key channels of four value channels in registers, two
// key channels to a 64-bit register (fma.rn.f32x2), for all of the sequence's rows.  A chunk's pack and its 16 x 32 values come
// through a ring of asynchronous copies.
#define CHUNK_THREADS 128
#define CHUNK_STAGES 3         // chunks on their way or worked on
#define CHUNK_SORTED 64        // sequences of a step that are put in order (two a lane)
#define CHUNK_ALONE (120 * 1024)      // bytes of shared memory of which an SM holds one block's
// A sequence, the step's row it starts at, its rows and its slot.  Of at most 64 the one that comes z-th when the longest come first, by eighths of the
// longest's rows (of those alike the earlier); every warp works it out for itself, two sequences a lane.
struct ChunkSequence {
    int seq, row0, rows, slot;
};
__device__ __forceinline__ ChunkSequence chunk_long_first(int z, const int* seq_rows, const int* seq_slot, int seqs) {
    const int lane = threadIdx.x & 31;
    int row0[2], rows[2], slot[2], eighth[2];
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int seq = lane + 32 * i;
        row0[i] = seq < seqs ? seq_rows[seq] : 0;
        rows[i] = seq < seqs ? seq_rows[seq + 1] - row0[i] : -1;
        slot[i] = seq < seqs ? seq_slot[seq] : -1;
    }
    const int longest = max(__reduce_max_sync(0xffffffffu, max(rows[0], rows[1])), 1);
#pragma unroll
    for (int i = 0; i < 2; i++) eighth[i] = rows[i] < 0 ? -1 : (int)min(7ll, 8ll * rows[i] / longest);
    int before = 0;
    for (int e = 7; e >= 0; e--) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const unsigned here = __ballot_sync(0xffffffffu, eighth[i] == e);
            if (z < before + __popc(here)) {
                const unsigned found = __ballot_sync(0xffffffffu, eighth[i] == e && before + __popc(here & ((1u << lane) - 1u)) == z);
                const int from = __ffs(found) - 1;
                return {from + 32 * i, __shfl_sync(0xffffffffu, row0[i], from), __shfl_sync(0xffffffffu, rows[i], from), __shfl_sync(0xffffffffu, slot[i], from)};
            }
            before += __popc(here);
        }
    }
    return {z, 0, 0, -1};
}

template <int DL, bool DELTA, bool LONG_FIRST>      // D = 32 DL
__global__ void __launch_bounds__(CHUNK_THREADS)
chunk_scan_kernel(const ChunkSpan span, const float* pack, const float* v, int v_stride, float* __restrict__ state, const int* __restrict__ seq_rows,
                  const int* __restrict__ seq_slot, float* __restrict__ out, int H, int N, int P, int n_slots, int write_state, float out_scale) {
    constexpr int DT = 2 * DL, D = 16 * DT, PT = 4, MATS = DELTA ? 4 : 2, PACK = chunk_pack_floats(D, DELTA), V_AT = PACK, STAGE = V_AT + CHUNK * 32;
    extern __shared__ __align__(16) float chunk_smem[];
    const int dg = threadIdx.x & 15, pg = threadIdx.x >> 4;
    float* mine = chunk_smem + CHUNK_STAGES * STAGE + pg * CHUNK * PT;      // what a half warp hands to itself: -E of its value channels
    pdl_launch_dependents_if_resident();
    pdl_wait();
    PDL_FRESH(pack); PDL_FRESH(v);
    const int h = blockIdx.y, p0 = blockIdx.x * 32;
    int seq = blockIdx.z, row0, n_rows, slot;
    if constexpr (LONG_FIRST) {
        const ChunkSequence of = chunk_long_first(seq, seq_rows, seq_slot, gridDim.z);
        seq = of.seq, row0 = of.row0, n_rows = of.rows, slot = of.slot;
    } else {
        slot = seq_slot[seq];
        row0 = seq_rows[seq];
        n_rows = seq_rows[seq + 1] - row0;
    }
    if (slot < 0 || slot >= n_slots || n_rows <= 0 || n_rows < span.min_rows) return;
    const int n_chunks = min(span.first + span.count, (n_rows + CHUNK - 1) / CHUNK);
    if (span.first >= n_chunks) return;
    const int pv = min(32, P - p0);                                        // value channels that exist (a multiple of four)
    // The values past the head's channels are never copied: they stay zero.  (Those past the sequence's last row are set to zero with its chunk,
    // whose place may have held another's: rows of zeros in Z0, times an infinity, would be none.)
    for (int i = threadIdx.x; i < CHUNK_STAGES * CHUNK * 32; i += CHUNK_THREADS) chunk_smem[(i / (CHUNK * 32)) * STAGE + V_AT + i % (CHUNK * 32)] = 0.0f;
    __syncthreads();
    // The chunk that is asked for next (a sequence's chunks lie at neighbouring places): where this thread's first quads come from, the rows from there on, its stage.
    const int t = threadIdx.x >> 3, at = 4 * (threadIdx.x & 7);
    const float* next = pack + (chunk_place(span, row0, seq, span.first) * H + h) * PACK + 4 * threadIdx.x;
    const float* next_v = v + (size_t)(row0 + span.first * CHUNK + t) * v_stride + (size_t)h * P + p0 + at;
    int next_rows = min(n_rows, (span.first + span.count) * CHUNK) - span.first * CHUNK, next_at = 0;
    auto issue = [&] {
        if (next_rows > 0) {
            float* stage = chunk_smem + next_at;
            const uint32_t dst = ad_smem(stage) + 16 * threadIdx.x;
#pragma unroll
            for (int i = 0; i < PACK / 4 / CHUNK_THREADS; i++) cp_async16(dst + 16 * CHUNK_THREADS * i, next + 4 * CHUNK_THREADS * i);
            if (threadIdx.x < PACK / 4 % CHUNK_THREADS) cp_async16(dst + 4 * (PACK - PACK % (4 * CHUNK_THREADS)), next + (PACK - PACK % (4 * CHUNK_THREADS)));
            if (t >= next_rows) *reinterpret_cast<float4*>(stage + V_AT + t * 32 + at) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            else if (at < pv) cp_async16(ad_smem(stage) + 4 * (V_AT + t * 32 + at), next_v);
        }
        cp_async_commit();
        next += (size_t)H * PACK;
        next_v += (size_t)CHUNK * v_stride;
        next_rows -= CHUNK;
        next_at = next_at == (CHUNK_STAGES - 1) * STAGE ? 0 : next_at + STAGE;
    };
#pragma unroll
    for (int i = 0; i < CHUNK_STAGES - 1; i++) issue();
    uint64_t S[DT / 2][PT];
    const bool p_ok = pg * PT < pv;
    float* st = state + (((size_t)slot * H + h) * P + p0 + (p_ok ? pg * PT : 0)) * N + 4 * dg;
#pragma unroll
    for (int m = 0; m < DT / 4; m++)
#pragma unroll
        for (int p = 0; p < PT; p++) {
            const bool ok = p_ok && 4 * dg + 64 * m < N;
            const float4 x = ok ? *reinterpret_cast<const float4*>(st + (size_t)p * N + 64 * m) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            S[2 * m][p] = pack_f32x2(x.x, x.y);
            S[2 * m + 1][p] = pack_f32x2(x.z, x.w);
        }
    int now_at = 0;               // the stage worked on
    for (int c = span.first; c < n_chunks; c++) {
        cp_async_wait<CHUNK_STAGES - 2>();
        __syncthreads();          // the chunk is there for all, and all have left the one whose stage is filled next
        issue();
        const float* sx = chunk_smem + now_at;
        now_at = now_at == (CHUNK_STAGES - 1) * STAGE ? 0 : now_at + STAGE;
        const float *x0 = sx + 4 * dg, *z0 = x0 + (DELTA ? 2 : 1) * CHUNK * D, *z1 = z0 + CHUNK * D, *g = sx + MATS * CHUNK * D, *tot = g + CHUNK * CHUNK_G;
        const float* sv = sx + V_AT + pg * PT;
        float vr[CHUNK][PT];      // sixteen rows of this half warp's values
#pragma unroll
        for (int t = 0; t < CHUNK; t++) {
            const float4 x = *reinterpret_cast<const float4*>(sv + t * 32);
            vr[t][0] = x.x, vr[t][1] = x.y, vr[t][2] = x.z, vr[t][3] = x.w;
        }
        float o[PT], removed[PT], of_group[4][PT];
        ChunkRows<DT> rows_now, rows_next;
        rows_now.load(DELTA ? x0 + CHUNK * D : x0, 0, dg);
        if (DELTA) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                rows_next.load(i < 3 ? x0 + CHUNK * D : x0, (i + 1) & 3, dg);
                rows_now.template times<PT>(S, of_group[i]);
                rows_now = rows_next;
            }
            chunk_groups<PT>(of_group, removed);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (i < 3) rows_next.load(x0, i + 1, dg);
            rows_now.template times<PT>(S, of_group[i]);
            rows_now = rows_next;
        }
        chunk_groups<PT>(of_group, o);
        // The rows' own part, G V: this lane's row of G against the values up to its own (later rows' are not touched: a zero of G times
        // an infinity would be none).  Without what is removed, the first eight rows' sum is taken by itself: fewer roundings of the whole.
        float own[PT] = {};
#pragma unroll
        for (int s4 = 0; s4 < CHUNK / 4; s4++) {
            const float4 gg = *reinterpret_cast<const float4*>(g + dg * CHUNK_G + 4 * s4);
            const float gs[4] = {gg.x, gg.y, gg.z, gg.w};
            if (!DELTA && s4 == 2)
#pragma unroll
                for (int p = 0; p < PT; p++) o[p] += own[p];
            float* to = !DELTA && s4 < 2 ? own : o;
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int p = 0; p < PT; p++)
                    if (4 * s4 + e <= dg) to[p] = fmaf(gs[e], vr[4 * s4 + e][p], to[p]);
        }
        if (p_ok && c * CHUNK + dg < n_rows)
            *reinterpret_cast<float4*>(out + (size_t)(row0 + c * CHUNK + dg) * H * P + (size_t)h * P + p0 + pg * PT) = make_float4(out_scale * o[0], out_scale * o[1], out_scale * o[2], out_scale * o[3]);
        if (DELTA) {              // (handed over no sooner than it is needed: what is removed is still being summed while O is begun)
            *reinterpret_cast<float4*>(mine + dg * PT) = make_float4(-removed[0], -removed[1], -removed[2], -removed[3]);
            __syncwarp();
        }
        // The state after the chunk.  Of a delta rule: what was, less what is removed, then what is added (removed last, the sums carry parts that
        // cancel: 1.8 times as far from 64-bit sums).  Else: twelve rows' sum from nothing, what was, the last four rows (what was first: 1.1 times
        // as far where decays are slow; what was last: 1.2 times where they are fast).
        float s[DT][PT];
        auto decayed = [&](bool first) {
#pragma unroll
            for (int m = 0; m < DT / 4; m++) {
                const ulonglong2 t2 = *reinterpret_cast<const ulonglong2*>(tot + 4 * dg + 64 * m);
#pragma unroll
                for (int p = 0; p < PT; p++) {
                    const uint64_t lo = first ? 0ull : pack_f32x2(s[4 * m][p], s[4 * m + 1][p]), hi = first ? 0ull : pack_f32x2(s[4 * m + 2][p], s[4 * m + 3][p]);
                    unpack_f32x2(fma_f32x2(t2.x, S[2 * m][p], lo), s[4 * m][p], s[4 * m + 1][p]);
                    unpack_f32x2(fma_f32x2(t2.y, S[2 * m + 1][p], hi), s[4 * m + 2][p], s[4 * m + 3][p]);
                }
            }
        };
        if (DELTA) {
            decayed(true);
#pragma unroll
            for (int r = 0; r < CHUNK; r++) {
                const float4 e4 = *reinterpret_cast<const float4*>(mine + r * PT);
                const float es[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
                for (int m = 0; m < DT / 4; m++) {
                    const float4 z = *reinterpret_cast<const float4*>(z1 + r * D + 64 * m);
                    const float zs[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int p = 0; p < PT; p++) s[4 * m + i][p] = fmaf(zs[i], es[p], s[4 * m + i][p]);
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < DT; i++)
#pragma unroll
                for (int p = 0; p < PT; p++) s[i][p] = 0.0f;
        }
#pragma unroll
        for (int r = 0; r < CHUNK; r++) {
            if (!DELTA && r == 12) decayed(false);
#pragma unroll
            for (int m = 0; m < DT / 4; m++) {
                const float4 z = *reinterpret_cast<const float4*>(z0 + r * D + 64 * m);
                const float zs[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int p = 0; p < PT; p++) s[4 * m + i][p] = fmaf(zs[i], vr[r][p], s[4 * m + i][p]);
            }
        }
#pragma unroll
        for (int i = 0; i < DT / 2; i++)
#pragma unroll
            for (int p = 0; p < PT; p++) S[i][p] = pack_f32x2(s[2 * i][p], s[2 * i + 1][p]);
    }
    if (write_state && p_ok) {
#pragma unroll
        for (int m = 0; m < DT / 4; m++)
#pragma unroll
            for (int p = 0; p < PT; p++)
                if (4 * dg + 64 * m < N) {
                    float4 x;
                    unpack_f32x2(S[2 * m][p], x.x, x.y);
                    unpack_f32x2(S[2 * m + 1][p], x.z, x.w);
                    *reinterpret_cast<float4*>(st + (size_t)p * N + 64 * m) = x;
                }
    }
}

template <int DL, bool DELTA>
static cudaError_t chunk_scan_launch(const ChunkSpan& span, const float* pack, const float* v, int v_stride, float* state, const int* seq_rows, const int* seq_slot,
                                     float* out, int rows, int max_new, int seqs, int H, int N, int P, int n_slots, int write_state, float out_scale, cudaStream_t s) {
    constexpr size_t NEEDS = (CHUNK_STAGES * (chunk_pack_floats(32 * DL, DELTA) + CHUNK * 32) + (DELTA ? 32 * CHUNK : 0)) * sizeof(float);
    static_assert(NEEDS <= CHUNK_ALONE, "shared memory of one block");
    // Sequences of several lengths go longest first: the first blocks get an SM each and, being the oldest there, its schedulers; in the order they came, the
    // longest may share an SM with its like.  16 heads of 128 x 256, 400 + 1,100 + 1,800 rows: 403 -> 351 us the whole call (before, the longest's blocks
    // alone 168 to 308 us), 64 heads of a delta rule 580 -> 528.
    // Where the longest sequence's chain is as long as all SMs' work, an SM to itself for every block of it (and for the others one at a time, through
    // the shared memory a block asks for): 16 heads of 128 x 256, sequences of 2,000 and three of 100 rows 347 -> 243 us the whole call, 8 heads, 400, 1,100 and 1,800 rows 227 -> 208;
    // not for 16 heads of the latter, half as much again for all SMs as for the longest, nor for two of 2,048 (382 and 452).
    const long long work = (long long)((P + 31) / 32) * H * rows;
    const size_t SMEM = seqs > 1 && work * 7 <= (long long)bc_sm_count() * max_new * 8 ? CHUNK_ALONE : NEEDS;
    auto launch = [&](auto long_first) {
        constexpr auto* kernel = chunk_scan_kernel<DL, DELTA, decltype(long_first)::value>;
        if (cudaError_t e = bc_allow_shared<kernel>(SMEM); e != cudaSuccess) return e;
        return bc_launch(kernel, dim3((P + 31) / 32, H, seqs), dim3(CHUNK_THREADS), SMEM, s, span, pack, v, v_stride, state, seq_rows, seq_slot, out, H, N, P, n_slots,
                         write_state, out_scale);
    };
    const bool mixed = seqs > 1 && seqs <= CHUNK_SORTED && (long long)rows < (long long)seqs * max_new;
    return mixed ? launch(std::true_type()) : launch(std::false_type());
}

// A step's chunks through `prepare` (the kernel that fills the pack) and the scan: at once where `capacity` chunks of scratch hold them, else
// segment by segment (at least one chunk a sequence, and the state must be written).
static inline bool chunk_fits(long long capacity, long long rows, long long seqs, int min_rows, int write_state) {
    return capacity >= chunk_places(rows, seqs, min_rows) || (write_state && capacity >= seqs);
}
// prepare(span, places): the kernel over the places that the span's chunks lie at; scan(span).
template <class Prepare, class Scan>
static cudaError_t chunk_step(long long capacity, int rows, int seqs, int max_new, int min_rows, Prepare prepare, Scan scan) {
    const int most = (max_new + CHUNK - 1) / CHUNK;
    const long long all = chunk_places(rows, seqs, min_rows);
    const bool whole = capacity >= all;
    const int segment = whole ? most : (int)(capacity / seqs < most ? capacity / seqs : most);
    cudaError_t e = cudaSuccess;
    for (int at = 0; at < most && e == cudaSuccess; at += segment) {
        const ChunkSpan span = {at, segment < most - at ? segment : most - at, whole ? 0 : segment, whole && chunk_crowded(rows, seqs, min_rows), min_rows};
        e = prepare(span, whole ? all : (long long)seqs * segment);
        if (e == cudaSuccess) e = scan(span);
    }
    return e;
}
