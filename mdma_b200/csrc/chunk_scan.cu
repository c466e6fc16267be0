// Prompts through the recurrences that are linear in their state: linear attention with a decay per head, and Mamba-2.
//
//     S_t = a_t S_(t-1) + k_t u_t^T,   o_t = S_t^T q_t          S [n][v] per head, all in float
//
//   linear attention   a_t = the head's decay, u = v; q, k, v: what `LinInput` makes of a projection row
//   Mamba-2            a_t = exp(-exp(A_log) dt_t), u = dt_t x, k = B, q = C (shared by the heads of a group), o += D x
//
// Every sequence is cut into chunks of 64 rows that are worked on side by side, in three launches:
//   chunk_sums    what a chunk adds to the state, sum_j (a_(j+1) .. a_last) k_j u_j^T, from zero;
//   chunk_starts  in order over the chunks: the state at every chunk's start, and the sequence's state at the end;
//   chunk_out     o_i = (a_0 .. a_i) S_start^T q_i + sum_(j <= i) (a_(j+1) .. a_i) (q_i . k_j) u_j.
// Bound by the float multiply-adds: 2 n v for every token and head, and about 64 (n + v) for the rows of its chunk, all of
// them in tiles of 4 x 4 (chunk_sums: 4 x 8) outputs a thread whose operands are read 16 bytes at a time, without bank
// conflicts, from rows that lie along the sum.  Chunks of 64: with 32 the states that travel between the launches are
// twice as many (64 KB a chunk and head of 128 x 128), with 128 the products inside a chunk are.  The blocks of Mamba-2
// take several heads each: C B^T is the same for all heads of a group and stays in registers.
//
// Measured against the runs of 128 (256) rows that walk their chunks one after another: linear attention, 1,500 rows, 16
// heads of 128 x 128, 209 -> 147 us (801 rows 112 -> 92); Mamba-2, 2,048 rows, 64 heads of 128 x 64, 560 -> 235 us (250 in
// a chain of calls; 801 rows 366 -> 100).  Of that chunk_out takes 95 (62) us, about half of the multiply-adds' rate: two blocks an SM are what the
// registers and the shared memory allow.
//
// States between the launches: `states` [sequence * max_chunks + chunk][head][v][n], and for Mamba-2 every chunk's whole
// decay behind them.
#include "rows_product.cuh"
#include "linear_input.cuh"

namespace mdma {

constexpr int kScanChunk = 64, kScanCols = 64, kScanThreads = 256;
constexpr int kScanPitch = kScanChunk + 4;          // of the rows of q k^T
constexpr int kScanMostN = 128, kScanMostHeads = 8;

struct ChunkScan {
    const int* seq_start; const int* seq_slot;
    float* state; size_t state_stride;
    float* states; float* decays;                   // decays: Mamba-2 only
    float* out;                                     // [rows][heads * vdim]
    int heads, n, vdim, max_chunks;
    int heads_per_block;                            // Mamba-2: a block's heads; else its parts of 64 columns of v
    // linear attention
    const void* proj; int row_stride, q_col, k_col, v_col;
    const float* decay;
    LinInput in;
    // Mamba-2: `conv` rows [x | B | C], the raw step sizes at dt + row * dt_stride + head
    const float* conv; int conv_stride, groups;
    const float* dt; int dt_stride;
    const void* dt_bias; const void* A_log; const void* D; int w_dtype;
};
__device__ __forceinline__ float scan_vector(const void* p, int dtype, int h) {
    return dtype == kF32 ? reinterpret_cast<const float*>(p)[h] : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[h]);
}
__device__ __forceinline__ float softplus_scan(float v) { return v > 20.0f ? v : log1pf(expf(v)); }
__host__ __device__ inline int scan_padded(int n) { return (n + 7) & ~7; }

__device__ __forceinline__ void scan_copy16(float* dst_shared, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst_shared)), "l"(src) : "memory");
}
__device__ __forceinline__ void scan_copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// rows 0 .. 63 of `width` numbers, `stride` apart, as float rows of `padded` numbers `pitch` apart; f(number, row); zeros
// from row n and from column `width` on
template <typename T, class F>
__device__ __forceinline__ void scan_fill(float* dst, int pitch, int padded, const T* __restrict__ src, size_t stride, int width, int n, F f) {
    const int quads = padded >> 2;
    const bool vec = rows_of_four(src, (long)stride, width);
#pragma unroll 4
    for (int e = threadIdx.x; e < kScanChunk * quads; e += kScanThreads) {
        const int i = e / quads, c = (e - i * quads) << 2;
        float4 v = i < n ? load4_of(src + i * stride, c, width, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n && c < width) { v.x = f(v.x, i); v.y = f(v.y, i); v.z = f(v.z, i); v.w = f(v.w, i); }
        if (c + 3 >= width) { if (c >= width) v.x = 0.f; if (c + 1 >= width) v.y = 0.f; if (c + 2 >= width) v.z = 0.f; if (c + 3 >= width) v.w = 0.f; }
        st4(dst + i * pitch + c, v);
    }
}
// the same of float rows as they are: copied without passing through registers where they lie on 16-byte boundaries (ask
// for `scan_copies_done` and a barrier before reading)
__device__ __forceinline__ void scan_fetch(float* dst, int pitch, int padded, const float* __restrict__ src, size_t stride, int width, int n) {
    if (!rows_of_four(src, (long)stride, width)) {
        scan_fill(dst, pitch, padded, src, stride, width, n, [](float z, int) { return z; });
        return;
    }
    const int quads = padded >> 2;
    for (int e = threadIdx.x; e < kScanChunk * quads; e += kScanThreads) {
        const int i = e / quads, c = (e - i * quads) << 2;
        if (i < n && c < width) scan_copy16(dst + i * pitch + c, src + i * stride + c);
        else st4(dst + i * pitch + c, make_float4(0.f, 0.f, 0.f, 0.f));
    }
}
// q or k rows turned by their positions where they lie
__device__ __forceinline__ void scan_rotate(float* q, float* k, int pitch, int t0, int n, const LinInput& in) {
    for (int e = threadIdx.x; e < n * in.half; e += kScanThreads) {
        const int i = e / in.half, p = e - i * in.half;
        const int d0 = in.interleaved ? 2 * p : p, d1 = in.interleaved ? 2 * p + 1 : p + in.half;
        float sn, cs;
        sincosf((float)in.tok_pos[t0 + i] * in.inv_freq[p], &sn, &cs);
        float* kr = k + i * pitch;
        const float a = kr[d0], b = kr[d1];
        kr[d0] = fmaf(a, cs, -(b * sn));
        kr[d1] = fmaf(b, cs, a * sn);
        if (q != nullptr) {
            float* qr = q + i * pitch;
            const float u = qr[d0], v = qr[d1];
            qr[d0] = fmaf(u, cs, -(v * sn));
            qr[d1] = fmaf(v, cs, u * sn);
        }
    }
}
// Mamba-2, one warp: step sizes of the chunk's rows (0 from row n on) and the running sums of the decays' logarithms.  The
// sums are made in double and kept as two floats: a decay between two rows is the exponential of a difference of sums that
// may be hundreds of times as large.
__device__ __forceinline__ void scan_steps(const ChunkScan& p, int h, int t0, int n, float* dt, float* cum, float* rest) {
    const int lane = threadIdx.x & 31;
    const float rate = expf(scan_vector(p.A_log, p.w_dtype, h)), bias = scan_vector(p.dt_bias, p.w_dtype, h);
    const float d0 = 2 * lane < n ? softplus_scan(p.dt[(size_t)(t0 + 2 * lane) * p.dt_stride + h] + bias) : 0.f;
    const float d1 = 2 * lane + 1 < n ? softplus_scan(p.dt[(size_t)(t0 + 2 * lane + 1) * p.dt_stride + h] + bias) : 0.f;
    const double a0 = -(double)rate * d0, a1 = -(double)rate * d1;
    double upto = a0 + a1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const double v = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += v; }
    // (from the rows before, not as upto - a1: a later row that is not finite must leave this one alone)
    const double before = __shfl_up_sync(0xffffffffu, upto, 1), first = (lane > 0 ? before : 0.0) + a0;
    dt[2 * lane] = d0; dt[2 * lane + 1] = d1;
    cum[2 * lane] = (float)first; rest[2 * lane] = (float)(first - (double)(float)first);
    cum[2 * lane + 1] = (float)upto; rest[2 * lane + 1] = (float)(upto - (double)(float)upto);
}
// the decay from behind row j to row i
__device__ __forceinline__ float scan_decay(const float* cum, const float* rest, int i, int j) {
    return expf((cum[i] - cum[j]) + (rest[i] - rest[j]));
}

struct ChunkRows { int seq, t0, n; };
__device__ __forceinline__ ChunkRows chunk_rows(const ChunkScan& p, int slot) {
    const int s = slot / p.max_chunks, c = slot - s * p.max_chunks;
    const int t0 = p.seq_start[s] + c * kScanChunk;
    return ChunkRows{s, t0, min(kScanChunk, p.seq_start[s + 1] - t0)};
}

// ---------------------------------------------------------------- what a chunk adds to the state
// Block = (chunk, heads_per_block heads, 64 columns of v); a thread owns 4 columns of v and two quads of n.  Mamba-2: B is
// fetched once for all heads, the next head's rows are on their way while a head is computed.
template <typename T, bool MAMBA>
__global__ void __launch_bounds__(kScanThreads, 3)
chunk_sums_kernel(const ChunkScan p) {
    chain_release();
    chain_wait();
    extern __shared__ __align__(16) float sm[];
    const ChunkRows at = chunk_rows(p, blockIdx.x);
    const int n = at.n;
    if (n <= 0) return;
    const int h0 = MAMBA ? blockIdx.y * p.heads_per_block : blockIdx.y;
    int c0 = (MAMBA ? blockIdx.z : blockIdx.z * p.heads_per_block) * kScanCols, cw = min(kScanCols, p.vdim - c0);
    const int NP = scan_padded(p.n), warp = threadIdx.x >> 5;
    float* k = sm;                                  // [64][NP]
    float* u = k + kScanChunk * NP;                 // [64][64], Mamba-2: twice
    float* weight = u + (MAMBA ? 2 : 1) * kScanChunk * kScanCols;      // [heads][64]
    float* cum = weight + (MAMBA ? kScanMostHeads : 1) * kScanChunk;   // Mamba-2: [heads][64], and the rests
    const float* conv = MAMBA ? p.conv + (size_t)at.t0 * p.conv_stride : nullptr;
    if (MAMBA) {
        scan_fetch(k, NP, NP, conv + p.heads * p.vdim + (h0 / (p.heads / p.groups)) * p.n, p.conv_stride, p.n, n);
        scan_fetch(u, kScanCols, kScanCols, conv + h0 * p.vdim + c0, p.conv_stride, cw, n);
        if (warp < p.heads_per_block) {
            float* w = weight + warp * kScanChunk;
            float* c = cum + warp * 2 * kScanChunk;
            scan_steps(p, h0 + warp, at.t0, n, w, c, c + kScanChunk);
            __syncwarp();
            for (int j = threadIdx.x & 31; j < kScanChunk; j += 32) w[j] *= scan_decay(c, c + kScanChunk, kScanChunk - 1, j);
            if ((threadIdx.x & 31) == 0 && blockIdx.z == 0) p.decays[(size_t)blockIdx.x * p.heads + h0 + warp] = expf(c[kScanChunk - 1] + c[2 * kScanChunk - 1]);
        }
    } else {
        if (threadIdx.x < kScanChunk) weight[threadIdx.x] = (int)threadIdx.x < n ? powf(p.decay[h0], (float)(n - 1 - (int)threadIdx.x)) : 0.f;
        const T* rows = reinterpret_cast<const T*>(p.proj) + (size_t)at.t0 * p.row_stride;
        const int silu = p.in.silu;
        const float k_scale = p.in.k_scale;
        scan_fill(k, NP, NP, rows + p.k_col + h0 * p.n, p.row_stride, p.n, n, [=](float z, int) { return lin_act(z, silu) * k_scale; });
        __syncthreads();
        scan_fill(u, kScanCols, kScanCols, rows + p.v_col + h0 * p.vdim + c0, p.row_stride, cw, n, [=](float z, int i) { return lin_act(z, silu) * weight[i]; });
        if (p.in.half > 0) scan_rotate(nullptr, k, NP, at.t0, n, p.in);
    }
    const int groups = NP >> 3;                     // pairs of quads of n: 4 g .. and NP / 2 + 4 g ..
    for (int hh = 0; hh < p.heads_per_block; ++hh) {
        float* v = u + (MAMBA ? (hh & 1) * kScanChunk * kScanCols : 0);
        if (!MAMBA && hh > 0) {                     // the next 64 columns
            c0 += kScanCols;
            if (c0 >= p.vdim) break;
            cw = min(kScanCols, p.vdim - c0);
            __syncthreads();
            const int silu = p.in.silu;
            scan_fill(u, kScanCols, kScanCols, reinterpret_cast<const T*>(p.proj) + (size_t)at.t0 * p.row_stride + p.v_col + h0 * p.vdim + c0, p.row_stride, cw, n,
                      [=](float z, int i) { return lin_act(z, silu) * weight[i]; });
        }
        if (MAMBA) {
            scan_copies_done();
            __syncthreads();
            if (hh + 1 < p.heads_per_block)
                scan_fetch(u + ((hh + 1) & 1) * kScanChunk * kScanCols, kScanCols, kScanCols, conv + (h0 + hh + 1) * p.vdim + c0, p.conv_stride, cw, n);
            const float* w = weight + hh * kScanChunk;
#pragma unroll
            for (int e = threadIdx.x; e < kScanChunk * kScanCols / 4; e += kScanThreads) {
                float4 x = ld4(v + 4 * e);
                scale4(x, w[e >> 4]);
                st4(v + 4 * e, x);
            }
        }
        __syncthreads();
        float* to = p.states + ((size_t)blockIdx.x * p.heads + (MAMBA ? h0 + hh : h0)) * p.vdim * p.n;
        for (int tile = threadIdx.x; tile < groups * (kScanCols / 4); tile += kScanThreads) {
            const int na = (tile % groups) << 2, nb = na + (NP >> 1), c = (tile / groups) << 2;
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int j = 0; j < n; ++j) {
                const float4 x = ld4(v + j * kScanCols + c), ka = ld4(k + j * NP + na), kb = ld4(k + j * NP + nb);
                fma4(a[0], x.x, ka); fma4(a[1], x.y, ka); fma4(a[2], x.z, ka); fma4(a[3], x.w, ka);
                fma4(b[0], x.x, kb); fma4(b[1], x.y, kb); fma4(b[2], x.z, kb); fma4(b[3], x.w, kb);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (c + i >= cw) break;
                float* row = to + (size_t)(c0 + c + i) * p.n;
                if ((p.n & 3) == 0) {
                    if (na < p.n) st4(row + na, a[i]);
                    if (nb < p.n) st4(row + nb, b[i]);
                } else {
                    const float va[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, vb[4] = {b[i].x, b[i].y, b[i].z, b[i].w};
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (na + e < p.n) row[na + e] = va[e];
                        if (nb + e < p.n) row[nb + e] = vb[e];
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------- the state at every chunk's start
// `states` holds every chunk's sum on entry and the state at its start on return; the sequence's state is brought up to
// date.  Bound by the memory that keeps the chunks' states (the second-level cache, for prompts of a few thousand rows): a
// thread owns one number and has eight chunks' loads in flight.
template <bool MAMBA>
__global__ void __launch_bounds__(256)
chunk_starts_kernel(const ChunkScan p) {
    chain_release();
    chain_wait();
    const size_t per_head = (size_t)p.vdim * p.n, all = per_head * p.heads;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int s = blockIdx.y;
    const int rows = p.seq_start[s + 1] - p.seq_start[s], chunks = (rows + kScanChunk - 1) / kScanChunk;
    if (e >= all || chunks <= 0) return;
    const int h = (int)(e / per_head);
    const int in_head = (int)(e - (size_t)h * per_head), v = in_head / p.n, d = in_head - v * p.n;
    // the sequence's state: Mamba-2 keeps [head][v][n], linear attention [head][n][v]
    float* st = p.state + (size_t)p.seq_slot[s] * p.state_stride + (size_t)h * per_head + (MAMBA ? (size_t)in_head : (size_t)d * p.vdim + v);
    float cur = *st;
    float* at = p.states + (size_t)s * p.max_chunks * all + e;
    const float* decays = MAMBA ? p.decays + (size_t)s * p.max_chunks * p.heads + h : nullptr;
    const float whole = MAMBA ? 0.f : powf(p.decay[h], (float)kScanChunk);
    const float last = MAMBA ? 0.f : powf(p.decay[h], (float)(rows - (chunks - 1) * kScanChunk));
    constexpr int U = 8;
    for (int c0 = 0; c0 < chunks; c0 += U) {
        float sum[U], decay[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool there = c0 + u < chunks;
            sum[u] = there ? at[(size_t)(c0 + u) * all] : 0.f;
            decay[u] = !there ? 0.f : MAMBA ? decays[(size_t)(c0 + u) * p.heads] : c0 + u == chunks - 1 ? last : whole;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (c0 + u >= chunks) break;
            at[(size_t)(c0 + u) * all] = cur;
            cur = fmaf(decay[u], cur, sum[u]);
        }
    }
    *st = cur;
}

// ---------------------------------------------------------------- a chunk's rows
// Sums are taken 16 terms at a time and those added up, so that their rounding does not grow with the length (one chain of
// 128 had twice the error of the row-by-row walk).
constexpr int kScanTerms = 16;
// acc[i][j] += sum_d a[row i][d] b[column j][d] for the thread's four rows (pitch pa) and NJ columns (16 apart, pitch pb)
template <int NJ>
__device__ __forceinline__ void scan_dots(float (&acc)[4][4], const float* a, int pa, const float* b, int pb, int len) {
    for (int d0 = 0; d0 < len; d0 += kScanTerms) {
        float2 part[4][NJ] = {};
        const int stop = min(len, d0 + kScanTerms);
#pragma unroll 2
        for (int d = d0; d < stop; d += 4) {
            float4 x[4], y[NJ];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = ld4(a + i * pa + d);
#pragma unroll
            for (int j = 0; j < NJ; ++j) y[j] = ld4(b + 16 * j * pb + d);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) dot4(part[i][j], x[i], y[j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) acc[i][j] += part[i][j].x + part[i][j].y;
    }
}
// acc[i][j] += sum_d a[row i][d] b[4 tx + j][d], b's rows of 128 numbers with their quads permuted (`scan_state_quad`)
__device__ __forceinline__ int scan_state_quad(int row, int quad) { return row * kScanMostN + 4 * (quad ^ ((row >> 2) & 7)); }
__device__ __forceinline__ void scan_dots_state(float (&acc)[4][4], const float* a, int pa, const float* b, int tx, int len) {
    const float* bt = b + 4 * tx * kScanMostN;
    const int turn = tx & 7;
    for (int d0 = 0; d0 < len; d0 += kScanTerms) {
        float2 part[4][4] = {};
        const int stop = min(len, d0 + kScanTerms);
#pragma unroll 2
        for (int d = d0; d < stop; d += 4) {
            const int at = 4 * ((d >> 2) ^ turn);
            float4 x[4], y[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = ld4(a + i * pa + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = ld4(bt + j * kScanMostN + at);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dot4(part[i][j], x[i], y[j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j].x + part[i][j].y;
    }
}

// Block = (chunk, heads_per_block heads, 64 columns of v).  Warp w owns rows 8 w .. 8 w + 7, so it needs the columns of
// q k^T and the rows of u up to 8 w + 7 only (a thread's rows take none beyond their own); a thread owns four neighbouring
// rows, of q k^T the columns tx, tx + 16, .., of the result the columns 4 tx .. 4 tx + 3.
template <typename T, bool MAMBA>
__global__ void __launch_bounds__(kScanThreads, 2)
chunk_out_kernel(const ChunkScan p) {
    chain_release();
    chain_wait();
    extern __shared__ __align__(16) float sm[];
    const ChunkRows at = chunk_rows(p, blockIdx.x);
    const int n = at.n;
    if (n <= 0) return;
    const int h0 = MAMBA ? blockIdx.y * p.heads_per_block : blockIdx.y;
    int c0 = (MAMBA ? blockIdx.z : blockIdx.z * p.heads_per_block) * kScanCols, cw = min(kScanCols, p.vdim - c0);
    const int NP = scan_padded(p.n), P = NP + 4;
    float* q = sm;                                  // [64][P]
    float* ks = q + kScanChunk * P;                 // k [64][P], then the state's columns [64 v][128]
    float* A = ks + max(kScanChunk * P, kScanCols * kScanMostN);      // [64][kScanPitch]
    float* u = A + kScanChunk * kScanPitch;         // [64][64]
    float* dt = u + kScanChunk * kScanCols;         // Mamba-2: [heads][step sizes 64 | sums 64 | rests 64]; else decay^0 .. decay^64
    const T* rows = MAMBA ? nullptr : reinterpret_cast<const T*>(p.proj) + (size_t)at.t0 * p.row_stride;
    const float* conv = MAMBA ? p.conv + (size_t)at.t0 * p.conv_stride : nullptr;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tx = lane & 15, row = 8 * warp + (lane >> 4) * 4;
    if (MAMBA) {
        const float* B = conv + p.heads * p.vdim + (h0 / (p.heads / p.groups)) * p.n;
        scan_fetch(ks, P, NP, B, p.conv_stride, p.n, n);
        scan_fetch(q, P, NP, B + p.groups * p.n, p.conv_stride, p.n, n);
        if (warp < p.heads_per_block) {
            float* mine = dt + warp * 3 * kScanChunk;
            scan_steps(p, h0 + warp, at.t0, n, mine, mine + kScanChunk, mine + 2 * kScanChunk);
        }
        scan_copies_done();
    } else {
        const int silu = p.in.silu;
        const float k_scale = p.in.k_scale;
        scan_fill(ks, P, NP, rows + p.k_col + h0 * p.n, p.row_stride, p.n, n, [=](float z, int) { return lin_act(z, silu) * k_scale; });
        scan_fill(q, P, NP, rows + p.q_col + h0 * p.n, p.row_stride, p.n, n, [=](float z, int) { return lin_act(z, silu); });
        scan_fill(u, kScanCols, kScanCols, rows + p.v_col + h0 * p.vdim + c0, p.row_stride, cw, n, [=](float z, int) { return lin_act(z, silu); });
        if (threadIdx.x <= kScanChunk) dt[threadIdx.x] = powf(p.decay[h0], (float)threadIdx.x);
        if (p.in.half > 0) {
            __syncthreads();
            scan_rotate(q, ks, P, at.t0, n, p.in);
        }
    }
    __syncthreads();
    float raw[4][4] = {};
    const int nj = (8 * warp + 7) / 16 + 1;
    if (nj == 1) scan_dots<1>(raw, q + row * P, P, ks + tx * P, P, NP);
    else if (nj == 2) scan_dots<2>(raw, q + row * P, P, ks + tx * P, P, NP);
    else if (nj == 3) scan_dots<3>(raw, q + row * P, P, ks + tx * P, P, NP);
    else scan_dots<4>(raw, q + row * P, P, ks + tx * P, P, NP);
    for (int hh = 0; hh < p.heads_per_block; ++hh) {
        const int h = MAMBA ? h0 + hh : h0;
        if (!MAMBA && hh > 0) {                     // the next 64 columns: q k^T stays
            c0 += kScanCols;
            if (c0 >= p.vdim) break;
            cw = min(kScanCols, p.vdim - c0);
        }
        __syncthreads();                            // k, or the state and u before these, are done with
        const float* S = p.states + ((size_t)blockIdx.x * p.heads + h) * p.vdim * p.n + (size_t)c0 * p.n;
        if ((p.n & 3) == 0) {
            const int quads = NP >> 2, full = p.n >> 2;
            for (int e = threadIdx.x; e < kScanCols * quads; e += kScanThreads) {
                const int c = e / quads, d = e - c * quads;
                if (c < cw && d < full) scan_copy16(ks + scan_state_quad(c, d), S + (size_t)c * p.n + 4 * d);
                else st4(ks + scan_state_quad(c, d), make_float4(0.f, 0.f, 0.f, 0.f));
            }
        } else {
            for (int e = threadIdx.x; e < kScanCols * NP; e += kScanThreads) {
                const int c = e / NP, d = e - c * NP;
                ks[scan_state_quad(c, d >> 2) + (d & 3)] = c < cw && d < p.n ? S[(size_t)c * p.n + d] : 0.f;
            }
        }
        if (MAMBA) {
            scan_fetch(u, kScanCols, kScanCols, conv + h * p.vdim + c0, p.conv_stride, cw, n);
        } else if (hh > 0) {
            const int silu = p.in.silu;
            scan_fill(u, kScanCols, kScanCols, rows + p.v_col + h * p.vdim + c0, p.row_stride, cw, n, [=](float z, int) { return lin_act(z, silu); });
        }
        const float* steps = MAMBA ? dt + hh * 3 * kScanChunk : dt;
        const float *cum = steps + kScanChunk, *rest = steps + 2 * kScanChunk;        // Mamba-2 only
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j >= nj || (!MAMBA && hh > 0)) break;
            const int c = tx + 16 * j;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = row + i;
                float f = 0.f;                      // (chosen, not multiplied: a later row may hold anything)
                if (c <= r) f = raw[i][j] * (MAMBA ? scan_decay(cum, rest, r, c) * steps[c] : steps[r - c]);
                A[r * kScanPitch + c] = f;
            }
        }
        scan_copies_done();
        __syncthreads();
        float acc[4][4] = {};
        scan_dots_state(acc, q + row * P, P, ks, tx, NP);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float start = MAMBA ? expf(cum[row + i] + rest[row + i]) : steps[row + i + 1];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] *= start;
        }
        // the thread's rows see the rows of u up to their own, no later one: 0 times a number that is not finite is not 0
        for (int j0 = 0; j0 < row + 4; j0 += kScanTerms) {
            float4 o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            const int stop = min(row, j0 + kScanTerms);
#pragma unroll 2
            for (int j = j0; j < stop; j += 4) {
                float4 x[4], y[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = ld4(A + (row + i) * kScanPitch + j);
#pragma unroll
                for (int e = 0; e < 4; ++e) y[e] = ld4(u + (j + e) * kScanCols + 4 * tx);
#pragma unroll
                for (int i = 0; i < 4; ++i) { fma4(o[i], x[i].x, y[0]); fma4(o[i], x[i].y, y[1]); fma4(o[i], x[i].z, y[2]); fma4(o[i], x[i].w, y[3]); }
            }
            if (row < j0 + kScanTerms) {            // the thread's own four rows
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float4 y = ld4(u + (row + e) * kScanCols + 4 * tx);
#pragma unroll
                    for (int i = e; i < 4; ++i) fma4(o[i], A[(row + i) * kScanPitch + row + e], y);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) { acc[i][0] += o[i].x; acc[i][1] += o[i].y; acc[i][2] += o[i].z; acc[i][3] += o[i].w; }
        }
        const float Dh = MAMBA ? scan_vector(p.D, p.w_dtype, h) : 0.f;
        const bool quads = (p.vdim & 3) == 0 && ((uintptr_t)p.out & 15) == 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = row + i;
            if (r >= n) break;
            float4 o = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            if (MAMBA) fma4(o, Dh, ld4(u + r * kScanCols + 4 * tx));
            float* to = p.out + (size_t)(at.t0 + r) * p.heads * p.vdim + (size_t)h * p.vdim + c0 + 4 * tx;
            if (quads) {
                if (4 * tx < cw) st4(to, o);
            } else {
                if (4 * tx < cw) to[0] = o.x;
                if (4 * tx + 1 < cw) to[1] = o.y;
                if (4 * tx + 2 < cw) to[2] = o.z;
                if (4 * tx + 3 < cw) to[3] = o.w;
            }
        }
    }
}

static size_t chunk_sums_smem(int n, bool mamba) {
    return sizeof(float) * ((size_t)kScanChunk * (scan_padded(n) + (mamba ? 2 : 1) * kScanCols) + (mamba ? 3 * kScanMostHeads : 1) * kScanChunk);
}
static size_t chunk_out_smem(int n, bool mamba) {
    const size_t k = (size_t)kScanChunk * (scan_padded(n) + 4), state = (size_t)kScanCols * kScanMostN;
    return sizeof(float) * (k + (k > state ? k : state) + (size_t)kScanChunk * (kScanPitch + kScanCols) + (mamba ? 3 * kScanMostHeads * kScanChunk : kScanChunk + 4));
}

template <typename T, bool MAMBA>
static int run_chunk_scan(ChunkScan p, int n_seqs, cudaStream_t stream) {
    const int parts = (p.vdim + kScanCols - 1) / kScanCols;
    const long slots = (long)n_seqs * p.max_chunks;
    const size_t sums_smem = chunk_sums_smem(p.n, MAMBA), out_smem = chunk_out_smem(p.n, MAMBA);
    cudaError_t e = cudaFuncSetAttribute(chunk_sums_kernel<T, MAMBA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sums_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_out_kernel<T, MAMBA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)out_smem);
    if (e != cudaSuccess) return fail("chunk_scan: cannot reserve shared memory: %s", cudaGetErrorString(e));
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // Mamba-2: up to eight heads of a group a block, as long as the blocks are three quarters of what the device holds of
    // them at once (two an SM)
    p.heads_per_block = 1;
    if (MAMBA)
        while (p.heads_per_block < kScanMostHeads && (p.heads / p.groups) % (2 * p.heads_per_block) == 0 &&
               2 * slots * (p.heads / (2 * p.heads_per_block)) * parts >= 3l * sms) p.heads_per_block *= 2;
    dim3 grid((unsigned)slots, p.heads / p.heads_per_block, parts);
    // Linear attention: a block takes all parts of v, so that q, k and their products are made once, unless that leaves more of
    // the last round of blocks empty (costs of a block of one part in the same units, by count of instructions)
    auto whole = [&](long at_once, double shared, double each) {
        const long blocks = slots * p.heads;
        auto rounds = [&](long n) { return (double)((n + at_once - 1) / at_once); };
        return rounds(blocks) * (shared + each * parts) <= rounds(blocks * parts) * (shared + each);
    };
    auto set_parts = [&](bool all_of_them) { p.heads_per_block = all_of_them ? parts : 1; grid = dim3((unsigned)slots, p.heads, all_of_them ? 1 : parts); };
    if (!MAMBA) set_parts(whole(3l * sms, 0.8, 2.6));
    launch_chained(chunk_sums_kernel<T, MAMBA>, grid, dim3(kScanThreads), sums_smem, stream, p);
    const size_t all = (size_t)p.heads * p.vdim * p.n;
    launch_chained(chunk_starts_kernel<MAMBA>, dim3((unsigned)((all + 255) / 256), n_seqs), dim3(256), 0, stream, p);
    if (!MAMBA) set_parts(whole(2l * sms, 2.9, 3.5));
    launch_chained(chunk_out_kernel<T, MAMBA>, grid, dim3(kScanThreads), out_smem, stream, p);
    MDMA_LAUNCH_OK("chunk_scan");
    return 0;
}

}  // namespace mdma

using namespace mdma;

extern "C" {

// Rows of a chunk; 0: heads of n x vdim do not fit these kernels.
int mdma_chunk_scan_rows(int n, int vdim) { return n >= 1 && n <= kScanMostN && vdim >= 1 ? kScanChunk : 0; }

// `states`: n_seqs * max_chunks * heads * n * vdim floats, 16-byte aligned.  The rest as in mdma_linear_attention.
int mdma_linear_attention_chunks(const void* proj, int dtype, int row_stride, int q_col, int k_col, int v_col, const float* decay,
                                 const int* seq_start, const int* seq_slot, float* state, long state_stride, float* out, int n_seqs,
                                 int heads, int dim, int vdim, int max_chunks, float* states, long states_floats, int silu,
                                 int rotary_dim, int interleaved, const float* inv_freq, const int* tok_pos, float k_scale,
                                 cudaStream_t stream) {
    MDMA_REQUIRE(rotary_dim >= 0 && rotary_dim % 2 == 0 && rotary_dim <= dim && (rotary_dim == 0 || (inv_freq && tok_pos)),
                 "linear_attention: %d turned numbers of a head of %d", rotary_dim, dim);
    MDMA_REQUIRE(n_seqs >= 0 && n_seqs <= 65535 && heads > 0 && heads <= 65535 && mdma_chunk_scan_rows(dim, vdim) > 0 && max_chunks >= 1 &&
                 (vdim + kScanCols - 1) / kScanCols <= 65535, "linear_attention: bad sizes");
    if (n_seqs == 0) return 0;
    const long need = (long)n_seqs * max_chunks * heads * dim * vdim;
    MDMA_REQUIRE(states != nullptr && ((uintptr_t)states & 15) == 0 && states_floats >= need && (long)n_seqs * max_chunks <= 65535l * 32,
                 "linear_attention: %ld floats of scratch needed, %ld given", need, states_floats);
    ChunkScan p = {};
    p.seq_start = seq_start; p.seq_slot = seq_slot; p.state = state; p.state_stride = (size_t)state_stride; p.states = states; p.out = out;
    p.heads = heads; p.n = dim; p.vdim = vdim; p.max_chunks = max_chunks;
    p.proj = proj; p.row_stride = row_stride; p.q_col = q_col; p.k_col = k_col; p.v_col = v_col; p.decay = decay;
    p.in = LinInput{silu, rotary_dim / 2, interleaved, k_scale, inv_freq, tok_pos};
    MDMA_DISPATCH_DTYPE(dtype, T, { return (run_chunk_scan<T, false>(p, n_seqs, stream)); });
    return 0;
}

// `states`: n_seqs * max_chunks * (heads * N * vdim + heads) floats, 16-byte aligned.  The rest as in mdma_mamba2_scan.
int mdma_mamba2_chunks(const float* conv, int conv_stride, const float* proj, int proj_stride, int dt_col, const void* dt_bias,
                       const void* A_log, const void* D, int w_dtype, const int* seq_start, const int* seq_slot, float* state,
                       long state_stride, float* y, int n_seqs, int heads, int vdim, int N, int G, int max_chunks, float* states,
                       long states_floats, cudaStream_t stream) {
    MDMA_REQUIRE(heads > 0 && heads <= 65535 && G > 0 && heads % G == 0 && mdma_chunk_scan_rows(N, vdim) > 0 && max_chunks >= 1 &&
                 n_seqs >= 0 && n_seqs <= 65535 && (vdim + kScanCols - 1) / kScanCols <= 65535, "mamba2_scan: bad geometry");
    MDMA_REQUIRE(w_dtype == kF32 || w_dtype == kBF16, "mamba2_scan: unknown dtype %d", w_dtype);
    MDMA_REQUIRE(state_stride >= (long)heads * N * vdim, "mamba2_scan: the state rows are too short");
    if (n_seqs == 0) return 0;
    const long slots = (long)n_seqs * max_chunks, state_floats = (long)heads * N * vdim;
    MDMA_REQUIRE(states != nullptr && ((uintptr_t)states & 15) == 0 && states_floats >= slots * (state_floats + heads) && slots <= 65535l * 16,
                 "mamba2_scan: %ld chunks need %ld floats of scratch, %ld given", slots, slots * (state_floats + heads), states_floats);
    ChunkScan p = {};
    p.seq_start = seq_start; p.seq_slot = seq_slot; p.state = state; p.state_stride = (size_t)state_stride; p.states = states;
    p.decays = states + slots * state_floats; p.out = y;
    p.heads = heads; p.n = N; p.vdim = vdim; p.max_chunks = max_chunks;
    p.conv = conv; p.conv_stride = conv_stride; p.groups = G; p.dt = proj + dt_col; p.dt_stride = proj_stride;
    p.dt_bias = dt_bias; p.A_log = A_log; p.D = D; p.w_dtype = w_dtype;
    return run_chunk_scan<float, true>(p, n_seqs, stream);
}

}  // extern "C"
