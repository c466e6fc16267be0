// Matrix products on the CUDA cores, sum_k A[m, k] * W[n, k], in two shapes that give the same bits.
//
// Order of additions of every output, whatever the shape, the number of rows or the way the operands lie in memory:
// the products of each run of 16 values of k are summed from zero, the runs' sums of each quarter of K (a whole number
// of runs) are added up in order, then the four quarters.  A row's result therefore does not depend on how many other
// rows are in the call, the chains of roundings are short (16, K / 64 and 4 long), and four groups of threads can walk
// the four quarters side by side.
//
//   few_rows_product  up to 8 rows.  Bound by reading W once: a thread holds one run (16 values, 64 bytes) of two rows
//                     of W in registers, loaded before the rows of A are there, and multiplies it with all rows of A
//                     out of shared memory; the runs' sums meet in shared memory.
//                     Measured, 1,024 x 1,024 floats: 4 rows 3.3 us (a tile of 64 rows x 64 features walked by one block
//                     without anything on its way took 67), 8 rows 4.5.
//   few_rows_stream   the same for float matrices of K up to 1,024 that are larger than what the blocks hold at once: a block
//                     walks over groups of features, the next groups' rows on their way by cp.async in two stages of shared
//                     memory (laid out for a thread's run, while the loads are of whole lines).  Measured, 4 rows x 32,000 x 1,024: 34 us, a block a group 50.
//   tile_product      32 rows x 32 rows of W per block of 256 threads.  Bound by the fused multiply-adds: each quarter
//                     of K belongs to 64 threads (4 x 4 outputs each, 16 multiply-adds for two 16-byte shared-memory
//                     reads); float rows have three runs on their way while one is computed.
#pragma once
#include "common.cuh"
#include "float4.cuh"

namespace mdma {

enum RowsShape : int { kTile = 0, kFew = 1, kStream = 2 };
constexpr int kRun = 16;                       // values of k summed from zero
constexpr int kFewRows = 8;                    // rows of A of one few_rows_product
constexpr int kTileRows = 32, kTileFeats = 32; // of one tile_product
constexpr int kRunPitch = 20;                  // floats from one row's run to the next in shared memory (16-byte reads without bank conflicts)
constexpr int kRowsThreads = 256;

__device__ __forceinline__ float4 load4(const float* p) { return ld4(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
// four values from p[k..], zeros from K on; `vec`: K is a multiple of 4 and every row starts on a four-element boundary
template <typename T>
__device__ __forceinline__ float4 load4_of(const T* p, int k, int K, bool vec) {
    if (p == nullptr || k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) return load4(p + k);
    return make_float4(to_float(p[k]), k + 1 < K ? to_float(p[k + 1]) : 0.f, k + 2 < K ? to_float(p[k + 2]) : 0.f,
                       k + 3 < K ? to_float(p[k + 3]) : 0.f);
}
template <typename T>
__device__ __forceinline__ bool rows_of_four(const T* p, long stride, int K) {
    return K % 4 == 0 && stride % 4 == 0 && ((uintptr_t)p & (4 * sizeof(T) - 1)) == 0;
}
__device__ __forceinline__ int quarter_runs(int K) { return ((K + kRun - 1) / kRun + 3) / 4; }

// How many runs of K a block of few_rows_product takes at a time (a power of two); the block covers 256 / that pairs of
// rows of W.  32 where K has no more (all threads have work), else 64.
__host__ __device__ inline int few_rows_chunk(int K) { return (K + kRun - 1) / kRun <= 32 ? 32 : 64; }
// features per block: a pair is two features, or one feature of the two matrices of a gated product
__host__ __device__ inline int few_rows_features(int K, bool dual) { return kRowsThreads / few_rows_chunk(K) * (dual ? 1 : 2); }
constexpr int kFewRowsSmem = kFewRows * 64 * kRun;        // floats: the rows of A (64 runs of 8 rows), then the runs' sums

// rows of A: row_of(m) for m < rows (called after `arrived()`); store(m, f, sum, sum2) is called by one thread for each
// m < rows and feature f0 <= f < N of this block.  All 256 threads call this together; `smem` is kFewRowsSmem floats.
template <typename TA, typename TW, bool DUAL, class RowOf, class Arrived, class Store>
__device__ __forceinline__ void few_rows_product(int rows, RowOf row_of, const TW* __restrict__ W, const TW* __restrict__ W2,
                                                 int f0, int N, int K, bool vec_a, bool vec_w, float* smem,
                                                 Arrived arrived, Store store) {
    const int chunk = few_rows_chunk(K), t = threadIdx.x;
    const int run_l = t & (chunk - 1), pair = t / chunk, pairs = kRowsThreads / chunk;
    const int R = (K + kRun - 1) / kRun, q = quarter_runs(K);
    const int fa = DUAL ? f0 + pair : f0 + 2 * pair, fb = DUAL ? fa : fa + 1;
    const TW* wa = fa < N ? W + (size_t)fa * K : nullptr;
    const TW* wb = fb < N ? (DUAL ? W2 : W) + (size_t)fb * K : nullptr;
    float4 a[4], b[4];
    auto load_w = [&](int c0) {
        const int k = (c0 + run_l) * kRun;
#pragma unroll
        for (int i = 0; i < 4; ++i) { a[i] = load4_of(wa, k + 4 * i, K, vec_w); b[i] = load4_of(wb, k + 4 * i, K, vec_w); }
    };
    load_w(0);
    arrived();
    // sums by (row of W in the block, row of A, quarter): 256 of them, 512 with chunks of 32 runs
    const int sums = 2 * pairs * kFewRows * 4;
    float acc[2] = {0.f, 0.f};
    for (int c0 = 0; c0 < R; c0 += chunk) {
        // the rows' runs lie 64 bytes apart; a run's four quads are permuted so that eight threads read eight runs at once
        for (int i = t; i < rows * chunk * 4; i += kRowsThreads) {
            const int m = i / (chunk * 4), at = i - m * chunk * 4, run = at >> 2, quad = at & 3;
            st4(smem + (m * chunk + run) * kRun + 4 * (quad ^ ((run >> 1) & 3)), load4_of(row_of(m), (c0 + run) * kRun + 4 * quad, K, vec_a));
        }
        __syncthreads();
        float pa[kFewRows], pb[kFewRows];
#pragma unroll
        for (int m = 0; m < kFewRows; ++m) {
            if (m >= rows) break;
            const float* x = smem + (m * chunk + run_l) * kRun;
            float sa = 0.f, sb = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = ld4(x + 4 * (i ^ ((run_l >> 1) & 3)));
                sa = dot4(v, a[i], sa);
                sb = dot4(v, b[i], sb);
            }
            pa[m] = sa; pb[m] = sb;
        }
        if (c0 + chunk < R) load_w(c0 + chunk);
        __syncthreads();
        // [row of W][row of A][run]
#pragma unroll
        for (int m = 0; m < kFewRows; ++m) {
            if (m >= rows) break;
            smem[((2 * pair) * kFewRows + m) * (chunk + 1) + run_l] = pa[m];
            smem[((2 * pair + 1) * kFewRows + m) * (chunk + 1) + run_l] = pb[m];
        }
        __syncthreads();
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const int i = t + s * kRowsThreads;
            if (i >= sums || ((i >> 2) & (kFewRows - 1)) >= rows) continue;
            const float* p = smem + (i >> 2) * (chunk + 1);
            const int lo = max((i & 3) * q, c0) - c0, hi = min(min(((i & 3) + 1) * q, R), c0 + chunk) - c0;
            for (int r = lo; r < hi; ++r) acc[s] += p[r];
        }
        __syncthreads();
    }
    float* total = smem;                       // [row of W][row of A]
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int i = t + s * kRowsThreads;
        const float v1 = __shfl_down_sync(0xffffffffu, acc[s], 1), v2 = __shfl_down_sync(0xffffffffu, acc[s], 2);
        const float v3 = __shfl_down_sync(0xffffffffu, acc[s], 3);
        if (i < sums && (i & 3) == 0) total[i >> 2] = ((acc[s] + v1) + v2) + v3;
    }
    __syncthreads();
    const int feats = DUAL ? pairs : 2 * pairs;
    for (int i = t; i < feats * rows; i += kRowsThreads) {
        const int f = i % feats, m = i / feats;
        if (f0 + f >= N) continue;
        if (DUAL) store(m, f0 + f, total[2 * f * kFewRows + m], total[(2 * f + 1) * kFewRows + m]);
        else store(m, f0 + f, total[f * kFewRows + m], 0.f);
    }
}

// ---- the same, streaming -----------------------------------------------------------------------------------------------
constexpr int kStreamStage = 2 * kRowsThreads * kRun;     // floats of a stage: two rows' runs a thread
constexpr int kStreamMaxK = 64 * kRun;
// shared memory: two stages, the rows of A, the runs' sums (2 pairs x rows x (chunk + 1)), their totals
__host__ __device__ inline int few_rows_stream_floats(int rows, int K) {
    const int chunk = few_rows_chunk(K);
    return 2 * kStreamStage + rows * chunk * kRun + 2 * (kRowsThreads / chunk) * (rows * (chunk + 1) + kFewRows) + 64;
}
// Whether a product of float matrices takes this form on so many blocks: their rows lie on 16 bytes, there are two groups a block,
// and a block's two stages carry enough of W.  A stage is as long as a chunk of runs, whatever K leaves empty of it, so one matrix
// streams from 2.75 full stages a block on, or where K fills the chunk; two matrices always (they are half of the groups).
// us, a block a group / streamed, 1 and 5 rows: 14,000 x 128 6.9 / 9.1, 9.9 / 11.0, x 384 8.4 / 9.7, 11.3 / 11.5, x 512 9.7 / 9.7,
// 12.8 / 11.7; 20,000 x 256 11.0 / 12.3, 15.4 / 14.3, x 384 13.4 / 12.7, 17.9 / 15.2; 32,000 x 64 14.3 / 14.6, 20.4 / 21.4, x 256
// 17.3 / 14.7, 23.4 / 21.9; 4,736 x 768 5.6 / 6.1, 8.7 / 8.5, 4,800 x 1,024 7.3 / 7.2, 11.0 / 9.4; gated 9,472 x 64 9.2 / 8.2, 13.0 / 12.3.
static inline bool few_rows_streams(const void* W, const void* W2, int N, int K, bool dual, int blocks) {
    if (K > kStreamMaxK || K % 4 != 0 || (((uintptr_t)W | (uintptr_t)W2) & 15) != 0) return false;
    const int feats = few_rows_features(K, dual);
    if ((N + feats - 1) / feats < 2 * blocks) return false;
    return dual || 32 * ((K + kRun - 1) / kRun) >= 31 * few_rows_chunk(K) || 4l * N * K >= 11l * blocks * kStreamStage;
}

// As few_rows_product for the groups of features `group`, `group` + `groups`, ..; the same sums in the same order.  Where the rows of
// A, the sums and the totals lie in `smem` depends on `rows`: a barrier belongs between two calls in one block, and W is asked
// for before `arrived()`, so its address may not depend on anything that the kernel in front writes.
template <typename TA, bool DUAL, class RowOf, class Arrived, class Store>
__device__ __forceinline__ void few_rows_stream(int rows, RowOf row_of, const float* __restrict__ W, const float* __restrict__ W2,
                                                int group, int groups, int N, int K, bool vec_a, float* smem, Arrived arrived, Store store) {
    const int chunk = few_rows_chunk(K), t = threadIdx.x;
    const int run_l = t & (chunk - 1), pair = t / chunk, pairs = kRowsThreads / chunk, feats = DUAL ? pairs : 2 * pairs;
    const int R = (K + kRun - 1) / kRun, q = quarter_runs(K), turn = (run_l >> 1) & 3;
    float* const rows_a = smem + 2 * kStreamStage;
    float* const run_sums = rows_a + rows * chunk * kRun;            // [row of W][row of A][run]
    float* const total = run_sums + 2 * pairs * rows * (chunk + 1);  // [row of W][row of A of kFewRows]
    auto issue = [&](int f0, int stage) {
        float* to = smem + stage * kStreamStage;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int i = t + x * kRowsThreads, r = i / (chunk * 4), at = i - r * chunk * 4, run = at >> 2, quad = at & 3, k = run * kRun + 4 * quad;
            const int f = DUAL ? f0 + (r >> 1) : f0 + r;
            const bool there = f < N && k < K;
            const float* src = there ? (DUAL && (r & 1) ? W2 : W) + (size_t)f * K + k : W;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to + (r * chunk + run) * kRun + 4 * (quad ^ ((run >> 1) & 3)))),
                         "l"(src), "r"(there ? 16 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int step = groups * feats;
    issue(group * feats, 0);
    issue(group * feats + step, 1);
    arrived();
    for (int i = t; i < rows * chunk * 4; i += kRowsThreads) {
        const int m = i / (chunk * 4), at = i - m * chunk * 4, run = at >> 2, quad = at & 3;
        st4(rows_a + (m * chunk + run) * kRun + 4 * (quad ^ ((run >> 1) & 3)), load4_of(row_of(m), run * kRun + 4 * quad, K, vec_a));
    }
    for (int f0 = group * feats, stage = 0; f0 < N; f0 += step, stage ^= 1) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* wa = smem + stage * kStreamStage + (2 * pair * chunk + run_l) * kRun;
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { a[i] = ld4(wa + 4 * (i ^ turn)); b[i] = ld4(wa + chunk * kRun + 4 * (i ^ turn)); }
#pragma unroll
        for (int m = 0; m < kFewRows; ++m) {
            if (m >= rows) break;
            const float* x = rows_a + (m * chunk + run_l) * kRun;
            float sa = 0.f, sb = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = ld4(x + 4 * (i ^ turn));
                sa = dot4(v, a[i], sa);
                sb = dot4(v, b[i], sb);
            }
            run_sums[(2 * pair * rows + m) * (chunk + 1) + run_l] = sa;
            run_sums[((2 * pair + 1) * rows + m) * (chunk + 1) + run_l] = sb;
        }
        __syncthreads();
        issue(f0 + 2 * step, stage);
        // a quarter of K a thread: (row of W, row of A, quarter)
        for (int i = t; i < 2 * pairs * rows * 4; i += kRowsThreads) {
            const float* p = run_sums + (i >> 2) * (chunk + 1);
            const int lo = (i & 3) * q, hi = min(((i & 3) + 1) * q, R);
            float acc = 0.f;
            for (int r = lo; r < hi; ++r) acc += p[r];
            const float v1 = __shfl_down_sync(0xffffffffu, acc, 1), v2 = __shfl_down_sync(0xffffffffu, acc, 2), v3 = __shfl_down_sync(0xffffffffu, acc, 3);
            if ((i & 3) == 0) total[(i >> 2) / rows * kFewRows + (i >> 2) % rows] = ((acc + v1) + v2) + v3;
        }
        __syncthreads();
        for (int i = t; i < feats * rows; i += kRowsThreads) {
            const int f = i % feats, m = i / feats;
            if (f0 + f >= N) continue;
            if (DUAL) store(m, f0 + f, total[2 * f * kFewRows + m], total[(2 * f + 1) * kFewRows + m]);
            else store(m, f0 + f, total[f * kFewRows + m], 0.f);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

constexpr int kTileStages = 4;                 // runs of a quarter on their way or being computed
constexpr int kTileBuf = (kTileRows + kTileFeats) * kRunPitch;
constexpr int kTileSmemBytes = 4 * kTileStages * kTileBuf * (int)sizeof(float);

// Rows row_of(0 .. 31) (null: none) times 32 rows of W from f0 on; gated products: 16 features of both matrices.
// `smem` is kTileSmemBytes; all 256 threads call this together.
template <typename TA, typename TW, bool DUAL, class RowOf, class Store>
__device__ __forceinline__ void tile_product(int rows, RowOf row_of, const TW* __restrict__ W, const TW* __restrict__ W2,
                                             int f0, int N, int K, bool vec_a, bool vec_w, float* smem, Store store) {
    const int quarter = threadIdx.x >> 6, u = threadIdx.x & 63, tx = u & 7, ty = u >> 3;
    const int R = (K + kRun - 1) / kRun, q = quarter_runs(K);
    const int lo = quarter * q, hi = min(lo + q, R);
    float* mine = smem + quarter * kTileStages * kTileBuf;
    // thread u fills quad u & 3 of rows u / 4 and 16 + u / 4 of either operand
    const int quad = u & 3, lr = u >> 2;
    const TA* src_a[2];
    const TW* src_w[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        src_a[i] = lr + 16 * i < rows ? row_of(lr + 16 * i) : nullptr;
        const int f = DUAL ? f0 + lr : f0 + lr + 16 * i;
        src_w[i] = f < N ? (DUAL && i == 1 ? W2 : W) + (size_t)f * K : nullptr;
    }
    float acc[4][4] = {};
    auto compute = [&](const float* buf) {
        float part[4][4] = {};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            float4 a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = ld4(buf + (ty + 8 * i) * kRunPitch + 4 * kk);
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = ld4(buf + (kTileRows + tx + 8 * j) * kRunPitch + 4 * kk);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j] = dot4(a[i], w[j], part[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
    };
    auto meet = [&] { asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); };       // this quarter's 64 threads
    if (sizeof(TA) == 4 && sizeof(TW) == 4 && vec_a && vec_w) {
        // float rows on 16-byte boundaries: three runs on their way (cp.async; what is beyond a matrix arrives as zeros)
        auto copy = [&](float* dst, const void* src) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                         "l"(src != nullptr ? src : (const void*)W), "r"(src != nullptr ? 16 : 0) : "memory");
        };
        auto issue = [&](int run) {
            if (run < hi) {
                float* buf = mine + ((run - lo) % kTileStages) * kTileBuf;
                const int k = run * kRun + 4 * quad;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    copy(buf + (lr + 16 * i) * kRunPitch + 4 * quad, src_a[i] != nullptr && k < K ? src_a[i] + k : nullptr);
                    copy(buf + (kTileRows + lr + 16 * i) * kRunPitch + 4 * quad, src_w[i] != nullptr && k < K ? src_w[i] + k : nullptr);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int s = 0; s < kTileStages - 1; ++s) issue(lo + s);
        for (int run = lo; run < hi; ++run) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kTileStages - 2) : "memory");
            meet();                            // this run is there for everyone, the one before it is done with
            issue(run + kTileStages - 1);
            compute(mine + ((run - lo) % kTileStages) * kTileBuf);
        }
    } else {
        float4 na[2], nw[2];
        auto fetch = [&](int run) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                na[i] = load4_of(src_a[i], run * kRun + 4 * quad, K, vec_a);
                nw[i] = load4_of(src_w[i], run * kRun + 4 * quad, K, vec_w);
            }
        };
        if (lo < hi) fetch(lo);
        for (int run = lo; run < hi; ++run) {
            float* buf = mine + ((run - lo) & 1) * kTileBuf;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                st4(buf + (lr + 16 * i) * kRunPitch + 4 * quad, na[i]);
                st4(buf + (kTileRows + lr + 16 * i) * kRunPitch + 4 * quad, nw[i]);
            }
            meet();
            if (run + 1 < hi) fetch(run + 1);
            compute(buf);
        }
    }
    __syncthreads();
    float* sums = smem;                        // [quarter][16 outputs][64 threads]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sums[(quarter * 16 + i * 4 + j) * 64 + u] = acc[i][j];
    __syncthreads();
    float r[4];                                // this quarter's threads finish the rows ty + 8 * quarter
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float* s = sums + (quarter * 4 + j) * 64 + u;
        r[j] = ((s[0] + s[16 * 64]) + s[32 * 64]) + s[48 * 64];
    }
    const int m = ty + 8 * quarter;
    if (m < rows) {
#pragma unroll
        for (int j = 0; j < (DUAL ? 2 : 4); ++j) {
            const int f = f0 + tx + 8 * j;
            if (f < N) store(m, f, r[j], DUAL ? r[j + 2] : 0.f);
        }
    }
}

// Blocks of few_rows_stream that the device holds: two an SM (115,456 bytes each at most, with eight rows of A and 1,024 of K).
static inline int few_rows_stream_blocks() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return 2 * (sms > 0 ? sms : 1);
}
template <class Kernel>
static inline size_t few_rows_stream_smem(Kernel kernel, int rows, int K) {
    const int bytes = few_rows_stream_floats(rows < kFewRows ? rows : kFewRows, K) * (int)sizeof(float);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, few_rows_stream_floats(kFewRows, kStreamMaxK) * (int)sizeof(float));
    return bytes;
}

// The shared memory of a kernel made of either, which is allowed to it (per launch: the attribute belongs to the device).
template <class Kernel>
static inline size_t rows_product_smem(Kernel kernel, bool few) {
    if (few) return kFewRowsSmem * sizeof(float);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmemBytes);
    return kTileSmemBytes;
}

}  // namespace mdma
