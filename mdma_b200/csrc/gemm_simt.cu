// Matrix products on the CUDA cores: out[m,n] = sum_k A[m,k] * W[n,k].
//
// This is the product of the true 32-bit engine (float inputs, float FMA, no
// reduced-precision matrix mode) and the fallback of the bfloat16 engine for
// shapes the tensor-core kernel refuses.  The order of additions is that of
// rows_product.cuh: one order for every shape, so a row's result does not
// depend on how many other rows are in the call.
#include <type_traits>

#include "rows_product.cuh"

namespace mdma {

// The blocks that stream W are the faster ones for up to 8 rows, and beyond as long as (rows of the matrices) x (passes of 8
// rows of A) is small, since every pass reads W again (from the second-level cache).  Up to K = 512, where a block takes 16 rows
// of the matrices: 9,216, nearly what four blocks an SM hold; beyond, with 8 rows a block: 8,192 for two passes, 6,144 for
// more (a second round of blocks, which costs less than a second row of tiles).  Both give the same bits.  Measured in a
// graph, few against tile, us: K 512, 1,024 rows of the matrix x 64 rows of A (8,192) 8.8 / 10.3, 1,536 x 48 (9,216) 9.1 / 11.1,
// 1,024 x 80 (10,240) 12.4 / 11.1; K 768, 1,536 x 24 (4,608) 10.2 / 10.8, x 32 (6,144) 14.8 / 11.0, x 40 (7,680) 19.0 / 15.7;
// K 1,024, 1,024 x 32 (4,096) 10.3 / 13.9, x 48 (6,144) 15.2 / 18.4, x 56 (7,168) 18.4 / 18.4, x 64 (8,192) 20.0 / 18.0,
// 2,048 x 24 (6,144) 15.2 / 17.9, x 32 20.0 / 17.7, 4,096 x 16 (two passes, 8,192) 19.0 / 20.3; K 4,096, 1,024 x 48 58.3 / 65.0,
// x 64 77.0 / 62.3; gated, K 1,024, 1,024 x 24 (6,144) 15.8 / 17.2, x 32 20.7 / 17.8, 2,048 x 16 (two passes, 8,192) 19.7 / 20.3.
inline long few_rows_limit(int K, long passes) { return few_rows_chunk(K) == 32 ? 9216 : passes == 2 ? 8192 : 6144; }

enum GemmMode : int {
    kStore = 0,        // out = acc
    kAccumulate = 1,   // out += acc        (the residual stream, float)
    kSwiGLU = 2,       // out = act(acc_gate) * acc_up, with a second weight (act: SiLU or GELU)
    kStoreAct = 3,     // out = act(acc): a feed-forward without a gate
};

// SHAPE: blocks of up to 8 rows that stream W (kFew: a group of features each, kStream: one group after another); else tiles
// of 32 rows.
template <typename TA, typename TW, typename TO, int MODE, int SHAPE>
__global__ void __launch_bounds__(kRowsThreads)
gemm_nt_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, const TW* __restrict__ W2,
               TO* __restrict__ out, int ldo, int M, int N, int K, const Ending e,
               long batch_a, long batch_w, long batch_o, int w_fixed) {
    constexpr bool kDual = MODE == kSwiGLU, FEW = SHAPE != kTile;
    extern __shared__ __align__(16) float smem[];
    chain_release();
    // blockIdx.z: one of several products of the same sizes (a head each), operands `batch_*` elements apart
    A += (size_t)blockIdx.z * batch_a;
    W += (size_t)blockIdx.z * batch_w;
    if (kDual) W2 += (size_t)blockIdx.z * batch_w;
    out += (size_t)blockIdx.z * batch_o;
    constexpr int kRows = FEW ? kFewRows : kTileRows;
    const bool vec_a = rows_of_four(A, lda, K), vec_w = rows_of_four(W, K, K) && (!kDual || rows_of_four(W2, K, K));
    // A matrix that no kernel on its way can write (a model's weight) is asked for while the kernel before this one ends: 4 % of
    // a generation of the 32-bit engine.
    if (!FEW || !w_fixed) chain_wait();
    for (int m0 = blockIdx.y * kRows; m0 < M; m0 += gridDim.y * kRows) {
        const int rows = min(kRows, M - m0);
        auto row_of = [&](int m) { return A + (size_t)(m0 + m) * lda; };
        auto store = [&](int m, int n, float acc, float acc2) {
            TO* o = out + (size_t)(m0 + m) * ldo + n;
            const float r = acc + ending_bias(e.bias, e.bias_dtype, n);
            if (MODE == kStore) *o = from_float<TO>(r);
            else if (MODE == kAccumulate) *o = from_float<TO>(to_float(*o) + r);
            else if (MODE == kStoreAct) *o = from_float<TO>(gate_activation(r, e.act));
            else *o = from_float<TO>(gated_pair(r, acc2 + ending_bias(e.bias2, e.bias_dtype, n), e.act, e.act_limit, e.act_alpha));
        };
        if constexpr (SHAPE == kStream)
            few_rows_stream<TA, kDual>(rows, row_of, W, W2, blockIdx.x, gridDim.x, N, K, vec_a, smem, [] { chain_wait(); }, store);
        else if (FEW) few_rows_product<TA, TW, kDual>(rows, row_of, W, W2, blockIdx.x * few_rows_features(K, kDual), N, K, vec_a, vec_w,
                                                 smem, [] { chain_wait(); }, store);
        else tile_product<TA, TW, kDual>(rows, row_of, W, W2, blockIdx.x * (kDual ? kTileFeats / 2 : kTileFeats), N, K, vec_a, vec_w, smem, store);
        __syncthreads();
    }
}

template <typename TA, typename TW, typename TO, int MODE>
static void launch_mode(const void* A, int lda, const void* W, const void* W2, void* out, int ldo, int M, int N, int K,
                        const Ending& e, int w_fixed, cudaStream_t stream, int batch, long batch_a, long batch_w, long batch_o) {
    constexpr bool kDual = MODE == kSwiGLU;
    const long passes = (M + kFewRows - 1) / kFewRows;
    const bool few = passes == 1 || (long)N * (kDual ? 2 : 1) * passes <= few_rows_limit(K, passes);
    const auto launch = [&](auto kernel, int rows, int across, size_t smem) {
        launch_chained(kernel, dim3(across, min((M + rows - 1) / rows, 65535), batch), dim3(kRowsThreads), smem, stream, (const TA*)A, lda,
                       (const TW*)W, (const TW*)W2, (TO*)out, ldo, M, N, K, e, batch_a, batch_w, batch_o, w_fixed);
    };
    const int feats = few ? few_rows_features(K, kDual) : kDual ? kTileFeats / 2 : kTileFeats;
    const int groups = (N + feats - 1) / feats;
    if constexpr (std::is_same<TW, float>::value) {
        const int most = few_rows_stream_blocks();
        if (passes == 1 && batch == 1 && few_rows_streams(W, W2, N, K, kDual, most)) {
            const auto kernel = gemm_nt_kernel<TA, TW, TO, MODE, kStream>;
            launch(kernel, kFewRows, most, few_rows_stream_smem(kernel, M, K));
            return;
        }
    }
    const auto kernel = few ? gemm_nt_kernel<TA, TW, TO, MODE, kFew> : gemm_nt_kernel<TA, TW, TO, MODE, kTile>;
    launch(kernel, few ? kFewRows : kTileRows, groups, rows_product_smem(kernel, few));
}

template <typename TA, typename TW, typename TO>
static int launch_gemm(int mode, const void* A, int lda, const void* W, const void* W2, void* out, int ldo,
                       int M, int N, int K, const Ending& e, int w_fixed, cudaStream_t stream,
                       int batch = 1, long batch_a = 0, long batch_w = 0, long batch_o = 0) {
    if (mode == kStore) launch_mode<TA, TW, TO, kStore>(A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    else if (mode == kAccumulate) launch_mode<TA, TW, TO, kAccumulate>(A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    else if (mode == kSwiGLU) launch_mode<TA, TW, TO, kSwiGLU>(A, lda, W, W2, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    else if (mode == kStoreAct) launch_mode<TA, TW, TO, kStoreAct>(A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    else return fail("gemm_simt: unknown mode %d", mode);
    MDMA_LAUNCH_OK("gemm_simt");
    return 0;
}

}  // namespace mdma

using namespace mdma;
// Returns 1 if a product of up to 8 rows with a 16-byte aligned float matrix (`gated`: two of them) [N, K] streams it through
// shared memory on a device of so many SMs.
extern "C" int mdma_gemm_simt_streams(int N, int K, int gated, int sm_count) { return few_rows_streams(nullptr, nullptr, N, K, gated != 0, 2 * sm_count) ? 1 : 0; }

extern "C" int mdma_gemm_simt(int mode, const void* A, int a_dtype, int lda, const void* W, const void* W2,
                              int w_dtype, void* out, int out_dtype, int ldo, int M, int N, int K,
                              const void* bias, const void* bias2, int bias_dtype, int act, float act_limit, float act_alpha,
                              int w_fixed, cudaStream_t stream) {
    MDMA_REQUIRE(M >= 0 && N > 0 && K > 0 && lda >= K && ldo >= N, "gemm_simt: bad sizes M=%d N=%d K=%d lda=%d ldo=%d", M, N, K, lda, ldo);
    MDMA_REQUIRE(mode != kSwiGLU || W2 != nullptr, "gemm_simt: SwiGLU needs two weights");
    MDMA_REQUIRE(mode != kAccumulate || out_dtype == kF32, "gemm_simt: the residual stream is float");
    MDMA_REQUIRE((M + 63) / 64 <= 65535, "gemm_simt: too many rows (%d)", M);
    MDMA_REQUIRE(act >= kActSilu && act <= kActReluSquared, "gemm_simt: unknown activation %d", act);
    MDMA_REQUIRE(act != kActSwishLimit || mode == kSwiGLU, "gemm_simt: the limited activation belongs to a gated product");
    MDMA_REQUIRE(bias_dtype == kF32 || bias_dtype == kBF16, "gemm_simt: unknown bias dtype %d", bias_dtype);
    if (M == 0) return 0;
    const Ending e{bias, mode == kSwiGLU ? bias2 : nullptr, bias_dtype, act, 0, act_limit, act_alpha};
    if (a_dtype == kF32 && w_dtype == kF32 && out_dtype == kF32)
        return launch_gemm<float, float, float>(mode, A, lda, W, W2, out, ldo, M, N, K, e, w_fixed, stream);
    if (a_dtype == kBF16 && w_dtype == kBF16 && out_dtype == kBF16)
        return launch_gemm<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(mode, A, lda, W, W2, out, ldo, M, N, K, e, w_fixed, stream);
    if (a_dtype == kBF16 && w_dtype == kBF16 && out_dtype == kF32)
        return launch_gemm<__nv_bfloat16, __nv_bfloat16, float>(mode, A, lda, W, W2, out, ldo, M, N, K, e, w_fixed, stream);
    return fail("gemm_simt: unsupported dtypes a=%d w=%d out=%d", a_dtype, w_dtype, out_dtype);
}

// `batch` products of the same sizes in one launch: product z reads A + z * batch_a (rows `lda` apart),
// W + z * batch_w ([N, K], contiguous) and writes out + z * batch_o (rows `ldo` apart).  A projection
// applied head by head is one call: the heads lie side by side in the rows of A and of out.
extern "C" int mdma_gemm_simt_batched(const void* A, int a_dtype, int lda, long batch_a, const void* W, int w_dtype,
                                      long batch_w, void* out, int out_dtype, int ldo, long batch_o, int batch,
                                      int M, int N, int K, int w_fixed, cudaStream_t stream) {
    MDMA_REQUIRE(M >= 0 && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm_simt_batched: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
    MDMA_REQUIRE((M + 63) / 64 <= 65535, "gemm_simt_batched: too many rows (%d)", M);
    if (M == 0) return 0;
    const Ending e{nullptr, nullptr, kF32, kActSilu};
    if (a_dtype == kF32 && w_dtype == kF32 && out_dtype == kF32)
        return launch_gemm<float, float, float>(kStore, A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    if (a_dtype == kBF16 && w_dtype == kBF16 && out_dtype == kBF16)
        return launch_gemm<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(kStore, A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    if (a_dtype == kBF16 && w_dtype == kBF16 && out_dtype == kF32)
        return launch_gemm<__nv_bfloat16, __nv_bfloat16, float>(kStore, A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    if (a_dtype == kF32 && w_dtype == kBF16 && out_dtype == kF32)       // float rows through matrices kept in bfloat16 (a recurrence's gates)
        return launch_gemm<float, __nv_bfloat16, float>(kStore, A, lda, W, nullptr, out, ldo, M, N, K, e, w_fixed, stream, batch, batch_a, batch_w, batch_o);
    return fail("gemm_simt_batched: unsupported dtypes a=%d w=%d out=%d", a_dtype, w_dtype, out_dtype);
}
