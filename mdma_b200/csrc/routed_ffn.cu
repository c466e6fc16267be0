// A feed-forward made of many small gated feed-forwards ("experts") of which each token uses a few.
//
// Router (one block per token, float arithmetic):
//     z = R h (+ bias)                     logits over all routed outputs (experts, then identity experts)
//     s = softmax(z), or sigmoid(z) element by element (`scoring` 1)
//     c = s + correction                   choice scores
//     experts form `n_groups` equal groups of neighbours; a group's score is the sum of its `group_top`
//     largest c (1: its largest); only the `keep_groups` best groups stay eligible (the others count as
//     minus infinity)
//     the `top` eligible experts with the largest c are chosen (ties: the lower number)
//     weight_j = s[chosen_j] / (sum of the chosen s + 1e-20), or s[chosen_j] itself (`renormalize` 0), times a constant
// and, if the layer has a shared expert with a gate, sg = sigmoid(g . h), one number per token.
//
// Experts: expert e maps h to D_e pair(G_e h, U_e h), pair(g, u) = SiLU(g) * u or another gated form of
// `gated_pair`, or without U (a null pointer) to D_e act(G_e h); the last `n_identity` routed
// outputs have no matrices, their output is h itself.  The matrices of all experts are stacked:
// G and U [experts * ff, width], D [experts * width, ff].
//
// Two ways to compute the chosen experts.  Token by token (steps of few tokens): a block per (token,
// choice) reads its expert's matrices; every output element is one warp's sum in a fixed order.  Expert
// by expert (steps of many tokens): the (token, choice) pairs are counted and sorted by expert on the
// device, and a block computes a tile of pairs x features of ONE expert with the expert's matrix tile
// staged in shared memory once for all its pairs.  No step of either way reads anything on the host.
#include "rows_product.cuh"

namespace mdma {

// Pairs per expert up to which the blocks that stream an expert's matrices are the faster ones.  Measured, 14 experts of 512
// on rows of 1,024 floats, four a token, the whole feed-forward: 16 tokens (4.6 pairs an expert) 45 us against 75 with
// tiles, 32 tokens (9.1) 70 against 76, 64 tokens (18) 117 against 78; 4 tokens 29 (385 with tiles that had nothing on
// their way and four launches to sort the pairs).
constexpr int kFewPairsPerExpert = 10;

constexpr int kMaxRouted = 1024, kMaxTop = 32, kMaxGroupTop = 8;

// eight consecutive elements as floats, by 16-byte loads (the address must be 16-byte aligned)
__device__ __forceinline__ void load8(const float* p, float* v) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float* v) {
    const uint4 q = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
        v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
}

// A warp's dot product over n elements; `vec`: n is a multiple of 8 and both rows start on 16-byte boundaries, so a lane
// takes eight consecutive elements at a time.  Either way the order of additions is fixed.
template <typename TA, typename TW>
__device__ __forceinline__ float warp_dot(const TA* __restrict__ a, const TW* __restrict__ w, int n, int lane, bool vec = false) {
    float acc = 0.f;
    if (vec) {
#pragma unroll 4                                          // four loads of either row in flight
        for (int k = lane * 8; k < n; k += 256) {
            float x[8], y[8];
            load8(a + k, x);
            load8(w + k, y);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc = fmaf(x[i], y[i], acc);
        }
    } else {
        for (int k = lane; k < n; k += 32) acc = fmaf(to_float(a[k]), to_float(w[k]), acc);
    }
    return warp_sum(acc);
}

// The place of the largest of n values above minus infinity (ties: the lower place), -1 without one; a whole warp calls it.
__device__ __forceinline__ int warp_largest(const float* v, int n, int lane) {
    int at = -1;
    float best = -INFINITY;
    for (int i = lane; i < n; i += 32)
        if (v[i] > best) { best = v[i]; at = i; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, best, o);
        const int place = __shfl_xor_sync(0xffffffffu, at, o);
        if (place >= 0 && (at < 0 || other > best || (other == best && place < at))) { best = other; at = place; }
    }
    return at;
}

// ---------------------------------------------------------------- router
constexpr int kRouteWide = 32, kRouteNarrow = 8;

// Warps of a token's block.  Where every token has an SM of its own, a warp an output (and one for the shared gate), as long as
// there are no more than kRouteWide: the sums side by side are one round trip.  Of more tokens eight warps, six blocks an SM: one
// warp's serial tail then lies under other tokens' sums.  16 outputs and a gate of 2,048 in bfloat16, us, wide / eight: 4 tokens
// 7.9 / 9.9, 148 8.2 / 10.4, 200 14.3 / 10.5, 512 16 / 13.3, 6,000 142 / 70; 64 outputs 12 / 18, 12 / 18, 23 / 19, 46 / 32, 459 / 166.
static int route_warps(int n_tokens, int outputs, int sm_count) {
    if (n_tokens > sm_count || outputs <= kRouteNarrow) return kRouteNarrow;
    return outputs < kRouteWide ? outputs : kRouteWide;
}

template <typename TA, typename TW, typename TC, int MAX_WARPS>
__global__ void __launch_bounds__(MAX_WARPS * 32, MAX_WARPS == kRouteNarrow ? 6 : 1)
route_kernel(const TA* __restrict__ h, int h_stride, const TW* __restrict__ router, const TC* __restrict__ correction,
             const TW* __restrict__ shared_gate, int width, int n_routed, int top, int n_groups, int keep_groups,
             int scoring, int group_top, int renormalize, int logit_bias, float weight_scale,
             int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ shared_scale) {
    chain_release();
    // the router's rows come from memory: on their way while the kernel before this one ends (4 tokens, 16 outputs of 1,024
    // floats: 22 us with a warp waiting for every 256 numbers of every row)
    const size_t router_bytes = (size_t)n_routed * width * sizeof(TW);
    for (size_t at = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 128; at < router_bytes; at += (size_t)gridDim.x * blockDim.x * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(router) + at));
    chain_wait();
    __shared__ float z[kMaxRouted];
    __shared__ float c[kMaxRouted];
    __shared__ float group_score[kMaxRouted];
    __shared__ unsigned kept[kMaxRouted / 32];
    const int t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const TA* row = h + (size_t)t * h_stride;
    const bool vec_row = width % 8 == 0 && ((uintptr_t)row & 15) == 0;
    const bool vec = vec_row && ((uintptr_t)router & 15) == 0, vec_gate = vec_row && ((uintptr_t)shared_gate & 15) == 0;
    for (int e = warp; e < n_routed + (shared_gate != nullptr); e += n_warps) {
        const bool gate = e == n_routed;
        const float v = warp_dot(row, gate ? shared_gate : router + (size_t)e * width, width, lane, gate ? vec_gate : vec);
        if (lane != 0) continue;
        if (gate) shared_scale[t] = 1.0f / (1.0f + expf(-v));
        else z[e] = v + (logit_bias ? to_float(correction[e]) : 0.f);
    }
    __syncthreads();
    // the rest is a few hundred operations of one warp: exponentials, group scores and the search for a largest score side
    // by side, every sum by one lane in one order
    if (warp != 0) return;
    if (scoring == 1) {
        for (int e = lane; e < n_routed; e += 32) z[e] = 1.0f / (1.0f + expf(-z[e]));
    } else {
        float m = -INFINITY;
        for (int e = lane; e < n_routed; e += 32) m = fmaxf(m, z[e]);
        m = warp_max(m);
        for (int e = lane; e < n_routed; e += 32) z[e] = expf(z[e] - m);
        __syncwarp();
        float sum = 0.f;
        for (int e = 0; e < n_routed; ++e) sum += z[e];
        __syncwarp();
        for (int e = lane; e < n_routed; e += 32) z[e] = z[e] / sum;
    }
    for (int e = lane; e < n_routed; e += 32) c[e] = z[e] + (correction && !logit_bias ? to_float(correction[e]) : 0.f);   // z: s; c: choice score
    __syncwarp();
    if (n_groups > 1 && keep_groups < n_groups) {
        const int per = n_routed / n_groups;
        for (int g = lane; g < n_groups; g += 32) {
            float gs = -INFINITY;
            if (group_top <= 1) {
                for (int e = g * per; e < (g + 1) * per; ++e) gs = fmaxf(gs, c[e]);
            } else {
                // the group's largest scores, largest first, are added up (a group of fewer members: all of them)
                float best_of[kMaxGroupTop];
#pragma unroll
                for (int i = 0; i < kMaxGroupTop; ++i) best_of[i] = -INFINITY;
                for (int e = g * per; e < (g + 1) * per; ++e) {
                    float v = c[e];
#pragma unroll
                    for (int i = 0; i < kMaxGroupTop; ++i)
                        if (v > best_of[i]) { const float tmp = best_of[i]; best_of[i] = v; v = tmp; }
                }
                gs = 0.f;
#pragma unroll
                for (int i = 0; i < kMaxGroupTop; ++i) if (i < group_top && i < per) gs += best_of[i];
            }
            group_score[g] = gs;
        }
        __syncwarp();
        for (int w = lane; w < (n_groups + 31) / 32; w += 32) kept[w] = 0u;
        __syncwarp();
        // the best group not yet kept is looked for keep_groups times (ties: the lower number); a bit per group
        for (int k = 0; lane == 0 && k < keep_groups; ++k) {
            int best = -1;
            float best_score = -INFINITY;
            for (int g = 0; g < n_groups; ++g) {
                if (kept[g >> 5] >> (g & 31) & 1u) continue;
                const float gs = group_score[g];
                if (best < 0 || gs > best_score) { best = g; best_score = gs; }
            }
            if (best >= 0) kept[best >> 5] |= 1u << (best & 31);
        }
        __syncwarp();
        for (int e = lane; e < n_routed; e += 32) {
            const int g = e / per;
            if (!(kept[g >> 5] >> (g & 31) & 1u)) c[e] = -INFINITY;
        }
        __syncwarp();
    }
    int mine = -1;                                        // lane k keeps the k-th choice
    float total = 0.f;
    for (int k = 0; k < top; ++k) {
        const int best = warp_largest(c, n_routed, lane);
        if (lane == k) mine = best;
        if (best >= 0) { total += z[best]; if (lane == 0) c[best] = -INFINITY; }
        __syncwarp();
    }
    if (lane < top) {
        chosen[(size_t)t * top + lane] = mine;
        weights[(size_t)t * top + lane] = mine < 0 ? 0.f : weight_scale * (renormalize ? z[mine] / (total + 1e-20f) : z[mine]);
    }
}

// ---------------------------------------------------------------- token by token
// act[t * top + j, f] = silu(G_e[f] . h_t) * (U_e[f] . h_t), e = chosen[t, j] (nothing for identity experts)
template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
expert_gate_up_kernel(const TA* __restrict__ h, int h_stride, const TW* __restrict__ G, const TW* __restrict__ U,
                      const int* __restrict__ chosen, int n_experts, int top, int width, int ff, TA* __restrict__ act,
                      int pair_act, float act_limit, float act_alpha) {
    chain_release();
    chain_wait();
    extern __shared__ float hs[];
    const int pair = blockIdx.x;
    const int e = chosen[pair];
    if (e < 0 || e >= n_experts) return;
    const int t = pair / top;
    const TA* row = h + (size_t)t * h_stride;
    for (int k = threadIdx.x; k < width; k += blockDim.x) hs[k] = to_float(row[k]);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const bool vec = width % 8 == 0 && (((uintptr_t)G | (uintptr_t)U) & 15) == 0;
    if (U == nullptr) {
        for (int f = blockIdx.y * n_warps + warp; f < ff; f += gridDim.y * n_warps) {
            const float z = warp_dot(hs, G + ((size_t)e * ff + f) * width, width, lane, vec);
            if (lane == 0) act[(size_t)pair * ff + f] = from_float<TA>(gate_activation(z, pair_act));
        }
        return;
    }
    for (int f = blockIdx.y * n_warps + warp; f < ff; f += gridDim.y * n_warps) {
        const TW* g = G + ((size_t)e * ff + f) * width;
        const TW* u = U + ((size_t)e * ff + f) * width;
        float ag = 0.f, au = 0.f;
        if (vec) {
            for (int k = lane * 8; k < width; k += 256) {
                float x[8], a[8], b[8];
                load8(hs + k, x);
                load8(g + k, a);
                load8(u + k, b);
#pragma unroll
                for (int i = 0; i < 8; ++i) { ag = fmaf(x[i], a[i], ag); au = fmaf(x[i], b[i], au); }
            }
        } else {
            for (int k = lane; k < width; k += 32) {
                ag = fmaf(hs[k], to_float(g[k]), ag);
                au = fmaf(hs[k], to_float(u[k]), au);
            }
        }
        ag = warp_sum(ag);
        au = warp_sum(au);
        if (lane == 0) act[(size_t)pair * ff + f] = from_float<TA>(gated_pair(ag, au, pair_act, act_limit, act_alpha));
    }
}

// x[t, f] += sum_j w[t, j] * (D_e[f] . act[t * top + j]  or, for an identity expert,  h[t, f])
template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
expert_down_kernel(const TA* __restrict__ act, const TA* __restrict__ h, int h_stride, const TW* __restrict__ D,
                   const int* __restrict__ chosen, const float* __restrict__ weights, int n_experts, int top,
                   int width, int ff, float* __restrict__ x) {
    chain_release();
    chain_wait();
    const int t = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const bool vec = ff % 8 == 0 && (((uintptr_t)D | (uintptr_t)act) & 15) == 0;
    for (int f = blockIdx.y * n_warps + warp; f < width; f += gridDim.y * n_warps) {
        float total = 0.f;
        for (int j = 0; j < top; ++j) {
            const int e = chosen[(size_t)t * top + j];
            if (e < 0) continue;
            const float w = weights[(size_t)t * top + j];
            if (e >= n_experts) { total += w * to_float(h[(size_t)t * h_stride + f]); continue; }
            total += w * warp_dot(act + ((size_t)t * top + j) * ff, D + ((size_t)e * width + f) * ff, ff, lane, vec);
        }
        if (lane == 0) x[(size_t)t * width + f] += total;
    }
}

// ---------------------------------------------------------------- expert by expert
// The (token, choice) pairs sorted by expert: first[e] is where expert e's run starts in `order` (first[n_experts]: the
// total; identity experts are not counted), order[] lists the pairs expert after expert and where[] is its inverse.
// Three small kernels: every pair adds one to its expert's counter; one block turns the counters into starts (and
// clears them); every pair takes the next place of its expert's run.  The order inside a run depends on who comes
// first, the results do not: every pair's row is computed on its own.
__global__ void __launch_bounds__(256)
expert_count_kernel(const int* __restrict__ chosen, int n_pairs, int n_experts, int* __restrict__ counters) {
    chain_release();
    chain_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pairs) return;
    const int e = chosen[p];
    if (e >= 0 && e < n_experts) atomicAdd(&counters[e], 1);
}

__global__ void __launch_bounds__(32)
expert_starts_kernel(int n_experts, int* __restrict__ first, int* __restrict__ counters) {
    chain_release();
    chain_wait();
    if (threadIdx.x != 0) return;
    int run = 0;
    for (int e = 0; e < n_experts; ++e) { first[e] = run; run += counters[e]; counters[e] = 0; }
    first[n_experts] = run;
}

__global__ void __launch_bounds__(256)
expert_place_kernel(const int* __restrict__ chosen, int n_pairs, int n_experts, const int* __restrict__ first,
                    int* __restrict__ counters, int* __restrict__ order, int* __restrict__ where) {
    chain_release();
    chain_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n_pairs) return;
    const int e = chosen[p];
    if (e < 0 || e >= n_experts) return;
    const int at = first[e] + atomicAdd(&counters[e], 1);
    order[at] = p;
    if (where) where[p] = at;
}

// The same three in one block, for steps of up to kSortPairs pairs: one launch instead of a memset and three.
constexpr int kSortPairs = 8192, kSortThreads = 512;
__global__ void __launch_bounds__(kSortThreads)
expert_sort_kernel(const int* __restrict__ chosen, int n_pairs, int n_experts, int* __restrict__ first,
                   int* __restrict__ order, int* __restrict__ where) {
    chain_release();
    chain_wait();
    __shared__ int place[kMaxRouted];
    for (int e = threadIdx.x; e < n_experts; e += kSortThreads) place[e] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += kSortThreads) {
        const int e = chosen[p];
        if (e >= 0 && e < n_experts) atomicAdd(&place[e], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int run = 0;
        for (int e0 = 0; e0 < n_experts; e0 += 32) {
            const int n = e0 + lane < n_experts ? place[e0 + lane] : 0;
            int upto = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += v; }
            if (e0 + lane < n_experts) { place[e0 + lane] = run + upto - n; first[e0 + lane] = run + upto - n; }
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) first[n_experts] = run;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += kSortThreads) {
        const int e = chosen[p];
        if (e < 0 || e >= n_experts) continue;
        const int at = atomicAdd(&place[e], 1);
        order[at] = p;
        if (where) where[p] = at;
    }
}

// `first` holds 2 * (n_experts + 1) ints: the starts, then the counters
static int sort_pairs(const int* chosen, int n_pairs, int n_experts, int* first, int* order, int* where, cudaStream_t stream) {
    if (n_pairs <= kSortPairs && n_experts <= kMaxRouted) {
        launch_chained(expert_sort_kernel, dim3(1), dim3(kSortThreads), 0, stream, chosen, n_pairs, n_experts, first, order, where);
        MDMA_LAUNCH_OK("expert sort");
        return 0;
    }
    int* counters = first + n_experts + 1;
    if (cudaMemsetAsync(counters, 0, sizeof(int) * (size_t)(n_experts + 1), stream) != cudaSuccess) return fail("experts: memset failed");
    const int blocks = (n_pairs + 255) / 256;
    expert_count_kernel<<<blocks, 256, 0, stream>>>(chosen, n_pairs, n_experts, counters);
    expert_starts_kernel<<<1, 32, 0, stream>>>(n_experts, first, counters);
    expert_place_kernel<<<blocks, 256, 0, stream>>>(chosen, n_pairs, n_experts, first, counters, order, where);
    MDMA_LAUNCH_OK("expert sort");
    return 0;
}

// rows[i] = h[order[i] / top] for the sorted pairs i < first[n_experts]: the experts' inputs, expert after expert,
// as contiguous rows that a matrix product can take
template <typename TA>
__global__ void __launch_bounds__(256)
expert_gather_kernel(const TA* __restrict__ h, int h_stride, const int* __restrict__ first, const int* __restrict__ order,
                     int n_experts, int top, int width, TA* __restrict__ rows) {
    chain_release();
    chain_wait();
    const int i = blockIdx.x;
    if (i >= first[n_experts]) return;
    const TA* src = h + (size_t)(order[i] / top) * h_stride;
    TA* dst = rows + (size_t)i * width;
    for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < width; e += gridDim.y * blockDim.x) dst[e] = src[e];
}

// The products of expert blockIdx.z with its run of pairs, in the shapes and with the order of additions of
// rows_product.cuh: FEW blocks stream the expert's matrices over up to 8 pairs, else tiles of 32 pairs.
// act[pair, f] = pair_act(G_e h, U_e h), or act(G_e h) without U
template <typename TA, typename TW, bool DUAL, bool FEW>
__global__ void __launch_bounds__(kRowsThreads)
expert_gate_up_sorted_kernel(const TA* __restrict__ h, int h_stride, const TW* __restrict__ G, const TW* __restrict__ U,
                             const int* __restrict__ first, const int* __restrict__ order, int top, int width, int ff,
                             TA* __restrict__ act, int pair_act, float act_limit, float act_alpha) {
    chain_release();
    chain_wait();
    constexpr int kRows = FEW ? kFewRows : kTileRows;
    extern __shared__ __align__(16) float smem[];
    __shared__ int pair_of[kRows];
    const int e = blockIdx.z, stop = first[e + 1];
    G += (size_t)e * ff * width;
    if (DUAL) U += (size_t)e * ff * width;
    const bool vec_h = rows_of_four(h, h_stride, width), vec_w = rows_of_four(G, width, width) && (!DUAL || rows_of_four(U, width, width));
    for (int begin = first[e] + blockIdx.y * kRows; begin < stop; begin += gridDim.y * kRows) {
        const int n = min(kRows, stop - begin);
        if (threadIdx.x < n) pair_of[threadIdx.x] = order[begin + threadIdx.x];
        __syncthreads();
        auto row_of = [&](int m) { return h + (size_t)(pair_of[m] / top) * h_stride; };
        auto store = [&](int m, int f, float g, float u) {
            act[(size_t)pair_of[m] * ff + f] = from_float<TA>(DUAL ? gated_pair(g, u, pair_act, act_limit, act_alpha) : gate_activation(g, pair_act));
        };
        if (FEW) few_rows_product<TA, TW, DUAL>(n, row_of, G, U, blockIdx.x * few_rows_features(width, DUAL), ff, width, vec_h, vec_w, smem, [] {}, store);
        else tile_product<TA, TW, DUAL>(n, row_of, G, U, blockIdx.x * (DUAL ? kTileFeats / 2 : kTileFeats), ff, width, vec_h, vec_w, smem, store);
        __syncthreads();
    }
}

// y[pair, f] = D_e[f] . act[pair] for the pairs of expert blockIdx.z (float rows, one per pair)
template <typename TA, typename TW, bool FEW>
__global__ void __launch_bounds__(kRowsThreads)
expert_down_sorted_kernel(const TA* __restrict__ act, const TW* __restrict__ D, const int* __restrict__ first,
                          const int* __restrict__ order, int width, int ff, float* __restrict__ y) {
    chain_release();
    chain_wait();
    constexpr int kRows = FEW ? kFewRows : kTileRows;
    extern __shared__ __align__(16) float smem[];
    __shared__ int pair_of[kRows];
    const int e = blockIdx.z, stop = first[e + 1];
    D += (size_t)e * width * ff;
    const bool vec_a = rows_of_four(act, ff, ff), vec_w = rows_of_four(D, ff, ff);
    for (int begin = first[e] + blockIdx.y * kRows; begin < stop; begin += gridDim.y * kRows) {
        const int n = min(kRows, stop - begin);
        if (threadIdx.x < n) pair_of[threadIdx.x] = order[begin + threadIdx.x];
        __syncthreads();
        auto row_of = [&](int m) { return act + (size_t)pair_of[m] * ff; };
        auto store = [&](int m, int f, float v, float) { y[(size_t)pair_of[m] * width + f] = v; };
        if (FEW) few_rows_product<TA, TW, false>(n, row_of, D, D, blockIdx.x * few_rows_features(ff, false), width, ff, vec_a, vec_w, smem, [] {}, store);
        else tile_product<TA, TW, false>(n, row_of, D, D, blockIdx.x * kTileFeats, width, ff, vec_a, vec_w, smem, store);
        __syncthreads();
    }
}

// x[t, f] += sum_j w[t, j] * (y[row of pair t * top + j, f]  or, for an identity expert,  h[t, f]), j in order;
// the row of a pair is the pair's number, or where[pair] when y holds the sorted list's rows
template <typename TA>
__global__ void __launch_bounds__(256)
expert_combine_kernel(const float* __restrict__ y, const TA* __restrict__ h, int h_stride, const int* __restrict__ chosen,
                      const float* __restrict__ weights, const int* __restrict__ where, int n_experts, int top, int width,
                      float* __restrict__ x) {
    chain_release();
    chain_wait();
    const int t = blockIdx.x;
    for (int f = blockIdx.y * blockDim.x + threadIdx.x; f < width; f += gridDim.y * blockDim.x) {
        float total = 0.f;
        for (int j = 0; j < top; ++j) {
            const int e = chosen[(size_t)t * top + j];
            if (e < 0) continue;
            const size_t pair = (size_t)t * top + j;
            const float v = e >= n_experts ? to_float(h[(size_t)t * h_stride + f]) : y[(where ? (size_t)where[pair] : pair) * width + f];
            total += weights[(size_t)t * top + j] * v;
        }
        x[(size_t)t * width + f] += total;
    }
}

}  // namespace mdma

using namespace mdma;

#define MDMA_DISPATCH_2(a_code, TA, w_code, TW, ...) \
    MDMA_DISPATCH_DTYPE(a_code, TA, MDMA_DISPATCH_DTYPE(w_code, TW, __VA_ARGS__))

extern "C" {

// Warps of a token's block in mdma_route for so many outputs, the shared gate's among them.
int mdma_route_warps(int n_tokens, int outputs, int sm_count) { return route_warps(n_tokens, outputs, sm_count); }

int mdma_route(const void* h, int h_dtype, int h_stride, const void* router, int w_dtype, const void* correction,
               int c_dtype, const void* shared_gate, int n_tokens, int width, int n_routed, int top, int n_groups,
               int keep_groups, int scoring, int group_top, int renormalize, int logit_bias, float weight_scale, int* chosen,
               float* weights, float* shared_scale, cudaStream_t stream) {
    MDMA_REQUIRE(!logit_bias || correction, "route: a bias on the logits needs its numbers");
    MDMA_REQUIRE(scoring >= 0 && scoring <= 1 && group_top >= 1 && group_top <= kMaxGroupTop,
                 "route: scoring %d, a group's score over its %d largest (at most %d)", scoring, group_top, kMaxGroupTop);
    MDMA_REQUIRE(n_tokens >= 0 && width > 0, "route: bad sizes");
    MDMA_REQUIRE(n_routed > 0 && n_routed <= kMaxRouted, "route: %d routed outputs, the kernel takes up to %d", n_routed, kMaxRouted);
    MDMA_REQUIRE(top > 0 && top <= kMaxTop && top <= n_routed, "route: top %d of %d (at most %d)", top, n_routed, kMaxTop);
    MDMA_REQUIRE(n_groups >= 1 && n_routed % n_groups == 0 && keep_groups >= 1 && keep_groups <= n_groups,
                 "route: %d groups (keep %d) over %d outputs", n_groups, keep_groups, n_routed);
    MDMA_REQUIRE(shared_gate == nullptr || shared_scale != nullptr, "route: the shared gate needs a place for its result");
    if (n_tokens == 0) return 0;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int warps = route_warps(n_tokens, n_routed + (shared_gate != nullptr), sms);
    MDMA_DISPATCH_2(h_dtype, TA, w_dtype, TW,
        MDMA_DISPATCH_DTYPE(c_dtype, TC,
            launch_chained(warps == kRouteNarrow ? route_kernel<TA, TW, TC, kRouteNarrow> : route_kernel<TA, TW, TC, kRouteWide>,
                           dim3(n_tokens), dim3(warps * 32), 0, stream, (const TA*)h, h_stride,
                           (const TW*)router, (const TC*)correction, (const TW*)shared_gate, width, n_routed, top,
                           n_groups, keep_groups, scoring, group_top, renormalize, logit_bias, weight_scale, chosen, weights, shared_scale)));
    MDMA_LAUNCH_OK("route");
    return 0;
}

// Token by token: act [n_tokens * top, ff] in h's dtype is scratch; x [n_tokens, width] float takes the sum.
int mdma_experts_by_token(const void* h, int h_dtype, int h_stride, const void* G, const void* U, const void* D,
                          int w_dtype, const int* chosen, const float* weights, int n_tokens, int n_experts, int top,
                          int width, int ff, void* act, float* x, int pair_act, float act_limit, float act_alpha,
                          cudaStream_t stream) {
    MDMA_REQUIRE(n_tokens >= 0 && width > 0 && ff > 0 && top > 0 && n_experts >= 0, "experts: bad sizes");
    MDMA_REQUIRE((size_t)width * sizeof(float) <= 160 * 1024, "experts: width %d is beyond the kernel's shared memory", width);
    if (n_tokens == 0) return 0;
    const int fparts = (ff + 7) / 8 > 64 ? 64 : (ff + 7) / 8;
    const int wparts = (width + 7) / 8 > 128 ? 128 : (width + 7) / 8;
    MDMA_DISPATCH_2(h_dtype, TA, w_dtype, TW, {
        if (n_experts > 0) {
            static bool raised = false;
            if (!raised) {
                cudaFuncSetAttribute(expert_gate_up_kernel<TA, TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
                raised = true;
            }
            launch_chained(expert_gate_up_kernel<TA, TW>, dim3(n_tokens * top, fparts), dim3(256),
                           (size_t)width * sizeof(float), stream, (const TA*)h, h_stride, (const TW*)G, (const TW*)U, chosen,
                           n_experts, top, width, ff, (TA*)act, pair_act, act_limit, act_alpha);
        }
        launch_chained(expert_down_kernel<TA, TW>, dim3(n_tokens, wparts), dim3(256), 0, stream, (const TA*)act, (const TA*)h,
                       h_stride, (const TW*)D, chosen, weights, n_experts, top, width, ff, x);
    });
    MDMA_LAUNCH_OK("experts_by_token");
    return 0;
}

// Expert by expert: first [2 * (n_experts + 1)] and order [n_tokens * top] ints, act [n_tokens * top, ff] in h's dtype and
// y [n_tokens * top, width] floats are scratch.
int mdma_experts_sorted(const void* h, int h_dtype, int h_stride, const void* G, const void* U, const void* D,
                        int w_dtype, const int* chosen, const float* weights, int n_tokens, int n_experts, int top,
                        int width, int ff, int* first, int* order, void* act, float* y, float* x, int pair_act,
                        float act_limit, float act_alpha, cudaStream_t stream) {
    MDMA_REQUIRE(n_tokens >= 0 && width > 0 && ff > 0 && top > 0 && n_experts >= 0 && n_experts <= kMaxRouted, "experts: bad sizes");
    if (n_tokens == 0) return 0;
    const int n_pairs = n_tokens * top;
    MDMA_REQUIRE((n_pairs + 31) / 32 <= 65535, "experts: too many pairs (%d)", n_pairs);
    // by the pairs an expert has on average: the blocks take more tiles each where one has more
    const bool few = n_pairs <= kFewPairsPerExpert * n_experts;
    const int rows = few ? kFewRows : kTileRows;
    const int pair_tiles = n_experts > 0 ? (n_pairs / n_experts + rows) / rows + 1 : 1;
    const int wparts = (width + 255) / 256 > 64 ? 64 : (width + 255) / 256;
    MDMA_DISPATCH_2(h_dtype, TA, w_dtype, TW, {
        if (n_experts > 0) {
            if (int rc = sort_pairs(chosen, n_pairs, n_experts, first, order, nullptr, stream)) return rc;
            const bool dual = U != nullptr;
            const int gf = few ? few_rows_features(width, dual) : dual ? kTileFeats / 2 : kTileFeats;
            const int df = few ? few_rows_features(ff, false) : kTileFeats;
            auto up = dual ? (few ? expert_gate_up_sorted_kernel<TA, TW, true, true> : expert_gate_up_sorted_kernel<TA, TW, true, false>)
                           : (few ? expert_gate_up_sorted_kernel<TA, TW, false, true> : expert_gate_up_sorted_kernel<TA, TW, false, false>);
            launch_chained(up, dim3((ff + gf - 1) / gf, pair_tiles, n_experts), dim3(kRowsThreads), rows_product_smem(up, few), stream, (const TA*)h, h_stride,
                           (const TW*)G, (const TW*)U, first, order, top, width, ff, (TA*)act, pair_act, act_limit, act_alpha);
            auto down = few ? expert_down_sorted_kernel<TA, TW, true> : expert_down_sorted_kernel<TA, TW, false>;
            launch_chained(down, dim3((width + df - 1) / df, pair_tiles, n_experts), dim3(kRowsThreads), rows_product_smem(down, few), stream, (const TA*)act,
                           (const TW*)D, first, order, width, ff, y);
        }
        launch_chained(expert_combine_kernel<TA>, dim3(n_tokens, wparts), dim3(256), 0, stream, y, (const TA*)h, h_stride,
                       chosen, weights, (const int*)nullptr, n_experts, top, width, x);
    });
    MDMA_LAUNCH_OK("experts_sorted");
    return 0;
}

// The two ends of the expert-by-expert way when the products in between are the caller's (one matrix product per
// expert over its run of gathered rows).  Sort and gather: first [n_experts + 1], order and where [n_tokens * top],
// rows [n_tokens * top, width] in h's dtype.
int mdma_experts_gather(const void* h, int h_dtype, int h_stride, const int* chosen, int n_tokens, int n_experts, int top,
                        int width, int* first, int* order, int* where, void* rows, cudaStream_t stream) {
    MDMA_REQUIRE(n_tokens >= 0 && width > 0 && top > 0 && n_experts > 0 && n_experts <= kMaxRouted, "experts: bad sizes");
    if (n_tokens == 0) return 0;
    const int n_pairs = n_tokens * top;
    const int wparts = (width + 255) / 256 > 64 ? 64 : (width + 255) / 256;
    if (int rc = sort_pairs(chosen, n_pairs, n_experts, first, order, where, stream)) return rc;
    MDMA_DISPATCH_DTYPE(h_dtype, TA,
        launch_chained(expert_gather_kernel<TA>, dim3(n_pairs, wparts), dim3(256), 0, stream, (const TA*)h, h_stride,
                       (const int*)first, (const int*)order, n_experts, top, width, (TA*)rows));
    MDMA_LAUNCH_OK("experts_gather");
    return 0;
}

// Combine: y [sorted rows, width] floats hold the experts' results in the sorted list's order.
int mdma_experts_combine(const float* y, const void* h, int h_dtype, int h_stride, const int* chosen, const float* weights,
                         const int* where, int n_tokens, int n_experts, int top, int width, float* x, cudaStream_t stream) {
    MDMA_REQUIRE(n_tokens >= 0 && width > 0 && top > 0, "experts: bad sizes");
    if (n_tokens == 0) return 0;
    const int wparts = (width + 255) / 256 > 64 ? 64 : (width + 255) / 256;
    MDMA_DISPATCH_DTYPE(h_dtype, TA,
        launch_chained(expert_combine_kernel<TA>, dim3(n_tokens, wparts), dim3(256), 0, stream, y, (const TA*)h, h_stride,
                       chosen, weights, where, n_experts, top, width, x));
    MDMA_LAUNCH_OK("experts_combine");
    return 0;
}

}  // extern "C"
