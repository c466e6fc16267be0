// RMS norm in groups, and the weighted sum over the depth of the model.
//
// group_rmsnorm: a row of `width` floats is split into `groups` equal consecutive parts; every part is divided by
// its own sqrt(mean(part^2) + eps) and the whole row is multiplied by w.  Rows may be gathered by index.  Written
// in the compute dtype.  group_rmsnorm_add is the same norm on a sublayer's result y, added into the residual stream:
// x += norm(y); partial sums that a K-split product left of y are added up first (or are all there is of y: `only`).  All
// sums are float, in one fixed order: every warp sums a slice of a part, the slices of a part are added in slice order.
// Slices of up to 256 numbers in fours stay in registers between the two passes, and what the second pass adds to and
// multiplies with is asked for in the first: a block of a few rows is bound by the round trips it waits for.
//
// depth_mix: the model keeps the result of every layer so far; after run i the stream that goes on is
// x <- w[0] x0 + sum_{j=1..i+1} w[j] X_j, x0 the embedding's rows and X_j the result of run j-1 (X_(i+1) is x as the
// run left it, stored first).  Float throughout, terms added in the order of j.
#include "common.cuh"

namespace mdma {

constexpr int kGroupNormMaxWarps = 16;

constexpr int kGroupNormKeep = 2;                // groups of four numbers a lane keeps

template <typename T> __device__ __forceinline__ float4 four_of(const T* p);
template <> __device__ __forceinline__ float4 four_of<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 four_of<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xffff0000u), __uint_as_float(q.y << 16), __uint_as_float(q.y & 0xffff0000u));
}
__device__ __forceinline__ void put_four(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void put_four(__nv_bfloat16* p, const float4& v) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
// v += the partial sums at pp, four splits on their way at a time, added in split order
__device__ __forceinline__ void add_splits(float4& v, const float* pp, int splits, size_t split_stride) {
    int k = 0;
    for (; k + 4 <= splits; k += 4) {
        const float4 p0 = four_of(pp + (size_t)k * split_stride), p1 = four_of(pp + (size_t)(k + 1) * split_stride);
        const float4 p2 = four_of(pp + (size_t)(k + 2) * split_stride), p3 = four_of(pp + (size_t)(k + 3) * split_stride);
        v.x = (((v.x + p0.x) + p1.x) + p2.x) + p3.x;
        v.y = (((v.y + p0.y) + p1.y) + p2.y) + p3.y;
        v.z = (((v.z + p0.z) + p1.z) + p2.z) + p3.z;
        v.w = (((v.w + p0.w) + p1.w) + p2.w) + p3.w;
    }
    for (; k < splits; ++k) {
        const float4 p0 = four_of(pp + (size_t)k * split_stride);
        v.x += p0.x; v.y += p0.y; v.z += p0.z; v.w += p0.w;
    }
}

// Blocks of groups * slices warps (or fewer warps that walk the groups when there are more than 16 groups).
template <typename TW, typename TO, bool ADD>
__global__ void __launch_bounds__(kGroupNormMaxWarps * 32, 2)       // 64 registers (ADD spills 4 to 16 bytes): the block starts beside those of the product in front
group_rmsnorm_kernel(const float* src, float* y_complete, const float* __restrict__ partial,
                     int splits, size_t split_stride, int only, const int* __restrict__ rows, const TW* __restrict__ w,
                     TO* __restrict__ out, float* __restrict__ x_add, int width, int groups, int slices, int fours, float eps) {
    chain_release();
    chain_wait();
    __shared__ float sums[kGroupNormMaxWarps];
    const size_t t = blockIdx.x;
    const size_t r = rows ? (size_t)rows[t] : t;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    const int part = width / groups;
    const int per_slice = (part + slices - 1) / slices;
    const float* xr = src + r * width;
    for (int g0 = 0; g0 < groups; g0 += n_warps / slices) {
        const int g = g0 + warp / slices, s = warp % slices;
        const int lo = g * part + s * per_slice, hi = g < groups ? min(g * part + part, lo + per_slice) : lo;
        float sq = 0.f;
        // four numbers a lane at a time where the slices allow 16-byte accesses, kept if they are few enough
        const bool vec = fours && (lo & 3) == 0 && (hi & 3) == 0, keep = vec && hi - lo <= 128 * kGroupNormKeep;
        float4 v[kGroupNormKeep], x[kGroupNormKeep], f[kGroupNormKeep];
        if (keep) {
#pragma unroll
            for (int i = 0; i < kGroupNormKeep; ++i) {
                const int e = lo + lane * 4 + 128 * i;
                if (e >= hi) break;
                v[i] = ADD && only ? make_float4(0.f, 0.f, 0.f, 0.f) : four_of(xr + e);
                f[i] = four_of(w + e);
                if (ADD) x[i] = four_of(x_add + r * width + e);
            }
#pragma unroll
            for (int i = 0; i < kGroupNormKeep; ++i) {
                const int e = lo + lane * 4 + 128 * i;
                if (e >= hi) break;
                if (ADD && splits > 0) {
                    add_splits(v[i], partial + r * width + e, splits, split_stride);
                    put_four(y_complete + r * width + e, v[i]);
                }
                sq = fmaf(v[i].x, v[i].x, sq); sq = fmaf(v[i].y, v[i].y, sq); sq = fmaf(v[i].z, v[i].z, sq); sq = fmaf(v[i].w, v[i].w, sq);
            }
        } else if (vec) {
            for (int e = lo + lane * 4; e < hi; e += 128) {
                float4 u = ADD && only ? make_float4(0.f, 0.f, 0.f, 0.f) : four_of(xr + e);
                if (ADD && splits > 0) {
                    add_splits(u, partial + r * width + e, splits, split_stride);
                    put_four(y_complete + r * width + e, u);
                }
                sq = fmaf(u.x, u.x, sq); sq = fmaf(u.y, u.y, sq); sq = fmaf(u.z, u.z, sq); sq = fmaf(u.w, u.w, sq);
            }
        } else {
            for (int e = lo + lane; e < hi; e += 32) {
                float u = ADD && only ? 0.f : xr[e];
                if (ADD) {
                    for (int k = 0; k < splits; ++k) u += partial[(size_t)k * split_stride + r * width + e];
                    if (splits > 0) y_complete[r * width + e] = u;
                }
                sq = fmaf(u, u, sq);
            }
        }
        sq = warp_sum(sq);
        __syncthreads();
        if (lane == 0) sums[warp] = sq;
        __syncthreads();
        if (g < groups) {
            float total = 0.f;
            for (int k = 0; k < slices; ++k) total += sums[(warp / slices) * slices + k];
            const float inv = 1.0f / sqrtf(total / (float)part + eps);
            if (keep) {
#pragma unroll
                for (int i = 0; i < kGroupNormKeep; ++i) {
                    const int e = lo + lane * 4 + 128 * i;
                    if (e >= hi) break;
                    const float4 n = make_float4(v[i].x * inv * f[i].x, v[i].y * inv * f[i].y, v[i].z * inv * f[i].z, v[i].w * inv * f[i].w);
                    if (ADD) put_four(x_add + r * width + e, make_float4(x[i].x + n.x, x[i].y + n.y, x[i].z + n.z, x[i].w + n.w));
                    else put_four(out + t * width + e, n);
                }
            } else if (vec) {
                // (by the lane that made it: y_complete is read where it was written)
                for (int e = lo + lane * 4; e < hi; e += 128) {
                    const float4 u = four_of((ADD && splits > 0 ? y_complete + r * width : xr) + e), m = four_of(w + e);
                    const float4 n = make_float4(u.x * inv * m.x, u.y * inv * m.y, u.z * inv * m.z, u.w * inv * m.w);
                    if (ADD) {
                        const float4 old = four_of(x_add + r * width + e);
                        put_four(x_add + r * width + e, make_float4(old.x + n.x, old.y + n.y, old.z + n.z, old.w + n.w));
                    } else put_four(out + t * width + e, n);
                }
            } else {
                for (int e = lo + lane; e < hi; e += 32) {
                    const float u = (ADD && splits > 0) ? y_complete[r * width + e] : xr[e];
                    if (ADD) x_add[r * width + e] += u * inv * to_float(w[e]);
                    else out[t * width + e] = from_float<TO>(u * inv * to_float(w[e]));
                }
            }
        }
    }
}

template <typename TW>
__global__ void __launch_bounds__(256)
depth_mix_kernel(float* __restrict__ x, const float* __restrict__ x0, float* __restrict__ history, int depth, int run,
                 const TW* __restrict__ w, int width) {
    chain_release();
    chain_wait();
    const size_t t = blockIdx.x;
    float* hist = history + t * (size_t)depth * width;
    if ((width & 3) == 0) {
        // four numbers a thread; the earlier results are asked for four at a time, added in the order of j
        const int e = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
        if (e >= width) return;
        const float4 mine = *reinterpret_cast<const float4*>(x + t * width + e);
        *reinterpret_cast<float4*>(hist + (size_t)run * width + e) = mine;
        const float4 first = *reinterpret_cast<const float4*>(x0 + t * width + e);
        const float w0 = to_float(w[0]);
        float4 acc = make_float4(w0 * first.x, w0 * first.y, w0 * first.z, w0 * first.w);
        int j = 0;
        for (; j + 4 <= run; j += 4) {
            float4 h[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) h[i] = *reinterpret_cast<const float4*>(hist + (size_t)(j + i) * width + e);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float wj = to_float(w[j + i + 1]);
                acc.x = fmaf(wj, h[i].x, acc.x); acc.y = fmaf(wj, h[i].y, acc.y);
                acc.z = fmaf(wj, h[i].z, acc.z); acc.w = fmaf(wj, h[i].w, acc.w);
            }
        }
        for (; j < run; ++j) {
            const float4 h = *reinterpret_cast<const float4*>(hist + (size_t)j * width + e);
            const float wj = to_float(w[j + 1]);
            acc.x = fmaf(wj, h.x, acc.x); acc.y = fmaf(wj, h.y, acc.y); acc.z = fmaf(wj, h.z, acc.z); acc.w = fmaf(wj, h.w, acc.w);
        }
        const float wl = to_float(w[run + 1]);
        acc.x = fmaf(wl, mine.x, acc.x); acc.y = fmaf(wl, mine.y, acc.y); acc.z = fmaf(wl, mine.z, acc.z); acc.w = fmaf(wl, mine.w, acc.w);
        *reinterpret_cast<float4*>(x + t * width + e) = acc;
        return;
    }
    for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < width; e += gridDim.y * blockDim.x) {
        const float mine = x[t * width + e];
        hist[(size_t)run * width + e] = mine;
        float acc = to_float(w[0]) * x0[t * width + e];
        for (int j = 0; j < run; ++j) acc = fmaf(to_float(w[j + 1]), hist[(size_t)j * width + e], acc);
        x[t * width + e] = fmaf(to_float(w[run + 1]), mine, acc);
    }
}

static inline void group_norm_shape(int width, int groups, int* slices, int* warps) {
    const int part = width / groups;
    int s = 1;
    if (groups <= kGroupNormMaxWarps) {
        s = kGroupNormMaxWarps / groups;
        while (s > 1 && part / s < 128) s >>= 1;      // a slice of fewer than 128 numbers is not worth a warp
        int p2 = 1;
        while (p2 * 2 <= s) p2 *= 2;
        s = p2;
    }
    *slices = s;
    *warps = groups <= kGroupNormMaxWarps ? groups * s : kGroupNormMaxWarps;
}

}  // namespace mdma

using namespace mdma;

extern "C" {

int mdma_group_rmsnorm(const float* x, const void* w, int w_dtype, const int* rows, void* out, int out_dtype, int n_rows,
                       int width, int groups, float eps, cudaStream_t stream) {
    MDMA_REQUIRE(n_rows >= 0 && width > 0 && groups > 0 && width % groups == 0, "group_rmsnorm: %d numbers do not split into %d parts", width, groups);
    if (n_rows == 0) return 0;
    int slices, warps;
    group_norm_shape(width, groups, &slices, &warps);
    const int fours = (width & 3) == 0 && (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) == 0;
    MDMA_DISPATCH_DTYPE(w_dtype, TW, MDMA_DISPATCH_DTYPE(out_dtype, TO,
        launch_chained(group_rmsnorm_kernel<TW, TO, false>, dim3(n_rows), dim3(warps * 32), 0, stream, x, (float*)nullptr,
                       (const float*)nullptr, 0, (size_t)0, 0, rows, (const TW*)w, (TO*)out, (float*)nullptr, width, groups,
                       slices, fours, eps)));
    MDMA_LAUNCH_OK("group_rmsnorm");
    return 0;
}

// `only`: y is the sum of its partial sums (which there are), else they are added to it; it is left complete either way.
int mdma_group_rmsnorm_add(float* x, float* y, const float* partial, int splits, long split_stride, int only, const void* w,
                           int w_dtype, int n_rows, int width, int groups, float eps, cudaStream_t stream) {
    MDMA_REQUIRE(n_rows >= 0 && width > 0 && groups > 0 && width % groups == 0, "group_rmsnorm_add: %d numbers do not split into %d parts", width, groups);
    MDMA_REQUIRE(splits >= 0 && (splits == 0 || partial), "group_rmsnorm_add: partial sums need a pointer");
    MDMA_REQUIRE(splits == 0 || (((uintptr_t)partial & 15) == 0 && (split_stride & 3) == 0) || (width & 3) != 0, "group_rmsnorm_add: partial sums must be 16-byte aligned");
    if (n_rows == 0) return 0;
    MDMA_REQUIRE(!only || splits > 0, "group_rmsnorm_add: there are no partial sums");
    int slices, warps;
    group_norm_shape(width, groups, &slices, &warps);
    const int fours = (width & 3) == 0 && (((uintptr_t)x | (uintptr_t)y | (uintptr_t)w | (splits > 0 ? (uintptr_t)partial : 0)) & 15) == 0;
    MDMA_DISPATCH_DTYPE(w_dtype, TW,
        launch_chained(group_rmsnorm_kernel<TW, float, true>, dim3(n_rows), dim3(warps * 32), 0, stream, (const float*)y, y,
                       partial, splits, (size_t)split_stride, only, (const int*)nullptr, (const TW*)w, (float*)nullptr, x, width,
                       groups, slices, fours, eps));
    MDMA_LAUNCH_OK("group_rmsnorm_add");
    return 0;
}

int mdma_depth_mix(float* x, const float* x0, float* history, int depth, int run, const void* w, int w_dtype, int n_rows,
                   int width, cudaStream_t stream) {
    MDMA_REQUIRE(n_rows >= 0 && width > 0 && depth > 0 && run >= 0 && run < depth, "depth_mix: run %d of %d", run, depth);
    if (n_rows == 0) return 0;
    MDMA_DISPATCH_DTYPE(w_dtype, TW,
        launch_chained(depth_mix_kernel<TW>, dim3(n_rows, (width & 3) == 0 ? (width / 4 + 255) / 256 : (width + 1023) / 1024),
                       dim3(256), 0, stream, x, x0, history, depth, run, (const TW*)w, width));
    MDMA_LAUNCH_OK("depth_mix");
    return 0;
}

}  // extern "C"
