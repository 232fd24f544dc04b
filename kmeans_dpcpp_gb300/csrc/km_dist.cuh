// Squared distances of samples to the centroids of their labels
// (src/compute_inertia.hpp:11-99): acc = fma(x_f - c_f, x_f - c_f, acc) over
// f = 0..d-1, in that order.
#pragma once

#include "km_common.cuh"

namespace kmc {

__device__ __forceinline__ float fma_dist(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_dist(double a, double b, double c) { return __fma_rn(a, b, c); }

// Feature-major X (element (f, i) at X[f * fs + i * ss]), C (d, k): one thread
// per sample; eight features' loads in flight before the sequential chain.
template <typename T>
__device__ __forceinline__ T sq_dist_cols(const T *X, int64_t fs, int64_t ss, const T *C, int64_t d,
                                          int64_t k, int64_t i, int64_t c) {
    T acc = T(0);
    const T *x = X + i * ss, *q = C + c;
    int64_t f = 0;
    for (; f + 8 <= d; f += 8) {
        T v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = x[(f + u) * fs] - q[(f + u) * k];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = fma_dist(v[u], v[u], acc);
    }
    for (; f < d; ++f) {
        const T diff = x[f * fs] - q[f * k];
        acc = fma_dist(diff, diff, acc);
    }
    return acc;
}

// Row-major X and C of at most kRowVec features, rows padded with zeros to a
// multiple of four: one thread per sample, four features per load.
constexpr int64_t kRowVec = 32;
__device__ __forceinline__ float sq_dist_row(const float *x, const float *q, int64_t d) {
    float acc = 0.f;
#pragma unroll 4
    for (int64_t f = 0; f < d; f += 4) {
        const float4 a = *reinterpret_cast<const float4 *>(x + f);
        const float4 b = *reinterpret_cast<const float4 *>(q + f);
        const float d0 = a.x - b.x, d1 = a.y - b.y, d2 = a.z - b.z, d3 = a.w - b.w;
        acc = __fmaf_rn(d0, d0, acc);
        acc = __fmaf_rn(d1, d1, acc);
        acc = __fmaf_rn(d2, d2, acc);
        acc = __fmaf_rn(d3, d3, acc);
    }
    return acc;
}

// Longer rows: a warp takes 32 samples.  It reads 32 features of one sample
// and of its centroid at a time (whole 128-byte lines; a thread per row would
// touch 32 lines per load), leaves the differences in its 32 x 33 tile of
// shared memory, and each lane then continues its own sample's chain.
// c < 0: no such sample.  Returns lane r's squared distance.
constexpr int kDistTile = 32 * 33;
__device__ __forceinline__ float sq_dist_warp(const float *X, int64_t ss, const float *C,
                                              int64_t cs, int64_t d, int64_t i0, int64_t c,
                                              float *tile) {
    const int lane = threadIdx.x & 31;
    float acc = 0.f;
    for (int64_t f0 = 0; f0 < d; f0 += 32) {
        const bool in = f0 + lane < d;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
            const long long cr = __shfl_sync(0xffffffffu, (long long)c, r);
            float v = 0.f;
            if (in && cr >= 0) v = X[(i0 + r) * ss + f0 + lane] - __ldg(C + cr * cs + f0 + lane);
            tile[r * 33 + lane] = v;
        }
        __syncwarp();
        const int fn = d - f0 < 32 ? (int)(d - f0) : 32;
#pragma unroll 8
        for (int f = 0; f < fn; ++f) {
            const float v = tile[lane * 33 + f];
            acc = __fmaf_rn(v, v, acc);
        }
        __syncwarp();
    }
    return acc;
}

}  // namespace kmc
