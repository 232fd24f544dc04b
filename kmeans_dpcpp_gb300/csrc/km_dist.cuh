// Squared distances of samples to the centroids of their labels
// (src/compute_inertia.hpp:11-99): acc = fma(x_f - c_f, x_f - c_f, acc) over
// f = 0..d-1, in that order.
#pragma once

#include "km_common.cuh"

namespace kmc {

// Predicated read-only loads (0 when not in).  Volatile: plain loads would be
// moved into a branch that uses them, one latency each.
__device__ __forceinline__ float4 load_f4_if(const float4 *p, bool in) {
    float4 v;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %5, 0;\n\t"
        "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
        "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
        "@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
        : "l"(p), "r"((uint32_t)in));
    return v;
}
__device__ __forceinline__ float load_f_if(const float *p, bool in) {
    float v;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %2, 0;\n\t"
        "mov.f32 %0, 0f00000000;\n\t"
        "@p ld.global.nc.f32 %0, [%1];\n\t}"
        : "=&f"(v)
        : "l"(p), "r"((uint32_t)in));
    return v;
}
__device__ __forceinline__ int load_i_if(const int *p, bool in) {
    int v;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.u32 p, %2, 0;\n\t"
        "mov.s32 %0, 0;\n\t"
        "@p ld.global.nc.s32 %0, [%1];\n\t}"
        : "=&r"(v)
        : "l"(p), "r"((uint32_t)in));
    return v;
}

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
        for (int u = 0; u < 8; ++u) acc = fma_rn(v[u], v[u], acc);
    }
    for (; f < d; ++f) {
        const T diff = x[f * fs] - q[f * k];
        acc = fma_rn(diff, diff, acc);
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

// Longer rows (16-byte aligned, padded as above): a warp takes 32 samples.  It
// reads 32 features at a time, eight lanes per row and four rows per load, of
// the samples and of their centroids, leaves the differences in its 32 x 33
// tile of shared memory, and each lane then continues its own sample's chain.
// c < 0: no such sample.  Returns lane r's squared distance.
// 10M x 64: 2.97 ms with a thread per row and 4-byte loads, 1.57 ms with a warp
// per row and feature, 0.52 ms (5.0 TB/s) now.
constexpr int kDistTile = 32 * 33;
__device__ __forceinline__ float sq_dist_warp(const float *X, int64_t ss, const float *C,
                                              int64_t cs, int64_t d, int64_t i0, int64_t c,
                                              float *tile) {
    constexpr int kBatch = 4;
    const int lane = threadIdx.x & 31, rr = lane >> 3, q = 4 * (lane & 7);
    float acc = 0.f;
    for (int64_t f0 = 0; f0 < d; f0 += 32) {
#pragma unroll
        for (int r0 = 0; r0 < 32; r0 += 4 * kBatch) {
            float4 x[kBatch], y[kBatch];
#pragma unroll
            for (int t = 0; t < kBatch; ++t) {
                const int r = r0 + 4 * t + rr;
                const int64_t cr = __shfl_sync(0xffffffffu, (int)c, r);
                const bool in = cr >= 0 && f0 + q < d;
                x[t] = load_f4_if(reinterpret_cast<const float4 *>(X + (i0 + r) * ss + f0 + q), in);
                y[t] = load_f4_if(reinterpret_cast<const float4 *>(C + cr * cs + f0 + q), in);
            }
#pragma unroll
            for (int t = 0; t < kBatch; ++t) {
                float *o = tile + (r0 + 4 * t + rr) * 33 + q;
                o[0] = x[t].x - y[t].x;
                o[1] = x[t].y - y[t].y;
                o[2] = x[t].z - y[t].z;
                o[3] = x[t].w - y[t].w;
            }
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
