// Device helpers of the label kernels (km_reg_kernel.cuh, km_panel_kernel.cuh):
// paired float32 arithmetic, widening, and the float64 label of one sample.
#pragma once

#include "km_common.cuh"

namespace kmc {

using u64 = unsigned long long;

__device__ __forceinline__ u64 pack(float lo, float hi) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack(u64 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// float -> double.  The conversion instruction shares the float64 unit (2 per
// clock and SM); a normal float is widened with integer operations instead.
__device__ __forceinline__ double widen(float v) {
    const unsigned b = __float_as_uint(v), e = (b >> 23) & 0xffu;
    if (e - 1u < 254u)
        return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)),
                                (int)(b << 29));
    return (double)v;
}

// The label of one float64 sample, x[f * n], in float64 by a whole warp: the
// reference's arithmetic and first minimum, the lanes over the centroids.
template <typename T>
__device__ __forceinline__ int exact_label(const T *x, int64_t n, const T *C, const T *hn, int d,
                                           int64_t k) {
    T bv = pos_inf<T>();
    int bj = 0;
    for (int64_t j = threadIdx.x & 31; j < k; j += 32) {
        T dot = T(0);
#pragma unroll 4
        for (int f = 0; f < d; ++f) dot = fma_rn(x[(int64_t)f * n], C[(int64_t)f * k + j], dot);
        const T e = hn[j] - dot;
        if (e < bv) {
            bv = e;
            bj = (int)j;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const T ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
        if (ov < bv || (ov == bv && oj < bj)) {
            bv = ov;
            bj = oj;
        }
    }
    return bj;
}

}  // namespace kmc
