// The kernel of km_reg.cuh (included by the reg_*.cu translation units).
#pragma once

#include <algorithm>
#include <type_traits>

#include "km_pair.cuh"
#include "km_reg.cuh"

namespace kmc {
namespace reg {

// Certification of float64 labels by float32 scores.  In units scaled by the
// power of two sigma (largest |centroid coordinate| about 2^10), with u = 2^-24,
// x and c rounded to float32 and the sequential float32 dot product:
//   |score32 - score64| <= E_i = 1.002 u ((d + 3) ||x_i|| Cmax + 2 Hmax) + floor
// (d + 2 roundings of the products and operands, one of the subtraction, one of
// the half norm; the factor also covers the reference's own float64 rounding),
// floor for subnormal operands and products.  A sample whose best score is more
// than 2 E_i below the second best has the same winner in float64; any other
// (also every NaN or infinite bound) is evaluated in float64 by its warp.
struct Bound {
    float slope, base;  // E_i = slope ||x_i|| + base
};

template <int DP, int MODE, typename T, typename A>
__global__ void __launch_bounds__(max_threads(DP), 1) reg_kernel(Args<T, A> a) {
    wait_for_previous();
    if (a.guard != nullptr && *reinterpret_cast<const volatile int *>(&a.guard->done)) return;
    constexpr bool kF64 = sizeof(T) == 8;  // float64 samples: certified labels
    constexpr bool kPair = paired(DP, MODE), kDist = MODE == MODE_DIST;
    constexpr int S = samples_per_thread(DP), RS = row_floats(DP, MODE), KC = chunk_rows(DP, MODE);
    constexpr int S2 = S / 2;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t n = a.n, k = a.k;
    const int d = (int)a.d;
    const int kc = (int)(k < KC ? k : KC);
    float *cs = smem, *hs = smem + (size_t)kc * RS;
    // Always so: fits() admits fewer centroids.  Written as a choice because the
    // compiler schedules the float32 loops worse without the streamed form (1M x
    // 32, k = 64: 111 us with it, 120 to 135 without, in five ways of writing the
    // loop; a whole 200,003 x 32 estimator fit 2601 / 2735).
    const bool resident = k <= KC;

    float sigma = 1.f;
    Bound bound{0.f, 0.f};
    __shared__ float red_sh[32];
    auto block_max = [&](float v) {
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();
        if (lane == 0) red_sh[tid >> 5] = v;
        __syncthreads();
        v = red_sh[0];
        for (int q = 1; q < (int)(blockDim.x >> 5); ++q) v = fmaxf(v, red_sh[q]);
        return v;
    };
    if constexpr (kF64) {
        // sigma from the largest centroid coordinate (NaNs fail the
        // certification later: their scores never compare)
        float m = 0.f;
        for (int64_t e = tid; e < (int64_t)d * k; e += blockDim.x)
            m = fmaxf(m, fabsf((float)a.C[e]));
        m = block_max(m);
        const int ex = (int)(__float_as_uint(m) >> 23) - 127;
        const int sh = min(100, max(-100, 10 - ex));
        if (m > 0.f && m < pos_inf<float>()) sigma = __uint_as_float((unsigned)(127 + sh) << 23);
    }

    // Centroids j0 .. j0 + rows - 1 into shared memory; 8 centroids x 4
    // features per warp step.
    auto stage = [&](int64_t j0, int rows) {
        constexpr int Q = DP / 4;
        const int warps = blockDim.x >> 5, steps = ((rows + 7) / 8) * Q;
        const int jj = lane & 7, ff = lane >> 3;
        for (int t = tid >> 5; t < steps; t += warps) {
            const int j = (t / Q) * 8 + jj, f = (t % Q) * 4 + ff;
            if (j < rows) {
                float v = 0.f;
                if (f < d) v = (float)a.C[(int64_t)f * k + j0 + j];
                if (kF64) v *= sigma;
                if (kPair)
                    *reinterpret_cast<float2 *>(cs + (size_t)j * RS + 2 * f) = make_float2(v, v);
                else
                    cs[(size_t)j * RS + f] = v;
            }
        }
        if (!kDist)
            for (int j = tid; j < rows; j += blockDim.x) {
                if constexpr (kF64)
                    hs[j] = (float)((double)a.hn[j0 + j] * ((double)sigma * (double)sigma));
                else
                    hs[j] = a.hn[j0 + j];
            }
    };
    auto widen_bound = [&](int rows, float &c2, float &h) {
        for (int j = tid; j < rows; j += blockDim.x) {
            float q = 0.f;
            for (int f = 0; f < DP; ++f) {
                const float v = cs[(size_t)j * RS + (kPair ? 2 * f : f)];
                q = __fmaf_rn(v, v, q);
            }
            c2 = fmaxf(c2, q);
            h = fmaxf(h, fabsf(hs[j]));
        }
    };
    if (resident) stage(0, (int)k);
    __syncthreads();
    if constexpr (kF64) {
        float c2 = 0.f, h = 0.f;
        if (resident) {
            widen_bound((int)k, c2, h);
        } else {
            for (int64_t j0 = 0; j0 < k; j0 += kc) {
                const int rows = (int)(k - j0 < kc ? k - j0 : kc);
                stage(j0, rows);
                __syncthreads();
                widen_bound(rows, c2, h);
                __syncthreads();
            }
        }
        c2 = block_max(c2);
        h = block_max(h);
        const float cmax = __fadd_ru(__fsqrt_ru(__fmul_ru(c2, 1.f + 0x1p-15f)), 0x1p-60f);
        const float tiny = sigma * 0x1p-146f;  // 8 sigma 2^-149: subnormal operands
        bound.slope = __fadd_ru(__fmul_ru(1.002f * 0x1p-24f * (float)(d + 3), cmax), tiny);
        bound.base = __fadd_ru(__fmul_ru(1.002f * 0x1p-23f, h),
                               __fadd_ru(__fmul_ru(tiny, cmax), 0x1p-120f));
    }

    const int64_t wtiles = ceil_div<int64_t>(n, 32 * S);
    const int64_t wstride = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t wfirst = (int64_t)blockIdx.x * (blockDim.x >> 5) + (tid >> 5);
    // warps of a CTA step together only when they share streamed centroids
    const int64_t rounds = ceil_div<int64_t>(wtiles, wstride);
    for (int64_t r = 0; r < rounds; ++r) {
        const int64_t wt = wfirst + r * wstride;
        if (resident && wt >= wtiles) break;
        const int64_t i0 = wt * (32 * S) + lane;
        float x[S][DP];
#pragma unroll
        for (int f = 0; f < DP; ++f)
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int64_t i = i0 + 32 * s;
                float v = 0.f;
                if (f < d && i < n) v = (float)a.X[(int64_t)f * n + i];
                if (kF64) v *= sigma;
                x[s][f] = kDist ? -v : v;
            }
        u64 xp[kPair ? S2 : 1][kPair ? DP : 1];
        if constexpr (kPair) {
#pragma unroll
            for (int f = 0; f < DP; ++f)
#pragma unroll
                for (int p = 0; p < S2; ++p) xp[p][f] = pack(x[2 * p][f], x[2 * p + 1][f]);
        }
        float best[S], second[S];
        int idx[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            best[s] = second[s] = pos_inf<float>();
            idx[s] = 0;
        }

        for (int64_t j0 = 0; j0 < k; j0 += kc) {
            const int rows = (int)(k - j0 < kc ? k - j0 : kc);
            if (!resident) {
                __syncthreads();
                stage(j0, rows);
                __syncthreads();
            }
            const float *crow = cs;
            for (int j = 0; j < rows; ++j, crow += RS) {
                float v[S];
                if constexpr (kPair) {
                    u64 acc[S2];
#pragma unroll
                    for (int p = 0; p < S2; ++p) acc[p] = 0ull;
#pragma unroll
                    for (int f = 0; f < DP; f += 2) {
                        const ulonglong2 c = *reinterpret_cast<const ulonglong2 *>(crow + 2 * f);
#pragma unroll
                        for (int p = 0; p < S2; ++p) {
                            if (kDist) {
                                const u64 e0 = add2(c.x, xp[p][f]);
                                acc[p] = fma2(e0, e0, acc[p]);
                            } else {
                                acc[p] = fma2(xp[p][f], c.x, acc[p]);
                            }
                        }
#pragma unroll
                        for (int p = 0; p < S2; ++p) {
                            if (kDist) {
                                const u64 e1 = add2(c.y, xp[p][f + 1]);
                                acc[p] = fma2(e1, e1, acc[p]);
                            } else {
                                acc[p] = fma2(xp[p][f + 1], c.y, acc[p]);
                            }
                        }
                    }
#pragma unroll
                    for (int p = 0; p < S2; ++p) unpack(acc[p], v[2 * p], v[2 * p + 1]);
                } else {
#pragma unroll
                    for (int s = 0; s < S; ++s) v[s] = 0.f;
#pragma unroll
                    for (int f = 0; f < DP; f += 4) {
                        const float4 c = *reinterpret_cast<const float4 *>(crow + f);
#pragma unroll
                        for (int s = 0; s < S; ++s) v[s] = __fmaf_rn(x[s][f], c.x, v[s]);
#pragma unroll
                        for (int s = 0; s < S; ++s) v[s] = __fmaf_rn(x[s][f + 1], c.y, v[s]);
#pragma unroll
                        for (int s = 0; s < S; ++s) v[s] = __fmaf_rn(x[s][f + 2], c.z, v[s]);
#pragma unroll
                        for (int s = 0; s < S; ++s) v[s] = __fmaf_rn(x[s][f + 3], c.w, v[s]);
                    }
                }
                if constexpr (kDist) {
                    float *out = reinterpret_cast<float *>(a.dist) + (j0 + j) * n;
#pragma unroll
                    for (int s = 0; s < S; ++s)
                        if (i0 + 32 * s < n) out[i0 + 32 * s] = __fsqrt_rn(v[s]);
                } else {
                    const float h = hs[j];
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        const float e = h - v[s];
                        if (kF64) second[s] = fmaxf(best[s], fminf(second[s], e));
                        if (e < best[s]) {
                            best[s] = e;
                            idx[s] = (int)j0 + j;
                        }
                    }
                }
            }
        }
        if constexpr (kDist) continue;

        if constexpr (kF64) {
#pragma unroll
            for (int s = 0; s < S; ++s) {
                float q = 0.f;
#pragma unroll
                for (int f = 0; f < DP; ++f) q = __fmaf_rn(x[s][f], x[s][f], q);
                const float nx = __fadd_ru(__fsqrt_ru(__fmul_ru(q, 1.f + 0x1p-15f)), 0x1p-60f);
                const float e2 = 2.f * __fadd_ru(__fmul_ru(nx, bound.slope), bound.base);
                const bool sure = __fsub_rd(second[s], best[s]) > e2;
                unsigned todo = __ballot_sync(0xffffffffu, !sure && i0 + 32 * s < n);
                while (todo != 0u) {
                    // one uncertified sample at a time, the warp's lanes over its centroids
                    const int src = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    const T *xc = a.X + (i0 - lane + src + 32 * s);
                    const int bj = exact_label(xc, n, a.C, a.hn, d, k);
                    if (lane == src) idx[s] = bj;
                }
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int64_t i = i0 + 32 * s;
            if (i < n) {
                if (a.label64)
                    reinterpret_cast<int64_t *>(a.labels)[i] = idx[s];
                else
                    reinterpret_cast<int32_t *>(a.labels)[i] = idx[s];
            }
        }
        if constexpr (!kF64) {
            if (a.sums != nullptr) {
                // w x into this CTA's copy (this warp's, where there are more
                // copies than CTAs) with fire-and-forget reductions
                const int64_t copy = (a.P > (int64_t)gridDim.x ? wfirst : (int64_t)blockIdx.x) % a.P;
                A *sums = a.sums + copy * (int64_t)d * k, *sizes = a.sizes + copy * k;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const int64_t i = i0 + 32 * s;
                    if (i < n) {
                        const float wv = a.w[i];
                        A *p = sums + idx[s];
#pragma unroll
                        for (int f = 0; f < DP; ++f) {
                            if (f < d) {
                                float xv;
                                if constexpr (kPair) {
                                    float lo, hi;
                                    unpack(xp[s / 2][f], lo, hi);
                                    xv = (s & 1) ? hi : lo;
                                } else {
                                    xv = x[s][f];
                                }
                                const float t = __fmul_rn(xv, wv);
                                if constexpr (std::is_same<A, double>::value)
                                    atomicAdd(p, widen(t));
                                else
                                    atomicAdd(p, t);
                                p += k;
                            }
                        }
                        if constexpr (std::is_same<A, double>::value)
                            atomicAdd(sizes + idx[s], widen(wv));
                        else
                            atomicAdd(sizes + idx[s], wv);
                    }
                }
            }
        }
    }
}

template <int DP, int MODE, typename T, typename A>
int launch_class(const Args<T, A> &a, cudaStream_t s) {
    if (a.n == 0) return KMC_OK;
    auto kern = reg_kernel<DP, MODE, T, A>;
    const int64_t rows = std::min<int64_t>(a.k, chunk_rows(DP, MODE));
    const size_t smem = sizeof(float) * (size_t)rows * (row_floats(DP, MODE) + 1);
    static_assert(sizeof(float) * most_centroids(MODE) * (row_floats(DP, MODE) + 1) <= 47 * 1024,
                  "the centroids fit the shared memory that needs no opt-in");
    // one CTA per SM; few samples are spread over all SMs in smaller CTAs
    const int64_t wtiles = ceil_div<int64_t>(a.n, 32 * samples_per_thread(DP));
    const int64_t warps = std::max<int64_t>(
        1, std::min<int64_t>(max_threads(DP) / 32, ceil_div<int64_t>(wtiles, num_sms())));
    const int64_t grid = std::min<int64_t>(num_sms(), ceil_div<int64_t>(wtiles, warps));
    return launch_chained("reg_kernel", kern, dim3((unsigned)grid), dim3((unsigned)(32 * warps)), smem, s, a);
}

template <int MODE, typename T, typename A>
int launch_any(const Args<T, A> &a, cudaStream_t s) {
    if (a.d <= 4) return launch_class<4, MODE, T, A>(a, s);
    if (a.d <= 8) return launch_class<8, MODE, T, A>(a, s);
    if (a.d <= 12) return launch_class<12, MODE, T, A>(a, s);
    if (a.d <= 16) return launch_class<16, MODE, T, A>(a, s);
    if (a.d <= 20) return launch_class<20, MODE, T, A>(a, s);
    if (a.d <= 24) return launch_class<24, MODE, T, A>(a, s);
    if (a.d <= 28) return launch_class<28, MODE, T, A>(a, s);
    if (a.d <= 32) return launch_class<32, MODE, T, A>(a, s);
    if (a.d <= 40) return launch_class<40, MODE, T, A>(a, s);
    if (a.d <= 48) return launch_class<48, MODE, T, A>(a, s);
    if (a.d <= 56) return launch_class<56, MODE, T, A>(a, s);
    return launch_class<64, MODE, T, A>(a, s);
}

}  // namespace reg
}  // namespace kmc
