// The kernel of km_panel.cuh (included by the panel_*.cu translation units).
#pragma once

#include "km_pair.cuh"
#include "km_panel.cuh"

namespace kmc {
namespace panel {

// The micro-tile's own: volatile keeps the order below, in which consecutive
// instructions share an operand (the register file delivers two of the three
// 64-bit operands per issue; 10M x 64 against 256 ran 13 % slower reordered).
__device__ __forceinline__ void fma2_acc(u64 &acc, u64 a, u64 b) {
    asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ void copy_async4(float *dst, const float *src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(in ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// Certification of float64 labels by float32 scores.  In units scaled by the
// power of two sigma (largest |centroid coordinate| about 2^10), with u = 2^-24,
// x and c rounded to float32 and the sequential float32 dot product:
//   |score32 - score64| <= E_ij = 1.002 u ((d + 3) ||x_i|| ||c_j|| + 2 |hn_j|) + floor
// (d + 2 roundings of the products and operands, one of the subtraction, one of
// the half norm; the factor also covers the reference's own float64 rounding),
// floor for subnormal operands and products.  With the maxima over j of the
// norms this is a bound per sample.
//
// One centroid far from all others would spoil it for every sample.  Centroids
// beyond `reach` (8 harmonic means of the norms) whose half norm is at least
// 0.49 ||c_j||^2 are left out of the maxima for samples with ||x_i|| <= reach / 4:
// their ||x_i|| ||c_j|| <= ||c_j||^2 / 4, so their scores are at least
// 0.24 ||c_j||^2 and E_ij <= u (1.05 d + 7.3) score_ij, a relative error.
//
// A sample whose second best score exceeds its best by more than
//   2 E_i + u (1.06 d + 8) (|best| + |second|)
// has the same winner in float64; any other (also every NaN or infinite bound)
// is evaluated in float64 by its warp.
struct Bound {
    float slope, base;            // E_i = slope ||x_i|| + base, centroids within reach
    float slope_all, base_all;    // all centroids
    float reach4, rel;            // reach / 4, u (1.06 d + 8)
};

// Samples (of the panel) and centroids (of the column block) of a thread.
__device__ __forceinline__ int row_of(int m, int ty) {
    return m < 4 ? ty * 4 + m : 16 + ty * 4 + (m - 4);
}
template <int TN>
__device__ __forceinline__ int col_of(int q, int tx) {
    return TN == 8 ? (q < 4 ? tx * 4 + q : 32 + tx * 4 + (q - 4)) : tx * TN + q;
}

// F consecutive features of the micro-tile: samples from the panel, centroids
// from a block of 8 TN columns.
template <int F, int TN, bool DIST>
__device__ __forceinline__ void features(const float *panel, const float *cs, int ty, int tx,
                                         u64 (&acc)[8][TN / 2]) {
    constexpr int BN = 8 * TN;
#pragma unroll
    for (int f = 0; f < F; ++f) {
        const float *ar = panel + f * kRows, *br = cs + f * BN;
        u64 a[8], b[TN / 2];
#pragma unroll
        for (int m = 0; m < 8; m += 4) {
            const float4 v = *reinterpret_cast<const float4 *>(ar + row_of(m, ty));
            a[m] = pack(v.x, v.x);
            a[m + 1] = pack(v.y, v.y);
            a[m + 2] = pack(v.z, v.z);
            a[m + 3] = pack(v.w, v.w);
        }
        if constexpr (TN == 8) {
            *reinterpret_cast<ulonglong2 *>(b) = *reinterpret_cast<const ulonglong2 *>(br + tx * 4);
            *reinterpret_cast<ulonglong2 *>(b + 2) =
                *reinterpret_cast<const ulonglong2 *>(br + 32 + tx * 4);
        } else if constexpr (TN == 4) {
            *reinterpret_cast<ulonglong2 *>(b) = *reinterpret_cast<const ulonglong2 *>(br + tx * 4);
        } else {
            b[0] = *reinterpret_cast<const u64 *>(br + tx * 2);
        }
#pragma unroll
        for (int m = 0; m < 8; ++m) {
#pragma unroll
            for (int qq = 0; qq < TN / 2; ++qq) {
                const int q = (m & 1) ? TN / 2 - 1 - qq : qq;
                if (DIST) {
                    const u64 e = fma2(b[q], pack(-1.f, -1.f), a[m]);  // x - c, rounded once
                    fma2_acc(acc[m][q], e, e);
                } else {
                    fma2_acc(acc[m][q], a[m], b[q]);
                }
            }
        }
    }
}

// Lexicographic (value, index) minimum of a thread's 8 samples over the 8 lanes
// (tx) that hold them: recursive halving, after which lane tx holds sample
// m = the returned row in v[0], j[0].
__device__ __forceinline__ int rowmin8(float (&v)[8], int (&j)[8], int tx) {
    int base = 0;
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
        const bool upper = (tx & h) != 0;
#pragma unroll
        for (int r = 0; r < h; ++r) {
            const float sv = upper ? v[r] : v[r + h];
            const int sj = upper ? j[r] : j[r + h];
            float kv = upper ? v[r + h] : v[r];
            int kj = upper ? j[r + h] : j[r];
            const float ov = __shfl_xor_sync(0xffffffffu, sv, h);
            const int oj = __shfl_xor_sync(0xffffffffu, sj, h);
            if (ov < kv || (ov == kv && oj < kj)) {
                kv = ov;
                kj = oj;
            }
            v[r] = kv;
            j[r] = kj;
        }
        if (upper) base += h;
    }
    return base;
}
// The same with the runner-up's value: s is the second smallest of the values
// seen so far (equal values count separately).
__device__ __forceinline__ int rowmin8_second(float (&v)[8], int (&j)[8], float (&s)[8], int tx) {
    int base = 0;
#pragma unroll
    for (int h = 4; h > 0; h >>= 1) {
        const bool upper = (tx & h) != 0;
#pragma unroll
        for (int r = 0; r < h; ++r) {
            const float ov = __shfl_xor_sync(0xffffffffu, upper ? v[r] : v[r + h], h);
            const int oj = __shfl_xor_sync(0xffffffffu, upper ? j[r] : j[r + h], h);
            const float os = __shfl_xor_sync(0xffffffffu, upper ? s[r] : s[r + h], h);
            const float kv = upper ? v[r + h] : v[r], ks = upper ? s[r + h] : s[r];
            const int kj = upper ? j[r + h] : j[r];
            const bool other = ov < kv || (ov == kv && oj < kj);
            s[r] = fminf(fminf(ks, os), fmaxf(kv, ov));
            v[r] = other ? ov : kv;
            j[r] = other ? oj : kj;
        }
        if (upper) base += h;
    }
    return base;
}

// Warp tiles first + warp, + step, ... < end of a's samples by the first
// `warps` warps of the CTA (the others only join its barriers); `copy`: the
// private copy of the sums.
template <int TN, int MODE, typename T, typename A>
__device__ __forceinline__ void run_panels(const Args<T, A> &a, int warps, int64_t first,
                                           int64_t end, int64_t step, int64_t copy, float *smem) {
    constexpr bool kF64 = sizeof(T) == 8, kDist = MODE == MODE_DIST;
    constexpr int BN = 8 * TN;
    __shared__ float red_sh[kMaxWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = lane & 7, ty = lane >> 3;
    const int64_t n = a.n, k = a.k;
    const int d = (int)a.d;
    const Shape L = shape(d, k, TN, MODE, warps);
    const int dp = L.dp;
    const bool idle = warp >= warps;  // holds no panel
    float *panel = smem + L.panels + (size_t)(idle ? 0 : warp) * dp * kRows;
    int *labs = reinterpret_cast<int *>(smem + L.labs) + (idle ? 0 : warp) * kRows;

    float sigma = 1.f;
    Bound bound{};
    auto block_max = [&](float v) {
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        __syncthreads();
        if (lane == 0) red_sh[warp] = v;
        __syncthreads();
        v = red_sh[0];
        for (int q = 1; q < (int)(blockDim.x >> 5); ++q) v = fmaxf(v, red_sh[q]);
        return v;
    };
    if constexpr (kF64) {
        // sigma and the bound from the centroids.  NaN coordinates do not
        // count: their scores never win, in float32 or in float64
        float m = 0.f;
        for (int64_t e = tid; e < (int64_t)d * k; e += blockDim.x)
            m = fmaxf(m, fabsf((float)a.C[e]));
        m = block_max(m);
        const int sh = min(100, max(-100, 10 - ((int)(__float_as_uint(m) >> 23) - 127)));
        if (m > 0.f && m < pos_inf<float>()) sigma = __uint_as_float((unsigned)(127 + sh) << 23);
        // Norms twice: first the reach, then the maxima.  A float32 sum of
        // squares is within (1 + u)^(d + 1) of the exact one.
        auto norm = [&](int64_t j) {
            float q = 0.f;
            for (int f = 0; f < d; ++f) {
                const float v = (float)a.C[(int64_t)f * k + j] * sigma;
                q = __fmaf_rn(v, v, q);
            }
            return __fsqrt_rn(q);
        };
        float inv = 0.f;
        for (int64_t j = tid; j < k; j += blockDim.x) inv += 1.f / norm(j);
        for (int o = 16; o > 0; o >>= 1) inv += __shfl_xor_sync(0xffffffffu, inv, o);
        __syncthreads();
        if (lane == 0) red_sh[warp] = inv;
        __syncthreads();
        inv = 0.f;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) inv += red_sh[q];
        const float reach = 8.f * (float)k / inv;  // 0 when a norm is
        float cn = 0.f, hn = 0.f, ca = 0.f, ha = 0.f, out_of_reach = 0.f;
        for (int64_t j = tid; j < k; j += blockDim.x) {
            const float c = norm(j);
            const float h = (float)((double)a.hn[j] * ((double)sigma * (double)sigma));
            ca = fmaxf(ca, c);
            ha = fmaxf(ha, fabsf(h));
            const bool far = c * (1.f - 0x1p-12f) > reach && h >= 0.4905f * c * c;
            if (far) {
                out_of_reach = 1.f;
            } else {
                cn = fmaxf(cn, c);
                hn = fmaxf(hn, fabsf(h));
            }
        }
        out_of_reach = block_max(out_of_reach);
        cn = block_max(cn);
        hn = block_max(hn);
        ca = block_max(ca);
        ha = block_max(ha);
        const float tiny = sigma * 0x1p-145f;  // 16 sigma 2^-149: subnormal operands
        auto slope = [&](float c) {
            c = __fadd_ru(__fmul_ru(c, 1.f + 0x1p-14f), 0x1p-60f);
            return __fadd_ru(__fmul_ru(1.002f * 0x1p-24f * (float)(d + 3), c), tiny);
        };
        const float floor0 = __fadd_ru(__fmul_ru(tiny, __fmul_ru(ca, 1.01f)), 0x1p-120f);
        bound.slope = slope(cn);
        bound.base = __fadd_ru(__fmul_ru(1.002f * 0x1p-23f, hn), floor0);
        bound.slope_all = slope(ca);
        bound.base_all = __fadd_ru(__fmul_ru(1.002f * 0x1p-23f, ha), floor0);
        bound.reach4 = 0.25f * reach;
        bound.rel = out_of_reach > 0.f ? (1.06f * (float)d + 8.f) * 0x1p-24f : 0.f;
    }

    // Columns j0 .. j0 + kp - 1 (zero beyond k), in blocks of BN columns
    // ([block][feature][column]), and their half norms
    auto stage = [&](int64_t j0, int buf) {
        float *cs = smem + L.c + (size_t)buf * BN * dp, *hs = smem + L.hn + (size_t)buf * BN;
        for (int f = warp; f < dp; f += (int)(blockDim.x >> 5))
            for (int c = lane; c < L.kp; c += 32) {
                float *dst = cs + ((size_t)(c / BN) * dp + f) * BN + c % BN;
                const bool in = f < d && j0 + c < k;
                if constexpr (kF64)
                    *dst = in ? (float)a.C[(int64_t)f * k + j0 + c] * sigma : 0.f;
                else
                    copy_async4(dst, in ? a.C + (int64_t)f * k + j0 + c : a.C, in);
            }
        if (!kDist)
            for (int c = tid; c < L.kp; c += blockDim.x) {
                float h = pos_inf<float>();
                if (j0 + c < k) {
                    if constexpr (kF64)
                        h = (float)((double)a.hn[j0 + c] * ((double)sigma * (double)sigma));
                    else
                        h = a.hn[j0 + c];
                }
                hs[c] = h;
            }
    };
    if (L.resident) {
        stage(0, 0);
        copy_wait_all();
        __syncthreads();
    }
    // a last odd feature has a row of zeros behind it
    if (dp > d && !idle) panel[d * kRows + lane] = 0.f;

    const int64_t rounds = end > first ? ceil_div<int64_t>(end - first, step) : 0;
    for (int64_t r = 0; r < rounds; ++r) {
        const int64_t wt = first + warp + r * step;
        // warps step together only when they share streamed columns
        const bool mine = !idle && wt < end;
        if (L.resident && !mine) break;
        const int64_t i0 = mine ? wt * kRows : n, i = i0 + lane;
        __syncwarp();
        if (mine) {
            if constexpr (kF64) {
                // eight features' loads in flight
                for (int f0 = 0; f0 < d; f0 += 8) {
                    T v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = f0 + u < d && i < n ? a.X[(int64_t)(f0 + u) * n + i] : T(0);
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (f0 + u < d) panel[(f0 + u) * kRows + lane] = (float)v[u] * sigma;
                }
            } else {
                for (int f = 0; f < d; ++f)
                    copy_async4(panel + f * kRows + lane, i < n ? a.X + (int64_t)f * n + i : a.X,
                                i < n);
            }
        }
        if (!L.resident) {
            __syncthreads();  // the last round's last block has been read
            stage(0, 0);
        }
        copy_wait_all();
        __syncwarp();
        float best[8], second[8];
        int bidx[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            best[m] = second[m] = pos_inf<float>();
            bidx[m] = 0;
        }
        int buf = 0;
        for (int64_t j0 = 0; j0 < k; j0 += BN) {
            const float *cs = smem + L.c, *hs = smem + L.hn;
            if (L.resident) {
                cs += j0 * dp;
                hs += j0;
            } else {
                // the next block travels while this one is used
                copy_wait_all();
                __syncthreads();
                if (j0 + BN < k) stage(j0 + BN, buf ^ 1);
                cs += (size_t)buf * BN * dp;
                hs += (size_t)buf * BN;
                buf ^= 1;
            }
            if (!mine) continue;
            u64 acc[8][TN / 2];
#pragma unroll
            for (int m = 0; m < 8; ++m)
#pragma unroll
                for (int q = 0; q < TN / 2; ++q) acc[m][q] = 0ull;
            // unrolled blocks: addresses are immediates, loads run ahead
            int f = 0;
#pragma unroll 1
            for (; f + 16 <= dp; f += 16)
                features<16, TN, kDist>(panel + f * kRows, cs + f * BN, ty, tx, acc);
            if (dp & 8) {
                features<8, TN, kDist>(panel + f * kRows, cs + f * BN, ty, tx, acc);
                f += 8;
            }
            if (dp & 4) {
                features<4, TN, kDist>(panel + f * kRows, cs + f * BN, ty, tx, acc);
                f += 4;
            }
            if (dp & 2) features<2, TN, kDist>(panel + f * kRows, cs + f * BN, ty, tx, acc);
            if constexpr (kDist) {
                // through shared memory, 32 centroids at a time, so that each
                // store writes 32 consecutive samples of a centroid; samples
                // are permuted within fours by their thread column, so that
                // the writes hit 32 different banks
                float *out = smem + L.out + (size_t)warp * kRows * 33;
#pragma unroll
                for (int half = 0; half < (BN + 31) / 32; ++half) {
#pragma unroll
                    for (int q = 0; q < TN / 2; ++q) {
                        const int c = col_of<TN>(2 * q, tx) - 32 * half;
                        if (c >= 0 && c < 32) {
#pragma unroll
                            for (int m = 0; m < 8; ++m) {
                                float v0, v1;
                                unpack(acc[m][q], v0, v1);
                                const int at = row_of(m, ty) ^ (tx & 3);
                                out[c * 33 + at] = v0;
                                out[(c + 1) * 33 + at] = v1;
                            }
                        }
                    }
                    __syncwarp();
                    const int64_t jb = j0 + 32 * half;
                    const int cn = (int)(k - jb < 32 ? (k - jb < 0 ? 0 : k - jb) : 32);
                    if (i < n) {
#pragma unroll 8
                        for (int c = 0; c < cn && c < BN; ++c)
                            a.dist[(jb + c) * n + i] =
                                __fsqrt_rn(out[c * 33 + (lane ^ ((TN == 2 ? c >> 1 : c >> 2) & 3))]);
                    }
                    __syncwarp();
                }
            } else {
                // ascending centroid order within this thread's columns
#pragma unroll
                for (int q = 0; q < TN / 2; ++q) {
                    const int c = col_of<TN>(2 * q, tx);
                    const u64 hh = *reinterpret_cast<const u64 *>(hs + c);
                    const int j = (int)j0 + c;
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        float v0, v1;
                        unpack(fma2(acc[m][q], pack(-1.f, -1.f), hh), v0, v1);  // hn - dot
                        if (kF64) second[m] = fmaxf(best[m], fminf(second[m], v0));
                        if (v0 < best[m]) {
                            best[m] = v0;
                            bidx[m] = j;
                        }
                        if (kF64) second[m] = fmaxf(best[m], fminf(second[m], v1));
                        if (v1 < best[m]) {
                            best[m] = v1;
                            bidx[m] = j + 1;
                        }
                    }
                }
            }
        }
        if (kDist || !mine) continue;

        if constexpr (kF64) {
            const int row = row_of(rowmin8_second(best, bidx, second, tx), ty);
            float q = 0.f;
            for (int f = 0; f < d; ++f) {
                const float v = panel[f * kRows + row];
                q = __fmaf_rn(v, v, q);
            }
            const float nx = __fadd_ru(__fsqrt_ru(__fmul_ru(q, 1.f + 0x1p-14f)), 0x1p-60f);
            const bool near = nx <= bound.reach4;
            const float e = near ? __fadd_ru(__fmul_ru(nx, bound.slope), bound.base)
                                 : __fadd_ru(__fmul_ru(nx, bound.slope_all), bound.base_all);
            float need = 2.f * e;
            if (bound.rel > 0.f)
                need = __fadd_ru(
                    need, __fmul_ru(bound.rel, __fadd_ru(fabsf(best[0]), fabsf(second[0]))));
            const bool sure = __fsub_rd(second[0], best[0]) > need;
            unsigned todo = __ballot_sync(0xffffffffu, !sure && i0 + row < n);
            while (todo != 0u) {
                // one undecided sample at a time, the warp's lanes over its centroids
                const int src = __ffs(todo) - 1;
                todo &= todo - 1u;
                const T *x = a.X + i0 + __shfl_sync(0xffffffffu, row, src);
                const int bj = exact_label(x, n, a.C, a.hn, d, k);
                if (lane == src) bidx[0] = bj;
            }
            labs[row] = bidx[0];
        } else {
            const int m = rowmin8(best, bidx, tx);
            labs[row_of(m, ty)] = bidx[0];
        }
        __syncwarp();
        const int lab = labs[lane];
        if (i < n) {
            if (a.label64)
                reinterpret_cast<int64_t *>(a.labels)[i] = lab;
            else
                reinterpret_cast<int32_t *>(a.labels)[i] = lab;
        }
        if constexpr (!kF64) {
            if (a.sums != nullptr && i < n) {
                // w x into this CTA's copy with fire-and-forget reductions
                A *p = a.sums + copy * (int64_t)d * k + lab;
                const float wv = a.w[i];
#pragma unroll 4
                for (int f = 0; f < d; ++f, p += k) {
                    const float v = __fmul_rn(panel[f * kRows + lane], wv);
                    if constexpr (sizeof(A) == 8)
                        atomicAdd(p, widen(v));
                    else
                        atomicAdd(p, v);
                }
                if constexpr (sizeof(A) == 8)
                    atomicAdd(a.sizes + copy * k + lab, widen(wv));
                else
                    atomicAdd(a.sizes + copy * k + lab, wv);
            }
        }
    }
}

template <int TN, int MODE, typename T, typename A>
__global__ void __launch_bounds__(32 * kMaxWarps, 1) panel_kernel(Args<T, A> a, int warps) {
    wait_for_previous();
    if (a.guard != nullptr && *reinterpret_cast<const volatile int *>(&a.guard->done)) return;
    extern __shared__ __align__(16) float smem[];
    run_panels<TN, MODE, T, A>(a, warps, (int64_t)blockIdx.x * warps,
                               ceil_div<int64_t>(a.n, kRows), (int64_t)gridDim.x * warps,
                               (a.P > (int64_t)gridDim.x ? (int64_t)blockIdx.x * warps + (threadIdx.x >> 5)
                                         : (int64_t)blockIdx.x) % a.P,
               smem);
}

template <int TN, int MODE, typename T, typename A>
int launch_width(const Args<T, A> &a, cudaStream_t s) {
    if (a.n == 0) return KMC_OK;
    auto kern = panel_kernel<TN, MODE, T, A>;
    // One CTA per SM.  Warps without samples help to load the centroids (2000 x
    // 64 against 1000: 171 us without them, 66 with).  Up to three rounds are
    // made equal: with all warps in the first and few samples left for the last,
    // 80,000 x 64 against 600 took 232 us instead of 180 (with more rounds the
    // last counts less than warps left out: distances of 400,003 x 30 to 250,
    // six rounds of 16 warps 289 us, of 14 295).  Not for float64, whose undecided
    // samples want all warps (80,000 x 64 against 600: 321 us, in equal rounds 441).
    const int64_t wtiles = ceil_div<int64_t>(a.n, kRows), sms = num_sms();
    const int all = warps_for(a.d, MODE);
    int64_t rounds = ceil_div<int64_t>(wtiles, sms * all);
    if (sizeof(T) == 8 || rounds > 3) rounds = 1;
    const int warps = (int)std::min<int64_t>(all, ceil_div<int64_t>(wtiles, sms * rounds));
    const size_t smem = sizeof(float) * shape(a.d, a.k, TN, MODE, warps).total;
    KMC_TRY(allow_smem(kern, kSmemBytes));
    const int64_t grid = std::min<int64_t>(num_sms(), ceil_div<int64_t>(wtiles, warps));
    return launch_chained("panel", kern, dim3((unsigned)grid), dim3((unsigned)(32 * all)), smem, s, a,
                          warps);
}

// Columns of a step: 64, 32 or 16, whichever pads k least for its rate (the
// narrower micro-tiles reuse each operand less).
inline int columns_per_thread(int64_t k) {
    int best = 8;
    double cost = 1e300;
    const int tn[3] = {8, 4, 2};
    const double rate[3] = {1.0, 0.85, 0.6};
    for (int v = 0; v < 3; ++v) {
        const double c = (double)(ceil_div<int64_t>(k, 8 * tn[v]) * 8 * tn[v]) / rate[v];
        if (c < cost) {
            cost = c;
            best = tn[v];
        }
    }
    return best;
}

template <int MODE, typename T, typename A>
int launch_any(const Args<T, A> &a, cudaStream_t s) {
    const int tn = columns_per_thread(a.k);
    if (tn == 8) return launch_width<8, MODE, T, A>(a, s);
    if (tn == 4) return launch_width<4, MODE, T, A>(a, s);
    return launch_width<2, MODE, T, A>(a, s);
}

}  // namespace panel
}  // namespace kmc
