// Initialisation and input-layout kernels in front of the Lloyd path (the
// steps before the reference's driver, which takes X_t and initial centroids
// as given, python_api/_kmeans_lloyd.cpp:1153):
//   transpose     row-major X (n, d) -> the feature-major X_t (d, n) the
//                 engine reads, 32 x 32 tiles staged through shared memory so
//                 that both the reads and the writes are coalesced
//   gather_rows   C_t[:, j] = X_t[:, rows[j]] (random-row initialisation)
//   k-means++     D^2-weighted seeding (Arthur and Vassilvitskii, 2007), fully
//                 on the device and deterministic for a seed:
//                   draw u_t = SplitMix64(seed, t) / 2^64 in [0, 1)
//                   pick the first i whose running sum of v_i exceeds
//                   u_t * sum(v), with v_i = w_i (t = 0) or
//                   w_i * min_j ||x_i - c_j||^2 (t > 0) in float64, summed
//                   sequentially within fixed blocks of 4096 samples and then
//                   over the blocks in order
//                 so that a sequential CPU restatement selects the same rows.
//                 Squared distances use the engine's order: one fused
//                 multiply-add per feature, f = 0..d-1.
#include <cstdint>
#include <vector>

#include "km_kernels.cuh"
#include "kmeans_gb300.h"

namespace kmc {
namespace {

constexpr int kPPBlock = 4096;  // samples per partial sum of the k-means++ draw

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
    // SplitMix64 output function (S. Vigna, public domain)
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

template <typename T>
__global__ void transpose_kernel(const T *X, T *Xt, int64_t n, int64_t d) {
    __shared__ T tile[32][33];
    const int64_t i0 = (int64_t)blockIdx.x * 32, f0 = (int64_t)blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int64_t i = i0 + r, f = f0 + threadIdx.x;
        if (i < n && f < d) tile[r][threadIdx.x] = X[i * d + f];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int64_t f = f0 + r, i = i0 + threadIdx.x;
        if (i < n && f < d) Xt[f * n + i] = tile[threadIdx.x][r];
    }
}

template <typename T>
__global__ void gather_kernel(const T *Xt, int64_t n, int64_t d, const int32_t *rows, int64_t k,
                              T *Ct, int *bad) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < d * k;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t f = e / k, j = e % k;
        const int64_t i = rows[j];
        if (i >= 0 && i < n) {
            Ct[e] = Xt[f * n + i];
        } else {
            Ct[e] = T(0);
            atomicOr(bad, 1);
        }
    }
}

// k-means++ draw, one launch per centre.  Each CTA takes blocks of kPPBlock
// samples: it lowers the samples' min_d2 by the distance to the previous
// centre (one fused multiply-add per feature, f = 0..d-1) and forms the
// block's sum of v_i in the defined order; the CTA that finishes last walks
// the block sums and the chosen block, records the sample and copies its row.
//
// The defined order is sequential, one float64 addition after another, and
// float64 additions are slow here (2 per clock and SM), so a thread summing a
// block of 4096 samples from global memory took 0.55 ms whatever n.  A sum of
// non-negative terms that are all multiples of some power of two L and stay
// below 2^53 L is exact in any order, so it is formed by a tree whenever that
// holds (exact_key below; unit weights and float32 data nearly always) and
// sequentially, from shared memory, otherwise.  Updating, summing and picking
// in one launch leaves one pass over X_t per centre.  A whole estimator fit of
// 200,003 x 32, 64 centres, 20 iterations: 70.8 -> 7.8 ms, labels unchanged.
//
// A block is split into kPPParts parts, a CTA's work at a time, so that few
// samples still fill the SMs (a CTA per block: 49 CTAs and 42 us per centre at
// 200,003 x 32, now 15 us).  The CTA that finishes a block's last part forms the
// block's sum, and the one that finishes the last block draws; the parts' sums
// also narrow the draw to one part, which a single warp searches.
constexpr int kPPThreads = 256;
constexpr int kPPOwn = kPPBlock / kPPThreads;  // samples per thread and block
constexpr int kPPParts = 8;
constexpr int kPPPart = kPPBlock / kPPParts;
constexpr int kPPMine = kPPPart / kPPThreads;  // samples per thread and part
constexpr int kPPWarpBlocks = 1024;  // block sums that one warp draws from
constexpr int kPPWarps = kPPThreads / 32;
constexpr int kKeyNone = 1 << 20, kKeyFail = -(1 << 20);

// Exponent field of v's lowest set bit plus 52: v is a multiple of
// 2^(key - 1075), and a float64 with exponent field E holds every multiple of
// 2^(key - 1075) up to its magnitude when key >= E.  Zero divides by
// everything; negative, subnormal, infinite and NaN values never qualify.
__device__ __forceinline__ int exact_key(double v) {
    const long long b = __double_as_longlong(v);
    if ((b & 0x7fffffffffffffffll) == 0) return kKeyNone;
    const int e = (int)((b >> 52) & 0x7ff);
    if (b < 0 || e == 0 || e == 0x7ff) return kKeyFail;
    return e + __ffsll((b & 0xfffffffffffffll) | 0x10000000000000ll) - 1;
}
__device__ __forceinline__ int exponent_field(double v) {
    return (int)((__double_as_longlong(v) >> 52) & 0x7ff);
}

// Sums whose terms are all multiples of L = 2^(key - 1075) and stay below
// 2^53 L are formed in units of L with 64-bit integers: float64 operations run
// at 2 per clock and SM with 60 clocks of latency (the draw took 19 K of a
// centre's 33 K clocks with them).

// v / L; v a non-negative multiple of L.  ok is cleared at 2^53 and above.
__device__ __forceinline__ long long units_of(double v, int key, bool &ok) {
    const long long b = __double_as_longlong(v);
    if (b == 0) return 0;
    const int s = exponent_field(v) - key;
    if (s > 0) {
        ok = false;
        return 0;
    }
    return s < -52 ? 0 : ((b & 0xfffffffffffffll) | 0x10000000000000ll) >> -s;
}
// units L as a float64; exact below 2^53.
__device__ __forceinline__ double from_units(long long units, int key) {
    return units == 0 ? 0.0 : ldexp((double)units, key - 1075);
}

// w m = p 2^(e - 1075) of two floats, p < 2^48 exact; false when negative,
// infinite or NaN.
__device__ __forceinline__ bool float_term(float w, float m, unsigned long long &p, int &e) {
    const unsigned a = __float_as_uint(w), b = __float_as_uint(m);
    const unsigned ea = (a >> 23) & 0xffu, eb = (b >> 23) & 0xffu;
    const unsigned ma = (a & 0x7fffffu) | (ea != 0u ? 0x800000u : 0u);
    const unsigned mb = (b & 0x7fffffu) | (eb != 0u ? 0x800000u : 0u);
    p = (unsigned long long)ma * mb;
    e = (int)(max(ea, 1u) + max(eb, 1u)) - 300 + 1075;
    return ea != 255u && eb != 255u && (p == 0 || (a | b) >> 31 == 0u);
}
__device__ __forceinline__ int term_key(unsigned long long p, int e) {
    return p == 0 ? kKeyNone : e + __ffsll((long long)p) - 1;
}
__device__ __forceinline__ long long term_units(unsigned long long p, int e, int key, bool &ok) {
    if (p == 0) return 0;
    const int s = e - key;
    if (64 - __clzll((long long)p) + s > 53) {
        ok = false;
        return 0;
    }
    return (long long)(s >= 0 ? p << s : p >> -s);
}

// Block-wide sum (tree) and minimum key; valid in every thread.
struct PPShared {
    double v[kPPBlock];
    double wsum[kPPWarps];
    int wkey[kPPWarps];
    long long usum[kPPWarps];
    double scalar;
    int first, last;
    int flag;
};

__device__ __forceinline__ void pp_block_sum(PPShared &sh, double &sum, int &key) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        key = min(key, __shfl_xor_sync(0xffffffffu, key, o));
    }
    __syncthreads();  // earlier readers of wsum / wkey are done
    if (lane == 0) {
        sh.wsum[wid] = sum;
        sh.wkey[wid] = key;
    }
    __syncthreads();
    if (wid == 0) {
        // float64 additions share 2 lanes per clock: by one warp only
        sum = lane < kPPWarps ? sh.wsum[lane] : 0.0;
        key = lane < kPPWarps ? sh.wkey[lane] : kKeyNone;
        for (int o = kPPWarps / 2; o > 0; o >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
            key = min(key, __shfl_xor_sync(0xffffffffu, key, o));
        }
        __syncwarp();
        if (lane == 0) {
            sh.wsum[0] = sum;
            sh.wkey[0] = key;
        }
    }
    __syncthreads();
    sum = sh.wsum[0];
    key = sh.wkey[0];
}

// Sum of sh.v[0..count) added to `run` one after another (thread 0), each
// running value written back to sh.v when `keep`.
__device__ __forceinline__ double pp_sequential(PPShared &sh, double run, int count, bool keep) {
    int q = 0;
    for (; q + 8 <= count; q += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = sh.v[q + u];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            run += x[u];
            if (keep) sh.v[q + u] = run;
        }
    }
    for (; q < count; ++q) {
        run += sh.v[q];
        if (keep) sh.v[q] = run;
    }
    return run;
}

// Exclusive block-wide scan of one value per thread (sums exact by the
// caller's check, so any association gives the same bits).
__device__ __forceinline__ double pp_exclusive(PPShared &sh, double x) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double inc = x;
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    double exc = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) exc = 0.0;
    __syncthreads();
    if (lane == 31) sh.wsum[wid] = inc;
    __syncthreads();
    double before = 0.0;
    for (int q = 0; q < wid; ++q) before += sh.wsum[q];
    return before + exc;
}

// v of sample i.
template <typename T>
__device__ __forceinline__ double pp_value(const T *w, const T *min_d2, int64_t i, int t) {
    const double v = w ? (double)w[i] : 1.0;
    return t > 0 ? __dmul_rn(v, (double)__ldcg(min_d2 + i)) : v;
}

// The draw among exact sums, by one warp and in units of their common L: the
// block, its part, the sample.  Returns -1 when some sum's order matters (or
// none exceeds the target).
template <typename T>
__device__ __forceinline__ int64_t pp_draw_exact(const T *w, const T *min_d2, int64_t n, int64_t nb,
                                                 int t, double u, const double *partials,
                                                 const int *keys, const double *parts) {
    const int lane = threadIdx.x & 31;
    const int per = (int)((nb + 31) / 32);
    const int b0 = min(lane * per, (int)nb), b1 = min(b0 + per, (int)nb);
    auto scan = [&](long long x) {
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        return x;
    };
    auto least = [&](int x) { return __reduce_min_sync(0xffffffffu, x); };
    bool ok = true;
    int key = kKeyNone;
    for (int q = b0; q < b1; ++q) key = min(key, __ldcg(keys + q));
    key = least(key);
    if (key == kKeyNone || key < 0) return -1;  // nothing to draw, or an order that matters
    long long own = 0;
    for (int q = b0; q < b1; ++q) own += units_of(__ldcg(partials + q), key, ok);
    const long long incl = scan(own), total = __shfl_sync(0xffffffffu, incl, 31);
    if (__any_sync(0xffffffffu, !ok) || total >= (1ll << 53)) return -1;
    // a running sum exceeds the target when its units exceed the target's floor
    const double target = u * from_units(total, key);
    bool fits = true;
    long long goal = 0;
    {
        const int s = exponent_field(target) - key;
        if (target > 0.0 && exponent_field(target) > 0 && s > -53)
            goal = units_of(target, key, fits);
    }
    if (!fits) return -1;
    long long run = incl - own, before = 0;
    int mine = (int)nb;
    for (int q = b0; q < b1 && mine == (int)nb; ++q) {
        before = run;
        run += units_of(__ldcg(partials + q), key, ok);
        if (run > goal) mine = q;
    }
    const int b = least(mine);
    if (b >= (int)nb) return -1;
    before = __shfl_sync(0xffffffffu, before, __ffs(__ballot_sync(0xffffffffu, mine == b)) - 1);
    // the part
    const long long part =
        lane < kPPParts && (int64_t)b * kPPBlock + (int64_t)lane * kPPPart < n
            ? units_of(__ldcg(parts + (int64_t)b * kPPParts + lane), key, ok)
            : 0;
    const long long pincl = before + scan(part);
    const unsigned past = __ballot_sync(0xffffffffu, lane < kPPParts && pincl > goal);
    if (past == 0u) return -1;
    const int p = __ffs(past) - 1;
    before = __shfl_sync(0xffffffffu, pincl - part, p);
    // the sample: consecutive ones per lane, their loads unconditional and in
    // flight together
    constexpr int kOwn = kPPPart / 32;
    const int64_t i0 = (int64_t)b * kPPBlock + p * kPPPart + lane * kOwn;
    long long v[kOwn], sum = 0;
    {
        T m[kOwn], wv[kOwn];
#pragma unroll
        for (int r = 0; r < kOwn; ++r) m[r] = t > 0 ? __ldcg(min_d2 + min(i0 + r, n - 1)) : T(1);
#pragma unroll
        for (int r = 0; r < kOwn; ++r) wv[r] = w ? w[min(i0 + r, n - 1)] : T(1);
#pragma unroll
        for (int r = 0; r < kOwn; ++r) {
            if constexpr (sizeof(T) == 4) {
                unsigned long long q;
                int e;
                ok = float_term(wv[r], m[r], q, e) && ok;
                v[r] = term_units(q, e, key, ok);
            } else {
                v[r] = units_of(__dmul_rn((double)wv[r], (double)m[r]), key, ok);
            }
            if (i0 + r >= n) v[r] = 0;
            sum += v[r];
        }
    }
    long long x = before + scan(sum) - sum;
    int hit = kPPPart;
#pragma unroll
    for (int r = 0; r < kOwn; ++r) {
        x += v[r];
        if (hit == kPPPart && v[r] > 0 && x > goal) hit = lane * kOwn + r;
    }
    hit = least(hit);
    return hit < kPPPart ? (int64_t)b * kPPBlock + p * kPPPart + hit : -1;
}

// Sum of one part's v and its key (kKeyFail: the order matters), valid in every
// thread; float data in units of L.
__device__ __forceinline__ void pp_part_sum(PPShared &sh, const unsigned long long (&p)[kPPMine],
                                            const int (&e)[kPPMine], bool valid, double &sum,
                                            int &key) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    key = kKeyNone;
#pragma unroll
    for (int r = 0; r < kPPMine; ++r) key = min(key, term_key(p[r], e[r]));
    key = __reduce_min_sync(0xffffffffu, valid ? key : kKeyFail);
    if (lane == 0) sh.wkey[wid] = key;
    __syncthreads();
    key = kKeyNone;
#pragma unroll
    for (int q = 0; q < kPPWarps; ++q) key = min(key, sh.wkey[q]);
    long long units = 0;
    bool ok = key >= 0;
    if (ok) {
#pragma unroll
        for (int r = 0; r < kPPMine; ++r) units += term_units(p[r], e[r], key, ok);
    }
    for (int o = 16; o > 0; o >>= 1) units += __shfl_xor_sync(0xffffffffu, units, o);
    if (lane == 0) sh.usum[wid] = units;
    ok = !__syncthreads_or(!ok);
    units = 0;
#pragma unroll
    for (int q = 0; q < kPPWarps; ++q) units += sh.usum[q];
    if (!ok || units >= (1ll << 53)) key = kKeyFail;
    sum = key == kKeyFail || key == kKeyNone ? 0.0 : from_units(units, key);
}

template <typename T>
__global__ void __launch_bounds__(kPPThreads) pp_step_kernel(
    const T *__restrict__ Xt, const T *__restrict__ w, T *min_d2, int64_t n, int64_t d, int64_t k,
    int t, uint64_t seed, double *partials, double *prefix, int *keys, double *parts, int *part_keys,
    unsigned *arrived, int32_t *chosen, T *Ct, unsigned *ticket) {
    wait_for_previous();
    allow_next();
    __shared__ PPShared sh;
    __shared__ T centre[kPPThreads];
    const int tid = threadIdx.x;
    const int64_t nb = (n + kPPBlock - 1) / kPPBlock, items = (n + kPPPart - 1) / kPPPart;
    bool last_of_all = false;

    for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const int64_t i0 = item * kPPPart;
        T acc[kPPMine];
#pragma unroll
        for (int r = 0; r < kPPMine; ++r) acc[r] = T(0);
        for (int64_t f0 = 0; t > 0 && f0 < d; f0 += kPPThreads) {
            __syncthreads();
            // the previous centre
            if (f0 + tid < d) centre[tid] = Ct[(f0 + tid) * k + t - 1];
            __syncthreads();
            const int fn = (int)(d - f0 < kPPThreads ? d - f0 : kPPThreads);
            const T *row = Xt + f0 * n + i0 + tid;
            if (i0 + kPPPart <= n) {
#pragma unroll 8
                for (int f = 0; f < fn; ++f) {
                    const T cf = centre[f];
#pragma unroll
                    for (int r = 0; r < kPPMine; ++r) {
                        const T diff = row[f * n + r * kPPThreads] - cf;
                        acc[r] = fma_rn(diff, diff, acc[r]);
                    }
                }
            } else if (i0 + (tid & ~31) < n) {
                // A ragged part: warps leave out the samples that all lie past the
                // end (a predicate alone would still cost the float64 unit its
                // slots: 42 samples of 163 features took 59 us per centre in
                // float64, 32 now); the last sample stands for the others past the
                // end, so that no load waits behind a condition.
                static_assert(kPPMine == 2, "one or two samples of a thread");
                const int64_t i = i0 + tid;
                const T *x0 = Xt + f0 * n + min(i, n - 1);
                const T *x1 = Xt + f0 * n + min(i + kPPThreads, n - 1);
                if (i0 + (tid & ~31) + kPPThreads < n) {
#pragma unroll 8
                    for (int f = 0; f < fn; ++f) {
                        const T d0 = x0[f * n] - centre[f], d1 = x1[f * n] - centre[f];
                        acc[0] = fma_rn(d0, d0, acc[0]);
                        acc[1] = fma_rn(d1, d1, acc[1]);
                    }
                } else {
#pragma unroll 8
                    for (int f = 0; f < fn; ++f) {
                        const T d0 = x0[f * n] - centre[f];
                        acc[0] = fma_rn(d0, d0, acc[0]);
                    }
                }
            }
        }
        double sum = 0.0;
        int key = kKeyNone;
        T old[kPPMine], wv[kPPMine], m[kPPMine];
#pragma unroll
        for (int r = 0; r < kPPMine; ++r) {
            const int64_t i = min(i0 + tid + r * kPPThreads, n - 1);
            old[r] = t > 1 ? min_d2[i] : T(0);
            wv[r] = w ? w[i] : T(1);
        }
#pragma unroll
        for (int r = 0; r < kPPMine; ++r) {
            const int64_t i = i0 + tid + r * kPPThreads;
            m[r] = T(1);
            if (t > 0) {
                m[r] = acc[r];
                if (t > 1) m[r] = (m[r] < old[r]) ? m[r] : old[r];
                if (i < n) min_d2[i] = m[r];
            }
            if (i >= n) wv[r] = m[r] = T(0);
        }
        if constexpr (sizeof(T) == 4) {
            unsigned long long p[kPPMine];
            int e[kPPMine];
            bool valid = true;
#pragma unroll
            for (int r = 0; r < kPPMine; ++r) valid = float_term(wv[r], m[r], p[r], e[r]) && valid;
            pp_part_sum(sh, p, e, valid, sum, key);
        } else {
#pragma unroll
            for (int r = 0; r < kPPMine; ++r) {
                const double v = __dmul_rn((double)wv[r], (double)m[r]);
                sum += v;
                key = min(key, exact_key(v));
            }
            pp_block_sum(sh, sum, key);
        }
        // the CTA that finishes the block's last part sums the block
        const int64_t b = item / kPPParts;
        const int have = (int)(items - b * kPPParts < kPPParts ? items - b * kPPParts : kPPParts);
        if (tid == 0) {
            parts[item] = sum;
            part_keys[item] = key;
            __threadfence();
            sh.flag = atomicAdd(arrived + b, 1u) == (unsigned)have - 1u;
        }
        __syncthreads();
        if (!sh.flag) continue;
        __threadfence();
        if (tid < 32) {
            double all = tid < have ? __ldcg(parts + b * kPPParts + tid) : 0.0;
            int least = tid < have ? __ldcg(part_keys + b * kPPParts + tid) : kKeyNone;
            for (int o = kPPParts / 2; o > 0; o >>= 1) {
                all += __shfl_xor_sync(0xffffffffu, all, o);
                least = min(least, __shfl_xor_sync(0xffffffffu, least, o));
            }
            if (tid == 0) {
                sh.scalar = all;
                sh.first = least >= exponent_field(all) ? least : kKeyFail;
            }
        }
        __syncthreads();
        double block_sum = sh.scalar;
        const int block_key = sh.first;
        if (block_key == kKeyFail) {
            const int64_t j0 = b * kPPBlock;
            const int count = (int)(n - j0 < kPPBlock ? n - j0 : kPPBlock);
            for (int q = tid; q < count; q += kPPThreads) sh.v[q] = pp_value(w, min_d2, j0 + q, t);
            __syncthreads();
            if (tid == 0) block_sum = pp_sequential(sh, 0.0, count, false);
        }
        if (tid == 0) {
            partials[b] = block_sum;
            keys[b] = block_key;
            arrived[b] = 0u;  // for the next centre's launch
            __threadfence();
            sh.flag = atomicAdd(ticket, 1u) == (unsigned)nb - 1u;
        }
        __syncthreads();
        // the last block: nothing is left for any CTA
        last_of_all = sh.flag;
        __syncthreads();  // sh.flag is rewritten by the next part
    }
    if (!last_of_all) return;
    __threadfence();

    // the CTA that finished the last block draws the sample
    const double u = (double)(splitmix64(seed ^ splitmix64((uint64_t)t)) >> 11) * 0x1p-53;
    if (nb <= kPPWarpBlocks) {
        if (tid < 32) {
            const int64_t hit = pp_draw_exact(w, min_d2, n, nb, t, u, partials, keys, parts);
            if (tid == 0) sh.first = (int)hit;  // n < 2^31
        }
        __syncthreads();
        const int64_t hit = sh.first;
        if (hit >= 0) {
            if (tid == 0) {
                chosen[t] = (int32_t)hit;
                *ticket = 0u;  // for the next centre's launch
            }
            for (int64_t f = tid; f < d; f += kPPThreads) Ct[f * k + t] = Xt[f * n + hit];
            return;
        }
        __syncthreads();
    }

    // total of the block sums, and the running sums when their order matters
    const int64_t per = (nb + kPPThreads - 1) / kPPThreads;
    const int64_t b0 = tid * per < nb ? tid * per : nb;
    const int64_t b1 = b0 + per < nb ? b0 + per : nb;
    double own = 0.0, total;
    int key = kKeyNone;
    for (int64_t b = b0; b < b1; ++b) {
        own += __ldcg(partials + b);
        key = min(key, __ldcg(keys + b));
    }
    total = own;
    pp_block_sum(sh, total, key);
    const bool exact_blocks = key >= exponent_field(total);
    if (!exact_blocks) {
        double run = 0.0;
        for (int64_t q0 = 0; q0 < nb; q0 += kPPBlock) {
            const int count = (int)(nb - q0 < kPPBlock ? nb - q0 : kPPBlock);
            for (int q = tid; q < count; q += kPPThreads) sh.v[q] = __ldcg(partials + q0 + q);
            __syncthreads();
            if (tid == 0) run = pp_sequential(sh, run, count, true);
            __syncthreads();
            for (int q = tid; q < count; q += kPPThreads) prefix[q0 + q] = sh.v[q];
            __syncthreads();
        }
        if (tid == 0) sh.scalar = run;
        __syncthreads();
        total = sh.scalar;
        __syncthreads();
    }
    int64_t sel = -1;
    if (total > 0.0) {
        const double target = u * total;
        // first block whose running sum exceeds the target
        if (tid == 0) sh.first = (int)nb;
        __syncthreads();
        double run = 0.0, before = 0.0;
        int64_t mine = nb;
        if (exact_blocks) {
            run = pp_exclusive(sh, own);
            for (int64_t b = b0; b < b1 && mine == nb; ++b) {
                before = run;
                run += __ldcg(partials + b);
                if (run > target) mine = b;
            }
        } else {
            for (int64_t b = b0; b < b1 && mine == nb; ++b) {
                if (prefix[b] > target) {
                    mine = b;
                    before = b > 0 ? prefix[b - 1] : 0.0;
                }
            }
        }
        if (mine < nb) atomicMin(&sh.first, (int)mine);
        __syncthreads();
        if (mine < nb && sh.first == (int)mine) sh.scalar = before;
        __syncthreads();
        // no such block: rounding at the very end of the range
        const bool none = sh.first >= (int)nb;
        const int64_t b = none ? nb - 1 : sh.first;
        const double run0 = none ? total : sh.scalar;
        const int64_t i0 = b * kPPBlock;
        const int count = (int)(n - i0 < kPPBlock ? n - i0 : kPPBlock);
        // its samples, each thread kPPOwn consecutive ones
        __syncthreads();
        for (int q = tid; q < kPPBlock; q += kPPThreads) {
            sh.v[q] = q < count ? pp_value(w, min_d2, i0 + q, t) : 0.0;
        }
        if (tid == 0) {
            sh.first = kPPBlock;
            sh.last = -1;
        }
        __syncthreads();
        double part = 0.0;
        int vkey = exact_key(run0);
        for (int r = 0; r < kPPOwn; ++r) {
            const double v = sh.v[tid * kPPOwn + r];
            part += v;
            vkey = min(vkey, exact_key(v));
        }
        double all = part;
        if (tid == 0) all += run0;
        pp_block_sum(sh, all, vkey);
        if (vkey >= exponent_field(all)) {
            double x = run0 + pp_exclusive(sh, part);
            for (int r = 0; r < kPPOwn; ++r) {
                const double v = sh.v[tid * kPPOwn + r];
                x += v;
                if (v > 0.0) {
                    atomicMax(&sh.last, tid * kPPOwn + r);
                    if (x > target) atomicMin(&sh.first, tid * kPPOwn + r);
                }
            }
        } else if (tid == 0) {
            double x = run0;
            for (int q = 0; q < count; ++q) {
                const double v = sh.v[q];
                if (v > 0.0) sh.last = q;  // last positive sample if rounding overshoots
                x += v;
                if (x > target && v > 0.0) {
                    sh.first = q;
                    break;
                }
            }
        }
        __syncthreads();
        if (sh.first < kPPBlock)
            sel = i0 + sh.first;
        else if (sh.last >= 0)
            sel = i0 + sh.last;
    }
    if (sel < 0) sel = t > 0 ? ((int64_t)chosen[t - 1] + 1) % n : 0;  // every weight is zero
    if (tid == 0) {
        chosen[t] = (int32_t)sel;
        *ticket = 0u;  // for the next centre's launch
    }
    for (int64_t f = tid; f < d; f += kPPThreads) Ct[f * k + t] = Xt[f * n + sel];
}

// Population variance of each feature in float64: the mean, then the mean
// squared deviation.  A feature's samples are split over gridDim.x CTAs whose
// partial sums are added in CTA order, so the result does not depend on the
// schedule.  Bound by the float64 unit (2 operations per clock and SM); one
// CTA per feature left most SMs idle (0.33 ms at 200,003 x 32).
constexpr int kVarThreads = 256;

__device__ __forceinline__ double var_block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
        r = (threadIdx.x < kVarThreads / 32) ? sh[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;  // valid in thread 0
}

// SQUARE = 0: partial sums of the samples; 1: of the squared deviations from
// the mean that `sums` holds the partial sums of.
template <typename T, int SQUARE>
__global__ void __launch_bounds__(kVarThreads) feature_sum_kernel(const T *Xt, int64_t n,
                                                                  const double *sums, double *out) {
    __shared__ double sh[kVarThreads / 32];
    const int64_t f = blockIdx.y;
    const T *row = Xt + f * n;
    double mean = 0.0;
    if (SQUARE) {
        for (unsigned q = 0; q < gridDim.x; ++q) mean += sums[f * gridDim.x + q];
        mean /= (double)n;
    }
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)kVarThreads + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * kVarThreads) {
        const double v = (double)row[i] - mean;
        s += SQUARE ? v * v : v;
    }
    s = var_block_sum(s, sh);
    if (threadIdx.x == 0) out[f * gridDim.x + blockIdx.x] = s;
}

template <typename T>
int mean_variance(const T *Xt, int64_t n, int64_t d, double *out, cudaStream_t s) {
    KMC_CHECK_ARG(n >= 1 && d >= 1, "invalid dimensions");
    KMC_CHECK_ARG(d <= (int64_t(1) << 31) - 1, "n_features too large");
    // about four CTAs per SM over all features, at least 2048 samples each
    const int64_t parts = std::max<int64_t>(
        1, std::min<int64_t>(ceil_div<int64_t>(n, 2048), ceil_div<int64_t>(4 * num_sms(), d)));
    Scratch mem;
    KMC_TRY(mem.alloc(2 * sizeof(double) * d * parts, s));
    double *sums = mem.as<double>(), *sq = sums + d * parts;
    // the grid's y extent is limited: features in slices of 65,535
    for (int64_t f0 = 0; f0 < d; f0 += 65535) {
        const dim3 grid((unsigned)parts, (unsigned)std::min<int64_t>(d - f0, 65535));
        feature_sum_kernel<T, 0><<<grid, kVarThreads, 0, s>>>(Xt + f0 * n, n, nullptr,
                                                              sums + f0 * parts);
        KMC_TRY(check_launch("feature_mean"));
        feature_sum_kernel<T, 1><<<grid, kVarThreads, 0, s>>>(Xt + f0 * n, n, sums + f0 * parts,
                                                              sq + f0 * parts);
        KMC_TRY(check_launch("feature_variance"));
    }
    std::vector<double> h((size_t)(d * parts));
    KMC_CUDA_TRY(cudaMemcpyAsync(h.data(), sq, sizeof(double) * d * parts, cudaMemcpyDeviceToHost,
                                 s));
    KMC_CUDA_TRY(cudaStreamSynchronize(s));
    double acc = 0.0;
    for (int64_t f = 0; f < d; ++f) {
        double tot = 0.0;
        for (int64_t q = 0; q < parts; ++q) tot += h[(size_t)(f * parts + q)];
        acc += tot / (double)n;
    }
    *out = acc / (double)d;
    return KMC_OK;
}

template <typename T>
int transpose(const T *X, T *Xt, int64_t n, int64_t d, cudaStream_t s) {
    KMC_CHECK_ARG(n >= 0 && d >= 0, "array dimensions must be non-negative");
    if (n == 0 || d == 0) return KMC_OK;
    KMC_CHECK_ARG(ceil_div<int64_t>(d, 32) <= 65535, "n_features too large");
    dim3 grid((unsigned)ceil_div<int64_t>(n, 32), (unsigned)ceil_div<int64_t>(d, 32));
    transpose_kernel<T><<<grid, dim3(32, 8), 0, s>>>(X, Xt, n, d);
    return check_launch("transpose");
}

template <typename T>
int gather(const T *Xt, int64_t n, int64_t d, const int32_t *rows, int64_t k, T *Ct,
           cudaStream_t s) {
    KMC_CHECK_ARG(n >= 1 && d >= 0 && k >= 0, "invalid dimensions");
    if (d * k == 0) return KMC_OK;
    Scratch flag;
    KMC_TRY(flag.alloc(sizeof(int), s));
    KMC_CUDA_TRY(cudaMemsetAsync(flag.ptr, 0, sizeof(int), s));
    const int64_t g = std::min<int64_t>(ceil_div<int64_t>(d * k, 256), 4096);
    gather_kernel<T><<<(unsigned)g, 256, 0, s>>>(Xt, n, d, rows, k, Ct, flag.as<int>());
    KMC_TRY(check_launch("gather_rows"));
    int bad = 0;
    KMC_CUDA_TRY(cudaMemcpyAsync(&bad, flag.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    KMC_CUDA_TRY(cudaStreamSynchronize(s));
    KMC_CHECK_ARG(bad == 0, "row index out of range [0, n_samples)");
    return KMC_OK;
}

template <typename T>
int kmeanspp(const T *Xt, const T *w, int64_t n, int64_t d, int64_t k, uint64_t seed, T *Ct,
             int32_t *chosen, cudaStream_t s) {
    KMC_CHECK_ARG(n >= 1 && d >= 1 && k >= 1, "invalid dimensions");
    KMC_CHECK_ARG(k <= n, "n_clusters exceeds n_samples");
    KMC_CHECK_ARG(n < (int64_t(1) << 31), "n_samples must fit int32 indices");
    const int64_t nb = ceil_div<int64_t>(n, kPPBlock);
    Scratch mem;
    const size_t o_p = align256(sizeof(T) * n), o_f = o_p + align256(sizeof(double) * nb);
    const size_t o_k = o_f + align256(sizeof(double) * nb), o_s = o_k + align256(sizeof(int) * nb);
    const size_t o_sk = o_s + align256(sizeof(double) * nb * kPPParts);
    const size_t o_t = o_sk + align256(sizeof(int) * nb * kPPParts);
    KMC_TRY(mem.alloc(o_t + sizeof(unsigned) * (nb + 1), s));
    char *b = mem.as<char>();
    T *min_d2 = reinterpret_cast<T *>(b);
    double *partials = reinterpret_cast<double *>(b + o_p);
    double *prefix = reinterpret_cast<double *>(b + o_f);
    int *keys = reinterpret_cast<int *>(b + o_k);
    unsigned *ticket = reinterpret_cast<unsigned *>(b + o_t);
    double *parts = reinterpret_cast<double *>(b + o_s);
    int *part_keys = reinterpret_cast<int *>(b + o_sk);
    KMC_CUDA_TRY(cudaMemsetAsync(ticket, 0, sizeof(unsigned) * (nb + 1), s));
    // four CTAs fit an SM
    const unsigned grid = (unsigned)std::min<int64_t>(ceil_div<int64_t>(n, kPPPart),
                                                      4 * (int64_t)num_sms());
    for (int64_t t = 0; t < k; ++t) {
        KMC_TRY(launch_chained("kmeanspp_step", pp_step_kernel<T>, dim3(grid), dim3(kPPThreads), 0, s, Xt, w,
                               min_d2, n, d, k, (int)t, seed, partials, prefix, keys, parts, part_keys,
                               ticket + 1, chosen, Ct, ticket));
    }
    KMC_CUDA_TRY(cudaStreamSynchronize(s));
    return KMC_OK;
}

}  // namespace
}  // namespace kmc

using namespace kmc;

extern "C" {

int kmc_transpose_f32(const float *X, float *X_t, int64_t n_samples, int64_t n_features,
                      kmc_stream_t stream) {
    return transpose<float>(X, X_t, n_samples, n_features, reinterpret_cast<cudaStream_t>(stream));
}

int kmc_transpose_f64(const double *X, double *X_t, int64_t n_samples, int64_t n_features,
                      kmc_stream_t stream) {
    return transpose<double>(X, X_t, n_samples, n_features,
                             reinterpret_cast<cudaStream_t>(stream));
}

int kmc_gather_rows_f32(const float *X_t, int64_t n_samples, int64_t n_features,
                        const int32_t *rows, int64_t n_clusters, float *centroids_t,
                        kmc_stream_t stream) {
    return gather<float>(X_t, n_samples, n_features, rows, n_clusters, centroids_t,
                         reinterpret_cast<cudaStream_t>(stream));
}

int kmc_gather_rows_f64(const double *X_t, int64_t n_samples, int64_t n_features,
                        const int32_t *rows, int64_t n_clusters, double *centroids_t,
                        kmc_stream_t stream) {
    return gather<double>(X_t, n_samples, n_features, rows, n_clusters, centroids_t,
                          reinterpret_cast<cudaStream_t>(stream));
}

int kmc_mean_feature_variance_f32(const float *X_t, int64_t n_samples, int64_t n_features,
                                  double *mean_variance_out, kmc_stream_t stream) {
    KMC_CHECK_ARG(mean_variance_out != nullptr, "null output");
    return mean_variance<float>(X_t, n_samples, n_features, mean_variance_out,
                                reinterpret_cast<cudaStream_t>(stream));
}

int kmc_mean_feature_variance_f64(const double *X_t, int64_t n_samples, int64_t n_features,
                                  double *mean_variance_out, kmc_stream_t stream) {
    KMC_CHECK_ARG(mean_variance_out != nullptr, "null output");
    return mean_variance<double>(X_t, n_samples, n_features, mean_variance_out,
                                 reinterpret_cast<cudaStream_t>(stream));
}

int kmc_kmeans_plusplus_f32(const float *X_t, const float *sample_weight, int64_t n_samples,
                            int64_t n_features, int64_t n_clusters, uint64_t seed,
                            float *centroids_t, int32_t *chosen_rows, kmc_stream_t stream) {
    return kmeanspp<float>(X_t, sample_weight, n_samples, n_features, n_clusters, seed,
                           centroids_t, chosen_rows, reinterpret_cast<cudaStream_t>(stream));
}

int kmc_kmeans_plusplus_f64(const double *X_t, const double *sample_weight, int64_t n_samples,
                            int64_t n_features, int64_t n_clusters, uint64_t seed,
                            double *centroids_t, int32_t *chosen_rows, kmc_stream_t stream) {
    return kmeanspp<double>(X_t, sample_weight, n_samples, n_features, n_clusters, seed,
                            centroids_t, chosen_rows, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
