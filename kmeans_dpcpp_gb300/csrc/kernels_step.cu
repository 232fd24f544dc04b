// relocate_kernel: empty clusters at the end of an iteration (km_step.cuh).
#include "km_dist.cuh"
#include "km_step.cuh"

namespace kmc {

namespace {

// Order-preserving unsigned keys (larger value -> larger key) and their digits.
// Not of NaN, whose bits are the compiler's to choose: its key could differ
// between the histograms of one selection.
__device__ __forceinline__ unsigned long long order_of(float v) {
    const unsigned b = __float_as_uint(v);
    return (b & 0x80000000u) ? (unsigned)~b : (b | 0x80000000u);
}
__device__ __forceinline__ unsigned long long order_of(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ float value_of(unsigned long long k, float) {
    const unsigned u = (unsigned)k;
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
__device__ __forceinline__ double value_of(unsigned long long k, double) {
    return __longlong_as_double(
        (long long)((k & 0x8000000000000000ull) ? (k & 0x7fffffffffffffffull) : ~k));
}

// Barrier over the (cooperatively launched) grid, number `*round` so far.  A
// wait that runs out fails the fit: every CTA then leaves.
__device__ __forceinline__ bool grid_barrier(StepCtl *ctl, unsigned *round, long long limit) {
    __shared__ int ok_sh;
    __threadfence();
    __syncthreads();
    ++*round;
    if (threadIdx.x == 0) {
        atomicAdd(&ctl->barrier, 1u);
        const unsigned want = *round * gridDim.x;
        const long long t0 = clock64();
        int ok = 1;
        while (*reinterpret_cast<volatile unsigned *>(&ctl->barrier) < want) {
            if (*reinterpret_cast<volatile int *>(&ctl->failed)) ok = 0;
            if (clock64() - t0 > limit) {
                atomicExch(&ctl->failed, 1);
                ok = 0;
            }
            if (!ok) break;
        }
        ok_sh = ok;
    }
    __syncthreads();
    const bool ok = ok_sh != 0;
    __threadfence();
    __syncthreads();
    return ok;
}

// Sample a comes before sample b: farther first, the lower index on ties.
template <typename T>
__device__ __forceinline__ bool farther(const T *dist, int64_t a, int64_t b) {
    const T va = __ldcg(dist + a), vb = __ldcg(dist + b);
    return va > vb || (va == vb && a < b);
}

// fn(distance) of samples i, i + kRelocThreads, ... below end, eight loads in
// flight (one at a time, a pass over a CTA's 16,000 samples was 32 latencies;
// the relocation of a 5M x 14 fit 237 -> 202 us).
template <typename T, typename F>
__device__ __forceinline__ void each_distance(const T *dist, int64_t i, int64_t end, F fn) {
    constexpr int kBatch = 8;
    for (; i < end; i += kBatch * kRelocThreads) {
        T v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            v[u] = dist[i + u * kRelocThreads < end ? i + u * kRelocThreads : i];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (i + u * kRelocThreads < end) fn(v[u]);
    }
}

constexpr int64_t kRankAll = 4096;  // ranked by counting all pairs; beyond, by merging

// The relocation of src/util_kernels.hpp:163-476: the r-th empty cluster (in
// ascending order) takes the r-th farthest sample (ties: the lower index); the
// threshold is found by a radix select over 8-bit digits.  Samples whose distance
// is NaN rank last and stay; where too few others are left, the last empty
// clusters get none.  Every CTA of the
// grid works on its range of samples, with a grid barrier between the phases.
// Bounded by the pass over X for the distances; the selection reads 4 bytes a
// sample and pass from L2.
template <typename T, typename I>
__device__ __noinline__ bool relocate(const RelocArgs<T, I> &a, unsigned *round) {
    __shared__ unsigned long long h[256];
    __shared__ long long wsum[2][kRelocThreads / 32];
    __shared__ unsigned long long pick[2];
    extern __shared__ float tiles[];  // row-major path: kDistTile floats per warp
    StepCtl *ctl = a.ctl;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t n = a.n, d = a.d, k = a.k;
    const int64_t n_empty = *reinterpret_cast<volatile int *>(&ctl->n_empty);
    const int64_t m = n_empty < n ? n_empty : n;
    if (m <= 0) return true;
    // this CTA's samples (a multiple of the CTA's threads each)
    const int64_t per =
        ceil_div<int64_t>(ceil_div<int64_t>(n, gridDim.x), kRelocThreads) * kRelocThreads;
    const int64_t b0 = blockIdx.x * per < n ? blockIdx.x * per : n;
    const int64_t b1 = b0 + per < n ? b0 + per : n;

    // distances to the iteration's centroids, and the first digit's histogram
    constexpr int kDigits = (int)sizeof(T);
    for (int q = tid; q < 256; q += kRelocThreads) h[q] = 0ull;
    __syncthreads();
    unsigned *h32 = reinterpret_cast<unsigned *>(h);  // counts of one CTA fit 32 bits
    for (int64_t i = b0 + tid; i < b0 + per; i += kRelocThreads) {
        const int64_t c = i < b1 ? (int64_t)a.labels[i] : -1;
        const bool ok = c >= 0 && c < k;
        T v = pos_inf<T>();
        if constexpr (sizeof(T) == 4) {
            if (a.c_rows != nullptr && d > kRowVec) {
                const float r = sq_dist_warp(a.X, a.ss, a.c_rows, a.c_stride, d, i - lane,
                                             ok ? c : -1, tiles + wid * kDistTile);
                if (ok) v = r;
            } else if (a.c_rows != nullptr) {
                if (ok) v = sq_dist_row(a.X + i * a.ss, a.c_rows + c * a.c_stride, d);
            } else if (ok) {
                v = sq_dist_cols<T>(a.X, a.fs, a.ss, a.prev, d, k, i, c);
            }
        } else if (ok) {
            v = sq_dist_cols<T>(a.X, a.fs, a.ss, a.prev, d, k, i, c);
        }
        if (!(v == v)) v = -pos_inf<T>();  // no distance
        if (i < b1) a.sq_dist[i] = v;
        // the leading digits of similar distances are the same few: lanes that
        // share the first lane's digit count once
        const unsigned digit = (unsigned)(order_of(v) >> (8 * kDigits - 8));
        const unsigned in = __ballot_sync(0xffffffffu, i < b1);
        const unsigned lead = __shfl_sync(0xffffffffu, digit, 0);
        const unsigned same = __ballot_sync(0xffffffffu, digit == lead) & in;
        if (lane == 0 && same != 0u) atomicAdd(&h32[lead], (unsigned)__popc(same));
        if (i < b1 && digit != lead) atomicAdd(&h32[digit], 1u);
    }
    unsigned long long prefix = 0ull, rank = (unsigned long long)(m - 1);
    for (int p = 0; p < kDigits; ++p) {
        const int shift = 8 * (kDigits - 1 - p);
        if (p > 0) {
            for (int q = tid; q < 256; q += kRelocThreads) h[q] = 0ull;
            __syncthreads();
            each_distance(a.sq_dist, b0 + tid, b1, [&](T v) {
                const unsigned long long key = order_of(v);
                if ((key >> (shift + 8)) == (prefix >> (shift + 8)))
                    atomicAdd(&h32[(key >> shift) & 0xffu], 1u);
            });
        }
        __syncthreads();
        for (int q = tid; q < 256; q += kRelocThreads)
            if (h32[q] != 0u) atomicAdd(&ctl->hist[p][q], (unsigned long long)h32[q]);
        if (!grid_barrier(ctl, round, a.wait_limit)) return false;
        // the digit holding the rank-th largest key (every CTA finds it itself)
        if (tid < 256) h[tid] = __ldcg(&ctl->hist[p][255 - tid]);
        __syncthreads();
        for (int o = 1; o < 256; o <<= 1) {  // inclusive sums from the largest digit down
            unsigned long long v = 0ull;
            if (tid < 256) v = h[tid] + (tid >= o ? h[tid - o] : 0ull);
            __syncthreads();
            if (tid < 256) h[tid] = v;
            __syncthreads();
        }
        if (tid < 256) {
            const unsigned long long before = tid > 0 ? h[tid - 1] : 0ull;
            if (before <= rank && h[tid] > rank) {
                pick[0] = (unsigned long long)(255 - tid);
                pick[1] = rank - before;
            }
        }
        __syncthreads();
        prefix |= pick[0] << shift;
        rank = pick[1];
        __syncthreads();
    }
    const T thr = value_of(prefix, T(0));

    // samples beyond and at the threshold, in index order
    long long ng = 0, ne = 0;
    each_distance(a.sq_dist, b0 + tid, b1, [&](T v) {
        ng += v > thr;
        ne += v == thr;
    });
    for (int o = 16; o > 0; o >>= 1) {
        ng += __shfl_down_sync(0xffffffffu, ng, o);
        ne += __shfl_down_sync(0xffffffffu, ne, o);
    }
    if (lane == 0) {
        wsum[0][wid] = ng;
        wsum[1][wid] = ne;
    }
    __syncthreads();
    if (tid == 0) {
        long long g = 0, e = 0;
        for (int q = 0; q < kRelocThreads / 32; ++q) {
            g += wsum[0][q];
            e += wsum[1][q];
        }
        ctl->counts[blockIdx.x] = g;
        ctl->counts[kMaxRelocCtas + blockIdx.x] = e;
        pick[0] = (unsigned long long)(g + e);
    }
    if (!grid_barrier(ctl, round, a.wait_limit)) return false;
    const bool any = pick[0] != 0ull;  // of this CTA's samples
    // samples of the CTAs before this one, and of all CTAs
    long long pg = 0, pe = 0, tg = 0, te = 0;
    for (int b = tid; b < (int)gridDim.x; b += kRelocThreads) {
        const long long g = __ldcg(&ctl->counts[b]), e = __ldcg(&ctl->counts[kMaxRelocCtas + b]);
        tg += g;
        te += e;
        if (b < (int)blockIdx.x) {
            pg += g;
            pe += e;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        pg += __shfl_down_sync(0xffffffffu, pg, o);
        pe += __shfl_down_sync(0xffffffffu, pe, o);
        tg += __shfl_down_sync(0xffffffffu, tg, o);
        te += __shfl_down_sync(0xffffffffu, te, o);
    }
    if (lane == 0) {
        wsum[0][wid] = pg;
        wsum[1][wid] = pe;
        h[wid] = (unsigned long long)tg;
        h[kRelocThreads / 32 + wid] = (unsigned long long)te;
    }
    __syncthreads();
    pg = pe = tg = te = 0;
    for (int q = 0; q < kRelocThreads / 32; ++q) {
        pg += wsum[0][q];
        pe += wsum[1][q];
        tg += (long long)h[q];
        te += (long long)h[kRelocThreads / 32 + q];
    }
    // at the threshold (fewer than m lie beyond it; none when only samples
    // without a distance are left)
    const long long need = thr == -pos_inf<T>() ? 0 : (m - tg < te ? m - tg : te);
    __syncthreads();
    for (int64_t i0 = b0; any && i0 < b1; i0 += kRelocThreads) {
        const int64_t i = i0 + tid;
        const T v = i < b1 ? a.sq_dist[i] : T(0);
        const bool g = i < b1 && v > thr, e = i < b1 && v == thr;
        const unsigned mg = __ballot_sync(0xffffffffu, g), me = __ballot_sync(0xffffffffu, e);
        if (lane == 0) {
            wsum[0][wid] = __popc(mg);
            wsum[1][wid] = __popc(me);
        }
        __syncthreads();
        long long og = pg, oe = pe;
        for (int q = 0; q < kRelocThreads / 32; ++q) {
            if (q < wid) {
                og += wsum[0][q];
                oe += wsum[1][q];
            }
            pg += wsum[0][q];
            pe += wsum[1][q];
        }
        const unsigned lm = (1u << lane) - 1u;
        og += __popc(mg & lm);
        oe += __popc(me & lm);
        if (g && og < k) a.gt_list[og] = i;
        if (e && oe < need && tg + oe < k) a.far[tg + oe] = i;
        __syncthreads();
    }
    if (!grid_barrier(ctl, round, a.wait_limit)) return false;

    // rank of the samples beyond the threshold
    const int64_t total = tg < k ? tg : k;
    const int64_t gid = blockIdx.x * (int64_t)kRelocThreads + tid;
    const int64_t gstride = (int64_t)gridDim.x * kRelocThreads;
    if (total <= kRankAll) {
        // a warp per entry, its lanes over the others (a thread per entry waited
        // for each of them in turn: 2 ms for 3000)
        const int64_t warps = (int64_t)gridDim.x * (kRelocThreads / 32);
        for (int64_t e = (int64_t)wid * gridDim.x + blockIdx.x; e < total; e += warps) {
            const int64_t ie = __ldcg(a.gt_list + e);
            int r = 0;
#pragma unroll 4
            for (int64_t q = lane; q < total; q += 32) {
                const int64_t iq = __ldcg(a.gt_list + q);
                r += iq != ie && farther(a.sq_dist, iq, ie);
            }
            r = __reduce_add_sync(0xffffffffu, r);
            if (lane == 0) a.far[r] = ie;
        }
    } else {
        // merge sort: an entry's place is its place in its own run plus the
        // partner run's entries before it
        const int64_t *src = a.gt_list;
        int64_t *dst = a.gt_tmp;
        for (int64_t len = 1; len < total; len <<= 1) {
            const bool last = 2 * len >= total;
            if (last) dst = a.far;
            for (int64_t e = gid; e < total; e += gstride) {
                const int64_t base = (e / (2 * len)) * (2 * len);
                const int64_t mid = base + len < total ? base + len : total;
                const int64_t end = mid + len < total ? mid + len : total;
                const int64_t v = __ldcg(src + e);
                const int64_t o0 = e < mid ? mid : base, o1 = e < mid ? end : mid;
                int64_t lo = o0, hi = o1;
                while (lo < hi) {
                    const int64_t c = (lo + hi) >> 1;
                    if (farther(a.sq_dist, __ldcg(src + c), v)) lo = c + 1;
                    else hi = c;
                }
                dst[(e < mid ? e : base + (e - mid)) + (lo - o0)] = v;
            }
            if (!last && !grid_barrier(ctl, round, a.wait_limit)) return false;
            int64_t *t = const_cast<int64_t *>(src);
            src = dst;
            dst = t;
        }
    }
    if (!grid_barrier(ctl, round, a.wait_limit)) return false;

    // move the samples, one thread per feature (one more for the sizes), empty
    // clusters in order; the loads of eight moves in flight
    constexpr int kMoves = 8;
    const int64_t moves = m < tg + need ? m : tg + need;
    for (int64_t f = gid; f <= d; f += gstride) {
        T *const row = f < d ? a.sums + f * k : a.sizes;
        for (int64_t r0 = 0; r0 < moves; r0 += kMoves) {
            int64_t s[kMoves], from[kMoves], to[kMoves];
            T xw[kMoves], left[kMoves];
#pragma unroll
            for (int u = 0; u < kMoves; ++u) {
                const int64_t r = r0 + u < moves ? r0 + u : r0;
                s[u] = __ldcg(a.far + r);
                to[u] = __ldcg(a.empty_list + r);
                if (r0 + u >= moves || s[u] < 0 || s[u] >= n) s[u] = -1;
            }
#pragma unroll
            for (int u = 0; u < kMoves; ++u) {
                const int64_t i = s[u] < 0 ? 0 : s[u];
                from[u] = (int64_t)a.labels[i];
                if (s[u] < 0 || from[u] < 0 || from[u] >= k || to[u] < 0 || to[u] >= k)
                    from[u] = to[u] = -1;
                xw[u] = a.w[i];
                if (f < d) xw[u] = mul_rn(a.X[f * a.fs + i * a.ss], xw[u]);  // rounded, as the reference
            }
#pragma unroll
            for (int u = 0; u < kMoves; ++u) left[u] = row[from[u] < 0 ? 0 : from[u]];
#pragma unroll
            for (int u = 0; u < kMoves; ++u) {
                // what the moves before it, loaded with it, made of that sum
#pragma unroll
                for (int v = 0; v < u; ++v) {
                    if (from[v] == from[u]) left[u] = left[v];
                    if (to[v] == from[u]) left[u] = xw[v];
                }
                left[u] -= xw[u];
                if (from[u] < 0) continue;
                row[from[u]] = left[u];
                row[to[u]] = xw[u];
            }
        }
    }
    return grid_barrier(ctl, round, a.wait_limit);
}

template <typename T, typename I>
__global__ void __launch_bounds__(kRelocThreads, 2) relocate_kernel(RelocArgs<T, I> a) {
    if (*reinterpret_cast<volatile int *>(&a.state->done) != kPaused) return;
    __shared__ double sh[32];
    StepCtl *ctl = a.ctl;
    unsigned round = 0;
    if (relocate<T, I>(a, &round)) {
        // 32 clusters to a warp, the warps of all CTAs in turn: the divisions,
        // float64 ones above all, want every SM
        constexpr int kBatch = 4;
        const int64_t warps = (int64_t)gridDim.x * (kRelocThreads / 32);
        for (int64_t g = (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; g * 32 < a.k; g += warps) {
            const int64_t j = g * 32 + (threadIdx.x & 31);
            if (j >= a.k) continue;
            const T size = __ldcg(a.sizes + j);
            T shift = T(0);
            for (int64_t f0 = 0; f0 < a.d; f0 += kBatch) {
                T sum[kBatch], old[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const int64_t at = (f0 + u < a.d ? f0 + u : f0) * a.k + j;
                    sum[u] = __ldcg(a.sums + at);
                    old[u] = a.prev[at];
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    if (f0 + u >= a.d) break;
                    const int64_t at = (f0 + u) * a.k + j;
                    const T c = sum[u] / size, diff = old[u] - c;
                    a.nxt[at] = c;
                    a.cur[at] = c;
                    shift = fma_rn(diff, diff, shift);
                }
            }
            a.shifts[j] = shift;
        }
    }
    // every CTA has read `done` before the last one resumes the loop
    if (!last_cta(&ctl->reloc_ticket)) return;
    if (*reinterpret_cast<volatile int *>(&ctl->failed)) {
        if (threadIdx.x == 0) {
            atomicOr(&a.state->err, 1u);
            atomicExch(&a.state->done, 1);
        }
    } else {
        stop_rule<T>(a.shifts, a.k, a.state, sh);
    }
    for (int q = threadIdx.x; q < 8 * 256; q += kRelocThreads) ctl->hist[q / 256][q % 256] = 0ull;
    if (threadIdx.x == 0) {
        ctl->n_empty = 0;
        ctl->barrier = 0u;
        ctl->reloc_ticket = 0u;
    }
}

}  // namespace

template <typename T, typename I>
int launch_relocation(const RelocArgs<T, I> &a, cudaStream_t s) {
    // enough CTAs for the distances, and for the divisions; two per SM are resident
    // together (a cooperative launch)
    const int64_t want = std::max(ceil_div<int64_t>(a.n, 4 * kRelocThreads),
                                  std::min(ceil_div<int64_t>(a.k, 32), a.d * a.k / 4096));
    const int64_t most = std::min<int64_t>(2 * (int64_t)num_sms(), kMaxRelocCtas);
    const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, most));
    const size_t smem = sizeof(T) == 4 && a.c_rows != nullptr && a.d > kRowVec
                            ? sizeof(float) * kDistTile * (kRelocThreads / 32)
                            : 0;
    auto kern = relocate_kernel<T, I>;
    if (smem > 0) KMC_TRY(allow_smem(kern, smem));
    RelocArgs<T, I> args = a;
    void *params[] = {&args};
    KMC_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kern), dim3(grid),
                                             dim3(kRelocThreads), params, smem, s));
    return KMC_OK;
}

template int launch_relocation<float, int32_t>(const RelocArgs<float, int32_t> &, cudaStream_t);
template int launch_relocation<float, int64_t>(const RelocArgs<float, int64_t> &, cudaStream_t);
template int launch_relocation<double, int32_t>(const RelocArgs<double, int32_t> &, cudaStream_t);
template int launch_relocation<double, int64_t>(const RelocArgs<double, int64_t> &, cudaStream_t);

}  // namespace kmc
