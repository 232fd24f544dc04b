// Float64 cluster sums of float64 samples whose labels are known, in a fixed
// order: a fit whose labels stop changing reproduces its centroids bit for
// bit, so a zero tolerance stops it on the same iteration as a sequential
// implementation (atomics in arbitrary order would leave last-bit noise in
// every centroid shift).
//
// Bound by float64 additions (2 per clock and SM): each sample costs d + 1, so
// they must not run on a lane or two of a warp.  A lane takes a feature (the
// weight is one more), a half-warp (up to 15 features) or a warp a sample at a
// time, and adds into its own copy of the sums in shared memory, which no
// other lane touches: no atomics, no barriers, and the samples of a copy are
// added in ascending order.  A warp's next 32 samples are copied in
// asynchronously while it adds the current ones.  The copies of a CTA are
// added in order into the CTA's copy in global memory.  An iteration of 2M x 14,
// k = 127 took 12.2 ms when the float64 tiles also added the sums, one thread
// owning each cluster; labels and sums together take 0.44 ms now (the sums 0.15;
// 0.21 with a predicated product per sample).
#include <algorithm>

#include "km_reg.cuh"

namespace kmc {

namespace {

constexpr size_t kSumsSmem = 220 * 1024;
constexpr int kSumsWarps = 12;  // at most
constexpr int kPitch = 33;      // doubles per staged feature row

__host__ __device__ constexpr size_t stage_doubles(int64_t d) { return (size_t)(d + 1) * kPitch; }
__host__ __device__ constexpr bool half_warps(int64_t d) { return d + 1 <= 16; }

// Shared memory of one warp: its copies, two staged tiles and their labels.
size_t warp_bytes(int64_t d, int64_t k) {
    const size_t units = half_warps(d) ? 2 : 1;
    return units * sizeof(double) * (size_t)((d + 1) * k) + 2 * sizeof(double) * stage_doubles(d) +
           2 * sizeof(int64_t) * 32;
}

int warps_for(int64_t d, int64_t k) {
    return (int)std::min<size_t>(kSumsWarps, kSumsSmem / warp_bytes(d, k));
}

__device__ __forceinline__ void copy_async8(void *dst, const void *src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_async4(void *dst, const void *src, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(in ? 4 : 0)
                 : "memory");
}

// A warp's staged tile into its copies.  Four samples at a time: with different
// labels their additions do not depend on one another; else in order.
template <typename I, bool HALF, bool UNIT>
__device__ __forceinline__ void add_tile(const double *st, const I *lb, double *mine, int d, int half,
                                         int f0) {
    constexpr int kStep = HALF ? 16 : 32, kMine = HALF ? 16 : 32, kAhead = 4;
    const int s0 = half * 16, ds = d + 1;
    for (int f = f0; f < ds; f += kStep) {
        const double *xf = st + f * kPitch + s0, *wf = st + d * kPitch + s0;
#pragma unroll 2
        for (int q = 0; q < kMine; q += kAhead) {
            int l[kAhead];
            double v[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                l[u] = (int)lb[s0 + q + u];
                v[u] = xf[q + u];
                if (!UNIT && f < d) v[u] = __dmul_rn(v[u], wf[q + u]);  // rounded, as the reference
            }
            const bool apart = l[0] != l[1] && l[0] != l[2] && l[0] != l[3] && l[1] != l[2] &&
                               l[1] != l[3] && l[2] != l[3];
            if (apart) {
                double sum[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) sum[u] = mine[l[u] * ds + f];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) sum[u] += v[u];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) mine[l[u] * ds + f] = sum[u];
            } else {
#pragma unroll
                for (int u = 0; u < kAhead; ++u) mine[l[u] * ds + f] += v[u];
            }
        }
    }
}

template <typename I, bool HALF>
__global__ void __launch_bounds__(32 * kSumsWarps, 1)
    sums64_kernel(const double *X, const double *w, const I *labels, double *out, double *out_sizes,
                  int64_t n, int d, int64_t k, const LoopState *guard) {
    wait_for_previous();
    if (guard != nullptr && *reinterpret_cast<const volatile int *>(&guard->done)) return;
    extern __shared__ __align__(16) double sh[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
    constexpr int kUnits = HALF ? 2 : 1;
    const int ds = d + 1;
    const int64_t copy = (int64_t)ds * k;
    const int units = warps * kUnits;
    double *stage = sh + (size_t)units * copy + (size_t)warp * 2 * stage_doubles(d);
    I *lab = reinterpret_cast<I *>(reinterpret_cast<int64_t *>(
                 sh + (size_t)units * copy + (size_t)warps * 2 * stage_doubles(d)) + warp * 64);
    for (int64_t e = tid; e < units * copy; e += blockDim.x) sh[e] = 0.0;
    __syncthreads();
    const int half = HALF ? lane >> 4 : 0;
    const int f0 = HALF ? (lane & 15) : lane;
    double *mine = sh + (size_t)(warp * kUnits + half) * copy;

    const int64_t wtiles = ceil_div<int64_t>(n, 32);
    const int64_t wstride = (int64_t)gridDim.x * warps;
    auto fetch = [&](int64_t wt, int b) {
        const int64_t i = wt * 32 + lane;
        const bool in = wt < wtiles && i < n;
        double *st = stage + (size_t)b * stage_doubles(d);
        for (int f = 0; f < d; ++f)
            copy_async8(st + f * kPitch + lane, X + (in ? (int64_t)f * n + i : 0), in);
        copy_async8(st + d * kPitch + lane, w + (in ? i : 0), in);
        if (sizeof(I) == 8)
            copy_async8(lab + 32 * b + lane, labels + (in ? i : 0), in);
        else
            copy_async4(lab + 32 * b + lane, labels + (in ? i : 0), in);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int64_t wt = (int64_t)blockIdx.x * warps + warp;
    if (wt < wtiles) fetch(wt, 0);
    for (int b = 0; wt < wtiles; wt += wstride, b ^= 1) {
        fetch(wt + wstride, b ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const double *st = stage + (size_t)b * stage_doubles(d);
        const I *lb = lab + 32 * b;
        // Samples past n were staged as zeros with label 0: they add nothing.
        // Weights of one (by their bits: a float64 compare costs as much as an
        // addition) take a loop without the product, whose instruction costs
        // its slots even where a predicate turns it off.
        if (__all_sync(0xffffffffu, __double_as_longlong(st[d * kPitch + lane]) == 0x3ff0000000000000ll))
            add_tile<I, HALF, true>(st, lb, mine, d, half, f0);
        else
            add_tile<I, HALF, false>(st, lb, mine, d, half, f0);
        __syncwarp();  // the buffer is refilled two tiles later
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    for (int64_t e = tid; e < copy; e += blockDim.x) {
        const int64_t j = e / ds, f = e - j * ds;
        double s = sh[e];
        for (int u = 1; u < units; ++u) s += sh[(size_t)u * copy + e];
        if (f < d)
            out[(int64_t)blockIdx.x * d * k + f * k + j] = s;
        else
            out_sizes[(int64_t)blockIdx.x * k + j] = s;
    }
}

}  // namespace

bool sums64_fits(int64_t d, int64_t k) {
    return d >= 1 && warps_for(d, k) >= 1;
}

int64_t sums64_copies(int64_t n, int64_t d, int64_t k) {
    return std::max<int64_t>(1, std::min<int64_t>(num_sms(), ceil_div<int64_t>(
                                                                 n, 32 * (int64_t)warps_for(d, k))));
}

template <typename I>
int launch_sums64(const double *X, const double *w, const I *labels, double *sums, double *sizes,
                  int64_t n, int64_t d, int64_t k, int64_t copies, cudaStream_t s,
                  const LoopState *guard) {
    const int warps = warps_for(d, k);
    const size_t smem = warp_bytes(d, k) * (size_t)warps;
    auto kern = half_warps(d) ? sums64_kernel<I, true> : sums64_kernel<I, false>;
    if (smem > 48 * 1024) KMC_TRY(allow_smem(kern, kSumsSmem));
    return launch_chained("sums64", kern, dim3((unsigned)copies), dim3((unsigned)(32 * warps)), smem, s, X,
                          w, labels, sums, sizes, n, (int)d, k, guard);
}

template int launch_sums64<int32_t>(const double *, const double *, const int32_t *, double *,
                                    double *, int64_t, int64_t, int64_t, int64_t, cudaStream_t,
                                    const LoopState *);
template int launch_sums64<int64_t>(const double *, const double *, const int64_t *, double *,
                                    double *, int64_t, int64_t, int64_t, int64_t, cudaStream_t,
                                    const LoopState *);

}  // namespace kmc
