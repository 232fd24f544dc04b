// The end of a Lloyd iteration: cluster sums -> next centroids, shifts, stop
// rule (reduce_sums_kernel, finish_kernel), and the relocation of empty
// clusters (relocate_kernel, kernels_step.cu).
//
// An iteration used to end in about 20 launches (copy reduction, empty list,
// gate, 15 relocation kernels that mostly returned at once, division, stop
// rule, copy), 2 to 3 us each: a 50,000-sample fit spent 100 of its 150 us per
// iteration there.  Now finish_kernel assumes that no cluster is empty and
// does everything, keeping the sums and the previous centroids; its last CTA
// either applies the stop rule or, when clusters are empty, lists them and
// pauses the loop, and the relocation (one cooperative launch) redoes the
// division from the kept sums and resumes it.  The driver and the request
// server launch the relocation when they find the loop paused; kmc_fit_step,
// which never waits for the device, enqueues it with every iteration.
//
// Semantics: reduction of the private copies and the empty-cluster list
// (src/util_kernels.hpp:87-161, ascending order), division and shifts
// (util_kernels.hpp:9-41, 481-516; kmeans_lloyd_driver.hpp:317-341), stop rule
// (kmeans_lloyd_driver.hpp:83, 343-353), relocation (util_kernels.hpp:163-476).
#pragma once

#include <algorithm>

#include "km_kernels.cuh"

namespace kmc {

// Control block of a fit's iterations (device memory, zero between kernels).
struct StepCtl {
    unsigned finish_ticket;  // CTAs of finish_kernel that are through
    unsigned reloc_ticket;
    int n_empty;             // empty clusters of this iteration (the loop is paused: > 0)
    unsigned barrier;        // arrivals at relocate_kernel's grid barriers
    int failed;              // a grid barrier gave up its wait
    long long counts[2 * 512];            // relocation: greater / equal samples per CTA
    unsigned long long hist[8][256];      // radix-select histograms
};

constexpr int kFinishThreads = 256;
constexpr int kFinishOwn = 4;  // elements of a round per thread
constexpr int kFinishElems = kFinishThreads * kFinishOwn;
constexpr int kRelocThreads = 512;
constexpr int kMaxRelocCtas = 512;
// LoopState::done of a loop that waits for relocate_kernel
constexpr int kPaused = 2;

template <typename T>
struct FinishArgs {
    T *cur;             // (d, k) current centroids, overwritten
    T *nxt;             // (d, k) result buffer
    T *prev;            // (d, k) the centroids before, and the
    T *sums;            // (d, k) cluster sums, kept for a relocation
    T *sizes;           // (k)
    T *shifts;          // (k)
    T *hn;              // (k) half norms of the new centroids, or null
    int64_t *empty_list;  // (k), ascending
    int64_t d, k;
    int jc;             // clusters per CTA
    LoopState *state;
    StepCtl *ctl;
};

// Sums as float64 private copies in (d, k) order.
struct PlainSums {
    double *sums, *sizes;  // [copies][d*k], [copies][k]
    int64_t dk, k, copies;
    struct Part {
        double v;
    };
    // feature f (d: the sizes) and cluster j of element e
    __device__ __forceinline__ void at(int64_t e, int64_t d, int64_t *f, int64_t *j) const {
        *f = e / k;
        *j = e - *f * k;
    }
    static __device__ __forceinline__ Part zero() { return Part{0.0}; }
    static __device__ __forceinline__ void add(Part &a, const Part &b) { a.v += b.v; }
    __device__ __forceinline__ double value(const Part &p) const { return p.v; }
    // Copies g, g + groups, ... in order, zeroed once read; eight loads in flight.
    __device__ __forceinline__ Part load(int64_t f, int64_t j, int64_t d, int g, int groups) const {
        double *p = f < d ? sums + f * k + j : sizes + j;
        const int64_t stride = f < d ? dk : k;
        double acc = 0.0;
        for (int64_t c = g; c < copies; c += 8 * groups) {
            double v[8];
            // unconditional (the first again in the place of those past the last
            // copy): a load behind a condition waits for the one before it
#pragma unroll
            for (int u = 0; u < 8; ++u)
                v[u] = load_in_order(p + (c + u * groups < copies ? c + u * groups : c) * stride);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (c + u * groups < copies) p[(c + u * groups) * stride] = 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (c + u * groups < copies) acc += v[u];
        }
        return Part{acc};
    }
};

// Sums already reduced (by reduce_sums_kernel).
template <typename T>
struct ReducedSums {
    T *sums, *sizes;
    int64_t k;
    struct Part {
        T v;
    };
    __device__ __forceinline__ T value(const Part &p) const { return p.v; }
    __device__ __forceinline__ Part load(int64_t f, int64_t j, int64_t d, int, int) const {
        return Part{f < d ? sums[f * k + j] : sizes[j]};
    }
};

// Private copies -> sums and sizes.  G threads share an element's copies (g, g +
// G, ..., then the G partial sums in order: a fixed order, so float64 fits stay
// reproducible); a CTA takes kReduceThreads / G consecutive elements.  One
// thread per element walked 304 copies as a chain of memory latencies: 46 us
// for 240 elements, 5 us with 16.  Up to kFewCopies copies four threads do, and
// the grid is a quarter (4 copies of 132,096 elements: 39 -> 23 us).
constexpr int kReduceLanes = 32, kReduceGroups = 16;
constexpr int kReduceThreads = kReduceLanes * kReduceGroups, kFewCopies = 8;

template <typename T, typename Src, int G>
__global__ void __launch_bounds__(kReduceThreads)
    reduce_sums_kernel(Src src, T *sums, T *sizes, int64_t d, int64_t k, const LoopState *state) {
    wait_for_previous();
    allow_next();
    if (*reinterpret_cast<const volatile int *>(&state->done)) return;
    constexpr int kLanes = kReduceThreads / G;
    __shared__ typename Src::Part red[G][kLanes];
    const int el = threadIdx.x % kLanes, g = threadIdx.x / kLanes;
    const int64_t e = blockIdx.x * (int64_t)kLanes + el;
    int64_t f = 0, j = 0;
    typename Src::Part p = Src::zero();
    if (e < (d + 1) * k) {
        src.at(e, d, &f, &j);
        p = src.load(f, j, d, g, G);
    }
    red[g][el] = p;
    __syncthreads();
    if constexpr (G > 4) {
        if (g < 4) {
            p = red[G / 4 * g][el];
#pragma unroll
            for (int q = 1; q < G / 4; ++q) Src::add(p, red[G / 4 * g + q][el]);
        }
        __syncthreads();
        if (g < 4) red[g][el] = p;
        __syncthreads();
    }
    if (g == 0 && e < (d + 1) * k) {
#pragma unroll
        for (int q = 1; q < 4; ++q) Src::add(p, red[q][el]);
        if (f < d)
            sums[f * k + j] = (T)src.value(p);
        else
            sizes[j] = (T)src.value(p);
    }
}

// Total shift and stop rule (kmeans_lloyd_driver.hpp:83, 343-353) by one CTA.
// sh: 32 doubles.
template <typename T>
__device__ __forceinline__ void stop_rule(const T *shifts, int64_t k, LoopState *st, double *sh) {
    double acc = 0.0;
    for (int64_t j = threadIdx.x; j < k; j += blockDim.x) acc += (double)__ldcg(shifts + j);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = acc;
    __syncthreads();
    if (wid == 0) {
        double r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
        if (lane == 0) {
            st->last_shift = r;
            st->n_iter += 1;
            const T shift_t = (T)r;
            const T tol_t = (T)st->tol;
            st->done = (st->n_iter < st->max_iter) && (shift_t > tol_t) ? 0 : 1;
        }
    }
}

// True in every thread of the CTA that finishes last (its reads of the other
// CTAs' results bypass L1).
__device__ __forceinline__ bool last_cta(unsigned *ticket) {
    __shared__ int last_sh;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_sh = atomicAdd(ticket, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (last_sh) __threadfence();
    return last_sh != 0;
}

// Division, each cluster's shift (features in order, as the reference adds
// them), the plain forms' half norms for the next iteration (a launch of their
// own before: 50,000 x 14, k = 16, 20 iterations 707 -> 629 us) and, in the last CTA, the stop rule or the empty-cluster list.  A CTA
// takes jc clusters.  Latency-bound: all loads of a round are issued together
// (sums, previous centroids, sizes), and the CTAs meet once, at the ticket.
template <typename T, typename Src>
__global__ void __launch_bounds__(kFinishThreads) finish_kernel(Src src, FinishArgs<T> a) {
    wait_for_previous();
    allow_next();
    if (*reinterpret_cast<const volatile int *>(&a.state->done)) return;
    __shared__ T diff_sh[kFinishElems], new_sh[kFinishElems];
    __shared__ T size_sh[32];
    __shared__ double sh[32];
    __shared__ int warp_counts[kFinishThreads / 32];
    const int tid = threadIdx.x;
    const int64_t d = a.d, k = a.k, j0 = (int64_t)blockIdx.x * a.jc;
    const int jn = (int)(k - j0 < a.jc ? k - j0 : a.jc);
    const int64_t fc = kFinishElems / a.jc;  // features per round
    T shift = T(0), norm = T(0);
    for (int64_t f0 = 0; f0 == 0 || f0 < d; f0 += fc) {
        const int nf = (int)(d - f0 < fc ? d - f0 : fc), cnt = nf * jn;
        T s[kFinishOwn], old[kFinishOwn];
#pragma unroll
        for (int u = 0; u < kFinishOwn; ++u) {
            const int e = tid + u * kFinishThreads;
            s[u] = old[u] = T(0);
            if (e < cnt) {
                const int f = e / jn, j = e - f * jn;
                s[u] = (T)src.value(src.load(f0 + f, j0 + j, d, 0, 1));
                old[u] = a.cur[(f0 + f) * k + j0 + j];
            }
        }
        if (f0 == 0 && tid < jn) {
            const T v = (T)src.value(src.load(d, j0 + tid, d, 0, 1));
            size_sh[tid] = v;
            a.sizes[j0 + tid] = v;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kFinishOwn; ++u) {
            const int e = tid + u * kFinishThreads;
            if (e < cnt) {
                const int f = e / jn, j = e - f * jn;
                const int64_t at = (f0 + f) * k + j0 + j;
                const T c = s[u] / size_sh[j];
                a.sums[at] = s[u];
                a.prev[at] = old[u];
                a.cur[at] = c;
                a.nxt[at] = c;
                diff_sh[e] = old[u] - c;
                new_sh[e] = c;
            }
        }
        __syncthreads();
        if (tid < jn) {
#pragma unroll 4
            for (int f = 0; f < nf; ++f) {
                const T diff = diff_sh[f * jn + tid];
                shift = fma_rn(diff, diff, shift);
            }
        } else if (tid >= 32 && tid < 32 + jn) {
            // the next iteration's half norms, by another warp
#pragma unroll 4
            for (int f = 0; f < nf; ++f) {
                const T c = new_sh[f * jn + tid - 32];
                norm = fma_rn(c, c, norm);
            }
        }
        __syncthreads();
    }
    if (a.hn != nullptr && tid >= 32 && tid < 32 + jn) a.hn[j0 + tid - 32] = norm / T(2);
    if (tid < 32) {
        const bool empty = tid < jn && size_sh[tid] == T(0);
        if (tid < jn) a.shifts[j0 + tid] = shift;
        const unsigned m = __ballot_sync(0xffffffffu, empty);
        if (tid == 0 && m != 0u) atomicAdd(&a.ctl->n_empty, __popc(m));
    }
    if (!last_cta(&a.ctl->finish_ticket)) return;
    const int n_empty = *reinterpret_cast<volatile int *>(&a.ctl->n_empty);
    if (n_empty == 0) {
        stop_rule<T>(a.shifts, k, a.state, sh);
    } else {
        // ascending list of the empty clusters
        const int lane = tid & 31, wid = tid >> 5;
        int64_t base = 0;
        for (int64_t c0 = 0; c0 < k; c0 += kFinishThreads) {
            const int64_t j = c0 + tid;
            const bool empty = j < k && __ldcg(a.sizes + j) == T(0);
            const unsigned m = __ballot_sync(0xffffffffu, empty);
            if (lane == 0) warp_counts[wid] = __popc(m);
            __syncthreads();
            int before = 0, total = 0;
            for (int q = 0; q < kFinishThreads / 32; ++q) {
                if (q < wid) before += warp_counts[q];
                total += warp_counts[q];
            }
            if (empty) a.empty_list[base + before + __popc(m & ((1u << lane) - 1u))] = j;
            base += total;
            __syncthreads();
        }
        if (tid == 0) a.state->done = kPaused;
    }
    if (tid == 0) a.ctl->finish_ticket = 0u;
}

// Few clusters per CTA, so that the CTAs' latencies run side by side: one up
// to 128 clusters, 8 at 1024, at most 32.
template <typename T, typename Src>
int launch_finish(const Src &src, FinishArgs<T> a, cudaStream_t s) {
    a.jc = (int)std::min<int64_t>(32, ceil_div<int64_t>(a.k, 128));
    return launch_chained("finish", finish_kernel<T, Src>, dim3((unsigned)ceil_div<int64_t>(a.k, a.jc)),
                          dim3(kFinishThreads), 0, s, src, a);
}

// Up to this many private copies finish_kernel reads them itself.
constexpr int64_t kDirectCopies = 2;

// Reduction (where there are several copies) and finish; *n_launches kernels.
template <typename T, typename Src>
int launch_reduce_and_finish(const Src &src, int64_t copies, const FinishArgs<T> &a,
                             int64_t *n_launches, cudaStream_t s) {
    *n_launches = 1;
    if (copies <= kDirectCopies) return launch_finish<T>(src, a, s);
    *n_launches = 2;
    const bool few = copies <= kFewCopies;
    const int64_t grid = ceil_div<int64_t>((a.d + 1) * a.k, kReduceThreads / (few ? 4 : kReduceGroups));
    auto kern = few ? reduce_sums_kernel<T, Src, 4> : reduce_sums_kernel<T, Src, kReduceGroups>;
    KMC_TRY(launch_chained("reduce_sums", kern, dim3((unsigned)grid), dim3(kReduceThreads), 0, s, src,
                           a.sums, a.sizes, a.d, a.k, (const LoopState *)a.state));
    return launch_finish<T>(ReducedSums<T>{a.sums, a.sizes, a.k}, a, s);
}

// Relocation of the empty clusters of a paused loop, then division, stop rule
// and the resumption of the loop.  Returns at once when the loop is not paused.
template <typename T, typename I>
struct RelocArgs {
    T *cur, *nxt, *prev, *sums, *sizes, *shifts;
    const int64_t *empty_list;
    int64_t *far, *gt_list, *gt_tmp;  // (k) each: samples, farthest first; scratch
    const T *X, *w;
    const I *labels;
    T *sq_dist;  // (n)
    int64_t n, d, k, fs, ss;  // X element (f, i) at X[f * fs + i * ss]
    const T *c_rows;          // row-major copy of prev ([k][c_stride]), or null
    int64_t c_stride;
    long long wait_limit;
    LoopState *state;
    StepCtl *ctl;
};

template <typename T, typename I>
int launch_relocation(const RelocArgs<T, I> &a, cudaStream_t s);

}  // namespace kmc
