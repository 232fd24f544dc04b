// Kernels of the batched Lloyd engine (km_batch.cuh), the device-side
// synthetic-data generator used by the serving loop, and the tile autotuner.
//
// Per engine step (every active instance advances one Lloyd iteration):
//   batch_prep    half norms of the centroids (src/util_kernels.hpp:47-82
//                 order), reset work-queue counters
//   batch_panel   persistent CTAs pop (instance, run of 128-sample tiles)
//                 items from a device work queue and walk them in panels of 32
//                 samples per warp (km_panel.cuh).  Each (sample, centroid)
//                 pair gets the plain form's arithmetic -- sequential FMA dot
//                 over f = 0..d-1, D = hn - dot, strict < over ascending j
//                 (src/device_functions.hpp:106-162) -- so labels equal a
//                 single fit's bit for bit.  Fitting instances add w*x into
//                 float64 copies of the sums.  Three variants differ in the
//                 centroids per thread (16, 32 or 64 columns per step); the
//                 autotuner picks one per (d, k)
//   batch_assign  the same for instances of more features than a panel takes,
//                 in 128-sample tiles (centroid windows of 32, 64 or 128)
//   batch_reduce  sums rounded once to float32, sizes, ascending empty-cluster
//                 list (src/util_kernels.hpp:87-161), the copies zeroed again
//   batch_update  divide, per-cluster shifts, float64 total, the driver's stop
//                 rule (src/kmeans_lloyd_driver.hpp:317-353), copy-back
//                 (several CTAs per fitting instance in both)
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <map>
#include <tuple>
#include <mutex>
#include <sstream>
#include <string>
#include <sys/stat.h>

#include "km_batch.cuh"
#include "km_panel_kernel.cuh"
#include "km_step.cuh"

namespace kmc {

namespace {

constexpr int kThreadsB = 256;
constexpr int kBK = 16;
constexpr int kTM = 8;
constexpr size_t kPrivBytes = 72 * 1024;  // with the tiles: two CTAs per SM
constexpr int kSumCopies = 48;            // global copies of small instances' sums
constexpr int kFewSumCopies = 8;          // and of larger ones'

constexpr int kPrepThreads = 128;

// Half norms, a thread per cluster (gridDim.x CTAs per instance).
__global__ void __launch_bounds__(kPrepThreads)
    batch_prep_kernel(BInst *tab, const int *idx, int count, int *counters) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < kBatchCounters)
        counters[threadIdx.x] = 0;
    if ((int)blockIdx.y >= count) return;
    BInst &in = tab[idx[blockIdx.y]];
    const int d = in.d, k = in.k, j = blockIdx.x * kPrepThreads + threadIdx.x;
    if (j >= k) return;
    const float *C = in.C + j;
    float acc = 0.f;
    int f = 0;
    for (; f + 8 <= d; f += 8) {
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = C[(int64_t)(f + u) * k];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = __fmaf_rn(v[u], v[u], acc);
    }
    for (; f < d; ++f) {
        const float v = C[(int64_t)f * k];
        acc = __fmaf_rn(v, v, acc);
    }
    in.hn[j] = acc / 2.f;
}

template <int HN>
__device__ __forceinline__ void vld(const float *p, float *o) {
    if constexpr (HN == 1) {
        o[0] = p[0];
    } else if constexpr (HN == 2) {
        const float2 v = *reinterpret_cast<const float2 *>(p);
        o[0] = v.x;
        o[1] = v.y;
    } else {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        o[0] = v.x;
        o[1] = v.y;
        o[2] = v.z;
        o[3] = v.w;
    }
}

template <int TN>
struct BTile {
    static constexpr int BM = 16 * kTM, BN = 16 * TN, HM = kTM / 2, HN = TN / 2;
    static constexpr int XR = kBK * BM / kThreadsB, CR = kBK * BN / kThreadsB;
    static constexpr size_t base_bytes =
        sizeof(float) * (2 * kBK * BM + 2 * kBK * BN + BN + BM) + sizeof(long long) * BM;
};

// DIST = 1: the items are B_TRANSFORM instances, whose (k, n) Euclidean
// distances sqrt(sum_f (c - x)^2) are written instead of labels (the plain
// form's MODE_DIST arithmetic, compute_euclidean_distance.hpp:12-114).
template <int TN, int DIST>
__global__ void __launch_bounds__(kThreadsB, 2)
    batch_assign_kernel(const BInst *tab, const BItem *items, int n_items, int *counter) {
    using G = BTile<TN>;
    constexpr int BM = G::BM, BN = G::BN, HM = G::HM, HN = G::HN, XR = G::XR, CR = G::CR;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float *Xs = reinterpret_cast<float *>(smem_raw);
    float *Cs = Xs + 2 * kBK * BM;
    float *hs = Cs + 2 * kBK * BN;
    float *ws = hs + BN;
    long long *labs = reinterpret_cast<long long *>(ws + BM);
    double *psums = reinterpret_cast<double *>(labs + BM);
    __shared__ int item_sh;

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    while (true) {
        if (tid == 0) item_sh = atomicAdd(counter, 1);
        __syncthreads();
        const int it = item_sh;
        __syncthreads();
        if (it >= n_items) break;
        const BItem item = items[it];
        const BInst &in = tab[item.inst];
        const float *X = in.X, *C = in.C, *hn = in.hn, *w = in.w;
        int32_t *labels = in.labels;
        const int64_t n = in.n;
        const int d = in.d, k = in.k;
        const bool fit = in.mode == B_FIT;
        const int64_t dk = (int64_t)d * k;
        const bool priv = fit && in.copies == 1 && (size_t)(dk + k) * sizeof(double) <= kPrivBytes;
        double *tsums = priv ? psums : in.sums + (int64_t)(blockIdx.x % (unsigned)in.copies) * (dk + k);
        double *tsizes = tsums + dk;
        if (priv) {
            for (int64_t e = tid; e < dk + k; e += kThreadsB) psums[e] = 0.0;
            __syncthreads();
        }
        const int nchunks = (d + kBK - 1) / kBK;
        const int64_t tile_end = item.tile0 + item.ntiles;
        // Feature chunk ch of samples li0.. and centroids lc0.. into registers;
        // chunk 0 of the item's next (tile, centroid window) step is loaded
        // while the current step's last chunk is multiplied (the widest
        // window has no registers to spare for it: it loads at the step).
        constexpr bool kAhead = TN <= 4;
        float xr[XR], cr[CR];
        auto load_regs = [&](int64_t li0, int lc0, int ch) {
            const int f0 = ch * kBK;
#pragma unroll
            for (int r = 0; r < XR; ++r) {
                const int e = tid + r * kThreadsB;
                const int kk = e / BM, s = e % BM;
                const int f = f0 + kk;
                const int64_t i = li0 + s;
                xr[r] = (f < d && i < n) ? X[(int64_t)f * n + i] : 0.f;
            }
#pragma unroll
            for (int r = 0; r < CR; ++r) {
                const int e = tid + r * kThreadsB;
                const int kk = e / BN, c = e % BN;
                const int f = f0 + kk, j = lc0 + c;
                cr[r] = (f < d && j < k) ? C[(int64_t)f * k + j] : 0.f;
            }
        };
        auto store_smem = [&](int buf) {
#pragma unroll
            for (int r = 0; r < XR; ++r) Xs[buf * kBK * BM + tid + r * kThreadsB] = xr[r];
#pragma unroll
            for (int r = 0; r < CR; ++r) Cs[buf * kBK * BN + tid + r * kThreadsB] = cr[r];
        };
        if (kAhead) load_regs(item.tile0 * BM, 0, 0);

        for (int64_t tile = item.tile0; tile < tile_end; ++tile) {
            const int64_t i0 = tile * BM;
            float best[kTM];
            int bidx[kTM];
#pragma unroll
            for (int m = 0; m < kTM; ++m) {
                best[m] = pos_inf<float>();
                bidx[m] = 0;
            }
            for (int c0 = 0; c0 < k; c0 += BN) {
                float acc[kTM][TN];
#pragma unroll
                for (int m = 0; m < kTM; ++m)
#pragma unroll
                    for (int q = 0; q < TN; ++q) acc[m][q] = 0.f;
                for (int c = tid; c < BN; c += kThreadsB)
                    hs[c] = (c0 + c < k) ? hn[c0 + c] : pos_inf<float>();

                if (!kAhead) load_regs(i0, c0, 0);
                store_smem(0);  // chunk 0 (loaded during the previous step when kAhead)
                __syncthreads();
                for (int ch = 0; ch < nchunks; ++ch) {
                    const int buf = ch & 1;
                    if (ch + 1 < nchunks)
                        load_regs(i0, c0, ch + 1);
                    else if (kAhead && c0 + BN < k)
                        load_regs(i0, c0 + BN, 0);
                    else if (kAhead && tile + 1 < tile_end)
                        load_regs(i0 + BM, 0, 0);
                    const float *xb = Xs + buf * kBK * BM;
                    const float *cb = Cs + buf * kBK * BN;
#pragma unroll
                    for (int kk = 0; kk < kBK; ++kk) {
                        float xv[kTM], cv[TN];
                        vld<HM>(xb + kk * BM + ty * HM, xv);
                        vld<HM>(xb + kk * BM + BM / 2 + ty * HM, xv + HM);
                        vld<HN>(cb + kk * BN + tx * HN, cv);
                        vld<HN>(cb + kk * BN + BN / 2 + tx * HN, cv + HN);
#pragma unroll
                        for (int m = 0; m < kTM; ++m)
#pragma unroll
                            for (int q = 0; q < TN; ++q) {
                                if (DIST) {
                                    const float diff = cv[q] - xv[m];
                                    acc[m][q] = __fmaf_rn(diff, diff, acc[m][q]);
                                } else {
                                    acc[m][q] = __fmaf_rn(xv[m], cv[q], acc[m][q]);
                                }
                            }
                    }
                    if (ch + 1 < nchunks) store_smem(buf ^ 1);
                    __syncthreads();
                }
                if (DIST) {
#pragma unroll
                    for (int m = 0; m < kTM; ++m) {
                        const int s = (m < HM) ? ty * HM + m : BM / 2 + ty * HM + (m - HM);
                        const int64_t i = i0 + s;
#pragma unroll
                        for (int q = 0; q < TN; ++q) {
                            const int cl = (q < HN) ? tx * HN + q : BN / 2 + tx * HN + (q - HN);
                            const int j = c0 + cl;
                            if (i < n && j < k) in.dist[(int64_t)j * n + i] = __fsqrt_rn(acc[m][q]);
                        }
                    }
                    continue;  // smem buffers are rewritten only after the next step's barrier
                }
                // ascending centroid order within this thread's columns
#pragma unroll
                for (int q = 0; q < TN; ++q) {
                    const int cl = (q < HN) ? tx * HN + q : BN / 2 + tx * HN + (q - HN);
                    const float h = hs[cl];
                    const int j = c0 + cl;
#pragma unroll
                    for (int m = 0; m < kTM; ++m) {
                        const float v = h - acc[m][q];
                        if (v < best[m]) {
                            best[m] = v;
                            bidx[m] = j;
                        }
                    }
                }
                __syncthreads();
            }
            if (DIST) continue;
            // (value, index) minimum over the 16 threads sharing these samples
            {
                const int m = rowmin16<float, kTM>(best, bidx, tx);
                if ((tx & (16 / kTM - 1)) == 0) {
                    const int s = (m < HM) ? ty * HM + m : BM / 2 + ty * HM + (m - HM);
                    const int64_t i = i0 + s;
                    if (i < n) labels[i] = bidx[0];
                    labs[s] = bidx[0];
                }
            }
            if (fit) {
                for (int s = tid; s < BM; s += kThreadsB) {
                    const int64_t i = i0 + s;
                    ws[s] = (i < n) ? w[i] : 0.f;
                }
                __syncthreads();
                for (int64_t e = tid; e < (int64_t)BM * d; e += kThreadsB) {
                    const int s = (int)(e % BM);
                    const int64_t f = e / BM;
                    const int64_t i = i0 + s;
                    if (i < n) {
                        // up to kBK features the samples are still in chunk buffer 0
                        const float x = (nchunks == 1) ? Xs[f * BM + s] : X[f * n + i];
                        const float v = __fmul_rn(x, ws[s]);
                        atomicAdd(&tsums[f * k + labs[s]], (double)v);
                    }
                }
                for (int s = tid; s < BM; s += kThreadsB) {
                    const int64_t i = i0 + s;
                    if (i < n) atomicAdd(&tsizes[labs[s]], (double)ws[s]);
                }
            }
            __syncthreads();
        }
        if (priv) {
            for (int64_t e = tid; e < dk + k; e += kThreadsB) {
                const double v = psums[e];
                if (v != 0.0) atomicAdd(&in.sums[e], v);
            }
        }
        __syncthreads();
    }
}

// The same items for instances whose samples fit panels (km_panel.cuh): the
// CTA takes an item, its warps the item's panels of 32 samples; the instance's
// variant chooses the centroids per thread (2, 4 or 8, so 16, 32 or 64 columns
// per step).  One kernel and one queue for all variants: a kernel per variant
// ran one after another, each with its own tail.
template <int DIST>
__global__ void __launch_bounds__(32 * panel::kMaxWarps, 1)
    batch_panel_kernel(const BInst *tab, const BItem *items, int n_items, int *counter) {
    extern __shared__ __align__(16) float psmem[];
    __shared__ int item_sh;
    constexpr int mode = DIST ? panel::MODE_DIST : panel::MODE_LABELS;
    while (true) {
        __syncthreads();  // the last item's shared memory is free
        if (threadIdx.x == 0) item_sh = atomicAdd(counter, 1);
        __syncthreads();
        const int it = item_sh;
        if (it >= n_items) break;
        const BItem item = items[it];
        const BInst &in = tab[item.inst];
        const int warps = panel::warps_for(in.d, mode);
        const int64_t copy =
            DIST ? 0 : (int64_t)((blockIdx.x * panel::kMaxWarps + (threadIdx.x >> 5)) % (unsigned)in.copies);
        const int64_t dk = (int64_t)in.d * in.k;
        // the copies lie one after another, each with its sizes
        double *sums = in.mode == B_FIT ? in.sums + copy * (dk + in.k) : nullptr;
        constexpr int64_t per_tile = kBatchTileM / panel::kRows;
        const int64_t first = item.tile0 * per_tile, end = first + item.ntiles * per_tile;
        if constexpr (DIST) {
            const panel::Args<float, float> a{in.X, nullptr, in.C, nullptr, nullptr, 0, nullptr,
                                              nullptr, in.dist, in.n, in.d, in.k, 1, nullptr};
            if (in.variant == 0)
                panel::run_panels<2, mode, float, float>(a, warps, first, end, warps, 0, psmem);
            else if (in.variant == 1)
                panel::run_panels<4, mode, float, float>(a, warps, first, end, warps, 0, psmem);
            else
                panel::run_panels<8, mode, float, float>(a, warps, first, end, warps, 0, psmem);
        } else {
            const panel::Args<float, double> a{in.X, in.w, in.C, in.hn, in.labels, 0, sums,
                                               sums ? sums + dk : nullptr, nullptr, in.n, in.d,
                                               in.k, 1, nullptr};
            if (in.variant == 0)
                panel::run_panels<2, mode, float, double>(a, warps, first, end, warps, 0, psmem);
            else if (in.variant == 1)
                panel::run_panels<4, mode, float, double>(a, warps, first, end, warps, 0, psmem);
            else
                panel::run_panels<8, mode, float, double>(a, warps, first, end, warps, 0, psmem);
        }
    }
}

// True in the CTA of an instance (gridDim.x of them) that finishes last.
__device__ __forceinline__ bool last_of_instance(unsigned *ticket) {
    __shared__ int last_sh;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last_sh = atomicAdd(ticket, 1u) == gridDim.x - 1u;
        if (last_sh) *ticket = 0u;
    }
    __syncthreads();
    if (last_sh) __threadfence();
    return last_sh != 0;
}

// Private copies -> float32 sums and sizes, the copies zeroed once read, and
// the ascending empty-cluster list.  An instance gets gridDim.x CTAs; a CTA
// takes 32 elements at a time, their copies shared by 16 threads (as in
// reduce_sums_kernel).  One CTA per instance left most SMs idle and walked the
// copies one latency after another: 124 us for 24 instances.
constexpr int kBatchReduceThreads = kReduceLanes * kReduceGroups;

__global__ void __launch_bounds__(kBatchReduceThreads)
    batch_reduce_kernel(BInst *tab, const int *idx, int count, int *n_empty_out) {
    if ((int)blockIdx.y >= count) return;
    __shared__ double red[kReduceGroups][kReduceLanes];
    __shared__ int warp_counts[32];
    BInst &in = tab[idx[blockIdx.y]];
    const int d = in.d, k = in.k;
    const int64_t dk = (int64_t)d * k, total = dk + k;
    const int el = threadIdx.x % kReduceLanes, g = threadIdx.x / kReduceLanes;
    if (in.copies <= kFewSumCopies) {
        // a thread per element, its copies' loads in flight together
        for (int64_t e = blockIdx.x * (int64_t)kBatchReduceThreads + threadIdx.x; e < total;
             e += (int64_t)gridDim.x * kBatchReduceThreads) {
            double x[kFewSumCopies], acc = 0.0;
#pragma unroll
            for (int c = 0; c < kFewSumCopies; ++c)
                x[c] = in.sums[(c < in.copies ? c : 0) * total + e];
#pragma unroll
            for (int c = 0; c < kFewSumCopies; ++c)
                if (c < in.copies) {
                    in.sums[c * total + e] = 0.0;
                    acc += x[c];
                }
            const float v = (float)acc;
            if (e < dk)
                in.Cn[e] = v;
            else
                in.sizes[e - dk] = v;
        }
    } else {
        for (int64_t e0 = blockIdx.x * (int64_t)kReduceLanes; e0 < total;
             e0 += (int64_t)gridDim.x * kReduceLanes) {
            const int64_t e = e0 + el;
            double acc = 0.0;
            if (e < total) {
                for (int c = g; c < in.copies; c += 4 * kReduceGroups) {
                    double v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        v[u] = c + u * kReduceGroups < in.copies
                                   ? in.sums[(int64_t)(c + u * kReduceGroups) * total + e]
                                   : 0.0;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (c + u * kReduceGroups < in.copies) {
                            in.sums[(int64_t)(c + u * kReduceGroups) * total + e] = 0.0;
                            acc += v[u];
                        }
                }
            }
            red[g][el] = acc;
            __syncthreads();
            if (g == 0 && e < total) {
#pragma unroll
                for (int q = 1; q < kReduceGroups; ++q) acc += red[q][el];
                if (e < dk)
                    in.Cn[e] = (float)acc;
                else
                    in.sizes[e - dk] = (float)acc;
            }
            __syncthreads();
        }
    }
    if (!last_of_instance(&in.tickets[0])) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarps = kBatchReduceThreads / 32;
    int base = 0;
    for (int j0 = 0; j0 < k; j0 += kBatchReduceThreads) {
        const int j = j0 + threadIdx.x;
        const bool empty = (j < k) && (__ldcg(in.sizes + j) == 0.f);
        const unsigned ballot = __ballot_sync(0xffffffffu, empty);
        if (lane == 0) warp_counts[wid] = __popc(ballot);
        __syncthreads();
        int before = 0, all = 0;
        for (int q = 0; q < nwarps; ++q) {
            if (q < wid) before += warp_counts[q];
            all += warp_counts[q];
        }
        if (empty) in.empty_list[base + before + __popc(ballot & ((1u << lane) - 1u))] = j;
        base += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        in.empty_list[k] = base;
        in.n_empty = base;
        n_empty_out[blockIdx.y] = base;
    }
}

// Division, shifts (kept in hn, which the next step recomputes) and, in the
// instance's last CTA, the driver's stop rule.  A CTA takes 32 clusters.
__global__ void __launch_bounds__(kFinishThreads)
    batch_update_kernel(BInst *tab, const int *idx, int count, int *done_out, int relocated) {
    if ((int)blockIdx.y >= count) return;
    BInst &in = tab[idx[blockIdx.y]];
    if (!relocated && in.n_empty != 0) return;  // the host relocates first
    __shared__ float diff_sh[kFinishElems];
    __shared__ double sh[32];
    constexpr int kClusters = 32, kFeatures = kFinishElems / kClusters;
    const int d = in.d, k = in.k, tid = threadIdx.x;
    for (int j0 = blockIdx.x * kClusters; j0 < k; j0 += gridDim.x * kClusters) {
        const int j = j0 + (tid & 31);
        const float size = j < k ? in.sizes[j] : 1.f;
        float shift = 0.f;
        for (int f0 = 0; f0 < d; f0 += kFeatures) {
            float s[kFinishOwn], old[kFinishOwn];
#pragma unroll
            for (int u = 0; u < kFinishOwn; ++u) {
                const int f = f0 + (tid >> 5) + u * (kFinishThreads / 32);
                s[u] = old[u] = 0.f;
                if (f < d && j < k) {
                    s[u] = in.Cn[(int64_t)f * k + j];
                    old[u] = in.C[(int64_t)f * k + j];
                }
            }
#pragma unroll
            for (int u = 0; u < kFinishOwn; ++u) {
                const int fl = (tid >> 5) + u * (kFinishThreads / 32), f = f0 + fl;
                if (f < d && j < k) {
                    const float c = s[u] / size;
                    in.Cn[(int64_t)f * k + j] = c;
                    in.C[(int64_t)f * k + j] = c;
                    diff_sh[fl * kClusters + (tid & 31)] = old[u] - c;
                }
            }
            __syncthreads();
            if (tid < 32 && j < k) {
                const int fn = d - f0 < kFeatures ? d - f0 : kFeatures;
#pragma unroll 8
                for (int fl = 0; fl < fn; ++fl) {
                    const float v = diff_sh[fl * kClusters + tid];
                    shift = __fmaf_rn(v, v, shift);
                }
            }
            __syncthreads();
        }
        if (tid < 32 && j < k) in.hn[j] = shift;
    }
    if (!last_of_instance(&in.tickets[1])) return;
    stop_rule<float>(in.hn, k, &in.st, sh);
    if (tid == 0) done_out[blockIdx.y] = in.st.done;
}

// SplitMix64 output function (S. Vigna, public domain).
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float unit01(uint64_t h) {  // [0, 1), 24 bits
    return (float)(h >> 40) * 0x1p-24f;
}

// Gaussian blobs: sample i belongs to centre c(i) = hash(i) mod n_centers;
// centre coordinates uniform in [box_lo, box_hi), per-centre standard
// deviation uniform in [std_lo, std_hi], normal deviates by Box-Muller.
__global__ void blobs_kernel(float *X, int64_t n, int64_t d, int64_t n_centers, float box_lo,
                             float box_hi, float std_lo, float std_hi, uint64_t seed) {
    const uint64_t s_c = mix64(seed ^ 0x1111), s_m = mix64(seed ^ 0x2222),
                   s_s = mix64(seed ^ 0x3333), s_z = mix64(seed ^ 0x4444);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n * d;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t f = e / n, i = e % n;
        const int64_t c = (int64_t)(mix64(s_c ^ (uint64_t)i) % (uint64_t)n_centers);
        const float centre = box_lo + (box_hi - box_lo) * unit01(mix64(s_m ^ (uint64_t)(c * d + f)));
        const float sd = std_lo + (std_hi - std_lo) * unit01(mix64(s_s ^ (uint64_t)c));
        const uint64_t h = mix64(s_z ^ (uint64_t)e);
        const float u1 = ((float)(h >> 40) + 1.f) * 0x1p-24f;  // (0, 1]
        const float u2 = (float)(h & 0xFFFFFFull) * 0x1p-24f;
        const float z = sqrtf(-2.f * logf(u1)) * cospif(2.f * u2);
        X[e] = centre + sd * z;
    }
}

__global__ void gather_rows_kernel(const float *X, int64_t n, int64_t d, const int32_t *idx,
                                   int64_t k, float *C) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < d * k;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t f = e / k, j = e % k;
        const int64_t i = idx[j];
        C[e] = (i >= 0 && i < n) ? X[f * n + i] : 0.f;
    }
}

// Launch shape of each assign variant (shared memory attribute set once, so
// the launch itself can be captured into a graph).
struct AssignShape {
    size_t smem = 0;
    int grid = 0;
};
std::mutex g_shape_mu;
AssignShape g_shape[2][kBatchVariants][64];  // [dist][variant][device]

template <int TN, int DIST>
int assign_shape(int variant, AssignShape *out) {
    int dev = 0;
    KMC_CUDA_TRY(cudaGetDevice(&dev));
    KMC_CHECK_ARG(dev >= 0 && dev < 64, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_shape_mu);
    AssignShape &sh = g_shape[DIST][variant][dev];
    if (sh.grid == 0) {
        const size_t smem = BTile<TN>::base_bytes + kPrivBytes;
        auto kern = batch_assign_kernel<TN, DIST>;
        KMC_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)smem));
        int per_sm = 0;
        KMC_CUDA_TRY(
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreadsB, smem));
        sh.smem = smem;
        sh.grid = num_sms() * (per_sm < 1 ? 1 : per_sm);
    }
    *out = sh;
    return KMC_OK;
}

template <int TN, int DIST>
int launch_assign_v(int variant, const BInst *tab, const BItem *items, int n_items,
                    int *counter, cudaStream_t s) {
    AssignShape sh;
    KMC_TRY((assign_shape<TN, DIST>(variant, &sh)));
    int grid = sh.grid;
    if (grid > n_items) grid = n_items;
    if (grid < 1) return KMC_OK;
    batch_assign_kernel<TN, DIST><<<grid, kThreadsB, sh.smem, s>>>(tab, items, n_items, counter);
    return check_launch("batch_assign");
}

template <int DIST>
int prepare_panels() {
    KMC_CUDA_TRY(cudaFuncSetAttribute(batch_panel_kernel<DIST>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)panel::kSmemBytes));
    return KMC_OK;
}

template <int DIST>
int launch_panels(const BInst *tab, const BItem *items, int n_items, int *counter,
                  cudaStream_t s) {
    const int grid = std::min(n_items, num_sms());
    batch_panel_kernel<DIST><<<grid, 32 * panel::kMaxWarps, panel::kSmemBytes, s>>>(
        tab, items, n_items, counter);
    return check_launch("batch_panel");
}

std::mutex g_tune_mu;
// autotuner choices by (d, power-of-two bucket of k, tag); tag "f32-panel" is
// the batched engine's centroid window, "fit-f32" / "fit-f64" the single-fit tile
std::map<std::tuple<int64_t, int64_t, std::string>, int> g_tune;
bool g_tune_loaded = false;

std::string tune_path() {
    if (const char *p = std::getenv("KMC_TILE_CACHE")) return p;
    std::string base;
    if (const char *x = std::getenv("XDG_CACHE_HOME"))
        base = x;
    else if (const char *h = std::getenv("HOME"))
        base = std::string(h) + "/.cache";
    else
        return "";
    return base + "/kmeans_gb300/tiles.txt";
}

// Lines "d k tag variant"; later lines win.
void tune_load() {
    const std::string p = tune_path();
    if (p.empty()) return;
    std::ifstream f(p);
    std::string line;
    while (std::getline(f, line)) {
        std::istringstream is(line);
        int64_t d = 0, k = 0;
        std::string tag;
        int v = -1;
        if (is >> d >> k >> tag >> v && v >= 0 && v < 8) g_tune[{d, k, tag}] = v;
    }
}

void tune_store(int64_t d, int64_t k, const std::string &tag, int v) {
    const std::string p = tune_path();
    if (p.empty()) return;
    const size_t slash = p.rfind('/');
    if (slash != std::string::npos) {
        // create the cache directory (and its parent) if needed
        const std::string dir = p.substr(0, slash);
        const size_t s2 = dir.rfind('/');
        if (s2 != std::string::npos && s2 > 0) mkdir(dir.substr(0, s2).c_str(), 0755);
        mkdir(dir.c_str(), 0755);
    }
    std::ofstream f(p, std::ios::app);
    if (f) f << d << " " << k << " " << tag << " " << v << "\n";
}

}  // namespace

int batch_sum_copies(int64_t n, int64_t d, int64_t k) {
    // larger sums: a few copies (24 fits of 2,000 to 500,000 samples, d = 8 to
    // 128, k = 4 to 512, 10 iterations: 10.3 -> 10.0 ms)
    const int64_t elems = (d + 1) * k;
    if (elems * (int64_t)sizeof(double) <= (int64_t)kPrivBytes) {
        // few clusters: more copies (207,209 x 32, k = 4 alone: 48 copies 141 us,
        // 404 89)
        const int64_t c = std::min<int64_t>(608, 4864 / std::max<int64_t>(k, 1));
        return (int)std::max<int64_t>(kSumCopies, std::min<int64_t>(c, n / 512));
    }
    return elems <= 65536 ? kFewSumCopies : elems <= 524288 ? 4 : 1;
}

namespace {
// Instances of a launch: its grid counts them along y, whose extent is limited.
// (Along x, with an instance's CTAs far apart, 24 fits ran 1 % slower.)
constexpr int kSliceInstances = 65535;

// launch(first, instances) for slices of `count` instances, at least once.
template <typename F>
int in_slices(int count, const char *what, F launch) {
    for (int first = 0; first == 0 || first < count; first += kSliceInstances) {
        launch(first, std::min(count - first, kSliceInstances));
        KMC_TRY(check_launch(what));
    }
    return KMC_OK;
}
}  // namespace

int launch_batch_prep(BInst *tab, const int *idx, int count, int64_t max_k, int *counters,
                      cudaStream_t s) {
    const unsigned parts = (unsigned)std::max<int64_t>(1, ceil_div<int64_t>(max_k, kPrepThreads));
    return in_slices(count, "batch_prep", [&](int first, int m) {
        const dim3 grid(parts, (unsigned)std::max(m, 1));
        batch_prep_kernel<<<grid, kPrepThreads, 0, s>>>(tab, idx + first, m, counters);
    });
}

int prepare_batch_assign() {
    AssignShape sh;
    KMC_TRY((assign_shape<2, 0>(0, &sh)));
    KMC_TRY((assign_shape<4, 0>(1, &sh)));
    KMC_TRY((assign_shape<8, 0>(2, &sh)));
    KMC_TRY((assign_shape<2, 1>(0, &sh)));
    KMC_TRY((assign_shape<4, 1>(1, &sh)));
    KMC_TRY((assign_shape<8, 1>(2, &sh)));
    KMC_TRY((prepare_panels<0>()));
    return prepare_panels<1>();
}

bool batch_in_panels(int64_t d, int dist) {
    return panel::fits(d, dist ? panel::MODE_DIST : panel::MODE_LABELS);
}

int batch_panel_round(int64_t d, int dist) {
    return panel::warps_for(d, dist ? panel::MODE_DIST : panel::MODE_LABELS) * panel::kRows /
           kBatchTileM;
}

int launch_batch_panels(int dist, const BInst *tab, const BItem *items, int n_items, int *counter,
                        cudaStream_t s) {
    if (n_items <= 0) return KMC_OK;
    return dist ? launch_panels<1>(tab, items, n_items, counter, s)
                : launch_panels<0>(tab, items, n_items, counter, s);
}

int launch_batch_assign(int variant, int dist, const BInst *tab, const BItem *items, int n_items,
                        int *counter, cudaStream_t s) {
    if (n_items <= 0) return KMC_OK;
    if (dist) {
        if (variant == 0) return launch_assign_v<2, 1>(0, tab, items, n_items, counter, s);
        if (variant == 1) return launch_assign_v<4, 1>(1, tab, items, n_items, counter, s);
        return launch_assign_v<8, 1>(2, tab, items, n_items, counter, s);
    }
    if (variant == 0) return launch_assign_v<2, 0>(0, tab, items, n_items, counter, s);
    if (variant == 1) return launch_assign_v<4, 0>(1, tab, items, n_items, counter, s);
    return launch_assign_v<8, 0>(2, tab, items, n_items, counter, s);
}

namespace {
// CTAs per instance: enough for the largest, together about four per SM.
unsigned ctas_per_instance(int64_t most, int count) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(most, 4 * (int64_t)num_sms() / count));
}
}  // namespace

int launch_batch_reduce(BInst *tab, const int *idx, int count, int64_t max_elems,
                        int *n_empty_out, cudaStream_t s) {
    if (count <= 0) return KMC_OK;
    const unsigned parts = ctas_per_instance(ceil_div<int64_t>(max_elems, 2 * kReduceLanes), count);
    return in_slices(count, "batch_reduce", [&](int first, int m) {
        batch_reduce_kernel<<<dim3(parts, (unsigned)m), kBatchReduceThreads, 0, s>>>(
            tab, idx + first, m, n_empty_out + first);
    });
}

int launch_batch_update(BInst *tab, const int *idx, int count, int64_t max_k, int *done_out,
                        bool relocated, cudaStream_t s) {
    if (count <= 0) return KMC_OK;
    const unsigned parts = ctas_per_instance(ceil_div<int64_t>(max_k, 32), count);
    return in_slices(count, "batch_update", [&](int first, int m) {
        batch_update_kernel<<<dim3(parts, (unsigned)m), kFinishThreads, 0, s>>>(
            tab, idx + first, m, done_out + first, relocated ? 1 : 0);
    });
}

int launch_blobs(float *X, int64_t n, int64_t d, int64_t n_centers, float box_lo,
                 float box_hi, float std_lo, float std_hi, uint64_t seed, cudaStream_t s) {
    if (n * d == 0) return KMC_OK;
    KMC_CHECK_ARG(n_centers > 0, "n_centers must be positive");
    const int64_t g = std::min<int64_t>(ceil_div<int64_t>(n * d, 256), 65536);
    blobs_kernel<<<(unsigned)g, 256, 0, s>>>(X, n, d, n_centers, box_lo, box_hi, std_lo, std_hi,
                                             seed);
    return check_launch("blobs");
}

int launch_gather_rows(const float *X, int64_t n, int64_t d, const int32_t *idx, int64_t k,
                       float *C, cudaStream_t s) {
    if (d * k == 0) return KMC_OK;
    const int64_t g = std::min<int64_t>(ceil_div<int64_t>(d * k, 256), 4096);
    gather_rows_kernel<<<(unsigned)g, 256, 0, s>>>(X, n, d, idx, k, C);
    return check_launch("gather_rows");
}

void seeded_rows(int64_t n, int64_t k, uint64_t seed, std::vector<int32_t> *out) {
    out->resize((size_t)k);
    if (n <= 0) return;
    uint64_t a = (mix64(seed) % (uint64_t)n) | 1ull;
    auto gcd = [](uint64_t x, uint64_t y) {
        while (y) {
            const uint64_t t = x % y;
            x = y;
            y = t;
        }
        return x;
    };
    while (gcd(a, (uint64_t)n) != 1) a += 2;
    const uint64_t b = mix64(seed ^ 0x5555) % (uint64_t)n;
    for (int64_t j = 0; j < k; ++j)
        (*out)[(size_t)j] = (int32_t)((a % (uint64_t)n * (uint64_t)j + b) % (uint64_t)n);
}

bool tune_lookup(int64_t d, int64_t k, const char *tag, int *v) {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    if (!g_tune_loaded) {
        tune_load();
        g_tune_loaded = true;
    }
    auto it = g_tune.find({d, k, std::string(tag)});
    if (it == g_tune.end()) return false;
    *v = it->second;
    return true;
}

void tune_record(int64_t d, int64_t k, const char *tag, int v) {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tune[{d, k, std::string(tag)}] = v;
    tune_store(d, k, tag, v);
}

int tune_variant(int64_t d, int64_t k_in, cudaStream_t s, int *variant) {
    // one measurement per (d, power-of-two bucket of k)
    int64_t k = 1;
    while (k < k_in) k <<= 1;
    if (tune_lookup(d, k, "f32-panel", variant) && *variant < kBatchVariants) return KMC_OK;
    KMC_TRY(prepare_batch_assign());
    // Time the three assign kernels on a synthetic fitting instance of this
    // (d, k): 256 tiles of 128 samples, blobs around k centres.
    const int64_t n = 256 * kBatchTileM;
    Scratch mem;
    const size_t off_C = align256(sizeof(float) * d * n);
    const size_t off_hn = off_C + align256(sizeof(float) * d * k);
    const size_t off_w = off_hn + align256(sizeof(float) * k);
    const size_t off_lab = off_w + align256(sizeof(float) * n);
    const size_t off_sum = off_lab + align256(sizeof(int32_t) * n);
    const size_t off_tab = off_sum + align256(sizeof(double) * (d * k + k));
    const size_t off_item = off_tab + align256(sizeof(BInst));
    const size_t off_cnt = off_item + align256(sizeof(BItem) * 64);
    KMC_TRY(mem.alloc(off_cnt + 256, s));
    char *b = mem.as<char>();
    float *X = reinterpret_cast<float *>(b);
    float *C = reinterpret_cast<float *>(b + off_C);
    BInst h{};
    h.X = X;
    h.w = reinterpret_cast<float *>(b + off_w);
    h.C = C;
    h.hn = reinterpret_cast<float *>(b + off_hn);
    h.sums = reinterpret_cast<double *>(b + off_sum);
    h.copies = 1;
    h.labels = reinterpret_cast<int32_t *>(b + off_lab);
    h.n = n;
    h.d = (int)d;
    h.k = (int)k;
    h.mode = B_FIT;
    KMC_TRY(launch_blobs(X, n, d, k, -5.f, 5.f, 1.f, 1.f, 7, s));
    KMC_TRY(launch_blobs(C, k, d, k, -5.f, 5.f, 1.f, 1.f, 8, s));
    KMC_TRY(launch_fill<float>(const_cast<float *>(h.w), 1.f, n, s));
    KMC_TRY(launch_fill<float>(h.hn, 0.f, k, s));
    KMC_TRY(launch_fill<double>(h.sums, 0.0, d * k + k, s));
    BItem hi[64];
    for (int q = 0; q < 64; ++q) hi[q] = BItem{0, 4, (long long)q * 4};
    BInst *tab = reinterpret_cast<BInst *>(b + off_tab);
    BItem *items = reinterpret_cast<BItem *>(b + off_item);
    int *cnt = reinterpret_cast<int *>(b + off_cnt);
    KMC_CUDA_TRY(cudaMemcpyAsync(items, hi, sizeof(hi), cudaMemcpyHostToDevice, s));
    cudaEvent_t e0, e1;
    KMC_CUDA_TRY(cudaEventCreate(&e0));
    KMC_CUDA_TRY(cudaEventCreate(&e1));
    float best_ms = 0.f;
    int best = 2;
    for (int v = 0; v < kBatchVariants; ++v) {
        float tot = 0.f;
        h.variant = v;
        KMC_CUDA_TRY(cudaMemcpyAsync(tab, &h, sizeof(h), cudaMemcpyHostToDevice, s));
        for (int rep = 0; rep < 3; ++rep) {
            KMC_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int), s));
            KMC_CUDA_TRY(cudaEventRecord(e0, s));
            if (batch_in_panels(d, 0))
                KMC_TRY(launch_batch_panels(0, tab, items, 64, cnt, s));
            else
                KMC_TRY(launch_batch_assign(v, 0, tab, items, 64, cnt, s));
            KMC_CUDA_TRY(cudaEventRecord(e1, s));
            KMC_CUDA_TRY(cudaEventSynchronize(e1));
            float ms = 0.f;
            KMC_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
            if (rep > 0) tot += ms;  // first run warms up
        }
        if (v == 0 || tot < best_ms) {
            best_ms = tot;
            best = v;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    KMC_CUDA_TRY(cudaStreamSynchronize(s));
    tune_record(d, k, "f32-panel", best);
    *variant = best;
    return KMC_OK;
}

}  // namespace kmc
