// O(k*d) and O(n) kernels of the Lloyd engine: half norms, broadcast
// division, private-copy reduction with empty-cluster detection, centroid
// shifts, per-sample inertia and deterministic float64 sums.
//
// Arithmetic order follows the SYCL kernels cited on each function: sums over
// features run sequentially f = 0..d-1 with a fused multiply-add, exactly as
// `acc += a * b` is contracted by the reference's device compiler.
#include <algorithm>

#include "km_dist.cuh"
#include "km_kernels.cuh"

namespace kmc {

namespace {

__device__ __forceinline__ bool stopped(const LoopState *g) {
    return g != nullptr && *reinterpret_cast<const volatile int *>(&g->done) != 0;
}

// broadcast_division_kernel, src/util_kernels.hpp:9-41: X[r, c] /= y[c].
template <typename T>
__global__ void broadcast_divide_kernel(T *X, const T *y, int64_t rows, int64_t cols) {
    int64_t total = rows * cols;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = e % cols;
        X[e] = X[e] / y[c];
    }
}

// half_l2_norm_kernel, src/util_kernels.hpp:47-82: out[j] = (sum_f C[f,j]^2) / 2.
template <typename T>
__global__ void half_norm_kernel(const T *C, T *out, int64_t d, int64_t k,
                                 const LoopState *guard) {
    if (stopped(guard)) return;
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= k) return;
    T acc = T(0);
    // eight features' loads in flight before the sequential chain
    int64_t f = 0;
    for (; f + 8 <= d; f += 8) {
        T v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = C[(f + u) * k + j];
#pragma unroll
        for (int u = 0; u < 8; ++u) acc = fma_rn(v[u], v[u], acc);
    }
    for (; f < d; ++f) {
        const T v = C[f * k + j];
        acc = fma_rn(v, v, acc);
    }
    out[j] = acc / T(2);
}

// reduce_centroid_data_kernel, src/util_kernels.hpp:87-161, part 1: sums of
// the private copies (sums and sizes).  A CTA takes 32 consecutive elements;
// G threads share an element's copies (g, g + G, ... in order, eight loads in
// flight; then the G partial sums in order), because one thread per element
// walks thousands of copies as a chain of memory latencies (8448 elements,
// 2642 copies: 206 us).  Float sums then also round less: P / G + G additions
// follow one another instead of P.
constexpr int kCopyLanes = 32;

template <typename T, int G>
__global__ void __launch_bounds__(kCopyLanes * G)
    reduce_copies_kernel(const T *sizes_cp, const T *cent_cp, T *out_sizes, T *out_cent, int64_t P,
                         int64_t d, int64_t k) {
    __shared__ T red[G][kCopyLanes];
    const int64_t dk = d * k;
    const int el = threadIdx.x % kCopyLanes, g = threadIdx.x / kCopyLanes;
    for (int64_t e0 = blockIdx.x * (int64_t)kCopyLanes; e0 < dk + k;
         e0 += (int64_t)gridDim.x * kCopyLanes) {
        const int64_t e = e0 + el;
        T s = T(0);
        if (e < dk + k) {
            const T *src = (e < dk) ? cent_cp + e : sizes_cp + (e - dk);
            const int64_t stride = (e < dk) ? dk : k;
            for (int64_t p = g; p < P; p += 8 * G) {
                T v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = p + u * G < P ? src[(p + u * G) * stride] : T(0);
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (p + u * G < P) s += v[u];
            }
        }
        red[g][el] = s;
        __syncthreads();
        if (g == 0 && e < dk + k) {
#pragma unroll
            for (int q = 1; q < G; ++q) s += red[q][el];
            if (e < dk)
                out_cent[e] = s;
            else
                out_sizes[e - dk] = s;
        }
        __syncthreads();
    }
}

// The same sums, bit for bit, by one thread per element that holds the G partial
// sums.  With enough elements (wide_sums) there are threads enough, and whole
// warps read consecutive ones.  float64 additions bound the float64 form, so its
// CTAs are small, for equal shares of the SMs.  137,004 elements: 16 copies 23.6 ->
// 9.3 us (float64 48 -> 17), 152 copies 38 -> 15 (90 -> 64); 4 copies 11.3 -> 9.3.
template <typename T>
constexpr int kWideThreads = sizeof(T) == 8 ? 64 : 256;

// 16 threads per element are as fast below (21,000 elements of 304 float copies
// 13.4 us, by one thread 15.4; 31,000: 15.4, 15.4; 16,000 of 64: 11.3, 9.3;
// float64 41,000 of 304: 49, 60; 61,000: 68, 66).
template <typename T>
bool wide_sums(int64_t elems, int64_t P) {
    return elems >= std::max<int64_t>(16384, (sizeof(T) == 8 ? 200 : 100) * P);
}

template <typename T, int G>
__global__ void __launch_bounds__(kWideThreads<T>)
    reduce_copies_wide_kernel(const T *sizes_cp, const T *cent_cp, T *out_sizes, T *out_cent,
                              int64_t P, int64_t d, int64_t k) {
    const int64_t dk = d * k, e = blockIdx.x * (int64_t)kWideThreads<T> + threadIdx.x;
    if (e >= dk + k) return;
    const T *src = (e < dk) ? cent_cp + e : sizes_cp + (e - dk);
    const int64_t stride = (e < dk) ? dk : k;
    constexpr int kBatch = G > 1 ? G : 4;
    T s[G];
#pragma unroll
    for (int g = 0; g < G; ++g) s[g] = T(0);
    int64_t p = 0;
    for (; p + kBatch <= P; p += kBatch) {
        T v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) v[u] = load_in_order(src + (p + u) * stride);
#pragma unroll
        for (int u = 0; u < kBatch; ++u) s[u % G] += v[u];
    }
    if constexpr (G == 1) {
        for (; p < P; ++p) s[0] += src[p * stride];
    } else if (p < P) {
        T v[G];
#pragma unroll
        for (int u = 0; u < G; ++u)
            v[u] = load_in_order(src + (p + u < P ? p + u : p) * stride);
#pragma unroll
        for (int u = 0; u < G; ++u)
            if (p + u < P) s[u] += v[u];
    }
#pragma unroll
    for (int g = 1; g < G; ++g) s[0] += s[g];
    if (e < dk)
        out_cent[e] = s[0];
    else
        out_sizes[e - dk] = s[0];
}

// Part 2: empty-cluster list.  The reference appends through an atomic
// counter in arbitrary order (util_kernels.hpp:143-153, marked FIXME there);
// here the list is built in ascending cluster order by one block, starting
// at the counter's current value.
template <typename T, typename I>
__global__ void empty_list_kernel(const T *sizes, I *list, I *n_empty, int64_t k) {
    __shared__ int warp_counts[32];
    __shared__ long long base_sh;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    if (threadIdx.x == 0) base_sh = (long long)(*n_empty);
    __syncthreads();
    for (int64_t j0 = 0; j0 < k; j0 += blockDim.x) {
        int64_t j = j0 + threadIdx.x;
        bool empty = (j < k) && (sizes[j] == T(0));
        unsigned ballot = __ballot_sync(0xffffffffu, empty);
        if (lane == 0) warp_counts[wid] = __popc(ballot);
        __syncthreads();
        long long before = 0, total = 0;
        for (int w = 0; w < nwarps; ++w) {
            if (w < wid) before += warp_counts[w];
            total += warp_counts[w];
        }
        if (empty) {
            long long pos = base_sh + before + __popc(ballot & ((1u << lane) - 1u));
            if (pos >= 0 && pos < k) list[pos] = (I)j;  // the counter is caller-initialised
        }
        __syncthreads();
        if (threadIdx.x == 0) base_sh += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *n_empty = (I)base_sh;
}

// compute_centroid_shifts_squared_kernel, src/util_kernels.hpp:481-516.
template <typename T>
__global__ void shifts_kernel(const T *old_c, const T *new_c, T *out, int64_t d, int64_t k) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= k) return;
    T acc = T(0);
    for (int64_t f = 0; f < d; ++f) {
        T diff = old_c[f * k + j] - new_c[f * k + j];
        acc = fma_rn(diff, diff, acc);
    }
    out[j] = acc;
}

// Fixed-order block reduction of doubles (deterministic for a given grid).
__device__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (wid == 0) {
        r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    __syncthreads();
    return r;  // valid in thread 0
}

// compute_inertia_kernel / compute_uniform_weight_inertia_kernel,
// src/compute_inertia.hpp:11-99.  w == nullptr gives the unit-weight form.
template <typename T, typename I>
__global__ void inertia_kernel(const T *X, const T *w, const T *C, const I *labels, T *out,
                               int64_t n, int64_t d, int64_t k, int64_t fs, int64_t ss) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = (int64_t)labels[i];
        if (c < 0 || c >= k) {  // caller-supplied label out of range
            out[i] = pos_inf<T>();
            continue;
        }
        const T acc = sq_dist_cols<T>(X, fs, ss, C, d, k, i, c);
        out[i] = (w != nullptr) ? mul_rn(acc, w[i]) : acc;
    }
}

// The same for row-major samples and centroids (zero-padded to a multiple of
// four features).  Bound by reading X once: 10M x 64 took 2.97 ms with a thread
// per row reading X and the (d, k) centroids 4 bytes at a time.
constexpr int kInertiaThreads = 256;
template <typename I>
__global__ void __launch_bounds__(kInertiaThreads)
    inertia_rows_kernel(const float *X, int64_t ss, const float *w, const float *C, int64_t cs,
                        const I *labels, float *out, int64_t n, int64_t d, int64_t k) {
    extern __shared__ float tiles[];
    const int lane = threadIdx.x & 31;
    float *tile = tiles + (threadIdx.x >> 5) * kDistTile;
    for (int64_t i0 = blockIdx.x * (int64_t)kInertiaThreads; i0 < n;
         i0 += (int64_t)gridDim.x * kInertiaThreads) {
        const int64_t i = i0 + threadIdx.x;
        const int64_t c = i < n ? (int64_t)labels[i] : -1;
        const bool ok = c >= 0 && c < k;
        float v = pos_inf<float>();
        if (d > kRowVec) {
            const float r = sq_dist_warp(X, ss, C, cs, d, i - lane, ok ? c : -1, tile);
            if (ok) v = r;
        } else if (ok) {
            v = sq_dist_row(X + i * ss, C + c * cs, d);
        }
        if (i < n) out[i] = ok && w != nullptr ? mul_rn(v, w[i]) : v;
    }
}

constexpr int kSumGrid = 1024;
constexpr int kSumBlock = 256;

template <typename T>
__global__ void sum_stage1_kernel(const T *data, int64_t n, double *partials) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        acc += (double)data[i];
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = r;
}

__global__ void sum_stage2_kernel(const double *partials, int count, double *out) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < count; i += blockDim.x) acc += partials[i];
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) *out = r;
}

template <typename T>
__global__ void fill_kernel(T *p, T v, int64_t count) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < count;
         e += (int64_t)gridDim.x * blockDim.x)
        p[e] = v;
}

inline unsigned grid_for(int64_t work, int block, int max_blocks = 4096) {
    int64_t g = ceil_div<int64_t>(work, block);
    if (g < 1) g = 1;
    if (g > max_blocks) g = max_blocks;
    return (unsigned)g;
}

}  // namespace

template <typename T>
int launch_broadcast_divide(T *X, const T *y, int64_t rows, int64_t cols, cudaStream_t s) {
    if (rows * cols == 0) return KMC_OK;
    broadcast_divide_kernel<T><<<grid_for(rows * cols, 256, 8192), 256, 0, s>>>(X, y, rows, cols);
    return check_launch("broadcast_divide");
}

template <typename T>
int launch_half_norm(const T *C, T *out, int64_t d, int64_t k, cudaStream_t s,
                     const LoopState *guard) {
    if (k == 0) return KMC_OK;
    half_norm_kernel<T><<<grid_for(k, 128, 1 << 20), 128, 0, s>>>(C, out, d, k, guard);
    return check_launch("half_l2_norm");
}

template <typename T, typename I>
int launch_reduce_centroids(const T *sizes_cp, const T *cent_cp, T *out_sizes, T *out_cent,
                            I *empty_list, I *n_empty, int64_t P, int64_t d, int64_t k,
                            cudaStream_t s) {
    if (k == 0) return KMC_OK;
    const int64_t elems = d * k + k;
    const unsigned wide = (unsigned)ceil_div<int64_t>(elems, kWideThreads<T>);
    if (P <= 8)
        reduce_copies_wide_kernel<T, 1><<<wide, kWideThreads<T>, 0, s>>>(
            sizes_cp, cent_cp, out_sizes, out_cent, P, d, k);
    else if (wide_sums<T>(elems, P))
        reduce_copies_wide_kernel<T, 16><<<wide, kWideThreads<T>, 0, s>>>(
            sizes_cp, cent_cp, out_sizes, out_cent, P, d, k);
    else
        reduce_copies_kernel<T, 16><<<grid_for(elems, kCopyLanes, 16384), kCopyLanes * 16, 0, s>>>(
            sizes_cp, cent_cp, out_sizes, out_cent, P, d, k);
    KMC_TRY(check_launch("reduce_centroids_data"));
    empty_list_kernel<T, I><<<1, 1024, 0, s>>>(out_sizes, empty_list, n_empty, k);
    return check_launch("empty_clusters_list");
}

template <typename T>
int launch_shifts(const T *old_c, const T *new_c, T *out, int64_t d, int64_t k,
                  cudaStream_t s) {
    if (k == 0) return KMC_OK;
    shifts_kernel<T><<<grid_for(k, 128, 1 << 20), 128, 0, s>>>(old_c, new_c, out, d, k);
    return check_launch("centroid_shifts");
}

template <typename T, typename I>
int launch_inertia(const T *X, const T *w, const T *C, const I *labels, T *out, int64_t n,
                   int64_t d, int64_t k, cudaStream_t s, int64_t x_fstride, int64_t x_sstride,
                   const T *c_rows, int64_t c_stride) {
    if (n == 0) return KMC_OK;
    const int64_t fs = x_fstride > 0 ? x_fstride : n, ss = x_fstride > 0 ? x_sstride : 1;
    if constexpr (sizeof(T) == 4) {
        if (c_rows != nullptr && fs == 1) {
            const size_t smem =
                d > kRowVec ? sizeof(float) * kDistTile * (kInertiaThreads / 32) : 0;
            inertia_rows_kernel<I><<<grid_for(n, kInertiaThreads, num_sms() * 16), kInertiaThreads,
                                     smem, s>>>(X, ss, w, c_rows, c_stride, labels, out, n, d, k);
            return check_launch("compute_inertia_rows");
        }
    }
    inertia_kernel<T, I><<<grid_for(n, 256, 16384), 256, 0, s>>>(X, w, C, labels, out, n, d, k, fs,
                                                                 ss);
    return check_launch("compute_inertia");
}

int64_t sum_partials_size() { return kSumGrid; }

template <typename T>
int launch_sum_f64(const T *data, int64_t n, double *partials, double *out, cudaStream_t s) {
    sum_stage1_kernel<T><<<kSumGrid, kSumBlock, 0, s>>>(data, n, partials);
    KMC_TRY(check_launch("sum_stage1"));
    sum_stage2_kernel<<<1, 1024, 0, s>>>(partials, kSumGrid, out);
    return check_launch("sum_stage2");
}

template <typename T>
int launch_fill(T *p, T v, int64_t count, cudaStream_t s) {
    if (count == 0) return KMC_OK;
    fill_kernel<T><<<grid_for(count, 256, 8192), 256, 0, s>>>(p, v, count);
    return check_launch("fill");
}

#define KMC_INST_T(T)                                                                        \
    template int launch_broadcast_divide<T>(T *, const T *, int64_t, int64_t, cudaStream_t); \
    template int launch_half_norm<T>(const T *, T *, int64_t, int64_t, cudaStream_t,          \
                                     const LoopState *);                                      \
    template int launch_shifts<T>(const T *, const T *, T *, int64_t, int64_t, cudaStream_t); \
    template int launch_sum_f64<T>(const T *, int64_t, double *, double *, cudaStream_t);     \
    template int launch_fill<T>(T *, T, int64_t, cudaStream_t);

#define KMC_INST_TI(T, I)                                                                     \
    template int launch_reduce_centroids<T, I>(const T *, const T *, T *, T *, I *, I *,      \
                                               int64_t, int64_t, int64_t, cudaStream_t);      \
    template int launch_inertia<T, I>(const T *, const T *, const T *, const I *, T *,        \
                                      int64_t, int64_t, int64_t, cudaStream_t, int64_t,       \
                                      int64_t, const T *, int64_t);

KMC_INST_T(float)
KMC_INST_T(double)
template int launch_fill<int32_t>(int32_t *, int32_t, int64_t, cudaStream_t);
template int launch_fill<int64_t>(int64_t *, int64_t, int64_t, cudaStream_t);
KMC_INST_TI(float, int32_t)
KMC_INST_TI(float, int64_t)
KMC_INST_TI(double, int32_t)
KMC_INST_TI(double, int64_t)

}  // namespace kmc
