// Labels, fused step and distances of up to 64 features and few centroids, with
// the samples in registers.
//
// A thread holds S samples (S x DP registers, DP = features rounded up to a
// multiple of 4, the rest zero) and walks the centroids, which the CTA keeps
// in shared memory: every lane of a warp reads the same centroid, nothing is
// exchanged between threads, and warps never wait for one another.  With few
// centroids the samples' loads are what counts, and S x d of them are in
// flight per thread; with more, the panels' micro-tiles (km_panel.cuh) use the
// FMA pipe better (labels of 1M samples, registers against panels: 14 features
// and 32 centroids 36 / 40 us, 64 and 20: 90 / 127 us, 8 and 8: 11 / 25 us,
// 4 and 64: 27 / 35 us; but 16 and 1000: 859 / 630 us).
//
// Each score keeps the reference's arithmetic (sequential fma over f = 0..d-1,
// hn - dot, strict < over ascending centroids; src/device_functions.hpp:
// 106-162).  Padded features add 0 * 0, which leaves every sum as it is.
//
// Up to 32 features two samples share an instruction (fma.rn.f32x2: the same
// rounding per half, one issue slot for two products).  Both halves need the
// same centroid value, so shared memory holds each value twice; beyond 32
// features that would saturate the shared-memory port, and single fmas are
// used.
#pragma once

#include "km_kernels.cuh"

namespace kmc {
namespace reg {

constexpr int kMaxFeatures = 64;
constexpr size_t kSmemBytes = 220 * 1024;

constexpr int MODE_LABELS = 0, MODE_DIST = 1;

__host__ __device__ constexpr bool paired(int DP, int mode) { return DP <= 32 || mode == MODE_DIST; }
__host__ __device__ constexpr int samples_per_thread(int DP) { return DP <= 32 ? 4 : 2; }
__host__ __device__ constexpr int max_threads(int DP) { return DP <= 16 ? 512 : 384; }
// Floats per centroid in shared memory: a multiple of 4 that is 4 mod 8, so
// that staging 8 centroids x 4 features writes 32 different banks.
__host__ __device__ constexpr int row_floats(int DP, int mode) {
    const int w = paired(DP, mode) ? 2 * DP : DP;
    return (w % 8 == 4) ? w : w + 4;
}
// Centroids held at once.
__host__ __device__ constexpr int chunk_rows(int DP, int mode) {
    return (int)(kSmemBytes / sizeof(float)) / (row_floats(DP, mode) + 1);
}

template <typename T, typename A>
struct Args {
    const T *X;   // (d, n)
    const T *w;   // (n), with sums
    const T *C;   // (d, k)
    const T *hn;  // (k)
    void *labels;
    int label64;
    A *sums, *sizes;  // private copies ([P][d k], [P][k]); null: labels only
    T *dist;          // MODE_DIST: (k, n)
    int64_t n, d, k, P;
    const LoopState *guard;
};

// f32 input, A = float or double sums, and float64 input (labels only); one
// launcher per feature class, defined in reg_*.cu.
template <typename T, typename A>
int launch_labels(const Args<T, A> &a, cudaStream_t s);
int launch_dist(const Args<float, float> &a, cudaStream_t s);

// Up to this many centroids the registers are used for labels / distances.
constexpr int64_t most_centroids(int mode) { return mode == MODE_DIST ? 32 : 64; }
inline bool fits(int64_t d, int64_t k, int mode) {
    return d >= 1 && d <= kMaxFeatures && k <= most_centroids(mode);
}
// With less than two warps per SM, a thread's own chain over all centroids bounds
// the call, and the panels, which share it among eight lanes, are faster (labels of
// 2000 samples, registers against panels, float32: 14 features and 64 centroids
// 13.1 / 4.0 us, 32 and 16 8.5 / 3.9, 64 and 64 36 / 7.3; but 32 and 4 at 32,000
// 4.4 / 4.8; float64: 32 and 64 49 / 16, but 4 and 53 7.5 / 8.6).
inline bool few_samples(int64_t n, int64_t d, int64_t k, bool f64) {
    const int64_t two_warps = 2 * 32 * (int64_t)num_sms() * samples_per_thread((int)d);
    return n < two_warps && k >= 12 && k * d >= (f64 ? 500 : 200);
}

}  // namespace reg

// ---- sums64.cu: float64 cluster sums of float64 samples, given the labels ----
// Whether a CTA can hold its own copies of the sums.
bool sums64_fits(int64_t d, int64_t k);
// Number of private copies written ([copies][d k] then sizes [copies][k]).
int64_t sums64_copies(int64_t n, int64_t d, int64_t k);
template <typename I>
int launch_sums64(const double *X, const double *w, const I *labels, double *sums, double *sizes,
                  int64_t n, int64_t d, int64_t k, int64_t copies, cudaStream_t s,
                  const LoopState *guard);

}  // namespace kmc
