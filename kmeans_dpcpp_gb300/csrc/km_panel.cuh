// Labels (and cluster sums) or distances of samples in panels, one per warp.
//
// A warp takes 32 samples at a time, all their features as a panel in shared
// memory (d x 32 floats), and walks the centroids, which the whole CTA shares:
// resident when they fit, else streamed in double-buffered blocks of columns.
// Each thread forms an 8 x TN micro-tile (8 samples, TN centroids) of dot
// products or squared distances.  With resident centroids no warp ever waits
// for another.
//
// Each element keeps the reference's arithmetic: one fused multiply-add per
// feature, f = 0..d-1 in order, then hn - dot and the first minimum over
// ascending centroids (src/device_functions.hpp:106-162).  Features are padded
// to an even number with zeros, which change nothing.
//
// What bounds it and why it looks like this:
//  - the FMA pipe takes 128 products per clock and SM as single fmas or as
//    pairs (fma.rn.f32x2); pairs leave half the issue slots to the loads and
//    the argmin.  In isolation this micro-tile reaches 93 % of the pipe,
//    single fmas 82 %, and samples held in registers against broadcast
//    centroids 70 % (each operand is then read from the register file once);
//  - tiles shared by a CTA, 16 features per barrier, ran at 61 %: all warps
//    load, compute and wait together.  Panels need no barrier (1M x 64 against
//    512: 1.17 ms, 74 %; 1.57 ms before);
//  - operands held twice in shared memory, which saves the moves that double
//    them, were slower (2M x 14 against 127: 0.22 against 0.19 ms);
//  - the panel also serves the cluster sums (a lane per sample), which went
//    back to global memory before.
//
// Float64 samples: labels from float32 scores with a rounding bound (Bound
// below), the undecided samples in float64 by their warp.
#pragma once

#include <algorithm>
#include <type_traits>

#include "km_reg.cuh"

namespace kmc {
namespace panel {

constexpr int MODE_LABELS = 0, MODE_DIST = 1;
constexpr int kMaxWarps = 16;
constexpr int kRows = 32;  // samples of a panel
constexpr size_t kSmemBytes = 224 * 1024;

template <typename T, typename A>
using Args = reg::Args<T, A>;

// Shared memory of a launch: offsets and sizes in floats.
struct Shape {
    int dp;        // features padded to even
    int bn;        // columns of a warp's step
    int kp;        // columns held: all of them padded to bn, or a block of bn
    int resident;  // all centroids are held
    size_t c, hn, panels, labs, out, total;
};

__host__ __device__ inline Shape shape(int64_t d, int64_t k, int tn, int mode, int warps) {
    Shape s;
    s.dp = (int)(d + (d & 1));
    s.bn = 8 * tn;
    const int64_t kall = ceil_div<int64_t>(k, s.bn) * s.bn;
    const size_t per_warp =
        (size_t)s.dp * kRows + kRows + (mode == MODE_DIST ? (size_t)kRows * 33 : 0);
    s.resident = kall * (s.dp + 1) + warps * per_warp <= kSmemBytes / sizeof(float);
    s.kp = s.resident ? (int)kall : s.bn;
    size_t off = 0;
    s.c = off;
    off += (size_t)s.kp * s.dp * (s.resident ? 1 : 2);
    s.hn = off;
    off += (size_t)s.kp * (s.resident ? 1 : 2);
    s.panels = off;
    off += (size_t)warps * s.dp * kRows;
    s.labs = off;
    off += (size_t)warps * kRows;
    s.out = off;
    if (mode == MODE_DIST) off += (size_t)warps * kRows * 33;
    s.total = off;
    return s;
}

// Warps of a CTA for d features: as many as fit beside two column blocks.
__host__ __device__ inline int warps_for(int64_t d, int mode) {
    for (int w = kMaxWarps; w >= 8; w -= 4) {
        const Shape s = shape(d, int64_t(1) << 40, 8, mode, w);
        if (s.total * sizeof(float) <= kSmemBytes) return w;
    }
    return 0;
}
__host__ __device__ inline bool fits(int64_t d, int mode = MODE_LABELS) { return d >= 1 && warps_for(d, mode) > 0; }

// T float with A float or double sums, and T = A = double (labels only).
template <typename T, typename A>
int launch_labels(const Args<T, A> &a, cudaStream_t s);
int launch_dist(const Args<float, float> &a, cudaStream_t s);

}  // namespace panel
}  // namespace kmc
