// Instances of km_reg.cuh: distances of float samples to the centroids.
#include "km_reg_kernel.cuh"

namespace kmc {
namespace reg {
int launch_dist(const Args<float, float> &a, cudaStream_t s) {
    return launch_any<MODE_DIST, float, float>(a, s);
}
}  // namespace reg
}  // namespace kmc
