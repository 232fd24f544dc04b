// Instances of km_panel.cuh: distances of float samples to the centroids.
#include "km_panel_kernel.cuh"

namespace kmc {
namespace panel {
int launch_dist(const Args<float, float> &a, cudaStream_t s) {
    return launch_any<MODE_DIST, float, float>(a, s);
}
}  // namespace panel
}  // namespace kmc
