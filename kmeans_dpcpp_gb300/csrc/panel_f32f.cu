// Instances of km_panel.cuh: labels (and float32 sums) of float samples.
#include "km_panel_kernel.cuh"

namespace kmc {
namespace panel {
template <>
int launch_labels<float, float>(const Args<float, float> &a, cudaStream_t s) {
    return launch_any<MODE_LABELS, float, float>(a, s);
}
}  // namespace panel
}  // namespace kmc
