// Instances of km_panel.cuh: labels (and float64 sums) of float samples.
#include "km_panel_kernel.cuh"

namespace kmc {
namespace panel {
template <>
int launch_labels<float, double>(const Args<float, double> &a, cudaStream_t s) {
    return launch_any<MODE_LABELS, float, double>(a, s);
}
}  // namespace panel
}  // namespace kmc
