// Instances of km_panel.cuh: labels of float64 samples.
#include "km_panel_kernel.cuh"

namespace kmc {
namespace panel {
template <>
int launch_labels<double, double>(const Args<double, double> &a, cudaStream_t s) {
    return launch_any<MODE_LABELS, double, double>(a, s);
}
}  // namespace panel
}  // namespace kmc
