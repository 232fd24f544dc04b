// Instances of km_reg.cuh: labels (and sums) of float samples, double sums.
#include "km_reg_kernel.cuh"

namespace kmc {
namespace reg {
template <>
int launch_labels<float, double>(const Args<float, double> &a, cudaStream_t s) {
    return launch_any<MODE_LABELS, float, double>(a, s);
}
}  // namespace reg
}  // namespace kmc
