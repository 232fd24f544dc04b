// Instances of km_reg.cuh: labels (and sums) of double samples, double sums.
#include "km_reg_kernel.cuh"

namespace kmc {
namespace reg {
template <>
int launch_labels<double, double>(const Args<double, double> &a, cudaStream_t s) {
    return launch_any<MODE_LABELS, double, double>(a, s);
}
}  // namespace reg
}  // namespace kmc
