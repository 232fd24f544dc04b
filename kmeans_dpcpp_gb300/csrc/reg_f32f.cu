// Instances of km_reg.cuh: labels (and sums) of float samples, float sums.
#include "km_reg_kernel.cuh"

namespace kmc {
namespace reg {
template <>
int launch_labels<float, float>(const Args<float, float> &a, cudaStream_t s) {
    return launch_any<MODE_LABELS, float, float>(a, s);
}
}  // namespace reg
}  // namespace kmc
