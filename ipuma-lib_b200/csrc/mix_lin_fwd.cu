// Forward pass of the classes of model kMixLin (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixLin, true>() {
  return k_mix<kMixLin, true>;
}
}  // namespace ipuma_dev
