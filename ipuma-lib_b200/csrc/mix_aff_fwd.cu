// Forward pass of the classes of model kMixAff (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixAff, true>() {
  return k_mix<kMixAff, true>;
}
}  // namespace ipuma_dev
