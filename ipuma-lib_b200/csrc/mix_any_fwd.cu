// Forward pass of the classes of model kMixAny (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixAny, true>() {
  return k_mix<kMixAny, true>;
}
}  // namespace ipuma_dev
