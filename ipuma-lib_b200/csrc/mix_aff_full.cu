// Forward and reverse pass of the classes of model kMixAff (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixAff, false>() {
  return k_mix<kMixAff, false>;
}
}  // namespace ipuma_dev
