// Forward and reverse pass of the classes of model kMixAny (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixAny, false>() {
  return k_mix<kMixAny, false>;
}
}  // namespace ipuma_dev
