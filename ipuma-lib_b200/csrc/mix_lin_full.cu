// Forward and reverse pass of the classes of model kMixLin (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixLin, false>() {
  return k_mix<kMixLin, false>;
}
}  // namespace ipuma_dev
