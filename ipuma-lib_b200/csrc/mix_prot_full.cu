// Forward and reverse pass of the classes of model kMixProt (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixProt, false>() {
  return k_mix<kMixProt, false>;
}
}  // namespace ipuma_dev
