// Forward pass of the classes of model kMixProt (k_mix).
#include "class_mix.cuh"

namespace ipuma_dev {
template <>
MixKernel mix_kernel<kMixProt, true>() {
  return k_mix<kMixProt, true>;
}
}  // namespace ipuma_dev
