// The pass kernels of one butterfly kind (ntt_kernels.cuh).
#include "ntt_kernels.cuh"

namespace aoa {
AOA_NTT_KIND(, kButterflyLazyQ1)
}  // namespace aoa
