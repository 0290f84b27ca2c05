// Per-coefficient arithmetic of the key-switch results (Q limbs, transform
// domain), shared by ks_finish.cu and the whole-limb kernels.
#pragma once
#include "aoa_internal.h"

namespace aoa {

__device__ __forceinline__ void mac_wide(uint64_t& lo, uint64_t& hi, uint64_t a, uint64_t b) {
  const uint64_t l = a * b;
  hi += __umul64hi(a, b);
  lo += l;
  hi += lo < l;
}

// 2^33 <= q < 2^60: a sum of three products below q^2 is in one Barrett step's
// range (2^(64 + s), s = bit length - 2)
__device__ __forceinline__ bool sums_fit(const PrimeConst& P) { return P.bar_sh && P.bar_sh <= 58; }

// a0 b0 + d2 kb mod q (the first poly of HMult)
__device__ __forceinline__ uint64_t ks_sum2(uint64_t a0, uint64_t b0, uint64_t d2, uint64_t kb, bool fit,
                                            const PrimeConst& P) {
  if (!fit) return add_mod(mul_mod(a0, b0, P), mul_mod(d2, kb, P), P.q);
  uint64_t lo = a0 * b0, hi = __umul64hi(a0, b0);
  mac_wide(lo, hi, d2, kb);
  return barrett_wide(lo, hi, P.q, P.bar_mu, (uint32_t)P.bar_sh);
}

// a0 b1 + a1 b0 + d2 ka mod q (the second)
__device__ __forceinline__ uint64_t ks_sum3(uint64_t a0, uint64_t a1, uint64_t b0, uint64_t b1, uint64_t d2,
                                            uint64_t ka, bool fit, const PrimeConst& P) {
  if (!fit)
    return add_mod(add_mod(mul_mod(a0, b1, P), mul_mod(a1, b0, P), P.q), mul_mod(d2, ka, P), P.q);
  uint64_t lo = a0 * b1, hi = __umul64hi(a0, b1);
  mac_wide(lo, hi, a1, b0);
  mac_wide(lo, hi, d2, ka);
  return barrett_wide(lo, hi, P.q, P.bar_mu, (uint32_t)P.bar_sh);
}

}  // namespace aoa
