// Division by a small whole number whose reciprocal is at hand.
#pragma once

#include <cmath>
#include <cstring>

namespace hos {

// v / d from r = 1 / d rounded: q = v r, corrected by its exact remainder
// (Markstein, 1990): three operations in place of a division's dozen, which at
// 64 issue cycles each held the steep tank's k_pow_run at 895 us a call.  A v
// whose remainder could underflow, or that is not finite, is divided.
#ifdef __CUDACC__
__host__ __device__ __forceinline__
#else
inline
#endif
double div_by(double v, double d, double r) {
#ifdef __CUDA_ARCH__
  const int hi = __double2hiint(v);
#else
  unsigned long long b;
  std::memcpy(&b, &v, 8);
  const int hi = (int)(b >> 32);
#endif
  const int e = (hi >> 20) & 0x7ff;
  if (e < 64 || e == 0x7ff) return v / d;
  const double q = v * r;
  return fma(fma(-d, q, v), r, q);
}

}  // namespace hos
