// Cosines and sines of the vertical modes of the wavemaker potential at the free
// surface, angles pi (2 i + 1) u e with u = 1 / (2 l_add) and e = eta + 1
// (kx_add of HOS-NWT.f90:390-406 times e): one evaluation per run of modes and a
// rotation by pi 2 u e from each to the next.
//
// The angles reach 800: cos(kx_add e) errs by the rounding of kx_add and of the
// product, 4e-15 (rms) at mode 50 and 2.9e-14 over modes 128 to 512.  In units of pi
// nothing is lost but the product's rounding, which the start of a run gives back,
// so that a run errs by its rotations alone: 4.5e-16 over runs of 32 modes
// wherever they lie, below the direct evaluation's from the first mode on.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define HOSNWT_HD __host__ __device__ __forceinline__
#else
#define HOSNWT_HD inline
#endif

namespace hos {

// sin and cos of pi a e; F: (x, *s, *c) -> sin(pi x), cos(pi x)
template <typename F>
HOSNWT_HD void mode_start(double a, double e, F&& sin_cos_pi, double& s, double& c) {
  const double p = a * e;
  const double r = 3.141592653589793238462643 * fma(a, e, -p);
  double s0, c0;
  sin_cos_pi(p, &s0, &c0);
  s = fma(r, c0, s0);
  c = fma(-r, s0, c0);
}
// the next mode's, from the rotation's s2, c2
HOSNWT_HD void mode_next(double s2, double c2, double& s, double& c) {
  const double cn = fma(c, c2, -(s * s2));
  s = fma(s, c2, c * s2);
  c = cn;
}

}  // namespace hos
