// sin and cos together in FP64 for the phases exp(i q.r) of the reconstruction.
#pragma once

namespace fame {

// Cody & Waite argument reduction (W. J. Cody, W. Waite, Software Manual for the Elementary
// Functions, 1980) with pi/2 as the sum of two doubles, each product exact in its FMA, then the
// Taylor polynomials of sin (to x^17) and cos (to x^16) on [-pi/4, pi/4], whose truncation is
// below 3e-18.  Absolute error below 3e-16, tested at and around multiples of pi/2; arguments beyond
// 2^19 pi/2, infinities and NaN go to sincos.  Branch-free otherwise, with the two polynomials
// as independent chains, about 35 FP64 instructions: it shares the FP64 pipe with the products
// of the Taylor moments.
__device__ __forceinline__ void sincos_phase(double x, double* s, double* c) {
  if (!(fabs(x) < 823549.0)) {
    sincos(x, s, c);
    return;
  }
  const double k = rint(x * 0.63661977236758134308);            // 2 / pi
  const double r0 = fma(-k, 1.5707963267948965580, x);            // pi / 2 rounded to a double
  const double r = fma(-k, 6.1232339957367658860e-17, r0);        // and the rest of pi / 2
  const double z = r * r;
  double ps = 1.0 / 355687428096000.0;                            // 1/17!
  double pc = 1.0 / 20922789888000.0;                             // 1/16!
  ps = fma(-ps, z, 1.0 / 1307674368000.0);                        // 1/15!
  pc = fma(-pc, z, 1.0 / 87178291200.0);                          // 1/14!
  ps = fma(-ps, z, 1.0 / 6227020800.0);
  pc = fma(-pc, z, 1.0 / 479001600.0);
  ps = fma(-ps, z, 1.0 / 39916800.0);
  pc = fma(-pc, z, 1.0 / 3628800.0);
  ps = fma(-ps, z, 1.0 / 362880.0);
  pc = fma(-pc, z, 1.0 / 40320.0);
  ps = fma(-ps, z, 1.0 / 5040.0);
  pc = fma(-pc, z, 1.0 / 720.0);
  ps = fma(-ps, z, 1.0 / 120.0);
  pc = fma(-pc, z, 1.0 / 24.0);
  ps = fma(-ps, z, 1.0 / 6.0);
  pc = fma(-pc, z, 0.5);
  const double sn = fma(-ps * z, r, r);
  const double cs = fma(-pc, z, 1.0);
  const int q = (int)k;
  const double a = (q & 1) ? cs : sn, b = (q & 1) ? sn : cs;
  *s = (q & 2) ? -a : a;
  *c = ((q + 1) & 2) ? -b : b;
}

}  // namespace fame
