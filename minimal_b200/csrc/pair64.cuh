// FP64 body pairs (3d/kernel.h:122-150), shared by the near field and the
// direct sums.
#pragma once
#include <cuda_runtime.h>

namespace fmm {

// One pair with every case handled: a pair at distance zero contributes
// nothing.
__device__ __forceinline__ void pair(double xi, double yi, double zi, const double4 s, double &pot, double &ax,
                                     double &ay, double &az) {
  const double dx = xi - s.x, dy = yi - s.y, dz = zi - s.z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double ir = r2 > 0 ? rsqrt(r2) : 0.0;
  const double qir = s.w * ir;
  const double qir3 = qir * ir * ir;
  pot += qir;
  ax += dx * qir3;
  ay += dy * qir3;
  az += dz * qir3;
}

// The same pair for a normal r2: 1/sqrt(r2) by one third-order Householder
// step from the hardware's estimate y (relative error e/2 of about 2^-21,
// e = 1 - r2 y^2): y (1 + e/2 + 3 e^2/8), the next term e^3 5/16 below
// 2^-60.  Without rsqrt()'s special cases the pairs of an unrolled sweep
// overlap: the near field of 1M uniform bodies takes 3398 us against 4368
// with rsqrt(), the direct sum of 1M bodies on 1,000 targets 1395 against
// 2062 (the 18 FP64 instructions of a pair take 2730 and 1155 us at the FP64
// peak).
// r2 zero, subnormal, infinite or NaN gives a potential that is not finite
// (0 and infinity: NaN; subnormal: the flushed estimate is infinite), for
// any charge, so a sum of these pairs with a finite potential had none.
__device__ __forceinline__ void pair_normal(double xi, double yi, double zi, const double4 s, double &pot, double &ax,
                                            double &ay, double &az) {
  const double dx = xi - s.x, dy = yi - s.y, dz = zi - s.z;
  const double r2 = dx * dx + dy * dy + dz * dz;
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
  const double e = fma(-(r2 * y), y, 1.0);
  const double ir = fma(y * e, fma(0.375, e, 0.5), y);
  const double qir = s.w * ir;
  const double qir3 = qir * ir * ir;
  pot += qir;
  ax += dx * qir3;
  ay += dy * qir3;
  az += dz * qir3;
}

}  // namespace fmm
