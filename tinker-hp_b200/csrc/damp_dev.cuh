// Ewald screening of one pair in FP64: exp(-x^2) and erfc(x) from one exponential.
#pragma once
#include <cuda_runtime.h>

namespace thp {

// ex = exp(-x^2), er = erfc(x) = ex * erfcx(x), x >= 0: erfc() forms the same
// exponential again.  The rounding of x^2 (up to x^2 / 2 ulp of ex) is made
// good to first order.  Over 0 <= x <= 4 (4.2 M points against 80-bit
// references) the largest errors are 1.3 ulp for ex and 3.7 for er; exp(-x*x)
// and erfc(x) have 8.4 and 3.7.  With one rsqrt (0.5 ulp; 1/sqrt 1.5) for the
// root and the division, and the p field formed only where a pair's two scales
// differ, the FP64 direct-field pass at 288,000 atoms takes 1.24 ms (1.39
// before).  The FP32 passes keep exp and erfc: there the same form measured
// 317 against 299 us in the gradient's pair pass at 96,000 atoms.
__device__ __forceinline__ void screen(double x, double& ex, double& er) {
  const double x2 = x * x;
  const double lo = fma(x, x, -x2);
  ex = exp(-x2);
  ex = fma(-lo, ex, ex);
  er = ex * erfcx(x);
}
__device__ __forceinline__ void screen(float x, float& ex, float& er) {
  ex = expf(-x * x);
  er = erfcf(x);
}

}  // namespace thp
