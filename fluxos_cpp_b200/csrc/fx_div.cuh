// FP64 quotients that cost less than a division and have its bits.
#pragma once
#include <cuda_runtime.h>

namespace fx {

// Quotients over a shared denominator, the bits of a / b: y = 1 / b, correctly
// rounded, then two Newton corrections of a * y. The first leaves a faithful
// quotient, so by Markstein's theorem (IBM J. Res. Dev. 34, 1990; Muller et al.,
// Handbook of Floating-Point Arithmetic, ch. 4) the second rounds correctly; its
// residual is exact for |a| >= 2^-700 and b, a below 2^200, 2^700. Anything else
// divides, except 0, whose quotient is a * y (an FP64 division of 0 takes 436
// cycles against 146 of an ordinary one, measured, and dry and resting cells
// divide 0 all the time). The division stays out of line: a dozen copies of it
// in the kernel cost more in instruction fetches than the quotients save
// (2048 x 2048 cells 0.82 ms a step with them inline, 0.70 ms without, 0.80 ms
// with plain divisions).
static __device__ __noinline__ double plain_div(double a, double b) { return a / b; }
struct Over {
  double b, y;
  bool ok;
  Over() = default;
  __device__ __forceinline__ explicit Over(double b_) : b(b_), y(1.0 / b_) {
    ok = (b > 6.223015277861142e-61) & (b < 1.6069380442589903e60);  // 2^-200, 2^200
  }
  __device__ __forceinline__ double of(double a) const {
    const double q0 = a * y;
    const double q1 = fma(fma(-b, q0, a), y, q0);
    double q = fma(fma(-b, q1, a), y, q1);
    const unsigned e = (unsigned)(__double2hiint(a) & 0x7ff00000) - ((1023u - 700u) << 20);
    const bool zero = a == 0.0;
    q = zero ? q0 : q;
    if (!ok | ((e >= (1400u << 20)) & !zero)) q = plain_div(a, b);
    return q;
  }
};
// The same over a constant between 2^-200 and 2^200.
__device__ __forceinline__ double over(double a, double b, double y) {
  const double q0 = a * y;
  const double q1 = fma(fma(-b, q0, a), y, q0);
  double q = fma(fma(-b, q1, a), y, q1);
  const unsigned e = (unsigned)(__double2hiint(a) & 0x7ff00000) - ((1023u - 700u) << 20);
  const bool zero = a == 0.0;
  q = zero ? q0 : q;
  if ((e >= (1400u << 20)) & !zero) q = plain_div(a, b);
  return q;
}

}  // namespace fx
