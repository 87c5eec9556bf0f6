// Division of many values by one, and a reciprocal from an approximate one.
#pragma once
#include <math.h>

namespace b200 {

// a / b rounded to nearest, with r = 1 / b rounded to nearest: a product, its remainder and one correction, "division when the
// divisor is known in advance" (Brisebarre, Muller, Raina, IEEE Transactions on Computers 53(8), 2004; that the correction ends at the
// correctly rounded quotient is Markstein's theorem, IBM Journal of Research and Development 34(1), 1990).  For b >= 1: the same
// bits as a division while |a| >= 2^-100 (below, the remainder is a subnormal number: an ulp, at least 2^-149, at most); zero loses its
// sign; infinities and NaN of a stay what they are (the remainder is a NaN then).
__host__ __device__ __forceinline__ float quotient(float a, float b, float r) {
  const float q = a * r, e = fmaf(-b, q, a);
  return e == e ? fmaf(e, r, q) : q;
}

// A step of the Newton-Raphson iteration for 1 / b from r, an approximation of it: r + r (1 - b r).  The relative error e of r becomes
// e^2 and the two roundings: from one of 2^-22 the result is within an ulp, and so is a product with it within an ulp and a half.
__host__ __device__ __forceinline__ float newton_reciprocal(float b, float r) { return fmaf(r, fmaf(-b, r, 1.0f), r); }

} // namespace b200
