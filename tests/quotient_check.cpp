// The division by a value known in advance (quotient.cuh) against the machine's, which rounds to nearest: the arithmetic of both is
// IEEE's, so what holds here holds on the GPU, whose reciprocal (__frcp_rn), product and fmaf round the same way.
#define __host__
#define __device__
#define __forceinline__ inline
#include "../buddy_mlir_b200/csrc/quotient.cuh"

#include <cstdint>
#include <cstring>

static float bits(uint32_t u) {
  float f;
  memcpy(&f, &u, 4);
  return f;
}
static uint32_t of(float f) {
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
}

extern "C" {

// Quotients that differ, over all 2^23 significands of a at one exponent, for each of n divisors.
long all_significands(const float *b, int n) {
  long wrong = 0;
  for (int j = 0; j < n; ++j) {
    const float d = b[j], r = 1.0f / d;
    for (uint32_t m = 0; m < 1u << 23; ++m) {
      const float a = bits(0x3f800000u | m);
      wrong += of(b200::quotient(a, d, r)) != of(a / d);
    }
  }
  return wrong;
}

void pairs(const float *a, const float *b, float *out, float *want, long n) {
  for (long i = 0; i < n; ++i) {
    out[i] = b200::quotient(a[i], b[i], 1.0f / b[i]);
    want[i] = a[i] / b[i];
  }
}

// Quotients a * newton_reciprocal(b, r) with r = 1 / b rounded and moved by `ulps`: what an approximate reciprocal may give.
void newton(const float *a, const float *b, float *out, long n, int ulps) {
  for (long i = 0; i < n; ++i)
    out[i] = a[i] * b200::newton_reciprocal(b[i], bits(of(1.0f / b[i]) + ulps));
}

}
