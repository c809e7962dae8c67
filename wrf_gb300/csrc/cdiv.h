// Division by a constant without a divide instruction, bit-identical to IEEE
// round-to-nearest division.
//
// Method of Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE Trans.
// Computers 53(8), 2004: with zh = RN(1/c),
//     q = RN(x * zh),  r = x - q c (exact, one fma),  result = RN(q + r zh).
// Whether this returns RN(x / c) for every x depends on c; for c = 12 and
// c = 60 (the flux denominators of the advection operators) it was checked
// against IEEE division for all 2^32 single-precision inputs (tests run the
// range below 2^-96, two whole binades and a sample of the rest, which covers
// every input by scale invariance).  Nonzero inputs of magnitude
// below 2^-110, where the quotient nears the subnormal range and the remainder
// stops being exact, and infinities and NaNs take the division itself.
//
// Zeros take the fast path (a field at rest or a tracer outside its plume has
// zero differences everywhere: with the division there, the first large step
// of a horizontally uniform wind issued 20-55% more instructions in the tendency
// kernels), so the steps are arranged to keep a zero's sign: they form
// w = -(x / c) as q' = RN(x (-zh)), r = x + q' c, w = RN(q' + r (-zh)), and a
// difference of two quotients is the difference of two such w.
//
// Shared by the kernels (nvcc) and the host-side check (gcc, with
// -ffp-contract=off so that x * zh is not fused).
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define WRFGPU_HD __host__ __device__ __forceinline__
#else
#define WRFGPU_HD static inline
#endif

/* 2 |x|'s bits - 1: the largest value for a zero, else ordered as |x|.  At
 * least WRFGPU_DIV_MIN: x is zero or not below 2^-110 in magnitude. */
#define WRFGPU_DIV_MIN 0x10FFFFFFu
WRFGPU_HD uint32_t wrfgpu_div_key(float x) {
#if defined(__CUDA_ARCH__)
  return 2u * __float_as_uint(x) - 1u;
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return 2u * u - 1u;
#endif
}
/* -(x / c), nz = -RN(1/c) */
WRFGPU_HD float wrfgpu_div_neg(float x, float c, float nz) {
  const float q = x * nz;
  return fmaf(fmaf(q, c, x), nz, q);
}

WRFGPU_HD float wrfgpu_div_const(float x, float c, float zh) {
  const float w = wrfgpu_div_neg(x, c, -zh);
  if (!(wrfgpu_div_key(x) >= WRFGPU_DIV_MIN && fabsf(w) <= 3.40282347e38f)) return x / c;
  return -w;
}

WRFGPU_HD float wrfgpu_div12(float x) { return wrfgpu_div_const(x, 12.0f, 1.0f / 12.0f); }
WRFGPU_HD float wrfgpu_div60(float x) { return wrfgpu_div_const(x, 60.0f, 1.0f / 60.0f); }

/* x / c - y / c with both quotients rounded as IEEE division, one test for the
 * pair: the fast path is taken when neither numerator is a nonzero below
 * 2^-110 and the result is finite (an infinite or NaN numerator makes it a
 * NaN).  The 5th- and 3rd-order fluxes each divide two numerators by the
 * same constant. */
WRFGPU_HD float wrfgpu_div_const_sub(float x, float y, float c, float zh) {
  const uint32_t kx = wrfgpu_div_key(x), ky = wrfgpu_div_key(y);
  const float z = wrfgpu_div_neg(y, c, -zh) - wrfgpu_div_neg(x, c, -zh);
  if (!((kx < ky ? kx : ky) >= WRFGPU_DIV_MIN && fabsf(z) <= 3.40282347e38f)) return x / c - y / c;
  return z;
}
/* x / 12 + y / 12 = x / 12 - (-y) / 12 */
WRFGPU_HD float wrfgpu_div12_add(float x, float y) { return wrfgpu_div_const_sub(x, -y, 12.0f, 1.0f / 12.0f); }
WRFGPU_HD float wrfgpu_div60_sub(float x, float y) { return wrfgpu_div_const_sub(x, y, 60.0f, 1.0f / 60.0f); }
