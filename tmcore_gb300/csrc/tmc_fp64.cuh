// FP64 arithmetic that keeps off the FP64 pipe.
//
// GB300 executes FP64 at 2 lanes per clock and SM: one warp-wide FP64
// instruction occupies its sub-partition's pipe for 64 cycles, an integer or
// FP32 instruction for one.  The FP64 kernels are bound by that pipe (80-85%
// busy with DRAM at 11-13% of peak), so here everything that an exponent or a
// sign bit can express is done on the integer units, and quotients by a
// divisor whose reciprocal is at hand cost three FP64 instructions.  Results
// are those of IEEE division, square root and multiplication bit for bit.
#pragma once

#include <cuda_runtime.h>

namespace tmc {
namespace f64 {

// |x| in [2^-400, 2^401): products, quotients and residuals of two such
// values neither overflow nor lose bits to subnormals
__host__ __device__ __forceinline__ bool mid_exponent(int hi) {
  return (unsigned)(hi & 0x7fffffff) - (623u << 20) < (801u << 20);
}
__device__ __forceinline__ bool mid(double x) { return mid_exponent(__double2hiint(x)); }

// 1/b rounded to nearest for div_r, or 0 (which makes div_r divide) for a
// divisor outside the range its three-instruction form is proved for
__host__ inline double recip_host(double b) {
  union {
    double d;
    unsigned long long u;
  } v{b};
  return mid_exponent((int)(v.u >> 32)) ? 1.0 / b : 0.0;
}

// x / 2: the exponent field less one for normal results
__device__ __forceinline__ double half(double x) {
  const int hi = __double2hiint(x);
  if ((unsigned)((hi >> 20) & 0x7ff) - 2u < 2045u) return __hiloint2double(hi - 0x00100000, __double2loint(x));
  return 0.5 * x;
}

// sign * x for a sign of +1 or -1
__device__ __forceinline__ double with_sign(double x, int sign) {
  return __hiloint2double(__double2hiint(x) ^ (sign & 0x80000000), __double2loint(x));
}

// a / b rounded to nearest from r = RN(1/b): quotient estimate, its exact
// residual by FMA, one correction (Markstein 1990; Brisebarre, Muller and
// Raina 2004 prove the form for a divisor known in advance).  Outside the
// range where the residual is exact (zeros, infinities, NaN, extreme
// exponents) the plain division.
__device__ __forceinline__ double div_r(double a, double b, double r) {
  const double q = __dmul_rn(a, r);
  if (mid(q)) return __fma_rn(__fma_rn(-q, b, a), r, q);
  return a / b;
}

// 1/b for div_r: Newton iterations from the 20-bit hardware estimate
__device__ __forceinline__ double recip(double b) {
  if (!mid(b)) return 0.0;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  return __fma_rn(__fma_rn(-b, y, 1.0), y, y);
}

// s = sqrt(a) rounded to nearest and r = 1/s (for div_r): coupled iteration
// (Goldschmidt 1964) from the hardware's reciprocal square root estimate, g
// -> sqrt(a), h -> 1/(2 sqrt(a)), and one residual correction of g
// (Markstein 1990)
struct SqrtR {
  double s, r;
};
__device__ __forceinline__ SqrtR sqrt_r(double a) {
  if (!mid(a) || __double2hiint(a) < 0) return {sqrt(a), 0.0};
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  double g = __dmul_rn(a, y);
  double h = half(y);
  double e = __fma_rn(-g, h, 0.5);
  g = __fma_rn(g, e, g);
  h = __fma_rn(h, e, h);
  e = __fma_rn(-g, h, 0.5);
  g = __fma_rn(g, e, g);
  h = __fma_rn(h, e, h);
  const double s = __fma_rn(__fma_rn(-g, g, a), h, g);
  y = __hiloint2double(__double2hiint(h) + 0x00100000, __double2loint(h));
  return {s, __fma_rn(__fma_rn(-s, y, 1.0), y, y)};
}

}  // namespace f64
}  // namespace tmc
