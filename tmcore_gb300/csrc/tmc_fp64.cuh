// FP64 arithmetic that keeps off the FP64 pipe.
//
// GB300 executes FP64 at 2 lanes per clock and SM: one warp-wide FP64
// instruction occupies its sub-partition's pipe for 64 cycles, an integer or
// FP32 instruction for one.  The FP64 kernels are bound by that pipe (80-85%
// busy with DRAM at 11-13% of peak), so here everything that an exponent or a
// sign bit can express is done on the integer units, and quotients by a
// divisor whose reciprocal is at hand cost three FP64 instructions.  Results
// are those of IEEE division, square root and multiplication bit for bit; the
// reasons stand at div_r and sqrt_r.
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

// sign * x for a sign of +1, -1 or 0 (an element that lists an edge which is not
// its own)
__device__ __forceinline__ double with_sign(double x, int sign) {
  const int mask = -(sign & 1);
  return __hiloint2double((__double2hiint(x) ^ (sign & 0x80000000)) & mask, __double2loint(x) & mask);
}

// a / b rounded to nearest from r = RN(1/b), or from r = 0 (which makes it
// divide): quotient estimate q, its residual by FMA, one correction (Markstein
// 1990; Brisebarre, Muller and Raina 2004 for a divisor known in advance).
// Why, in units in the last place of q: with the mantissas of b and r as
// integers B and R, B R = 2^105 + h with |h| <= B/2 (h = 0 for a power of two).
// The corrected value, before its rounding, is off a/b by |a/b - q| |h| / 2^105,
// at most 1.5 2^-53.  a/b itself is a midpoint plus N / (2 B), N a nonzero
// integer, so only |N| <= 2 could round the wrong way.  So near a midpoint q is
// one of its two neighbours, |a/b - q| is a half, and the deviation at most
// B/4 2^-105 < 1 / (2 B) stays on the quotient's side.
// That needs r correctly rounded: with the reciprocal one unit off, 1 / (2 -
// 2^-52) comes out one unit off.  Outside the range where the residual is
// exact (zeros, infinities, NaN, extreme exponents) the plain division.
__device__ __forceinline__ double div_r(double a, double b, double r) {
  const double q = __dmul_rn(a, r);
  if (mid(q)) return __fma_rn(__fma_rn(-q, b, a), r, q);
  return a / b;
}

// y if it is 1/b rounded to nearest, else 0, for y within a few units of 1/b.
// A Newton iteration ends within 2^-80 of 1/b before its rounding and so may
// round the other way where 1/b is next to a midpoint.  With the mantissas as
// integers the product's distance from the power of two is its low 64 bits:
// 14 integer instructions, where a residual in FP64 would hold the pipe for 64
// cycles.  (Where y is a power of two and b is not, the distance is 2^52 or
// more, above B/2: the closer spacing below y needs no case.)
__device__ __forceinline__ double nearest_or_zero(double b, double y) {
  auto mantissa = [](double x) {
    return (unsigned long long)(unsigned)((__double2hiint(x) & 0xfffff) | 0x100000) << 32 |
           (unsigned)__double2loint(x);
  };
  const unsigned long long B = mantissa(b);
  const long long h = (long long)(B * mantissa(y));
  return 2 * (unsigned long long)(h < 0 ? -h : h) <= B ? y : 0.0;
}

// 1/b rounded to nearest for div_r, or 0: Newton iterations from the 20-bit
// hardware estimate
__device__ __forceinline__ double recip(double b) {
  if (!mid(b)) return 0.0;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = __fma_rn(__fma_rn(-b, y, 1.0), y, y);
  return nearest_or_zero(b, __fma_rn(__fma_rn(-b, y, 1.0), y, y));
}

// s = sqrt(a) rounded to nearest and r = 1/s rounded to nearest, or 0 (for
// div_r): coupled iteration (Goldschmidt 1964) from the hardware's reciprocal
// square root estimate, g -> sqrt(a), h -> 1/(2 sqrt(a)), and one residual
// correction of g (Markstein 1990).  g and h end within 2^-52 (relative), so
// the corrected root is within 2^-50 units in the last place of sqrt(a) before
// its rounding.  A root that near a midpoint m (54 bits) has a 2^s = m^2 - c
// with |c| <= 64: some 25 mantissas, for which (and for 150 more) equality
// with the IEEE square root is tested.
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
  return {s, nearest_or_zero(s, __fma_rn(__fma_rn(-s, y, 1.0), y, y))};
}

// ---------------------------------------------------------------------------
// sums across lanes in integers: every term is aligned to the largest
// exponent as a 128-bit integer (53 bits of mantissa, 64 bits below them,
// further bits dropped), the integers are added exactly and the sum is rounded
// once.  A warp sum costs about a hundred integer instructions and twenty for
// each further term of a lane; the five additions of an FP64 shuffle tree
// occupy the FP64 pipe for 320 cycles, a double-double tree's for 6,400.
// ---------------------------------------------------------------------------
struct Fixed {
  __int128 m;  // the sum is m 2^(e - 1139)
  int e;       // largest biased exponent of the terms; < 0: m holds the bits of an FP64 tree sum
};
struct HiLo {
  double hi, lo;
};

__device__ __forceinline__ double from_fixed(bool neg, unsigned __int128 u, int e, unsigned __int128* rest) {
  const unsigned long long uh = (unsigned long long)(u >> 64), ul = (unsigned long long)u;
  const int n = uh ? 128 - __clzll(uh) : 64 - __clzll(ul);  // bits of u (u != 0)
  unsigned long long bits;
  const int E = n + e - 117;  // biased exponent of the leading bit
  if (n <= 53) {
    bits = ul << (53 - n);
    *rest = 0;
  } else {
    const int sh = n - 53;
    bits = (unsigned long long)(u >> sh);
    *rest = u - ((unsigned __int128)bits << sh);  // truncated here; lo takes the rest
  }
  bits += (unsigned long long)(E - 1) << 52;
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}
// the sum as hi + lo with lo of hi's sign, to 2^-106 of hi
__device__ __forceinline__ HiLo split(const Fixed& f) {
  if (f.e < 0) return {__longlong_as_double((long long)f.m), 0.0};
  const bool neg = f.m < 0;
  unsigned __int128 u = neg ? (unsigned __int128)0 - (unsigned __int128)f.m : (unsigned __int128)f.m, rest = 0;
  if (u == 0) return {0.0, 0.0};
  const double hi = from_fixed(neg, u, f.e, &rest);
  if (rest == 0) return {hi, 0.0};
  return {hi, from_fixed(neg, rest, f.e, &u)};
}
__device__ __forceinline__ double value(const Fixed& f) {
  const HiLo v = split(f);
  return v.hi + v.lo;
}

// the sum over the warp of each lane's n <= 64 terms (the limbs leave 6 bits above
// 32 terms), in every lane; all 32 lanes call, with the same n
template <int kUnroll>
__device__ __forceinline__ Fixed warp_sum(const double* v, int n) {
  const unsigned all = 0xffffffffu;
  int ex = 0;
#pragma unroll kUnroll
  for (int k = 0; k < n; ++k) ex = max(ex, (__double2hiint(v[k]) >> 20) & 0x7ff);
  const int e = (int)__reduce_max_sync(all, (unsigned)ex);
  if ((unsigned)(e - 200) > 1700u) {  // zeros, extreme exponents, infinities, NaN: in FP64
    double t = 0.0;
#pragma unroll kUnroll
    for (int k = 0; k < n; ++k) t += v[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(all, t, off);
    return {(__int128)__double_as_longlong(t), -1};
  }
  unsigned __int128 acc = 0;
#pragma unroll kUnroll
  for (int k = 0; k < n; ++k) {
    const int hi = __double2hiint(v[k]), x = (hi >> 20) & 0x7ff;
    long long m = (long long)(((unsigned long long)(unsigned)(hi & 0xfffff) << 32) | (unsigned)__double2loint(v[k]));
    if (x) m |= 1ll << 52;
    if (hi < 0) m = -m;
    const int sh = e - (x ? x : 1);
    const long long H = m >> (sh < 63 ? sh : 63);
    unsigned long long L = 0;
    if (sh >= 64)
      L = sh < 127 ? (unsigned long long)(m >> (sh - 64)) : (unsigned long long)H;
    else if (sh > 0)
      L = (unsigned long long)m << (64 - sh);
    acc += (unsigned __int128)(unsigned long long)H << 64 | L;
  }
  const long long H = (long long)(unsigned long long)(acc >> 64);
  const unsigned long long L = (unsigned long long)acc;
  const unsigned M26 = (1u << 26) - 1;
  const unsigned s0 = __reduce_add_sync(all, (unsigned)L & M26);
  const unsigned s1 = __reduce_add_sync(all, (unsigned)(L >> 26) & M26);
  const unsigned s2 = __reduce_add_sync(all, ((unsigned)(L >> 52) | (unsigned)((unsigned long long)H << 12)) & M26);
  const unsigned s3 = __reduce_add_sync(all, (unsigned)(H >> 14) & M26);
  const int s4 = (int)__reduce_add_sync(all, (unsigned)(int)(H >> 40));
  const unsigned __int128 s = (unsigned __int128)s0 + ((unsigned __int128)s1 << 26) + ((unsigned __int128)s2 << 52) +
                              ((unsigned __int128)s3 << 78) + ((unsigned __int128)(__int128)s4 << 104);
  return {(__int128)s, e};
}
template <int N>
__device__ __forceinline__ Fixed warp_sum(const double (&v)[N]) {
  return warp_sum<N>(v, N);
}
__device__ __forceinline__ Fixed warp_sum(double v) {
  const double t[1] = {v};
  return warp_sum(t);
}

}  // namespace f64
}  // namespace tmc
