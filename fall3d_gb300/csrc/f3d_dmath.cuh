// f3d_dmath.cuh -- binary64 functions in few operations: those of the
// settling-velocity iteration (vsettl), whose cost on GB300 is the number of
// binary64 operations per drag iteration (further down), and a table-driven
// logarithm and exponential, which only the diagnostic f3d_dmath_eval reaches.
//
// Methods of the latter (published):
//  * exp: P. T. P. Tang, "Table-driven implementation of the exponential
//    function in IEEE floating-point arithmetic", ACM TOMS 15(2), 1989.
//    a = (64 m + j) ln2/64 + r with |r| <= ln2/128, exp(a) = 2^m 2^(j/64) e^r,
//    2^(j/64) from a 64-entry table, e^r - 1 by its Taylor series to r^6.
//  * log: P. T. P. Tang, "Table-driven implementation of the logarithm
//    function in IEEE floating-point arithmetic", ACM TOMS 16(4), 1990.
//    x = 2^k z, z in [1, 2); the top seven fraction bits of z pick the
//    breakpoint c = 1 + (j + 1/2)/128, r = z/c - 1 (one fused multiply-add
//    with the tabulated reciprocal), |r| <= 2^-8, and
//    log x = k ln2 - log(1/c) + log1p(r), log1p by its Taylor series to r^7.
//
// Accuracy of these: the truncated series are below 2^-64; the results are
// within a few units in the last place (the tests bound both against a
// high-precision evaluation).  Arguments outside the reduced ranges (log of
// a non-normal or huge value, exp beyond +-700) fall back to CUDA's log/exp.
#pragma once

#include "f3d_common.cuh"

namespace f3d {

struct DMathTab {
  double invc[128];  // RN(1 / (1 + (j + 1/2)/128))
  double logc[128];  // RN(-log(invc[j]))
  double e2[64];     // RN(2^(j/64))
};

// Fills the tables with all threads of the block (the caller synchronises).
__device__ __forceinline__ void dmath_tab_init(DMathTab& t) {
  for (int j = threadIdx.x; j < 128; j += blockDim.x) {
    const double ic = 1.0 / (1.0 + (j + 0.5) / 128.0);
    t.invc[j] = ic;
    t.logc[j] = -log(ic);
  }
  for (int j = threadIdx.x; j < 64; j += blockDim.x) t.e2[j] = exp2(j / 64.0);
}

__device__ __forceinline__ double dm_log(const DMathTab& t, double x) {
  const long long ix = dbits(x);
  // 2^-1000 <= x <= 2^1000 (positive, normal, finite), as one unsigned compare
  if ((unsigned long long)(ix - 0x0170000000000000LL) > 0x7d00000000000000ULL) return log(x);
  const int k = (int)(ix >> 52) - 1023;
  const int j = (int)((ix >> 45) & 127);
  const double z = bitsd((ix & 0x000FFFFFFFFFFFFFLL) | 0x3FF0000000000000LL);
  const double r = fma(z, t.invc[j], -1.0);
  double q = fma(r, 1.0 / 7.0, -1.0 / 6.0);
  q = fma(q, r, 1.0 / 5.0);
  q = fma(q, r, -1.0 / 4.0);
  q = fma(q, r, 1.0 / 3.0);
  q = fma(q, r, -1.0 / 2.0);
  const double p = fma(q, r * r, r);  // log1p(r)
  const double kd = (double)k;
  const double hi = fma(kd, 0x1.62e42fefa3800p-1, t.logc[j]);  // kd * ln2_hi is exact
  const double lo = fma(kd, 0x1.ef35793c76730p-45, p);
  return hi + lo;
}

__device__ __forceinline__ double dm_exp(const DMathTab& t, double a) {
  // |a| <= 700 (NaN excluded), as one integer compare on the magnitude bits
  if ((dbits(a) & 0x7fffffffffffffffLL) > 0x4085e00000000000LL) return exp(a);
  const double shift = 0x1.8p52;                        // rounds a*64/ln2 to an integer
  const double kd = fma(a, 0x1.71547652b82fep+6, shift);
  const long long n = dbits(kd) - dbits(shift);
  const double kn = kd - shift;
  double r = fma(kn, -0x1.62e42fefa0000p-7, a);        // kn * (ln2/64)_hi is exact
  r = fma(kn, -0x1.cf79abc9e3b3ap-46, r);
  double q = fma(r, 1.0 / 720.0, 1.0 / 120.0);
  q = fma(q, r, 1.0 / 24.0);
  q = fma(q, r, 1.0 / 6.0);
  q = fma(q, r, 0.5);
  const double em1 = fma(q, r * r, r);  // e^r - 1
  const long long m52 = (long long)((unsigned long long)(n >> 6) << 52);  // 2^m in the exponent field
  const double s = bitsd(dbits(t.e2[n & 63]) + m52);
  return fma(s, em1, s);
}

// ---------------------------------------------------------------- Ganser
// The three functions of a Ganser drag iteration in as few binary64
// operations as their accuracy (about an ulp) allows, for arguments in the
// normal range the callers check.

// x^a, a = 0.6567 - 1: with x = 2^k z, z in [1, 2), and the breakpoint c of
// the top eight fraction bits of z, x^a = 2^(ka) c^a (1 + r)^a, r = z/c - 1,
// |r| <= 2^-9: two table values and the binomial series to r^5 (the next term
// is below 2^-57), 8 operations in place of the 23 of a logarithm and an
// exponential.  Within 8.2 * 2^-53 of the value: the tables' 2 and 1 ulp, their
// product and the last rounding.  (The power of two's exponent a*k is rounded,
// by up to 2^-49 at the ends of the range, which the table corrects: without
// that the error was 12.9 * 2^-53.)
constexpr double kPowA = 0.6567 - 1.0;
constexpr int kPowEmin = -64, kPowN = 128;  // exponents k of the table
struct PowTab {
  double invc[256];   // RN(1 / (1 + (j + 1/2)/256))
  double powc[256];   // invc[j]^-a
  double pow2[kPowN]; // 2^(a (kPowEmin + j))
};
__device__ __forceinline__ void pow_tab_init(PowTab& t) {
  for (int j = threadIdx.x; j < 256; j += blockDim.x) {
    const double ic = 1.0 / (1.0 + (j + 0.5) / 256.0);
    t.invc[j] = ic;
    t.powc[j] = pow(ic, -kPowA);
  }
  for (int j = threadIdx.x; j < kPowN; j += blockDim.x) {
    const double k = kPowEmin + j, p = kPowA * k, l = fma(kPowA, k, -p);  // a*k = p + l
    const double e = exp2(p);
    t.pow2[j] = fma(e, l * 0.6931471805599453, e);  // 2^l = 1 + l ln 2, l below 2^-49
  }
}
// the biased exponent lies in the table's range
__device__ __forceinline__ bool pow_in_range(double x) {
  return (unsigned)((__double2hiint(x) >> 20) - (1023 + kPowEmin)) < (unsigned)kPowN;
}
__device__ __forceinline__ double pow_a(const PowTab& t, double x) {
  const int hi = __double2hiint(x);
  const int j = (hi >> 12) & 255;
  const double z = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
  const double s = t.pow2[(hi >> 20) - (1023 + kPowEmin)] * t.powc[j];
  const double r = fma(z, t.invc[j], -1.0);
  constexpr double a = kPowA, c1 = a, c2 = c1 * (a - 1.0) / 2.0, c3 = c2 * (a - 2.0) / 3.0, c4 = c3 * (a - 3.0) / 4.0,
                   c5 = c4 * (a - 4.0) / 5.0;
  double q = fma(r, c5, c4);
  q = fma(q, r, c3);
  q = fma(q, r, c2);
  q = fma(q, r, c1);
  return fma(s * r, q, s);
}

// 1/sqrt(x) and 1/x, x in [2^-1000, 2^1000], from the hardware's approximations
// y by one step of Chebyshev's method (J. F. Traub, Iterative Methods for the
// Solution of Equations, 1964), y - f/f' (1 + f f''/(2 f'^2)), of third order:
//   f(y) = 1/y - x,   e = 1 - x y:    y (1 + e + e^2);
//   f(y) = 1/y^2 - x, h = 1 - x y^2:  y (1 + h/2 + 3/8 h^2).
// With a relative error d of y, the first leaves d^3 and the second, the next term
// of the series of (1 - h)^(-1/2) being 5/16 h^3 at h = 2 d, 5/2 d^3.  d measured over
// 1.3e9 arguments in [1, 4): 2^-19.94 and 2^-20.04; so 2^-59.8 and 2^-58.8, beside
// the roundings of the last operations (1.02 and 1.6 times 2^-53 in all).
__device__ __forceinline__ double rsqrt_fast(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = fma(-(x * y), y, 1.0);
  return fma(y * h, fma(0.375, h, 0.5), y);
}
__device__ __forceinline__ double rcp_fast(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

}  // namespace f3d
