// f3d_common.cuh -- device helpers shared by the transport kernels.
//
// Semantics that the reference leaves to the Fortran processor are fixed
// here exactly as in the CPU oracle:
//  * MAX/MIN follow gfortran 4.8 (the compiler of the reference build):
//    mvar = a; if (b .op. mvar .or. isnan(mvar)) mvar = b.  They return the
//    non-NaN operand and keep the first operand on ties (so MAX(0,-0) = +0).
//  * SIGN(1,b) is copysign(1,b), with a NaN b counted as positive (the CUDA
//    and aarch64 default NaN is positive).
// The binary64 kernels are compiled with --fmad=false so that every
// expression is rounded operation by operation, as the Fortran is.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#define F3D_HD __host__ __device__ __forceinline__

template <class T>
F3D_HD T fmax2(T a, T b) { return (b > a || isnan(a)) ? b : a; }
template <class T>
F3D_HD T fmin2(T a, T b) { return (b < a || isnan(a)) ? b : a; }
template <class T>
F3D_HD T sign1(T b) { return isnan(b) ? T(1) : (signbit(b) ? T(-1) : T(1)); }

// A binary64 value's bit pattern and back, by moves that the compiler does
// not look through: it turns integer operations on the pattern that it
// recognises (a cleared sign bit, a comparison with zero's pattern) back into
// binary64 instructions, which issue at 1/32 of the integer rate.  The plain
// form's vertical sweep of 400x300x20 cells and 4 classes issued 28.1 of them
// per cell with the plain reinterpretation.
__device__ __forceinline__ long long dbits(double x) {
  long long r;
  asm("mov.b64 %0, %1;" : "=l"(r) : "d"(x));
  return r;
}
__device__ __forceinline__ double bitsd(long long b) {
  double r;
  asm("mov.b64 %0, %1;" : "=d"(r) : "l"(b));
  return r;
}

// A binary32 value widened with integer operations (the conversion
// instruction goes through the binary64 pipe, which the kernels of
// binary64 sums are bound by); exponent 0 and 255 take the conversion.
__device__ __forceinline__ double widen(float v) {
  const unsigned u = __float_as_uint(v), e = (u >> 23) & 255u;
  if (e - 1u >= 254u) return (double)v;
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}
__device__ __forceinline__ double widen(double v) { return v; }

// |x| and x > 0 of binary64 values on the bit patterns (integer operations;
// the binary64 pipe is the plain form's bottleneck): clearing the sign bit
// is fabs, NaN included; x > 0 holds exactly for the patterns of positive
// finite values and +inf, 1 .. 0x7ff0000000000000 as signed integers.
__device__ __forceinline__ double absd(double x) { return bitsd(dbits(x) & 0x7fffffffffffffffLL); }
__device__ __forceinline__ float absd(float x) { return fabsf(x); }
__device__ __forceinline__ bool gt0(double x) {
  const long long b = dbits(x);
  return b > 0 && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool gt0(float x) { return x > 0.0f; }

// MAX(0,x) and MIN(0,x) (+0 for a zero or a NaN) by selection on the bit
// pattern: no binary64 comparison and no branch.  A branch in a column march's
// first iteration left its warps split to the end of the column.
__device__ __forceinline__ double max0(double x) { return bitsd(gt0(x) ? dbits(x) : 0LL); }
__device__ __forceinline__ double min0(double x) {
  const long long b = dbits(x);
  return bitsd(b < 0 && (unsigned long long)b <= 0xfff0000000000000ULL && (b << 1) != 0 ? b : 0LL);
}
__device__ __forceinline__ float max0(float x) { return x > 0.0f ? x : 0.0f; }
__device__ __forceinline__ float min0(float x) { return x < 0.0f ? x : 0.0f; }

// 0.5*x: the exponent one less (integer operations), the product where that
// is not a normal number.
static __device__ __noinline__ double half_product(double x) { return 0.5 * x; }
__device__ __forceinline__ double half_of(double x) {
  const long long b = dbits(x);
  if (((unsigned)(b >> 32) & 0x7fffffffu) - 0x00200000u >= 0x7fd00000u) return half_product(x);
  return bitsd(b - (1LL << 52));
}
__device__ __forceinline__ float half_of(float x) { return 0.5f * x; }

// RN(a/b) from y = RN(1/b) with a single binary64 operation.  GB300 issues
// two lanes of binary64 per SM and clock against 64 of integer, so the
// quotient q0 = RN(a*y), which is within 1.5 ulp of a/b, is corrected in
// integers: with the significands A, B, Q (53-bit integers) and
// a - q0*b = 2^e * (A*2^s - Q*B), R = A*2^s - Q*B is below 1.5*B in magnitude,
// so 64-bit arithmetic modulo 2^64 gives it exactly, and q0 is the nearest
// value when |R| <= B/2, else its neighbour is (a quotient of two such values
// is never half-way between two).  Adding +-1 to the bit pattern of q0 is that
// neighbour unless q0 is a power of two, below which the spacing halves.
// A zero a gives a*y (the signed zero of a/b).  A q0 that is a power of two,
// subnormal or non-finite operands and results, and a b whose reciprocal may
// not be normal take the IEEE division: the result is RN(a/b) for all inputs.
// (Markstein's correction by four multiply-adds before this: the plain form's
// x sweep of 400x300x50 cells and 16 classes 4.08 ms, now 3.42 ms.  The range
// matters where a plume's tail falls off to zero: with operands below 2^-900
// left to the division, the diffusion sweep in z of 400x300x20 cells and 4
// classes issued 13.7 binary64 instructions per cell.)
// the rare paths out of line, so that they cost the callers no registers
static __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }
static __device__ __noinline__ double minmod_div_ieee(double a, double b, double dx) {
  const double dr = a / dx, dl = b / dx;
  return 0.5 * (sign1(dr) + sign1(dl)) * fmin2(fabs(dr), fabs(dl));
}
__device__ __forceinline__ unsigned mag_hi(double x) { return (unsigned)(dbits(x) >> 32) & 0x7fffffffu; }
// a normal number; 2^-1000 <= |x| < 2^1000 (its reciprocal is normal as well)
__device__ __forceinline__ bool is_normal(double x) { return mag_hi(x) - 0x00100000u < 0x7fe00000u; }
__device__ __forceinline__ bool div_in_range(double x) { return mag_hi(x) - 0x01700000u < 0x7d000000u; }
__device__ __forceinline__ double div_rn_recip(double a, double b, double y) {
  const double q0 = a * y;
  const long long ba = dbits(a), bb = dbits(b), bq = dbits(q0);
  const unsigned long long one = 1ULL << 52, mask = one - 1;
  const bool zero = (ba & 0x7fffffffffffffffLL) == 0;
  // y may be inexact, infinite or zero for a b out of range; one rare branch
  if (!div_in_range(b) || (!zero && (!is_normal(a) || !is_normal(q0) || (bq & mask) == 0)))
    return div_ieee(a, b);
  const unsigned long long B = (bb & mask) | one;
  const int s = (int)((ba >> 52) & 2047) - (int)((bb >> 52) & 2047) - (int)((bq >> 52) & 2047) + 1075;
  const long long R = (long long)((((ba & mask) | one) << (s & 63)) - ((bq & mask) | one) * B);
  const long long h = (long long)(B >> 1);
  return bitsd(zero ? bq : bq + (R > h ? 1 : 0) - (R < -h ? 1 : 0));
}

// The slope limiter of advctx.f90:34-40 (and advcty), with
// deltar = a/dx, deltal = b/dx:
//   sigma = 0.5*(SIGN(1,deltar)+SIGN(1,deltal))*MIN(|deltar|,|deltal|).
// For dx > 0, x -> RN(x/dx) is monotonic and keeps the sign of x (zeros and
// underflows included), so SIGN(1,RN(a/dx)) = SIGN(1,a) and
// MIN(|RN(a/dx)|,|RN(b/dx)|) = RN(m/dx) with m = MIN(|a|,|b|) under the same
// MIN rule (NaN operands included): one division instead of two, the same
// bits.  Other dx take the reference's two divisions.
template <class T>
__device__ __forceinline__ T minmod_div(T a, T b, T dx, T rdx) {
  (void)rdx;
  if (!(dx > T(0))) {
    const T dr = a / dx, dl = b / dx;
    return T(0.5) * (sign1(dr) + sign1(dl)) * fmin2(absd(dr), absd(dl));
  }
  return T(0.5) * (sign1(a) + sign1(b)) * (fmin2(absd(a), absd(b)) / dx);
}

// The limiter 0.5*(SIGN(1,dr)+SIGN(1,dl))*MIN(|dr|,|dl|) (advctzc.f90:44).
template <class T>
__device__ __forceinline__ T minmod_ref(T dr, T dl) {
  return T(0.5) * (sign1(dr) + sign1(dl)) * fmin2(absd(dr), absd(dl));
}

// binary64 forms of both limiters on the bit patterns.  GB300 issues
// binary64 arithmetic at 1/64 of the binary32 rate while integer operations
// run at full rate, so the sign and minimum logic moves to integers.  For
// finite operands (the others take the formula):
//  * 0.5*(s_r + s_l) is +-1 when the sign bits agree (SIGN(1,-0) = -1), and
//    +0 when they differ, where +0 * (a finite m >= 0) = +0;
//  * |x| of finite binary64 values orders like the integers of their bit
//    patterns with the sign cleared, and MIN keeps the first operand on
//    ties, which has the same bits as the second;
//  * (+-1) * m is m with the sign bit of the first operand.
// The results are the formula's bits.
__device__ __forceinline__ double minmod_ref(double dr, double dl) {
  const long long br = dbits(dr), bl = dbits(dl);
  const long long mr = br & 0x7fffffffffffffffLL, ml = bl & 0x7fffffffffffffffLL;
  if (mr >= 0x7ff0000000000000LL || ml >= 0x7ff0000000000000LL)
    return 0.5 * (sign1(dr) + sign1(dl)) * fmin2(fabs(dr), fabs(dl));
  // one selected pattern: a branch would duplicate what follows it
  return bitsd((br ^ bl) < 0 ? 0LL : (ml < mr ? ml : mr) | (br & (long long)0x8000000000000000ULL));
}
// rdx = RN(1/dx): the division by dx goes through div_rn_recip.
__device__ __forceinline__ double minmod_div(double a, double b, double dx, double rdx) {
  const long long ba = dbits(a), bb = dbits(b);
  const long long ma = ba & 0x7fffffffffffffffLL, mb = bb & 0x7fffffffffffffffLL;
  if (!gt0(dx) || ma >= 0x7ff0000000000000LL || mb >= 0x7ff0000000000000LL)
    return minmod_div_ieee(a, b, dx);
  const double q = div_rn_recip(bitsd(mb < ma ? mb : ma), dx, rdx);  // >= 0, +inf on overflow
  const long long bq = dbits(q);
  if (bq == 0x7ff0000000000000LL) return minmod_div_ieee(a, b, dx);  // 0 * inf for opposite signs
  return bitsd((ba ^ bb) < 0 ? 0LL : bq | (ba & (long long)0x8000000000000000ULL));
}

// Grid geometry of one scenario (interior nx, ny, nz; halo arrays are rows of
// px values, (ny+2)(nz+2) rows, x fastest).  The row pitch px is nx+2, or for
// the precision form's state nx+2 rounded up to a multiple of 4 values, so
// that tensor copies (16-byte row strides) can stage it; the padding stays 0.
struct Dims {
  int nx, ny, nz, px;
  Dims() = default;
  F3D_HD Dims(int nx_, int ny_, int nz_) : nx(nx_), ny(ny_), nz(nz_), px(nx_ + 2) {}
  F3D_HD Dims(int nx_, int ny_, int nz_, int px_) : nx(nx_), ny(ny_), nz(nz_), px(px_) {}
  F3D_HD long long C(int i, int j, int k) const {
    return (long long)i + (long long)px * ((long long)j + (long long)(ny + 2) * k);
  }
  F3D_HD long long M(int i, int j, int k) const {
    return (long long)(i - 1) + (long long)nx * ((long long)(j - 1) + (long long)ny * (k - 1));
  }
  F3D_HD long long P(int i, int j) const { return (long long)(i - 1) + (long long)nx * (j - 1); }
  F3D_HD long long halo() const { return (long long)px * (ny + 2) * (nz + 2); }
  F3D_HD long long cells() const { return (long long)nx * ny * nz; }
  F3D_HD long long plane() const { return (long long)nx * ny; }
};

// Double-double accumulator (Knuth TwoSum): sums that are exact to well
// below one binary64 ulp, and independent of the reduction order up to the
// final rounding.  Used for the mass budgets.
struct DD {
  double hi, lo;
};
F3D_HD DD dd_zero() { return DD{0.0, 0.0}; }
F3D_HD DD dd_add_d(DD a, double b) {
  double s = a.hi + b;
  double bb = s - a.hi;
  double err = (a.hi - (s - bb)) + (b - bb);
  double lo = a.lo + err;
  double hi = s + lo;
  lo = lo - (hi - s);
  return DD{hi, lo};
}
