// f3d_fused_math.cuh -- device arithmetic of the precision form's step kernel
// (f3d_fused2.cu).
//
// The formulas are the reference's (sizloop's routines, cited at each
// function) in binary32, in the form that needs the fewest operations per
// cell: everything that does not depend on the class or on the step is part
// of a coefficient, formed in binary64 at the meteo update and rounded once
// (launch_step_fields), and the two upwind differences of a cell are taken
// from one flux per face.  Contractions are explicit (fused multiply-adds;
// the unit is built with --fmad=false), every kernel variant calls these
// functions on the same values, so all of them give the same bits for the
// same cell.
#pragma once

#include <type_traits>

#include "f3d_fused.h"

namespace f3d {
namespace fz {

constexpr unsigned FULL = 0xffffffffu;

// MAX(0,x), MIN(0,x); 0 for a NaN
__device__ __forceinline__ float clip0(float x) { return fmaxf(x, 0.0f); }
__device__ __forceinline__ float2 max0(float2 v) { return make_float2(fmaxf(v.x, 0.0f), fmaxf(v.y, 0.0f)); }
__device__ __forceinline__ float2 min0(float2 v) { return make_float2(fminf(v.x, 0.0f), fminf(v.y, 0.0f)); }

__device__ __forceinline__ float shup(float v) { return __shfl_up_sync(FULL, v, 1); }
__device__ __forceinline__ float shdn(float v) { return __shfl_down_sync(FULL, v, 1); }

// Pairs of binary32 values, the two columns of a lane: the packed f32x2
// instructions, one issue slot for both columns.  A difference is the fused
// multiply-add b*(-1) + a (exactly RN(a - b)): the packed subtraction itself
// was measured to be contracted with a product it follows, which the packed
// addition, product and multiply-add are not.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, splat(-1.0f), a); }
__device__ __forceinline__ float2 abs2(float2 v) { return make_float2(fabsf(v.x), fabsf(v.y)); }
__device__ __forceinline__ float2 sel2(bool cx, bool cy, float2 a, float2 b) {
  return make_float2(cx ? a.x : b.x, cy ? a.y : b.y);
}

// The limiter 0.5*(SIGN(1,r)+SIGN(1,l))*MIN(|r|,|l|) of advctx.f90:34-40:
// the common minimum with the product of the signs, clamped at 0 (opposite
// signs), with the sign of r.
__device__ __forceinline__ float minmod(float r, float l) {
  float m;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(m) : "f"(r), "f"(l));
  return __uint_as_float(__float_as_uint(fmaxf(m, 0.0f)) | (__float_as_uint(r) & 0x80000000u));
}
__device__ __forceinline__ float2 minmod2(float2 r, float2 l) { return make_float2(minmod(r.x, l.x), minmod(r.y, l.y)); }

// The limiter's coefficient in work(k,2) of advctzc.f90:36-44 with this
// level's factors (ZTab::a, b) and s = |vk + vk_1|: s*(a - b*s).
__device__ __forceinline__ float2 lim_coef_z(float2 vk, float2 vk_1, float za, float zb) {
  const float2 s = abs2(add2(vk, vk_1));
  return mul2(s, fma2(s, splat(-zb), splat(za)));
}

// The upwind side's difference (advctx.f90:48-54): the face flux below the
// cell for a positive velocity, the one above otherwise.
__device__ __forceinline__ float2 upwind(float2 c, float2 v, float2 g, float2 gp) {
  return sub2(c, make_float2(v.x > 0.0f ? g.x : gp.x, v.y > 0.0f ? g.y : gp.y));
}

// Staged fields of iteration t (plane index in parentheses): c(t+2),
// vz+vset(t+1), the Courant velocities and limiter coefficients of x and y and
// 1/rho (t), and the diffusion's face coefficients (t-1).
enum : int { F_C = 0, F_VK, F_UX, F_KX, F_UY, F_KY, F_L, F_FZ, F_FX, F_FY, NF };
// their plane in iteration t, minus t
__host__ __device__ constexpr int field_plane(int f) { return f == F_C ? 2 : f == F_VK ? 1 : f >= F_FZ ? -1 : 0; }

using False_ = std::integral_constant<bool, false>;
using True_ = std::integral_constant<bool, true>;

}  // namespace fz
}  // namespace f3d
