// f3d_output.cu -- the output variables of Sources/printres_nc.f90 computed
// on the device, so that a results record leaves the GPU as a few (nx,ny)
// planes (binary64, or binary32 as the reference's netCDF variables are
// NF90_FLOAT, printres_nc.f90:805-841) instead of the whole state.
//
// Every variable is evaluated in binary64 in the reference's order of
// operations (--fmad=false): a sum over classes is accumulated from 0 in
// class order and divided by Hm1 afterwards, the column trapezoid runs
// upwards from the first layer, and the final unit factor multiplies the
// sum.  In the precision form the binary32 state is widened first.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "f3d_ctx_impl.h"

namespace f3d {
namespace {

constexpr int OB = 128;  // threads per block: one column (i, j) each

// The classes of an output variable (0-based) with AOT's qeff and
// rhop*reff of each, as a kernel parameter; more than CMAX go to device arrays.
constexpr int CMAX = 128;
struct OutClasses {
  int n;
  const int* cls_more;
  const double *q_more, *r_more;
  int cls[CMAX];
  double q[CMAX], r[CMAX];
  __device__ int at(int i) const { return cls_more ? cls_more[i] : cls[i]; }
};

// x != 0 with no binary64 comparison
__device__ __forceinline__ bool nonzero(float x) { return x != 0.0f; }
__device__ __forceinline__ bool nonzero(double x) { return (dbits(x) << 1) != 0; }

// sum over the listed classes of c(i,j,k,ic) (0 + c1 + c2 + ...).  A zero
// leaves the sum as it is and is skipped; eight loads are in flight.
template <class T>
__device__ __forceinline__ double class_sum(const T* c, long long hb, long long q, const OutClasses& cl) {
  double s = 0.0;
  for (int n0 = 0; n0 < cl.n; n0 += 8) {
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = n0 + u < cl.n ? c[(long long)cl.at(n0 + u) * hb + q] : T(0);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (nonzero(v[u])) s = s + widen(v[u]);
  }
  return s;
}

// one result value, in binary64 or rounded to binary32
__device__ __forceinline__ void put(void* out, long long p, double v, int f32) {
  if (f32)
    reinterpret_cast<float*>(out)[p] = (float)v;
  else
    reinterpret_cast<double*>(out)[p] = v;
}

// The column variables take blocks of 32 columns by 8 warps: the warps form
// the values of 8 levels at a time, the first warp adds their terms in the
// reference's order.  They are bound by binary64 operations (a class's
// addition and its conversion); with the conversion in integers, zeros
// skipped and the division by Hm1 through its reciprocal (div_rn_recip) the
// column mass of 400x300x50 cells and 16 classes takes 323 us instead of
// 418 us, the optical thickness 187 us instead of 400 us.
constexpr int CW = 8;

// z-cumulative concentration, g/m2 (printres_nc.f90:216-246 particles and
// gases, :281-387 PM05/PM10/PM20): w(k) = (sum over the classes)/Hm1,
// work2d = sum_{k<nz} dz(k)*0.5*(w(k)+w(k+1)), times 1e3.
template <class T>
__global__ void __launch_bounds__(32 * CW) k_out_column(const T* c, Dims d, const OutClasses cl, const double* dz,
                                                        const double* Hm1, void* out, int f32) {
  __shared__ double w[CW][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long p = blockIdx.x * 32LL + lane, pc = min(p, d.plane() - 1);
  const int i = (int)(pc % d.nx) + 1, j = (int)(pc / d.nx) + 1;
  const long long hb = d.halo();
  const double h = Hm1[pc], rh = 1.0 / h;
  double acc = 0.0, wp = 0.0;
  for (int k0 = 1; k0 <= d.nz; k0 += CW) {
    const int k = k0 + warp;
    if (k <= d.nz) w[warp][lane] = div_rn_recip(class_sum<T>(c, hb, d.C(i, j, k), cl), h, rh);
    __syncthreads();
    if (warp == 0)
      for (int u = 0; u < CW && k0 + u <= d.nz; ++u) {
        const double wn = w[u][lane];
        const double two = wp + wn;
        if (k0 + u > 1 && two != 0.0) acc = acc + dz[k0 + u - 1] * 0.5 * two;
        wp = wn;
      }
    __syncthreads();
  }
  if (warp == 0 && p < d.plane()) put(out, p, 1e3 * acc, f32);
}

// concentration at the first layer, g/m3 (printres_nc.f90:389-493):
// 1e3*(sum over the classes of c(i,j,1,ic))/Hm1.
template <class T>
__global__ void k_out_ground(const T* c, Dims d, const OutClasses cl, const double* Hm1, void* out, int f32) {
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  if (p >= d.plane()) return;
  const int i = (int)(p % d.nx) + 1, j = (int)(p / d.nx) + 1;
  const double s = class_sum<T>(c, d.halo(), d.C(i, j, 1), cl);
  put(out, p, 1e3 * s / Hm1[p], f32);
}

// aerosol optical thickness (printres_nc.f90:495-540): for each aerosol
// class in class order and each layer upwards,
// work2d += dz(k)*0.5*(w(k)+w(k+1))*0.75*Qeff(ieff)/(rhop(ic)*reff(ieff))
// with w = c(ic)/Hm1; q[n] = qeff and r[n] = rhop*reff belong to class n.
template <class T>
__global__ void __launch_bounds__(32 * CW) k_out_aot(const T* c, Dims d, const OutClasses cl, const double* dz,
                                                     const double* Hm1, void* out, int f32) {
  __shared__ double w[CW + 1][32], term[CW][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long p = blockIdx.x * 32LL + lane, pc = min(p, d.plane() - 1);
  const int i = (int)(pc % d.nx) + 1, j = (int)(pc / d.nx) + 1;
  const long long hb = d.halo();
  const double h = Hm1[pc], rh = 1.0 / h;
  const bool h_plain = div_in_range(h);  // 0/h is 0
  double acc = 0.0;
  for (int n = 0; n < cl.n; ++n) {
    const T* cc = c + (long long)cl.at(n) * hb;
    const double q = cl.q_more ? cl.q_more[n] : cl.q[n], r = cl.r_more ? cl.r_more[n] : cl.r[n], rr = 1.0 / r;
    const bool q_plain = div_in_range(r) && fabs(q) < 1e300;  // 0*q/r is 0
    for (int k0 = 1; k0 <= d.nz - 1; k0 += CW) {  // layers k0 .. k0+CW-1, levels to k0+CW
      const int k = k0 + warp;
      auto W = [&](int kk) {
        const T v = cc[d.C(i, j, kk)];
        return v == T(0) && h_plain ? 0.0 : div_rn_recip(widen(v), h, rh);
      };
      if (k <= d.nz) w[warp][lane] = W(k);
      if (warp == 0 && k0 + CW <= d.nz) w[CW][lane] = W(k0 + CW);
      __syncthreads();
      if (k <= d.nz - 1) {
        const double two = w[warp][lane] + w[warp + 1][lane];
        term[warp][lane] = two == 0.0 && q_plain ? 0.0 : div_rn_recip(dz[k] * 0.5 * two * 0.75 * q, r, rr);
      }
      __syncthreads();
      if (warp == 0)
        for (int u = 0; u < CW && k0 + u <= d.nz - 1; ++u)
          if (term[u][lane] != 0.0) acc = acc + term[u][lane];
    }
    __syncthreads();
  }
  if (warp == 0 && p < d.plane()) put(out, p, acc, f32);
}

// deposit plane (printres_nc.f90:105-189): field(:,:,ic)/Hm1 of cload or cwet
__global__ void k_out_plane(const double* f, long long n, const double* Hm1, void* out, int f32) {
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  if (p < n) put(out, p, f[p] / Hm1[p], f32);
}

// deposit thickness, cm (printres_nc.f90:191-214): 1e2*(sum over particle
// classes of cload(ic)/rhop(ic))/Hm1; the reciprocals of rhop once per block,
// for OB classes at a time.
__global__ void k_out_thick(const double* cload, long long pl, int np, const double* rhop,
                            const double* Hm1, void* out, int f32) {
  __shared__ double rr[OB];
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  double s = 0.0;
  for (int i0 = 0; i0 < np; i0 += OB) {
    const int n = min(OB, np - i0);
    __syncthreads();  // the previous group's are read
    if (threadIdx.x < n) rr[threadIdx.x] = 1.0 / rhop[i0 + threadIdx.x];
    __syncthreads();
    for (int u = 0; u < n && p < pl; ++u)
      s = s + div_rn_recip(cload[(i0 + u + 1LL) * pl + p], rhop[i0 + u], rr[u]);
  }
  if (p < pl) put(out, p, 1e2 * s / Hm1[p], f32);
}

// concentration at a flight level, g/m3 (printres_nc.f90:542-573 and
// Sources/setcut.f90:1-54): the particle concentration w = (sum c)/Hm1
// interpolated linearly in pressure between the two layers whose
// pressures bracket pnom (p(k) >= pnom > p(k+1)), 0 below the first layer
// or when no pair of layers brackets it; times 1e3.
template <class T>
__global__ void k_out_fl(const T* c, Dims d, const OutClasses cl, const double* pres,
                         double pnom, const double* Hm1, void* out, int f32) {
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  const long long pl = d.plane();
  if (p >= pl) return;
  const int i = (int)(p % d.nx) + 1, j = (int)(p / d.nx) + 1;
  double v = 0.0;
  if (!(pnom > pres[p])) {
    for (int k = 1; k <= d.nz - 1; ++k) {
      const double pk = pres[(long long)(k - 1) * pl + p], pk1 = pres[(long long)k * pl + p];
      if (pnom <= pk && pnom > pk1) {
        const double s = (pnom - pk) / (pk1 - pk);
        const double h = Hm1[p];
        const long long hb = d.halo();
        const double wk = class_sum<T>(c, hb, d.C(i, j, k), cl) / h;
        const double wk1 = class_sum<T>(c, hb, d.C(i, j, k + 1), cl) / h;
        v = wk * (1.0 - s) + wk1 * s;
        break;
      }
    }
  }
  put(out, p, 1e3 * v, f32);
}

// 3-D concentration, g/m3 (printres_nc.f90:575-601 all particles,
// :646-671 one class): 1e3*((sum over the classes)/Hm1) on the model
// levels, or with `asl` moved to heights above sea level by
// Sources/ter2asl.f90:1-55 (linear in height between the terrain-following
// levels that bracket zlayer(k) above max(0,topg); 0 below the first level
// and above the last).
// The model levels take a thread per column and level.
template <class T>
__global__ void k_out_con(const T* c, Dims d, const OutClasses cl, const double* Hm1, void* out, int f32) {
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  const long long pl = d.plane();
  if (p >= pl) return;
  const int i = (int)(p % d.nx) + 1, j = (int)(p / d.nx) + 1;
  const long long hb = d.halo();
  const double h = Hm1[p], rh = 1.0 / h;
  for (int k = blockIdx.y + 1; k <= d.nz; k += gridDim.y)
    put(out, (long long)(k - 1) * pl + p, 1e3 * div_rn_recip(class_sum<T>(c, hb, d.C(i, j, k), cl), h, rh), f32);
}
template <class T>
__global__ void k_out_con_asl(const T* c, Dims d, const OutClasses cl, const double* Hm1, const double* zlayer,
                              const double* topg, void* out, int f32) {
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  const long long pl = d.plane();
  if (p >= pl) return;
  const int i = (int)(p % d.nx) + 1, j = (int)(p / d.nx) + 1;
  const long long hb = d.halo();
  const double h = Hm1[p];
  // the levels of the last pair: the next one mostly shares one of them (400x300x50
  // cells, the plain form, sums of 8 classes: 2.05 ms; 2.67 ms with each pair formed
  // anew and zeros found by binary64 comparisons)
  int ka = 0;
  double w[2] = {0.0, 0.0};
  const double zo = fmax2(0.0, topg[p]);
  for (int k = 1; k <= d.nz; ++k) {
    const double zasl = zlayer[k - 1];
    double v = 0.0;
    if (!(zasl < zo + zlayer[0])) {
      for (int kk = 1; kk <= d.nz - 1; ++kk) {
        if (zasl >= zo + zlayer[kk - 1] && zasl <= zo + zlayer[kk]) {
          const double s = (zo + zlayer[kk] - zasl) / (zlayer[kk] - zlayer[kk - 1]);
          if (kk != ka) {
            const bool next = ka > 0 && kk == ka + 1;
            if (next) w[0] = w[1];
            for (int u = next ? 1 : 0; u < 2; ++u) {
              const double x = 1e3 * (class_sum<T>(c, hb, d.C(i, j, kk + u), cl) / h);
              if (u == 0) w[0] = x;
              else w[1] = x;
            }
            ka = kk;
          }
          v = s * w[0] + (1.0 - s) * w[1];
          break;
        }
      }
    }
    put(out, (long long)(k - 1) * pl + p, v, f32);
  }
}

// a binary64 3-D field (x fastest) times Hm1 or not, with `asl` moved to
// heights above sea level by ter2asl: the gravity-current winds
// (printres_nc.f90:603-644: vx*Hm1, vy*Hm1) and Maggr (:673-690)
__global__ void k_out_field(const double* f, int times_hm1, Dims d, const double* Hm1,
                            const double* zlayer, const double* topg, int asl, void* out, int f32) {
  const long long p = blockIdx.x * (long long)OB + threadIdx.x;
  const long long pl = d.plane();
  if (p >= pl) return;
  const double h = Hm1[p];
  auto val = [&](int k) {
    const double v = f[(long long)(k - 1) * pl + p];
    return times_hm1 ? v * h : v;
  };
  if (!asl) {
    for (int k = 1; k <= d.nz; ++k) put(out, (long long)(k - 1) * pl + p, val(k), f32);
    return;
  }
  const double zo = fmax2(0.0, topg[p]);
  for (int k = 1; k <= d.nz; ++k) {
    const double zasl = zlayer[k - 1];
    double v = 0.0;
    if (!(zasl < zo + zlayer[0])) {
      for (int kk = 1; kk <= d.nz - 1; ++kk) {
        if (zasl >= zo + zlayer[kk - 1] && zasl <= zo + zlayer[kk]) {
          const double s = (zo + zlayer[kk] - zasl) / (zlayer[kk] - zlayer[kk - 1]);
          v = s * val(kk) + (1.0 - s) * val(kk + 1);
          break;
        }
      }
    }
    put(out, (long long)(k - 1) * pl + p, v, f32);
  }
}

// Tracking points (Sources/writps.f90, writps_air.f90): one thread per
// point, bilinear weights of the cell (ip, jp) at (s, t) in (-1,1)^2.
// out per point: [0..6] load, thickness, ground concentration, PM05, PM10,
// PM20, column mass (writps.f90:64-148); then nz concentrations, nz
// extinctions, nz number concentrations and the AOD (writps_air.f90:
// 64-109); then np class loads (writps.f90:215-222, writps_end).
struct TrackClass {
  double diam, rhop;
  int aer;         // an aerosol class of get_AOT_prop's range
  double q, r;     // Qeff(ieff), reff(ieff)
};
template <class T>
__global__ void k_track(const T* c, const double* cload, Dims d, int np, const int* ip, const int* jp,
                        const double* sp, const double* tp, int npts, const TrackClass* cls,
                        const double* dz, const double* Hm1, double* out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= npts) return;
  const int nz = d.nz;
  const long long pl = d.plane(), hb = d.halo();
  const int stride = 7 + 3 * nz + 1 + np;
  double* o = out + (long long)n * stride;
  const int i = ip[n], j = jp[n];
  const double s = sp[n], t = tp[n], st = s * t;
  const double v1 = (1.0 - t - s + st) * 0.25, v2 = (1.0 - t + s - st) * 0.25;
  const double v3 = (1.0 + t + s + st) * 0.25, v4 = (1.0 + t - s - st) * 0.25;
  const long long p1 = d.P(i, j), p2 = d.P(i + 1, j), p3 = d.P(i + 1, j + 1), p4 = d.P(i, j + 1);
  const double h1 = Hm1[p1], h2 = Hm1[p2], h3 = Hm1[p3], h4 = Hm1[p4];
  auto pl4 = [&](const double* f) {  // v1*(f1/h1) + ... of a 2-D field
    return v1 * (f[p1] / h1) + v2 * (f[p2] / h2) + v3 * (f[p3] / h3) + v4 * (f[p4] / h4);
  };
  auto c4 = [&](int ic, int k) {  // the same of c(:,:,k,ic)
    const T* cc = c + (long long)(ic - 1) * hb;
    return v1 * ((double)cc[d.C(i, j, k)] / h1) + v2 * ((double)cc[d.C(i + 1, j, k)] / h2) +
           v3 * ((double)cc[d.C(i + 1, j + 1, k)] / h3) + v4 * ((double)cc[d.C(i, j + 1, k)] / h4);
  };
  o[0] = pl4(cload);
  double thick = 0.0;
  for (int ic = 1; ic <= np; ++ic) {
    const double* f = cload + (long long)ic * pl;
    const double rp = cls[ic - 1].rhop;
    thick = thick + v1 * (f[p1] / h1 / rp) + v2 * (f[p2] / h2 / rp) + v3 * (f[p3] / h3 / rp) + v4 * (f[p4] / h4 / rp);
  }
  o[1] = 1e2 * thick;
  auto acc4 = [&](double a, int ic, int k) {  // a + v1*(c1/h1) + ... term by term
    const T* cc = c + (long long)(ic - 1) * hb;
    return a + v1 * ((double)cc[d.C(i, j, k)] / h1) + v2 * ((double)cc[d.C(i + 1, j, k)] / h2) +
           v3 * ((double)cc[d.C(i + 1, j + 1, k)] / h3) + v4 * ((double)cc[d.C(i, j + 1, k)] / h4);
  };
  double cg = 0.0, pm5 = 0.0, pm10 = 0.0, pm20 = 0.0;
  for (int ic = 1; ic <= np; ++ic) cg = acc4(cg, ic, 1);
  for (int ic = 1; ic <= np; ++ic)
    if (cls[ic - 1].diam <= 5e-6) pm5 = acc4(pm5, ic, 1);
  for (int ic = 1; ic <= np; ++ic)
    if (cls[ic - 1].diam <= 1e-5) pm10 = acc4(pm10, ic, 1);
  for (int ic = 1; ic <= np; ++ic)
    if (cls[ic - 1].diam <= 2e-5) pm20 = acc4(pm20, ic, 1);
  o[2] = cg * 1e3;
  o[3] = pm5 * 1e3;
  o[4] = pm10 * 1e3;
  o[5] = pm20 * 1e3;
  double cummc = 0.0;
  for (int ic = 1; ic <= np; ++ic)
    for (int k = 1; k <= nz - 1; ++k) {
      const double cp1 = c4(ic, k), cp2 = c4(ic, k + 1);
      cummc = cummc + dz[k] * 0.5 * (cp1 + cp2);
    }
  o[6] = 1e3 * cummc;
  double* cz = o + 7;
  double* ext = cz + nz;
  double* nco = ext + nz;
  double aod = 0.0;
  const double pi = 3.14159265358979323846;
  for (int k = 1; k <= nz; ++k) {
    double a = 0.0, e = 0.0, q = 0.0;
    for (int ic = 1; ic <= np; ++ic) {
      const double cc = c4(ic, k);
      a = a + cc;
      const TrackClass& k1 = cls[ic - 1];
      if (k1.aer) {
        e = e + (cc * 0.75 * k1.q) / (k1.rhop * k1.r);
        aod = aod + (dz[k] * cc * 0.75 * k1.q) / (k1.rhop * k1.r);
      }
      if (0.5 * k1.diam <= 32e-6) q = q + (6.0 * cc) / (k1.rhop * pi * k1.diam * k1.diam * k1.diam);
    }
    cz[k - 1] = a * 1e3;
    ext[k - 1] = e * 1e6;
    nco[k - 1] = q * 1e-6;
  }
  o[7 + 3 * nz] = aod;
  for (int ic = 1; ic <= np; ++ic) o[8 + 3 * nz + ic - 1] = pl4(cload + (long long)ic * pl);
}

unsigned blocks(long long n) { return (unsigned)((n + OB - 1) / OB); }

// Sources/printres_nc.f90:2066-2123 (get_AOT_prop): effective radii in
// micrometres and extinction efficiencies of the 20 aerosol bins.
const double kReffUm[20] = {0.014, 0.020, 0.028, 0.040, 0.056, 0.079, 0.112, 0.158, 0.224, 0.316,
                            0.447, 0.631, 0.891, 1.259, 1.778, 2.512, 3.548, 5.012, 7.079, 10.000};
const double kQeff[20] = {0.00213, 0.00386, 0.00864, 0.02324, 0.06674, 0.18285, 0.44613,
                          0.93225, 1.63000, 2.35760, 2.83130, 2.90880, 2.72340, 2.50530,
                          2.35970, 2.27100, 2.21020, 2.16410, 2.12830, 2.10050};

}  // namespace
}  // namespace f3d

using namespace f3d;

namespace {

#define OK(call)                                                                      \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess) return f3d::ctx_error(F3D_ERR_CUDA, cudaGetErrorString(e_)); \
  } while (0)

// Pressure at a flight level of the ICAO standard atmosphere
// (Sources/setcut.f90:60-107, standard_atm): three layers up to 32 km.
double standard_pressure(double z) {
  const double goo = 9.80665, Roo = 8.31432, Moo = 0.0289644;
  const double zoo = 0.0, Too = 288.15, poo = 101325.0, Loo = -0.0065;
  const double zo1 = 11000.0, To1 = 216.65, po1 = 22632.0;
  const double zo2 = 20000.0, To2 = 216.65, po2 = 5474.0, Lo2 = 0.001;
  if (z < zo1) {
    const double T = Too + Loo * (z - zoo);
    return poo * std::pow(Too / T, goo * Moo / (Roo * Loo));
  } else if (z < zo2) {
    return po1 * std::exp(-(goo * Moo * (z - zo1) / (Roo * To1)));
  }
  const double T = To2 + Lo2 * (z - zo2);
  return po2 * std::pow(To2 / T, goo * Moo / (Roo * Lo2));
}

// A device allocation of one call, given back on its stream.
struct Scratch {
  void* p = nullptr;
  cudaStream_t s = nullptr;
  ~Scratch() {
    if (p) cudaFreeAsync(p, s);
  }
};

// Where a call's kernel writes its n values of the wanted type: the
// destination itself if it is aligned memory of this device, else the
// context's plane buffer (2-D variables) or a buffer of the call (3-D), from
// which finish() copies.
struct Result {
  void* p = nullptr;
  size_t bytes = 0;
  Scratch own;
};

int result_buffer(f3d_ctx* x, long long n, void* dst, int dst_type, Result& r) {
  const size_t size = dst_type == F3D_OUT_BINARY32 ? sizeof(float) : sizeof(double);
  r.bytes = size * (size_t)n;
  cudaPointerAttributes at{};
  int dev = -1;
  if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
    cudaGetLastError();
    at.type = cudaMemoryTypeHost;
  }
  OK(cudaGetDevice(&dev));
  if (at.type == cudaMemoryTypeDevice && at.device == dev && reinterpret_cast<size_t>(dst) % size == 0) {
    r.p = dst;
  } else if (n <= x->d.plane()) {
    if (!x->out_plane)
      if (int rc = f3d::ctx_alloc(x, &x->out_plane, sizeof(double) * (size_t)x->d.plane())) return rc;
    r.p = x->out_plane;
  } else {
    r.own.s = x->stream;
    OK(cudaMallocAsync(&r.own.p, r.bytes, x->stream));
    r.p = r.own.p;
  }
  return F3D_OK;
}

int finish(f3d_ctx* x, const Result& r, void* dst) {
  cudaStream_t s = x->stream;
  if (r.p != dst) OK(cudaMemcpyAsync(dst, r.p, r.bytes, cudaMemcpyDefault, s));
  OK(cudaGetLastError());
  OK(cudaStreamSynchronize(s));
  return F3D_OK;
}

// The kernel parameter of a class list; lists longer than it holds are copied
// to `more` (device memory of the call).
int class_list(f3d_ctx* x, const std::vector<int>& cls, const std::vector<double>& q, const std::vector<double>& r,
               OutClasses& o, Scratch& more) {
  o = OutClasses{};
  o.n = (int)cls.size();
  if (cls.size() <= (size_t)CMAX) {
    for (size_t i = 0; i < cls.size(); ++i) o.cls[i] = cls[i];
    for (size_t i = 0; i < q.size(); ++i) {
      o.q[i] = q[i];
      o.r[i] = r[i];
    }
    return F3D_OK;
  }
  const size_t n = cls.size();
  more.s = x->stream;
  OK(cudaMallocAsync(&more.p, (2 * sizeof(double) + sizeof(int)) * n, x->stream));
  double* dq = reinterpret_cast<double*>(more.p);
  int* dc = reinterpret_cast<int*>(dq + 2 * n);
  OK(cudaMemcpyAsync(dc, cls.data(), sizeof(int) * n, cudaMemcpyHostToDevice, x->stream));
  if (!q.empty()) {
    OK(cudaMemcpyAsync(dq, q.data(), sizeof(double) * n, cudaMemcpyHostToDevice, x->stream));
    OK(cudaMemcpyAsync(dq + n, r.data(), sizeof(double) * n, cudaMemcpyHostToDevice, x->stream));
    o.q_more = dq;
    o.r_more = dq + n;
  }
  o.cls_more = dc;
  return F3D_OK;
}

// classes of printres_nc.f90's selections (0-based)
std::vector<int> particle_classes(const f3d_ctx* x) {
  std::vector<int> v;
  for (int ic = 0; ic < x->g.np; ++ic) v.push_back(ic);
  return v;
}

}  // namespace

extern "C" {

int f3d_output(f3d_ctx* x, int var, int index, int asl, void* dst, int dst_type) {
  if (!x || !dst) return f3d::ctx_error(F3D_ERR_ARG, "NULL argument");
  if (dst_type != F3D_OUT_BINARY64 && dst_type != F3D_OUT_BINARY32)
    return f3d::ctx_error(F3D_ERR_ARG, "dst_type must be F3D_OUT_BINARY64 or F3D_OUT_BINARY32");
  const Dims d = x->d;
  const int nc = x->g.nc, np = x->g.np;
  const long long pl = d.plane();
  long long n = pl;  // values in the result
  std::vector<int> cls;
  std::vector<double> q, r;
  switch (var) {
    case F3D_OUT_LOAD:
    case F3D_OUT_WET:
      if (index < 0 || index > np) return f3d::ctx_error(F3D_ERR_ARG, "class index outside 0..np");
      break;
    case F3D_OUT_THICK:
      break;
    case F3D_OUT_COL_MASS:
      if (index == 0) {
        cls = particle_classes(x);
      } else {
        if (index < 1 || np + index > nc) return f3d::ctx_error(F3D_ERR_ARG, "gas index outside 1..nc-np");
        cls.push_back(np + index - 1);
      }
      break;
    case F3D_OUT_PM_COL:
    case F3D_OUT_PM_GRND: {
      double thr;
      if (index == 5)
        thr = 5e-6;
      else if (index == 10)
        thr = 1e-5;
      else if (index == 20)
        thr = 2e-5;
      else
        return f3d::ctx_error(F3D_ERR_ARG, "PM size must be 5, 10 or 20 (micrometres)");
      for (int ic = 0; ic < np; ++ic)
        if (x->h_diam[ic] <= thr) cls.push_back(ic);
      break;
    }
    case F3D_OUT_C_GRND:
      cls = particle_classes(x);
      break;
    case F3D_OUT_AOT05: {
      double reff[20];
      for (int b = 0; b < 20; ++b) reff[b] = kReffUm[b] * 1e-6;
      for (int ic = 0; ic < np; ++ic) {
        const double rad = 0.5 * x->h_diam[ic];
        if (!(rad >= reff[0] && rad <= reff[19])) continue;
        int ieff = 0;
        for (int b = 0; b < 19; ++b)
          if (rad >= reff[b] && rad <= reff[b + 1]) ieff = b + 1;
        cls.push_back(ic);
        q.push_back(kQeff[ieff]);
        r.push_back(x->h_rhop[ic] * reff[ieff]);
      }
      break;
    }
    case F3D_OUT_CON:
      if (index < 0 || index > nc) return f3d::ctx_error(F3D_ERR_ARG, "class index outside 0..nc");
      if (index == 0)
        cls = particle_classes(x);
      else
        cls.push_back(index - 1);
      n = d.cells();
      break;
    case F3D_OUT_WIND:
      if (index != 1 && index != 2) return f3d::ctx_error(F3D_ERR_ARG, "wind component must be 1 (u) or 2 (v)");
      n = d.cells();
      break;
    case F3D_OUT_MAGGR:
      if (!x->agr_on) return f3d::ctx_error(F3D_ERR_STATE, "aggregation is off");
      n = d.cells();
      break;
    default:
      return f3d::ctx_error(F3D_ERR_ARG, "unknown output variable");
  }
  cudaStream_t s = x->stream;
  Scratch more;
  OutClasses cl;
  Result res;
  if (int rc = class_list(x, cls, q, r, cl, more)) return rc;
  if (int rc = result_buffer(x, n, dst, dst_type, res)) return rc;
  const int o32 = dst_type == F3D_OUT_BINARY32;
  const unsigned cb = (unsigned)((pl + 31) / 32);
  const bool f32 = x->prec == F3D_PREC_FP32;
  switch (var) {
    case F3D_OUT_LOAD:
    case F3D_OUT_WET:
    case F3D_OUT_THICK:
      launch_getc0(x->cdry, x->cwet, x->cload, d, nc, np, s);
      if (var == F3D_OUT_THICK)
        k_out_thick<<<blocks(pl), OB, 0, s>>>(x->cload, pl, np, x->rhop, x->Hm1, res.p, o32);
      else
        k_out_plane<<<blocks(pl), OB, 0, s>>>((var == F3D_OUT_LOAD ? x->cload : x->cwet) + index * pl, pl,
                                              x->Hm1, res.p, o32);
      break;
    case F3D_OUT_COL_MASS:
    case F3D_OUT_PM_COL:
      if (f32)
        k_out_column<float><<<cb, 32 * CW, 0, s>>>(x->c32, d, cl, x->dz, x->Hm1, res.p, o32);
      else
        k_out_column<double><<<cb, 32 * CW, 0, s>>>(x->c64, d, cl, x->dz, x->Hm1, res.p, o32);
      break;
    case F3D_OUT_C_GRND:
    case F3D_OUT_PM_GRND:
      if (f32)
        k_out_ground<float><<<blocks(pl), OB, 0, s>>>(x->c32, d, cl, x->Hm1, res.p, o32);
      else
        k_out_ground<double><<<blocks(pl), OB, 0, s>>>(x->c64, d, cl, x->Hm1, res.p, o32);
      break;
    case F3D_OUT_AOT05:
      if (f32)
        k_out_aot<float><<<cb, 32 * CW, 0, s>>>(x->c32, d, cl, x->dz, x->Hm1, res.p, o32);
      else
        k_out_aot<double><<<cb, 32 * CW, 0, s>>>(x->c64, d, cl, x->dz, x->Hm1, res.p, o32);
      break;
    case F3D_OUT_WIND:
    case F3D_OUT_MAGGR:
      k_out_field<<<blocks(pl), OB, 0, s>>>(var == F3D_OUT_MAGGR ? x->agr_maggr : (index == 1 ? x->vx : x->vy),
                                            var == F3D_OUT_WIND, d, x->Hm1, x->zlayer, x->topg, asl, res.p, o32);
      break;
    case F3D_OUT_CON: {
      const dim3 grid(blocks(pl), (unsigned)std::min(d.nz, 65535));
      if (f32 && asl)
        k_out_con_asl<float><<<blocks(pl), OB, 0, s>>>(x->c32, d, cl, x->Hm1, x->zlayer, x->topg, res.p, o32);
      else if (asl)
        k_out_con_asl<double><<<blocks(pl), OB, 0, s>>>(x->c64, d, cl, x->Hm1, x->zlayer, x->topg, res.p, o32);
      else if (f32)
        k_out_con<float><<<grid, OB, 0, s>>>(x->c32, d, cl, x->Hm1, res.p, o32);
      else
        k_out_con<double><<<grid, OB, 0, s>>>(x->c64, d, cl, x->Hm1, res.p, o32);
      break;
    }
  }
  count_launch();
  return finish(x, res, dst);
}

int f3d_track_points(f3d_ctx* x, int npts, const double* xpts, const double* ypts, double xo, double yo,
                     double* out) {
  if (!x || (npts > 0 && (!xpts || !ypts || !out))) return f3d::ctx_error(F3D_ERR_ARG, "NULL argument");
  if (npts <= 0) return F3D_OK;
  const Dims d = x->d;
  const int np = x->g.np, nz = d.nz;
  // get_pts_st (Sources/reaout.f90:180-224): the cell and (s,t) of each point
  std::vector<int> ip(npts), jp(npts);
  std::vector<double> sp(npts), tp(npts);
  const double dxo = x->g.dx, dyo = x->g.dy;
  for (int n = 0; n < npts; ++n) {
    bool found = false;
    for (int ix = 1; ix <= d.nx - 1; ++ix) {
      const double xx = xo + (ix - 1) * dxo;
      if (xpts[n] >= xx && xpts[n] <= xx + dxo) {
        ip[n] = ix;
        sp[n] = (xpts[n] - xx) / dxo;
        sp[n] = 2.0 * sp[n] - 1.0;
        found = true;
      }
    }
    if (!found) return f3d::ctx_error(F3D_ERR_RANGE, "get_pts_st: value not found");
    found = false;
    for (int iy = 1; iy <= d.ny - 1; ++iy) {
      const double yy = yo + (iy - 1) * dyo;
      if (ypts[n] >= yy && ypts[n] <= yy + dyo) {
        jp[n] = iy;
        tp[n] = (ypts[n] - yy) / dyo;
        tp[n] = 2.0 * tp[n] - 1.0;
        found = true;
      }
    }
    if (!found) return f3d::ctx_error(F3D_ERR_RANGE, "get_pts_st: value not found");
  }
  std::vector<TrackClass> cls(np > 0 ? np : 1);
  double reff[20];
  for (int b = 0; b < 20; ++b) reff[b] = kReffUm[b] * 1e-6;
  for (int ic = 0; ic < np; ++ic) {
    TrackClass& k = cls[ic];
    k.diam = x->h_diam[ic];
    k.rhop = x->h_rhop[ic];
    k.aer = 0;
    k.q = k.r = 0.0;
    const double rad = (double)0.5f * k.diam;
    if (rad >= reff[0] && rad <= reff[19]) {
      int ieff = 0;
      for (int b = 0; b < 19; ++b)
        if (rad >= reff[b] && rad <= reff[b + 1]) ieff = b + 1;
      k.aer = 1;
      k.q = kQeff[ieff];
      k.r = reff[ieff];
    }
  }
  const int stride = 7 + 3 * nz + 1 + np;
  cudaStream_t s = x->stream;
  Scratch sc;
  sc.s = s;
  const size_t bo = sizeof(double) * (size_t)npts * stride;
  const size_t bi = (sizeof(int) * 2 + sizeof(double) * 2) * (size_t)npts;
  OK(cudaMallocAsync(&sc.p, bo + bi + sizeof(TrackClass) * cls.size() + 256, s));
  unsigned char* b = reinterpret_cast<unsigned char*>(sc.p);
  double* res = reinterpret_cast<double*>(b);
  double* dsp = reinterpret_cast<double*>(b + bo);
  double* dtp = dsp + npts;
  int* dip = reinterpret_cast<int*>(dtp + npts);
  int* djp = dip + npts;
  TrackClass* dcls = reinterpret_cast<TrackClass*>(b + ((bo + bi + 15) & ~size_t(15)));
  OK(cudaMemcpyAsync(dsp, sp.data(), sizeof(double) * npts, cudaMemcpyHostToDevice, s));
  OK(cudaMemcpyAsync(dtp, tp.data(), sizeof(double) * npts, cudaMemcpyHostToDevice, s));
  OK(cudaMemcpyAsync(dip, ip.data(), sizeof(int) * npts, cudaMemcpyHostToDevice, s));
  OK(cudaMemcpyAsync(djp, jp.data(), sizeof(int) * npts, cudaMemcpyHostToDevice, s));
  OK(cudaMemcpyAsync(dcls, cls.data(), sizeof(TrackClass) * cls.size(), cudaMemcpyHostToDevice, s));
  launch_getc0(x->cdry, x->cwet, x->cload, d, x->g.nc, np, s);
  const unsigned nb = (unsigned)((npts + 63) / 64);
  if (x->prec == F3D_PREC_FP32)
    k_track<float><<<nb, 64, 0, s>>>(x->c32, x->cload, d, np, dip, djp, dsp, dtp, npts, dcls, x->dz, x->Hm1, res);
  else
    k_track<double><<<nb, 64, 0, s>>>(x->c64, x->cload, d, np, dip, djp, dsp, dtp, npts, dcls, x->dz, x->Hm1, res);
  count_launch();
  OK(cudaMemcpyAsync(out, res, bo, cudaMemcpyDefault, s));
  OK(cudaGetLastError());
  OK(cudaStreamSynchronize(s));
  return F3D_OK;
}

int f3d_output_fl(f3d_ctx* x, double flight_level, const double* p, void* dst, int dst_type) {
  if (!x || !p || !dst) return f3d::ctx_error(F3D_ERR_ARG, "NULL argument");
  if (dst_type != F3D_OUT_BINARY64 && dst_type != F3D_OUT_BINARY32)
    return f3d::ctx_error(F3D_ERR_ARG, "dst_type must be F3D_OUT_BINARY64 or F3D_OUT_BINARY32");
  const Dims d = x->d;
  const long long pl = d.plane(), s3 = d.cells();
  const double pnom = standard_pressure(flight_level * 30.48);  // printres_nc.f90:559
  cudaStream_t s = x->stream;
  Scratch more, sc;
  OutClasses cl;
  Result res;
  if (int rc = class_list(x, particle_classes(x), {}, {}, cl, more)) return rc;
  if (int rc = result_buffer(x, pl, dst, dst_type, res)) return rc;
  sc.s = s;
  OK(cudaMallocAsync(&sc.p, sizeof(double) * s3, s));
  double* dp = reinterpret_cast<double*>(sc.p);
  OK(cudaMemcpyAsync(dp, p, sizeof(double) * s3, cudaMemcpyDefault, s));
  const int o32 = dst_type == F3D_OUT_BINARY32;
  if (x->prec == F3D_PREC_FP32)
    k_out_fl<float><<<blocks(pl), OB, 0, s>>>(x->c32, d, cl, dp, pnom, x->Hm1, res.p, o32);
  else
    k_out_fl<double><<<blocks(pl), OB, 0, s>>>(x->c64, d, cl, dp, pnom, x->Hm1, res.p, o32);
  count_launch();
  return finish(x, res, dst);
}

}  // extern "C"
