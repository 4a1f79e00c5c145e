// f3d_coeff.cu -- the per-meteo-update coefficient chain of
// Sources/meteo.f90:19-149 on the device (binary64, --fmad=false).
//
// Transcendentals (pow, log, log10, exp, atan, acos, tan) are CUDA's; the
// reference uses the host libm, so these fields agree to a few ulp, not
// bitwise.  Everything else is rounded operation by operation as written.
//
// setvset: vsettl keeps its drag coefficient cd between calls
// (Sources/setvset.f90:89, SAVE), so the reference evaluates one sequential
// chain over (ic, i, j, k) with k fastest, continued across meteo updates.
// The chain is split into segments; each segment starts from a guess after a
// warm-up over the cells that precede it, and is accepted only if its entry
// cd equals, bit for bit, the exit cd of the previous segment (from then on
// the computation is identical to the sequential one).  The iteration
// contracts, so the warm-up reaches the exact chain value within a few to a
// few tens of cells; any segment that fails the check is recomputed in order
// from the verified exit of its predecessor.
//
// The drag iteration is binary64-pipe bound on GB300 (two lanes per SM and
// clock), so its Ganser form is restated to issue about 26 binary64 operations
// (GanserCell) in place of the reference's four divisions, square root and
// pow: the same iteration and stopping test on values that differ from the
// reference's by a few ulp.
#include <algorithm>

#include "f3d_dmath.cuh"
#include "f3d_internal.h"

namespace f3d {

static int sms() {
  static int nsm = 0;
  if (!nsm) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }
  return std::max(1, nsm);
}

// ------------------------------------------------------------- kappa3
// Sources/kappa3.f90:50-236.  A thread takes up to K3_LEV levels of a column: what
// depends on the column alone (the power of RAMS, the divisors) is formed once
// and divisions by a column's or a level's divisor use its reciprocal
// (div_rn_recip: the same quotient), since binary64 operations bound it
// (400x300x50 cells: 2.72 ms one cell per thread, 0.98 ms so).
constexpr int K3_LEV = 10, K3_B = 128;

struct K3Level {  // of level k (kappa3.f90:64-96)
  double zl, dzs, rdzs;  // zlayer, dz(k)+dz(k-1) and its reciprocal
  double lc;             // 1/(1/(vkarm*zl) + 1/rlamb)
};

__global__ void k_kappa3(Dims d, int modkv, int modkh, int coord_sys, double rkv0, double rkh0,
                         double Csh, double dX1, double dX2, double dx, double dy,
                         const double* dz, const double* zlayer, const double* Hm1,
                         const double* vx, const double* vy, const double* vptemp,
                         const double* ustar, const double* zi, const double* rl,
                         double* rkver, double* rkhor, int levels) {
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const double vkarm = 0.4, beta1 = 9.2, beta2 = 13.0, rlamb = 30.0, rkhmin = 1e2, rkvmin = 1.0;
  const double hinf = 5.0, hsup = 5e3, alfa = 0.28, Khf = 8000.0, gi = 9.81;
  const bool vert = modkv != 0, horiz = modkh != 0;
  const int k0 = blockIdx.y * levels + 1, k1 = min(nz, k0 + levels - 1);
  __shared__ K3Level lev[K3_LEV + 1];  // levels k0-1 .. (k0-1: only for k = nz, below)
  if (vert && threadIdx.x <= levels) {
    const int k = k0 - 1 + threadIdx.x;
    if (k >= 1 && k <= nz) {
      K3Level z;
      z.zl = zlayer[k - 1];
      z.dzs = dz[k] + dz[k - 1];
      z.rdzs = 1.0 / z.dzs;
      z.lc = 1.0 / ((1.0 / (vkarm * z.zl)) + (1.0 / rlamb));
      lev[threadIdx.x] = z;
    }
  }
  __syncthreads();
  const long long p = blockIdx.x * (long long)K3_B + threadIdx.x, pl = d.plane();
  if (p >= pl) return;
  const int i = (int)(p % nx) + 1, j = (int)(p / nx) + 1;
  // shear and Richardson number of cell (a,b) at level k < nz (kappa3.f90:64-71)
  auto grad = [&](long long q, int k, double& dvdz2, double& rich) {
    const K3Level& z = lev[k - k0 + 1];
    const long long m = q + (k - 1) * pl;
    const double gx = div_rn_recip(vx[m + pl] - vx[m - pl], z.dzs, z.rdzs);
    const double gy = div_rn_recip(vy[m + pl] - vy[m - pl], z.dzs, z.rdzs);
    dvdz2 = gx * gx + gy * gy;
    dvdz2 = fmax2(dvdz2, 1e-10);
    rich = gi * div_rn_recip(vptemp[m + pl] - vptemp[m - pl], z.dzs, z.rdzs) / (vptemp[m] * dvdz2);
  };
  const double us = vert ? ustar[p] : 0.0, rlp = vert ? rl[p] : 0.0;
  const double h = vert ? fmin2(fmax2(zi[p], hinf), hsup) : 1.0, rh = vert ? 1.0 / h : 1.0;
  const double dXX = horiz ? Hm1[p] * dX1 : 1.0;
  const double ddx = i == 1 || i == nx ? dXX : 2.0 * dXX, rddx = horiz ? 1.0 / ddx : 1.0;
  const double ddy = j == 1 || j == ny ? dX2 : 2.0 * dX2, rddy = horiz ? 1.0 / ddy : 1.0;
  const double Kmh = modkh == 1 ? 0.075 * pow(dXX * dX2, 2.0 / 3.0) : 0.0;
  const long long e = i == nx ? p : p + 1, w = i == 1 ? p : p - 1;
  const long long n = j == ny ? p : p + nx, s = j == 1 ? p : p - nx;
  for (int k = k0; k <= k1; ++k) {
    const long long o = (k - 1) * pl, m = p + o;
    const double zl = vert ? lev[k - k0 + 1].zl : 0.0;
    // vertical
    if (modkv == 0) {
      rkver[m] = rkv0;
    } else if (modkv == 1) {
      if (k >= 2) {
        const double zeta = div_rn_recip(zl, h, rh);
        double kv;
        if (zeta < 1.0) {
          if (rlp >= 0.0)
            kv = vkarm * us * zl * (1.0 - zeta) / (1.0 + beta1 * zl * rlp);
          else
            kv = vkarm * us * zl * (1.0 - zeta) * sqrt(1.0 - beta2 * zl * rlp);
        } else {
          double dvdz2, rich;
          // at k = nz the reference reuses the values of the last point
          // computed at k = nz-1, i.e. (nx, ny, nz-1) (kappa3.f90:64-71)
          if (k < nz)
            grad(p, k, dvdz2, rich);
          else
            grad(pl - 1, nz - 1, dvdz2, rich);
          const double lc = lev[k - k0 + 1].lc;
          if (rich >= 0.0)
            kv = lc * lc * sqrt(dvdz2) / (1.0 + 10.0 * rich * (1.0 + 8.0 * rich));
          else
            kv = lc * lc * sqrt(dvdz2) * sqrt(1.0 - 18.0 * rich);
          kv = fmax2(kv, rkvmin);
        }
        rkver[m] = kv;
      }
    } else if (modkv == 2) {
      const double gh = 11.6, betah = 7.8, prt = 0.95;
      double zeta = zl * rlp;
      double kv;
      if (zeta < 0.0)
        kv = vkarm * us * zl * sqrt(1.0 - gh * zeta) / prt;
      else if (zeta > 0.0)
        kv = vkarm * us * zl / (prt + betah * zeta);
      else
        kv = vkarm * us * zl / prt;
      zeta = div_rn_recip(zl, h, rh);
      if (zeta > 1.0) zeta = 1.0;
      rkver[m] = kv * (1.0 - zeta);
    }
    // horizontal
    if (modkh == 0) {
      rkhor[m] = rkh0;
    } else if (modkh == 1 || modkh == 2) {
      const double dvxdx = div_rn_recip(vx[e + o] - vx[w + o], ddx, rddx);
      const double dvydx = div_rn_recip(vy[e + o] - vy[w + o], ddx, rddx);
      const double dvxdy = div_rn_recip(vx[n + o] - vx[s + o], ddy, rddy);
      const double dvydy = div_rn_recip(vy[n + o] - vy[s + o], ddy, rddy);
      double kh;
      if (modkh == 1) {
        const double s1 = dvxdy + dvydx;
        kh = Csh * Csh * dXX * dX2 * sqrt(s1 * s1 + 2.0 * (dvxdx * dvxdx + dvydy * dvydy));
        kh = 1.0 * fmax2(kh, Kmh);
        kh = fmax2(kh, rkhmin);
      } else {
        const double Khn0 = (coord_sys == 0) ? 3.6e-2 : 4000.0;
        const double s1 = dvxdx - dvydy, s2 = dvydx + dvxdy;
        const double Kht = alfa * alfa * dXX * dX2 * sqrt(s1 * s1 + s2 * s2);
        const double Khn = Khf * (Khn0 / Hm1[p] / dx) * (Khn0 / dy);
        kh = (1.0 / Kht) + (1.0 / Khn);
        kh = fmax2(1.0 / kh, rkhmin);
      }
      rkhor[m] = kh;
    }
  }
}

// both diffusivities constant
__global__ void k_kappa3_const(long long n, double rkv0, double rkh0, double* rkver, double* rkhor) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < n; m += (long long)gridDim.x * blockDim.x) {
    rkver[m] = rkv0;
    rkhor[m] = rkh0;
  }
}

void launch_kappa3(Dims d, int modkv, int modkh, int coord_sys, double rkv0, double rkh0,
                   double Csh, double dX1, double dX2, double dx, double dy, const double* dz,
                   const double* zlayer, const double* Hm1, const double* vx, const double* vy,
                   const double* vptemp, const double* ustar, const double* zi, const double* rl,
                   double* rkver, double* rkhor, cudaStream_t s) {
  const long long cb = (d.plane() + K3_B - 1) / K3_B;
  if (modkv == 0 && modkh == 0) {
    const long long n = d.cells();
    k_kappa3_const<<<(unsigned)std::min<long long>((n + 255) / 256, 8LL * sms()), 256, 0, s>>>(n, rkv0, rkh0, rkver,
                                                                                            rkhor);
    count_launch();
    return;
  }
  // as many levels per thread as leave three blocks on two SMs, in groups of
  // about the same size: 33x29x14 cells 40 us with one level, 83 with ten;
  // 80x80x25 75 with five, 85 with ten and 99 with one; 121x101x30 114 with ten,
  // 135 with three; 400x300x50 1.25 ms with ten, 2.49 with one (the call's wall clock)
  const long long most = std::max<long long>(1, std::min<long long>(K3_LEV, 2 * cb * d.nz / (3LL * sms())));
  const int groups = (int)((d.nz + most - 1) / most), levels = (d.nz + groups - 1) / groups;
  k_kappa3<<<dim3((unsigned)cb, groups), K3_B, 0, s>>>(
      d, modkv, modkh, coord_sys, rkv0, rkh0, Csh, dX1, dX2, dx, dy, dz, zlayer, Hm1, vx, vy, vptemp, ustar, zi, rl,
      rkver, rkhor, levels);
  count_launch();
}

// --------------------------------------------------------- setvdrydep
// Sources/setvdrydep.f90:74-264; the Feng (2008) coefficient tables of
// setvdrydep.f90:79-129 indexed [land use - 1][mode - 1].
__constant__ double c_feng_a[6][4] = {
    {0.0048, 0.0315, 1.2891, 1.0338}, {0.0037, 0.0120, 1.3977, 1.0707},
    {0.0042, 0.2928, 1.3970, 0.9155}, {0.0032, 0.1201, 1.1838, 1.0096},
    {0.0043, 0.1337, 1.2834, 1.1595}, {0.0045, 0.0925, 1.2654, 1.0891}};
__constant__ double c_feng_b[6][4] = {
    {1.0, 2.7925, 2.6878, 1.2644}, {1.0, 2.2413, 2.5838, 1.3247}, {1.0, 3.8581, 2.5580, 1.0364},
    {1.0, 3.4407, 2.8033, 1.2069}, {1.0, 3.5456, 2.7157, 1.4863}, {1.0, 3.2920, 2.7227, 1.4240}};
// USGS 24-category land use -> Feng land class (setvdrydep.f90:165-215).
__constant__ int c_usgs_feng[25] = {6, 1, 6, 6, 6, 6, 6, 6, 6, 6, 3, 6, 6, 6,
                                    6, 6, 5, 6, 6, 3, 2, 2, 2, 2, 4};

__device__ __forceinline__ int drydep_mode(double dm) {
  if (dm > 100e-6) return 0;
  if (dm > 10e-6) return 4;
  if (dm > 2.5e-6) return 3;
  if (dm > 0.1e-6) return 2;
  return 1;
}

__global__ void k_setvdrydep(Dims d, int nc, const double* diam, const double* zlayer,
                             const double* ldu, const double* rl, const double* znt,
                             const double* ustar, const double* tempe, const double* rho,
                             double* vdep) {
  const long long pl = d.plane();
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= pl) return;
  bool have_to_work = false;
  for (int ic = 0; ic < nc; ++ic) have_to_work |= drydep_mode(diam[ic]) > 0;
  if (!have_to_work) return;
  const double vkarm = 0.4, visc0 = 1.827e-5, Tair0 = 291.15;
  const double lv = ldu[p];
  int iland = 6;
  if (lv > -1.0 && lv < 25.0) {
    const int code = (int)lv;
    if (code >= 1 && code <= 24) iland = c_usgs_feng[code];
  }
  const double zeta = rl[p] * zlayer[0];
  const double zeta0 = rl[p] * znt[p];
  double ra;
  if (ustar[p] > 0.0) {
    ra = log(zlayer[0] / znt[p]);
    if (zeta > 0) {
      ra = ra + 4.7 * (zeta - zeta0);
    } else if (zeta < 0) {
      const double eta = pow(1.0 - 15.0 * zeta, 0.25);
      const double eta0 = pow(1.0 - 15.0 * zeta0, 0.25);
      ra = ra + log((eta0 * eta0 + 1) * ((eta0 + 1) * (eta0 + 1)) /
                    ((eta * eta + 1) * ((eta + 1) * (eta + 1))));
      ra = ra + 2 * (atan(eta) - atan(eta0));
    }
    ra = ra / (ustar[p] * vkarm);
  } else {
    ra = 1e20;
  }
  const double T = tempe[p];
  const double visc = visc0 * ((Tair0 + 120.0) / (T + 120.0)) * pow(T / Tair0, 1.5);
  double Re = ustar[p] * znt[p] * rho[p] / visc;
  if (Re > 40300.0) Re = 40300.0;
  double Vd1 = -0.5 * ((Re - 40300.0) / 15330.0) * ((Re - 40300.0) / 15330.0);
  Vd1 = 0.0226 * ustar[p] * exp(Vd1);
  for (int ic = 0; ic < nc; ++ic) {
    const int mode = drydep_mode(diam[ic]);
    if (mode > 0) {
      double Vd = Vd1 + c_feng_a[iland - 1][mode - 1] * pow(ustar[p], c_feng_b[iland - 1][mode - 1]);
      Vd = ra + 1.0 / Vd;
      vdep[(long long)ic * pl + p] = -1.0 / Vd;
    }
  }
}

void launch_setvdrydep(Dims d, int nc, const double* diam, const double* zlayer,
                       const double* ldu, const double* rl, const double* znt,
                       const double* ustar, const double* tempe, const double* rho,
                       double* vdep, cudaStream_t s) {
  const long long pl = d.plane();
  k_setvdrydep<<<(unsigned)((pl + 127) / 128), 128, 0, s>>>(d, nc, diam, zlayer, ldu, rl, znt, ustar,
                                                           tempe, rho, vdep);
  count_launch();
}

// ------------------------------------------ scaling, corvver, setdivu
// Sources/meteo.f90:108-112 (scaling), Sources/corvver.f90:21-34,
// Sources/setdivu.f90:16-30.
__global__ void k_scale_corvver(Dims d, int coord_sys, double dX1, double dX2, const double* Hm1,
                                const double* topg, double* vx, const double* vy, double* vz,
                                double* rho, const double* rkhor, double* rkh1) {
  const int nx = d.nx, ny = d.ny;
  const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (m >= d.cells()) return;
  const int ix = (int)(m % nx) + 1;
  const int iy = (int)((m / nx) % ny) + 1;
  const long long p = d.P(ix, iy);
  const double h = Hm1[p];
  const double vxs = vx[m] / h;
  vx[m] = vxs;
  rho[m] = rho[m] * h;
  rkh1[m] = rkhor[m] / (h * h);
  if (coord_sys == 0) {
    const double dyinv = 1.0 / dX2;
    const double dxinv = 1.0 / (h * dX1);
    const double zx = dxinv * (topg[d.P(ix + 1 <= nx ? ix + 1 : nx, iy)] - topg[p]);
    const double zy = dyinv * (topg[d.P(ix, iy + 1 <= ny ? iy + 1 : ny)] - topg[p]);
    const double vs = zx * vxs + zy * vy[m];
    vz[m] = vz[m] - vs;
  }
}

__global__ void k_setdivu(Dims d, double dX1, double dX2, const double* dz, const double* Hm1,
                          const double* vx, const double* vy, const double* vz, double* divu) {
  const int nx = d.nx, ny = d.ny;
  const long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (m >= d.cells()) return;
  const int i = (int)(m % nx) + 1;
  const int j = (int)((m / nx) % ny) + 1;
  const int k = (int)(m / ((long long)nx * ny)) + 1;
  const double vi = vx[m], vi_1 = vx[d.M(i > 1 ? i - 1 : 1, j, k)];
  const double vj = vy[m], vj_1 = vy[d.M(i, j > 1 ? j - 1 : 1, k)];
  const double vk = vz[m], vk_1 = vz[d.M(i, j, k > 1 ? k - 1 : 1)];
  divu[m] = (vi - vi_1) / (Hm1[d.P(i, j)] * dX1) + (vj - vj_1) / dX2 + (vk - vk_1) / dz[k];
}

void launch_meteo_scale(Dims d, int coord_sys, double dX1, double dX2, const double* dz,
                        const double* Hm1, const double* topg, double* vx, double* vy,
                        double* vz, double* rho, const double* rkhor, double* rkh1,
                        double* divu, cudaStream_t s) {
  const long long n = d.cells();
  const unsigned nb = (unsigned)((n + 255) / 256);
  k_scale_corvver<<<nb, 256, 0, s>>>(d, coord_sys, dX1, dX2, Hm1, topg, vx, vy, vz, rho, rkhor, rkh1);
  count_launch();
  if (divu) {
    k_setdivu<<<nb, 256, 0, s>>>(d, dX1, dX2, dz, Hm1, vx, vy, vz, divu);
    count_launch();
  }
}

void launch_setdivu(Dims d, double dX1, double dX2, const double* dz, const double* Hm1,
                    const double* vx, const double* vy, const double* vz, double* divu,
                    cudaStream_t s) {
  const long long n = d.cells();
  k_setdivu<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(d, dX1, dX2, dz, Hm1, vx, vy, vz, divu);
  count_launch();
}

// reamet.f90:146 (PRATE mm/s -> mm/h when wet deposition is on) and
// reamet.f90:153 (vz(:,:,1) = 0); with wet deposition also the highest level
// it reaches at any column, max over zi of the levels with zlayer <= zi
// (wetdep.f90:37), for the step kernel's column pieces.
__global__ void k_reamet_fix(Dims d, int wetdep, double* vz, double* prate, const double* zi, const double* zlayer,
                             int* nwet) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= d.plane()) return;
  vz[p] = 0.0;
  if (!wetdep) return;
  prate[p] = prate[p] * 3600.0;
  const double z = zi[p];
  int top = 0;
  for (int k = 1; k <= d.nz; ++k)
    if (zlayer[k - 1] <= z) top = k;
  if (top > 0) atomicMax(nwet, top);
}

void launch_reamet_fix(Dims d, int wetdep, double* vz, double* prate, const double* zi, const double* zlayer,
                       int* nwet, cudaStream_t s) {
  k_reamet_fix<<<(unsigned)((d.plane() + 255) / 256), 256, 0, s>>>(d, wetdep, vz, prate, zi, zlayer, nwet);
  count_launch();
}

// ------------------------------------------------------------ setvset
struct ClassConst {
  double diam, rhop, psi;
  double num;       // 4*gi*diam*rhop, the numerator of setvset.f90:104
  double cd100;     // Wilson
  // Ganser: sqrt(num); num^(1/2)*diam*rk1*rk2; 24*rk2/that; rk2*24*0.1118; rk2*0.4305; rk2
  double ft, fg, fi, fp, fq, rk2;
  int ok;           // get_gama converged
};

// Sources/setpsi.f90:65-127
__device__ int get_gama_dev(double diam, double sphe, double& gama) {
  const double d = diam * 1e3;
  const double toler = 1e-8;
  double gmin = 1e-3, gmax = 1.0;
  const double pi = 4.0 * atan(1.0);
  const double h = 0.5 * d;
  const double Vp = 4.0 * pi * (h * h * h) / 3.0;
  const double Ap = pow(pi, 1.0 / 3.0) * pow(6.0 * Vp, 2.0 / 3.0) / sphe;
  gama = 0.0;
  for (int it = 1; it <= 1000; ++it) {
    gama = 0.5 * (gmin + gmax);
    const double e = acos(gama);
    const double Ao = 0.5 * pi * d * d * pow(gama, -4.0 / 3.0) * (gama * gama + (e / tan(e)));
    if (Ao < Ap)
      gmax = gama;
    else
      gmin = gama;
    if ((it > 1) && (fabs(Ao - Ap) < toler)) return it;
  }
  return -1;
}

__global__ void k_class_consts(int np, int modv, const double* diam, const double* rhop,
                               const double* psi, const double* sphe, ClassConst* cc) {
  const int ic = blockIdx.x * blockDim.x + threadIdx.x;
  if (ic >= np) return;
  const double gi = 9.81;
  ClassConst k;
  k.diam = diam[ic];
  k.rhop = rhop[ic];
  k.psi = psi[ic];
  k.num = 4.0 * gi * k.diam * k.rhop;
  k.cd100 = k.ft = k.fg = k.fi = k.fp = k.fq = k.rk2 = 0.0;
  k.ok = 1;
  if (modv == 2) {
    double gama;
    if (get_gama_dev(k.diam, sphe[ic], gama) < 0) k.ok = 0;
    // gama**(-2.0/3.0): binary32 exponent (setvset.f90:120)
    const double dnd = 0.5 * (1.0 + gama) * pow(gama, (double)(-2.0f / 3.0f));
    const double rk1 = 1.0 / (dnd / 3.0 + 2.0 / (3.0 * sqrt(k.psi)));
    k.rk2 = pow(10.0, 1.8148 * pow(-log10(k.psi), 0.5743));
    k.ft = sqrt(k.num);
    // ft*diam*rk1*rk2 and 24*rk2/that rounded once (products and quotient in
    // double-double): their errors would be the same in every cell of a class
    double h = k.ft * k.diam, l = fma(k.ft, k.diam, -h);
    for (const double f : {rk1, k.rk2}) {
      const double p = h * f;
      l = fma(h, f, -p) + l * f;
      h = p;
    }
    k.fg = h + l;
    l = l - (k.fg - h);
    const double n = 24.0 * k.rk2, q = n / k.fg;
    k.fi = q + (fma(-q, k.fg, n) + fma(24.0, k.rk2, -n) - q * l) / k.fg;
    k.fp = k.rk2 * (24.0 * 0.1118);
    k.fq = k.rk2 * 0.4305;
  } else if (modv == 3) {
    k.cd100 = 0.24 * pow(k.psi, -0.828) + 2.0 * sqrt(1.0 - k.psi);
  }
  cc[ic] = k;
}

// A Ganser call (setvset.f90:117-136) between iterations.  With
// R = rey*rk1*rk2 = G*v and v = T/sqrt(cd),
//   cd = 24/(rey*rk1)*(1 + 0.1118*R^0.6567) + 0.4305*rk2/(1 + 3305/R)
//      = rk2*(24*0.1118*R^(0.6567-1) + 24/R + 0.4305*R/(R + 3305)),
// and 24/R = 24/(G*T)*cd*(1/sqrt(cd)).  y = 1/sqrt(cd) is carried: it gives
// v, R and 24/R of an iteration, the result T*y after the last one, and the
// next call's first v.  The cell's factors come from k_visc (cf.x =
// sqrt(1/(3*rhoa)), cf.y = cf.x*rhoa/visc, ci = 1/cf.y), the class's from
// k_class_consts.
struct GanserCell {
  double T, g, i;  // v = T*y, R = g*y, rk2*24/R = i*(cd*y)
};
__device__ __forceinline__ bool mid_range(double x) {  // 2^-1000 <= x < 2^1000 (positive)
  return (unsigned)(__double2hiint(x) - 0x01700000) < 0x7d000000u;
}
// an argument outside the fast functions' ranges
__device__ __noinline__ double ganser_cd_slow(double rk2, double R) {
  const double Q = R + 3305.0, N = fma(0.4305 * R, R, 24.0 * Q);
  return rk2 * fma(24.0 * 0.1118, pow(R, kPowA), N / (R * Q));
}
static __device__ __noinline__ double rsqrt_slow(double x) { return rsqrt(x); }
__device__ __forceinline__ double ganser_rsqrt(double cd) { return mid_range(cd) ? rsqrt_fast(cd) : rsqrt_slow(cd); }
__device__ __forceinline__ void ganser_step(const ClassConst& k, const GanserCell& c, const PowTab& tab, double& cd,
                                            double& y, double& v) {
  v = c.T * y;
  const double R = c.g * y;
  if (pow_in_range(R) && mid_range(cd)) {
    const double u = R * rcp_fast(R + 3305.0);
    cd = fma(k.fp, pow_a(tab, R), fma(k.fq, u, c.i * (cd * y)));
  } else {
    cd = ganser_cd_slow(k.rk2, R);
  }
  y = ganser_rsqrt(cd);
}
// |v - vold| <= 1e-3 on the magnitude bits (the same order for non-negative
// values; a NaN difference is above it as in binary64)
__device__ __forceinline__ bool ganser_done(double v, double vold) {
  return (dbits(v - vold) & 0x7fffffffffffffffLL) <= dbits(1e-3);
}

// Sources/setvset.f90:65-181 for one call of the other drag models; returns
// iterations (0 for the closed-form Dellino model) or -1 when maxit is
// reached.
__device__ int vsettl_dev(const ClassConst& k, int model, double rhoa, double visc, double& cd, double& vset) {
  const double eps = 1e-3;
  double vold = 1e5, v = 0.0;
  if (model == 4) {
    const double gi = 9.81, diam = k.diam;
    v = pow((diam * diam * diam * gi * (k.rhop - rhoa) * rhoa * pow(k.psi, 1.6)) / (visc * visc),
            0.5206);
    vset = (1.2065 * visc * v) / (diam * rhoa);
    return 0;
  }
  for (int it = 1; it <= 100; ++it) {
    v = sqrt(k.num / (3.0 * cd * rhoa));
    const double rey = rhoa * v * k.diam / visc;
    if (model == 1) {
      if (rey <= 988.947)
        cd = 24.0 / rey * (1.0 + 0.15 * pow(rey, 0.687));
      else
        cd = 0.44;
    } else {  // model 3
      if (rey <= 100.0) {
        cd = 24.0 / rey * pow(k.psi, -0.828) + 2.0 * sqrt(1.0 - k.psi);
      } else if (rey > 100.0 && rey < 1000.0) {
        const double a = (1.0 - k.cd100) / 900.0;
        const double b = 1.0 - 1000.0 * a;
        cd = a * rey + b;
      } else {
        cd = 1.0;
      }
    }
    if (it > 1 && fabs(v - vold) <= eps) {
      vset = sqrt(k.num / (3.0 * cd * rhoa));
      return it;
    }
    vold = v;
  }
  vset = v;
  return -1;
}

struct ChainGeom {
  Dims d;
  long long L;    // np * nx * ny * nz
  long long S;    // segment length
  long long W;    // warm-up length
  long long nseg;
};

// chain position q -> (ic, i, j, k) with k fastest (setvset.f90:25-33)
__device__ __forceinline__ void chain_cell(const ChainGeom& g, long long q, int& ic, long long& m) {
  const int nz = g.d.nz, ny = g.d.ny, nx = g.d.nx;
  const int k = (int)(q % nz) + 1;
  long long r = q / nz;
  const int j = (int)(r % ny) + 1;
  r /= ny;
  const int i = (int)(r % nx) + 1;
  ic = (int)(r / nx);
  m = g.d.M(i, j, k);
}

__device__ __forceinline__ double sutherland(double T) {
  const double visc0 = 1.827e-5;
  const double Tair0 = (double)291.15f;  // default-real literal (setvset.f90:23)
  const double t = T / Tair0;
  return visc0 * ((Tair0 + 120.0) / (T + 120.0)) * (t * sqrt(t));  // t**1.5
}

// The air viscosity of every cell, shared by all classes (setvset.f90:95-97),
// or for the Ganser iteration (model 2) its cell factors: with
// f = sqrt(1/(3*rho)) and g = f*rho/visc, cf = (f, g) and 1/g in visc.
__global__ void k_visc(long long s3, int modv, const double* tempe, const double* rho, double* visc, double2* cf) {
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < s3;
       m += (long long)gridDim.x * blockDim.x) {
    const double vs = sutherland(tempe[m]), r = rho[m];
    if (modv == 2) {
      const double f = sqrt(1.0 / (3.0 * r)), g = f * r / vs;
      cf[m] = make_double2(f, g);
      visc[m] = 1.0 / g;
    } else {
      visc[m] = vs;
    }
  }
}

// What a chain run reads and writes.
struct ChainIO {
  const ClassConst* cc;
  const double* visc;
  const double2* cf;
  const double* rho;
  double* vset;
  int* iters;
};

// Runs chain cells [q0, q1) from cd; writes -vset (setvset.f90:60) and the
// iteration counts when `write`.
__device__ void chain_run(const ChainGeom& g, long long q0, long long q1, int modv, const ChainIO& io, double& cd,
                          bool write, int& nonconv) {
  const long long s3 = g.d.cells();
  for (long long q = q0; q < q1; ++q) {
    int ic;
    long long m;
    chain_cell(g, q, ic, m);
    double v;
    const int it = vsettl_dev(io.cc[ic], modv, io.rho[m], io.visc[m], cd, v);
    if (write) {
      io.vset[(long long)ic * s3 + m] = -v;
      if (io.iters) io.iters[(long long)ic * s3 + m] = it;
      if (it < 0 || !io.cc[ic].ok) nonconv = 1;
    }
  }
}

// The same for the Ganser model, cells q0 <= q < q1 written from qw on: one
// loop over the iterations of all cells, in which a thread goes on to its
// next cell when it is done with one, so that the lanes of a warp need not
// wait for the one with the most iterations at every cell.  The next cell's
// factors are loaded while the current one iterates.
__device__ void chain_run_ganser(const ChainGeom& g, long long q0, long long qw, long long q1, const ChainIO& io,
                                 const PowTab& tab, double& cd, double& cd_w, int& nonconv) {
  if (q0 >= q1) return;
  const long long s3 = g.d.cells(), pl = g.d.plane();
  const int nz = g.d.nz;
  int ic;
  long long m, q = q0;
  chain_cell(g, q, ic, m);
  int left = nz - (int)(q % nz);  // cells of this column from q on
  ClassConst k = io.cc[ic];
  auto factors = [&](double2 f, double fi) { return GanserCell{k.ft * f.x, k.fg * f.y, k.fi * fi}; };
  GanserCell c = factors(io.cf[m], io.visc[m]);
  int icn = ic;  // the next cell, its class and factors
  long long mn = m;
  double2 fn;
  double fin;
  auto look = [&]() {
    if (q + 1 >= q1) return;
    if (left > 1) {
      mn = m + pl;
    } else {
      chain_cell(g, q + 1, icn, mn);
    }
    fn = io.cf[mn];
    fin = io.visc[mn];
  };
  look();
  double y = ganser_rsqrt(cd), vold = 1e5, v;
  int it = 0;
  if (q == qw) cd_w = cd;
  for (;;) {
    ++it;
    ganser_step(k, c, tab, cd, y, v);
    const bool done = it > 1 && ganser_done(v, vold);
    vold = v;
    if (!done && it < 100) continue;
    if (q >= qw) {
      io.vset[(long long)ic * s3 + m] = done ? -(c.T * y) : -v;
      if (io.iters) io.iters[(long long)ic * s3 + m] = done ? it : -1;
      if (!done || !k.ok) nonconv = 1;
    }
    if (++q >= q1) break;
    if (q == qw) cd_w = cd;
    left = left > 1 ? left - 1 : nz;
    m = mn;
    if (icn != ic) {
      ic = icn;
      k = io.cc[ic];
    }
    c = factors(fn, fin);
    it = 0;
    vold = 1e5;
    look();
  }
}

// Segment s of the chain: its entry cd (the chain's state for the first
// segment, else the value a warm-up of W cells from cd = 1 reaches), its
// cells and its exit cd.
__device__ __forceinline__ void chain_segment(const ChainGeom& g, long long s, int modv, const ChainIO& io,
                                              const double* cd_state, double* entry, double* exitv, int* nonconv,
                                              const PowTab& tab) {
  const long long q0 = s * g.S, q1 = min(g.L, q0 + g.S), qs = s == 0 ? 0 : max(0LL, q0 - g.W);
  double cd = s == 0 ? *cd_state : 1.0, cd0 = cd;
  int nc_flag = 0, dummy = 0;
  if (modv == 2) {
    chain_run_ganser(g, qs, q0, q1, io, tab, cd, cd0, nc_flag);
  } else {
    chain_run(g, qs, q0, modv, io, cd, false, dummy);
    cd0 = cd;
    chain_run(g, q0, q1, modv, io, cd, true, nc_flag);
  }
  entry[s] = cd0;
  exitv[s] = cd;
  nonconv[s] = nc_flag;
}

// One segment per thread; a segment's result does not depend on the thread
// or block that computes it.
__global__ void __launch_bounds__(64, 8)
    k_chain_segments(ChainGeom g, int modv, ChainIO io, const double* cd_state, double* entry, double* exitv,
                     int* nonconv) {
  __shared__ PowTab tab;
  pow_tab_init(tab);
  __syncthreads();
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= g.nseg) return;
  chain_segment(g, s, modv, io, cd_state, entry, exitv, nonconv, tab);
}

// The same segments computed beside the step kernel (a look-ahead meteo
// update on a second stream): blocks of four warps, one per SM sub-partition.
// Only the first block that starts on an SM works (claim[smid]); later ones on
// the same SM return at once, so that an SM idle at launch time does not fill
// up with chain blocks and shut the steps out.  The working blocks take
// segments from a counter until none is left.
__global__ void __launch_bounds__(128, 8)
    k_chain_beside(ChainGeom g, int modv, ChainIO io, const double* cd_state, double* entry, double* exitv,
                   int* nonconv, int* claim, unsigned long long* next) {
  __shared__ PowTab tab;
  __shared__ int mine;
  if (threadIdx.x == 0) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    mine = atomicCAS(claim + (smid & 255u), 0, 1) == 0;
  }
  __syncthreads();
  if (!mine) return;
  pow_tab_init(tab);
  __syncthreads();
  for (;;) {
    const unsigned long long s = atomicAdd(next, 1ULL);
    if (s >= (unsigned long long)g.nseg) break;
    chain_segment(g, (long long)s, modv, io, cd_state, entry, exitv, nonconv, tab);
  }
}

// Collects segments whose speculative entry differs from the predecessor's exit.
__global__ void k_chain_check(ChainGeom g, const double* entry, const double* exitv, int* bad,
                              int* nbad, int cap) {
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s < 1 || s >= g.nseg) return;
  if (dbits(entry[s]) != dbits(exitv[s - 1])) {
    const int slot = atomicAdd(nbad, 1);
    if (slot < cap) bad[slot] = (int)s;
  }
}

// Sequential repair in chain order (single thread).  Segments verified above
// stay; a recomputed segment may change its exit, so its successor is
// re-checked until the chain agrees again.  cap overflow -> full scan.
__global__ void k_chain_fix(ChainGeom g, int modv, ChainIO io, double* entry, double* exitv, int* nonconv, int* bad,
                            const int* nbad, int cap, double* cd_state) {
  __shared__ PowTab tab;
  if (*nbad > 0) pow_tab_init(tab);
  __syncthreads();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const int nb = *nbad;
  if (nb > 0) {
    const bool full = nb > cap;
    int cnt = full ? 0 : nb;
    // insertion sort of the (few) bad segment ids
    for (int a = 1; a < cnt; ++a) {
      const int v = bad[a];
      int b = a - 1;
      while (b >= 0 && bad[b] > v) {
        bad[b + 1] = bad[b];
        --b;
      }
      bad[b + 1] = v;
    }
    long long s = full ? 1 : bad[0];
    int next = 1;  // index into bad[] of the next listed segment after s
    while (s < g.nseg) {
      const double expect = exitv[s - 1];
      if (dbits(entry[s]) != dbits(expect)) {
        double cd = expect;
        int nc_flag = 0;
        entry[s] = cd;
        const long long q0 = s * g.S, q1 = min(g.L, q0 + g.S);
        double cd0;
        if (modv == 2)
          chain_run_ganser(g, q0, q0, q1, io, tab, cd, cd0, nc_flag);
        else
          chain_run(g, q0, q1, modv, io, cd, true, nc_flag);
        exitv[s] = cd;
        nonconv[s] = nc_flag;
        ++s;  // the successor must be re-checked
        continue;
      }
      if (full) {
        ++s;
        continue;
      }
      while (next < cnt && bad[next] <= s) ++next;
      if (next >= cnt) break;
      s = bad[next];
    }
  }
  *cd_state = exitv[g.nseg - 1];
}

__global__ void k_chain_status(ChainGeom g, const int* nonconv, int* status) {
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s < g.nseg && nonconv[s]) atomicOr(status, 1);
}

// f3d_dmath_eval; ops 4 to 6: the Ganser iteration's power, 1/sqrt and 1/x
__global__ void k_dmath_eval(int op, long long n, const double* x, double* y) {
  __shared__ DMathTab tab;
  __shared__ PowTab pow_tab;
  dmath_tab_init(tab);
  pow_tab_init(pow_tab);
  __syncthreads();
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    const double v = x[op == 2 ? 2 * q : q];
    y[q] = op == 0   ? dm_log(tab, v)
           : op == 1 ? dm_exp(tab, v)
           : op == 2 ? div_rn_recip(v, x[2 * q + 1], 1.0 / x[2 * q + 1])
           : op == 4 ? (pow_in_range(v) ? pow_a(pow_tab, v) : pow(v, kPowA))
           : op == 5 ? ganser_rsqrt(v)
                     : (mid_range(v) ? rcp_fast(v) : 1.0 / v);
  }
}

void launch_dmath_eval(int op, long long n, const double* x, double* y, cudaStream_t s) {
  if (n <= 0) return;
  k_dmath_eval<<<(unsigned)std::min<long long>((n + 255) / 256, 152LL * 8), 256, 0, s>>>(op, n, x, y);
  count_launch();
}

// setvset.f90:48-60 for the gas classes np+1..nc, which the chain does not
// touch: the aggregate loop multiplies class np+1 (a gas class with vset = 0
// when nc > np), then vset = -vset over all classes.  They keep their previous
// value (zero of alternating sign, as the reference negates the whole array
// at every update).
__global__ void k_vset_finish(long long s3, int nc, int np, int aggregate, double vset_factor,
                              double* vset) {
  const long long n = s3 * (nc - np);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
       q += (long long)gridDim.x * blockDim.x) {
    double* v = vset + (long long)np * s3 + q;
    *v = -(aggregate && q < s3 ? vset_factor * *v : *v);
  }
}

static ChainGeom chain_geom(Dims d, int np, int modv) {
  ChainGeom g;
  g.d = d;
  g.L = d.cells() * np;
  g.W = 64;
  // The segments are the threads of one launch.  Every one costs the W cells of
  // its warm-up and the longest ends the launch (2 to 6 iterations per cell by
  // class): segments of about 256 cells, but no fewer than 8 warps per SM hold, and
  // at most 12 warps' worth.  Whole columns of an iterating model, so that the
  // lanes of a warp go through the levels together; the closed form reads in order
  // with segments of any length.  Update, ms, with segments of 1024 cells and 3 warps
  // at least, with 256 and 8, and with whole columns:
  //   300x220x30, 8 classes: Ganser 7.5, 6.2, 5.3; Wilson 29.1, 20.4, 16.0; Dellino 10.0, 7.5, 8.1
  //   243x191x37, 11:        Ganser 9.5, 7.3, 5.5; Wilson 43.0, 27.1, 16.9; Dellino  9.9, 8.5, 8.7
  //   400x300x50, 16:        Ganser 24.2, 24.2, 21.3; Wilson 88.1, 88.1, 69.6 (12 warps in all cases)
  const long long warp_row = 32LL * sms();
  const long long n = std::min(12 * warp_row, std::max(8 * warp_row, g.L / 256));
  g.S = std::max<long long>(64, (g.L + n - 1) / n);
  if (modv != 4) g.S = (g.S + d.nz - 1) / d.nz * d.nz;
  g.nseg = (g.L + g.S - 1) / g.S;
  return g;
}

static constexpr int kBadCap = 8192;

// The regions of launch_setvset's scratch, each on a 256-byte boundary (so
// that what a caller puts behind them is aligned too).
static constexpr size_t region(size_t bytes) { return (bytes + 255) & ~size_t(255); }

size_t setvset_scratch_bytes(Dims d, int np) {
  const ChainGeom g = chain_geom(d, np, 4);  // the model with the most segments
  return region(sizeof(ClassConst) * (size_t)(np + 1)) + 2 * region(sizeof(double) * (size_t)g.nseg) +
         region(sizeof(int) * (size_t)g.nseg) + region(sizeof(int) * 8) + region(sizeof(int) * kBadCap) +
         region(sizeof(double) * (size_t)d.cells()) + region(2 * sizeof(double) * (size_t)d.cells()) +
         region(sizeof(int) * 256) + region(sizeof(unsigned long long));
}

void launch_setvset(Dims d, int nc, int np, int modv, const double* diam, const double* rhop,
                    const double* psi, const double* sphe, const double* tempe,
                    const double* rho, int aggregate, double vset_factor, double* vset,
                    int* iters, double* cd_state, void* scratch, int* status, cudaStream_t s,
                    int beside_step, int have_classes) {
  const ChainGeom g = chain_geom(d, np, modv);
  unsigned char* p = reinterpret_cast<unsigned char*>(scratch);
  auto take = [&](size_t bytes) {
    unsigned char* r = p;
    p += region(bytes);
    return r;
  };
  ClassConst* cc = reinterpret_cast<ClassConst*>(take(sizeof(ClassConst) * (size_t)(np + 1)));
  double* entry = reinterpret_cast<double*>(take(sizeof(double) * (size_t)g.nseg));
  double* exitv = reinterpret_cast<double*>(take(sizeof(double) * (size_t)g.nseg));
  int* nonconv = reinterpret_cast<int*>(take(sizeof(int) * (size_t)g.nseg));
  int* nbad = reinterpret_cast<int*>(take(sizeof(int) * 8));
  int* bad = reinterpret_cast<int*>(take(sizeof(int) * kBadCap));
  double* visc = reinterpret_cast<double*>(take(sizeof(double) * (size_t)d.cells()));
  double2* cf = reinterpret_cast<double2*>(take(2 * sizeof(double) * (size_t)d.cells()));
  int* claim = reinterpret_cast<int*>(take(sizeof(int) * 256));
  unsigned long long* next = reinterpret_cast<unsigned long long*>(take(sizeof(unsigned long long)));
  cudaMemsetAsync(nbad, 0, sizeof(int), s);
  cudaMemsetAsync(status, 0, sizeof(int), s);
  if (np > 0 && g.L > 0) {
    if (!have_classes) {
      k_class_consts<<<(np + 31) / 32, 32, 0, s>>>(np, modv, diam, rhop, psi, sphe, cc);
      count_launch();
    }
    k_visc<<<(int)std::min<long long>((d.cells() + 255) / 256, 152LL * 16), 256, 0, s>>>(d.cells(), modv, tempe,
                                                                                         rho, visc, cf);
    const ChainIO io{cc, visc, cf, rho, vset, iters};
    const int bs = 64;
    const long long nb = (g.nseg + bs - 1) / bs;
    if (beside_step) {
      // an SM holding this block must still take a step-kernel block
      static const cudaError_t carveout = cudaFuncSetAttribute(
          k_chain_beside, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      (void)carveout;
      cudaMemsetAsync(claim, 0, sizeof(int) * 256, s);
      cudaMemsetAsync(next, 0, sizeof(unsigned long long), s);
      k_chain_beside<<<(unsigned)(4 * sms()), 128, 0, s>>>(g, modv, io, cd_state, entry, exitv, nonconv, claim,
                                                                 next);
    } else {
      k_chain_segments<<<(unsigned)nb, bs, 0, s>>>(g, modv, io, cd_state, entry, exitv, nonconv);
    }
    k_chain_check<<<(unsigned)((g.nseg + 255) / 256), 256, 0, s>>>(g, entry, exitv, bad, nbad, kBadCap);
    k_chain_fix<<<1, 32, 0, s>>>(g, modv, io, entry, exitv, nonconv, bad, nbad, kBadCap, cd_state);
    k_chain_status<<<(unsigned)((g.nseg + 255) / 256), 256, 0, s>>>(g, nonconv, status);
    count_launch(5);
  }
  if (nc > np) {
    const long long n = d.cells() * (nc - np);
    k_vset_finish<<<(int)std::min<long long>((n + 255) / 256, 152LL * 16), 256, 0, s>>>(
        d.cells(), nc, np, aggregate, vset_factor, vset);
    count_launch();
  }
}

}  // namespace f3d
