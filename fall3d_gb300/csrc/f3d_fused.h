// f3d_fused.h -- arguments of the precision form's fused step kernel.
#pragma once

#include <cuda.h>  // CUtensorMap (types only; the encoder is reached through the runtime)

#include "f3d_internal.h"

namespace f3d {

// Per-level factors of the step (binary32, rounded once from binary64), with
// dzz = 2/(dz(k)+dz(k-1)) of advctzc.f90:34 and diffz.f90:25.
struct ZTab {
  float a, b;     // lim_coef_z: dt/4*dz(k-1)*dzz, dt^2/8*dzz
  float rdz;      // 1/dz(k): the slope between k and k+1
  float dtdzz;    // dt*dzz
  float dtrdz;    // dt/dz(k)
  float pad[3];
};

// Fields of the step kernel, filled at every meteo update.  3-D fields have
// the halo layout of the precision form's c: rows of d.px values (nx+2
// rounded up to a multiple of 4, so that tensor copies can stage them),
// planes 0..nz+1; ghost rows and columns hold what makes the interior
// formulas give the reference's boundary faces.
struct StepFields {
  float* ux;  // Courant velocity vx*dt/dX1, ghost columns = the adjacent cell's
  float* kx;  // limiter coefficient of work(i,2), advctx.f90:40-43: 0.5*C*(1-C), C = 0.5*|ux(i)+ux(i-1)|
  float* uy;  // vy*dt/dX2, ghost rows = the adjacent cell's
  float* ky;
  float* l;   // 1/rho, ghosts = the adjacent cell's
  float* fx;  // face (i,i+1): 0.5*dt/dX1^2*(P(i)+P(i+1)), P = rkh1*rho; faces 0 and nx: dt/dX1^2*P(1), P(nx)
  float* fy;  // face (j,j+1) likewise, P = rkhor*rho
  float* fz;  // face (k,k+1): 0.5*(P(k)+P(k+1))/dz(k), P = rkver*rho; plane 0: P(1)/dz(0),
              // plane nz: P(nz)/dz(nz), plane nz+1: P(nz-1)/dz(nz-1)
  float* vk;  // vz+vset, class blocks
  // the faces of the first and last cells on their inner side, which the
  // reference does not average (diffx.f90:22-33, 44-55): dt/dX1^2*P(2) and
  // P(nx-1) at [side][k][j] (nz+2 planes of ny+2), dt/dX2^2*P(2), P(ny-1) at
  // [side][k][i] (nz+2 planes of px), P(2)/dz(1) of diffz at [j][i] (px)
  float *ex, *ey, *ez;
  ZTab* tab;  // levels 0..nz+1
};

struct FusedArgs {
  const float* c_in;  // class blocks of d.halo() values, after setsrc
  float* c_out;       // same layout; receives the step's result incl. ghosts
  long long cstride;
  Dims d;
  int ncls;
  int xfirst;  // iiter even: x before y (sizloop.f90:42-48)
  // the column is cut into nchunk pieces marched by different blocks: levels
  // 1..kfirst, then pieces of klen levels
  int nchunk, kfirst, klen;
  double dt64;
  StepFields f;
  const float* vdep;  // class blocks of nx*ny
  const float* rkver1;  // rkver(:,:,1) (setbcc bottom)
  float dz0;
  // binary64 deposits
  const unsigned char* wet_class;  // per class: wet deposition applies (or NULL)
  const double* lambda2d;          // min(dt*a*prate^b,1) per column
  const double* zi;
  const double* zlayer;
  const double* dz64;
  double* cwet;  // (nx,ny,0:nc)
  double* cdry;
  const double* vset64;  // class blocks of nx*ny*nz
  const double* vdep64;  // class blocks of nx*ny
  int* status;           // device status word: F3D_STEP_STAGING_TIMEOUT is or-ed into it
};

// a staging wait of the step kernel gave up (a tensor copy did not arrive)
#define F3D_STEP_STAGING_TIMEOUT 0x100

// Tensor maps of a context's met fields and of a state buffer for the step
// kernel's tensor copies: boxes of 68 values (x) by the tile region's rows by
// one plane.  [0]: 32-row boxes, [1]: 16-row boxes.
struct F2Maps {
  enum { VK = 0, UX, KX, UY, KY, L, FZ, FX, FY, N };
  CUtensorMap m[2][N];
};
struct CMaps {
  CUtensorMap m[2];
};
// 0 on success
int make_step_maps(const FusedArgs& a, F2Maps* out);
int make_c_maps(Dims d, int ncls, const float* c, CMaps* out);
// the largest nz whose per-level table fits into the step kernel's shared memory,
// for a context's own step or in a batch (whose kernel keeps tables of its own)
int fused2_max_nz(bool batch);
inline int halo_pitch(int nx) { return (nx + 2 + 3) & ~3; }

// How a context's column is cut (nchunk, kfirst, klen) so that the tiles of
// all classes fill the device: nwet = highest level any wet deposition
// reaches (0: none), which the first piece must hold.  batch_items: the uncut
// tiles of all classes of all scenarios of the launch (0: its own); a batch
// that fills the device gains nothing from pieces, which cost four iterations
// each (64 members of 64..320 by 64..320 cells: 10.2 ms per step, cut as for
// launches of their own 10.7 ms).
void step_chunks(FusedArgs& a, int shape, int nwet, long long batch_items);

// Tile shapes (F3D_OPT_TILE), region x by y / threads: 0, 1 and 2 = 64x16 /
// 512 (a row per warp, two blocks per SM), 3 = 64x32 / 512 (two rows per
// warp); two columns per lane.  Results do not depend on the shape.
// step_shape: the faster one for a launch of its own, where none was set.
int step_shape(Dims d, int ncls);
// beside: a look-ahead meteo update may run at the same time.
void launch_step_fused(const FusedArgs& a, const F2Maps& maps, const CMaps& c, int shape, cudaStream_t s,
                       bool beside = false);
// The step kernel's fields from the scaled binary64 fields of a meteo update
// whose finddt maximum is at *dtcn (dt = safety/max(dtcn,1e-13)).
void launch_step_fields(Dims d, int nc, double safety, double dX1, double dX2, const double* dz,
                        const unsigned long long* dtcn, const double* vx, const double* vy, const double* vz,
                        const double* rho, const double* rkh1, const double* rkhor, const double* rkver,
                        const double* vset, const StepFields& f, cudaStream_t s);
// vz+vset of one class block
void launch_step_vk(Dims d, int nc, const double* vz, const double* vset, float* vk, cudaStream_t s);
// tiles of one class of an nx x ny grid for a tile shape
int fused_tiles(int nx, int ny, int shape);

// Batched form: a persistent launch per sweep order over the work items of all
// scenarios (at most F3D_BATCH_MAX) that take it.  args: device array of the
// scenarios' arguments, whose c_in / c_out are the scenario's two buffers; counter: two.
#define F3D_BATCH_MAX 128
struct BatchMaps {  // a scenario's tensor maps (device array in batch order)
  F2Maps met;
  CMaps a, b;
};
// sets the kernels' shared-memory limit (that of the longest column) and returns their persistent grid (-1 on error)
int fused_batch_grid(int shape, int max_nz);
void launch_step_fused_batch(int shape, int grid, const FusedArgs* args, const int* item_off, int nscen, int* counter,
                             const int* bstep, const int* iiter0, int commit, int max_nz, const BatchMaps* maps,
                             cudaStream_t s);
void launch_wet_lambda(long long n, double dt, const double* prate, double* lam, cudaStream_t s);

}  // namespace f3d
