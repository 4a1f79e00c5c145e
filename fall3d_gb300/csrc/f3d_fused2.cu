// f3d_fused2.cu -- the precision form's whole transport step in one kernel.
//
// One block owns an output tile of one class and marches up the column (or a
// piece of it), so each concentration is read from and written to HBM once
// per step.  The sweeps of Sources/sizloop.f90:35-71 are pipelined per
// horizontal plane; iteration t runs
//
//   A  setbcc + advctzc   plane t, per column in registers (window of the
//                         original column c(t), c(t+1), c(t+2) and the flux
//                         difference of the face below)
//   B  advctx / advcty    plane t; x: warp shuffles along a row; y: the
//                         lane's own rows and shared memory
//   C  diffz              plane k = t-1 (needs plane t of B)
//   D  diffx / diffy      plane k
//   E  wetdep, accum, clip, store (plane k)
//
// A lane owns two neighbouring columns (every field of a position pair is one
// 64-bit value), a warp HY/NW adjacent rows of the 64 x HY tile region.  The
// x/y sweeps need +-2 cells (advection) then +-1 (diffusion), so the output
// tile is 58 x (HY-6); halo cells are recomputed by neighbouring blocks.  The
// ghost cells of setbcc are formed from the original column
// (setbcc.f90:53-83) and stay unchanged through the sweeps (the reference's
// stale ghosts).  Input and output are distinct buffers.
//
// Each advection sweep takes a cell's two upwind differences from one flux
// per face, F = u*c + K*minmod (u the Courant velocity, K the limiter's
// coefficient): c - (F(q) - F(q-1)) or c - (F(q+1) - F(q)); each diffusion
// sweep adds the difference of its two face fluxes.  Everything that does not
// depend on the class is part of the staged coefficients (StepFields); the
// boundary faces of the reference come from the coefficients' ghost values.
//
// Staging: the ten fields iteration t+1 reads (c two planes ahead, vz+vset
// one, the Courant velocities and limiter coefficients, 1/rho and the three
// face coefficients) arrive by tensor copies, in two buffers; one lane of each
// warp issues a field's box as soon as the last warp has read the field's
// buffer.  A box starts at the region's first column rounded down to a
// multiple of 4 values (16 bytes, what a tensor copy needs; the region then
// starts 0 or 2 values into it) and is 68 wide.
//
// What bounds it: 400x300x50 cells and 16 classes take 0.889 ms (1.255 ms
// before the flux form, the packed arithmetic, the coefficients formed at the
// meteo update and the shared-memory addressing), 1.32 GB of algorithmic bytes
// or 0.19 ms at the copy bandwidth.  A warp issues about 500 instructions per
// plane for its 128 positions, 200 of them binary32 arithmetic, at half the
// issue rate: with one block of 16 warps per SM (174 KB of staged fields, 128
// registers) the dependency chains of the sweeps and the three block barriers
// of a plane are not all covered.  The tensor copies bring 87 KB per plane and
// SM, 6.7 TB/s over the device; when the copies of t+1 were issued after
// iteration t's first barrier, waiting for them was the largest stall (0.999
// ms with c and vz+vset in a third buffer, 1.03 ms without; all fields issued
// after the iteration's last barrier 0.915 ms).
//
// Column pieces: a march over levels k0..k1 starts at t = k0-1 from the
// original column's planes k0-3..k0 (the advection fluxes of plane k0-1 need
// them), so pieces are independent of one another; they let grids with few
// tiles fill the device.  Every value is formed by the same operations
// whatever the tile shape or the pieces, so results do not depend on them.
#include <algorithm>
#include <type_traits>

#include "f3d_fused_math.cuh"

namespace f3d {

namespace {

using namespace fz;

constexpr int HX = 64, TX = HX - 6, RS = HX + 4;
constexpr int GUARD = 512;  // bytes before the staging area (reads one row above a field)

template <int HY_, int NW_>
struct Shape {
  static constexpr int HYR = HY_, NT = 32 * NW_, RPW = HY_ / NW_, TY = HY_ - 6, FS = RS * HY_,
                       NP = HX * HY_, MAP = HY_ == 32 ? 0 : 1, UNROLL = HY_ == 32 ? 1 : 2;
  static_assert(HY_ % NW_ == 0 && NW_ >= NF, "rows must divide among warps; a warp issues one field's copies");
};
constexpr int HY = 32, NW = 16;  // the default shape
using Tall = Shape<HY, NW>;
using Flat = Shape<16, 16>;

// value of the column to the left / right of each of the lane's two columns
__device__ __forceinline__ float2 left2(float2 v) { return make_float2(shup(v.y), v.x); }
__device__ __forceinline__ float2 right2(float2 v) { return make_float2(v.y, shdn(v.x)); }
__device__ __forceinline__ float& cmp(float2& v, int c) { return c ? v.y : v.x; }

__device__ __forceinline__ float2 lds2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ void sts2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ float2 ldg2(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }

template <class S>
size_t step_smem(int nz) {
  return GUARD + sizeof(float) * ((size_t)2 * NF * S::FS + 3 * (size_t)S::NP + HX) +
         sizeof(ZTab) * (size_t)(nz + 2) + 64;
}

// ------------------------------------------------ tensor copies (TMA)
__device__ __forceinline__ void mbar_init(unsigned bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// waits for the phase of the given parity, at most 4096 polls, each of which
// the hardware may suspend for up to a millisecond; false on a timeout
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  for (int i = 0; i < 4096; ++i) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(1000000)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load3(unsigned dst, const CUtensorMap* map, int x, int y, int z, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// One piece of the column of one tile of one class.  maps, cmap: tensor maps
// of the scenario's met fields and of c_in.  commit = 0 skips the deposit
// writes (cdry, cwet) so that the autotuner can time the kernel on a live
// state.
template <class S, bool XFIRST>
__device__ __forceinline__ void step_tile(const FusedArgs& a, const F2Maps* maps, const CMaps* cmap,
                                          const float* c_in, float* c_out, const int commit, const int cls,
                                          const int tile, const int chunk) {
  constexpr int RPW = S::RPW, TY = S::TY, FS = S::FS, NP = S::NP, NT = S::NT, HYR = S::HYR;
  // The block's shared memory, addressed from the array itself with no detour
  // through an integer or a parameter: the compiler then knows the address
  // space and emits shared-memory instructions with 32-bit addresses (with
  // generic ones the step of 400x300x50 cells, 16 classes took 1.125 ms
  // instead of 1.055 ms).
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* stage = reinterpret_cast<float*>(smem_raw + GUARD);  // [2][NF][FS], 128-byte aligned fields
  float* P0s = stage + 2 * NF * FS;                       // planes the y sweeps exchange rows through:
  float* Ws = P0s + NP;                                   // c, the advection flux, c/rho
  float* P1s = Ws + NP;
  ZTab* tab = reinterpret_cast<ZTab*>(P1s + NP + HX);
  // one per staging buffer
  unsigned long long* mbar = reinterpret_cast<unsigned long long*>(tab + (a.d.nz + 2));

  const Dims d = a.d;
  const int nx = d.nx, ny = d.ny, nz = d.nz;
  const int tiles_x = (nx + TX - 1) / TX;
  const int i0 = 1 + (tile % tiles_x) * TX, j0 = 1 + (tile / tiles_x) * TY;
  const int gx0 = i0 - 3, gy0 = j0 - 3;
  const int oi1 = min(nx, i0 + TX - 1), oj1 = min(ny, j0 + TY - 1);
  const int lane = threadIdx.x & 31, warp = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);  // uniform
  const int gi = gx0 + 2 * lane;       // the lane's first column (even); the second is gi + 1
  const int gj0 = gy0 + RPW * warp;    // the warp's first row
  const int px = d.px;                 // row pitch of c and of the fields (a multiple of 4)
  const int cs = px * (ny + 2);        // their plane
  const int xs = gx0 & ~3;             // first column of the staged boxes
  const int sft = gx0 - xs;            // the region's offset in a box row (0 or 2)
  const int pl = nx * ny;
  const bool edge = !(gx0 >= 1 && gx0 + HX - 1 <= nx && gy0 >= 1 && gy0 + HYR - 1 <= ny);
  const bool xedge = gx0 <= 1 || gx0 + HX - 1 >= nx;  // the region holds column 1 or nx
  // levels k0..k1 of the column, iterations ts..te
  const int k0 = chunk == 0 ? 1 : a.kfirst + 1 + (chunk - 1) * a.klen;
  const int k1 = chunk == 0 ? (a.nchunk > 1 ? a.kfirst : nz) : min(nz, k0 + a.klen - 1);
  const int ts = max(1, k0 - 1), te = k1 + 1;

  const unsigned mbar0 = (unsigned)__cvta_generic_to_shared(mbar);
  __shared__ int s_kzmax;  // the highest wet layer of the tile: above it the wet code is skipped
  if (threadIdx.x == 0) {
    mbar_init(mbar0, NF);
    mbar_init(mbar0 + 8, NF);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_kzmax = 0;
  }
  __syncthreads();

  // ------------------------------------------------ staging
  // The staged inputs of iteration t are in buffer (t-ts)&1.  Those of t+2
  // are issued during iteration t, a field's box after the block barrier that
  // follows every warp's last read of the field: the advection's fields after
  // the second barrier (early), the others, and x's when its sweep is the
  // second, after the last.  One barrier object per buffer: with one for each
  // of the two groups the wait is shorter but the second wait of a plane costs
  // more (0.961 ms against 0.889 ms at 400x300x50, 16 classes).  One lane of
  // warp f issues field f's box.  Outside the arrays it fills zeros; planes
  // outside 1..nz are not read and not copied.
  const unsigned stage0 = (unsigned)__cvta_generic_to_shared(stage);
  const bool issuer = lane == 0 && warp < NF;
  const int f_plane = field_plane(warp);
  const int f_z = warp <= F_VK ? cls * (nz + 2) : 0;
  const CUtensorMap* f_map = warp == F_C ? &cmap->m[S::MAP] : &maps->m[S::MAP][issuer ? warp - 1 : 0];
  const bool early = warp < F_L && (XFIRST || (warp != F_UX && warp != F_KX));
  auto prefetch = [&](const int t, const bool mine) {
    if (!issuer || !mine || t > te) return;
    const unsigned buf = (unsigned)(t - ts) & 1u, bar = mbar0 + 8u * buf;
    const int p = t + f_plane;
    // the warps' reads of this buffer (ordered before this point by a block
    // barrier) come before the tensor copy overwrites it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const bool ok = p >= 1 && p <= nz;
    mbar_expect(bar, ok ? (unsigned)(FS * sizeof(float)) : 0u);
    if (ok) tma_load3(stage0 + 4u * (buf * NF + warp) * FS, f_map, xs, gy0, f_z + p, bar);
  };
  bool timed_out = false;
  auto staged = [&](const int t) {
    if (!mbar_wait(mbar0 + 8u * ((unsigned)(t - ts) & 1u), (unsigned)((t - ts) >> 1) & 1u)) timed_out = true;
  };
  prefetch(ts, true);
  prefetch(ts + 1, true);

  for (int k = threadIdx.x; k < (nz + 2) * (int)(sizeof(ZTab) / 4); k += NT)
    reinterpret_cast<float*>(tab)[k] = __ldg(reinterpret_cast<const float*>(a.f.tab) + k);
  // wet deposition reaches only the first piece (step_chunks)
  const bool wet = a.wet_class && chunk == 0 && a.wet_class[cls];
  // zlayer is non-decreasing (checked on the host): the layers below the
  // mixing height are a prefix of the column (wetdep.f90:37)
  if (wet)
    for (int o = threadIdx.x; o < TX * TY; o += NT) {
      const int oi = i0 + o % TX, oj = j0 + o / TX;
      if (oi > oi1 || oj > oj1) continue;
      const double zi = a.zi[(oi - 1) + nx * (oj - 1)];
      int kz = s_kzmax;
      while (kz < nz && a.zlayer[kz] <= zi) ++kz;
      if (kz > 0) atomicMax(&s_kzmax, kz);
    }

  const float* __restrict__ cin = c_in + (long long)cls * a.cstride;
  float* __restrict__ cout = c_out + (long long)cls * a.cstride;
  const float* __restrict__ vkc = a.f.vk + (long long)cls * a.cstride;

  // ------------------------------------------------ per-position state
  // bit 2r+c: row r (gj0 + r), column c (gi + c) is an output cell; is stored
  // at the planes 1..nz (output cells and the tile's ghosts on the grid's faces)
  unsigned kout = 0, kst = 0;
#pragma unroll
  for (int r = 0; r < RPW; ++r) {
    const int gj = gj0 + r;
    const bool rows_out = gj >= j0 && gj <= oj1;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int g = gi + c;
      const bool cols_out = g >= i0 && g <= oi1;
      const unsigned bit = 1u << (2 * r + c);
      if (rows_out && cols_out) kout |= bit;
      if ((rows_out && ((g == 0 && i0 == 1) || (g == nx + 1 && oi1 == nx))) ||
          (cols_out && ((gj == 0 && j0 == 1) || (gj == ny + 1 && oj1 == ny))))
        kst |= bit;
    }
  }
  kst |= kout;
  // ghost columns of the lane's pair, ghost rows of the warp (uniform)
  const bool gx_0 = gi == 0 || gi == nx + 1, gx_1 = gi + 1 == nx + 1;
  auto ghost_row = [&](int r) { return gj0 + r == 0 || gj0 + r == ny + 1; };
  const bool pair_in = gi >= 0 && gi < px;  // the pair lies in the arrays' rows
  auto row_in = [&](int r) { return gj0 + r >= 0 && gj0 + r <= ny + 1; };
  const int h0 = gi + px * gj0;  // offset of the first row's pair at plane 0
  // original column c(t), c(t+1), vz+vset(t), slope(t) = (c(t+1)-c(t))/dz(t),
  // work(t,2), the flux difference below plane t; then the advected plane
  // t-1, 1/rho there, and the diffusive flux below it
  float2 o0[RPW], o1[RPW], vk[RPW], sl[RPW], w2[RPW], gk[RPW], gtop[RPW];
  float2 rb[RPW], lb[RPW], fp[RPW], gb[RPW], dqn[RPW], gy[RPW];

  __syncthreads();  // tables and wet state

  // ------------------------------------------------ the first plane's window
#pragma unroll
  for (int r = 0; r < RPW; ++r) {
    const int gj = gj0 + r, h = h0 + r * px;
    const float2 z2 = make_float2(0.0f, 0.0f);
    const bool in = pair_in && row_in(r);
    rb[r] = lb[r] = fp[r] = gb[r] = gtop[r] = dqn[r] = gy[r] = z2;
    auto C = [&](int k) { return in ? *reinterpret_cast<const float2*>(cin + h + k * cs) : z2; };
    auto V = [&](int k) { return in ? ldg2(vkc + h + k * cs) : z2; };
    const ZTab zt = tab[ts], zm = tab[ts - 1];
    o0[r] = C(ts);
    o1[r] = C(ts + 1);
    vk[r] = V(ts);
    const float2 pk = mul2(vk[r], o0[r]);
    sl[r] = mul2(sub2(o1[r], o0[r]), splat(zt.rdz));
    if (ts == 1) {  // the bottom ghost (setbcc.f90:19-33); work(0,2) = work(1,2)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int g = gi + c;
        if (g < 1 || g > nx || gj < 1 || gj > ny) continue;
        const int mb = (g - 1) + nx * (gj - 1);
        const float c1 = cmp(o0[r], c);
        float b = 0.0f;
        if (!(cmp(vk[r], c) >= 0.0f))
          b = c1 * (1.0f + a.dz0 * __ldg(a.vdep + (long long)cls * pl + mb) / __ldg(a.rkver1 + mb));
        cmp(gb[r], c) = b;
        if (kout >> (2 * r + c) & 1u) {
          cout[h + c] = clip0(b);  // clipped ghost (sizloop.f90:77)
          if (g == 1 && gj == 1) cout[d.C(0, 0, 0)] = clip0(c1);  // setbcc.f90:87-91
          if (g == nx && gj == 1) cout[d.C(nx + 1, 0, 0)] = clip0(c1);
          if (g == 1 && gj == ny) cout[d.C(0, ny + 1, 0)] = clip0(c1);
          if (g == nx && gj == ny) cout[d.C(nx + 1, ny + 1, 0)] = clip0(c1);
        }
      }
      // a NaN ghost (0/0 where the diffusivity is 0) counts as a positive
      // slope that the other one limits, as SIGN and MIN of a NaN do
      float2 s0 = mul2(sub2(o0[r], gb[r]), splat(zm.rdz));
      s0 = sel2(isnan(s0.x), isnan(s0.y), splat(__int_as_float(0x7f800000)), s0);
      w2[r] = mul2(lim_coef_z(vk[r], vk[r], zt.a, zt.b), minmod2(sl[r], s0));
      gk[r] = mul2(splat(zt.dtdzz), sub2(pk, mul2(vk[r], gb[r])));
    } else {  // ts >= 3: the planes below are inside the column
      const float2 cm = C(ts - 1), cmm = C(ts - 2), vm = V(ts - 1), vmm = V(ts - 2);
      const float2 s1 = mul2(sub2(o0[r], cm), splat(zm.rdz));
      const float2 s2 = mul2(sub2(cm, cmm), splat(tab[ts - 2].rdz));
      const float2 w2m = mul2(lim_coef_z(vm, vmm, zm.a, zm.b), minmod2(s1, s2));
      w2[r] = mul2(lim_coef_z(vk[r], vm, zt.a, zt.b), minmod2(sl[r], s1));
      gk[r] = fma2(splat(zt.dtdzz), sub2(pk, mul2(vm, cm)), sub2(w2[r], w2m));
    }
    // the adjacent row's c of plane ts, for a y-face ghost row
    if (edge && (gj == 0 || gj == ny + 1) && in)
      gy[r] = *reinterpret_cast<const float2*>(cin + h + (gj == 0 ? px : -px) + ts * cs);
  }

  // ------------------------------------------------ one iteration of the march
  const int kzmax = s_kzmax;
  auto plane = [&](auto edge_c, auto steady_c, const int t) {
    constexpr bool EDGE = decltype(edge_c)::value;
    constexpr bool STEADY = decltype(steady_c)::value;  // 3 <= t <= nz-2, plane t-1 is an output plane
    const int k = t - 1;
    // ghosts keep their value through the sweeps
    auto keep = [&](float2 out, float2 in, int r) {
      if constexpr (EDGE) {
        if (xedge) out = sel2(gx_0, gx_1, in, out);
        if (ghost_row(r)) out = in;
      }
      return out;
    };
    // inner faces of the grid's first and last columns and rows, plane k
    float ex[RPW];
    float2 ey[RPW];
    if constexpr (EDGE) {
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        const int gj = gj0 + r;
        ex[r] = 0.0f;
        ey[r] = make_float2(0.0f, 0.0f);
        if (k < k0) continue;
        // gi is even: column 1 is a pair's second
        if (xedge && (gi == 0 || gi == nx || gi + 1 == nx) && row_in(r))
          ex[r] = __ldg(a.f.ex + (gi == 0 ? 0 : (nz + 2) * (ny + 2)) + k * (ny + 2) + gj);
        if ((gj == 1 || gj == ny) && pair_in) ey[r] = ldg2(a.f.ey + (gj == 1 ? 0 : (nz + 2) * px) + k * px + gi);
      }
    }
    staged(t);
    const float* sb = stage + ((t - ts) & 1) * (NF * FS) + RPW * warp * RS + sft + 2 * lane;  // the row-0 pair
    auto at = [&](int field, int r) { return sb + field * FS + r * RS; };
    float2 s2[RPW];
    if (STEADY || t <= nz) {
      float2 s1[RPW];
      const ZTab zn = tab[(STEADY || t + 1 <= nz) ? t + 1 : nz];
      // ---------------- A: setbcc ghosts + advctzc for plane t
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        const int gj = gj0 + r;
        float2 gxv = make_float2(0.0f, 0.0f), gyv = gxv;
        if constexpr (EDGE) {
          if (xedge) {  // x-face ghosts from the neighbouring column's original c; their own ux is the
                        // neighbour's (setbcc.f90:53-66)
            const float2 u = lds2(at(F_UX, r));
            const float cl = shup(o0[r].y);
            gxv.x = gi == 0 ? (u.x >= 0.0f ? 0.0f : o0[r].y) : (u.x <= 0.0f ? 0.0f : cl);
            gxv.y = u.y <= 0.0f ? 0.0f : o0[r].x;
          }
          if (ghost_row(r)) {  // y-face ghosts (setbcc.f90:70-83)
            const float2 v = lds2(at(F_UY, r));
            const bool lo = gj == 0;
            gyv = sel2(lo ? v.x >= 0.0f : v.x <= 0.0f, lo ? v.y >= 0.0f : v.y <= 0.0f, gyv, gy[r]);
            if (t < min(te, nz) && pair_in)  // the next plane's
              gy[r] = *reinterpret_cast<const float2*>(cin + h0 + r * px + (lo ? px : -px) + (t + 1) * cs);
          }
        }
        {  // the column update, on every position
          float2 c2 = make_float2(0.0f, 0.0f), vkp = make_float2(0.0f, 0.0f), gn, w2n = w2[r], sln = sl[r];
          if (STEADY || t + 1 <= nz) {
            vkp = lds2(at(F_VK, r));
            if (STEADY || t + 2 <= nz) {
              c2 = lds2(at(F_C, r));
            } else {  // the top ghost (setbcc.f90:37-49), vkp = vk(nz)
              c2 = sel2(vkp.x <= 0.0f, vkp.y <= 0.0f, make_float2(0.0f, 0.0f), o1[r]);
              gtop[r] = c2;
#pragma unroll
              for (int c = 0; c < 2; ++c) {
                const int g = gi + c;
                if (kout >> (2 * r + c) & 1u) {
                  const float top = cmp(o1[r], c);
                  cout[h0 + r * px + c + (nz + 1) * cs] = clip0(cmp(c2, c));
                  if (g == 1 && gj == 1) cout[d.C(0, 0, nz + 1)] = clip0(top);
                  if (g == nx && gj == 1) cout[d.C(nx + 1, 0, nz + 1)] = clip0(top);
                  if (g == 1 && gj == ny) cout[d.C(0, ny + 1, nz + 1)] = clip0(top);
                  if (g == nx && gj == ny) cout[d.C(nx + 1, ny + 1, nz + 1)] = clip0(top);
                }
              }
            }
            sln = mul2(sub2(c2, o1[r]), splat(zn.rdz));
            w2n = mul2(lim_coef_z(vkp, vk[r], zn.a, zn.b), minmod2(sln, sl[r]));
            gn = fma2(splat(zn.dtdzz), sub2(mul2(vkp, o1[r]), mul2(vk[r], o0[r])), sub2(w2n, w2[r]));
          } else {  // t == nz: work(nz+1,1) (advctzc.f90:58-64), work(nz+1,2) = work(nz,2)
            gn = mul2(splat(zn.dtrdz), mul2(vk[r], sub2(gtop[r], o0[r])));
          }
          s1[r] = upwind(o0[r], vk[r], gk[r], gn);
          w2[r] = w2n;
          sl[r] = sln;
          gk[r] = gn;
          o0[r] = o1[r];
          o1[r] = c2;
          vk[r] = vkp;
        }
        if constexpr (EDGE) {
          if (xedge) s1[r] = sel2(gx_0, gx_1, gxv, s1[r]);
          if (ghost_row(r)) s1[r] = gyv;
        }
      }
      // ---------------- B: advctx (shuffles) and advcty (shared memory)
      auto adv_x = [&](const float2* in, float2* out) {
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
          const float2 c0 = in[r], u = lds2(at(F_UX, r)), cp = right2(c0);
          const float2 dc = sub2(cp, c0);
          const float2 wx = mul2(lds2(at(F_KX, r)), minmod2(dc, left2(dc)));
          const float2 F = fma2(u, c0, wx);
          float2 Fl = left2(F);
          if constexpr (EDGE) {
            if (xedge) {  // work(0,2) = work(1,2) (advctx.f90:48-50)
              if (gi == 0) Fl.y = __fmaf_rn(u.y, c0.x, wx.y);
            }
          }
          const float2 G = sub2(F, Fl);
          float2 Gp = right2(G);
          if constexpr (EDGE) {
            if (xedge) {  // work(n+1,1), work(n+1,2) = work(n,2) (advctx.f90:46, 52-54)
              if (gi == nx) Gp.x = __fsub_rn(__fmaf_rn(u.x, cp.x, wx.x), F.x);
              if (gi + 1 == nx) Gp.y = __fsub_rn(__fmaf_rn(u.y, cp.y, wx.y), F.y);
            }
          }
          out[r] = keep(upwind(c0, u, G, Gp), c0, r);
        }
      };
      auto adv_y = [&](const float2* in, float2* out) {
        float* P0 = P0s + RPW * warp * HX + 2 * lane;
        float* W = Ws + RPW * warp * HX + 2 * lane;
        sts2(P0, in[0]);
        if (RPW > 1) sts2(P0 + (RPW - 1) * HX, in[RPW - 1]);
        __syncthreads();
        const float2 cb = lds2(P0 - HX), ca = lds2(P0 + RPW * HX);
        float2 u[RPW], wy[RPW], F[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) u[r] = lds2(at(F_UY, r));
        float2 dl = sub2(in[0], cb);
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
          const float2 dr = sub2(r < RPW - 1 ? in[r + 1] : ca, in[r]);
          wy[r] = mul2(lds2(at(F_KY, r)), minmod2(dr, dl));
          F[r] = fma2(u[r], in[r], wy[r]);
          dl = dr;
        }
        sts2(W, F[0]);
        if (RPW > 1) sts2(W + (RPW - 1) * HX, F[RPW - 1]);
        __syncthreads();
        prefetch(t + 2, early);
        float2 G[RPW + 1];
#pragma unroll
        for (int r = 0; r <= RPW; ++r) {
          const float2 Fb = r ? F[r - 1] : lds2(W - HX), Fa = r < RPW ? F[r] : lds2(W + RPW * HX);
          G[r] = sub2(Fa, Fb);
        }
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
          float2 g = G[r], gp = G[r + 1];
          if constexpr (EDGE) {  // the line's ends, as in x (uniform across the warp)
            if (gj0 + r == 1) g = sub2(F[r], fma2(u[r], r ? in[r - 1] : cb, wy[r]));
            if (gj0 + r == ny) gp = sub2(fma2(u[r], r < RPW - 1 ? in[r + 1] : ca, wy[r]), F[r]);
          }
          out[r] = keep(upwind(in[r], u[r], g, gp), in[r], r);
        }
      };
      float2 sa[RPW];
      if constexpr (XFIRST) {  // sizloop.f90:42-48
        adv_x(s1, sa);
        adv_y(sa, s2);
      } else {
        adv_y(s1, sa);
        adv_x(sa, s2);
      }
    } else {
#pragma unroll
      for (int r = 0; r < RPW; ++r) s2[r] = make_float2(0.0f, 0.0f);
      __syncthreads();  // the y-sweep plane of the previous iteration is read by all warps
    }
    // ---------------- C: diffz for plane k (diffz.f90:22-62)
    float2 s3[RPW], lbv[RPW];
    const ZTab zk = tab[k];
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const float2 c0 = rb[r];
      lbv[r] = lb[r];
      if (STEADY || t <= nz) {
        const float2 l = lds2(at(F_L, r)), q = mul2(s2[r], l), qb = mul2(c0, lb[r]);
        if (STEADY || t > ts) {
          const float2 dq = sub2(q, qb);
          const float2 f = mul2(lds2(at(F_FZ, r)), dq);
          if (STEADY || k > 1) {
            s3[r] = fma2(splat(zk.dtdzz), sub2(f, fp[r]), c0);
          } else {  // the bottom cell: its upper face not averaged, the ground face MAX(0, ...)
            const int h = pair_in && row_in(r) ? h0 + r * px : 0;
            const float2 up = mul2(ldg2(a.f.ez + h), dq);
            const float2 lo = max0(mul2(ldg2(a.f.fz + h), sub2(qb, mul2(gb[r], lb[r]))));
            s3[r] = fma2(splat(zk.dtdzz), sub2(up, lo), c0);
          }
          fp[r] = f;
          if (!STEADY && t == nz) dqn[r] = dq;
        }
        rb[r] = s2[r];
        lb[r] = l;
      } else {  // k == nz: the top face MIN(0, ...) with the ghost c(nz+1) (diffz.f90:50-61)
        const int h = pair_in && row_in(r) ? h0 + r * px : 0;
        const float2 up = min0(mul2(ldg2(a.f.fz + h + nz * cs), sub2(mul2(gtop[r], lb[r]), mul2(c0, lb[r]))));
        const float2 lo = mul2(ldg2(a.f.fz + h + (nz + 1) * cs), dqn[r]);
        s3[r] = fma2(splat(zk.dtrdz), sub2(up, lo), c0);
      }
      if (STEADY || k >= k0) s3[r] = keep(s3[r], c0, r);
    }
    if (!STEADY && k < k0) {
      __syncthreads();
      prefetch(t + 2, !early);
      return;
    }
    // ---------------- D: diffx (shuffles) and diffy (shared memory); their
    // coefficients are read before the barrier that frees the staging buffer
    float2 cfx[RPW], cfy[RPW + 1];
#pragma unroll
    for (int r = 0; r < RPW; ++r) cfx[r] = lds2(at(F_FX, r));
#pragma unroll
    for (int r = 0; r <= RPW; ++r) cfy[r] = lds2(at(F_FY, r - 1));
    auto dif_x = [&](const float2* in, float2* out) {
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        const float2 c0 = in[r], q = mul2(c0, lbv[r]), qp = right2(q);
        const float2 dq = sub2(qp, q);
        float2 fr = mul2(cfx[r], dq);
        if constexpr (EDGE) {
          if (xedge) {  // the line's end faces MAX(0, ...), MIN(0, ...) (diffx.f90:22-33, 44-55)
            fr.x = gi == 0 ? fmaxf(fr.x, 0.0f) : gi == nx ? fminf(fr.x, 0.0f) : fr.x;
            if (gi + 1 == nx) fr.y = fminf(fr.y, 0.0f);
          }
        }
        float2 fl = left2(fr);
        if constexpr (EDGE) {
          if (xedge) {  // and the inner faces of the first and last cells
            const float dm = shup(dq.y);
            if (gi == 0) fr.y = ex[r] * dq.y;
            if (gi == nx) fl.x = ex[r] * dm;
            if (gi + 1 == nx) fl.y = ex[r] * dq.x;
          }
        }
        out[r] = keep(add2(c0, sub2(fr, fl)), c0, r);
      }
    };
    auto dif_y = [&](const float2* in, float2* out) {
      float* P1 = P1s + RPW * warp * HX + 2 * lane;
      float2 q[RPW];
#pragma unroll
      for (int r = 0; r < RPW; ++r) q[r] = mul2(in[r], lbv[r]);
      sts2(P1, q[0]);
      if (RPW > 1) sts2(P1 + (RPW - 1) * HX, q[RPW - 1]);
      __syncthreads();
      prefetch(t + 2, !early);
      const float2 qm = lds2(P1 - HX), qa = lds2(P1 + RPW * HX);
      float2 dq[RPW + 1], f[RPW + 1];  // faces gj0-1/2 .. gj0+RPW-1/2
#pragma unroll
      for (int r = 0; r <= RPW; ++r) {
        dq[r] = sub2(r < RPW ? q[r] : qa, r ? q[r - 1] : qm);
        f[r] = mul2(cfy[r], dq[r]);
      }
#pragma unroll
      for (int r = 0; r < RPW; ++r) {
        float2 lo = f[r], up = f[r + 1];
        if constexpr (EDGE) {  // the line's end and inner faces, as in x (uniform across the warp)
          if (gj0 + r == 1) {
            lo = max0(lo);
            up = mul2(ey[r], dq[r + 1]);
          }
          if (gj0 + r == ny) {
            lo = mul2(ey[r], dq[r]);
            up = min0(up);
          }
        }
        out[r] = keep(add2(in[r], sub2(up, lo)), in[r], r);
      }
    };
    float2 s3a[RPW], s4[RPW];
    if constexpr (XFIRST) {  // sizloop.f90:55-61
      dif_x(s3, s3a);
      dif_y(s3a, s4);
    } else {
      dif_y(s3, s3a);
      dif_x(s3a, s4);
    }
    // ---------------- E: wetdep, accum, clip, store (plane k); ghosts have kept their setbcc value
    float* const q = cout + (h0 + k * cs);
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      float2 res = s4[r];
      if (wet && k <= kzmax) {  // uniform across the block; wetdep.f90:37-49
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int p2 = (gi + c - 1) + nx * (gj0 + r - 1);
          if (!(kout >> (2 * r + c) & 1u) || !(a.zlayer[k - 1] <= a.zi[p2])) continue;
          double* cw = a.cwet + (long long)(cls + 1) * pl + p2;
          const double lam = a.lambda2d[p2], v = (double)cmp(res, c);
          if (commit) *cw = *cw + a.dz64[k] * lam * v;
          cmp(res, c) = (float)(v * (1.0 - lam));
        }
      }
      if (!STEADY && k == 1 && commit) {  // accum (accum.f90:17-25), binary64
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          if (!(kout >> (2 * r + c) & 1u)) continue;
          const int mb = (gi + c - 1) + nx * (gj0 + r - 1);
          double* cd = a.cdry + (long long)(cls + 1) * pl + mb;
          const double vsd = a.vset64[(long long)cls * d.cells() + mb] + a.vdep64[(long long)cls * pl + mb];
          *cd = *cd - a.dt64 * (double)cmp(res, c) * fmin2(0.0, vsd);
        }
      }
      res = max0(res);
      // predicated stores (no divergence): whole pairs, and the single
      // columns of the two lanes at the tile's sides
      const unsigned b = kst >> (2 * r) & 3u;
      float* const o = q + r * px;
      asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %0, 3;\n\t@p st.global.v2.f32 [%1], {%2, %3};\n\t}" ::"r"(b),
                   "l"(o), "f"(res.x), "f"(res.y)
                   : "memory");
      asm volatile(
          "{\n\t.reg .pred p, q, s;\n\tsetp.eq.u32 q, %0, 1;\n\tsetp.eq.u32 s, %0, 2;\n\t@q st.global.f32 [%1], %2;\n\t"
          "@s st.global.f32 [%1+4], %3;\n\t}" ::"r"(b),
          "l"(o), "f"(res.x), "f"(res.y)
          : "memory");
    }
  };

  auto march = [&](auto edge_c) {
    const int t1 = max(3, k0 + 1), t2 = max(t1 - 1, min(te, nz - 2));  // steady: t1..t2
    for (int t = ts; t < min(t1, te + 1); ++t) plane(edge_c, False_{}, t);
    // A body of two planes issues 9% fewer instructions (no moves of the
    // carried values) but misses the instruction cache more often: with two
    // rows per warp the second costs more (400x300x50, 16 classes: 0.912 ms
    // against 0.889 ms), with one row the first (0.976 ms against 1.014 ms).
#pragma unroll S::UNROLL
    for (int t = t1; t <= t2; ++t) plane(edge_c, True_{}, t);
    for (int t = t2 + 1; t <= te; ++t) plane(edge_c, False_{}, t);
  };
  if (edge)
    march(True_{});
  else
    march(False_{});

  if (timed_out) {  // a tensor copy did not arrive in time: report, and let copies in flight land
    atomicOr(a.status, F3D_STEP_STAGING_TIMEOUT);
    for (int t = max(ts, te - 1); t <= te; ++t) staged(t);
  }
  __syncthreads();  // nobody waits on the barriers any more: they may be reused (next batch item)
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(mbar0 + 8u * b) : "memory");
  }
}

template <class S>
constexpr int min_blocks() {
  return S::HYR == 16 ? 2 : 1;
}

struct StepMaps {
  F2Maps met;
  CMaps c;
};

template <class S, bool XFIRST>
__global__ void __launch_bounds__(S::NT, min_blocks<S>())
    k_step_fused2(const FusedArgs a, const __grid_constant__ StepMaps maps) {
  const int item = blockIdx.x / a.ncls;
  step_tile<S, XFIRST>(a, &maps.met, &maps.c, a.c_in, a.c_out, 1, (int)(blockIdx.x % a.ncls), item / a.nchunk,
                       item % a.nchunk);
}

// The 64x32 step while a look-ahead meteo update runs beside it: with at most
// 112 registers a block leaves the settling chain's four 64-register warps
// room on its SM (the 128 of the other build take the whole register file).
// A forecast of 400x300x50 cells and 16 classes over eight meteo updates runs at
// 9.84e10 cell-class-steps/s with it, 6.7e10 to 7.6e10 with the other build
// throughout (whose blocks and the chain's exclude each other) and 8.5e10 to
// 9.0e10 with every update made when due.
template <bool XFIRST>
__global__ void __maxnreg__(112) k_step_fused2_beside(const FusedArgs a, const __grid_constant__ StepMaps maps) {
  const int item = blockIdx.x / a.ncls;
  step_tile<Tall, XFIRST>(a, &maps.met, &maps.c, a.c_in, a.c_out, 1, (int)(blockIdx.x % a.ncls), item / a.nchunk,
                          item % a.nchunk);
}

// ------------------------------------------------------------ batched form
// The step of every scenario of a batch in persistent launches: the work
// items are (scenario, tile, piece, class), numbered scenario by scenario
// (item_off[s] .. item_off[s+1]-1, class fastest); each block takes the next
// item from a counter until none is left.  A scenario's arguments are copied
// to shared memory with each item; its buffers alternate with the number of batch steps it
// has taken (bstep[s] even: c_in -> c_out, odd: c_out -> c_in), and the x/y
// order follows iiter = iiter0[s] + bstep[s] + 1 (sizloop.f90:42-48).
static_assert(sizeof(FusedArgs) % 4 == 0, "copied by words");

// Two launches per batch step, one per sweep order, each over the scenarios
// whose step has that order (usually all or none): with both orders in one
// kernel the 64x32 march spills, 324 bytes when both are inlined, 104 and 228 as
// calls of their own, 20 to 48 in this form (four scenarios of 400x300x50 cells and
// 16 classes 9.48e10 -> 1.00e11 cell-class-steps/s, 64 members of 64..320 by
// 64..320 cells 7.18e10 -> 7.36e10; the 64x16 march, at 64 registers, spills 232 and
// 244).  Where both orders have scenarios the launches follow one another, each
// with a tail of its own: 12 members of 64..200 by 64..200 cells take 0.79 ms a step
// when they agree and 0.88 ms when half of them are a step behind, 12 of
// 200x180x40 cells and 12 classes 2.63 and 2.71 (0.99 and 1.00, 3.32 and 3.32 before the flux form).
template <class S, bool XFIRST>
__global__ void __launch_bounds__(S::NT, min_blocks<S>())
    k_step_fused2_batch(const FusedArgs* __restrict__ args, const int* __restrict__ item_off, int nscen, int* counter,
                        const int* __restrict__ bstep, const int* __restrict__ iiter0, int commit,
                        const BatchMaps* __restrict__ maps) {
  __shared__ int s_item;
  __shared__ int s_off[F3D_BATCH_MAX + 1], s_scn[F3D_BATCH_MAX + 1];  // this order's items and scenarios
  __shared__ FusedArgs s_args;
  for (int q = threadIdx.x; q < nscen; q += S::NT) {
    s_off[q] = item_off[q + 1] - item_off[q];
    s_scn[q] = ((iiter0[q] + bstep[q] + 1) % 2 == 0) == XFIRST;
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // compacted in place: entry n is written at or before it is read
    int n = 0, off = 0;
    for (int q = 0; q < nscen; ++q) {
      const int items = s_off[q];
      if (!s_scn[q]) continue;
      s_off[n] = off;
      s_scn[n++] = q;
      off += items;
    }
    s_off[n] = off;
    s_item = n;
  }
  __syncthreads();
  const int nsel = s_item, total = s_off[nsel];
  for (;;) {
    __syncthreads();  // the previous item is done with shared memory
    if (threadIdx.x == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= total) break;
    int lo = 0, hi = nsel;  // s_off[lo] <= item < s_off[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_off[mid] <= item) lo = mid;
      else hi = mid;
    }
    const int scn = s_scn[lo], local = item - s_off[lo];
    for (int w = threadIdx.x; w < (int)(sizeof(FusedArgs) / 4); w += S::NT)
      reinterpret_cast<int*>(&s_args)[w] = __ldg(reinterpret_cast<const int*>(args + scn) + w);
    __syncthreads();
    const FusedArgs& a = s_args;
    const int rest = local / a.ncls, bs = bstep[scn];
    const float* cin = (bs & 1) ? a.c_out : a.c_in;
    float* cout = (bs & 1) ? const_cast<float*>(a.c_in) : a.c_out;
    step_tile<S, XFIRST>(a, &maps[scn].met, (bs & 1) ? &maps[scn].b : &maps[scn].a, cin, cout, commit, local % a.ncls,
                         rest / a.nchunk, rest % a.nchunk);
  }
}

// ------------------------------------------------------------ step fields
// The class-independent fields of the step kernel from a meteo update's
// binary64 fields, one thread per position of the halo layout (see StepFields
// for what the ghosts hold).  dt is the update's own, formed as the host
// does (finddt.f90:58-66).
__global__ void k_step_fields(Dims d, double safety, double dX1, double dX2, const double* dz,
                              const unsigned long long* dtcn, const double* vx, const double* vy, const double* rho,
                              const double* rkh1, const double* rkhor, const double* rkver, StepFields f) {
  const double dt = safety * (1.0 / fmax2(__longlong_as_double((long long)*dtcn), 1e-13));
  const int nx = d.nx, ny = d.ny, nz = d.nz, px = d.px;
  // the divisions once per thread, which takes several positions of its plane
  const double ax = dt / dX1, ay = dt / dX2, bx = dt / (dX1 * dX1), by = dt / (dX2 * dX2);
  const int plane = px * (ny + 2), k = blockIdx.y;
  const double rdz = 1.0 / (k == 0 ? dz[0] : k <= nz ? dz[k] : dz[nz - 1]);
  for (int h = blockIdx.x * blockDim.x + threadIdx.x; h < plane; h += gridDim.x * blockDim.x) {
    const int i = h % px, j = h / px;
    if (h == 0 && k <= nz) {  // this level's factors
      ZTab z{};
      const double dk = dz[k], dm = k > 0 ? dz[k - 1] : dz[0], dzz = 2.0 / (dk + dm);
      z.a = (float)(0.25 * dt * dm * dzz);
      z.b = (float)(0.125 * dt * dt * dzz);
      z.rdz = (float)(1.0 / dk);
      z.dtdzz = (float)(dt * dzz);
      z.dtrdz = (float)(dt / dk);
      f.tab[k] = z;
    }
    if (i > nx + 1) continue;
    const int ic = min(max(i, 1), nx), jc = min(max(j, 1), ny);
    const long long m = d.M(ic, jc, 1), pl = d.plane();
    const long long o = h + (long long)k * plane;
    // rkver*rho at a level, for diffz
    auto Z = [&](int kk) { return rkver[m + (kk - 1) * pl] * rho[m + (kk - 1) * pl]; };
    if (k == 0 || k > nz) {
      f.fz[o] = (float)((k == 0 ? Z(1) : Z(nz - 1)) * rdz);
      if (k == 0) f.ez[h] = (float)(Z(2) / dz[1]);
      continue;
    }
    const long long q = m + (k - 1) * pl;
    const double r = rho[q];
    f.ux[o] = (float)(ax * vx[q]);
    f.uy[o] = (float)(ay * vy[q]);
    auto K = [](double c) { return (float)(0.5 * c * (1.0 - c)); };
    if (i >= 1 && i <= nx) f.kx[o] = K(0.5 * ax * absd(vx[q] + vx[i > 1 ? q - 1 : q]));
    if (j >= 1 && j <= ny) f.ky[o] = K(0.5 * ay * absd(vy[q] + vy[j > 1 ? q - nx : q]));
    f.l[o] = (float)(1.0 / r);
    f.fz[o] = (float)((k < nz ? 0.5 * (Z(k) + Z(k + 1)) : Z(nz)) * rdz);
    const double p = rkh1[q] * r, s = rkhor[q] * r;
    f.fx[o] = (float)(i >= 1 && i < nx ? 0.5 * bx * (p + rkh1[q + 1] * rho[q + 1]) : bx * p);
    f.fy[o] = (float)(j >= 1 && j < ny ? 0.5 * by * (s + rkhor[q + nx] * rho[q + nx]) : by * s);
    if (i == 2) f.ex[(long long)k * (ny + 2) + j] = (float)(bx * p);
    if (i == nx - 1) f.ex[(long long)(nz + 2) * (ny + 2) + (long long)k * (ny + 2) + j] = (float)(bx * p);
    if (j == 2) f.ey[(long long)k * px + i] = (float)(by * s);
    if (j == ny - 1) f.ey[(long long)(nz + 2) * px + (long long)k * px + i] = (float)(by * s);
  }
}

// vz + vset per class in the halo layout (the vertical velocity of
// advctzc.f90:23): every thread keeps vz of its cell through the classes.
__global__ void k_step_vk(Dims d, int nc, const double* vz, const double* vset, float* vk) {
  const long long s3 = d.cells(), hb = d.halo();
  for (long long m = blockIdx.x * (long long)blockDim.x + threadIdx.x; m < s3;
       m += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(m % d.nx) + 1;
    const long long r = m / d.nx;
    const int j = (int)(r % d.ny) + 1, k = (int)(r / d.ny) + 1;
    const double w = vz[m];
    float* o = vk + d.C(i, j, k);
    for (int c = 0; c < nc; ++c) o[c * hb] = (float)(w + vset[c * s3 + m]);
  }
}

// wet-deposition rate per column for the fused kernel: lambda =
// min(dt*a*prate^b, 1) (wetdep.f90:40), constant between meteo updates.
__global__ void k_wet_lambda(long long n, double dt, const double* prate, double* lam) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= n) return;
  const double aa = 8.4e-5, b = 0.79;
  lam[p] = fmin2(dt * aa * pow(prate[p], b), 1.0);
}

int device_sms() {
  static int nsm = 0;
  if (!nsm) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }
  return std::max(1, nsm);
}

// calls f with the tile shape's type
template <class F>
auto with_shape(int shape, F f) {
  return shape == 3 ? f(Tall{}) : f(Flat{});
}

}  // namespace

void launch_wet_lambda(long long n, double dt, const double* prate, double* lam, cudaStream_t s) {
  k_wet_lambda<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, dt, prate, lam);
  count_launch();
}

void launch_step_fields(Dims d, int nc, double safety, double dX1, double dX2, const double* dz,
                        const unsigned long long* dtcn, const double* vx, const double* vy, const double* vz,
                        const double* rho, const double* rkh1, const double* rkhor, const double* rkver,
                        const double* vset, const StepFields& f, cudaStream_t s) {
  const long long plane = (long long)d.px * (d.ny + 2);
  // about four blocks per SM over all planes
  const long long nb = std::max<long long>(1, 4LL * device_sms() / (d.nz + 2));
  k_step_fields<<<dim3((unsigned)std::min<long long>((plane + 255) / 256, nb), d.nz + 2), 256, 0, s>>>(d, safety, dX1, dX2, dz, dtcn, vx, vy,
                                                                               rho, rkh1, rkhor, rkver, f);
  count_launch();
  launch_step_vk(d, nc, vz, vset, f.vk, s);
}

void launch_step_vk(Dims d, int nc, const double* vz, const double* vset, float* vk, cudaStream_t s) {
  const int nb = (int)std::min<long long>((d.cells() + 255) / 256, 152LL * 16);
  k_step_vk<<<nb, 256, 0, s>>>(d, nc, vz, vset, vk);
  count_launch();
}

int fused_tiles(int nx, int ny, int shape) {
  const int ty = with_shape(shape, [](auto s) { return decltype(s)::TY; });
  return ((nx + TX - 1) / TX) * ((ny + ty - 1) / ty);
}

// 64x16 tiles of which every SM gets at most one take a plane in fewer
// operations per warp than the 64x32 tiles that would leave half of the SMs
// idle: 21.0 us against 27.2 at 12x10x8 cells and 3 classes, 24.1 against 39.9
// at 32x28x14 and 4, 40.5 against 50.6 at 80x80x25 and 6 (96 tiles), 60.7
// against 61.0 at 160x121x40 and 3 (117).  Beyond, their larger share of halo
// rows costs more: 66.0 against 63.0 us at 121x101x30 and 6 classes (198 tiles),
// 299 against 285 at 243x191x37 and 11, 976 against 889 at 400x300x50 and 16.
int step_shape(Dims d, int ncls) { return (long long)fused_tiles(d.nx, d.ny, 0) * ncls <= device_sms() ? 0 : 3; }

void step_chunks(FusedArgs& a, int shape, int nwet, long long batch_items) {
  const int nz = a.d.nz;
  a.nchunk = 1;
  a.kfirst = nz;
  a.klen = nz;
  const long long blocks = std::max(batch_items, (long long)fused_tiles(a.d.nx, a.d.ny, shape) * a.ncls);
  const long long slots = (long long)device_sms() * with_shape(shape, [](auto s) { return min_blocks<decltype(s)>(); });
  // waves of blocks times iterations of the longest piece (plus ~3 for the start)
  long long best = ((blocks + slots - 1) / slots) * (nz + 4);
  for (int n = 2; n <= 16; ++n) {
    const int len = (nz + n - 1) / n, first = std::max(len, nwet), rest = nz - first;
    if (len < 4 || rest < 4 * (n - 1)) break;
    const int each = (rest + n - 2) / (n - 1);
    if (rest - each * (n - 2) < 4) continue;
    const long long cost = ((blocks * n + slots - 1) / slots) * (std::max(first + 1, each + 2) + 3);
    if (cost < best) {
      best = cost;
      a.nchunk = n;
      a.kfirst = first;
      a.klen = each;
    }
  }
}

void launch_step_fused(const FusedArgs& a, const F2Maps& maps, const CMaps& c, int shape, cudaStream_t s, bool beside) {
  with_shape(shape, [&](auto sh) {
    using S = decltype(sh);
    const size_t sm = step_smem<S>(a.d.nz);
    StepMaps m;
    m.met = maps;
    m.c = c;
    auto go = [&](auto kernel) {
      // the limit of the longest column, not of this one: another thread may be
      // launching the kernel for a longer one
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)step_smem<S>(std::max(a.d.nz, fused2_max_nz(false))));
      kernel<<<fused_tiles(a.d.nx, a.d.ny, shape) * a.ncls * a.nchunk, S::NT, sm, s>>>(a, m);
    };
    if (beside && S::HYR == HY)
      a.xfirst ? go(k_step_fused2_beside<true>) : go(k_step_fused2_beside<false>);
    else
      a.xfirst ? go(k_step_fused2<S, true>) : go(k_step_fused2<S, false>);
    return 0;
  });
  count_launch();
}

int fused2_max_nz(bool batch) {
  static const auto limit = [](std::initializer_list<const void*> kernels) {
    size_t fixed = 0;  // the kernels' own shared memory beside the dynamic one
    for (const void* k : kernels) {
      cudaFuncAttributes at{};
      if (cudaFuncGetAttributes(&at, k) != cudaSuccess) return 0;
      fixed = std::max(fixed, at.sharedSizeBytes);
    }
    const size_t cap = (size_t)227 * 1024, base = step_smem<Tall>(0) + fixed;
    return cap > base ? (int)((cap - base) / sizeof(ZTab)) : 0;
  };
  static const int alone = limit({(const void*)k_step_fused2<Tall, true>, (const void*)k_step_fused2<Tall, false>,
                                  (const void*)k_step_fused2_beside<true>, (const void*)k_step_fused2_beside<false>});
  static const int in_batch = limit({(const void*)k_step_fused2_batch<Tall, true>,
                                     (const void*)k_step_fused2_batch<Tall, false>});
  return batch ? in_batch : alone;
}

// cuTensorMapEncodeTiled, reached through the runtime's driver entry point
// (no link against the driver library)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// the two maps (32- and 16-row boxes) of a field: x (the padded row), y (rows
// 0..ny+1), z (planes 0..nz+1, times the classes for class blocks)
static int step_map(Dims d, const float* p, long long planes, CUtensorMap* m32, CUtensorMap* m16) {
  static EncodeTiledFn enc = nullptr;
  if (!enc) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return 1;
    enc = reinterpret_cast<EncodeTiledFn>(fn);
  }
  if (d.px % 4 != 0 || d.px < d.nx + 2) return 2;
  const cuuint64_t dim[3] = {(cuuint64_t)d.px, (cuuint64_t)(d.ny + 2), (cuuint64_t)planes};
  const cuuint64_t stride[2] = {(cuuint64_t)d.px * sizeof(float), (cuuint64_t)d.px * (d.ny + 2) * sizeof(float)};
  const cuuint32_t es[3] = {1u, 1u, 1u};
  for (int q = 0; q < 2; ++q) {
    const cuuint32_t box[3] = {(cuuint32_t)RS, q ? 16u : 32u, 1u};
    if (enc(q ? m16 : m32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(p), dim, stride, box, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return 3;
  }
  return 0;
}

int make_step_maps(const FusedArgs& a, F2Maps* out) {
  const long long np = a.d.nz + 2;
  const float* p[F2Maps::N] = {a.f.vk, a.f.ux, a.f.kx, a.f.uy, a.f.ky, a.f.l, a.f.fz, a.f.fx, a.f.fy};
  for (int f = 0; f < F2Maps::N; ++f)
    if (int rc = step_map(a.d, p[f], f == F2Maps::VK ? np * a.ncls : np, &out->m[0][f], &out->m[1][f])) return rc;
  return 0;
}

int make_c_maps(Dims d, int ncls, const float* c, CMaps* out) {
  return step_map(d, c, (long long)(d.nz + 2) * ncls, &out->m[0], &out->m[1]);
}

int fused_batch_grid(int shape, int max_nz) {
  return with_shape(shape, [&](auto sh) {
    using S = decltype(sh);
    const size_t sm = step_smem<S>(max_nz);
    auto fit = [&](auto kernel) {
      int per_sm = 0;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)step_smem<S>(std::max(max_nz, fused2_max_nz(true)))) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, S::NT, sm) != cudaSuccess)
        return 0;
      return per_sm;
    };
    const int per_sm = std::min(fit(k_step_fused2_batch<S, true>), fit(k_step_fused2_batch<S, false>));
    return per_sm < 1 ? -1 : per_sm * device_sms();
  });
}

void launch_step_fused_batch(int shape, int grid, const FusedArgs* args, const int* item_off, int nscen, int* counter,
                             const int* bstep, const int* iiter0, int commit, int max_nz, const BatchMaps* maps,
                             cudaStream_t s) {
  with_shape(shape, [&](auto sh) {
    using S = decltype(sh);
    const size_t sm = step_smem<S>(max_nz);
    k_step_fused2_batch<S, true><<<grid, S::NT, sm, s>>>(args, item_off, nscen, counter, bstep, iiter0, commit, maps);
    k_step_fused2_batch<S, false><<<grid, S::NT, sm, s>>>(args, item_off, nscen, counter + 1, bstep, iiter0, commit,
                                                         maps);
    return 0;
  });
  count_launch(2);
}

}  // namespace f3d
