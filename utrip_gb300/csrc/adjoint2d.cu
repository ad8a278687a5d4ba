// Discrete adjoint of the 2.5-D mLW step (cans2d/hdmlw/mlw_m3.f:2-377) and of
// the boundary fill, by hand: the transpose of the linearised step, applied to
// an adjoint state lambda (one array per primitive variable), on the device.
//
// Forward step, in the stage form the reverse follows (1-based indices,
// interior = 2..n-1 in both axes, dt frozen):
//   (1) cell values of the input primitives P: conserved U, fluxes FX, FY
//       (mlw_m3.f:107-202);
//   (2) du = -0.25 dt (dxi (FX(i+1)-FX(i-1)) + dyi (FY(j+1)-FY(j-1)))   interior
//       Uh(corner) = avg4(U) - dt dxim/2 (dx FX) - dt dyim/2 (dy FY)  (mlwhalf.f)
//   (3) corner primitives Ph = prim(Uh), corner fluxes GX, GY (:214-310)
//   (4) du -= 0.5 dt (dxi sum_uy (dx GX) + dyi sum_ux (dy GY))         (mlwfull.f)
//   (5) q = qav dxm max(0, |dv| - 1e-4) on faces; du += dt dxi (q dxim dU - ...)
//       for the 8 conserved variables (mlwartv.f, :324-345)
//   (6) P' = prim(U + du) on the interior; other cells keep P (:349-374)
// az is updated by sources of its own and feeds back into nothing, and the
// objective does not read it, so its adjoint is identically zero.
//
// Reverse, given lambda' for P' after the boundary fill (bc_transpose first):
//   k_adj_cells   a' = (dP'/dU')^T lambda' on the interior (= adjoint of du),
//                 plus the cell values U, FX, FY of P for the kernels below
//   k_adj_corners adjoint of GX, GY gathered from the four cells that read each
//                 corner (transpose of (4)), then of Uh through (3)
//   k_adj_gather  adjoint of U, FX, FY of every cell gathered from its corners
//                 (transpose of the predictor), its neighbours (transpose of
//                 the half step and of the viscosity in U), the adjoint of q
//                 on its two faces per axis, then (dU,FX,FY/dP)^T; cells
//                 outside the interior pass lambda' through unchanged.
// Every transpose is a gather: no atomics, deterministic results.
#include <cuda_runtime.h>

#include "cans_common.cuh"
#include "cans_internal.h"
#include "df64.cuh"

namespace cans {

namespace {

constexpr int kT = 128;
// four resident blocks per SM (at most 128 registers a thread): a 258^2
// grid's 520 blocks then fit in one wave of 152 x 4 slots, where three
// blocks per SM (the registers the reverse kernels would otherwise take)
// need two waves, the second nearly empty
constexpr int kMinBlocks = 4;
// primitive slots of the state (mlw_m3 order) and conserved slots
enum { P_RO = 0, P_PR, P_VX, P_VY, P_VZ, P_BX, P_BY, P_BZ, P_AZ };
enum { C_RO = 0, C_EE, C_RX, C_RY, C_RZ, C_BX, C_BY, C_BZ };

struct G2 {
  int ix, jx;
  size_t n;
};

__device__ __forceinline__ bool interior(const G2 &g, int i, int j) {
  return i >= 1 && i <= g.ix - 2 && j >= 1 && j <= g.jx - 2;  // 0-based
}

// The reverse kernels are written once for a number type R: double (FP64
// pipe) or df::DF (double-float on the FP32 pipes, about 2^-46 per
// operation; see df64.cuh).  The gradient is checked to 1e-6 relative, so the
// reverse sweep may run in double-float; the forward steps it linearises
// about are the run's own FP64 steps in either case.  Scratch arrays between
// the kernels hold R values (num_ld / num_st); the states read and the
// adjoint written are doubles (num_in / num_out).
template <class R> struct PhysR {
  R gm1, gm1i, ggm1, pi8i, pi4i, qav;
};
template <class R> __device__ __forceinline__ PhysR<R> phys_r(const Phys &ph) {
  return {num_in<R>(ph.gm1), num_in<R>(ph.gm1i), num_in<R>(ph.ggm1), num_in<R>(ph.pi8i),
          num_in<R>(ph.pi4i), num_in<R>(ph.qav)};
}

// (1): conserved values and fluxes of one primitive state (mlw_m3.f:107-202)
template <class R> struct CellF {
  R U[8], FX[8], FY[8];
};
template <class R>
__device__ __forceinline__ void cell_forward(const R *p, const PhysR<R> &ph, CellF<R> &o) {
  const R ro = p[P_RO], pr = p[P_PR], vx = p[P_VX], vy = p[P_VY], vz = p[P_VZ];
  const R bx = p[P_BX], by = p[P_BY], bz = p[P_BZ];
  const R vv = vx * vx + vy * vy + vz * vz, bb = bx * bx + by * by + bz * bz;
  const R ex = -vy * bz + vz * by, ey = -vz * bx + vx * bz, ez = -vx * by + vy * bx;
  const R ep = pr * ph.ggm1 + 0.5f * ro * vv;
  o.U[C_RO] = ro;
  o.U[C_EE] = pr * ph.gm1i + 0.5f * ro * vv + ph.pi8i * bb;
  o.U[C_RX] = ro * vx;
  o.U[C_RY] = ro * vy;
  o.U[C_RZ] = ro * vz;
  o.U[C_BX] = bx;
  o.U[C_BY] = by;
  o.U[C_BZ] = bz;
  o.FX[C_RO] = ro * vx;
  o.FY[C_RO] = ro * vy;
  o.FX[C_EE] = ep * vx + (bz * ey - by * ez) * ph.pi4i;
  o.FY[C_EE] = ep * vy + (bx * ez - bz * ex) * ph.pi4i;
  o.FX[C_RX] = ro * vx * vx + pr + ph.pi8i * (by * by + bz * bz - bx * bx);
  o.FY[C_RX] = ro * vx * vy - ph.pi4i * bx * by;
  o.FX[C_RY] = ro * vy * vx - ph.pi4i * by * bx;
  o.FY[C_RY] = ro * vy * vy + pr + ph.pi8i * (bx * bx + bz * bz - by * by);
  o.FX[C_RZ] = ro * vz * vx - ph.pi4i * bz * bx;
  o.FY[C_RZ] = ro * vz * vy - ph.pi4i * bz * by;
  o.FX[C_BX] = R(0.0f);
  o.FY[C_BX] = ez;
  o.FX[C_BY] = -ez;
  o.FY[C_BY] = R(0.0f);
  o.FX[C_BZ] = ey;
  o.FY[C_BZ] = -ex;
}

// primitives of a conserved state (mlw_m3.f:214-223, 365-374)
template <class R>
__device__ __forceinline__ void prim_forward(const R *u, const PhysR<R> &ph, R *p) {
  const R ro = u[C_RO];
  const R ri = R(1.0f) / ro;
  const R vx = u[C_RX] * ri, vy = u[C_RY] * ri, vz = u[C_RZ] * ri;
  const R vv = vx * vx + vy * vy + vz * vz;
  const R bb = u[C_BX] * u[C_BX] + u[C_BY] * u[C_BY] + u[C_BZ] * u[C_BZ];
  p[P_RO] = ro;
  p[P_PR] = ph.gm1 * (u[C_EE] - 0.5f * ro * vv - ph.pi8i * bb);
  p[P_VX] = vx;
  p[P_VY] = vy;
  p[P_VZ] = vz;
  p[P_BX] = u[C_BX];
  p[P_BY] = u[C_BY];
  p[P_BZ] = u[C_BZ];
}

// Transpose of (1): given the adjoints of U, FX, FY at the point p, read from aU, aX,
// aY with stride kT (HASU: of U too), return ap = (d(U,FX,FY)/dP)^T of them.  The sums
// over the terms are factored: the derivatives of the mass and momentum fluxes share
// sx = d(FX)/d(rho vx), sy and q = d(..)/d(rho v^2 / 2), 70 products where one term
// after the other takes 150.
template <class R, bool HASU>
__device__ __forceinline__ void cell_reverse(const R *p, const PhysR<R> &ph, const double *aU,
                                             const double *aX, const double *aY, R *ap) {
  const R ro = p[P_RO], pr = p[P_PR], vx = p[P_VX], vy = p[P_VY], vz = p[P_VZ];
  const R bx = p[P_BX], by = p[P_BY], bz = p[P_BZ];
  auto X = [&](int v) { return num_ld<R>(aX + v * kT); };
  auto Y = [&](int v) { return num_ld<R>(aY + v * kT); };
  auto U = [&](int v) { return num_ld<R>(aU + v * kT); };
  const R vv = fma(vx, vx, fma(vy, vy, vz * vz));
  const R ex = fma(vz, by, -(vy * bz)), ey = fma(vx, bz, -(vz * bx)), ez = fma(vy, bx, -(vx * by));
  const R ep = fma(pr, ph.ggm1, 0.5f * ro * vv);
  const R xe = X(C_EE), ye = Y(C_EE), tx = xe * ph.pi4i, ty = ye * ph.pi4i;
  const R xx = X(C_RX), xy = X(C_RY), xz = X(C_RZ), yx = Y(C_RX), yy = Y(C_RY), yz = Y(C_RZ);
  // adjoints of ep and E, and of rho v^2 / 2
  const R aep = fma(xe, vx, ye * vy);
  const R aex = -(fma(ty, bz, Y(C_BZ))), aey = fma(tx, bz, X(C_BZ));
  const R aez = fma(ty, bx, Y(C_BX)) - fma(tx, by, X(C_BY));
  R q = aep, db = yy - xx, mx, my, mz;
  if constexpr (HASU) q = q + U(C_EE);
  const R sx = fma(xx, vx, fma(xy, vy, fma(xz, vz, X(C_RO))));
  const R sy = fma(yx, vx, fma(yy, vy, fma(yz, vz, Y(C_RO))));
  mx = fma(xx, vx, fma(yx, vy, fma(vx, q, sx)));
  my = fma(xy, vx, fma(yy, vy, fma(vy, q, sy)));
  mz = fma(xz, vx, fma(yz, vy, vz * q));
  R aro = fma(vx, sx, fma(vy, sy, 0.5f * vv * q));
  R apr = fma(aep, ph.ggm1, xx + yy);
  const R p82 = 2.0f * ph.pi8i;
  // of pi8i times the squares of bx, by, bz
  R qx = db, qy = -db, qz = xx + yy;
  R abx, aby, abz;
  if constexpr (HASU) {
    const R ue = U(C_EE), ux = U(C_RX), uy = U(C_RY), uz = U(C_RZ);
    mx = mx + ux;
    my = my + uy;
    mz = mz + uz;
    aro = aro + fma(ux, vx, fma(uy, vy, fma(uz, vz, U(C_RO))));
    apr = fma(ue, ph.gm1i, apr);
    qx = qx + ue;
    qy = qy + ue;
    qz = qz + ue;
    abx = fma(p82 * bx, qx, U(C_BX));
    aby = fma(p82 * by, qy, U(C_BY));
    abz = fma(p82 * bz, qz, U(C_BZ));
  } else {
    abx = p82 * bx * qx;
    aby = p82 * by * qy;
    abz = p82 * bz * qz;
  }
  const R xyx = xy + yx;
  abx = fma(-ph.pi4i, fma(xyx, by, xz * bz), abx);
  aby = fma(-ph.pi4i, fma(xyx, bx, yz * bz), aby);
  abz = fma(-ph.pi4i, fma(xz, bx, yz * by), abz);
  ap[P_RO] = aro;
  ap[P_PR] = apr;
  ap[P_VX] = fma(ro, mx, fma(xe, ep, fma(aey, bz, -(aez * by))));
  ap[P_VY] = fma(ro, my, fma(ye, ep, fma(aez, bx, -(aex * bz))));
  ap[P_VZ] = fma(ro, mz, fma(aex, by, -(aey * bx)));
  ap[P_BX] = fma(ty, ez, fma(aez, vy, fma(-aey, vz, abx)));
  ap[P_BY] = fma(-tx, ez, fma(aex, vz, fma(-aez, vx, aby)));
  ap[P_BZ] = fma(tx, ey, fma(-ty, ex, fma(aey, vx, fma(-aex, vy, abz))));
}

// Transpose of prim_forward at the point whose primitives are p: given ap,
// return au = (dP/dU)^T ap.
template <class R>
__device__ __forceinline__ void prim_reverse(const R *p, const PhysR<R> &ph, const R *ap,
                                             R *au) {
  const R ro = p[P_RO], vx = p[P_VX], vy = p[P_VY], vz = p[P_VZ];
  const R vv = vx * vx + vy * vy + vz * vz;
  const R apr = ap[P_PR];
  const R avv = -ph.gm1 * 0.5f * ro * apr;
  const R abb = -ph.gm1 * ph.pi8i * apr;
  const R ri = R(1.0f) / ro;
  const R avx = ap[P_VX] + 2.0f * vx * avv, avy = ap[P_VY] + 2.0f * vy * avv,
          avz = ap[P_VZ] + 2.0f * vz * avv;
  au[C_EE] = ph.gm1 * apr;
  au[C_RX] = avx * ri;
  au[C_RY] = avy * ri;
  au[C_RZ] = avz * ri;
  au[C_RO] = ap[P_RO] - ph.gm1 * 0.5f * vv * apr - (avx * vx + avy * vy + avz * vz) * ri;
  au[C_BX] = ap[P_BX] + 2.0f * p[P_BX] * abb;
  au[C_BY] = ap[P_BY] + 2.0f * p[P_BY] * abb;
  au[C_BZ] = ap[P_BZ] + 2.0f * p[P_BZ] * abb;
}

template <class R>
__device__ __forceinline__ void load_prim(const double *S, size_t n, size_t c, R *p) {
#pragma unroll
  for (int v = 0; v < 8; v++) p[v] = num_in<R>(S[v * n + c]);
}

// a' on the interior, the cell values U, FX, FY of P everywhere
template <class R>
__global__ void __launch_bounds__(kT, kMinBlocks)
    k_adj_cells(const double *__restrict__ P, const double *__restrict__ Rw,
                const double *__restrict__ lam, double *__restrict__ A1,
                double *__restrict__ CU, G2 g, Phys ph_) {
  const size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (c >= g.n) return;
  const PhysR<R> ph = phys_r<R>(ph_);
  const int i = (int)(c % g.ix), j = (int)(c / g.ix);
  R p[8];
  load_prim(P, g.n, c, p);
  CellF<R> f;
  cell_forward(p, ph, f);
#pragma unroll
  for (int v = 0; v < 8; v++) {
    num_st(CU + v * g.n + c, f.U[v]);
    num_st(CU + (8 + v) * g.n + c, f.FX[v]);
    num_st(CU + (16 + v) * g.n + c, f.FY[v]);
  }
  R au[8];
#pragma unroll
  for (int v = 0; v < 8; v++) au[v] = R(0.0f);
  if (interior(g, i, j)) {
    R r[8], ap[8];
    load_prim(Rw, g.n, c, r);
    load_prim(lam, g.n, c, ap);
    prim_reverse(r, ph, ap, au);
  }
#pragma unroll
  for (int v = 0; v < 8; v++) num_st(A1 + v * g.n + c, au[v]);
}

// corners (p+1/2, q+1/2), p = 0..ix-2, q = 0..jx-2 (0-based), stored at p+q*ix
template <class R>
__global__ void __launch_bounds__(kT, kMinBlocks)
    k_adj_corners(const double *__restrict__ CU, const double *__restrict__ A1,
                  double *__restrict__ A2, G2 g, Axis ax, Axis ay, Phys ph_,
                  double dt_) {
  const size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (c >= g.n) return;
  __shared__ double sm[2 * 8 * kT];
  double *sX = sm + threadIdx.x, *sY = sX + 8 * kT;
  const PhysR<R> ph = phys_r<R>(ph_);
  const R dt = num_in<R>(dt_);
  const int p = (int)(c % g.ix), q = (int)(c / g.ix);
  R out[8];
#pragma unroll
  for (int v = 0; v < 8; v++) out[v] = R(0.0f);
  if (p <= g.ix - 2 && q <= g.jx - 2) {
    const size_t c00 = c, c10 = c + 1, c01 = c + g.ix, c11 = c + g.ix + 1;
    // The eight variables in rolled loops, their results in shared memory: unrolled,
    // the kernels outgrow the instruction cache (gather, 256^2: half of the stalled
    // cycles; 47.8 -> 31.8 us with the shorter cell_reverse, corners 24.4 -> 20.3).
    // forward corner state (mlwhalf.f part 2)
    const R cx = -(0.5f * dt * num_in<R>(ax.dim[p])), cy = -(0.5f * dt * num_in<R>(ay.dim[q]));
#pragma unroll 1
    for (int v = 0; v < 8; v++) {
      const double *U = CU + v * g.n, *FX = CU + (8 + v) * g.n, *FY = CU + (16 + v) * g.n;
      const R s = (num_ld<R>(U + c10) + num_ld<R>(U + c00)) +
                  (num_ld<R>(U + c11) + num_ld<R>(U + c01));
      const R dx = (num_ld<R>(FX + c10) - num_ld<R>(FX + c00)) +
                   (num_ld<R>(FX + c11) - num_ld<R>(FX + c01));
      const R dy = (num_ld<R>(FY + c01) - num_ld<R>(FY + c00)) +
                   (num_ld<R>(FY + c11) - num_ld<R>(FY + c10));
      num_st(sX + v * kT, fma(cy, dy, fma(cx, dx, 0.25f * s)));
    }
    R ph8[8];
    {
      R uh[8];
#pragma unroll
      for (int v = 0; v < 8; v++) uh[v] = num_ld<R>(sX + v * kT);
      prim_forward(uh, ph, ph8);
    }
    // adjoint of GX, GY at this corner: the cells (p,q), (p+1,q), (p,q+1),
    // (p+1,q+1) that read it in mlwfull (0-based cell indices); 0 for those the step
    // does not update
    const R zero(0.0f);
    const bool i00 = interior(g, p, q), i10 = interior(g, p + 1, q),
               i01 = interior(g, p, q + 1), i11 = interior(g, p + 1, q + 1);
    const R hx0 = 0.5f * dt * num_in<R>(ax.di[p]), hx1 = 0.5f * dt * num_in<R>(ax.di[p + 1]);
    const R hy0 = 0.5f * dt * num_in<R>(ay.di[q]), hy1 = 0.5f * dt * num_in<R>(ay.di[q + 1]);
    const R uy1q = num_in<R>(ay.u1[q]), uy0q1 = num_in<R>(ay.u0[q + 1]);
    const R ux1p = num_in<R>(ax.u1[p]), ux0p1 = num_in<R>(ax.u0[p + 1]);
    const R x00 = i00 ? -(hx0 * uy1q) : zero, x10 = i10 ? hx1 * uy1q : zero;
    const R x01 = i01 ? -(hx0 * uy0q1) : zero, x11 = i11 ? hx1 * uy0q1 : zero;
    const R y00 = i00 ? -(hy0 * ux1p) : zero, y10 = i10 ? -(hy0 * ux0p1) : zero;
    const R y01 = i01 ? hy1 * ux1p : zero, y11 = i11 ? hy1 * ux0p1 : zero;
#pragma unroll 1
    for (int v = 0; v < 8; v++) {  // A1 is 0 outside the interior
      const double *a = A1 + v * g.n;
      const R l00 = num_ld<R>(a + c00), l10 = num_ld<R>(a + c10);
      const R l01 = num_ld<R>(a + c01), l11 = num_ld<R>(a + c11);
      num_st(sX + v * kT, fma(x00, l00, fma(x10, l10, fma(x01, l01, x11 * l11))));
      num_st(sY + v * kT, fma(y00, l00, fma(y10, l10, fma(y01, l01, y11 * l11))));
    }
    R aP[8];
    cell_reverse<R, false>(ph8, ph, nullptr, sX, sY, aP);
    prim_reverse(ph8, ph, aP, out);
  }
#pragma unroll
  for (int v = 0; v < 8; v++) num_st(A2 + v * g.n + c, out[v]);
}

// adjoint of P for every cell
template <class R>
__global__ void __launch_bounds__(kT, kMinBlocks)
    k_adj_gather(const double *__restrict__ P, const double *__restrict__ CU,
                 const double *__restrict__ A1, const double *__restrict__ A2,
                 const double *__restrict__ lam, double *__restrict__ out, G2 g,
                 Axis ax, Axis ay, Phys ph_, double dt_) {
  const size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (c >= g.n) return;
  __shared__ double sm[3 * 8 * kT];
  double *sU = sm + threadIdx.x, *sX = sU + 8 * kT, *sY = sX + 8 * kT;
  const PhysR<R> ph = phys_r<R>(ph_);
  const R dt = num_in<R>(dt_);
  const int i = (int)(c % g.ix), j = (int)(c / g.ix);
  const size_t n = g.n, sx = 1, sy = (size_t)g.ix;
  R p[8];
  load_prim(P, n, c, p);
  const bool in_c = interior(g, i, j);
  const bool in_xm = interior(g, i - 1, j), in_xp = interior(g, i + 1, j);
  const bool in_ym = interior(g, i, j - 1), in_yp = interior(g, i, j + 1);
  // corners around the cell: (i-1+1/2, j-1+1/2) .. (i+1/2, j+1/2)
  const bool k_mm = i >= 1 && j >= 1, k_pm = i <= g.ix - 2 && j >= 1;
  const bool k_mp = i >= 1 && j <= g.jx - 2, k_pp = i <= g.ix - 2 && j <= g.jx - 2;
  // metrics the coefficients below read
  const R zero(0.0f);
  const R dim_xm = i >= 1 ? num_in<R>(ax.dim[i - 1]) : zero, dim_x = num_in<R>(ax.dim[i]);
  const R dim_ym = j >= 1 ? num_in<R>(ay.dim[j - 1]) : zero, dim_y = num_in<R>(ay.dim[j]);
  const R di_x = num_in<R>(ax.di[i]), di_y = num_in<R>(ay.di[j]);
  const R di_xm = i >= 1 ? num_in<R>(ax.di[i - 1]) : zero;
  const R di_xp = i <= g.ix - 2 ? num_in<R>(ax.di[i + 1]) : zero;
  const R di_ym = j >= 1 ? num_in<R>(ay.di[j - 1]) : zero;
  const R di_yp = j <= g.jx - 2 ? num_in<R>(ay.di[j + 1]) : zero;
  // artificial-viscosity coefficients of the four faces (mlw_m3.f:324-334)
  // and their derivatives in dv: q = qav dxm max(0, |dv| - eps)
  const double *VX = P + P_VX * n, *VY = P + P_VY * n;
  R qxm = zero, qxp = zero, qym = zero, qyp = zero, gxm = zero, gxp = zero, gym = zero,
    gyp = zero;
  const float eps = 1.0e-4f;  // the real*4 literal of the reference
  if (i >= 1) {
    const R d = num_in<R>(VX[c]) - num_in<R>(VX[c - sx]);
    const R e = fabs(d) - eps;
    const R qd = ph.qav * num_in<R>(ax.dm[i - 1]);
    qxm = e > 0.0f ? qd * e : zero;
    gxm = e > 0.0f ? (d > 0.0f ? qd : -qd) : zero;
  }
  if (i <= g.ix - 2) {
    const R d = num_in<R>(VX[c + sx]) - num_in<R>(VX[c]);
    const R e = fabs(d) - eps;
    const R qd = ph.qav * num_in<R>(ax.dm[i]);
    qxp = e > 0.0f ? qd * e : zero;
    gxp = e > 0.0f ? (d > 0.0f ? qd : -qd) : zero;
  }
  if (j >= 1) {
    const R d = num_in<R>(VY[c]) - num_in<R>(VY[c - sy]);
    const R e = fabs(d) - eps;
    const R qd = ph.qav * num_in<R>(ay.dm[j - 1]);
    qym = e > 0.0f ? qd * e : zero;
    gym = e > 0.0f ? (d > 0.0f ? qd : -qd) : zero;
  }
  if (j <= g.jx - 2) {
    const R d = num_in<R>(VY[c + sy]) - num_in<R>(VY[c]);
    const R e = fabs(d) - eps;
    const R qd = ph.qav * num_in<R>(ay.dm[j]);
    qyp = e > 0.0f ? qd * e : zero;
    gyp = e > 0.0f ? (d > 0.0f ? qd : -qd) : zero;
  }
  const bool aqxm_on = qxm != 0.0f, aqxp_on = qxp != 0.0f;
  const bool aqym_on = qym != 0.0f, aqyp_on = qyp != 0.0f;
  // coefficients shared by the 8 variables: viscosity in U (mlwartv.f),
  // half-step differences (mlwhalf.f part 1), corner predictor (part 2),
  // viscosity in q; zero where the reading cell is not updated
  const R cxm = in_xm ? dt * di_xm * qxm * dim_xm : zero;
  const R cxp = in_xp ? dt * di_xp * qxp * dim_x : zero;
  const R cym = in_ym ? dt * di_ym * qym * dim_ym : zero;
  const R cyp = in_yp ? dt * di_yp * qyp * dim_y : zero;
  const R c0 = in_c ? dt * (di_x * (qxp * dim_x + qxm * dim_xm) +
                            di_y * (qyp * dim_y + qym * dim_ym))
                    : zero;
  const bool av = aqxm_on | aqxp_on | aqym_on | aqyp_on;
  const R hxm = i >= 1 ? 0.25f * dt * di_xm : zero;
  const R hxp = i <= g.ix - 2 ? 0.25f * dt * di_xp : zero;
  const R hym = j >= 1 ? 0.25f * dt * di_ym : zero;
  const R hyp = j <= g.jx - 2 ? 0.25f * dt * di_yp : zero;
  const R pxm = i >= 1 ? 0.5f * dt * dim_xm : zero;
  const R pxp = i <= g.ix - 2 ? 0.5f * dt * dim_x : zero;
  const R pym = j >= 1 ? 0.5f * dt * dim_ym : zero;
  const R pyp = j <= g.jx - 2 ? 0.5f * dt * dim_y : zero;
  // d(du(o))/dq(face) per unit dU: the cell below the face gains, the cell
  // above loses (in_* already folded in)
  const R wxm_a = in_xm ? dt * dim_xm * di_xm : zero;
  const R wxm_b = (in_c && i >= 1) ? dt * dim_xm * di_x : zero;
  const R wxp_a = in_c ? dt * dim_x * di_x : zero;
  const R wxp_b = in_xp ? dt * dim_x * di_xp : zero;
  const R wym_a = in_ym ? dt * dim_ym * di_ym : zero;
  const R wym_b = (in_c && j >= 1) ? dt * dim_ym * di_y : zero;
  const R wyp_a = in_c ? dt * dim_y * di_y : zero;
  const R wyp_b = in_yp ? dt * dim_y * di_yp : zero;
  R aqxm = zero, aqxp = zero, aqym = zero, aqyp = zero;
#pragma unroll 1
  for (int v = 0; v < 8; v++) {
    const double *a = A1 + v * n, *h = A2 + v * n;
    const R l0 = in_c ? num_ld<R>(a + c) : zero;
    const R lxm = in_xm ? num_ld<R>(a + c - sx) : zero, lxp = in_xp ? num_ld<R>(a + c + sx) : zero;
    const R lym = in_ym ? num_ld<R>(a + c - sy) : zero, lyp = in_yp ? num_ld<R>(a + c + sy) : zero;
    const R hmm = k_mm ? num_ld<R>(h + c - sx - sy) : zero, hpm = k_pm ? num_ld<R>(h + c - sy) : zero;
    const R hmp = k_mp ? num_ld<R>(h + c - sx) : zero, hpp = k_pp ? num_ld<R>(h + c) : zero;
    const R ylo = hmm + hpm, yhi = hmp + hpp;  // corners below / above
    // U' = U + du on the interior; 0.25 of each surrounding corner
    R au = fma(R(0.25f), ylo + yhi, l0);
    if (av) au = fma(cxm, lxm, fma(cxp, lxp, fma(cym, lym, fma(cyp, lyp, fma(-c0, l0, au)))));
    num_st(sU + v * kT, au);
    num_st(sX + v * kT, fma(hxp, lxp, fma(-hxm, lxm, fma(pxp, hpm + hpp, -(pxm * (hmm + hmp))))));
    num_st(sY + v * kT, fma(hyp, lyp, fma(-hym, lym, fma(pyp, yhi, -(pym * ylo)))));
    if (av) {
      const double *U = CU + v * n;
      const R u0 = num_ld<R>(U + c);
      if (aqxm_on)
        aqxm = fma(u0 - num_ld<R>(U + c - sx), fma(wxm_a, lxm, -(wxm_b * l0)), aqxm);
      if (aqxp_on)
        aqxp = fma(num_ld<R>(U + c + sx) - u0, fma(wxp_a, l0, -(wxp_b * lxp)), aqxp);
      if (aqym_on)
        aqym = fma(u0 - num_ld<R>(U + c - sy), fma(wym_a, lym, -(wym_b * l0)), aqym);
      if (aqyp_on)
        aqyp = fma(num_ld<R>(U + c + sy) - u0, fma(wyp_a, l0, -(wyp_b * lyp)), aqyp);
    }
  }
  R ap[8];
  cell_reverse<R, true>(p, ph, sU, sX, sY, ap);
  // q(face) = qav dxm max(0, |v(+) - v(-)| - eps): the cell is (+) of the
  // lower face and (-) of the upper face
  ap[P_VX] += aqxm * gxm - aqxp * gxp;
  ap[P_VY] += aqym * gym - aqyp * gyp;
  // cells the step does not update pass the adjoint through
  if (!in_c) {
#pragma unroll
    for (int v = 0; v < 8; v++) ap[v] += num_in<R>(lam[v * n + c]);
  }
#pragma unroll
  for (int v = 0; v < 8; v++) out[v * n + c] = num_out(ap[v]);
  out[P_AZ * n + c] = 0.0;
}

// Transpose of the boundary program of one axis on one line, over all
// variables: the rules of bd_line (bc_line.cuh) in reverse order, each
// assignment dst = s*src turned into a(src) += s*a(dst), a(dst) = 0.
__device__ void bd_line_t(int kind, int mbnd, int m, double *q, int n, size_t st,
                          const double *dxm) {
#define QL(l) q[(size_t)((l)-1) * st]
  if (kind == BD_PER) {
    const int b0 = 1 + m, b1 = n - m;
    if (mbnd == 0)
      for (int i = m; i >= 1; i--) { QL(b1 + 1 - i) += QL(b0 - i); QL(b0 - i) = 0.0; }
    else
      for (int i = m; i >= 1; i--) { QL(b0 - 1 + i) += QL(b1 + i); QL(b1 + i) = 0.0; }
    return;
  }
  if (mbnd == 0) {
    const int b = 1 + m;
    switch (kind) {
      case BD_SPP: for (int i = m; i >= 1; i--) { QL(b - 1 + i) += QL(b - i); QL(b - i) = 0.0; } break;
      case BD_SPN: for (int i = m; i >= 1; i--) { QL(b - 1 + i) -= QL(b - i); QL(b - i) = 0.0; } break;
      case BD_SMP: for (int i = m; i >= 1; i--) { QL(b + i) += QL(b - i); QL(b - i) = 0.0; } break;
      case BD_SMN:
        QL(b) = 0.0;
        for (int i = m; i >= 1; i--) { QL(b + i) -= QL(b - i); QL(b - i) = 0.0; }
        break;
      case BD_FRE: for (int i = m; i >= 1; i--) { QL(b) += QL(b - i); QL(b - i) = 0.0; } break;
      case BD_CNS: for (int i = m; i >= 1; i--) QL(b - i) = 0.0; break;
      case BD_FRD: {
        double adq = 0.0;  // q(b-i) = q(b-i+1) - dqq dxm(b-i), dqq = (q(b+1)-q(b))/dxm(b)
        for (int i = m; i >= 1; i--) {
          QL(b - i + 1) += QL(b - i);
          adq -= QL(b - i) * dxm[b - i - 1];
          QL(b - i) = 0.0;
        }
        QL(b + 1) += adq / dxm[b - 1];
        QL(b) -= adq / dxm[b - 1];
        break;
      }
      default: break;
    }
  } else {
    const int b = n - m;
    switch (kind) {
      case BD_SPP: for (int i = m; i >= 1; i--) { QL(b + 1 - i) += QL(b + i); QL(b + i) = 0.0; } break;
      case BD_SPN: for (int i = m; i >= 1; i--) { QL(b + 1 - i) -= QL(b + i); QL(b + i) = 0.0; } break;
      case BD_SMP: for (int i = m; i >= 1; i--) { QL(b - i) += QL(b + i); QL(b + i) = 0.0; } break;
      case BD_SMN:
        QL(b) = 0.0;
        for (int i = m; i >= 1; i--) { QL(b - i) -= QL(b + i); QL(b + i) = 0.0; }
        break;
      case BD_FRE: for (int i = m; i >= 1; i--) { QL(b) += QL(b + i); QL(b + i) = 0.0; } break;
      case BD_CNS: for (int i = m; i >= 1; i--) QL(b + i) = 0.0; break;
      case BD_FRD: {
        double adq = 0.0;  // q(b+i) = q(b+i-1) + dqq dxm(b+i-1), dqq = (q(b)-q(b-1))/dxm(b-1)
        for (int i = m; i >= 1; i--) {
          QL(b + i - 1) += QL(b + i);
          adq += QL(b + i) * dxm[b + i - 2];
          QL(b + i) = 0.0;
        }
        QL(b) += adq / dxm[b - 2];
        QL(b - 1) -= adq / dxm[b - 2];
        break;
      }
      default: break;
    }
  }
#undef QL
}

__global__ void k_bc2d_t(int nvar, double *L, int ix, int jx, int axis, BcTable bc,
                         const double *dxm) {
  const int n = axis == 0 ? ix : jx;
  const size_t st = axis == 0 ? 1 : (size_t)ix;
  const long long nlines = axis == 0 ? jx : ix;
  const size_t nall = (size_t)ix * jx;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < nlines * nvar;
       t += (long long)gridDim.x * blockDim.x) {
    const int v = (int)(t / nlines);
    const long long line = t % nlines;
    double *q = L + (size_t)v * nall + (axis == 0 ? (size_t)line * ix : (size_t)line);
    const int klo = bc.kind[v][2 * axis], khi = bc.kind[v][2 * axis + 1];
    // the forward applies the lower then the upper rule: reverse order here
    if (khi >= 0) bd_line_t(khi, 1, bc.margin, q, n, st, dxm);
    if (klo >= 0) bd_line_t(klo, 0, bc.margin, q, n, st, dxm);
  }
}

// Error-free sum of two doubles (Knuth's TwoSum): s + e == a + b exactly.
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
  s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
}
// (s, c) += (t, d): a compensated partial sum, the rounding errors of every
// addition carried in c (the cascaded summation of Ogita, Rump and Oishi,
// "Accurate sum and dot product", 2005), so that J is the exact sum of its
// terms to about one rounding -- a finite difference of J then sees the
// state's rounding, not that of a 65k-term sum.
__device__ __forceinline__ void comp_add(double &s, double &c, double t, double d) {
  double e;
  two_sum(s, t, s, e);
  c = __dadd_rn(c, __dadd_rn(d, e));
}

// J = sum over the interior of (bx^2+by^2+bz^2)/(8 pi) dx dy (compensated
// block partial sums, reduced in a fixed order by k_sum_final) and its
// gradient
__global__ void __launch_bounds__(256)
    k_objective(const double *__restrict__ P, double *__restrict__ lam,
                double *__restrict__ part, G2 g, Axis ax, Axis ay, Phys ph) {
  __shared__ double red[2][256];
  double s = 0.0, c = 0.0;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < g.n;
       k += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(k % g.ix), j = (int)(k / g.ix);
    const double bx = P[P_BX * g.n + k], by = P[P_BY * g.n + k], bz = P[P_BZ * g.n + k];
    const bool in = interior(g, i, j);
    const double w = in ? ax.d[i] * ay.d[j] : 0.0;
    comp_add(s, c, (bx * bx + by * by + bz * bz) * ph.pi8i * w, 0.0);
    if (lam) {
#pragma unroll
      for (int v = 0; v < 9; v++) lam[v * g.n + k] = 0.0;
      lam[P_BX * g.n + k] = 2.0 * ph.pi8i * w * bx;
      lam[P_BY * g.n + k] = 2.0 * ph.pi8i * w * by;
      lam[P_BZ * g.n + k] = 2.0 * ph.pi8i * w * bz;
    }
  }
  red[0][threadIdx.x] = s;
  red[1][threadIdx.x] = c;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      double a = red[0][threadIdx.x], b = red[1][threadIdx.x];
      comp_add(a, b, red[0][threadIdx.x + o], red[1][threadIdx.x + o]);
      red[0][threadIdx.x] = a;
      red[1][threadIdx.x] = b;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = red[0][0];
    part[2 * blockIdx.x + 1] = red[1][0];
  }
}

__global__ void k_sum_final(const double *part, int nb, double *out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0, c = 0.0;
    for (int b = 0; b < nb; b++) comp_add(s, c, part[2 * b], part[2 * b + 1]);
    *out = __dadd_rn(s, c);
  }
}

}  // namespace

size_t adj2d_scratch_doubles(size_t ncells) { return 40 * ncells + 1024; }

cudaError_t launch_adj2d_step(const double *P, const double *R, const double *lam_in,
                              double *lam_out, double *scratch, int ix, int jx,
                              const Axis &ax, const Axis &ay, const Phys &ph,
                              double dt, bool df, cudaStream_t s) {
  G2 g{ix, jx, (size_t)ix * jx};
  double *A1 = scratch, *A2 = scratch + 8 * g.n, *CU = scratch + 16 * g.n;
  const unsigned blocks = (unsigned)((g.n + kT - 1) / kT);
  if (df) {
    k_adj_cells<df::DF><<<blocks, kT, 0, s>>>(P, R, lam_in, A1, CU, g, ph);
    k_adj_corners<df::DF><<<blocks, kT, 0, s>>>(CU, A1, A2, g, ax, ay, ph, dt);
    k_adj_gather<df::DF><<<blocks, kT, 0, s>>>(P, CU, A1, A2, lam_in, lam_out, g, ax, ay, ph,
                                               dt);
  } else {
    k_adj_cells<double><<<blocks, kT, 0, s>>>(P, R, lam_in, A1, CU, g, ph);
    k_adj_corners<double><<<blocks, kT, 0, s>>>(CU, A1, A2, g, ax, ay, ph, dt);
    k_adj_gather<double><<<blocks, kT, 0, s>>>(P, CU, A1, A2, lam_in, lam_out, g, ax, ay, ph,
                                               dt);
  }
  count_launch(3);
  return cudaGetLastError();
}

cudaError_t launch_bc2d_transpose(int nvar, double *lam, int ix, int jx,
                                  const Axis &ax, const Axis &ay, const BcTable &bc,
                                  cudaStream_t s) {
  // the forward fills x, then y: transpose y first
  for (int axis = 1; axis >= 0; axis--) {
    const long long total = (long long)(axis == 0 ? jx : ix) * nvar;
    int blocks = (int)((total + 127) / 128);
    if (blocks < 1) blocks = 1;
    k_bc2d_t<<<blocks, 128, 0, s>>>(nvar, lam, ix, jx, axis, bc, axis == 0 ? ax.dm : ay.dm);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Raw output of a step rebuilt from the two filled states around it: the
// step writes every cell but the outer layer, which it copies from its input,
// and a boundary program of margin 1 without bdsmn* rules then rewrites only
// that layer.  So R = P_next inside, P_cur on the outer layer.
__global__ void k_adj_merge(const double *__restrict__ P_next,
                            const double *__restrict__ P_cur, double *__restrict__ R,
                            int nvar, int ix, int jx) {
  const size_t n = (size_t)ix * jx;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n * nvar;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t c = t % n;
    const int i = (int)(c % ix), j = (int)(c / ix);
    const bool edge = i == 0 || i == ix - 1 || j == 0 || j == jx - 1;
    R[t] = edge ? P_cur[t] : P_next[t];
  }
}

cudaError_t launch_adj2d_merge(const double *P_next, const double *P_cur, double *R,
                               int nvar, int ix, int jx, cudaStream_t s) {
  const size_t total = (size_t)ix * jx * nvar;
  size_t blocks = (total + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  k_adj_merge<<<(unsigned)blocks, 256, 0, s>>>(P_next, P_cur, R, nvar, ix, jx);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_adj2d_objective(const double *P, double *lam, double *J,
                                   double *scratch, int ix, int jx, const Axis &ax,
                                   const Axis &ay, const Phys &ph, cudaStream_t s) {
  G2 g{ix, jx, (size_t)ix * jx};
  const int nb = 256;
  double *part = scratch;
  k_objective<<<nb, 256, 0, s>>>(P, lam, part, g, ax, ay, ph);
  k_sum_final<<<1, 32, 0, s>>>(part, nb, J);
  count_launch(2);
  return cudaGetLastError();
}

}  // namespace cans
