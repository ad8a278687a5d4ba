// Fused 3-D modified Lax-Wendroff step, fast policy (sm_103a, FP64): mlw_m
// (cans3d/hdmlw/mlw_m.f:2-453), with G mlw_m_g (mlw_m_g.f:2-469) and with R
// mlw_m_e (mlw_m_e.f:103-115, 257-270) given the eta J fields of mlw3d_e.cu,
// and the CFL of cans3d/common/cfl_m.f:39-85.  The exact policy's kernel, one
// operation of the reference after the other, is in mlw3d.cu.
//
// What bounds the step is the FP64 pipe (two lanes per SM and clock; HBM is at
// 2 %), so the kernel is laid out for the fewest FP64 warp instructions:
//  - A block owns a TX x TY column of cells and marches along z.  Per plane:
//    the cells of plane k+1 and, by other warps, the new primitives of plane k-1;
//    the predictor's sums of the corners of plane k+1/2; their fluxes; the full step
//    of plane k.  Each phase numbers its own work items (cells of the halo tile,
//    corners, interior cells) through the threads, so that its warps are full.
//  - The predictor's eight-cell sums and, on equally spaced axes, the corrector's
//    differences and face sums are integer sums (isum.cuh): no FP64 instruction.
//    They are chains of some 150 integer instructions, so two threads share a corner
//    and a cell, with four of the eight variables each: 20 warps a SM where one
//    thread for all eight leaves room for 10 (256^3: 16.7 against 16.3 ms, at the
//    same FP64 work for the shared part done twice).
//  - The corner quantities are kept at eight times their value (the eight-cell
//    mean is a sum, every flux is linear in the conserved variables at given
//    velocity), the factor is in constants and weights: no scaling products.
//  - The momentum flux is symmetric and the total pressure is formed once, as
//    in the double-float step.
//  - The corrector's x and y differences of a corner plane serve the cell
//    planes on both of its sides, and the z flux of a face (corner average,
//    central part and viscosity) the cells on both of its sides: each is formed
//    once and kept in shared memory (22 values a column).  So the corner ring
//    needs one plane, and nothing of the cell plane k-1 is kept.
//  - u_new = u + du with every term of du summed first: its terms round at
//    their own size.
//  - reciprocals of fd64.cuh; comparisons on the integer pipe; signs flipped on
//    the upper word (the compiler negates a double with an FP64 addition: 256^3
//    15.9 -> 14.1 ms for the loops over the variables).
// FP64 warp instructions a zone (32 a warp instruction, 16 x 8 tiles): 308, against
// 588 with all sums in FP64 (18.2 ms at 256^3) and 920 of one that forms each cell's
// sums for itself (29.9 ms).  Shared memory 114 KB, 96 registers: two blocks a SM,
// whose phases overlap.
#include <cuda_runtime.h>

#include <mutex>

#include "cans_common.cuh"
#include "cans_internal.h"
#include "cfl3.cuh"
#include "fd64.cuh"
#include "isum.cuh"
#include "mlw3d_march.cuh"

namespace cans {

namespace {

// x with its sign flipped where s < 0 (on its upper word: the negation of a double is
// an FP64 instruction)
__device__ __forceinline__ double signed_by(double x, int s) {
  return __hiloint2double(__double2hiint(x) ^ (s & (int)0x80000000), __double2loint(x));
}

// The predictor of four variables of one corner with FP64 sums, where an integer sum cannot be formed
// (isum::special): l and h the lower left cell of the corner's two planes, gl and gh
// that of the gravity sources, ks the corner's slots.
template <class T, bool G>
__device__ __noinline__ void predict_fp64(const double *l, const double *h, const double *gl,
                                          const double *gh, double *ks, int v0, double cxk,
                                          double cyk, double czk, double dt) {
  auto sum = [&](const double *p) { return (p[0] + p[1]) + (p[T::CX] + p[T::CX + 1]); };
  auto dx = [&](const double *p) { return (p[1] - p[0]) + (p[T::CX + 1] - p[T::CX]); };
  auto dy = [&](const double *p) { return (p[T::CX] - p[0]) + (p[T::CX + 1] - p[1]); };
#pragma unroll 1
  for (int v = v0; v < v0 + 4; v++) {
    const VarFields q = kVar[v];
    const size_t x = (size_t)q.fx * T::NC, y = (size_t)q.fy * T::NC, z = (size_t)q.fz * T::NC;
    const size_t o = (size_t)v * T::NC;
    double r = sum(l + o) + sum(h + o);
    if (q.fx >= 0) r = fma(signed_by(cxk, q.sx), dx(l + x) + dx(h + x), r);
    if (q.fy >= 0) r = fma(signed_by(cyk, q.sy), dy(l + y) + dy(h + y), r);
    if (q.fz >= 0) r = fma(signed_by(czk, q.sz), sum(h + z) - sum(l + z), r);
    if constexpr (G) {
      if (q.g >= 0) {
        const size_t s = (size_t)q.g * T::NC;
        r = fma(dt, sum(gl + s) + sum(gh + s), r);
      }
    }
    ks[(size_t)v * T::NK] = r;
  }
}

// isum::diff_planes and face_planes of one variable in FP64, with the weights
// themselves: o = tx, ty, tz, gx, gy, pu of the full step.
template <class T>
__device__ __noinline__ void cell_fp64(VarFields q, const double *s0, const double *s1,
                                       const double *kk, double gxl, double gyl, double pl,
                                       double w, double ux0, double ux1, double uy0, double uy1,
                                       double uz0, double uz1, double *o) {
  o[0] = o[1] = o[3] = o[4] = 0.0;
  o[5] = w;
  if (q.fx >= 0) {
    const double *k = kk + (size_t)q.kx * T::NK, *f = s0 + (size_t)q.fx * T::NC;
    o[3] = 2.0 * (uy0 * (k[1] - k[0]) + uy1 * (k[T::KX + 1] - k[T::KX]));
    o[0] = 2.0 * (uz0 * gxl + uz1 * o[3]) + 16.0 * (f[1] - f[-1]);
  }
  if (q.fy >= 0) {
    const double *k = kk + (size_t)q.ky * T::NK, *f = s0 + (size_t)q.fy * T::NC;
    o[4] = 2.0 * (ux0 * (k[T::KX] - k[0]) + ux1 * (k[T::KX + 1] - k[1]));
    o[1] = 2.0 * (uz0 * gyl + uz1 * o[4]) + 16.0 * (f[T::CX] - f[-T::CX]);
  }
  if (q.fz >= 0) {
    const double *k = kk + (size_t)q.kz * T::NK;
    const double *f0 = s0 + (size_t)q.fz * T::NC, *f1 = s1 + (size_t)q.fz * T::NC;
    const double s = 4.0 * (uy0 * (ux0 * k[0] + ux1 * k[1]) +
                            uy1 * (ux0 * k[T::KX] + ux1 * k[T::KX + 1]));
    const double p = s + 16.0 * (f0[0] + f1[0]);
    o[5] = (q.sz < 0 ? -p : p) + w;
  }
  o[2] = o[5] - pl;
}

}  // namespace

template <int TX, int TY, bool G, bool R, int MINB, bool U>
__global__ void __launch_bounds__(T3F<TX, TY, G>::NT, MINB)
    k_mlw3d_fast(const double *__restrict__ A, double *__restrict__ B, int ix, int jx, int kx,
                 Axis ax, Axis ay, Axis az, Phys ph, double dt_arg, Ctl *__restrict__ ctl,
                 Box3 box, int kchunk, const double *__restrict__ grav,
                 const double *__restrict__ res) {
  using T = T3F<TX, TY, G>;
  extern __shared__ double smem[];
  double *scell = smem;                               // [2][NCF][NC]
  double *sk = scell + 2 * (size_t)NCF * T::NC;       // [NKF][NK]
  double *sqx = sk + (size_t)NKF * T::NK;             // q / dxm of plane k
  double *sqy = sqx + T::NQX;
  double *sret = sqy + T::NQY;                        // [NR][NI]
  double *sun = sret + (size_t)T::NR * T::NI;         // [4][NI]: new values 4 .. 7
  double *sred = sun + 4 * (size_t)T::NI;
  double *szc = sred + 32;                            // of plane k: viscosity, flux factor
  double *sgc = szc + 2;                              // G: [2][4][NC]
  double *sgk = sgc + 2 * 4 * (size_t)T::NC;          // G: [4][NK]

  if (ctl != nullptr) {
    if (ctl->done | ctl->pause) return;
    A = ctl->buf[ctl->cur];
    B = ctl->buf[ctl->cur ^ 1];
  }
  const double dt = ctl != nullptr ? ctl->dt : dt_arg;
  const size_t plane = (size_t)ix * jx, n = plane * kx;
  const int tid = threadIdx.x;
  const int i0 = 1 + blockIdx.x * TX, j0 = 1 + blockIdx.y * TY;
  const int kb = 1 + blockIdx.z * kchunk, ke = min(kx - 2, kb + kchunk - 1);
  if (kb > ke) return;

  // the thread's cell of the halo tile; ghost cells keep their input values (mlw_m.f
  // updates only 2..n-1) and are copied by the block of their nearest interior cell
  const int ct = tid - T::T0, hx = ct % T::CX, hy = ct / T::CX;
  const int gi = i0 - 1 + hx, gj = j0 - 1 + hy;
  const bool cell = ct >= 0 && ct < T::NC, in_arr = cell && gi < ix && gj < jx;
  const int ci = min(max(gi, 1), ix - 2), cj = min(max(gj, 1), jx - 2);
  const bool owned = in_arr && ci >= i0 && ci < i0 + TX && cj >= j0 && cj < j0 + TY;
  const bool xy_ghost = owned && (gi != ci || gj != cj);
  // its corner (two threads a corner, four variables each), and the corner's
  // predictor coefficients -8 dt / (4 dxm)
  const int kt = tid % T::NKW, kv0 = tid < T::NKW ? 0 : 4;
  const int cx = kt % T::KX, cy = kt / T::KX;
  const bool corner = kt < T::NK;
  const bool cor_in = corner && i0 - 1 + cx <= ix - 2 && j0 - 1 + cy <= jx - 2;
  const int p00 = cx + cy * T::CX;
  const double cxk = cor_in ? -2.0 * dt * ax.dim[i0 - 1 + cx] : 0.0;
  const double cyk = cor_in ? -2.0 * dt * ay.dim[j0 - 1 + cy] : 0.0;
  // its interior cell (two threads a cell, four variables each)
  const int it = tid % T::NI, iv0 = tid < T::NI ? 0 : 4;
  const int lx = it % TX + 1, ly = it / TX + 1;
  const int ii = i0 - 1 + lx, jj = j0 - 1 + ly;
  const bool interior = tid < 2 * T::NI && ii <= ix - 2 && jj <= jx - 2;
  const int c0 = lx + ly * T::CX;
  const int kSW = (lx - 1) + (ly - 1) * T::KX;
  // the viscosity faces (qav dm dim of an x and a y face) of the upper threads
  const int ft = tid - T::NKW;
  const int fxx = ft % T::KX, fxr = ft / T::KX, fyx = ft % TX, fyr = ft / TX;
  const bool facex = ft >= 0 && ft < T::NQX && i0 + fxx < ix && j0 + fxr < jx;
  const bool facey = ft >= 0 && ft < T::NQY && i0 + fyx < ix && j0 + fyr < jx;
  const double qxc = facex ? ph.qav * ax.dm[i0 - 1 + fxx] * ax.dim[i0 - 1 + fxx] : 0.0;
  const double qyc = facey ? ph.qav * ay.dm[j0 - 1 + fyr] * ay.dim[j0 - 1 + fyr] : 0.0;

  auto cslot = [&](int k) { return scell + (size_t)(k & 1) * NCF * T::NC; };
  auto gslot = [&](int k) { return sgc + (size_t)(k & 1) * 4 * T::NC; };

  // ---- cells of plane k (mlw_m.f:74-202) -----------------------------------
  auto load_plane = [&](int k) {
    if (!cell) return;
    double *sl = cslot(k) + ct;
#define S(f) sl[(size_t)(f) * T::NC]
    if (!in_arr) {
#pragma unroll 1
      for (int f = 0; f < NCF; f++) S(f) = 0.0;
      if constexpr (G)
        for (int f = 0; f < 4; f++) gslot(k)[f * T::NC + ct] = 0.0;
      return;
    }
    const size_t g = (size_t)gi + (size_t)gj * ix + (size_t)k * plane;
    const double ro = A[P3::RO * n + g], pr = A[P3::PR * n + g];
    const double vx = A[P3::VX * n + g], vy = A[P3::VY * n + g], vz = A[P3::VZ * n + g];
    const double bx = A[P3::BX * n + g], by = A[P3::BY * n + g], bz = A[P3::BZ * n + g];
    if (xy_ghost ? k == 0 || k >= kb && k <= ke || k == kx - 1
                 : owned && (k == 0 || k == kx - 1)) {
      B[P3::RO * n + g] = ro;
      B[P3::PR * n + g] = pr;
      B[P3::VX * n + g] = vx;
      B[P3::VY * n + g] = vy;
      B[P3::VZ * n + g] = vz;
      B[P3::BX * n + g] = bx;
      B[P3::BY * n + g] = by;
      B[P3::BZ * n + g] = bz;
    }
    const double rx = ro * vx, ry = ro * vy, rz = ro * vz;
    const double ek = 0.5 * fma(rx, vx, fma(ry, vy, rz * vz));
    const double bb = fma(bx, bx, fma(by, by, bz * bz));
    const double ep = fma(pr, ph.ggm1, ek);
    double ex = fma(vz, by, -vy * bz), ey = fma(vx, bz, -vz * bx), ez = fma(vy, bx, -vx * by);
    if constexpr (R) {
      ex += res[g];
      ey += res[n + g];
      ez += res[2 * n + g];
    }
    const double pbx = ph.pi4i * bx, pby = ph.pi4i * by, pbz = ph.pi4i * bz;
    const double pt = fma(ph.pi8i, bb, pr);
    S(CRO) = ro; S(CEE) = fma(pr, ph.gm1i, fma(ph.pi8i, bb, ek));
    S(CRX) = rx; S(CRY) = ry; S(CRZ) = rz;
    S(CBX) = bx; S(CBY) = by; S(CBZ) = bz;
    S(CEX) = ex; S(CEY) = ey; S(CEZ) = ez;
    S(CVX) = vx; S(CVY) = vy; S(CVZ) = vz;
    S(CFX) = fma(ep, vx, fma(pbz, ey, -pby * ez));
    S(CFY) = fma(ep, vy, fma(pbx, ez, -pbz * ex));
    S(CFZ) = fma(ep, vz, fma(pby, ex, -pbx * ey));
    S(CXX) = fma(rx, vx, fma(-pbx, bx, pt));
    S(CYY) = fma(ry, vy, fma(-pby, by, pt));
    S(CZZ) = fma(rz, vz, fma(-pbz, bz, pt));
    S(CXY) = fma(rx, vy, -pbx * by);
    S(CXZ) = fma(rx, vz, -pbx * bz);
    S(CYZ) = fma(ry, vz, -pby * bz);
    if constexpr (G) {  // mlw_m_g.f:135-136, 154, 172, 190
      const double gx = grav[g], gy = grav[2 * n + g], gz = grav[4 * n + g];
      double *gs = gslot(k) + ct;
      gs[0] = fma(rx, gx, fma(ry, gy, rz * gz));
      gs[T::NC] = ro * gx;
      gs[2 * T::NC] = ro * gy;
      gs[3 * T::NC] = ro * gz;
    }
#undef S
  };

  // ---- eight times the state predicted at the corners of plane k + 1/2
  // (mlwhalf.f:49-65), into the corner's own slots 0 .. 7; 0 outside the array
  auto corner_sums = [&](int k) {
    if (!cor_in) return;
    double *ks = sk + kt;
    const double czk = -2.0 * dt * az.dim[k];
    const double *L = cslot(k) + p00, *H = cslot(k + 1) + p00;
    bool sp = false;
#pragma unroll 1
    for (int v = kv0; v < kv0 + 4; v++) {
      const VarFields q = kVar[v];
      auto at = [&](const double *p, int f) { return p + (size_t)f * T::NC; };
      double r = isum::eight<T::CX, isum::kSum>(at(L, v), at(H, v), sp);
      if (q.fx >= 0)
        r = fma(signed_by(cxk, q.sx), isum::eight<T::CX, isum::kDx>(at(L, q.fx), at(H, q.fx), sp),
                r);
      if (q.fy >= 0)
        r = fma(signed_by(cyk, q.sy), isum::eight<T::CX, isum::kDy>(at(L, q.fy), at(H, q.fy), sp),
                r);
      if (q.fz >= 0)
        r = fma(signed_by(czk, q.sz), isum::eight<T::CX, isum::kDz>(at(L, q.fz), at(H, q.fz), sp),
                r);
      if constexpr (G) {  // mlwsrch part 2: dt times the mean of the eight sources
        if (q.g >= 0) {
          const size_t o = (size_t)q.g * T::NC + p00;
          r = fma(dt, isum::eight<T::CX, isum::kSum>(gslot(k) + o, gslot(k + 1) + o, sp), r);
        }
      }
      ks[(size_t)v * T::NK] = r;
    }
    if (sp)  // a call, so that the FP64 sums are not predicated in
      predict_fp64<T, G>(L, H, G ? gslot(k) + p00 : nullptr, G ? gslot(k + 1) + p00 : nullptr, ks,
                         kv0, cxk, cyk, czk, dt);
  };

  // ---- fluxes of the corners of plane k + 1/2 (mlw_m.f:205-334) --------------
  auto corner_fluxes = [&](int k) {
    double *ks = sk + kt;
#define KS(f) ks[(size_t)(f) * T::NK]
    if (!cor_in) return;
    const size_t gc = (size_t)(i0 - 1 + cx) + (size_t)(j0 - 1 + cy) * ix + (size_t)k * plane;
    double rq[3] = {0.0, 0.0, 0.0}, gq[3] = {0.0, 0.0, 0.0};
    if constexpr (R) {
      rq[0] = res[3 * n + gc];
      rq[1] = res[4 * n + gc];
      rq[2] = res[5 * n + gc];
    }
    if constexpr (G) {
      gq[0] = grav[n + gc];
      gq[1] = grav[3 * n + gc];
      gq[2] = grav[5 * n + gc];
    }
    const double ro = KS(CRO), ee = KS(CEE), rx = KS(CRX), ry = KS(CRY), rz = KS(CRZ);
    const double bx = KS(CBX), by = KS(CBY), bz = KS(CBZ);
    // primitives and fluxes of the eightfold state: B B terms carry 64
    const double k4 = 0.125 * ph.pi4i, k8 = 0.125 * ph.pi8i;
    const double ri = fd::rcp(ro);
    const double vx = rx * ri, vy = ry * ri, vz = rz * ri;
    const double ek = 0.5 * fma(rx, vx, fma(ry, vy, rz * vz));
    const double bb = fma(bx, bx, fma(by, by, bz * bz));
    const double pr = ph.gm1 * fma(-k8, bb, ee - ek);
    const double ep = fma(pr, ph.ggm1, ek);
    double ex = fma(vz, by, -vy * bz), ey = fma(vx, bz, -vz * bx), ez = fma(vy, bx, -vx * by);
    if constexpr (R) {
      ex = fma(8.0, rq[0], ex);
      ey = fma(8.0, rq[1], ey);
      ez = fma(8.0, rq[2], ez);
    }
    const double pbx = k4 * bx, pby = k4 * by, pbz = k4 * bz;
    const double pt = fma(k8, bb, pr);
    KS(KRX) = rx; KS(KRY) = ry; KS(KRZ) = rz;
    KS(KEX) = ex; KS(KEY) = ey; KS(KEZ) = ez;
    KS(KFX) = fma(ep, vx, fma(pbz, ey, -pby * ez));
    KS(KFY) = fma(ep, vy, fma(pbx, ez, -pbz * ex));
    KS(KFZ) = fma(ep, vz, fma(pby, ex, -pbx * ey));
    KS(KXX) = fma(rx, vx, fma(-pbx, bx, pt));
    KS(KYY) = fma(ry, vy, fma(-pby, by, pt));
    KS(KZZ) = fma(rz, vz, fma(-pbz, bz, pt));
    KS(KXY) = fma(rx, vy, -pbx * by);
    KS(KXZ) = fma(rx, vz, -pbx * bz);
    KS(KYZ) = fma(ry, vz, -pby * bz);
    if constexpr (G) {  // mlw_m_g.f:289-290, 308, 326, 344
      sgk[kt] = fma(rx, gq[0], fma(ry, gq[1], rz * gq[2]));
      sgk[T::NK + kt] = ro * gq[0];
      sgk[2 * T::NK + kt] = ro * gq[1];
      sgk[3 * T::NK + kt] = ro * gq[2];
    }
#undef KS
  };

  // ---- per-column constants of the full step --------------------------------
  double uy0 = 0, uy1 = 0, ux0 = 0, ux1 = 0, dtx = 0, dty = 0, cx_ = 0, cy_ = 0, mxy = 0;
  float ex0 = 0, ex1 = 0, ey0 = 0, ey1 = 0;
  if (interior) {
    ux0 = ax.u0[ii];
    ux1 = ax.u1[ii];
    uy0 = ay.u0[jj];
    uy1 = ay.u1[jj];
    ex0 = ax.e0[ii];
    ex1 = ax.e1[ii];
    ey0 = ay.e0[jj];
    ey1 = ay.e1[jj];
    dtx = dt * ax.di[ii];
    dty = dt * ay.di[jj];
    cx_ = -0.015625 * dtx;
    cy_ = -0.015625 * dty;
    mxy = fd::maxp(ax.di[ii] * ax.di[ii], ay.di[jj] * ay.di[jj]);
  }
  auto ret = [&](int r) -> double & { return sret[(size_t)r * T::NI + it]; };

  double un[4] = {0.0, 0.0, 0.0, 0.0};  // the new values of the thread's variables
  double kmax = 0.0;                    // largest CFL key of the thread's cells
  bool bad = false;

  // ---- the new primitives of plane k and their CFL key -----------------------
  auto finish = [&](int k) {
    if (tid >= T::NI || !interior) return;
    const double ro = un[CRO], ee = un[CEE], rx = un[CRX], bx = un[CBX];
    const double ry = sun[tid], rz = sun[T::NI + tid], by = sun[2 * T::NI + tid];
    const double bz = sun[3 * T::NI + tid];
    const double ri = fd::rcp(ro);
    const double vx = rx * ri, vy = ry * ri, vz = rz * ri;
    const double ek = fma(rx, vx, fma(ry, vy, rz * vz));
    const double bb = fma(bx, bx, fma(by, by, bz * bz));
    const double pr = ph.gm1 * fma(-ph.pi8i, bb, fma(-0.5, ek, ee));
    const size_t g = (size_t)ii + (size_t)jj * ix + (size_t)k * plane;
    B[P3::RO * n + g] = ro;
    B[P3::PR * n + g] = pr;
    B[P3::VX * n + g] = vx;
    B[P3::VY * n + g] = vy;
    B[P3::VZ * n + g] = vz;
    B[P3::BX * n + g] = bx;
    B[P3::BY * n + g] = by;
    B[P3::BZ * n + g] = bz;
    if (ctl != nullptr && ii >= box.lo[0] && ii <= box.hi[0] && jj >= box.lo[1] &&
        jj <= box.hi[1] && k >= box.lo[2] && k <= box.hi[2]) {
      // the largest (v^2 + cs^2 + ca^2) max(1/dx^2, 1/dy^2, 1/dz^2) gives the
      // smallest time step (cfl_m.f:52-59, pi in single precision)
      const double s = fma(ph.pi4i_cfl, bb, fma(ph.gm, pr, ek)) * ri;
      const double key = s * fd::maxp(mxy, az.di[k] * az.di[k]);
      if (!fd::is_nan(key)) kmax = fd::max_(key, kmax);
      bad |= bad_cell(ro, pr, key);
    }
  };

  // outside the array the corners are never formed
  for (int q = tid; q < NKF * T::NK; q += T::NT) sk[q] = 0.0;
  if constexpr (G)
    for (int q = tid; q < 4 * T::NK; q += T::NT) sgk[q] = 0.0;
  for (int q = tid; q < T::NR * T::NI; q += T::NT) sret[q] = 0.0;
  load_plane(kb - 1);
  load_plane(kb);
  // k = kb - 1 only leaves what the columns keep of the corners kb - 1/2
  for (int k = kb - 1;; k++) {
    // (a) the primitives of plane k-1 (the first warps); cell plane k+1 over plane
    // k-1 (the others)
    if (k > kb) finish(k - 1);
    if (k > ke) break;
    if (k >= kb) load_plane(k + 1);
    __syncthreads();
    // (b) the sums of corner plane k+1/2
    corner_sums(k);
    __syncthreads();
    // (c) their fluxes (the lower half), viscosity faces of plane k (the upper)
    if (tid < T::NKW) {
      corner_fluxes(k);
    } else {
      const double *sl = cslot(k);
      if (ft == 0) {
        szc[0] = -64.0 * ph.qav * az.dm[k] * az.dim[k];
        szc[1] = -0.015625 * dt * az.di[k];
      }
      if (ft < T::NQX) {
        const double *v = sl + (size_t)CVX * T::NC + fxx + (fxr + 1) * T::CX;
        sqx[ft] = qxc * fd::pos_part(fd::abs_(v[1] - v[0]) - CANS_AV_EPS);
      }
      if (ft < T::NQY) {
        const double *v = sl + (size_t)CVY * T::NC + fyx + 1 + fyr * T::CX;
        sqy[ft] = qyc * fd::pos_part(fd::abs_(v[T::CX] - v[0]) - CANS_AV_EPS);
      }
    }
    __syncthreads();
    // (d) full step of plane k
    if (interior) {
      const double *s0 = cslot(k) + c0, *s1 = cslot(k + 1) + c0, *kk = sk + kSW;
      const double ae = dtx * sqx[lx + (ly - 1) * T::KX], aw = dtx * sqx[lx - 1 + (ly - 1) * T::KX];
      const double an = dty * sqy[lx - 1 + ly * TX], as = dty * sqy[lx - 1 + (ly - 1) * TX];
      const double aa = (ae + aw) + (an + as);
      // 64 times the z viscosity of the upper face, negative
      const double qz = szc[0] * fd::pos_part(fd::abs_(s1[(size_t)CVZ * T::NC] -
                                                       s0[(size_t)CVZ * T::NC]) - CANS_AV_EPS);
      // the corner sums carry 8 and weights of 1/2 a plane and axis, the z flux 32
      const double cz_ = szc[1];
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        const int v = iv0 + j;
        const VarFields q = kVar[v];
        const double *u = s0 + (size_t)v * T::NC;
        // the variable's fluxes at cell offset d and at the corners; called only where it
        // has one in the direction
        auto fx = [&](int d) { return s0[q.fx * T::NC + d]; };
        auto fy = [&](int d) { return s0[q.fy * T::NC + d]; };
        auto kx_ = [&](int d) { return kk[q.kx * T::NK + d]; };
        auto ky = [&](int d) { return kk[q.ky * T::NK + d]; };
        auto kz = [&](int d) { return kk[q.kz * T::NK + d]; };
        auto f0 = [&]() { return s0[q.fz * T::NC]; };
        auto f1 = [&]() { return s1[q.fz * T::NC]; };
        const double gxl = q.fx >= 0 ? ret(8 + q.rx) : 0.0, gyl = q.fy >= 0 ? ret(15 + q.ry) : 0.0;
        const double pl = ret(v);
        const double w = qz * (s1[(size_t)v * T::NC] - u[0]);
        double gx = 0.0, gy = 0.0, pu = w;           // what the next plane keeps
        double tx = 0.0, ty = 0.0, tz;               // differences of the directions
        double du = fma(ae, u[1], fma(aw, u[-1], fma(an, u[T::CX],
                                                     fma(as, u[-T::CX], -aa * u[0]))));
        if constexpr (U) {
          bool sp = false;
          const float ez0 = az.e0[k], ez1 = az.e1[k];
          if (q.fx >= 0)
            tx = isum::diff_planes(kx_(0), kx_(1), kx_(T::KX), kx_(T::KX + 1), gxl, fx(-1), fx(1),
                                   ey0, ey1, ez0, ez1, gx, sp);
          if (q.fy >= 0)
            ty = isum::diff_planes(ky(0), ky(T::KX), ky(1), ky(T::KX + 1), gyl, fy(-T::CX),
                                   fy(T::CX), ex0, ex1, ez0, ez1, gy, sp);
          if (q.fz >= 0)
            tz = isum::face_planes(kz(0), kz(1), kz(T::KX), kz(T::KX + 1), f0(), f1(), w, pl,
                                   q.sz < 0, ex0, ex1, ey0, ey1, pu, sp);
          else
            tz = w - pl;
          if (sp) {  // a call, as in corner_plane
            double o[6];
            cell_fp64<T>(q, s0, s1, kk, gxl, gyl, pl, w, ux0, ux1, uy0, uy1, az.u0[k], az.u1[k],
                         o);
            tx = o[0];
            ty = o[1];
            tz = o[2];
            gx = o[3];
            gy = o[4];
            pu = o[5];
          }
        } else {
          const double uz0 = 2.0 * az.u0[k], uz1 = 2.0 * az.u1[k];
          if (q.fx >= 0) {
            gx = fma(2.0 * uy1, kx_(T::KX + 1) - kx_(T::KX), 2.0 * uy0 * (kx_(1) - kx_(0)));
            tx = fma(16.0, fx(1) - fx(-1), fma(uz1, gx, uz0 * gxl));
          }
          if (q.fy >= 0) {
            gy = fma(2.0 * ux1, ky(T::KX + 1) - ky(1), 2.0 * ux0 * (ky(T::KX) - ky(0)));
            ty = fma(16.0, fy(T::CX) - fy(-T::CX), fma(uz1, gy, uz0 * gyl));
          }
          if (q.fz >= 0) {
            const double s = fma(2.0 * uy1, fma(2.0 * ux1, kz(T::KX + 1), 2.0 * ux0 * kz(T::KX)),
                                 2.0 * uy0 * fma(2.0 * ux1, kz(1), 2.0 * ux0 * kz(0)));
            pu = fma(q.sz < 0 ? -1.0 : 1.0, fma(16.0, f0() + f1(), s), w);
          }
          tz = pu - pl;
        }
        if (q.fx >= 0) ret(8 + q.rx) = gx;
        if (q.fy >= 0) ret(15 + q.ry) = gy;
        ret(v) = pu;
        du = fma(signed_by(cx_, q.sx), tx, du);
        du = fma(signed_by(cy_, q.sy), ty, du);
        du = fma(cz_, tz, du);
        if constexpr (G) {  // mlwsrch part 1 and mlwsrcf
          if (q.g >= 0) {
            const double *p = sgk + (size_t)q.g * T::NK + kSW;
            const double g1 = fma(uy1, fma(ux1, p[T::KX + 1], ux0 * p[T::KX]),
                                  uy0 * fma(ux1, p[1], ux0 * p[0]));
            const double g0 = ret(NRET + q.g);
            ret(NRET + q.g) = g1;
            du = fma(0.5 * dt, gslot(k)[(size_t)q.g * T::NC + c0], du);
            du = fma(0.0625 * dt, fma(az.u0[k], g0, az.u1[k] * g1), du);
          }
        }
        const double r = u[0] + du;
        if (iv0) {
          sun[(size_t)j * T::NI + it] = r;
        } else {
#pragma unroll
          for (int m = 0; m < 4; m++) un[m] = m == j ? r : un[m];
        }
      }
    }
    __syncthreads();
  }
  if (ctl != nullptr) {
    count_bad_block(bad, &ctl->nonfinite, tid);
    const double m = block_min(-kmax, sred, tid, T::NT);
    if (tid == 0 && m < 0.0) atomic_min_pos(&ctl->cfl_bits, ctl->safety / sqrt(-m));
  }
}

namespace {

constexpr int kMaxDevices3F = 64;

template <int TX, int TY, bool G, bool R, int MINB, bool U>
cudaError_t launch3f(const double *A, double *B, int ix, int jx, int kx, const Axis &ax,
                     const Axis &ay, const Axis &az, const Phys &ph, double dt, Ctl *ctl,
                     Box3 box, int kmax, cudaStream_t s, const double *grav,
                     const double *res) {
  using T = T3F<TX, TY, G>;
  // per device, once: the shared-memory attribute and the resident blocks
  static std::mutex mu;
  static int slots_of[kMaxDevices3F] = {};
  int dev = 0, slots = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices3F) return cudaErrorInvalidDevice;
  auto kern = k_mlw3d_fast<TX, TY, G, R, MINB, U>;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!slots_of[dev]) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)T::smem_bytes);
      if (e != cudaSuccess) return e;
      int sms = 0, per_sm = 0;
      if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, T::NT,
                                                             T::smem_bytes)) != cudaSuccess)
        return e;
      slots_of[dev] = sms * (per_sm > 0 ? per_sm : 1);
    }
    slots = slots_of[dev];
  }
  const int bx = (ix - 2 + TX - 1) / TX, by = (jx - 2 + TY - 1) / TY;
  const int kchunk = balance_kchunk((long long)bx * by, kx - 2, kmax, slots);
  const dim3 grid(bx, by, (kx - 2 + kchunk - 1) / kchunk);
  kern<<<grid, T::NT, T::smem_bytes, s>>>(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, kchunk,
                                          grav, res);
  count_launch();
  return cudaGetLastError();
}

template <bool G, bool R, bool U>
cudaError_t pick3f(int tile, const double *A, double *B, int ix, int jx, int kx, const Axis &ax,
                   const Axis &ay, const Axis &az, const Phys &ph, double dt, Ctl *ctl, Box3 box,
                   cudaStream_t s, const double *grav, const double *res) {
  if (tile == 2)
    return launch3f<16, 12, G, R, 1, U>(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, 64, s, grav,
                                        res);
  return launch3f<16, 8, G, R, G ? 1 : 2, U>(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box,
                                             tile == 1 ? 32 : 64, s, grav, res);
}
}  // namespace

// The fast policy's step.  Tiles 0 and 1: 16 x 8 columns, z chunks of at most 64
// and 32 planes; 2: 16 x 12 columns.
cudaError_t launch_mlw3d_fast(int tile, const double *A, double *B, int ix, int jx, int kx,
                              const Axis &ax, const Axis &ay, const Axis &az, const Phys &ph,
                              double dt, Ctl *ctl, Box3 box, cudaStream_t s, const double *grav,
                              const double *res) {
  if (ix < 3 || jx < 3 || kx < 3 || (grav && res)) return cudaErrorInvalidValue;
  const bool u = ax.uniform && ay.uniform && az.uniform;
  auto f = grav ? (u ? pick3f<true, false, true> : pick3f<true, false, false>)
           : res ? (u ? pick3f<false, true, true> : pick3f<false, true, false>)
                 : (u ? pick3f<false, false, true> : pick3f<false, false, false>);
  return f(tile, A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, s, grav, res);
}

}  // namespace cans
