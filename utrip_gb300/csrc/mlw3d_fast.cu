// Fused 3-D modified Lax-Wendroff step, fast policy (sm_103a, FP64): mlw_m
// (cans3d/hdmlw/mlw_m.f:2-453), with G mlw_m_g (mlw_m_g.f:2-469) and with R
// mlw_m_e (mlw_m_e.f:103-115, 257-270) given the eta J fields of mlw3d_e.cu,
// and the CFL of cans3d/common/cfl_m.f:39-85.  The exact policy's kernel, one
// operation of the reference after the other, is in mlw3d.cu.
//
// What bounds the step is the FP64 pipe (two lanes per SM and clock; HBM is at
// 2 %), so the kernel is laid out for the fewest FP64 warp instructions:
//  - A block owns a TX x TY column of cells and marches along z.  Per plane:
//    the cells of plane k+1, the corners of plane k+1/2, the full step of plane
//    k.  Each phase numbers its own work items (cells of the halo tile, corners,
//    interior cells) through the threads, so that its warps are full: 16 x 8
//    tiles take 6, 5 and 4 warps of a block of 6.
//  - The predictor's sums over the four cells of a plane (the mean of u, the x
//    and y differences of the fluxes, the sum of the z flux) are kept in
//    registers for the next corner plane, which is the other side of that cell
//    plane: 28 sums a corner, formed once.  Fields needed in two of these forms
//    (the off-diagonal momentum fluxes, E, the momenta) share their partial
//    sums: 97 additions a corner where eight-cell sums take 203.
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
//  - reciprocals of fd64.cuh; comparisons on the integer pipe.
// FP64 warp instructions a zone (32 a warp instruction, 16 x 8 tiles): about
// 550 against 920 of one that forms each cell's sums for itself.  Shared memory
// 110 KB, 168 registers: two blocks a SM, whose barriers overlap.
#include <cuda_runtime.h>

#include <mutex>

#include "cans_common.cuh"
#include "cans_internal.h"
#include "cfl3.cuh"
#include "fd64.cuh"

namespace cans {

namespace {

// cell slots: conserved, fluxes (XY = fx(ry) = fy(rx), ...), E, velocities
enum {
  CRO, CEE, CRX, CRY, CRZ, CBX, CBY, CBZ,
  CFX, CFY, CFZ,                  // energy fluxes
  CXX, CYY, CZZ, CXY, CXZ, CYZ,   // momentum fluxes
  CEX, CEY, CEZ, CVX, CVY, CVZ, NCF
};
// corner slots, all eight times their value; the mass fluxes are the momenta
enum { KRX, KRY, KRZ, KFX, KFY, KFZ, KXX, KYY, KZZ, KXY, KXZ, KYZ, KEX, KEY, KEZ, NKF };
// what a corner keeps of its lower cell plane: S the sum over the four cells, X
// and Y the differences along x and y
enum {
  S_RO, S_EE, S_RX, X_RX, S_RY, Y_RY, S_RZ, S_BX, S_BY, S_BZ, X_FX, Y_FY, S_FZ, X_XX, Y_YY,
  S_ZZ, X_XY, Y_XY, X_XZ, S_XZ, Y_YZ, S_YZ, Y_EX, S_EX, X_EY, S_EY, X_EZ, Y_EZ, NPS
};
// what an interior column keeps of its lower corner plane: the x and y
// differences of seven variables (ro, ee, rx, ry, rz, two of B) and the z face
// fluxes of eight
constexpr int NRET = 22;

template <int TX, int TY, bool G> struct T3F {
  static constexpr int CX = TX + 2, CY = TY + 2, NC = CX * CY;
  static constexpr int KX = TX + 1, KY = TY + 1, NK = KX * KY;
  static constexpr int NI = TX * TY, NQX = KX * TY, NQY = TX * KY;
  static constexpr int NT = (NC + 31) / 32 * 32;
  static constexpr int NR = NRET + (G ? 4 : 0);
  static constexpr size_t smem_bytes =
      sizeof(double) * (2 * (size_t)NCF * NC + (size_t)NKF * NK + NQX + NQY + (size_t)NR * NI +
                        32 + (G ? 2 * 4 * (size_t)NC + 4 * (size_t)NK : 0));
};

}  // namespace

template <int TX, int TY, bool G, bool R, int MINB>
__global__ void __launch_bounds__(((TX + 2) * (TY + 2) + 31) / 32 * 32, MINB)
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
  double *sred = sret + (size_t)T::NR * T::NI;
  double *sgc = sred + 32;                            // G: [2][4][NC]
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

  // the thread's cell of the halo tile
  const int hx = tid % T::CX, hy = tid / T::CX;
  const int gi = i0 - 1 + hx, gj = j0 - 1 + hy;
  const bool cell = tid < T::NC, in_arr = cell && gi < ix && gj < jx;
  // its corner, and the corner's predictor coefficients 8 dt / (4 dxm)
  const int cx = tid % T::KX, cy = tid / T::KX;
  const bool corner = tid < T::NK;
  const bool cor_in = corner && i0 - 1 + cx <= ix - 2 && j0 - 1 + cy <= jx - 2;
  const int p00 = cx + cy * T::CX;
  const double cxk = cor_in ? 2.0 * dt * ax.dim[i0 - 1 + cx] : 0.0;
  const double cyk = cor_in ? 2.0 * dt * ay.dim[j0 - 1 + cy] : 0.0;
  // its interior cell
  const int lx = tid % TX + 1, ly = tid / TX + 1;
  const int ii = i0 - 1 + lx, jj = j0 - 1 + ly;
  const bool interior = tid < T::NI && ii <= ix - 2 && jj <= jx - 2;
  const int c0 = lx + ly * T::CX;
  const int kSW = (lx - 1) + (ly - 1) * T::KX;
  // its viscosity faces: qav dm dim of an x and a y face
  const int fxx = tid % T::KX, fxr = tid / T::KX, fyx = tid % TX, fyr = tid / TX;
  const bool facex = tid < T::NQX && i0 + fxx < ix && j0 + fxr < jx;
  const bool facey = tid < T::NQY && i0 + fyx < ix && j0 + fyr < jx;
  const double qxc = facex ? ph.qav * ax.dm[i0 - 1 + fxx] * ax.dim[i0 - 1 + fxx] : 0.0;
  const double qyc = facey ? ph.qav * ay.dm[j0 - 1 + fyr] * ay.dim[j0 - 1 + fyr] : 0.0;

  auto cslot = [&](int k) { return scell + (size_t)(k & 1) * NCF * T::NC; };
  auto gslot = [&](int k) { return sgc + (size_t)(k & 1) * 4 * T::NC; };

  // ---- cells of plane k (mlw_m.f:74-202) -----------------------------------
  auto load_plane = [&](int k) {
    if (!cell) return;
    double *sl = cslot(k) + tid;
#define S(f) sl[(size_t)(f) * T::NC]
    if (!in_arr) {
#pragma unroll 1
      for (int f = 0; f < NCF; f++) S(f) = 0.0;
      if constexpr (G)
        for (int f = 0; f < 4; f++) gslot(k)[f * T::NC + tid] = 0.0;
      return;
    }
    const size_t g = (size_t)gi + (size_t)gj * ix + (size_t)k * plane;
    const double ro = A[P3::RO * n + g], pr = A[P3::PR * n + g];
    const double vx = A[P3::VX * n + g], vy = A[P3::VY * n + g], vz = A[P3::VZ * n + g];
    const double bx = A[P3::BX * n + g], by = A[P3::BY * n + g], bz = A[P3::BZ * n + g];
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
      double *gs = gslot(k) + tid;
      gs[0] = fma(rx, gx, fma(ry, gy, rz * gz));
      gs[T::NC] = ro * gx;
      gs[2 * T::NC] = ro * gy;
      gs[3 * T::NC] = ro * gz;
    }
#undef S
  };

  // ---- the plane sums of a corner ------------------------------------------
  double P[NPS] = {}, PG[G ? 4 : 1] = {};
  // q(s, x): the new value of sum s; the caller combines it with P[s] and stores
  auto plane_sums = [&](int k, auto &&put) {
    const double *sl = cslot(k) + p00;
#define F4(f) \
  const double *q = sl + (size_t)(f) * T::NC; \
  const double a = q[0], b = q[1], c = q[T::CX], d = q[T::CX + 1]
    auto sum = [&](int f, int s) { F4(f); put(s, (a + b) + (c + d)); };
    auto dx = [&](int f, int s) { F4(f); put(s, (b - a) + (d - c)); };
    auto dy = [&](int f, int s) { F4(f); put(s, (c - a) + (d - b)); };
    auto sum_dx = [&](int f, int s, int x) {
      F4(f);
      const double l = a + c, r = b + d;
      put(s, l + r);
      put(x, r - l);
    };
    auto sum_dy = [&](int f, int s, int y) {
      F4(f);
      const double l = a + b, r = c + d;
      put(s, l + r);
      put(y, r - l);
    };
    auto dx_dy = [&](int f, int x, int y) {
      F4(f);
      const double u = d - a, w = b - c;
      put(x, u + w);
      put(y, u - w);
    };
    sum(CRO, S_RO);
    sum_dx(CRX, S_RX, X_RX);
    sum_dy(CRY, S_RY, Y_RY);
    sum(CRZ, S_RZ);
    sum(CEE, S_EE);
    dx(CFX, X_FX);
    dy(CFY, Y_FY);
    sum(CFZ, S_FZ);
    dx(CXX, X_XX);
    dx_dy(CXY, X_XY, Y_XY);
    sum_dx(CXZ, S_XZ, X_XZ);
    dy(CYY, Y_YY);
    sum_dy(CYZ, S_YZ, Y_YZ);
    sum(CZZ, S_ZZ);
    sum(CBX, S_BX);
    sum(CBY, S_BY);
    sum(CBZ, S_BZ);
    sum_dy(CEX, S_EX, Y_EX);
    sum_dx(CEY, S_EY, X_EY);
    dx_dy(CEZ, X_EZ, Y_EZ);
#undef F4
  };
  auto grav_sum = [&](int k, int f) {
    const double *q = gslot(k) + f * T::NC + p00;
    return (q[0] + q[1]) + (q[T::CX] + q[T::CX + 1]);
  };

  // ---- corners of plane k + 1/2 (mlwhalf.f:49-65, mlw_m.f:205-334) -----------
  auto corner_plane = [&](int k) {
    if (!corner) return;
    double *ks = sk + tid;
#define KS(f) ks[(size_t)(f) * T::NK]
    if (!cor_in) {
#pragma unroll 1
      for (int f = 0; f < NKF; f++) KS(f) = 0.0;
      if constexpr (G)
        for (int f = 0; f < 4; f++) sgk[f * T::NK + tid] = 0.0;
      return;
    }
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
    const double czk = 2.0 * dt * az.dim[k];
    // D[s]: sums and x, y differences over both planes, z differences (upper
    // less lower) of the sums that are z fluxes; S_RZ, S_XZ, ... serve both
    double D[NPS], Zrz, Zxz, Zyz;
    plane_sums(k + 1, [&](int s, double x) {
      const bool z = s == S_FZ || s == S_ZZ || s == S_EX || s == S_EY;
      if (s == S_RZ) Zrz = x - P[s];
      if (s == S_XZ) Zxz = x - P[s];
      if (s == S_YZ) Zyz = x - P[s];
      D[s] = z ? x - P[s] : x + P[s];
      P[s] = x;
    });
    const double ro = fma(-czk, Zrz, fma(-cyk, D[Y_RY], fma(-cxk, D[X_RX], D[S_RO])));
    double ee = fma(-czk, D[S_FZ], fma(-cyk, D[Y_FY], fma(-cxk, D[X_FX], D[S_EE])));
    double rx = fma(-czk, Zxz, fma(-cyk, D[Y_XY], fma(-cxk, D[X_XX], D[S_RX])));
    double ry = fma(-czk, Zyz, fma(-cyk, D[Y_YY], fma(-cxk, D[X_XY], D[S_RY])));
    double rz = fma(-czk, D[S_ZZ], fma(-cyk, D[Y_YZ], fma(-cxk, D[X_XZ], D[S_RZ])));
    // B: d(bx) = -(dy Ez - dz Ey), d(by) = -(dz Ex - dx Ez), d(bz) = -(dx Ey - dy Ex)
    const double bx = fma(czk, D[S_EY], fma(-cyk, D[Y_EZ], D[S_BX]));
    const double by = fma(-czk, D[S_EX], fma(cxk, D[X_EZ], D[S_BY]));
    const double bz = fma(cyk, D[Y_EX], fma(-cxk, D[X_EY], D[S_BZ]));
    if constexpr (G) {  // mlwsrch part 2: dt times the mean of the eight sources
      double x[4];
#pragma unroll
      for (int f = 0; f < 4; f++) {
        x[f] = grav_sum(k + 1, f);
        PG[f] += x[f];
      }
      ee = fma(dt, PG[0], ee);
      rx = fma(dt, PG[1], rx);
      ry = fma(dt, PG[2], ry);
      rz = fma(dt, PG[3], rz);
#pragma unroll
      for (int f = 0; f < 4; f++) PG[f] = x[f];
    }
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
      sgk[tid] = fma(rx, gq[0], fma(ry, gq[1], rz * gq[2]));
      sgk[T::NK + tid] = ro * gq[0];
      sgk[2 * T::NK + tid] = ro * gq[1];
      sgk[3 * T::NK + tid] = ro * gq[2];
    }
#undef KS
  };

  // ---- per-column constants of the full step --------------------------------
  double uy0 = 0, uy1 = 0, ux0 = 0, ux1 = 0, dtx = 0, dty = 0, w00 = 0, w10 = 0, w01 = 0,
         w11 = 0, mxy = 0;
  if (interior) {
    ux0 = ax.u0[ii];
    ux1 = ax.u1[ii];
    uy0 = ay.u0[jj];
    uy1 = ay.u1[jj];
    dtx = dt * ax.di[ii];
    dty = dt * ay.di[jj];
    // corner weights of a z face over 4: twice the mean of eightfold values
    w00 = 0.25 * (ux0 * uy0);
    w10 = 0.25 * (ux1 * uy0);
    w01 = 0.25 * (ux0 * uy1);
    w11 = 0.25 * (ux1 * uy1);
    mxy = fd::maxp(ax.di[ii] * ax.di[ii], ay.di[jj] * ay.di[jj]);
  }
  auto ret = [&](int r) -> double & { return sret[(size_t)r * T::NI + tid]; };
  // corner differences along x (uy0 (SE - SW) + uy1 (NE - NW)) and y, and the
  // corner average of the z face
  auto kdx = [&](int f) {
    const double *q = sk + (size_t)f * T::NK + kSW;
    return fma(uy1, q[T::KX + 1] - q[T::KX], uy0 * (q[1] - q[0]));
  };
  auto kdy = [&](int f) {
    const double *q = sk + (size_t)f * T::NK + kSW;
    return fma(ux1, q[T::KX + 1] - q[1], ux0 * (q[T::KX] - q[0]));
  };
  auto kz = [&](int f, double s) {  // s + the average
    const double *q = sk + (size_t)f * T::NK + kSW;
    return fma(w11, q[T::KX + 1], fma(w01, q[T::KX], fma(w10, q[1], fma(w00, q[0], s))));
  };
  auto gkz = [&](int f) {
    const double *q = sgk + (size_t)f * T::NK + kSW;
    return fma(w11, q[T::KX + 1], fma(w01, q[T::KX], fma(w10, q[1], w00 * q[0])));
  };
  // twice the z flux of variable v through the face between planes k and k+1:
  // F_k + F_k+1 + 2 (corner average) - 4 qz (u_k+1 - u_k)
  auto z_face = [&](const double *s0, const double *s1, int v, int sf, int kf, bool neg,
                    double qz4) {
    const size_t o = (size_t)v * T::NC + c0;
    const double du = s1[o] - s0[o];
    if (sf < 0) return -qz4 * du;
    const size_t of = (size_t)sf * T::NC + c0;
    const double s = kz(kf, s0[of] + s1[of]);
    return fma(-qz4, du, neg ? -s : s);
  };
  auto z_visc = [&](const double *s0, const double *s1, int k) {
    const double q =
        fd::abs_(s1[(size_t)CVZ * T::NC + c0] - s0[(size_t)CVZ * T::NC + c0]) - CANS_AV_EPS;
    return 4.0 * (ph.qav * az.dm[k] * az.dim[k]) * fd::pos_part(q);
  };

  // ---- prologue: the sums of plane kb-1, corners kb-1/2, what they leave ----
  load_plane(kb - 1);
  load_plane(kb);
  __syncthreads();
  if (cor_in) {
    plane_sums(kb - 1, [&](int s, double x) { P[s] = x; });
    if constexpr (G) {
#pragma unroll
      for (int f = 0; f < 4; f++) PG[f] = grav_sum(kb - 1, f);
    }
  }
  corner_plane(kb - 1);
  __syncthreads();
  // fields of the seven x differences, y differences and the z faces, in the
  // order of ret()
  auto each_x = [&](auto &&f) {
    f(0, CRO, CRX, KRX, false); f(1, CEE, CFX, KFX, false); f(2, CRX, CXX, KXX, false);
    f(3, CRY, CXY, KXY, false); f(4, CRZ, CXZ, KXZ, false); f(5, CBY, CEZ, KEZ, true);
    f(6, CBZ, CEY, KEY, false);
  };
  if (interior) {
    const double *s0 = cslot(kb - 1), *s1 = cslot(kb);
    const double qz4 = z_visc(s0, s1, kb - 1);
    each_x([&](int r, int, int, int kf, bool) { ret(r) = kdx(kf); });
    ret(7) = kdy(KRY); ret(8) = kdy(KFY); ret(9) = kdy(KXY); ret(10) = kdy(KYY);
    ret(11) = kdy(KYZ); ret(12) = kdy(KEZ); ret(13) = kdy(KEX);
    ret(14) = z_face(s0, s1, CRO, CRZ, KRZ, false, qz4);
    ret(15) = z_face(s0, s1, CEE, CFZ, KFZ, false, qz4);
    ret(16) = z_face(s0, s1, CRX, CXZ, KXZ, false, qz4);
    ret(17) = z_face(s0, s1, CRY, CYZ, KYZ, false, qz4);
    ret(18) = z_face(s0, s1, CRZ, CZZ, KZZ, false, qz4);
    ret(19) = z_face(s0, s1, CBX, CEY, KEY, true, qz4);
    ret(20) = z_face(s0, s1, CBY, CEX, KEX, false, qz4);
    ret(21) = z_face(s0, s1, CBZ, -1, 0, false, qz4);
    if constexpr (G) {
#pragma unroll
      for (int f = 0; f < 4; f++) ret(NRET + f) = gkz(f);
    }
  }
  __syncthreads();

  double kmax = 0.0;  // largest CFL key of the thread's cells
  bool bad = false;

  for (int k = kb; k <= ke; k++) {
    // (a) cell plane k+1 over plane k-1
    load_plane(k + 1);
    __syncthreads();
    // (b) corner plane k+1/2, viscosity faces of plane k
    corner_plane(k);
    {
      const double *sl = cslot(k);
      if (tid < T::NQX) {
        const double *v = sl + (size_t)CVX * T::NC + fxx + (fxr + 1) * T::CX;
        sqx[tid] = qxc * fd::pos_part(fd::abs_(v[1] - v[0]) - CANS_AV_EPS);
      }
      if (tid < T::NQY) {
        const double *v = sl + (size_t)CVY * T::NC + fyx + 1 + fyr * T::CX;
        sqy[tid] = qyc * fd::pos_part(fd::abs_(v[T::CX] - v[0]) - CANS_AV_EPS);
      }
    }
    __syncthreads();
    // (c) full step of plane k
    if (interior) {
      const double *s0 = cslot(k), *s1 = cslot(k + 1);
      const double ae = dtx * sqx[lx + (ly - 1) * T::KX], aw = dtx * sqx[lx - 1 + (ly - 1) * T::KX];
      const double an = dty * sqy[lx - 1 + ly * TX], as = dty * sqy[lx - 1 + (ly - 1) * TX];
      const double aa = (ae + aw) + (an + as);
      const double fcx = 0.25 * dtx, fcy = 0.25 * dty;
      const double uz0 = az.u0[k], uz1 = az.u1[k], dtz = dt * az.di[k];
      // the corner differences carry 8: hdt / 8 = dt / 16
      const double hx0 = 0.0625 * dtx * uz0, hx1 = 0.0625 * dtx * uz1;
      const double hy0 = 0.0625 * dty * uz0, hy1 = 0.0625 * dty * uz1;
      const double hz = 0.25 * dtz;
      const double qz4 = z_visc(s0, s1, k);
      auto visc = [&](int v) {
        const double *q = s0 + (size_t)v * T::NC + c0;
        return fma(ae, q[1], fma(aw, q[-1], fma(an, q[T::CX], fma(as, q[-T::CX], -aa * q[0]))));
      };
      auto add_x = [&](double du, int r, int sf, int kf, bool neg) {
        const double *q = s0 + (size_t)sf * T::NC + c0;
        const double g1 = kdx(kf), g0 = ret(r);
        ret(r) = g1;
        const double s = neg ? 1.0 : -1.0;
        return fma(s * hx1, g1, fma(s * hx0, g0, fma(s * fcx, q[1] - q[-1], du)));
      };
      auto add_y = [&](double du, int r, int sf, int kf, bool neg) {
        const double *q = s0 + (size_t)sf * T::NC + c0;
        const double g1 = kdy(kf), g0 = ret(r);
        ret(r) = g1;
        const double s = neg ? 1.0 : -1.0;
        return fma(s * hy1, g1, fma(s * hy0, g0, fma(s * fcy, q[T::CX] - q[-T::CX], du)));
      };
      auto add_z = [&](double du, int r, int v, int sf, int kf, bool neg) {
        const double f1 = z_face(s0, s1, v, sf, kf, neg, qz4), f0 = ret(r);
        ret(r) = f1;
        return fma(-hz, f1 - f0, du);
      };
      auto source = [&](double du, int f) {  // mlwsrch part 1 and mlwsrcf
        if constexpr (G) {
          const double g1 = gkz(f), g0 = ret(NRET + f);
          ret(NRET + f) = g1;
          du = fma(0.5 * dt, gslot(k)[(size_t)f * T::NC + c0], du);
          du = fma(0.25 * dt * uz0, g0, du);
          du = fma(0.25 * dt * uz1, g1, du);
        }
        return du;
      };
      auto old = [&](int v) { return s0[(size_t)v * T::NC + c0]; };
      const double ro = old(CRO) + add_z(add_y(add_x(visc(CRO), 0, CRX, KRX, false), 7, CRY, KRY,
                                               false), 14, CRO, CRZ, KRZ, false);
      const double rx = old(CRX) + source(add_z(add_y(add_x(visc(CRX), 2, CXX, KXX, false), 9, CXY,
                                                      KXY, false), 16, CRX, CXZ, KXZ, false), 1);
      const double ry = old(CRY) + source(add_z(add_y(add_x(visc(CRY), 3, CXY, KXY, false), 10, CYY,
                                                      KYY, false), 17, CRY, CYZ, KYZ, false), 2);
      const double rz = old(CRZ) + source(add_z(add_y(add_x(visc(CRZ), 4, CXZ, KXZ, false), 11, CYZ,
                                                      KYZ, false), 18, CRZ, CZZ, KZZ, false), 3);
      const double bx = old(CBX) + add_z(add_y(visc(CBX), 12, CEZ, KEZ, false), 19, CBX, CEY, KEY,
                                         true);
      const double by = old(CBY) + add_z(add_x(visc(CBY), 5, CEZ, KEZ, true), 20, CBY, CEX, KEX,
                                         false);
      const double bz = old(CBZ) + add_z(add_y(add_x(visc(CBZ), 6, CEY, KEY, false), 13, CEX, KEX,
                                               true), 21, CBZ, -1, 0, false);
      const double ee = old(CEE) + source(add_z(add_y(add_x(visc(CEE), 1, CFX, KFX, false), 8, CFY,
                                                      KFY, false), 15, CEE, CFZ, KFZ, false), 0);
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
    }
    // ghost cells keep their input values (mlw_m.f updates only 2..n-1); each
    // is copied by the block owning its nearest interior cell, plane by plane,
    // plus the z ghost planes at the chunk ends
    if (in_arr) {
      const int ci = min(max(gi, 1), ix - 2), cj = min(max(gj, 1), jx - 2);
      if (ci >= i0 && ci < i0 + TX && cj >= j0 && cj < j0 + TY) {
        const bool xy_ghost = (gi == 0 || gi == ix - 1 || gj == 0 || gj == jx - 1);
        auto copy = [&](int kk) {
          const size_t g = (size_t)gi + (size_t)gj * ix + (size_t)kk * plane;
#pragma unroll
          for (int v = 0; v < P3::N; v++) B[v * n + g] = A[v * n + g];
        };
        if (xy_ghost) copy(k);
        if (k == 1) copy(0);
        if (k == kx - 2) copy(kx - 1);
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

template <int TX, int TY, bool G, bool R, int MINB>
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
  auto kern = k_mlw3d_fast<TX, TY, G, R, MINB>;
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

template <bool G, bool R>
cudaError_t pick3f(int tile, const double *A, double *B, int ix, int jx, int kx, const Axis &ax,
                   const Axis &ay, const Axis &az, const Phys &ph, double dt, Ctl *ctl, Box3 box,
                   cudaStream_t s, const double *grav, const double *res) {
  if (tile == 2)
    return launch3f<16, 12, G, R, 1>(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, 64, s, grav,
                                     res);
  return launch3f<16, 8, G, R, G ? 1 : 2>(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box,
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
  if (grav)
    return pick3f<true, false>(tile, A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, s, grav, res);
  if (res)
    return pick3f<false, true>(tile, A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, s, grav, res);
  return pick3f<false, false>(tile, A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, s, grav, res);
}

}  // namespace cans
