// Fused 3-D mLW step, mlw_m (cans3d/hdmlw/mlw_m.f:2-453), in the double-float
// policy (df64.cuh): the arithmetic runs as pairs of floats on the FP32
// pipes and the density and field are accumulated in FP64, as in the 2-D
// double-float step.
//
// The block is the fast policy's (mlw3d_fast.cu; fields and layout in
// mlw3d_march.cuh): a column of cells marching along z, work items numbered phase by
// phase so that warps are full, two threads a corner and a cell with four variables
// each, corner values at eight times their size, one corner plane in shared memory
// and 22 retained values a column.  What bounds the step is the issue of FP32
// instructions and their latency (a double-float sum is 11 in a chain of 8), so sums
// of several values are formed at once: exact two-sums of the heads in a tree, the
// tails and the errors added up beside them, one normalisation (59 instructions for
// eight values, 77 for seven sums); and on equally spaced axes the corner weights,
// one half up to 2^-36, are a float correction to plain sums.  128^3: 12500 warp
// instructions a zone (32 a warp) at 72 % of the issue slots and 0.97 ms, where one
// thread a cell with its own sums took 15400 at 44 % and 1.94 ms.
#include <cuda_runtime.h>

#include <mutex>

#include "cans_common.cuh"
#include "cans_internal.h"
#include "cfl3.cuh"
#include "df64.cuh"
#include "mlw3d_march.cuh"

namespace cans {

namespace {

using df::D;

struct PhysD3 {
  D gm, gm1, gm1i, ggm1, pi4i, pi8i, qav, pi4i_cfl;
};

// the fluxes of one state (cell or corner): E = -v x B, the energy flux
// ep v + (B x E)/4pi and the momentum flux rho v v + p_T - B B/4pi
struct Flux3 {
  D ex, ey, ez, fxe, fye, fze, fxx, fyy, fzz, fxy, fxz, fyz;
};
__device__ __forceinline__ Flux3 fluxes3(D rx, D ry, D rz, D vx, D vy, D vz, D bx, D by, D bz,
                                         D ep, D pt, D pi4i) {
  Flux3 o;
  const D pbx = df::mul(pi4i, bx), pby = df::mul(pi4i, by), pbz = df::mul(pi4i, bz);
  o.ex = df::mad(vz, by, df::neg(df::mul(vy, bz)));
  o.ey = df::mad(vx, bz, df::neg(df::mul(vz, bx)));
  o.ez = df::mad(vy, bx, df::neg(df::mul(vx, by)));
  o.fxe = df::mad(ep, vx, df::mad(pbz, o.ey, df::neg(df::mul(pby, o.ez))));
  o.fye = df::mad(ep, vy, df::mad(pbx, o.ez, df::neg(df::mul(pbz, o.ex))));
  o.fze = df::mad(ep, vz, df::mad(pby, o.ex, df::neg(df::mul(pbx, o.ey))));
  o.fxx = df::mad(rx, vx, df::mad(df::neg(pbx), bx, pt));
  o.fyy = df::mad(ry, vy, df::mad(df::neg(pby), by, pt));
  o.fzz = df::mad(rz, vz, df::mad(df::neg(pbz), bz, pt));
  o.fxy = df::mad(rx, vy, df::neg(df::mul(pbx, by)));
  o.fxz = df::mad(rx, vz, df::neg(df::mul(pbx, bz)));
  o.fyz = df::mad(ry, vz, df::neg(df::mul(pby, bz)));
  return o;
}

// sums and differences of the eight cells of a corner (l, u: lower left cells of its
// planes), as isum::eight
enum Form { kSum, kDx, kDy, kDz };
template <int CX, int F> __device__ __forceinline__ D eight(const D *l, const D *u) {
  auto plane = [](const D *p, bool neg) {
    D v[4] = {p[0], p[1], p[CX], p[CX + 1]};
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (F == kDx ? !(i & 1) : F == kDy ? !(i & 2) : neg) v[i] = df::neg(v[i]);
    return df::raw4(v[0], v[1], v[2], v[3]);
  };
  return df::norm2(plane(l, F == kDz), plane(u, false));
}

// weights of a corner difference or average on one axis: 2 u0, 2 u1, which are
// 1 + e0, 1 + e1 on equally spaced axes (U)
template <bool U> struct Weights;
template <> struct Weights<true> {
  float e0, e1;
  __device__ __forceinline__ void set(const Axis &a, int i) {
    e0 = __fmul_rn(a.e0[i], 0x1p-32f);
    e1 = __fmul_rn(a.e1[i], 0x1p-32f);
  }
  // w0 (b - a) + w1 (d - c)
  __device__ __forceinline__ D diff(D a, D b, D c, D d) const {
    const D p = df::two_sum(b.h, -a.h), q = df::two_sum(d.h, -c.h), s = df::two_sum(p.h, q.h);
    const float k = __fmaf_rn(p.h, e0, __fmul_rn(q.h, e1));
    return df::fast_two_sum(
        s.h, __fadd_rn(__fadd_rn(__fsub_rn(b.l, a.l), __fsub_rn(d.l, c.l)),
                       __fadd_rn(df::fadd3(p.l, q.l, s.l), k)));
  }
  // w0 l + w1 u + 16 (g - f)
  __device__ __forceinline__ D planes(D l, D u, D f, D g) const {
    const D x = df::two_sum(l.h, u.h);
    const D y = df::two_sum(__fmul_rn(16.0f, g.h), __fmul_rn(-16.0f, f.h));
    const D s = df::two_sum(x.h, y.h);
    const float k = __fmaf_rn(l.h, e0, __fmul_rn(u.h, e1));
    const float t = __fmaf_rn(16.0f, __fsub_rn(g.l, f.l), __fadd_rn(l.l, u.l));
    return df::fast_two_sum(s.h, __fadd_rn(t, __fadd_rn(df::fadd3(x.l, y.l, s.l), k)));
  }
};
template <> struct Weights<false> {
  D w0, w1;
  __device__ __forceinline__ void set(const Axis &a, int i) {
    w0 = df::scale(df::from_double(a.u0[i]), 2.0f);
    w1 = df::scale(df::from_double(a.u1[i]), 2.0f);
  }
  __device__ __forceinline__ D diff(D a, D b, D c, D d) const {
    return df::mad(w1, df::sub(d, c), df::mul(w0, df::sub(b, a)));
  }
  __device__ __forceinline__ D planes(D l, D u, D f, D g) const {
    return df::add(df::mad(w1, u, df::mul(w0, l)), df::scale(df::sub(g, f), 16.0f));
  }
};
// the corner average of a z face, 32 times its value, + 16 (f + g)
__device__ __forceinline__ D face(const Weights<true> &x, const Weights<true> &y, D a, D b, D c,
                                  D d, D f, D g) {
  const D p = df::raw4(a, b, c, d);
  const float k = __fadd_rn(__fmaf_rn(__fadd_rn(a.h, b.h), y.e0, __fmul_rn(__fadd_rn(c.h, d.h), y.e1)),
                            __fmaf_rn(__fadd_rn(a.h, c.h), x.e0, __fmul_rn(__fadd_rn(b.h, d.h), x.e1)));
  const D q = df::two_sum(__fmul_rn(16.0f, f.h), __fmul_rn(16.0f, g.h));
  return df::norm2({p.h, __fadd_rn(p.l, k)}, {q.h, __fmaf_rn(16.0f, __fadd_rn(f.l, g.l), q.l)});
}
__device__ __forceinline__ D face(const Weights<false> &x, const Weights<false> &y, D a, D b, D c,
                                  D d, D f, D g) {
  const D lo = df::mad(x.w1, b, df::mul(x.w0, a)), up = df::mad(x.w1, d, df::mul(x.w0, c));
  return df::mad(y.w1, up, df::mad(y.w0, lo, df::scale(df::add(f, g), 16.0f)));
}

__device__ __forceinline__ D signed_by(D x, int s) {
  const unsigned m = (unsigned)s & 0x80000000u;
  return {__uint_as_float(__float_as_uint(x.h) ^ m), __uint_as_float(__float_as_uint(x.l) ^ m)};
}
// max(0, |b - a| - 1.0e-4), the threshold a single-precision literal
__device__ __forceinline__ D jump(D a, D b) {
  const D q = df::addf(df::absd(df::sub(b, a)), -1.0e-4f);
  return df::pos(q) ? q : df::mk(0.0f);
}

template <int TX, int TY, int MINB, bool U>
__global__ void __launch_bounds__(T3F<TX, TY, false>::NT, MINB)
    k_mlw3d_df(const double *__restrict__ A, double *__restrict__ B, int ix, int jx, int kx,
               Axis ax, Axis ay, Axis az, Phys ph, double dt_arg, Ctl *__restrict__ ctl,
               Box3 box, int kchunk) {
  using T = T3F<TX, TY, false>;
  extern __shared__ D smem3[];
  D *scell = smem3;                              // [2][NCF][NC]
  D *sk = scell + 2 * (size_t)NCF * T::NC;       // [NKF][NK]
  D *sqx = sk + (size_t)NKF * T::NK;             // q / dxm of plane k
  D *sqy = sqx + T::NQX;
  D *sret = sqy + T::NQY;                        // [NR][NI]
  D *sun = sret + (size_t)T::NR * T::NI;         // [4][NI]: new values 4 .. 7
  double *sred = (double *)(sun + 4 * (size_t)T::NI);
  D *szc = (D *)(sred + 32);                     // of plane k: viscosity, flux factor

  if (ctl != nullptr) {
    if (ctl->done | ctl->pause) return;
    A = ctl->buf[ctl->cur];
    B = ctl->buf[ctl->cur ^ 1];
  }
  const double dtv = (ctl != nullptr) ? ctl->dt : dt_arg;
  const size_t plane = (size_t)ix * jx, n = plane * kx;
  const int tid = threadIdx.x;
  const int i0 = 1 + blockIdx.x * TX, j0 = 1 + blockIdx.y * TY;
  const int kb = 1 + blockIdx.z * kchunk, ke = min(kx - 2, kb + kchunk - 1);
  if (kb > ke) return;
  const PhysD3 P = {df::from_double(ph.gm),   df::from_double(ph.gm1),
                    df::from_double(ph.gm1i), df::from_double(ph.ggm1),
                    df::from_double(ph.pi4i), df::from_double(ph.pi8i),
                    df::from_double(ph.qav),  df::from_double(ph.pi4i_cfl)};
  const D dt = df::from_double(dtv);

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
  const D cxk = cor_in ? df::scale(df::mul(dt, df::from_double(ax.dim[i0 - 1 + cx])), -2.0f)
                       : df::mk(0.0f);
  const D cyk = cor_in ? df::scale(df::mul(dt, df::from_double(ay.dim[j0 - 1 + cy])), -2.0f)
                       : df::mk(0.0f);
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
  const D qxc = facex ? df::mul(df::mul(P.qav, df::from_double(ax.dm[i0 - 1 + fxx])),
                                df::from_double(ax.dim[i0 - 1 + fxx]))
                      : df::mk(0.0f);
  const D qyc = facey ? df::mul(df::mul(P.qav, df::from_double(ay.dm[j0 - 1 + fyr])),
                                df::from_double(ay.dim[j0 - 1 + fyr]))
                      : df::mk(0.0f);

  auto cslot = [&](int k) { return scell + (size_t)(k & 1) * NCF * T::NC; };

  // ---- cells of plane k (mlw_m.f:74-202) -----------------------------------
  auto load_plane = [&](int k) {
    if (!cell) return;
    D *sl = cslot(k) + ct;
#define S(f) sl[(size_t)(f) * T::NC]
    if (!in_arr) {
#pragma unroll 1
      for (int f = 0; f < NCF; f++) S(f) = df::mk(0.0f);
      return;
    }
    const size_t g = (size_t)gi + (size_t)gj * ix + (size_t)k * plane;
    double q[P3::N];
#pragma unroll
    for (int v = 0; v < P3::N; v++) q[v] = A[v * n + g];
    if (xy_ghost ? k == 0 || k >= kb && k <= ke || k == kx - 1
                 : owned && (k == 0 || k == kx - 1)) {
#pragma unroll
      for (int v = 0; v < P3::N; v++) B[v * n + g] = q[v];
    }
    const D ro = df::from_double(q[P3::RO]), pr = df::from_double(q[P3::PR]);
    const D vx = df::from_double(q[P3::VX]), vy = df::from_double(q[P3::VY]);
    const D vz = df::from_double(q[P3::VZ]);
    const D bx = df::from_double(q[P3::BX]), by = df::from_double(q[P3::BY]);
    const D bz = df::from_double(q[P3::BZ]);
    const D vv = df::mad(vz, vz, df::mad(vy, vy, df::sqr(vx)));
    const D bb = df::mad(bz, bz, df::mad(by, by, df::sqr(bx)));
    const D ek = df::mul(df::scale(ro, 0.5f), vv);
    const D rx = df::mul(ro, vx), ry = df::mul(ro, vy), rz = df::mul(ro, vz);
    const Flux3 fl = fluxes3(rx, ry, rz, vx, vy, vz, bx, by, bz, df::mad(pr, P.ggm1, ek),
                             df::mad(P.pi8i, bb, pr), P.pi4i);
    S(CRO) = ro; S(CEE) = df::mad(pr, P.gm1i, df::mad(P.pi8i, bb, ek));
    S(CRX) = rx; S(CRY) = ry; S(CRZ) = rz;
    S(CBX) = bx; S(CBY) = by; S(CBZ) = bz;
    S(CVX) = vx; S(CVY) = vy; S(CVZ) = vz;
    S(CEX) = fl.ex; S(CEY) = fl.ey; S(CEZ) = fl.ez;
    S(CFX) = fl.fxe; S(CFY) = fl.fye; S(CFZ) = fl.fze;
    S(CXX) = fl.fxx; S(CYY) = fl.fyy; S(CZZ) = fl.fzz;
    S(CXY) = fl.fxy; S(CXZ) = fl.fxz; S(CYZ) = fl.fyz;
#undef S
  };

  // ---- eight times the state predicted at the corners of plane k + 1/2
  // (mlwhalf.f:49-65), into the corner's own slots 0 .. 7; 0 outside the array
  auto corner_sums = [&](int k) {
    if (!cor_in) return;
    const D czk = df::scale(df::mul(dt, df::from_double(az.dim[k])), -2.0f);
    const D *L = cslot(k) + p00, *H = cslot(k + 1) + p00;
#pragma unroll 1
    for (int v = kv0; v < kv0 + 4; v++) {
      const VarFields q = kVar[v];
      auto at = [&](const D *p, int f) { return p + (size_t)f * T::NC; };
      D r = eight<T::CX, kSum>(at(L, v), at(H, v));
      if (q.fx >= 0)
        r = df::mad(signed_by(cxk, q.sx), eight<T::CX, kDx>(at(L, q.fx), at(H, q.fx)), r);
      if (q.fy >= 0)
        r = df::mad(signed_by(cyk, q.sy), eight<T::CX, kDy>(at(L, q.fy), at(H, q.fy)), r);
      if (q.fz >= 0)
        r = df::mad(signed_by(czk, q.sz), eight<T::CX, kDz>(at(L, q.fz), at(H, q.fz)), r);
      sk[(size_t)v * T::NK + kt] = r;
    }
  };

  // ---- fluxes of the corners of plane k + 1/2 (mlw_m.f:205-334) --------------
  auto corner_fluxes = [&]() {
    if (!cor_in) return;
    D *ks = sk + kt;
#define KS(f) ks[(size_t)(f) * T::NK]
    const D ro = KS(CRO), ee = KS(CEE), rx = KS(CRX), ry = KS(CRY), rz = KS(CRZ);
    const D bx = KS(CBX), by = KS(CBY), bz = KS(CBZ);
    // primitives and fluxes of the eightfold state: B B terms carry 64
    const D k4 = df::scale(P.pi4i, 0.125f), k8 = df::scale(P.pi8i, 0.125f);
    const D ri = df::rcp(ro);
    const D vx = df::mul(rx, ri), vy = df::mul(ry, ri), vz = df::mul(rz, ri);
    const D vv = df::mad(vz, vz, df::mad(vy, vy, df::sqr(vx)));
    const D bb = df::mad(bz, bz, df::mad(by, by, df::sqr(bx)));
    const D ek = df::mul(df::scale(ro, 0.5f), vv);
    const D pr = df::mul(P.gm1, df::sub(df::sub(ee, ek), df::mul(k8, bb)));
    const Flux3 fl = fluxes3(rx, ry, rz, vx, vy, vz, bx, by, bz, df::mad(pr, P.ggm1, ek),
                             df::mad(k8, bb, pr), k4);
    KS(KRX) = rx; KS(KRY) = ry; KS(KRZ) = rz;
    KS(KFX) = fl.fxe; KS(KFY) = fl.fye; KS(KFZ) = fl.fze;
    KS(KXX) = fl.fxx; KS(KYY) = fl.fyy; KS(KZZ) = fl.fzz;
    KS(KXY) = fl.fxy; KS(KXZ) = fl.fxz; KS(KYZ) = fl.fyz;
    KS(KEX) = fl.ex; KS(KEY) = fl.ey; KS(KEZ) = fl.ez;
#undef KS
  };

  // ---- per-column constants of the full step --------------------------------
  Weights<U> wx{}, wy{}, wz{};
  D dtx = df::mk(0.0f), dty = df::mk(0.0f), m2 = df::mk(0.0f);
  if (interior) {
    wx.set(ax, ii);
    wy.set(ay, jj);
    const D dxi = df::from_double(ax.di[ii]), dyi = df::from_double(ay.di[jj]);
    dtx = df::mul(dt, dxi);
    dty = df::mul(dt, dyi);
    const D x2 = df::sqr(dxi), y2 = df::sqr(dyi);
    m2 = df::gt(x2, y2) ? x2 : y2;
  }
  auto ret = [&](int r) -> D & { return sret[(size_t)r * T::NI + it]; };

  // the new values of the thread's variables; of ro and B their changes, which are
  // added to the input doubles
  D un[4] = {};
  double old[4] = {0.0, 0.0, 0.0, 0.0};
  D kmax = df::mk(0.0f);  // largest CFL key of the thread's cells
  bool bad = false;

  // ---- the new primitives of plane k and their CFL key -----------------------
  auto finish = [&](int k) {
    if (tid >= T::NI || !interior) return;
    const double ro_new = old[0] + df::to_double(un[CRO]);
    const double bx_new = old[1] + df::to_double(un[CBX]);
    const double by_new = old[2] + df::to_double(sun[2 * T::NI + tid]);
    const double bz_new = old[3] + df::to_double(sun[3 * T::NI + tid]);
    const D ee = un[CEE], rx = un[CRX], ry = sun[tid], rz = sun[T::NI + tid];
    const D ro = df::from_double(ro_new);
    const D bx = df::from_double(bx_new), by = df::from_double(by_new);
    const D bz = df::from_double(bz_new);
    const D ri = df::rcp(ro);
    const D vx = df::mul(rx, ri), vy = df::mul(ry, ri), vz = df::mul(rz, ri);
    const D vv = df::mad(vz, vz, df::mad(vy, vy, df::sqr(vx)));
    const D bb = df::mad(bz, bz, df::mad(by, by, df::sqr(bx)));
    const D pr = df::mul(P.gm1, df::sub(df::sub(ee, df::mul(df::scale(ro, 0.5f), vv)),
                                        df::mul(P.pi8i, bb)));
    const double prd = df::to_double(pr);
    const size_t g = (size_t)ii + (size_t)jj * ix + (size_t)k * plane;
    B[P3::RO * n + g] = ro_new;
    B[P3::PR * n + g] = prd;
    B[P3::VX * n + g] = df::to_double(vx);
    B[P3::VY * n + g] = df::to_double(vy);
    B[P3::VZ * n + g] = df::to_double(vz);
    B[P3::BX * n + g] = bx_new;
    B[P3::BY * n + g] = by_new;
    B[P3::BZ * n + g] = bz_new;
    if (ctl != nullptr && ii >= box.lo[0] && ii <= box.hi[0] && jj >= box.lo[1] &&
        jj <= box.hi[1] && k >= box.lo[2] && k <= box.hi[2]) {
      // cans3d/common/cfl_m.f:52-59 (pi in single precision), as the
      // largest S max(1/dx^2, 1/dy^2, 1/dz^2)
      const D s = df::mad(df::mad(P.gm, pr, df::mul(P.pi4i_cfl, bb)), ri, vv);
      const D z2 = df::sqr(df::from_double(az.di[k]));
      const D key = df::mul(s, df::gt(z2, m2) ? z2 : m2);
      if (key.h == key.h && df::gt(key, kmax)) kmax = key;
      constexpr long long kInf = 0x7ff0000000000000LL;
      const long long ra = __double_as_longlong(ro_new), pa = __double_as_longlong(prd);
      bad |= ra <= 0 || ra > kInf || pa <= 0 || pa > kInf ||
             (__float_as_uint(key.h) & 0x7fffffffu) > 0x7f800000u;
    }
  };

  // outside the array the corners are never formed
  for (int q = tid; q < NKF * T::NK; q += T::NT) sk[q] = df::mk(0.0f);
  for (int q = tid; q < T::NR * T::NI; q += T::NT) sret[q] = df::mk(0.0f);
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
      corner_fluxes();
    } else {
      const D *sl = cslot(k);
      if (ft == 0) {
        szc[0] = df::scale(df::mul(df::mul(P.qav, df::from_double(az.dm[k])),
                                   df::from_double(az.dim[k])), -64.0f);
        szc[1] = df::scale(df::mul(dt, df::from_double(az.di[k])), -0.015625f);
      }
      if (ft < T::NQX) {
        const D *v = sl + (size_t)CVX * T::NC + fxx + (fxr + 1) * T::CX;
        sqx[ft] = df::mul(qxc, jump(v[0], v[1]));
      }
      if (ft < T::NQY) {
        const D *v = sl + (size_t)CVY * T::NC + fyx + 1 + fyr * T::CX;
        sqy[ft] = df::mul(qyc, jump(v[0], v[T::CX]));
      }
    }
    __syncthreads();
    // (d) full step of plane k
    if (interior) {
      if (iv0 == 0) {  // read here, used by finish
        const size_t g = (size_t)ii + (size_t)jj * ix + (size_t)k * plane;
        old[0] = A[P3::RO * n + g];
        old[1] = A[P3::BX * n + g];
        old[2] = A[P3::BY * n + g];
        old[3] = A[P3::BZ * n + g];
      }
      const D *s0 = cslot(k) + c0, *s1 = cslot(k + 1) + c0, *kk = sk + kSW;
      const D ae = df::mul(dtx, sqx[lx + (ly - 1) * T::KX]);
      const D aw = df::mul(dtx, sqx[lx - 1 + (ly - 1) * T::KX]);
      const D an = df::mul(dty, sqy[lx - 1 + ly * TX]);
      const D as = df::mul(dty, sqy[lx - 1 + (ly - 1) * TX]);
      // 64 times the z viscosity of the upper face, negative
      const D qz = df::mul(szc[0], jump(s0[(size_t)CVZ * T::NC], s1[(size_t)CVZ * T::NC]));
      wz.set(az, k);
      // the corner sums carry 8 and weights of 1/2 a plane and axis, the z flux 32
      const D cx_ = df::scale(dtx, -0.015625f), cy_ = df::scale(dty, -0.015625f), cz_ = szc[1];
#pragma unroll 1
      for (int j = 0; j < 4; j++) {
        const int v = iv0 + j;
        const VarFields q = kVar[v];
        const D *u = s0 + (size_t)v * T::NC;
        const D u0 = u[0];
        D du = df::mul(ae, df::sub(u[1], u0));
        du = df::mad(aw, df::sub(u[-1], u0), du);
        du = df::mad(an, df::sub(u[T::CX], u0), du);
        du = df::mad(as, df::sub(u[-T::CX], u0), du);
        if (q.fx >= 0) {
          const D *f = s0 + (size_t)q.fx * T::NC, *c = kk + (size_t)q.kx * T::NK;
          const D g = wy.diff(c[0], c[1], c[T::KX], c[T::KX + 1]);
          du = df::mad(signed_by(cx_, q.sx), wz.planes(ret(8 + q.rx), g, f[-1], f[1]), du);
          ret(8 + q.rx) = g;
        }
        if (q.fy >= 0) {
          const D *f = s0 + (size_t)q.fy * T::NC, *c = kk + (size_t)q.ky * T::NK;
          const D g = wx.diff(c[0], c[T::KX], c[1], c[T::KX + 1]);
          du = df::mad(signed_by(cy_, q.sy), wz.planes(ret(15 + q.ry), g, f[-T::CX], f[T::CX]),
                       du);
          ret(15 + q.ry) = g;
        }
        D pu = df::mul(qz, df::sub(s1[(size_t)v * T::NC], u0));
        if (q.fz >= 0) {
          const size_t o = (size_t)q.fz * T::NC;
          const D *c = kk + (size_t)q.kz * T::NK;
          const D s = face(wx, wy, c[0], c[1], c[T::KX], c[T::KX + 1], s0[o], s1[o]);
          pu = df::add(signed_by(s, q.sz), pu);
        }
        du = df::mad(cz_, df::sub(pu, ret(v)), du);
        ret(v) = pu;
        const D r = v == CRO || v == CBX || v == CBY || v == CBZ ? du : df::add(u0, du);
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
    // largest key of the block, one conversion, root and division
    D m = kmax;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      D w;
      w.h = __shfl_xor_sync(0xffffffffu, m.h, o);
      w.l = __shfl_xor_sync(0xffffffffu, m.l, o);
      if (df::gt(w, m)) m = w;
    }
    const int lane = tid & 31, w = tid >> 5;
    if (lane == 0) sred[w] = df::to_double(m);
    __syncthreads();
    if (w == 0) {
      double x = lane < T::NT / 32 ? sred[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = y > x ? y : x;
      }
      if (lane == 0 && x > 0.0) atomic_min_pos(&ctl->cfl_bits, ctl->safety / sqrt(x));
    }
  }
}

template <int TX, int TY, int MINB, bool U>
cudaError_t launch3df(const double *A, double *B, int ix, int jx, int kx, const Axis &ax,
                      const Axis &ay, const Axis &az, const Phys &ph, double dt, Ctl *ctl,
                      Box3 box, int kchunk, cudaStream_t s) {
  using T = T3F<TX, TY, false>;
  auto kern = k_mlw3d_df<TX, TY, MINB, U>;
  static std::mutex mu;
  static int slots_of[64] = {};
  int dev = 0, slots = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
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
  kchunk = balance_kchunk((long long)bx * by, kx - 2, kchunk, slots);
  dim3 grid(bx, by, (kx - 2 + kchunk - 1) / kchunk);
  kern<<<grid, T::NT, T::smem_bytes, s>>>(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, kchunk);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

int mlw3d_df_tile_count() { return 2; }

cudaError_t launch_mlw3d_df(int tile, const double *A, double *B, int ix, int jx, int kx,
                            const Axis &ax, const Axis &ay, const Axis &az, const Phys &ph,
                            double dt, Ctl *ctl, Box3 box, cudaStream_t s) {
  if (ix < 3 || jx < 3 || kx < 3) return cudaErrorInvalidValue;
  // z chunks of at most 64 planes; tile 0: 16 x 16 columns (fewer cells and corners
  // are formed twice: 128^3 0.97 ms), tile 1: 16 x 8, two blocks a SM (1.00 ms)
  const bool u = ax.uniform && ay.uniform && az.uniform;
  auto f = tile == 1 ? (u ? launch3df<16, 8, 2, true> : launch3df<16, 8, 2, false>)
                     : (u ? launch3df<16, 16, 1, true> : launch3df<16, 16, 1, false>);
  return f(A, B, ix, jx, kx, ax, ay, az, ph, dt, ctl, box, 64, s);
}

}  // namespace cans
