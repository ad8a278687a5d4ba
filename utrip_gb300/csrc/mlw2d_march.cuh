// The y-marching block of the fused 2-D mLW step (sm_103a): mlw_m3 and mlw_m
// (cans2d/hdmlw/mlw_m3.f:64-374, mlw_m.f), with gravity (G: mlw_m3_g.f:95-121,
// 194-220) and resistivity (R: mlw_m3_e.f:124-132, 236-244), for the fast policy
// (FP64) and, mlw_m3 only, the double-float policy.  The exact policy, one
// operation of the reference after the other, is the tile of mlw2d_tile.cuh.
//
// A block takes a strip of 32 interior columns and a segment of rows, in chunks
// of CH rows; between chunks it keeps the last two cell rows and the last corner
// row instead of recomputing them, so its halo work is that of a 32 x segment
// tile while its shared memory is that of a 32 x CH tile.  Per chunk:
//   phase 1  cells of the new rows: conserved variables, fluxes, E
//   phase 2  corners: predictor (mlwhalf part 2, mlwsrch), half-step state and
//            fluxes; viscosity faces
//   phase 3  the rows' own cells: central differences (mlwhalf part 1), corrector
//            (mlwfull, mlwsrcf), viscosity (mlwartv), update, primitives, CFL
// 34 CH threads (whole warps): one per cell of the new rows, per corner, and per
// updated cell (32 CH of them).
//
// The FP64 step is bound by the FP64 pipe (71 % busy at 512^2, 88 % at most; HBM at
// 3 %) and by the latency of the integer sums that relieve it: an FP64 warp
// instruction takes 64 issue slots, of which the step uses 30 %.  So the algebra is
// arranged for the fewest FP64 instructions, 219 a cell:
//   - the momentum flux is symmetric (fx(ry) = fy(rx)), the total pressure formed
//     once, the corner mass fluxes are the half-step momenta;
//   - the corner values are kept at four times their value (the mean of u is a
//     sum and every flux linear in the conserved variables at given velocity):
//     the factor is in constants and weights, no scaling products;
//   - a field needed as a sum and a difference, or as both differences, shares
//     its partial sums;
//   - viscosity as one linear combination of five values;
//   - the predictor's cell sums and, on equally spaced axes, the corner and central
//     differences of a direction are integer sums (isum.cuh);
//   - what depends on the column alone is formed once per block;
//   - reciprocals of fd64.cuh; comparisons on the integer pipe.
// u_new = u + du, the terms of du summed first; ro and B, which are state
// variables, are added to in FP64 in both policies.
//
// The double-float step takes the same sums with one normalisation each (df64.cuh) and
// its eight variables in a rolled loop.  Measured at 512^2, a step: FP64 217 (a tile
// that recomputes its halo) -> 145 us, double-float 98 -> 88 us.
//
// AVF records (1) or holds (2) the viscosity's branch of every face: see
// mlw2d_tile.cuh.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <type_traits>

#include "balance2d.h"
#include "cans_common.cuh"
#include "cans_internal.h"
#include "df64.cuh"
#include "fd64.cuh"
#include "isum.cuh"
#include "mlw2d_tile.cuh"  // Prim, av_branch

namespace cans {

namespace {

using df::D;

// a cell of the new state the CFL cannot use (see bad_cell): ro or pr not
// positive or not finite, or a key that is not a number
__device__ __forceinline__ bool bad_cell_d(double ro, double pr, D key) {
  constexpr long long kInf = 0x7ff0000000000000LL;
  const long long a = __double_as_longlong(ro), b = __double_as_longlong(pr);
  const bool knan = (__float_as_uint(key.h) & 0x7fffffffu) > 0x7f800000u;
  return a <= 0 || a > kInf || b <= 0 || b > kInf || knan;
}

// warp maximum of a double-float key (h, l compared lexicographically)
__device__ __forceinline__ D warp_max_d(D v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    D w;
    w.h = __shfl_xor_sync(0xffffffffu, v.h, o);
    w.l = __shfl_xor_sync(0xffffffffu, v.l, o);
    if (df::gt(w, v) || v.h != v.h) v = w;
  }
  return v;
}

// Number operations of the marching kernel, which is written once for
// both: DFN, double-float on the FP32 pipes (the double-float policy), and
// F64N, FP64 with FMA contraction (the fast policy).
struct DFN {
  using V = df::D;
  static __device__ __forceinline__ V in(double x) { return df::from_double(x); }
  static __device__ __forceinline__ double out(V x) { return df::to_double(x); }
  static __device__ __forceinline__ V zero() { return df::mk(0.0f); }
  static __device__ __forceinline__ V mad(V a, V b, V c) { return df::mad(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return df::mul(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return df::add(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return df::sub(a, b); }
  static __device__ __forceinline__ V neg(V a) { return df::neg(a); }
  static __device__ __forceinline__ V scale(V a, float p2) { return df::scale(a, p2); }
  static __device__ __forceinline__ V sqr(V a) { return df::sqr(a); }
  // ae (ue - u) + aw (uw - u) + an (un - u) + as (us - u), aa = -(ae + aw + an + as):
  // differences first here, where a product's rounding is 2^-48 of it
  static __device__ __forceinline__ V visc(V ae, V ue, V aw, V uw, V an, V un, V as, V us, V,
                                           V u) {
    return mad(as, sub(us, u), mad(an, sub(un, u), mad(aw, sub(uw, u), mul(ae, sub(ue, u)))));
  }
  static __device__ __forceinline__ V add4(V a, V b, V c, V d) { return df::add4(a, b, c, d); }
  static __device__ __forceinline__ V diff6(V a, V b, V c, V d, V f, V g, float e0, float e1,
                                            bool &) {
    return df::diff6(a, b, c, d, f, g, __fmul_rn(e0, 0x1p-32f), __fmul_rn(e1, 0x1p-32f));
  }
  static __device__ __forceinline__ V rcp(V a) { return df::rcp(a); }
  static __device__ __forceinline__ V addf(V a, float b) { return df::addf(a, b); }
  static __device__ __forceinline__ V absd(V a) { return df::absd(a); }
  static __device__ __forceinline__ V pos_part(V a) { return df::pos(a) ? a : zero(); }
  static __device__ __forceinline__ bool gt(V a, V b) { return df::gt(a, b); }
  static __device__ __forceinline__ bool isnan(V a) { return a.h != a.h; }
  static __device__ __forceinline__ V nan_probe(V a) { return a; }
  static __device__ __forceinline__ V warp_max(V v) { return warp_max_d(v); }
};
struct F64N {
  using V = double;
  static __device__ __forceinline__ V in(double x) { return x; }
  static __device__ __forceinline__ double out(V x) { return x; }
  static __device__ __forceinline__ V zero() { return 0.0; }
  static __device__ __forceinline__ V mad(V a, V b, V c) { return fma(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
  static __device__ __forceinline__ V add(V a, V b) { return a + b; }
  static __device__ __forceinline__ V sub(V a, V b) { return a - b; }
  static __device__ __forceinline__ V neg(V a) { return -a; }
  static __device__ __forceinline__ V scale(V a, float p2) { return a * (double)p2; }
  static __device__ __forceinline__ V sqr(V a) { return a * a; }
  static __device__ __forceinline__ V visc(V ae, V ue, V aw, V uw, V an, V un, V as, V us, V aa,
                                           V u) {
    return fma(as, us, fma(an, un, fma(aw, uw, fma(ae, ue, aa * u))));
  }
  static __device__ __forceinline__ V add4(V a, V b, V c, V d) { return (a + b) + (c + d); }
  static __device__ __forceinline__ V diff6(V a, V b, V c, V d, V f, V g, float e0, float e1,
                                            bool &sp) {
    return isum::diff6(a, b, c, d, f, g, e0, e1, sp);
  }
  static __device__ __forceinline__ V rcp(V a) { return fd::rcp(a); }
  static __device__ __forceinline__ V addf(V a, float b) { return a + (double)b; }
  static __device__ __forceinline__ V absd(V a) { return fabs(a); }
  // max(0, a), and comparisons of a key with values that are not negative, on the
  // integer pipe
  static __device__ __forceinline__ V pos_part(V a) { return fd::pos_part(a); }
  static __device__ __forceinline__ bool gt(V a, V b) { return fd::lt(b, a); }
  static __device__ __forceinline__ bool isnan(V a) { return fd::is_nan(a); }
  // a float whose NaN-ness is the key's, for bad_cell_d
  static __device__ __forceinline__ df::D nan_probe(V a) {
    return {fd::is_nan(a) ? __int_as_float(0x7fc00000) : 0.0f, 0.0f};
  }
  static __device__ __forceinline__ V warp_max(V v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v, o);
      if (w > v || v != v) v = w;
    }
    return v;
  }
};
template <class N> struct PhysN {
  typename N::V gm, gm1, gm1i, ggm1, pi4i, pi8i, qav;
};
template <class N> __device__ __forceinline__ PhysN<N> phys_n(const Phys &ph) {
  return {N::in(ph.gm),   N::in(ph.gm1),  N::in(ph.gm1i), N::in(ph.ggm1),
          N::in(ph.pi4i), N::in(ph.pi8i), N::in(ph.qav)};
}

// cell slots: conserved, fluxes (XY = fx(ry) = fy(rx)), E_z, velocities; the
// z components of mlw_m3 last
enum {
  CRO, CEE, CRX, CRY, CBX, CBY, CFX, CFY, CXX, CYY, CXY, CEZ, CVX, CVY, NC2,
  CRZ = NC2, CBZ, CXZ, CYZ, CEX, CEY, NC3
};
// corner slots, four times their value; the mass fluxes are the momenta
enum { KRX, KRY, KFX, KFY, KXX, KYY, KXY, KEZ, NK2, KXZ = NK2, KYZ, KEX, KEY, NK3 };
constexpr int NOF = -1;

// Rows of a chunk of the FP64 steps: 34 x 7 cells, 33 x 7 corners and 32 x 7 updated
// cells fill 8, 8 and 7 warps, and two blocks of 8 warps leave 128 registers a
// thread.
constexpr int kFastCH = 7;

template <int CH, bool M3, bool G> struct March {
  static constexpr int TX = 32, CX = TX + 2, KX = TX + 1;
  static constexpr int CR = CH + 2, KR = CH + 1;  // cell rows, corner rows
  static constexpr int NC = CX * CR, NK = KX * KR;
  static constexpr int NQX = KX * CH, NQY = TX * KR;
  static constexpr int NCS = (M3 ? NC3 : NC2) + (G ? 3 : 0);
  static constexpr int NKS = (M3 ? NK3 : NK2) + (G ? 3 : 0);
  static constexpr int GC = NCS - 3, GK = NKS - 3;  // gravity: ro (v.g), ro gx, ro gy
  static constexpr int NT = (CX * CH + 31) / 32 * 32;
  static constexpr size_t smem_bytes =
      sizeof(double) * ((size_t)NCS * NC + (size_t)NKS * NK + NQX + NQY + 32);
};

// What one step of one grid needs.
struct MarchArgs {
  const double *A;
  double *B;
  int ix, jx;
  double dt, safety;
  unsigned long long *cfl;  // null: no CFL is reduced
  int *bad;
  Box3 box;
  const double *grav, *res;  // as in mlw2d_tile.cuh
  unsigned char *avb;
  unsigned long long *nflip;
};

// Cell values of one cell (phase 1).
template <class N, class T, bool M3, bool G, bool R>
__device__ __forceinline__ void march_cell(const MarchArgs &a, size_t n, size_t g,
                                           typename N::V *sc, int c, const PhysN<N> &P) {
  using V = typename N::V;
  using Q = Prim<M3>;
#define SC(s) sc[(size_t)(s) * T::NC + c]
  auto in = [&](int v) { return N::in(a.A[(size_t)v * n + g]); };
  const V ro = in(Q::RO), pr = in(Q::PR), vx = in(Q::VX), vy = in(Q::VY);
  const V bx = in(Q::BX), by = in(Q::BY);
  V vz = N::zero(), bz = N::zero();
  if constexpr (M3) {
    vz = in(Q::VZ);
    bz = in(Q::BZ);
  }
  const V rx = N::mul(ro, vx), ry = N::mul(ro, vy);
  V bb = N::mad(by, by, N::sqr(bx)), rv = N::mad(rx, vx, N::mul(ry, vy));
  V ez = N::mad(vy, bx, N::neg(N::mul(vx, by)));
  if constexpr (M3) {
    bb = N::mad(bz, bz, bb);
    rv = N::mad(N::mul(ro, vz), vz, rv);
  }
  const V ek = N::scale(rv, 0.5f);
  const V ep = N::mad(pr, P.ggm1, ek), pt = N::mad(P.pi8i, bb, pr);
  const V pbx = N::mul(P.pi4i, bx), pby = N::mul(P.pi4i, by);
  if constexpr (R) ez = N::add(ez, N::in(a.res[(M3 ? 2 * n : 0) + g]));
  V fx = N::mad(N::neg(pby), ez, N::mul(ep, vx)), fy = N::mad(pbx, ez, N::mul(ep, vy));
  if constexpr (M3) {
    const V rz = N::mul(ro, vz), pbz = N::mul(P.pi4i, bz);
    V ex = N::mad(vz, by, N::neg(N::mul(vy, bz))), ey = N::mad(vx, bz, N::neg(N::mul(vz, bx)));
    if constexpr (R) {
      ex = N::add(ex, N::in(a.res[g]));
      ey = N::add(ey, N::in(a.res[n + g]));
    }
    fx = N::mad(pbz, ey, fx);
    fy = N::mad(N::neg(pbz), ex, fy);
    SC(CRZ) = rz; SC(CBZ) = bz; SC(CEX) = ex; SC(CEY) = ey;
    SC(CXZ) = N::mad(rz, vx, N::neg(N::mul(pbx, bz)));
    SC(CYZ) = N::mad(rz, vy, N::neg(N::mul(pby, bz)));
  }
  SC(CRO) = ro; SC(CRX) = rx; SC(CRY) = ry; SC(CBX) = bx; SC(CBY) = by;
  SC(CEE) = N::mad(pr, P.gm1i, N::mad(P.pi8i, bb, ek));
  SC(CEZ) = ez; SC(CVX) = vx; SC(CVY) = vy;
  SC(CFX) = fx;
  SC(CFY) = fy;
  SC(CXX) = N::mad(rx, vx, N::mad(N::neg(pbx), bx, pt));
  SC(CYY) = N::mad(ry, vy, N::mad(N::neg(pby), by, pt));
  SC(CXY) = N::mad(rx, vy, N::neg(N::mul(pbx, by)));
  if constexpr (G) {  // mlw_m3_g.f:95, 106, 117
    const V gx = N::in(a.grav[g]), gy = N::in(a.grav[2 * n + g]);
    SC(T::GC) = N::mad(rx, gx, N::mul(ry, gy));
    SC(T::GC + 1) = N::mul(ro, gx);
    SC(T::GC + 2) = N::mul(ro, gy);
  }
#undef SC
}

// The predictor's four-cell sums of a field: S the sum over the cells a, b (x+1),
// c (x+1, y+1), d (y+1), X and Y the differences along x and y.  Fields needed in
// two forms share their partial sums.
template <class N, class T> struct Cells4 {
  using V = typename N::V;
  const V *p;  // cell a of field 0
  bool sp = false;
  __device__ __forceinline__ void load(int f, V &a, V &b, V &c, V &d) const {
    const V *q = p + (size_t)f * T::NC;
    a = q[0];
    b = q[1];
    c = q[T::CX + 1];
    d = q[T::CX];
  }
  __device__ __forceinline__ V sum(int f) {
    V a, b, c, d;
    load(f, a, b, c, d);
    return N::add4(b, a, c, d);
  }
  __device__ __forceinline__ V dx(int f) {
    V a, b, c, d;
    load(f, a, b, c, d);
    return N::add4(b, N::neg(a), c, N::neg(d));
  }
  __device__ __forceinline__ V dy(int f) {
    V a, b, c, d;
    load(f, a, b, c, d);
    return N::add4(d, N::neg(a), c, N::neg(b));
  }
  __device__ __forceinline__ void sum_dx(int f, V &s, V &x) {
    V a, b, c, d;
    load(f, a, b, c, d);
    const V l = N::add(a, d), r = N::add(b, c);
    s = N::add(l, r);
    x = N::sub(r, l);
  }
  __device__ __forceinline__ void sum_dy(int f, V &s, V &y) {
    V a, b, c, d;
    load(f, a, b, c, d);
    const V l = N::add(a, b), r = N::add(d, c);
    s = N::add(l, r);
    y = N::sub(r, l);
  }
  __device__ __forceinline__ void dx_dy(int f, V &x, V &y) {
    V a, b, c, d;
    load(f, a, b, c, d);
    const V u = N::sub(c, a), w = N::sub(b, d);
    x = N::add(u, w);
    y = N::sub(u, w);
  }
};
// The same for doubles on the integer pipe (isum.cuh); sp is set where a sum must
// be formed in FP64.
template <class T> struct ICells4 {
  const double *p;
  bool sp = false;
  __device__ __forceinline__ isum::Four load(int f) {
    const double *q = p + (size_t)f * T::NC;
    return isum::four(q[0], q[1], q[T::CX + 1], q[T::CX], sp);
  }
  __device__ __forceinline__ double sum(int f) {
    const isum::Four q = load(f);
    return isum::out<8>((q.a + q.b) + (q.c + q.d), q.E);
  }
  __device__ __forceinline__ double dx(int f) {
    const isum::Four q = load(f);
    return isum::out<8>((q.b - q.a) + (q.c - q.d), q.E);
  }
  __device__ __forceinline__ double dy(int f) {
    const isum::Four q = load(f);
    return isum::out<8>((q.d - q.a) + (q.c - q.b), q.E);
  }
  __device__ __forceinline__ void sum_dx(int f, double &s, double &x) {
    const isum::Four q = load(f);
    const long long l = q.a + q.d, r = q.b + q.c;
    s = isum::out<8>(l + r, q.E);
    x = isum::out<8>(r - l, q.E);
  }
  __device__ __forceinline__ void sum_dy(int f, double &s, double &y) {
    const isum::Four q = load(f);
    const long long l = q.a + q.b, r = q.d + q.c;
    s = isum::out<8>(l + r, q.E);
    y = isum::out<8>(r - l, q.E);
  }
  __device__ __forceinline__ void dx_dy(int f, double &x, double &y) {
    const isum::Four q = load(f);
    const long long u = q.c - q.a, w = q.b - q.d;
    x = isum::out<8>(u + w, q.E);
    y = isum::out<8>(u - w, q.E);
  }
};

// The predictor of one corner (mlwhalf part 2): four times its conserved values
// (ro, ee, rx, ry, bx, by, rz, bz) from the cell sums `st`.
template <class N, class T, bool M3, bool G, class St>
__device__ __forceinline__ void march_predict(St &st, typename N::V cx4, typename N::V cy4,
                                              typename N::V dt, typename N::V *u) {
  using V = typename N::V;
  const V nx = N::neg(cx4), ny = N::neg(cy4);
  V sx, sy, x, y;
  st.sum_dx(CRX, sx, x);
  st.sum_dy(CRY, sy, y);
  u[0] = N::mad(ny, y, N::mad(nx, x, st.sum(CRO)));
  st.dx_dy(CXY, x, y);
  u[2] = N::mad(ny, y, N::mad(nx, st.dx(CXX), sx));
  u[3] = N::mad(ny, st.dy(CYY), N::mad(nx, x, sy));
  u[1] = N::mad(ny, st.dy(CFY), N::mad(nx, st.dx(CFX), st.sum(CEE)));
  st.dx_dy(CEZ, x, y);
  u[4] = N::mad(ny, y, st.sum(CBX));
  u[5] = N::mad(cx4, x, st.sum(CBY));
  if constexpr (M3) {
    u[6] = N::mad(ny, st.dy(CYZ), N::mad(nx, st.dx(CXZ), st.sum(CRZ)));
    u[7] = N::mad(cy4, st.dy(CEX), N::mad(nx, st.dx(CEY), st.sum(CBZ)));
  }
  if constexpr (G) {  // mlwsrch part 2: dt times the mean of the four sources
    u[1] = N::mad(dt, st.sum(T::GC), u[1]);
    u[2] = N::mad(dt, st.sum(T::GC + 1), u[2]);
    u[3] = N::mad(dt, st.sum(T::GC + 2), u[3]);
  }
}
// The same with FP64 sums, into the corner's slots: where an integer sum cannot be
// formed (isum::special).
template <class T, bool M3, bool G>
__device__ __noinline__ void march_predict_fp64(const double *p, double *sk, double cx4,
                                                double cy4, double dt) {
  Cells4<F64N, T> st{p};
  double u[8];
  march_predict<F64N, T, M3, G>(st, cx4, cy4, dt, u);
  for (int v = 0; v < (M3 ? 8 : 6); v++) sk[(size_t)v * T::NK] = u[v];
}

// Half-step values of one corner k from its four cells a, b (x+1), cc (x+1, y+1),
// d (y+1), at four times their value (phase 2).  cx4, cy4 = 2 dt / dxm, 2 dt / dym;
// g the corner's index in the global arrays.
template <class N, class T, bool M3, bool G, bool R>
__device__ __forceinline__ void march_corner(const MarchArgs &m, size_t n, size_t g,
                                             const typename N::V *sc, typename N::V *sk, int a,
                                             int k, typename N::V cx4, typename N::V cy4,
                                             typename N::V dt, const PhysN<N> &P) {
  using V = typename N::V;
#define SK(s) sk[(size_t)(s) * T::NK + k]
  // global operands first, so that their latency overlaps the predictor
  double gq[2] = {0.0, 0.0}, rq[3] = {0.0, 0.0, 0.0};
  if constexpr (G) {
    gq[0] = m.grav[n + g];
    gq[1] = m.grav[3 * n + g];
  }
  if constexpr (R) {
    rq[2] = m.res[(M3 ? 5 * n : n) + g];
    if constexpr (M3) {
      rq[0] = m.res[3 * n + g];
      rq[1] = m.res[4 * n + g];
    }
  }
  V u[8];
  if constexpr (std::is_same<N, F64N>::value) {
    ICells4<T> st{sc + a};
    march_predict<N, T, M3, G>(st, cx4, cy4, dt, u);
    if (st.sp) {  // a real branch: the FP64 sums must not be predicated in
      march_predict_fp64<T, M3, G>(sc + a, sk + k, cx4, cy4, dt);
#pragma unroll
      for (int v = 0; v < (M3 ? 8 : 6); v++) u[v] = SK(v);
    }
  } else {
    Cells4<N, T> st{sc + a};
    march_predict<N, T, M3, G>(st, cx4, cy4, dt, u);
  }
  const V ro = u[0], ee = u[1], rx = u[2], ry = u[3], bx = u[4], by = u[5];
  const V rz = M3 ? u[6] : N::zero(), bz = M3 ? u[7] : N::zero();
  const V ri = N::rcp(ro), vx = N::mul(rx, ri), vy = N::mul(ry, ri);
  const V k4 = N::scale(P.pi4i, 0.25f), k8 = N::scale(P.pi8i, 0.25f);
  V vz = N::zero(), bb = N::mad(by, by, N::sqr(bx)), rv = N::mad(rx, vx, N::mul(ry, vy));
  V ez = N::mad(vy, bx, N::neg(N::mul(vx, by)));
  if constexpr (M3) {
    vz = N::mul(rz, ri);
    bb = N::mad(bz, bz, bb);
    rv = N::mad(rz, vz, rv);
  }
  const V ek = N::scale(rv, 0.5f);
  const V pr = N::mul(P.gm1, N::mad(N::neg(k8), bb, N::sub(ee, ek)));
  const V ep = N::mad(pr, P.ggm1, ek), pt = N::mad(k8, bb, pr);
  const V pbx = N::mul(k4, bx), pby = N::mul(k4, by);
  const V four = N::in(4.0);
  if constexpr (R) ez = N::mad(four, N::in(rq[2]), ez);
  V fx = N::mad(N::neg(pby), ez, N::mul(ep, vx)), fy = N::mad(pbx, ez, N::mul(ep, vy));
  if constexpr (M3) {
    const V pbz = N::mul(k4, bz);
    V ex = N::mad(vz, by, N::neg(N::mul(vy, bz))), ey = N::mad(vx, bz, N::neg(N::mul(vz, bx)));
    if constexpr (R) {
      ex = N::mad(four, N::in(rq[0]), ex);
      ey = N::mad(four, N::in(rq[1]), ey);
    }
    fx = N::mad(pbz, ey, fx);
    fy = N::mad(N::neg(pbz), ex, fy);
    SK(KEX) = ex; SK(KEY) = ey;
    SK(KXZ) = N::mad(rz, vx, N::neg(N::mul(pbx, bz)));
    SK(KYZ) = N::mad(rz, vy, N::neg(N::mul(pby, bz)));
  }
  SK(KRX) = rx; SK(KRY) = ry; SK(KEZ) = ez;
  SK(KFX) = fx;
  SK(KFY) = fy;
  SK(KXX) = N::mad(rx, vx, N::mad(N::neg(pbx), bx, pt));
  SK(KYY) = N::mad(ry, vy, N::mad(N::neg(pby), by, pt));
  SK(KXY) = N::mad(rx, vy, N::neg(N::mul(pbx, by)));
  if constexpr (G) {  // mlw_m3_g.f:194, 205, 216
    const V gx = N::in(gq[0]), gy = N::in(gq[1]);
    SK(T::GK) = N::mad(rx, gx, N::mul(ry, gy));
    SK(T::GK + 1) = N::mul(ro, gx);
    SK(T::GK + 2) = N::mul(ro, gy);
  }
#undef SK
}

// Corner field f weighted to the cell whose lower left corner is kSW.
template <class N, class T>
__device__ __forceinline__ typename N::V march_to_cell(const typename N::V *sk, int f, int kSW,
                                                       typename N::V ux0, typename N::V ux1,
                                                       typename N::V uy0, typename N::V uy1) {
  const typename N::V *q = sk + (size_t)f * T::NK + kSW;
  const typename N::V s = N::mad(ux1, q[1], N::mul(ux0, q[0]));
  const typename N::V t = N::mad(ux1, q[T::KX + 1], N::mul(ux0, q[T::KX]));
  return N::mad(uy1, t, N::mul(uy0, s));
}

// The fields of march_du's variables, in the order of du: conserved slot, x flux at the
// cells and corners and whether it enters negated, y flux, gravity source.
struct VarFields2 {
  signed char su, fx, nx, kfx, fy, ny, kfy, gs;
};
__constant__ VarFields2 kVar2[8] = {
    {CRO, CRX, 0, KRX, CRY, 0, KRY, -1}, {CEE, CFX, 0, KFX, CFY, 0, KFY, 0},
    {CRX, CXX, 0, KXX, CXY, 0, KXY, 1},  {CRY, CXY, 0, KXY, CYY, 0, KYY, 2},
    {CBX, NOF, 0, NOF, CEZ, 0, KEZ, -1}, {CBY, CEZ, 1, KEZ, NOF, 0, NOF, -1},
    {CRZ, CXZ, 0, KXZ, CYZ, 0, KYZ, -1}, {CBZ, CEY, 0, KEY, CEX, 1, KEX, -1}};

// The changes of the conserved variables of cell c (ro, ee, rx, ry, bx, by, rz,
// bz): viscosity, central differences, corrector, gravity sources.  ae .. as are dt
// q / (dx dxm) of the four faces, dtx = dt / dx, dty = dt / dy.
//
// U: the weights u0, u1 are one half up to ex0 .. ey1 (Axis::e0, e1), and the two
// corner differences and the central difference of a direction are one integer
// sum (isum::diff6): one FP64 instruction a direction where six are needed; in
// double-float one sum (df::diff6) and one product.
// sp is set where such a sum must be formed in FP64.
template <class N, class T, bool M3, bool G, bool U>
__device__ __forceinline__ void march_du(const typename N::V *sc, const typename N::V *sk, int c,
                                         int kSW, typename N::V ae, typename N::V aw,
                                         typename N::V an, typename N::V as, typename N::V dtx,
                                         typename N::V dty, typename N::V dt, typename N::V ux0,
                                         typename N::V ux1, typename N::V uy0, typename N::V uy1,
                                         float ex0, float ex1, float ey0, float ey1,
                                         typename N::V *du, bool &sp) {
  using V = typename N::V;
  const int cE = c + 1, cW = c - 1, cN = c + T::CX, cS = c - T::CX;
  const int kSE = kSW + 1, kNW = kSW + T::KX, kNE = kNW + 1;
#define SC(s, c) sc[(size_t)(s) * T::NC + (c)]
#define SK(s, c) sk[(size_t)(s) * T::NK + (c)]
  const V aa = N::neg(N::add(N::add(ae, aw), N::add(an, as)));
  // the corner values carry 4: hdt / 4 = dt / 8, and dt / 16 with a weight of 1/2
  const V dtx16 = N::scale(dtx, 0.0625f), dty16 = N::scale(dty, 0.0625f);
  const V fcx = N::scale(dtx, 0.25f), fcy = N::scale(dty, 0.25f);
  const V hx = N::scale(dtx, 0.125f), hy = N::scale(dty, 0.125f);
  const V fx0 = N::mul(hx, uy0), fx1 = N::mul(hx, uy1);
  const V fy0 = N::mul(hy, ux0), fy1 = N::mul(hy, ux1);
  auto var = [&](int su, int fx, bool nx, int kfx, int fy, bool ny, int kfy, int gs = -1) -> V {
    V d = N::visc(ae, SC(su, cE), aw, SC(su, cW), an, SC(su, cN), as, SC(su, cS), aa, SC(su, c));
    if constexpr (U) {
      // fx0 (SE - SW) + fx1 (NE - NW) + fcx (E - W) = dtx/16 diff6
      if (fx != NOF) {
        const V q = N::diff6(SK(kfx, kSW), SK(kfx, kSE), SK(kfx, kNW), SK(kfx, kNE),
                             SC(fx, cW), SC(fx, cE), ey0, ey1, sp);
        d = N::mad(nx ? dtx16 : N::neg(dtx16), q, d);
      }
      if (fy != NOF) {
        const V q = N::diff6(SK(kfy, kSW), SK(kfy, kNW), SK(kfy, kSE), SK(kfy, kNE),
                             SC(fy, cS), SC(fy, cN), ex0, ex1, sp);
        d = N::mad(ny ? dty16 : N::neg(dty16), q, d);
      }
    } else {
      if (fx != NOF) {
        d = N::mad(nx ? fcx : N::neg(fcx), N::sub(SC(fx, cE), SC(fx, cW)), d);
        d = N::mad(nx ? fx0 : N::neg(fx0), N::sub(SK(kfx, kSE), SK(kfx, kSW)), d);
        d = N::mad(nx ? fx1 : N::neg(fx1), N::sub(SK(kfx, kNE), SK(kfx, kNW)), d);
      }
      if (fy != NOF) {
        d = N::mad(ny ? fcy : N::neg(fcy), N::sub(SC(fy, cN), SC(fy, cS)), d);
        d = N::mad(ny ? fy0 : N::neg(fy0), N::sub(SK(kfy, kNW), SK(kfy, kSW)), d);
        d = N::mad(ny ? fy1 : N::neg(fy1), N::sub(SK(kfy, kNE), SK(kfy, kSE)), d);
      }
    }
    if constexpr (G) {
      if (gs >= 0) {  // mlwsrch part 1 and mlwsrcf
        d = N::mad(N::scale(dt, 0.5f), SC(T::GC + gs, c), d);
        d = N::mad(N::scale(dt, 0.125f),
                   march_to_cell<N, T>(sk, T::GK + gs, kSW, ux0, ux1, uy0, uy1), d);
      }
    }
    return d;
  };
  if constexpr (std::is_same<N, DFN>::value) {
    // rolled: unrolled, the step outgrows the instruction cache (a sixth of the stalled
    // cycles at 512^2); FP64's sums are fewer instructions
#pragma unroll 1
    for (int v = 0; v < (M3 ? 8 : 6); v++) {
      const VarFields2 q = kVar2[v];
      const V d = var(q.su, q.fx, q.nx, q.kfx, q.fy, q.ny, q.kfy, G ? q.gs : -1);
#pragma unroll
      for (int k = 0; k < (M3 ? 8 : 6); k++)
        if (k == v) du[k] = d;
    }
  } else {
    du[0] = var(CRO, CRX, false, KRX, CRY, false, KRY);
    du[4] = var(CBX, NOF, false, NOF, CEZ, false, KEZ);
    du[5] = var(CBY, CEZ, true, KEZ, NOF, false, NOF);
    if constexpr (M3) du[7] = var(CBZ, CEY, false, KEY, CEX, true, KEX);
    du[1] = var(CEE, CFX, false, KFX, CFY, false, KFY, 0);
    du[2] = var(CRX, CXX, false, KXX, CXY, false, KXY, 1);
    du[3] = var(CRY, CXY, false, KXY, CYY, false, KYY, 2);
    if constexpr (M3) du[6] = var(CRZ, CXZ, false, KXZ, CYZ, false, KYZ);
  }
#undef SC
#undef SK
}
// The same in FP64, for the cells march_du's integer sums leave.
template <class T, bool M3, bool G>
__device__ __noinline__ void march_du_fp64(const double *sc, const double *sk, int c, int kSW,
                                           double ae, double aw, double an, double as, double dtx,
                                           double dty, double dt, double ux0, double ux1,
                                           double uy0, double uy1, double *du) {
  bool sp = false;
  double d[8];
  march_du<F64N, T, M3, G, false>(sc, sk, c, kSW, ae, aw, an, as, dtx, dty, dt, ux0, ux1, uy0,
                                  uy1, 0.0f, 0.0f, 0.0f, 0.0f, d, sp);
  for (int v = 0; v < (M3 ? 8 : 6); v++) du[v] = d[v];
}

// Rows jb .. je of strip `strip` (of nstrips) of one grid.  Every thread of the
// block calls it; smem holds March<CH, M3, G>::smem_bytes.
template <class N, int CH, bool M3, bool G, bool R, int AVF, bool U>
__device__ __forceinline__ void march_block(const MarchArgs &m, const Axis &ax, const Axis &ay,
                                            const Phys &ph, int strip, int nstrips, int jb,
                                            int je, double *smem) {
  using T = March<CH, M3, G>;
  using V = typename N::V;
  using Q = Prim<M3>;
  static_assert(T::NQX <= T::NT && T::NQY <= T::NT, "a thread takes one face of each kind");
  V *sc = reinterpret_cast<V *>(smem);      // cells   [NCS][CR][CX]
  V *sk = sc + (size_t)T::NCS * T::NC;      // corners [NKS][KR][KX]
  V *sqx = sk + (size_t)T::NKS * T::NK;     // q / dxm [CH][KX]
  V *sqy = sqx + T::NQX;                    // q / dym [KR][TX]
  double *sred = reinterpret_cast<double *>(sqy + T::NQY);
#define SC(s, c) sc[(size_t)(s) * T::NC + (c)]
#define SK(s, c) sk[(size_t)(s) * T::NK + (c)]
  const double *__restrict__ A = m.A;
  double *__restrict__ B = m.B;
  const int ix = m.ix, jx = m.jx, tid = threadIdx.x;
  const size_t n = (size_t)ix * (size_t)jx;
  const int i0 = 1 + strip * T::TX;
  const PhysN<N> P = phys_n<N>(ph);
  const V dt = N::in(m.dt), dt2 = N::scale(dt, 2.0f), dt8 = N::scale(dt, 0.125f);
  // the thread's column of phase 3 and its x face, the same in every chunk
  const int lx = tid % T::TX + 1, gi3 = i0 - 1 + lx;
  const bool col = gi3 <= ix - 2;
  const V dxi = N::in(col ? ax.di[gi3] : 0.0);
  const V ux0 = N::in(col ? ax.u0[gi3] : 0.0), ux1 = N::in(col ? ax.u1[gi3] : 0.0);
  const V dtx = N::mul(dt, dxi), ix2 = N::sqr(dxi);
  const int fxi = tid % T::KX, fxr = tid / T::KX;
  const bool facex = tid < T::NQX && i0 + fxi < ix;
  const V qxc = facex ? N::mul(N::mul(P.qav, N::in(ax.dm[i0 - 1 + fxi])),
                               N::in(ax.dim[i0 - 1 + fxi]))
                      : N::zero();
  // the coefficient of one viscosity face of jump d: c max(0, |d| - 1e-4), the
  // real*4 threshold 1.0e-4 a float
  auto visc_face = [&](V c, V d, size_t gf, bool real, bool owned) -> V {
    const V a = N::addf(N::absd(d), -1.0e-4f);
    if constexpr (AVF != 0) {
      if (!real) return N::zero();
      const unsigned char br = av_branch<AVF>(d, F<false>(a), m.avb + gf, m.nflip, owned);
      if (!(br & 1)) return N::zero();
      return N::mul(c, N::addf((br & 2) ? N::neg(d) : d, -1.0e-4f));
    }
    return N::mul(c, N::pos_part(a));
  };
  const bool edge_x = strip == 0 || strip == nstrips - 1;
  V kmax = N::zero();
  bool bad = false;

  for (int j0 = jb; j0 <= je; j0 += CH) {
    const bool first = j0 == jb;
    if (!first) {
      // keep the chunk's last two cell rows and last corner row
      for (int e = tid; e < T::NCS * 2 * T::CX; e += T::NT) {
        const int s = e / (2 * T::CX), r = e % (2 * T::CX);
        SC(s, r) = SC(s, CH * T::CX + r);
      }
      for (int e = tid; e < T::NKS * T::KX; e += T::NT) {
        const int s = e / T::KX, r = e % T::KX;
        SK(s, r) = SK(s, CH * T::KX + r);
      }
      __syncthreads();
    }
    // ---- phase 1: new cell rows (all CH + 2 of the first chunk) ----
    const int last_row = min(CH + 1, je + 1 - (j0 - 1));  // rows past je+1 are not read
    for (int c = (first ? 0 : 2 * T::CX) + tid; c < (last_row + 1) * T::CX; c += T::NT) {
      const int gi = i0 - 1 + c % T::CX, gj = j0 - 1 + c / T::CX;
      if (gi < ix && gj < jx) {
        march_cell<N, T, M3, G, R>(m, n, (size_t)gi + (size_t)gj * ix, sc, c, P);
      } else {
#pragma unroll 1
        for (int s = 0; s < T::NCS; s++) SC(s, c) = N::zero();
      }
    }
    __syncthreads();
    // ---- phase 2: new corner rows, and the viscosity faces ----
    for (int k = (first ? 0 : T::KX) + tid; k < last_row * T::KX; k += T::NT) {
      const int kx = k % T::KX, ky = k / T::KX;
      const int gi = i0 - 1 + kx, gj = j0 - 1 + ky;
      if (gi <= ix - 2 && gj <= jx - 2) {
        march_corner<N, T, M3, G, R>(m, n, (size_t)gi + (size_t)gj * ix, sc, sk,
                                     kx + ky * T::CX, k, N::mul(dt2, N::in(ax.dim[gi])),
                                     N::mul(dt2, N::in(ay.dim[gj])), dt, P);
      } else {
#pragma unroll 1
        for (int s = 0; s < T::NKS; s++) SK(s, k) = N::zero();
      }
    }
    if (tid < T::NQX) {
      const int gj = j0 + fxr, cl = fxi + (fxr + 1) * T::CX;
      sqx[tid] = visc_face(qxc, N::sub(SC(CVX, cl + 1), SC(CVX, cl)),
                           (size_t)(i0 - 1 + fxi) + (size_t)gj * ix,
                           facex && gj <= je, fxi > 0 || strip == 0);
    }
    if (tid < T::NQY) {
      const int r = tid / T::TX, gj = j0 - 1 + r, cl = lx + r * T::CX;
      V v = N::zero();
      if (gi3 < ix && gj + 1 < jx)
        v = visc_face(N::mul(N::mul(P.qav, N::in(ay.dm[gj])), N::in(ay.dim[gj])),
                      N::sub(SC(CVY, cl + T::CX), SC(CVY, cl)),
                      n + (size_t)gi3 + (size_t)gj * ix, gj <= je, r > 0 || j0 == 1);
      sqy[tid] = v;
    }
    __syncthreads();
    // ---- phase 3: the chunk's own cells ----
    const int ly = tid / T::TX + 1, gj = j0 - 1 + ly;
    if (tid < T::TX * CH && col && gj <= je) {
      const int gi = gi3;
      const size_t g = (size_t)gi + (size_t)gj * ix;
      // the doubles the update adds to, loaded ahead of the arithmetic
      const double ro0 = A[Q::RO * n + g], bx0 = A[Q::BX * n + g], by0 = A[Q::BY * n + g];
      const double az0 = A[Q::AZ * n + g];
      double bz0 = 0.0;
      if constexpr (M3) bz0 = A[Q::BZ * n + g];
      const int c = lx + ly * T::CX;
      const int kSW = (lx - 1) + (ly - 1) * T::KX;
      const V dyi = N::in(ay.di[gj]);
      const V uy0 = N::in(ay.u0[gj]), uy1 = N::in(ay.u1[gj]);
      const V dty = N::mul(dt, dyi);
      const V ae = N::mul(dtx, sqx[lx + (ly - 1) * T::KX]);
      const V aw = N::mul(dtx, sqx[lx - 1 + (ly - 1) * T::KX]);
      const V an = N::mul(dty, sqy[(lx - 1) + ly * T::TX]);
      const V as = N::mul(dty, sqy[(lx - 1) + (ly - 1) * T::TX]);
      V du[8];
      if constexpr (U) {
        bool sp = false;
        march_du<N, T, M3, G, true>(sc, sk, c, kSW, ae, aw, an, as, dtx, dty, dt, ux0, ux1, uy0,
                                    uy1, ax.e0[gi], ax.e1[gi], ay.e0[gj], ay.e1[gj], du, sp);
        if constexpr (std::is_same<N, F64N>::value) {
          if (sp) {  // a real branch, as in march_corner
            double slow[8];
            march_du_fp64<T, M3, G>(sc, sk, c, kSW, ae, aw, an, as, dtx, dty, dt, ux0, ux1, uy0,
                                    uy1, slow);
#pragma unroll
            for (int v = 0; v < (M3 ? 8 : 6); v++) du[v] = slow[v];
          }
        }
      } else {
        bool sp = false;
        march_du<N, T, M3, G, false>(sc, sk, c, kSW, ae, aw, an, as, dtx, dty, dt, ux0, ux1, uy0,
                                     uy1, 0.0f, 0.0f, 0.0f, 0.0f, du, sp);
      }
      const double ro_new = ro0 + N::out(du[0]), bx_new = bx0 + N::out(du[4]);
      const double by_new = by0 + N::out(du[5]);
      const V ee = N::add(SC(CEE, c), du[1]), rx = N::add(SC(CRX, c), du[2]);
      const V ry = N::add(SC(CRY, c), du[3]);
      double bz_new = 0.0;
      V rz = N::zero();
      if constexpr (M3) {
        rz = N::add(SC(CRZ, c), du[6]);
        bz_new = bz0 + N::out(du[7]);
      }
      // vector potential: mlwsrch part 1 + mlwsrcf with s = -ez, -ezh
      B[Q::AZ * n + g] =
          az0 - N::out(N::mad(dt8, march_to_cell<N, T>(sk, KEZ, kSW, ux0, ux1, uy0, uy1),
                              N::mul(N::scale(dt, 0.5f), SC(CEZ, c))));
      // back to primitives (mlw_m3.f:365-374)
      const V ro = N::in(ro_new), bx = N::in(bx_new), by = N::in(by_new);
      const V rinv = N::rcp(ro), vx = N::mul(rx, rinv), vy = N::mul(ry, rinv);
      V ek2 = N::mad(rx, vx, N::mul(ry, vy)), bb = N::mad(by, by, N::sqr(bx));
      if constexpr (M3) {
        const V bz = N::in(bz_new), vz = N::mul(rz, rinv);
        ek2 = N::mad(rz, vz, ek2);
        bb = N::mad(bz, bz, bb);
        B[Q::VZ * n + g] = N::out(vz);
        B[Q::BZ * n + g] = bz_new;
      }
      const V pr =
          N::mul(P.gm1, N::mad(N::neg(P.pi8i), bb, N::sub(ee, N::scale(ek2, 0.5f))));
      const double prd = N::out(pr);
      B[Q::RO * n + g] = ro_new;
      B[Q::PR * n + g] = prd;
      B[Q::VX * n + g] = N::out(vx);
      B[Q::VY * n + g] = N::out(vy);
      B[Q::BX * n + g] = bx_new;
      B[Q::BY * n + g] = by_new;
      if (m.cfl != nullptr && gi >= m.box.lo[0] && gi <= m.box.hi[0] && gj >= m.box.lo[1] &&
          gj <= m.box.hi[1]) {
        // the largest (v^2 + (gm p + B^2/4pi)/ro) max(1/dx^2, 1/dy^2) gives the
        // smallest time step (cfl_m3.f:46-55); ro v^2 = ek2
        const V s = N::mul(N::mad(P.gm, pr, N::mad(P.pi4i, bb, ek2)), rinv);
        const V iy2 = N::sqr(dyi);
        const V key = N::mul(s, N::gt(ix2, iy2) ? ix2 : iy2);
        if (!N::isnan(key) && N::gt(key, kmax)) kmax = key;
        bad |= bad_cell_d(ro_new, prd, N::nan_probe(key));
      }
    }
    // ghost cells of the output keep their input values; each is copied by
    // the chunk owning its nearest interior cell
    if (edge_x || j0 == 1 || j0 + CH - 1 >= jx - 2) {
      for (int c = tid; c < T::NC; c += T::NT) {
        const int gi = i0 - 1 + c % T::CX, gk = j0 - 1 + c / T::CX;
        if (gi >= ix || gk >= jx) continue;
        if (gi != 0 && gi != ix - 1 && gk != 0 && gk != jx - 1) continue;
        const int ci = min(max(gi, 1), ix - 2), cj = min(max(gk, 1), jx - 2);
        if (ci < i0 || ci >= i0 + T::TX || cj < j0 || cj >= j0 + CH || cj > je) continue;
        const size_t g = (size_t)gi + (size_t)gk * ix;
#pragma unroll
        for (int v = 0; v < Q::N; v++) B[v * n + g] = A[v * n + g];
      }
    }
    __syncthreads();
  }
#undef SC
#undef SK
  if (m.cfl != nullptr) {
    if (m.bad != nullptr) count_bad_block(bad, m.bad, tid);
    // 1 / sqrt(largest key): one conversion, root and division per block
    kmax = N::warp_max(kmax);
    const int lane = tid & 31, w = tid >> 5;
    if (lane == 0) sred[w] = N::out(kmax);
    __syncthreads();
    if (w == 0) {
      double x = lane < (T::NT + 31) / 32 ? sred[lane] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_xor_sync(0xffffffffu, x, o);
        x = (y > x || x != x) ? y : x;
      }
      if (lane == 0 && x > 0.0) atomic_min_pos(m.cfl, m.safety / sqrt(x));
    }
  }
}

// The marching step of one grid (U: both axes are uniform): block (strip, segment of `seg` rows).
template <class N, int CH, bool M3, bool G, bool R, int AVF, bool U>
__global__ void __launch_bounds__(March<CH, M3, G>::NT, 2)
    k_mlw2d_march(MarchArgs m, Axis ax, Axis ay, Phys ph, Ctl *__restrict__ ctl, int seg) {
  extern __shared__ double smem_march[];
  if (ctl != nullptr) {
    if (ctl->done | ctl->pause) return;
    m.A = ctl->buf[ctl->cur];
    m.B = ctl->buf[ctl->cur ^ 1];
    m.dt = ctl->dt;
    m.safety = ctl->safety;
    m.cfl = &ctl->cfl_bits;
    m.bad = &ctl->nonfinite;
  }
  const int jb = 1 + blockIdx.y * seg;
  march_block<N, CH, M3, G, R, AVF, U>(m, ax, ay, ph, blockIdx.x, gridDim.x, jb,
                                    min(m.jx - 2, jb + seg - 1), smem_march);
}

template <class N, int CH, bool M3, bool G, bool R, int AVF, bool U>
cudaError_t launch_march_u(const MarchArgs &m, const Axis &ax, const Axis &ay, const Phys &ph,
                         Ctl *ctl, cudaStream_t s, bool waves = false) {
  using T = March<CH, M3, G>;
  static std::mutex mu;
  static int sms_of[64] = {}, slots_of[64] = {};
  auto kern = k_mlw2d_march<N, CH, M3, G, R, AVF, U>;
  int dev = 0, sms = 0, slots = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!sms_of[dev]) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)T::smem_bytes);
      if (e != cudaSuccess) return e;
      int sm = 0, per_sm = 0;
      if ((e = cudaDeviceGetAttribute(&sm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
      if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, T::NT,
                                                             T::smem_bytes)) != cudaSuccess)
        return e;
      sms_of[dev] = sm > 0 ? sm : 1;
      slots_of[dev] = sms_of[dev] * (per_sm > 0 ? per_sm : 1);
    }
    sms = sms_of[dev];
    slots = slots_of[dev];
  }
  const int strips = (m.ix - 2 + T::TX - 1) / T::TX, rows = m.jx - 2;
  const int seg = waves ? balance_seg_waves(strips, rows, CH, slots)
                        : balance_seg(strips, rows, CH, sms);
  const dim3 grid(strips, (rows + seg - 1) / seg);
  kern<<<grid, T::NT, T::smem_bytes, s>>>(m, ax, ay, ph, ctl, seg);
  count_launch();
  return cudaGetLastError();
}

template <class N, int CH, bool M3, bool G, bool R, int AVF = 0>
cudaError_t launch_march(const MarchArgs &m, const Axis &ax, const Axis &ay, const Phys &ph,
                         Ctl *ctl, cudaStream_t s, bool waves = false) {
  if (ax.uniform && ay.uniform)
    return launch_march_u<N, CH, M3, G, R, AVF, true>(m, ax, ay, ph, ctl, s, waves);
  return launch_march_u<N, CH, M3, G, R, AVF, false>(m, ax, ay, ph, ctl, s, waves);
}

}  // namespace

}  // namespace cans
