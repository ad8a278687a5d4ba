// HLLD flux of one face on the device:
// cansxx-nosupport/hdhlld/hlld_flux.f90:148-480 (Miyoshi & Kusano, J. Comput.
// Phys. 208, 315 (2005)), Heaviside units (pb = B^2/2).
//
// Face states in the frame of the face normal: (ro, pr, vn, vt1, vt2, bn,
// bt1, bt2) with bn unused -- the normal field is the face value bxs; the
// flux comes back as (ro, ee, rn, rt1, rt2, bt1, bt2).
//
// hlld_flux_t is written once for its number type T:
//   F<true>   the exact policy: the expressions in the Fortran order with
//             separately rounded operations;
//   df::DF    the double-float policy: the same expressions with reciprocals in
//             place of the repeated divisions on the FP32 pipes (df64.cuh), face
//             states and fluxes converted once.
// hlld_flux_fast is the fast policy's flux, in FP64 (below).
#pragma once
#include <type_traits>

#include "cans_common.cuh"
#include "df64.cuh"
#include "fd64.cuh"
#include "roe_flux.cuh"  // fmax_, fsign_, the double-float rcp_ and sqrt_

namespace cans {

struct HlldK {
  double gm, gm1;   // gm, gm-1
  double zfloor;    // hlld_mh.f:34
  double gm1i;      // fast and double-float policies: 1/(gm-1)
};

// What the flux needs of its number type beyond the arithmetic operators:
// conversion from and to the caller's doubles, the sign tests of its
// branches and the reciprocal of the fast algebra.
template <class T> struct HNum;
template <> struct HNum<F<true>> {
  static constexpr bool exact = true;
  static __device__ __forceinline__ F<true> in(double x) { return F<true>(x); }
  static __device__ __forceinline__ double out(F<true> x) { return x.v; }
  static __device__ __forceinline__ bool ge0(F<true> x) { return x.v >= 0.0; }
  static __device__ __forceinline__ bool gt0(F<true> x) { return x.v > 0.0; }
  static __device__ __forceinline__ bool le0(F<true> x) { return x.v <= 0.0; }
  static __device__ __forceinline__ F<true> rcp(F<true> x) { return F<true>(1.0) / x; }
};
// a normalised double-float carries its sign in the head (a zero head has a
// zero tail)
template <> struct HNum<df::DF> {
  static constexpr bool exact = false;
  static __device__ __forceinline__ df::DF in(double x) { return num_in<df::DF>(x); }
  static __device__ __forceinline__ double out(df::DF x) { return num_out(x); }
  static __device__ __forceinline__ bool ge0(df::DF x) { return !(x.d.h < 0.0f); }
  static __device__ __forceinline__ bool gt0(df::DF x) { return x.d.h > 0.0f; }
  static __device__ __forceinline__ bool le0(df::DF x) { return !(x.d.h > 0.0f); }
  static __device__ __forceinline__ df::DF rcp(df::DF x) { return rcp_(x); }
};
// Fortran max, min, sign, abs and sqrt of double-floats, in the forms the
// F<E> versions take
__device__ __forceinline__ df::DF fmax_(df::DF a, df::DF b) {
  return df::gt(a.d, b.d) ? a : b;
}
__device__ __forceinline__ df::DF fmin_(df::DF a, df::DF b) {
  return df::gt(b.d, a.d) ? a : b;
}
__device__ __forceinline__ df::DF fsign_(df::DF a, df::DF b) {
  const df::D m = df::absd(a.d);
  return df::DF(signbit(b.d.h) ? df::neg(m) : m);
}
__device__ __forceinline__ df::DF fabs_(df::DF a) { return df::DF(df::absd(a.d)); }
__device__ __forceinline__ df::DF fsqrt(df::DF a) { return sqrt_(a); }

// ill (double-float instance): set when a subsonic face's star state is
// ill-conditioned for double-float -- its denominator
// ro (S - vn)(S - S_M) - bn^2 a difference of nearly equal terms, below
// kIllCond of them, where the star state's error grows as the rounding unit
// over that ratio -- so that the caller evaluates the face in FP64.
template <class T>
__device__ __forceinline__ void hlld_flux_t(const HlldK &K, const double *L,
                                            const double *R, double bxv,
                                            double *f, bool *ill = nullptr) {
  using N = HNum<T>;
  constexpr bool E = N::exact;
  const T gm = N::in(K.gm), gm1 = N::in(K.gm1), zf = N::in(K.zfloor);
  const T bxs = N::in(bxv);
  const T bxsq = bxs * bxs;
  // left and right states (:152-191)
  const T rol = N::in(L[0]), prl = N::in(L[1]), vxl = N::in(L[2]), vyl = N::in(L[3]),
          vzl = N::in(L[4]), byl = N::in(L[6]), bzl = N::in(L[7]);
  const T ror = N::in(R[0]), prr = N::in(R[1]), vxr = N::in(R[2]), vyr = N::in(R[3]),
          vzr = N::in(R[4]), byr = N::in(R[6]), bzr = N::in(R[7]);
  const T pbl = T(0.5) * (bxs * bxs + byl * byl + bzl * bzl);
  const T ptl = prl + pbl;
  T eel, eer;
  if constexpr (E) {
    eel = prl / gm1 + T(0.5) * rol * (vxl * vxl + vyl * vyl + vzl * vzl) + pbl;
  } else {
    eel = prl * N::in(K.gm1i) + T(0.5) * rol * (vxl * vxl + vyl * vyl + vzl * vzl) + pbl;
  }
  const T rxl = rol * vxl, ryl = rol * vyl, rzl = rol * vzl;
  const T pbr = T(0.5) * (bxs * bxs + byr * byr + bzr * bzr);
  const T ptr = prr + pbr;
  if constexpr (E) {
    eer = prr / gm1 + T(0.5) * (ror * (vxr * vxr + vyr * vyr + vzr * vzr)) + pbr;
  } else {
    eer = prr * N::in(K.gm1i) + T(0.5) * (ror * (vxr * vxr + vyr * vyr + vzr * vzr)) + pbr;
  }
  const T rxr = ror * vxr, ryr = ror * vyr, rzr = ror * vzr;
  // wave speeds (:197-207)
  const T gmpl = gm * prl, gmpr = gm * prr;
  const T gpbl = gmpl + T(2.0) * pbl, gpbr = gmpr + T(2.0) * pbr;
  const T cfl = fsqrt((gpbl + fsqrt(gpbl * gpbl - T(4.0) * gmpl * bxsq)) / (T(2.0) * rol));
  const T cfr = fsqrt((gpbr + fsqrt(gpbr * gpbr - T(4.0) * gmpr * bxsq)) / (T(2.0) * ror));
  const T cfm = fmax_(cfl, cfr);
  const T sl = fmin_(vxl, vxr) - cfm;
  const T sr = fmax_(vxl, vxr) + cfm;
  // physical fluxes (:214-229)
  const T frol = rxl;
  const T frxl = rxl * vxl + ptl - bxsq;
  const T fryl = rol * vxl * vyl - bxs * byl;
  const T frzl = rol * vxl * vzl - bxs * bzl;
  const T feel = vxl * (eel + ptl - bxsq) - bxs * (vyl * byl + vzl * bzl);
  const T fbyl = byl * vxl - bxs * vyl;
  const T fbzl = bzl * vxl - bxs * vzl;
  const T fror = rxr;
  const T frxr = rxr * vxr + ptr - bxsq;
  const T fryr = ror * vxr * vyr - bxs * byr;
  const T frzr = ror * vxr * vzr - bxs * bzr;
  const T feer = vxr * (eer + ptr - bxsq) - bxs * (vyr * byr + vzr * bzr);
  const T fbyr = byr * vxr - bxs * vyr;
  const T fbzr = bzr * vxr - bxs * vzr;
  // The double-float instance runs one straight-line path: its instruction
  // footprint, not its arithmetic, bounds it, so the branches below become
  // selects (SL: the face takes a one-sided state; the supersonic cases keep
  // the physical flux of their side).
  constexpr bool SL = std::is_same<T, df::DF>::value;
  // supersonic cases (:235-255)
  if (!SL && N::ge0(sl)) {
    f[0] = N::out(frol); f[1] = N::out(feel); f[2] = N::out(frxl); f[3] = N::out(fryl);
    f[4] = N::out(frzl); f[5] = N::out(fbyl); f[6] = N::out(fbzl);
    return;
  }
  if (!SL && N::le0(sr)) {
    f[0] = N::out(fror); f[1] = N::out(feer); f[2] = N::out(frxr); f[3] = N::out(fryr);
    f[4] = N::out(frzr); f[5] = N::out(fbyr); f[6] = N::out(fbzr);
    return;
  }
  // contact speed and star total pressure (:260-275)
  const T sdl = sl - vxl, sdr = sr - vxr;
  const T den = sdr * ror - sdl * rol;
  T sm, ptst;
  if constexpr (E) {
    sm = (sdr * ror * vxr - sdl * rol * vxl - ptr + ptl) / den;
    ptst = (sdr * ror * ptl - sdl * rol * ptr + rol * ror * sdr * sdl * (vxr - vxl)) / den;
  } else {
    const T di = N::rcp(den);
    sm = (sdr * ror * vxr - sdl * rol * vxl - ptr + ptl) * di;
    ptst = (sdr * ror * ptl - sdl * rol * ptr + rol * ror * sdr * sdl * (vxr - vxl)) * di;
  }
  const T sdml = sl - sm, sdmr = sr - sm;
  // one-sided star state (:281-342); side 0 left, 1 right
  T rost[2], rxst[2], ryst[2], rzst[2], vyst[2], vzst[2], byst[2], bzst[2], eest[2];
  T vdbst[2];
  // the star states' denominators first: where one is ill-conditioned for
  // double-float the caller evaluates the face in FP64, and the double-float
  // instance stops before the rest of the star states
  T temp_fst[2];
  bool illv = false;
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const T ro = s ? ror : rol, sd = s ? sdr : sdl, sdm = s ? sdmr : sdml;
    temp_fst[s] = ro * sd * sdm - bxsq;
    if constexpr (std::is_same<T, df::DF>::value) {
      if (ill != nullptr) {
        const float big = fabsf(ro.d.h * sd.d.h * sdm.d.h) + bxsq.d.h;
        if (!(fabsf(temp_fst[s].d.h) >= kIllCond * big)) illv = true;
      }
    }
  }
  if constexpr (SL) {
    if (ill != nullptr && illv && !(N::ge0(sl) || N::le0(sr))) {
      *ill = true;  // the caller evaluates the face in FP64
      return;
    }
  }
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const T ro = s ? ror : rol, vx = s ? vxr : vxl, vy = s ? vyr : vyl, vz = s ? vzr : vzl;
    const T by = s ? byr : byl, bz = s ? bzr : bzl, pt = s ? ptr : ptl, ee = s ? eer : eel;
    const T sd = s ? sdr : sdl, sdm = s ? sdmr : sdml;
    const T s3 = fsign_(T(1.0), temp_fst[s] + zf) * fsign_(T(1.0), temp_fst[s] - zf);
    const T mx = fmax_(T(0.0), s3), mn = fmin_(T(0.0), s3);
    const T dd = temp_fst[s] + mn;
    T tmp, tmp2, rsd, esd;
    if constexpr (E) {
      tmp = bxs * (sd - sdm) / dd;
      tmp2 = (ro * (sd * sd) - bxsq) / dd;
      rsd = ro * sd / sdm;
    } else {
      const T ddi = N::rcp(dd);
      tmp = bxs * (sd - sdm) * ddi;
      tmp2 = (ro * (sd * sd) - bxsq) * ddi;
      rsd = ro * sd * N::rcp(sdm);
    }
    rost[s] = mx * rsd - mn * ro;
    const T vxst = mx * sm - mn * vx;
    rxst[s] = rost[s] * vxst;
    vyst[s] = mx * (vy - by * tmp) - mn * vy;
    ryst[s] = rost[s] * vyst[s];
    vzst[s] = mx * (vz - bz * tmp) - mn * vz;
    rzst[s] = rost[s] * vzst[s];
    byst[s] = mx * (by * tmp2) - mn * by;
    bzst[s] = mx * (bz * tmp2) - mn * bz;
    vdbst[s] = vxst * bxs + vyst[s] * byst[s] + vzst[s] * bzst[s];
    const T num = sd * ee - pt * vx + ptst * sm + bxs * (vx * bxs + vy * by + vz * bz - vdbst[s]);
    if constexpr (E) esd = num / sdm;
    else esd = num * N::rcp(sdm);
    eest[s] = mx * esd - mn * ee;
  }
  // double-star states (:347-414)
  const T sqrtrol = fsqrt(rost[0]), sqrtror = fsqrt(rost[1]);
  T slst, srst;
  if constexpr (E) {
    slst = sm - fabs_(bxs) / sqrtrol;
    srst = sm + fabs_(bxs) / sqrtror;
  } else {
    slst = sm - fabs_(bxs) * N::rcp(sqrtrol);
    srst = sm + fabs_(bxs) * N::rcp(sqrtror);
  }
  T ryd[2], rzd[2], byd, bzd, eed[2];
  if (!SL && bxv == 0.0) {
    ryd[0] = ryst[0]; ryd[1] = ryst[1];
    rzd[0] = rzst[0]; rzd[1] = rzst[1];
    eed[0] = eest[0]; eed[1] = eest[1];
    byd = byst[0];  // unused: the flux takes byst of each side below
    bzd = bzst[0];
  } else {
    const T invsumro = N::rcp(sqrtrol + sqrtror);
    const T signbx = fsign_(T(1.0), bxs);
    const T vyd = invsumro * (sqrtrol * vyst[0] + sqrtror * vyst[1] + signbx * (byst[1] - byst[0]));
    ryd[0] = rost[0] * vyd;
    ryd[1] = rost[1] * vyd;
    const T vzd = invsumro * (sqrtrol * vzst[0] + sqrtror * vzst[1] + signbx * (bzst[1] - bzst[0]));
    rzd[0] = rost[0] * vzd;
    rzd[1] = rost[1] * vzd;
    byd = invsumro * (sqrtrol * byst[1] + sqrtror * byst[0] +
                      signbx * sqrtrol * sqrtror * (vyst[1] - vyst[0]));
    bzd = invsumro * (sqrtrol * bzst[1] + sqrtror * bzst[0] +
                      signbx * sqrtrol * sqrtror * (vzst[1] - vzst[0]));
    const T temp = sm * bxs + vyd * byd + vzd * bzd;
    eed[0] = eest[0] - sqrtrol * signbx * (vdbst[0] - temp);
    eed[1] = eest[1] + sqrtror * signbx * (vdbst[1] - temp);
  }
  const bool zb = bxv == 0.0;
  // flux (:446-480)
  if constexpr (SL) {
    // one side s and f = F_s + c1 (U*_s - U_s) + c2 (U**_s - U*_s): c1 = sl or
    // sr, c2 = slst or srst in the inner fans, 0 in the outer ones (the
    // branches of the reference, rearranged); the supersonic cases select the
    // physical flux.  With bx = 0 the double-star state is the star state.
    const bool right = !N::ge0(sm), sup = N::ge0(sl) || N::le0(sr);
    if (ill != nullptr) *ill = illv && !sup;
    const bool supr = N::le0(sr) && !N::ge0(sl);
    const bool inner = right ? N::gt0(srst) : !N::ge0(slst);
    const T c1 = right ? sr : sl;
    const T c2 = inner ? (right ? srst : slst) : T(0.0f);
    auto put = [&](int v, T fl, T fr, T ul, T ur, T usv, T udv) {
      const T fv = (right ? fr : fl) + c1 * (usv - (right ? ur : ul)) + c2 * (udv - usv);
      f[v] = N::out(sup ? (supr ? fr : fl) : fv);
    };
    // the star and double-star values of side s, picked by selects (an index
    // into the two-element arrays would place them in local memory)
    auto pick = [&](const T *x) { return right ? x[1] : x[0]; };
    const T ro_s = pick(rost), ee_s = pick(eest), ry_s = pick(ryst), rz_s = pick(rzst);
    const T by_s = pick(byst), bz_s = pick(bzst);
    put(0, frol, fror, rol, ror, ro_s, ro_s);
    put(1, feel, feer, eel, eer, ee_s, zb ? ee_s : pick(eed));
    put(2, frxl, frxr, rxl, rxr, pick(rxst), pick(rxst));
    put(3, fryl, fryr, ryl, ryr, ry_s, zb ? ry_s : pick(ryd));
    put(4, frzl, frzr, rzl, rzr, rz_s, zb ? rz_s : pick(rzd));
    put(5, fbyl, fbyr, byl, byr, by_s, zb ? by_s : byd);
    put(6, fbzl, fbzr, bzl, bzr, bz_s, zb ? bz_s : bzd);
  } else if (N::ge0(slst)) {
    f[0] = N::out(frol + sl * (rost[0] - rol));
    f[2] = N::out(frxl + sl * (rxst[0] - rxl));
    f[3] = N::out(fryl + sl * (ryst[0] - ryl));
    f[4] = N::out(frzl + sl * (rzst[0] - rzl));
    f[1] = N::out(feel + sl * (eest[0] - eel));
    f[5] = N::out(fbyl + sl * (byst[0] - byl));
    f[6] = N::out(fbzl + sl * (bzst[0] - bzl));
  } else if (N::ge0(sm)) {
    const T temp = slst - sl;
    const T byd0 = zb ? byst[0] : byd, bzd0 = zb ? bzst[0] : bzd;
    f[0] = N::out(frol - sl * rol - temp * rost[0] + slst * rost[0]);
    f[2] = N::out(frxl - sl * rxl - temp * rxst[0] + slst * rxst[0]);
    f[3] = N::out(fryl - sl * ryl - temp * ryst[0] + slst * ryd[0]);
    f[4] = N::out(frzl - sl * rzl - temp * rzst[0] + slst * rzd[0]);
    f[1] = N::out(feel - sl * eel - temp * eest[0] + slst * eed[0]);
    f[5] = N::out(fbyl - sl * byl - temp * byst[0] + slst * byd0);
    f[6] = N::out(fbzl - sl * bzl - temp * bzst[0] + slst * bzd0);
  } else if (N::gt0(srst)) {
    const T temp = srst - sr;
    const T byd1 = zb ? byst[1] : byd, bzd1 = zb ? bzst[1] : bzd;
    f[0] = N::out(fror - sr * ror - temp * rost[1] + srst * rost[1]);
    f[2] = N::out(frxr - sr * rxr - temp * rxst[1] + srst * rxst[1]);
    f[3] = N::out(fryr - sr * ryr - temp * ryst[1] + srst * ryd[1]);
    f[4] = N::out(frzr - sr * rzr - temp * rzst[1] + srst * rzd[1]);
    f[1] = N::out(feer - sr * eer - temp * eest[1] + srst * eed[1]);
    f[5] = N::out(fbyr - sr * byr - temp * byst[1] + srst * byd1);
    f[6] = N::out(fbzr - sr * bzr - temp * bzst[1] + srst * bzd1);
  } else {
    f[0] = N::out(fror + sr * (rost[1] - ror));
    f[2] = N::out(frxr + sr * (rxst[1] - rxr));
    f[3] = N::out(fryr + sr * (ryst[1] - ryr));
    f[4] = N::out(frzr + sr * (rzst[1] - rzr));
    f[1] = N::out(feer + sr * (eest[1] - eer));
    f[5] = N::out(fbyr + sr * (byst[1] - byr));
    f[6] = N::out(fbzr + sr * (bzst[1] - bzr));
  }
}

// The fast policy's flux.  The FP64 pipe bounds the HLLD step (two lanes per SM
// and clock), so the flux is written for the fewest FP64 instructions:
//  - the face lies in one fan, and its side is known from S_L, S_R and S_M:
//    the physical flux, the energies and the star state are formed for that
//    side s alone (selects of the inputs, no divergence), the star state of the
//    other side only where the face lies between the Alfven waves, whose states
//    mix both sides;
//  - f = F_s + c1 (U*_s - U_s) + c2 (U**_s - U*_s), c1 = S_s, c2 = S*_s between
//    the Alfven waves and 0 outside: the reference's branches with their
//    terms collected, differences of states in place of differences of products;
//  - the total pressure between the fast waves from side s,
//    p_s + ro_s (S_s - v_s)(S_M - v_s) (Miyoshi & Kusano 2005, eq. 23 with the
//    momentum jump), equal to the reference's symmetric form;
//  - the larger fast speed by comparing the squares: one outer root, not two;
//    the inner root's (g + B^2)^2 - 4 g Bx^2, g = gm p, as the sum of squares
//    (g - Bx^2)^2 + Bt^2 (2 (g + Bx^2) + Bt^2), which no rounding makes negative;
//  - reciprocals, roots and comparisons of fd64.cuh.
// Measured on the 128^3 box with an oblique field (134^3 cells): 6.6 ms a step (6.3 with isum.cuh)
// where the reference's branches with both sides formed took 12.3 ms.
// A star state within zfloor of its singular denominator keeps the side's own
// state (hlld_flux.f90:281-342), by selects.
__device__ __forceinline__ void hlld_flux_fast(const HlldK &K, const double *L,
                                               const double *R, double bx, double *f) {
  const double bb = bx * bx;
  const double btl = fma(L[6], L[6], L[7] * L[7]), btr = fma(R[6], R[6], R[7] * R[7]);
  const double b2l = bb + btl, b2r = bb + btr;  // twice the magnetic pressures
  // fast speeds
  const double gl = K.gm * L[1], gr = K.gm * R[1];
  const double hl = gl + bb, hr = gr + bb, el = gl - bb, er = gr - bb;
  const double kl = hl + btl, kr = hr + btr;
  const double c2l = (kl + fd::sqrt_(fma(btl, kl + hl, el * el))) * fd::rcp(L[0]);
  const double c2r = (kr + fd::sqrt_(fma(btr, kr + hr, er * er))) * fd::rcp(R[0]);
  // max(cfl, cfr), min(vl, vr) and max(vl, vr) as Fortran's on NaNs: the right one unless
  // the left one compares.  Unsigned, a negative square or a NaN is beyond infinity.
  // (On the upper words: an operation gives quiet NaNs, above 0x7ff00000.)
  auto up = [](double x) { return (unsigned)__double2hiint(x); };
  const bool cl = up(c2l) <= 0x7ff00000u && (unsigned long long)__double_as_longlong(c2l) >
                                                (unsigned long long)__double_as_longlong(c2r);
  const double cf = fd::sqrt_(0.5 * (cl ? c2l : c2r));
  const bool num = max(up(L[2]) & 0x7fffffffu, up(R[2]) & 0x7fffffffu) <= 0x7ff00000u;
  const bool lt = fd::lt(L[2], R[2]);
  const double sl = (lt && num ? L[2] : R[2]) - cf, sr = (lt || !num ? R[2] : L[2]) + cf;
  // contact speed
  const double dl = sl - L[2], dr = sr - R[2];
  const double ml = dl * L[0], mr = dr * R[0];
  const double ptl = fma(0.5, b2l, L[1]), ptr = fma(0.5, b2r, R[1]);
  const double sm = (fma(mr, R[2], -ml * L[2]) + (ptl - ptr)) * fd::rcp(mr - ml);
  // the side of the face and whether it is supersonic
  // (neither for a NaN, which the star states then carry into every component)
  const bool supl = up(sl) <= 0x7ff00000u;
  const bool supr = !supl && (up(sr) - 0x80000000u <= 0x7ff00000u || sr == 0.0);
  const bool right = !supl && (supr || __double2hiint(sm) < 0);
  const double ro = right ? R[0] : L[0], pr = right ? R[1] : L[1];
  const double vx = right ? R[2] : L[2], vy = right ? R[3] : L[3], vz = right ? R[4] : L[4];
  const double by = right ? R[6] : L[6], bz = right ? R[7] : L[7];
  const double pt = right ? ptr : ptl, b2 = right ? b2r : b2l;
  const double sd = right ? dr : dl, m = right ? mr : ml, sp = right ? sr : sl;
  // physical flux and conserved state of the side
  const double rx = ro * vx, ry = ro * vy, rz = ro * vz;
  const double ek = fma(rx, vx, fma(ry, vy, rz * vz));
  const double ee = fma(pr, K.gm1i, 0.5 * (ek + b2));
  const double vb = fma(vx, bx, fma(vy, by, vz * bz));
  double fro = rx;
  double frx = fma(rx, vx, pt - bb);
  double fry = fma(rx, vy, -bx * by);
  double frz = fma(rx, vz, -bx * bz);
  double fee = fma(vx, ee + pt, -bx * vb);
  double fby = fma(by, vx, -bx * vy);
  double fbz = fma(bz, vx, -bx * vz);
  if (!(supl || supr)) {
    // star state of one side: its density, transverse velocity and field
    auto star = [&](double ro_, double vx_, double vy_, double vz_, double by_, double bz_,
                    double sd_, double m_, double sdm, double rsdm, double &ros, double &vys,
                    double &vzs, double &bys, double &bzs) {
      const double t = fma(m_, sdm, -bb);
      const bool deg = fd::ltp(fd::abs_(t), K.zfloor);
      const double di = fd::rcp(deg ? 1.0 : t);
      const double a1 = bx * (sm - vx_) * di, a2 = fma(m_, sd_, -bb) * di;
      ros = deg ? ro_ : m_ * rsdm;
      vys = deg ? vy_ : fma(-by_, a1, vy_);
      vzs = deg ? vz_ : fma(-bz_, a1, vz_);
      bys = deg ? by_ : by_ * a2;
      bzs = deg ? bz_ : bz_ * a2;
      return deg;
    };
    const double sdm = sp - sm, rsdm = fd::rcp(sdm);
    double ros, vys, vzs, bys, bzs;
    const bool deg = star(ro, vx, vy, vz, by, bz, sd, m, sdm, rsdm, ros, vys, vzs, bys, bzs);
    const double vxs = deg ? vx : sm;
    const double vbs = fma(vxs, bx, fma(vys, bys, vzs * bzs));
    const double pts = fma(m, sm - vx, pt);
    const double es = fma(sd, ee, fma(-pt, vx, fma(pts, sm, bx * (vb - vbs)))) * rsdm;
    const double ees = deg ? ee : es;
    double rs, irs;
    fd::sqrt_rsqrt(ros, rs, irs);
    const double ca = fd::abs_(bx) * irs;
    const double sa = right ? sm + ca : sm - ca;  // the side's Alfven wave
    const double rys = ros * vys, rzs = ros * vzs;
    fro = fma(sp, ros - ro, fro);
    frx = fma(sp, fma(ros, vxs, -rx), frx);
    fry = fma(sp, rys - ry, fry);
    frz = fma(sp, rzs - rz, frz);
    fee = fma(sp, ees - ee, fee);
    fby = fma(sp, bys - by, fby);
    fbz = fma(sp, bzs - bz, fbz);
    // between the Alfven waves (with bx = 0 they are the contact)
    const int sah = __double2hiint(sa);
    const bool inner = right ? sah >= 0 && (sah | __double2loint(sa)) != 0 : sah < 0;
    if (inner) {
      const double sdo = right ? dl : dr, mo = right ? ml : mr;
      const double sdmo = (right ? sl : sr) - sm;
      double roo, vyo, vzo, byo, bzo;
      star(right ? L[0] : R[0], right ? L[2] : R[2], right ? L[3] : R[3],
           right ? L[4] : R[4], right ? L[6] : R[6], right ? L[7] : R[7], sdo, mo, sdmo,
           fd::rcp(sdmo), roo, vyo, vzo, byo, bzo);
      const double qo = fd::sqrt_(roo);
      const double iv = fd::rcp(rs + qo), qq = rs * qo;
      // sign(bx) with the sides exchanged for the right one
      const double flip =
          __hiloint2double(__double2hiint(bx) ^ (right ? (int)0x80000000 : 0), 0);
      const double vyd = iv * (fma(rs, vys, qo * vyo) + fd::mul_sign(byo - bys, flip));
      const double vzd = iv * (fma(rs, vzs, qo * vzo) + fd::mul_sign(bzo - bzs, flip));
      const double byd = iv * fma(rs, byo, fma(qo, bys, qq * fd::mul_sign(vyo - vys, flip)));
      const double bzd = iv * fma(rs, bzo, fma(qo, bzs, qq * fd::mul_sign(vzo - vzs, flip)));
      const double vbd = fma(sm, bx, fma(vyd, byd, vzd * bzd));
      fry = fma(sa, fma(ros, vyd, -rys), fry);
      frz = fma(sa, fma(ros, vzd, -rzs), frz);
      fee = fma(sa, rs * fd::mul_sign(vbd - vbs, flip), fee);
      fby = fma(sa, byd - bys, fby);
      fbz = fma(sa, bzd - bzs, fbz);
    }
  }
  f[0] = fro;
  f[1] = fee;
  f[2] = frx;
  f[3] = fry;
  f[4] = frz;
  f[5] = fby;
  f[6] = fbz;
}

template <bool E>
__device__ __forceinline__ void hlld_flux(const HlldK &K, const double *L,
                                          const double *R, double bxv,
                                          double *f) {
  if constexpr (E) hlld_flux_t<F<true>>(K, L, R, bxv, f);
  else hlld_flux_fast(K, L, R, bxv, f);
}

}  // namespace cans
