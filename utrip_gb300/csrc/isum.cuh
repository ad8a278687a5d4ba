// Stencil sums of doubles on the integer pipe (sm_103a).
//
// GB300 executes two FP64 lanes per SM and clock: an FP64 addition takes that
// pipe as long as 64 issue slots, while the integer pipes of a kernel bound by
// it stand idle.  A sum of a few doubles is formed here as an integer: the
// significands are aligned to the largest exponent of the operands, negated
// where the sign says so, added as 64-bit integers, and the sum is normalised and
// rounded once.  No FP64 instruction is used.
//
// Accuracy: the aligned operands keep G bits below the last place of the largest
// one (8 for a sum of four, 7 for one of up to eight: what 64 bits leave), so an
// operand up to 2^G smaller enters exactly and a smaller one is truncated below
// 2^-(52+G) of the largest one's power of two.  A sum of four is within 2^-58 of its
// largest operand before its one rounding (to nearest even), where the FP64
// chain rounds each partial sum to 2^-53; sums that cancel to zero are zero.
//
// The operands may be zero.  Where the largest exponent is not within the range
// of `special` (subnormals and their neighbourhood, the largest numbers,
// infinities, NaN) the caller forms its sums in FP64 instead.
#pragma once
#include <cuda_runtime.h>

namespace cans {
namespace isum {

// exponent field of x, in place
__device__ __forceinline__ unsigned expo(double x) {
  return (unsigned)__double2hiint(x) & 0x7ff00000u;
}
// no sum of operands with largest exponent E (in place) may be formed here
__device__ __forceinline__ bool special(unsigned E) {
  return E - 0x04000000u >= 0x7b800000u && E != 0u;  // fields 1 .. 63, 2040 .. 2047
}

// the significand bits of x (written on its words: the compiler turns a test of the
// whole against zero into an FP64 comparison)
__device__ __forceinline__ unsigned bits(double x) {
  return ((unsigned)__double2hiint(x) & 0x7fffffffu) | (unsigned)__double2loint(x);
}

// |x| 2^(e - expo(x)) as an integer in units of 2^-(52+G) of the power of two of
// exponent E >= e: below 2^(53+G).  E is not `special`, so it is 0 or the fields are
// 64 and up, and where e is 0 (zeros; subnormals beside a normal E) the hidden bit
// set here is shifted out with the rest.
template <int G> __device__ __forceinline__ unsigned long long mag(double x, unsigned e,
                                                                   unsigned E) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  unsigned long long m =
      (unsigned long long)(__funnelshift_l(lo, hi, 11) | 0x80000000u) << 32 | lo << 11;
  const unsigned top = max(E, 0x04000000u) + ((unsigned)(11 - G) << 20);
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"((top - e) >> 20));  // shifts beyond 63 give 0
  return m;
}
// the same with x's sign
template <int G> __device__ __forceinline__ long long at(double x, unsigned e, unsigned E) {
  const long long s = __double2hiint(x) >> 31;
  return ((long long)mag<G>(x, e, E) ^ s) - s;
}

// the double nearest to s in the units of E (ties to even)
template <int G> __device__ __forceinline__ double out(long long s, unsigned E) {
  const int sh = (int)(s >> 32);
  const long long sg = sh >> 31;
  unsigned long long m = (unsigned long long)((s ^ sg) - sg);
  const int lz = __clzll((long long)m);
  asm("shl.b64 %0, %0, %1;" : "+l"(m) : "r"(lz));
  const unsigned lo = (unsigned)m;
  const unsigned up = ((lo & 0x7ffu) + 0x3ffu + ((lo >> 11) & 1u)) >> 11;
  // a leading bit at 52 + G is the exponent E; the hidden bit adds one to the
  // field, and so does a carry of the rounding
  const unsigned f = m ? E + ((unsigned)(10 - G - lz) << 20) : 0u;
  const unsigned long long b = (m >> 11) + up;
  return __hiloint2double((int)((unsigned)(b >> 32) + f) | (sh & (int)0x80000000), (int)b);
}

// four operands aligned to their largest exponent
struct Four {
  long long a, b, c, d;
  unsigned E;
};
__device__ __forceinline__ Four four(double a, double b, double c, double d, bool &sp) {
  const unsigned E = max(max(expo(a), expo(b)), max(expo(c), expo(d)));
  sp |= special(E);
  if (E == 0u) sp |= (bits(a) | bits(b) | bits(c) | bits(d)) != 0u;  // a subnormal
  return {at<8>(a, expo(a), E), at<8>(b, expo(b), E), at<8>(c, expo(c), E),
          at<8>(d, expo(d), E), E};
}

// exponent field of 4 x
__device__ __forceinline__ unsigned expo4(double x) {
  const unsigned e = expo(x);
  return e + min(e, 0x200000u);
}
// 2^-32 m e for an integer m and a small factor e: |e| <= 2^-4, |m| < 2^61
__device__ __forceinline__ float scaled(long long m, float e) {
  return __fmul_rn(__int2float_rn((int)(m >> 32)), e);
}
// (b - a) (1 + e0 2^-32) + (d - c) (1 + e1 2^-32) + 4 (g - f), |e0|, |e1| <= 2^-4: two
// corner differences with weights near one and a central difference.  The
// correction is 2^-36 of the differences and is taken to 24 bits: 2^-60 of them.
__device__ __forceinline__ double diff6(double a, double b, double c, double d, double f,
                                        double g, float e0, float e1, bool &sp) {
  const unsigned ea = expo(a), eb = expo(b), ec = expo(c), ed = expo(d);
  const unsigned ef = expo4(f), eg = expo4(g);
  const unsigned E = max(max(max(ea, eb), max(ec, ed)), max(ef, eg));
  sp |= special(E);
  if (E == 0u) sp |= (bits(a) | bits(b) | bits(c) | bits(d) | bits(f) | bits(g)) != 0u;
  const long long x = at<7>(b, eb, E) - at<7>(a, ea, E);
  const long long y = at<7>(d, ed, E) - at<7>(c, ec, E);
  const long long z = at<7>(g, eg, E) - at<7>(f, ef, E);
  const int k = __float2int_rn(__fadd_rn(scaled(x, e0), scaled(y, e1)));
  return out<7>(x + y + z + (long long)k, E);
}

// exponent field of 16 x
__device__ __forceinline__ unsigned expo16(double x) {
  const unsigned e = expo(x);
  return e + min(e, 0x400000u);
}

// Sums over two planes of four cells each: l and u point at the lower left cell of
// the lower and the upper plane, a row is CX doubles.
// the sum of the eight, and the differences along x, y and from lower to upper
enum Form { kSum, kDx, kDy, kDz };
template <int CX, int F>
__device__ __forceinline__ double eight(const double *l, const double *u, bool &sp) {
  const double v[8] = {l[0], l[1], l[CX], l[CX + 1], u[0], u[1], u[CX], u[CX + 1]};
  unsigned e[8], E = 0u, any = 0u;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    e[i] = expo(v[i]);
    E = max(E, e[i]);
  }
  sp |= special(E);
  if (E == 0u) {
#pragma unroll
    for (int i = 0; i < 8; i++) any |= bits(v[i]);
    sp |= any != 0u;
  }
  long long s = 0;
  int n = 0;  // of negative terms: -m is ~m + 1
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const bool neg = F == kDx ? !(i & 1) : F == kDy ? !(i & 2) : F == kDz ? i < 4 : false;
    const int g = neg ? ~(__double2hiint(v[i]) >> 31) : __double2hiint(v[i]) >> 31;
    s += (long long)mag<7>(v[i], e[i], E) ^ (long long)g;
    n -= g;
  }
  return out<7>(s + n, E);
}

// The part of a direction of a cell's change that two corner planes and the central
// difference give, on axes whose weights are one half up to 2^-32 e:
//   gu   (b - a) (1 + e0) + (d - c) (1 + e1) of the upper corner plane
//   ret  gl (1 + ez0) + gu (1 + ez1) + 16 (g - f), gl being the lower plane's gu
__device__ __forceinline__ double diff_planes(double a, double b, double c, double d, double gl,
                                              double f, double g, float e0, float e1, float ez0,
                                              float ez1, double &gu, bool &sp) {
  const unsigned ea = expo(a), eb = expo(b), ec = expo(c), ed = expo(d), el = expo(gl);
  const unsigned ef = expo16(f), eg = expo16(g);
  const unsigned E = max(max(max(ea, eb), max(ec, ed)), max(max(ef, eg), el));
  sp |= special(E);
  if (E == 0u) sp |= (bits(a) | bits(b) | bits(c) | bits(d) | bits(f) | bits(g) | bits(gl)) != 0u;
  const long long x = at<6>(b, eb, E) - at<6>(a, ea, E);
  const long long y = at<6>(d, ed, E) - at<6>(c, ec, E);
  const long long z = at<6>(g, eg, E) - at<6>(f, ef, E);
  const long long l = at<6>(gl, el, E);
  const long long up = x + y + __float2int_rn(__fadd_rn(scaled(x, e0), scaled(y, e1)));
  gu = out<6>(up, E);
  return out<6>(l + up + z + __float2int_rn(__fadd_rn(scaled(l, ez0), scaled(up, ez1))), E);
}
// The z flux of a face, 16 times twice its value: the four corner values with
// weights (1 + ex + ey), 16 (f + g), and the viscosity's w; neg: less the former
// two.  pu is that of this face, the result its difference from the lower one pl.
__device__ __forceinline__ double face_planes(double a, double b, double c, double d, double f,
                                              double g, double w, double pl, bool neg, float ex0,
                                              float ex1, float ey0, float ey1, double &pu,
                                              bool &sp) {
  const unsigned ea = expo(a), eb = expo(b), ec = expo(c), ed = expo(d), el = expo(pl);
  const unsigned ef = expo16(f), eg = expo16(g), ew = expo(w);
  const unsigned E =
      max(max(max(ea, eb), max(ec, ed)), max(max(ef, eg), max(el, ew)));
  sp |= special(E);
  if (E == 0u)
    sp |= (bits(a) | bits(b) | bits(c) | bits(d) | bits(f) | bits(g) | bits(pl) | bits(w)) != 0u;
  const long long A = at<6>(a, ea, E), B = at<6>(b, eb, E), C = at<6>(c, ec, E);
  const long long D = at<6>(d, ed, E);
  const float k = __fadd_rn(__fadd_rn(scaled(A + B, ey0), scaled(C + D, ey1)),
                            __fadd_rn(scaled(A + C, ex0), scaled(B + D, ex1)));
  long long s = (A + B) + (C + D) + __float2int_rn(k) + (at<6>(f, ef, E) + at<6>(g, eg, E));
  s = (neg ? -s : s) + at<6>(w, ew, E);
  pu = out<6>(s, E);
  return out<6>(s - at<6>(pl, el, E), E);
}

// x + y rounded to nearest, the FP64 addition's result to the bit: the smaller operand
// is aligned to the larger with ten guard bits and what falls off them is kept as
// one sticky bit.  Some fifty integer instructions.  y's upper word is xored with flip
// (0x80000000: x - y).
constexpr unsigned kMinus = 0x80000000u;
__device__ __forceinline__ double add2(double x, double y, bool &sp, unsigned flip = 0u) {
  const unsigned hx = (unsigned)__double2hiint(x), lx = (unsigned)__double2loint(x);
  const unsigned hy = (unsigned)__double2hiint(y) ^ flip, ly = (unsigned)__double2loint(y);
  const bool sw = ((unsigned long long)(hy & 0x7fffffffu) << 32 | ly) >
                  ((unsigned long long)(hx & 0x7fffffffu) << 32 | lx);
  const unsigned hg = sw ? hy : hx, lg = sw ? ly : lx, hs = sw ? hx : hy, ls = sw ? lx : ly;
  const unsigned E = hg & 0x7ff00000u;
  sp |= special(E);
  if (E == 0u) sp |= ((hg & 0x7fffffffu) | lg) != 0u;
  auto sig = [](unsigned hi, unsigned lo) {  // the hidden bit at 62
    return (unsigned long long)((__funnelshift_l(lo, hi, 10) & 0x3fffffffu) | 0x40000000u) << 32 |
           lo << 10;
  };
  const unsigned sh = (E - (hs & 0x7ff00000u)) >> 20;
  const unsigned long long small = sig(hs, ls);
  unsigned long long t = small, back;
  asm("shr.u64 %0, %0, %1;" : "+l"(t) : "r"(sh));
  asm("shl.b64 %0, %1, %2;" : "=l"(back) : "l"(t), "r"(sh));
  t |= back != small ? 1ull : 0ull;
  const long long opp = (long long)((int)(hg ^ hs) >> 31);
  unsigned long long m = sig(hg, lg) + (unsigned long long)(((long long)t ^ opp) - opp);
  m = E != 0u ? m : 0ull;
  const int lz = __clzll((long long)m);
  asm("shl.b64 %0, %0, %1;" : "+l"(m) : "r"(lz));
  const unsigned lo = (unsigned)m;
  const unsigned up = ((lo & 0x7ffu) + 0x3ffu + ((lo >> 11) & 1u)) >> 11;
  const unsigned f = m ? E - ((unsigned)lz << 20) : 0u, sg = m ? hg : hg & hs;
  const unsigned long long b = (m >> 11) + up;
  return __hiloint2double((int)(((unsigned)(b >> 32) + f) | (sg & 0x80000000u)), (int)b);
}
static __device__ __noinline__ double sub_fp64(double x, double y) { return x - y; }
// x - y, the FP64 subtraction's result
__device__ __forceinline__ double sub_rn(double x, double y) {
  bool sp = false;
  const double r = add2(x, y, sp, kMinus);
  return sp ? sub_fp64(x, y) : r;
}
// x / 2 of a normal number or zero
__device__ __forceinline__ double half_of(double x, bool &sp) {
  const unsigned e = expo(x);
  if (e <= 0x100000u) sp |= bits(x) != 0u;
  return __hiloint2double(__double2hiint(x) - (int)min(e, 0x100000u), __double2loint(x));
}

// The minmod face states between cells 0 and 1 of a line of four: d0 + minmod(d0 - dm,
// d1 - d0) / 2 and d1 - minmod(d2 - d1, d1 - d0) / 2 (up to the sign of a zero
// minmod), bit for bit what five FP64 instructions give.
// Measured on the 128^3 boxes: Roe-MUSCL 9.0 -> 8.6 ms a step, HLLD 6.5 -> 6.2; with
// sub_rn in the updates 8.5 (the sums inside the Roe flux too: 8.9, as their
// integer temporaries halve the warps in flight).
__device__ __forceinline__ double minmod(double a, double b) {
  const long long x = __double_as_longlong(a) ^ __double_as_longlong(b);
  const unsigned long long p = (unsigned long long)__double_as_longlong(a) & 0x7fffffffffffffffull;
  const unsigned long long q = (unsigned long long)__double_as_longlong(b) & 0x7fffffffffffffffull;
  const unsigned long long m = p < q ? p : q;
  const unsigned long long s = (unsigned long long)__double_as_longlong(a) & 0x8000000000000000ull;
  return __longlong_as_double(x >= 0 ? (long long)(m | s) : 0ll);
}
static __device__ __noinline__ double2 muscl_fp64(double dm, double d0, double d1, double d2) {
  const double g = d1 - d0;
  return make_double2(fma(0.5, minmod(d0 - dm, g), d0), fma(-0.5, minmod(d2 - d1, g), d1));
}
__device__ __forceinline__ void muscl(double dm, double d0, double d1, double d2, double &wl,
                                      double &wr) {
  bool sp = false;
  const double g = add2(d1, d0, sp, kMinus);
  const double l = minmod(add2(d0, dm, sp, kMinus), g);
  const double r = minmod(add2(d2, d1, sp, kMinus), g);
  wl = add2(d0, half_of(l, sp), sp);
  wr = add2(d1, half_of(r, sp), sp, kMinus);
  if (sp) {
    const double2 w = muscl_fp64(dm, d0, d1, d2);
    wl = w.x;
    wr = w.y;
  }
}

}  // namespace isum
}  // namespace cans
