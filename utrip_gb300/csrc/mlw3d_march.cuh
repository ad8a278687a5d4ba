// The fields and the block layout that the marching 3-D mLW steps share: the fast
// policy's in FP64 (mlw3d_fast.cu) and the double-float one (mlw3d_df.cu).
#pragma once
#include <cuda_runtime.h>

namespace cans {
namespace {

// cell slots: conserved, fluxes (XY = fx(ry) = fy(rx), ...), E, velocities
enum {
  CRO, CEE, CRX, CBX, CRY, CRZ, CBY, CBZ,
  CFX, CFY, CFZ,                  // energy fluxes
  CXX, CYY, CZZ, CXY, CXZ, CYZ,   // momentum fluxes
  CEX, CEY, CEZ, CVX, CVY, CVZ, NCF
};
// corner slots, all eight times their value; the mass fluxes are the momenta
enum { KRX, KRY, KRZ, KFX, KFY, KFZ, KXX, KYY, KZZ, KXY, KXZ, KYZ, KEX, KEY, KEZ, NKF };
// what an interior column keeps of its lower corner plane: per variable the x and y
// differences (seven each) and the z face flux
constexpr int NRET = 22;

// The fields of variable v (cell slot v): its x, y, z fluxes at the cells and corners,
// -1 where it has none; their signs (of E in the induction equation); its retained x
// and y differences (a word of the column each, of one thread; -1 with the flux); its
// gravity source.  In constant memory: the loops over the
// variables stay rolled, so that their integer sums (some 600 instructions a pass)
// stay in the instruction cache.  The two halves of the variables have about the
// same number of sums (15 and 14 of the predictor, 11 and 10 of the corrector).
struct VarFields {
  signed char fx, kx, fy, ky, fz, kz, sx, sy, sz, rx, ry, g;
};
__constant__ VarFields kVar[8] = {
    {CRX, KRX, CRY, KRY, CRZ, KRZ, 1, 1, 1, 0, 0, -1},
    {CFX, KFX, CFY, KFY, CFZ, KFZ, 1, 1, 1, 1, 1, 0},
    {CXX, KXX, CXY, KXY, CXZ, KXZ, 1, 1, 1, 2, 2, 1},
    {-1, -1, CEZ, KEZ, CEY, KEY, 0, 1, -1, -1, 3, -1},
    {CXY, KXY, CYY, KYY, CYZ, KYZ, 1, 1, 1, 3, 4, 2},
    {CXZ, KXZ, CYZ, KYZ, CZZ, KZZ, 1, 1, 1, 4, 5, 3},
    {CEZ, KEZ, -1, -1, CEX, KEX, -1, 0, 1, 5, -1, -1},
    {CEY, KEY, CEX, KEX, -1, -1, 1, -1, 0, 6, 6, -1}};

template <int TX, int TY, bool G> struct T3F {
  static constexpr int CX = TX + 2, CY = TY + 2, NC = CX * CY;
  static constexpr int KX = TX + 1, KY = TY + 1, NK = KX * KY;
  static constexpr int NI = TX * TY, NQX = KX * TY, NQY = TX * KY;
  static constexpr int W = 32, NKW = (NK + W - 1) / W * W;  // whole warps of corners
  static constexpr int NT = 2 * NKW;                        // two threads a corner
  static constexpr int T0 = NT - (NC + W - 1) / W * W;      // the first of the cells' threads
  static_assert(NI % W == 0 && T0 >= NI && NT >= 2 * NI && NKW >= NQX && NKW >= NQY, "");
  static constexpr int NR = NRET + (G ? 4 : 0);
  static constexpr size_t smem_bytes =
      sizeof(double) * (2 * (size_t)NCF * NC + (size_t)NKF * NK + NQX + NQY +
                        (size_t)(NR + 4) * NI + 34 + (G ? 2 * 4 * (size_t)NC + 4 * (size_t)NK : 0));
};

}  // namespace
}  // namespace cans
