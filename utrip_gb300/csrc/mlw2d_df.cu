// The 2-D mLW step mlw_m3 (cans2d/hdmlw/mlw_m3.f:64-374) in the double-float
// policy: the y-marching block of mlw2d_march.cuh with its arithmetic in
// double-float (df64.cuh) on the FP32 pipes, and the conserved variables
// accumulated in FP64 (u_new = u + du, du in double-float).
//
// Precision: 48-bit significands (2^-48 per conversion, a few 2^-48 per
// operation).  The run holds the fast policy's bar against the oracle (the
// tests hold it to a relative 1e-10 per variable after 100 steps); the exact
// policy remains the bit-for-bit path.
#include "mlw2d_march.cuh"

namespace cans {

// Chunks of 8 or 6 rows, segments balanced by pairs of blocks an SM or by waves of
// resident blocks (balance_seg, balance_seg_waves): every configuration gives
// the same bits.
int mlw2d_df_tile_count() { return 7; }

cudaError_t launch_mlw2d_df(int tile, const double *A, double *B, int ix, int jx,
                            const Axis &ax, const Axis &ay, const Phys &ph, double dt,
                            Ctl *ctl, Box3 box, cudaStream_t s) {
  if (ix < 3 || jx < 3) return cudaErrorInvalidValue;
  MarchArgs m{};
  m.A = A;
  m.B = B;
  m.ix = ix;
  m.jx = jx;
  m.dt = dt;
  m.box = box;
  switch (tile) {
    case 1: case 5: return launch_march<DFN, 6, true, false, false>(m, ax, ay, ph, ctl, s);
    case 2: case 6: return launch_march<DFN, 8, true, false, false>(m, ax, ay, ph, ctl, s, true);
    case 3: return launch_march<DFN, 6, true, false, false>(m, ax, ay, ph, ctl, s, true);
    default: return launch_march<DFN, 8, true, false, false>(m, ax, ay, ph, ctl, s);
  }
}

}  // namespace cans
