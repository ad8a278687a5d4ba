// The 2-D mLW steps of the fast policy (FP64): mlw_m3 and mlw_m
// (cans2d/hdmlw/mlw_m3.f, mlw_m.f), with gravity (mlw_m3_g.f, mlw_m_g.f) and
// resistivity (mlw_m3_e.f, mlw_m_e.f, and both), as instances of the y-marching
// block of mlw2d_march.cuh.
#include "mlw2d_march.cuh"

namespace cans {

namespace {

template <bool M3, bool G, bool R>
cudaError_t pick(int tile, const MarchArgs &m, const Axis &ax, const Axis &ay, const Phys &ph,
                 Ctl *ctl, cudaStream_t s) {
  return launch_march<F64N, kFastCH, M3, G, R>(m, ax, ay, ph, ctl, s, (tile & 1) != 0);
}
template <bool M3>
cudaError_t pick_terms(int tile, const MarchArgs &m, const Axis &ax, const Axis &ay,
                       const Phys &ph, Ctl *ctl, cudaStream_t s) {
  if (m.grav && m.res) return pick<M3, true, true>(tile, m, ax, ay, ph, ctl, s);
  if (m.grav) return pick<M3, true, false>(tile, m, ax, ay, ph, ctl, s);
  if (m.res) return pick<M3, false, true>(tile, m, ax, ay, ph, ctl, s);
  return pick<M3, false, false>(tile, m, ax, ay, ph, ctl, s);
}

}  // namespace

// Even tiles balance the segments by pairs of blocks an SM, odd ones by waves of
// resident blocks; the results are the same bits.
cudaError_t launch_mlw2d_fast(int solver, int tile, const double *A, double *B, int ix, int jx,
                              const Axis &ax, const Axis &ay, const Phys &ph,
                              const double *grav, const double *res, double dt, Ctl *ctl,
                              Box3 box, cudaStream_t s) {
  if (ix < 3 || jx < 3) return cudaErrorInvalidValue;
  MarchArgs m{};
  m.A = A;
  m.B = B;
  m.ix = ix;
  m.jx = jx;
  m.dt = dt;
  m.box = box;
  m.grav = grav;
  m.res = res;
  return solver == 1 ? pick_terms<true>(tile, m, ax, ay, ph, ctl, s)
                     : pick_terms<false>(tile, m, ax, ay, ph, ctl, s);
}

// mlw_m3 with the viscosity's branch recorded (mode 1) or held (mode 2).
cudaError_t launch_mlw2d_av_fast(int mode, const double *A, double *B, int ix, int jx,
                                 const Axis &ax, const Axis &ay, const Phys &ph, double dt,
                                 unsigned char *avb, unsigned long long *nflip,
                                 cudaStream_t s) {
  MarchArgs m{};
  m.A = A;
  m.B = B;
  m.ix = ix;
  m.jx = jx;
  m.dt = dt;
  m.avb = avb;
  m.nflip = nflip;
  return mode == 1 ? launch_march<F64N, kFastCH, true, false, false, 1>(m, ax, ay, ph, nullptr, s)
                   : launch_march<F64N, kFastCH, true, false, false, 2>(m, ax, ay, ph, nullptr, s);
}

}  // namespace cans
