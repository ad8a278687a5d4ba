// Fused 2-D modified Lax-Wendroff step of the exact policy (sm_103a, FP64): the
// single-grid kernel; and the CFL kernels and the frame kernel of both policies.  The tile body itself
// (phases 1-3, one TX x TY tile) is in mlw2d_tile.cuh.
#include <cuda_runtime.h>

#include "bc_line.cuh"
#include "bcframe2d.cuh"
#include "cans_common.cuh"
#include "cans_internal.h"
#include "mlw2d_tile.cuh"

namespace cans {

// One tile per block.  With a control block the step takes dt and the
// buffers from it, does nothing once the run is done or paused, and reduces
// the CFL of the cells inside `box`.
template <bool M3, int TX, int TY, int RPT>
__global__ void __launch_bounds__(TX *TY / RPT, 1)
    k_mlw2d(const double *__restrict__ A, double *__restrict__ B, int ix,
            int jx, Axis ax, Axis ay, Phys ph, double dt_arg,
            Ctl *__restrict__ ctl, Box3 box) {
  extern __shared__ double smem[];
  double dt = dt_arg, safety = 0.0;
  unsigned long long *cfl = nullptr;
  if (ctl != nullptr) {
    if (ctl->done | ctl->pause) return;
    A = ctl->buf[ctl->cur];
    B = ctl->buf[ctl->cur ^ 1];
    dt = ctl->dt;
    safety = ctl->safety;
    cfl = &ctl->cfl_bits;
  }
  tile_step<M3, TX, TY, RPT>(A, B, ix, jx, ax, ay, ph, dt, safety, cfl, box,
                                blockIdx.x, blockIdx.y, gridDim.x, gridDim.y, smem,
                                nullptr, nullptr, ctl ? &ctl->nonfinite : nullptr);
}

// The mlw_m3 step with the artificial viscosity's branch recorded (AVF = 1)
// or held at the recorded one (AVF = 2): the forward of the adjoint's
// finite-difference check (see tile_step).  32 x 8 tiles, no control block.
template <int AVF>
__global__ void __launch_bounds__(128, 1)
    k_mlw2d_av(const double *__restrict__ A, double *__restrict__ B, int ix, int jx, Axis ax,
               Axis ay, Phys ph, double dt, unsigned char *avb, unsigned long long *nflip) {
  extern __shared__ double smem[];
  tile_step<true, 32, 8, 2, false, false, AVF>(
      A, B, ix, jx, ax, ay, ph, dt, 0.0, nullptr, Box3{}, blockIdx.x, blockIdx.y, gridDim.x,
      gridDim.y, smem, nullptr, nullptr, nullptr, avb, nflip);
}

cudaError_t launch_mlw2d_av(bool exact, int mode, const double *A, double *B, int ix, int jx,
                            const Axis &ax, const Axis &ay, const Phys &ph, double dt,
                            unsigned char *avb, unsigned long long *nflip, cudaStream_t s) {
  if (ix < 3 || jx < 3 || (mode != 1 && mode != 2) || !avb || (mode == 2 && !nflip))
    return cudaErrorInvalidValue;
  if (!exact)
    return launch_mlw2d_av_fast(mode, A, B, ix, jx, ax, ay, ph, dt, avb, nflip, s);
  using T = Tile<32, 8, true, 2>;
  auto k = mode == 1 ? k_mlw2d_av<1> : k_mlw2d_av<2>;
  cudaError_t e =
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem_bytes);
  if (e != cudaSuccess) return e;
  dim3 grid((ix - 2 + 31) / 32, (jx - 2 + 7) / 8);
  k<<<grid, T::NT, T::smem_bytes, s>>>(A, B, ix, jx, ax, ay, ph, dt, avb, nflip);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Tile configurations offered to the autotuner: (TX, TY).
namespace {
template <bool M3, int TX, int TY, int RPT = 2>
cudaError_t launch_tile(const double *A, double *B, int ix, int jx,
                        const Axis &ax, const Axis &ay, const Phys &ph,
                        double dt, Ctl *ctl, Box3 box, cudaStream_t s) {
  using T = Tile<TX, TY, M3, RPT>;
  static bool attr_set = false;  // per template instance
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(
        k_mlw2d<M3, TX, TY, RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
        (int)T::smem_bytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  dim3 grid((ix - 2 + TX - 1) / TX, (jx - 2 + TY - 1) / TY);
  k_mlw2d<M3, TX, TY, RPT><<<grid, T::NT, T::smem_bytes, s>>>(A, B, ix, jx, ax,
                                                                ay, ph, dt, ctl, box);
  count_launch();
  return cudaGetLastError();
}

template <bool M3>
cudaError_t launch_sel(int tile, const double *A, double *B, int ix, int jx,
                       const Axis &ax, const Axis &ay, const Phys &ph,
                       double dt, Ctl *ctl, Box3 box, cudaStream_t s) {
  // 32 x 9 and 32 x 10 give tile counts that fill whole waves of two blocks
  // per SM on grids where 32 x 8 leaves a partly empty last wave (512^2:
  // 1024 tiles = 3.4 waves of 304 blocks, 32 x 9: 912 = 3.0 waves)
  switch (tile) {
    case 1: return launch_tile<M3, 32, 8>(A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
    case 2: return launch_tile<M3, 16, 16>(A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
    case 3: return launch_tile<M3, 64, 8>(A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
    case 4: return launch_tile<M3, 32, 9, 1>(A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
    case 5: return launch_tile<M3, 32, 10>(A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
    default: return launch_tile<M3, 32, 16>(A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
  }
}
}  // namespace

// Tiles of the exact policy (6 and 7 stand for 32 x 9); the fast policy's are the
// marching block's (launch_mlw2d_fast).
int mlw2d_tile_count() { return 8; }

cudaError_t launch_mlw2d(int solver, bool exact, int tile, const double *A,
                         double *B, int ix, int jx, const Axis &ax,
                         const Axis &ay, const Phys &ph, double dt, Ctl *ctl,
                         Box3 box, cudaStream_t s) {
  if (ix < 3 || jx < 3) return cudaErrorInvalidValue;
  if (!exact)
    return launch_mlw2d_fast(solver, tile, A, B, ix, jx, ax, ay, ph, nullptr, nullptr, dt, ctl,
                             box, s);
  if (tile >= 6) tile = 4;
  return solver == 1 ? launch_sel<true>(tile, A, B, ix, jx, ax, ay, ph, dt, ctl, box, s)
                     : launch_sel<false>(tile, A, B, ix, jx, ax, ay, ph, dt, ctl, box, s);
}

// ---------------------------------------------------------------------------
// Standalone CFL over all cells (cfl_m3.f:46-65, cfl_m.f:46-65).
template <bool E, bool M3>
__global__ void k_cfl2d_full(const double *__restrict__ S, int ix, int jx,
                             Axis ax, Axis ay, Phys ph, double safety,
                             unsigned long long *out) {
  using FT = F<E>;
  using P = Prim<M3>;
  __shared__ double red[32];
  const size_t n = (size_t)ix * jx;
  double dmin = __longlong_as_double(0x7ff0000000000000LL);
  const FT gm(ph.gm), pi4i(ph.pi4i);
  for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < n;
       g += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(g % ix), j = (int)(g / ix);
    const FT ro(S[P::RO * n + g]), pr(S[P::PR * n + g]);
    const FT vx(S[P::VX * n + g]), vy(S[P::VY * n + g]);
    const FT bx(S[P::BX * n + g]), by(S[P::BY * n + g]);
    FT b2, v2;
    if constexpr (M3) {
      const FT vz(S[P::VZ * n + g]), bz(S[P::BZ * n + g]);
      b2 = bx * bx + by * by + bz * bz;
      v2 = vx * vx + vy * vy + vz * vz;
    } else {
      b2 = bx * bx + by * by;
      v2 = vx * vx + vy * vy;
    }
    double dtq;
    if constexpr (!E) {  // one reciprocal and one reciprocal root (see cfl3_cell)
      const double q = fma(fma(ph.gm, pr.v, b2.v * ph.pi4i), fd::rcp(ro.v), v2.v);
      dtq = safety * fd::minp(ax.d[i], ay.d[j]) * fd::rsqrt_(q);
    } else {
      const FT ca2 = b2 * pi4i / ro;
      const FT cs2 = gm * pr / ro;
      const FT dtcfl = fmin_(FT(ax.d[i]), FT(ay.d[j])) / fsqrt(v2 + cs2 + ca2);
      dtq = (FT(safety) * dtcfl).v;
    }
    if (dtq < dmin) dmin = dtq;
  }
  block_min_to(out, dmin, red, threadIdx.x, blockDim.x);
}

cudaError_t launch_cfl2d_full(int solver, bool exact, const double *S, int ix,
                              int jx, const Axis &ax, const Axis &ay,
                              const Phys &ph, double safety,
                              unsigned long long *out_bits, cudaStream_t s) {
  const size_t n = (size_t)ix * jx;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 152 * 8) blocks = 152 * 8;
  if (solver == 1) {
    if (exact) k_cfl2d_full<true, true><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, safety, out_bits);
    else k_cfl2d_full<false, true><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, safety, out_bits);
  } else {
    if (exact) k_cfl2d_full<true, false><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, safety, out_bits);
    else k_cfl2d_full<false, false><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, safety, out_bits);
  }
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// CFL over the frame of cells the boundary fill may have rewritten (ghost
// layers plus the first interior layer), then the start of the next loop
// iteration by the last block to finish.
// With all = 1 the CFL covers every cell: a loop whose chkdav changes cells
// after the step reduces its CFL here alone.

template <bool E, bool M3>
__device__ __forceinline__ double frame_dtq(const double *__restrict__ S, size_t n, int i,
                                            int j, int ix, const Axis &ax, const Axis &ay,
                                            const Phys &ph, double safety, bool &bad) {
  using P = Prim<M3>;
  const size_t g = (size_t)i + (size_t)j * ix;
  double q[P::N];
#pragma unroll
  for (int v = 0; v < P::N; v++) q[v] = (v == P::AZ) ? 0.0 : S[(size_t)v * n + g];
  return cell_dtq<E, M3>(q, i, j, ax, ay, ph, safety, bad);
}

template <bool E, bool M3>
__global__ void k_frame2d(const double *__restrict__ S, int ix, int jx,
                          Axis ax, Axis ay, Phys ph, int w, int all, Ctl *ctl) {
  __shared__ double red[32];
  if (ctl->done | ctl->pause) return;
  S = ctl->buf[ctl->cur ^ 1];  // the state the step just wrote
  const size_t n = (size_t)ix * jx;
  const long long total = frame_cells(ix, jx, w, all);
  double dmin = __longlong_as_double(0x7ff0000000000000LL);
  bool bad = false;
  for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x;
       f < total; f += (long long)gridDim.x * blockDim.x) {
    int i, j;
    frame_cell(f, ix, jx, w, all, i, j);
    const double dtq = frame_dtq<E, M3>(S, n, i, j, ix, ax, ay, ph, ctl->safety, bad);
    if (dtq < dmin) dmin = dtq;
  }
  count_bad_block(bad, &ctl->nonfinite, threadIdx.x);
  block_min_to(&ctl->cfl_bits, dmin, red, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(&ctl->frame_blocks_done, 1u);
    if (prev == gridDim.x - 1) {
      __threadfence();
      finish_iteration(ctl);
    }
  }
}

template <bool E, bool M3, bool MIX>
__global__ void __launch_bounds__(32 * Prim<M3>::N)
    k_bcframe2d(int ix, int jx, Axis ax, Axis ay, Phys ph, BcTable bc, Ctl *ctl) {
  bcframe2d<E, M3, MIX>(ix, jx, ax, ay, ph, bc, ctl, blockIdx.x, gridDim.x);
}

cudaError_t launch_bcframe2d(int solver, bool exact, int nvar, int ix, int jx, const Axis &ax,
                             const Axis &ay, const Phys &ph, const BcTable &bc, Ctl *ctl,
                             cudaStream_t s) {
  const int need = solver == 1 ? 9 : 7;
  if (nvar != need || ix < 2 * bc.margin + 3 || jx < 2 * bc.margin + 3)
    return cudaErrorInvalidValue;
  const int w = bc.margin + 1;
  int blocks = (int)((frame_cells(ix, jx, w, 0) + 31) / 32);
  if (blocks < 1) blocks = 1;
  if (blocks > 152 * 4) blocks = 152 * 4;
  const int nt = 32 * nvar;
  BcTable t = bc;
  t.mixed = bc_one_pass(bc, ix, jx) ? 0 : 1;
  auto k = solver == 1 ? (exact ? (t.mixed ? k_bcframe2d<true, true, true>
                                           : k_bcframe2d<true, true, false>)
                                : (t.mixed ? k_bcframe2d<false, true, true>
                                           : k_bcframe2d<false, true, false>))
                       : (exact ? (t.mixed ? k_bcframe2d<true, false, true>
                                           : k_bcframe2d<true, false, false>)
                                : (t.mixed ? k_bcframe2d<false, false, true>
                                           : k_bcframe2d<false, false, false>));
  k<<<blocks, nt, 0, s>>>(ix, jx, ax, ay, ph, t, ctl);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_frame2d(int solver, bool exact, const double *S, int ix,
                           int jx, const Axis &ax, const Axis &ay,
                           const Phys &ph, int margin, Ctl *ctl,
                           cudaStream_t s, int all) {
  const int w = margin + 1;
  const long long total = frame_cells(ix, jx, w, all);
  int blocks = (int)((total + 255) / 256);
  if (blocks < 1) blocks = 1;
  if (blocks > (all ? 152 * 4 : 152)) blocks = all ? 152 * 4 : 152;
  if (solver == 1) {
    if (exact) k_frame2d<true, true><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, w, all, ctl);
    else k_frame2d<false, true><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, w, all, ctl);
  } else {
    if (exact) k_frame2d<true, false><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, w, all, ctl);
    else k_frame2d<false, false><<<blocks, 256, 0, s>>>(S, ix, jx, ax, ay, ph, w, all, ctl);
  }
  count_launch();
  return cudaGetLastError();
}

}  // namespace cans
