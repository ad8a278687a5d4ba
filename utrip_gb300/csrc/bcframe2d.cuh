// The boundary program, the frame CFL and the end of one loop iteration of a 2-D
// run, shared by the single run's kernel (mlw2d.cu) and the batch's (batch2d.cu).
#pragma once
#include "bc_line.cuh"
#include "cans_common.cuh"
#include "cans_internal.h"
#include "fd64.cuh"
#include "mlw2d_tile.cuh"  // Prim

namespace cans {

// Cell (i, j) of frame index f: rows j < w or j >= jx-w (all i), then
// columns i < w or i >= ix-w of the remaining rows (every cell with all).
__device__ __forceinline__ void frame_cell(long long f, int ix, int jx, int w, int all,
                                           int &i, int &j) {
  const long long nrow = 2LL * w * ix;
  if (all) {
    i = (int)(f % ix);
    j = (int)(f / ix);
  } else if (f < nrow) {
    const long long r = f / ix;
    i = (int)(f % ix);
    j = (r < w) ? (int)r : (int)(jx - 2 * w + r);
  } else {
    const long long q = f - nrow;
    const long long r = q / (2 * w);
    const int cidx = (int)(q % (2 * w));
    j = (int)(w + r);
    i = (cidx < w) ? cidx : (ix - 2 * w + cidx);
  }
}
__host__ __device__ __forceinline__ long long frame_cells(int ix, int jx, int w, int all) {
  const long long inner_rows = jx - 2LL * w;
  return all ? (long long)ix * jx
             : 2LL * w * ix + (inner_rows > 0 ? inner_rows * 2LL * w : 0);
}

// cfl_m3 (cfl_m for the 7-array layout) of one cell from its values q[v]:
// safety * the cell's time-step limit; bad is set for a cell the CFL cannot
// use.
template <bool E, bool M3>
__device__ __forceinline__ double cell_dtq(const double *q, int i, int j, const Axis &ax,
                                           const Axis &ay, const Phys &ph, double safety,
                                           bool &bad) {
  using FT = F<E>;
  using P = Prim<M3>;
  const FT gm(ph.gm), pi4i(ph.pi4i);
  const FT ro(q[P::RO]), pr(q[P::PR]);
  const FT vx(q[P::VX]), vy(q[P::VY]);
  const FT bx(q[P::BX]), by(q[P::BY]);
  FT b2, v2;
  if constexpr (M3) {
    const FT vz(q[P::VZ]), bz(q[P::BZ]);
    b2 = bx * bx + by * by + bz * bz;
    v2 = vx * vx + vy * vy + vz * vz;
  } else {
    b2 = bx * bx + by * by;
    v2 = vx * vx + vy * vy;
  }
  if constexpr (!E) {  // one reciprocal and one reciprocal root (see cfl3_cell)
    const double s = fma(fma(ph.gm, pr.v, b2.v * ph.pi4i), fd::rcp(ro.v), v2.v);
    const double dtq = safety * fd::minp(ax.d[i], ay.d[j]) * fd::rsqrt_(s);
    bad |= bad_cell(ro.v, pr.v, dtq);
    return dtq;
  }
  const FT ca2 = b2 * pi4i / ro;
  const FT cs2 = gm * pr / ro;
  const FT dtcfl = fmin_(FT(ax.d[i]), FT(ay.d[j])) / fsqrt(v2 + cs2 + ca2);
  const double dtq = (FT(safety) * dtcfl).v;
  bad |= bad_cell(ro.v, pr.v, dtq);
  return dtq;
}
// The value at 1-based position l of row `row` after the x rules.  Not
// inlined: bc_xy_value calls it from each of its rule cases.
static __device__ __noinline__ double bc_x_value(const double *row, int ix, int m, int kxl, int kxh,
                                          double q0l, double q0h, const double *dxm, int l) {
  return bd_value(kxl, kxh, m, ix, q0l, q0h, dxm, l, [&](int p) { return row[p - 1]; });
}
// The value at 1-based (i, j) of one variable's array after the x rules of
// every row and then (cy: where they change the cell) the y rules of column i.
static __device__ __noinline__ double bc_xy_value(const double *sv, int ix, int jx, int m, int kxl,
                                           int kxh, int kyl, int kyh, double qxl, double qxh,
                                           double qyl, double qyh, const double *dxmx,
                                           const double *dxmy, int i, int j, bool cy) {
  auto xval = [&](int j1) {
    return bc_x_value(sv + (size_t)(j1 - 1) * ix, ix, m, kxl, kxh, qxl, qxh, dxmx, i);
  };
  if (!cy) return xval(j);
  return bd_value(kyl, kyh, m, jx, qyl, qyh, dxmy, j, xval);
}

// The boundary program and the frame CFL of one loop iteration in one
// launch, for a 2-D loop without chkdav.  A thread owns one frame cell and
// computes each variable's value there as the x rules and then the y rules
// of the program leave it (bd_value of the y rules over a column whose values
// are bd_value of the x rules over their rows): the same operations as
// k_bc_axis (x), k_bc_axis (y), so the same bits, with no barrier between the
// axes.  A thread reads only cells that no rule changes (the step's output)
// and writes only its own cell, so the threads are independent.  It then
// reduces the CFL over the frame as k_frame2d does, from the values in
// registers, and the last block ends the iteration.
// `block` of `nblocks` blocks of 32 Prim<M3>::N threads.
// MIX: the program may be one that bc_one_pass refuses; it is then filled rule by rule.
template <bool E, bool M3, bool MIX>
__device__ __forceinline__ void bcframe2d(int ix, int jx, const Axis &ax, const Axis &ay,
                                          const Phys &ph, const BcTable &bc, Ctl *ctl, int block,
                                          int nblocks) {
  using P = Prim<M3>;
  // a block takes 32 frame cells; thread (c, v) = (lane, warp) evaluates
  // variable v of cell c, and the first warp reduces the CFL of the 32 cells
  __shared__ double q[P::N][32];
  __shared__ double red[32];
  if (ctl->done | ctl->pause) return;
  double *S = ctl->buf[ctl->cur ^ 1];  // the state the step just wrote
  const size_t n = (size_t)ix * jx;
  const int m = bc.margin, w = m + 1;
  const long long total = frame_cells(ix, jx, w, 0);
  const int c = threadIdx.x & 31, v = threadIdx.x >> 5;
  // where a rule reads what another changes (!bc_one_pass): one block, rule by rule
  const bool mixed = MIX && bc.mixed != 0;
  if (mixed) {
    if (block != 0) return;
    nblocks = 1;
    for (int axis = 0; axis < 2; axis++) {
      const int len = axis ? jx : ix, lines = axis ? ix : jx;
      for (int t = threadIdx.x; t < lines * P::N; t += blockDim.x) {
        const int u = t / lines, line = t % lines;
        double *l = S + (size_t)u * n + (size_t)line * (axis ? 1 : ix);
        for (int f = 0; f < 2; f++)
          if (bc.kind[u][2 * axis + f] >= 0)
            bd_line(bc.kind[u][2 * axis + f], f, m, m, l, len, axis ? (size_t)ix : 1,
                    bc.q0[u][2 * axis + f], axis ? ay.dm : ax.dm);
      }
      __syncthreads();
    }
  }
  double dmin = __longlong_as_double(0x7ff0000000000000LL);
  bool bad = false;
  for (long long f0 = block * 32LL; f0 < total; f0 += nblocks * 32LL) {
    const long long f = f0 + c;
    int i = 0, j = 0;
    if (f < total) {
      frame_cell(f, ix, jx, w, 0, i, j);
      const double *sv = S + (size_t)v * n;
      const int kxl = bc.kind[v][0], kxh = bc.kind[v][1];
      const int kyl = bc.kind[v][2], kyh = bc.kind[v][3];
      const bool cx = bd_changes(kxl, kxh, m, ix, i + 1);
      const bool cy = bd_changes(kyl, kyh, m, jx, j + 1);
      const double val =
          mixed ? sv[(size_t)i + (size_t)j * ix]
                : bc_xy_value(sv, ix, jx, m, kxl, kxh, kyl, kyh, bc.q0[v][0], bc.q0[v][1],
                              bc.q0[v][2], bc.q0[v][3], ax.dm, ay.dm, i + 1, j + 1, cy);
      if (!mixed && (cx || cy)) S[(size_t)v * n + (size_t)i + (size_t)j * ix] = val;
      q[v][c] = val;
    }
    __syncthreads();
    if (v == 0 && f < total) {
      double qc[P::N];
#pragma unroll
      for (int u = 0; u < P::N; u++) qc[u] = q[u][c];
      const double dtq = cell_dtq<E, M3>(qc, i, j, ax, ay, ph, ctl->safety, bad);
      if (dtq < dmin) dmin = dtq;
    }
    __syncthreads();
  }
  count_bad_block(bad, &ctl->nonfinite, threadIdx.x);
  block_min_to(&ctl->cfl_bits, dmin, red, threadIdx.x, blockDim.x);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned prev = atomicAdd(&ctl->frame_blocks_done, 1u);
    if (prev == (unsigned)nblocks - 1) {
      __threadfence();
      finish_iteration(ctl);
    }
  }
}

}  // namespace cans
