// Many independent 2-D runs advanced together (sm_103a, FP64).
//
// A parameter sweep runs the same 2-D model (for example the magnetised shear
// layer of cans2d/md_mhdkh/hdmlw/model.f) for many grid sizes and plasma
// betas.  Run one at a time, a small grid fills a fraction of the 152 SMs and
// every step pays the launch latency of its kernels.  Here one loop iteration
// of every run is two launches in total (three where equally spaced and stretched
// meshes are in one batch):
//   1. a persistent step kernel: one block per resident slot; each block pulls
//      (run, tile) work items from a device work queue and applies the single
//      run's block (mlw2d_march.cuh; exact policy: mlw2d_tile.cuh) with the
//      run's own arrays, metrics, dt and CFL accumulator;
//   2. the boundary programs, frame CFLs and loop ends of all runs
//      (bcframe2d.cuh), and the reset of the work queue.
// Each run keeps its own dt, t, ns and termination exactly as if it ran
// alone, so the exact policy's results equal single-run results bit for bit.  The
// launches are captured in a CUDA graph; the tile shape and the cells per
// thread are picked by timing (cans_batch_autotune).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "bcframe2d.cuh"
#include "cans_common.cuh"
#include "cans_gpu.h"
#include "cans_internal.h"
#include "mlw2d_march.cuh"
#include "mlw2d_tile.cuh"

namespace cans {

// Device description of one run of the batch.
struct BatchGrid {
  Ctl *ctl;
  Axis ax, ay;
  Phys ph;
  Box3 box;       // cells whose CFL the step kernel reduces
  int ix, jx;
  int ntx, nty;   // tiles of the current configuration
  int tile0;      // first work item of this run
};

// The step's launches, each with a work queue of its own: the runs whose axes are all
// equally spaced and the others (exact policy: one launch for all).  A run is stepped by
// the instance of its own mesh whatever it shares the batch with.
constexpr int kQueues = 2;

// The next work item of a persistent block, or -1: the run it belongs to in *run,
// its tile in *tile.
__device__ __forceinline__ int next_item(const BatchGrid *__restrict__ grids, int ngrids,
                                         int nitems, unsigned int *queue, int *run, int *tile) {
  __shared__ int s_item;
  if (threadIdx.x == 0) s_item = (int)atomicAdd(queue, 1u);
  __syncthreads();
  const int item = s_item;
  __syncthreads();  // every thread has read s_item before it is rewritten
  if (item >= nitems) return -1;
  int lo = 0, hi = ngrids - 1;  // last run whose first item <= item
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (grids[mid].tile0 <= item) lo = mid;
    else hi = mid - 1;
  }
  *run = lo;
  *tile = item - grids[lo].tile0;
  return item;
}

// Step of every run in the exact policy: persistent blocks pull work items until
// the queue is exhausted.
template <bool M3, int TX, int TY, int RPT>
__global__ void __launch_bounds__(TX *TY / RPT, 1)
    k_mlw2d_batch(const BatchGrid *__restrict__ grids, int ngrids, int nitems,
                  unsigned int *queue) {
  extern __shared__ double smem[];
  int run, t;
  while (next_item(grids, ngrids, nitems, queue, &run, &t) >= 0) {
    const BatchGrid &G = grids[run];
    Ctl *ctl = G.ctl;
    if (ctl->done | ctl->pause) continue;
    tile_step<M3, TX, TY, RPT>(ctl->buf[ctl->cur], ctl->buf[ctl->cur ^ 1], G.ix,
                               G.jx, G.ax, G.ay, G.ph, ctl->dt, ctl->safety,
                               &ctl->cfl_bits, G.box, t % G.ntx, t / G.ntx,
                               G.ntx, G.nty, smem, nullptr, nullptr, &ctl->nonfinite);
  }
}

// The same in the fast policy: an item is a segment of `seg` rows of a strip of
// 32 columns, stepped by the single run's marching block (mlw2d_march.cuh), so
// that a batch runs its zones at the rate of a step that fills the GPU.
constexpr int kBatchCH = kFastCH;
template <bool M3, bool U>
__global__ void __launch_bounds__(March<kBatchCH, M3, false>::NT, 2)
    k_mlw2d_batch_fast(const BatchGrid *__restrict__ grids, int ngrids, int nitems, int seg,
                       unsigned int *queue) {
  extern __shared__ double smem_march[];
  int run, t;
  while (next_item(grids, ngrids, nitems, queue, &run, &t) >= 0) {
    const BatchGrid &G = grids[run];
    Ctl *ctl = G.ctl;
    if (ctl->done | ctl->pause) continue;
    MarchArgs m{};
    m.A = ctl->buf[ctl->cur];
    m.B = ctl->buf[ctl->cur ^ 1];
    m.ix = G.ix;
    m.jx = G.jx;
    m.dt = ctl->dt;
    m.safety = ctl->safety;
    m.cfl = &ctl->cfl_bits;
    m.bad = &ctl->nonfinite;
    m.box = G.box;
    const int jb = 1 + (t / G.ntx) * seg;
    march_block<F64N, kBatchCH, M3, false, false, 0, U>(m, G.ax, G.ay, G.ph, t % G.ntx, G.ntx, jb,
                                                     min(G.jx - 2, jb + seg - 1), smem_march);
  }
}

// Boundary program, frame CFL and loop end of every run (blockIdx.y) as a single
// run's k_bcframe2d does them, and the reset of the work queue for the next
// step.  One launch for what were three; the frame CFL of a run, on one SM
// before, spreads over the blocks of its row of the grid.
template <bool E, bool M3, bool MIX>
__global__ void __launch_bounds__(32 * Prim<M3>::N)
    k_bcframe_batch(const BatchGrid *__restrict__ grids, const BcTable *__restrict__ tables,
                    unsigned int *queue) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < kQueues) queue[threadIdx.x] = 0u;
  const BatchGrid &G = grids[blockIdx.y];
  bcframe2d<E, M3, MIX>(G.ix, G.jx, G.ax, G.ay, G.ph, tables[blockIdx.y], G.ctl, blockIdx.x,
                   gridDim.x);
}

// Start of every run (the first CFL is reduced into cfl_bits beforehand).
__global__ void k_prepare_batch(const BatchGrid *__restrict__ grids, int ngrids) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= ngrids) return;
  Ctl *ctl = grids[g].ctl;
  if (ctl->done || ctl->pause) return;
  start_iteration(ctl);
}

// ---------------------------------------------------------------------------
// Configurations the autotuner chooses from: tile shape and cells per thread of
// the exact policy; rows of a work item of the fast one (strips of 32 columns):
// long segments recompute fewer halo rows, short ones fill the last wave.
struct BatchConfig {
  int tx, ty, rpt;
};
static const BatchConfig kConfigs[] = {
    {32, 8, 2}, {32, 8, 1}, {32, 16, 2}, {16, 16, 2}, {32, 16, 4}, {64, 8, 2}};
static const BatchConfig kFastConfigs[] = {
    {32, 32, 0}, {32, 16, 0}, {32, 24, 0}, {32, 48, 0}, {32, 64, 0}, {32, 40, 0}};
constexpr int kNumConfigs = sizeof(kConfigs) / sizeof(kConfigs[0]);
static_assert(sizeof(kFastConfigs) == sizeof(kConfigs), "one index serves both policies");

// Blocks of a persistent kernel that a device holds at once: asked, and the kernel's
// shared memory set, once per device under a lock (batches of several host threads and
// devices share a kernel).
struct Resident {
  std::mutex mu;
  int of[64] = {};
};
template <class Kern, class... Args>
static cudaError_t launch_persistent(Kern kern, Resident &r, int nt, size_t smem, int nitems,
                                     cudaStream_t s, Args... args) {
  int dev = 0, resident = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  {
    std::lock_guard<std::mutex> lk(r.mu);
    if (!r.of[dev]) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      int per_sm = 0, sms = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, nt, smem);
      if (e != cudaSuccess) return e;
      e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return e;
      r.of[dev] = (per_sm > 0 ? per_sm : 1) * sms;
    }
    resident = r.of[dev];
  }
  const int blocks = resident < nitems ? resident : nitems;
  kern<<<blocks > 0 ? blocks : 1, nt, smem, s>>>(args...);
  count_launch();
  return cudaGetLastError();
}

template <bool M3, int TX, int TY, int RPT>
static cudaError_t launch_batch_cfg(const BatchGrid *grids, int ngrids, int nitems,
                                    unsigned int *queue, cudaStream_t s) {
  using T = Tile<TX, TY, M3, RPT>;
  static Resident resident;  // per template instance
  return launch_persistent(k_mlw2d_batch<M3, TX, TY, RPT>, resident, T::NT, T::smem_bytes, nitems,
                           s, grids, ngrids, nitems, queue);
}

template <bool M3>
static cudaError_t launch_batch(int cfg, const BatchGrid *grids, int ngrids,
                                int nitems, unsigned int *queue, cudaStream_t s) {
  switch (cfg) {
    case 1: return launch_batch_cfg<M3, 32, 8, 1>(grids, ngrids, nitems, queue, s);
    case 2: return launch_batch_cfg<M3, 32, 16, 2>(grids, ngrids, nitems, queue, s);
    case 3: return launch_batch_cfg<M3, 16, 16, 2>(grids, ngrids, nitems, queue, s);
    case 4: return launch_batch_cfg<M3, 32, 16, 4>(grids, ngrids, nitems, queue, s);
    case 5: return launch_batch_cfg<M3, 64, 8, 2>(grids, ngrids, nitems, queue, s);
    default: return launch_batch_cfg<M3, 32, 8, 2>(grids, ngrids, nitems, queue, s);
  }
}
template <bool M3, bool U>
static cudaError_t launch_batch_fast(int cfg, const BatchGrid *grids, int ngrids, int nitems,
                                     unsigned int *queue, cudaStream_t s) {
  using T = March<kBatchCH, M3, false>;
  static Resident resident;  // per template instance
  return launch_persistent(k_mlw2d_batch_fast<M3, U>, resident, T::NT, T::smem_bytes, nitems, s,
                           grids, ngrids, nitems, kFastConfigs[cfg].ty, queue);
}

}  // namespace cans

using namespace cans;

namespace {

thread_local std::string g_batch_error;
int bfail(cudaError_t e, const char *where) {
  g_batch_error = std::string(where) + ": " + cudaGetErrorString(e);
  return CANS_ERR_CUDA;
}
#define BK(call)                                            \
  do {                                                      \
    cudaError_t _e = (call);                                \
    if (_e != cudaSuccess) return bfail(_e, #call);         \
  } while (0)

unsigned long long r4_1e20() {
  const double d = (double)1.e20f;
  unsigned long long b;
  std::memcpy(&b, &d, sizeof b);
  return b;
}

}  // namespace

struct cans_batch {
  int ngrids = 0, solver = 1, nvar = 9, exact = 0, config = 0, margin = 1;
  cudaStream_t s = nullptr;
  bool own_stream = false;
  struct Grid {
    int ix = 0, jx = 0;
    size_t n = 0;
    double *buf[2] = {nullptr, nullptr};
    double *metrics = nullptr;  // the arrays of x, then of y
    Ctl *ctl = nullptr;
    BcTable bc{};
    Phys ph{};
    Axis ax, ay;
    int stop_on_bad = 0;
  };
  std::vector<Grid> g;
  std::vector<BatchGrid> hgrids;  // the runs of each of the step's launches in turn
  BatchGrid *d_grids = nullptr;
  BcTable *d_bc = nullptr;
  bool mixed = false;  // a run's program cannot be applied in one pass (bc_one_pass)
  unsigned int *d_queue = nullptr;
  int nruns[kQueues] = {}, nitems[kQueues] = {};  // of each of the step's launches
  int frame_blocks = 1;
  cudaGraphExec_t graph = nullptr;
  int graph_iters = 0, graph_nodes = 0;
};

namespace {

void drop_graph(cans_batch *b) {
  if (b->graph) cudaGraphExecDestroy(b->graph);
  b->graph = nullptr;
  b->graph_iters = 0;
}

// Tiles of every run under the current configuration, uploaded with the
// run descriptions and boundary tables.
int sync_tables(cans_batch *b) {
  const BatchConfig c = b->exact ? kConfigs[b->config] : kFastConfigs[b->config];
  int frame = 0;
  b->hgrids.clear();
  std::vector<int> order;  // runs by launch
  for (int q = 0; q < kQueues; q++) {
    b->nruns[q] = b->nitems[q] = 0;
    for (int r = 0; r < b->ngrids; r++)
      if ((b->exact || (b->g[r].ax.uniform && b->g[r].ay.uniform) ? 0 : 1) == q) {
        order.push_back(r);
        b->nruns[q]++;
      }
  }
  for (int k = 0; k < b->ngrids; k++) {
    auto &G = b->g[order[k]];
    int &item = b->nitems[k < b->nruns[0] ? 0 : 1];
    b->hgrids.emplace_back();
    BatchGrid &H = b->hgrids.back();
    H.ctl = G.ctl;
    H.ax = G.ax;
    H.ay = G.ay;
    H.ph = G.ph;
    const int w = b->margin + 1;
    H.box = Box3{{w, w, 0}, {G.ix - 1 - w, G.jx - 1 - w, 0}};
    H.ix = G.ix;
    H.jx = G.jx;
    H.ntx = (G.ix - 2 + c.tx - 1) / c.tx;
    H.nty = (G.jx - 2 + c.ty - 1) / c.ty;
    H.tile0 = item;
    item += H.ntx * H.nty;
    frame = std::max(frame, (int)frame_cells(G.ix, G.jx, w, 0));
  }
  b->frame_blocks = std::min((frame + 31) / 32, 152 * 4);
  std::vector<BcTable> bcs(b->ngrids);
  b->mixed = false;
  for (int k = 0; k < b->ngrids; k++) {
    auto &G = b->g[order[k]];
    bcs[k] = G.bc;
    bcs[k].mixed = bc_one_pass(G.bc, G.ix, G.jx) ? 0 : 1;
    b->mixed |= bcs[k].mixed != 0;
  }
  BK(cudaMemcpyAsync(b->d_grids, b->hgrids.data(), sizeof(BatchGrid) * b->ngrids,
                     cudaMemcpyHostToDevice, b->s));
  BK(cudaMemcpyAsync(b->d_bc, bcs.data(), sizeof(BcTable) * b->ngrids,
                     cudaMemcpyHostToDevice, b->s));
  BK(cudaStreamSynchronize(b->s));
  drop_graph(b);
  return CANS_OK;
}

int step_launch(cans_batch *b, int cfg) {
  const bool m3 = b->solver == CANS_SOLVER_MLW_M3_2D;
  for (int q = 0; q < kQueues; q++) {
    if (b->nruns[q] == 0) continue;
    const BatchGrid *grids = b->d_grids + (q ? b->nruns[0] : 0);
    if (b->exact)
      BK((m3 ? launch_batch<true> : launch_batch<false>)(cfg, grids, b->nruns[q], b->nitems[q],
                                                         b->d_queue + q, b->s));
    else
      BK((m3 ? q ? launch_batch_fast<true, false> : launch_batch_fast<true, true>
             : q ? launch_batch_fast<false, false> : launch_batch_fast<false, true>)(
          cfg, grids, b->nruns[q], b->nitems[q], b->d_queue + q, b->s));
  }
  return CANS_OK;
}

int enqueue_batch_iteration(cans_batch *b) {
  int rc = step_launch(b, b->config);
  if (rc) return rc;
  const bool m3 = b->solver == CANS_SOLVER_MLW_M3_2D;
  const dim3 grid(b->frame_blocks, b->ngrids);
  const int nt = 32 * b->nvar;
  const bool x = b->mixed;
  auto k = m3 ? (b->exact ? (x ? k_bcframe_batch<true, true, true>
                               : k_bcframe_batch<true, true, false>)
                          : (x ? k_bcframe_batch<false, true, true>
                               : k_bcframe_batch<false, true, false>))
              : (b->exact ? (x ? k_bcframe_batch<true, false, true>
                               : k_bcframe_batch<true, false, false>)
                          : (x ? k_bcframe_batch<false, false, true>
                               : k_bcframe_batch<false, false, false>));
  k<<<grid, nt, 0, b->s>>>(b->d_grids, b->d_bc, b->d_queue);
  count_launch();
  BK(cudaGetLastError());
  return CANS_OK;
}

int read_ctl(cans_batch *b, int r, Ctl *out) {
  BK(cudaMemcpyAsync(out, b->g[r].ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, b->s));
  BK(cudaStreamSynchronize(b->s));
  return CANS_OK;
}

}  // namespace

extern "C" int cans_batch_destroy(cans_batch *b) {
  if (!b) return CANS_ERR_ARG;
  if (b->s) cudaStreamSynchronize(b->s);
  drop_graph(b);
  for (auto &G : b->g) {
    for (int k = 0; k < 2; k++)
      if (G.buf[k]) cudaFree(G.buf[k]);
    if (G.metrics) cudaFree(G.metrics);
    if (G.ctl) cudaFree(G.ctl);
  }
  if (b->d_grids) cudaFree(b->d_grids);
  if (b->d_bc) cudaFree(b->d_bc);
  if (b->d_queue) cudaFree(b->d_queue);
  if (b->own_stream && b->s) cudaStreamDestroy(b->s);
  delete b;
  return CANS_OK;
}

extern "C" int cans_batch_create(cans_batch **out, int ngrids,
                                 const cans_run_desc *descs) {
  if (!out || ngrids < 1 || ngrids > 65535 || !descs) return CANS_ERR_ARG;
  const int solver = descs[0].solver;
  if (solver != CANS_SOLVER_MLW_M_2D && solver != CANS_SOLVER_MLW_M3_2D) return CANS_ERR_ARG;
  for (int r = 0; r < ngrids; r++) {
    const cans_run_desc &d = descs[r];
    const int wmin = 2 * (d.margin + 1) + 1;
    if (d.solver != solver || d.margin != descs[0].margin || d.exact != descs[0].exact ||
        d.ix < wmin || d.jx < wmin || d.kx != 1 || !d.dx || !d.dxm || !d.dy || !d.dym)
      return CANS_ERR_ARG;
    // the batch runs the plain mlw_m / mlw_m3 step: no source-term variant
    if (d.gx || d.et || d.etm) return CANS_ERR_ARG;
  }
  auto *b = new cans_batch();
  b->ngrids = ngrids;
  b->solver = solver;
  b->nvar = solver == CANS_SOLVER_MLW_M3_2D ? 9 : 7;
  b->exact = descs[0].exact;
  b->margin = descs[0].margin;
  b->g.resize(ngrids);
  auto bail = [&](int rc) {
    cans_batch_destroy(b);
    return rc;
  };
  cudaError_t e;
  if (descs[0].stream) {
    b->s = (cudaStream_t)descs[0].stream;
  } else {
    e = cudaStreamCreateWithFlags(&b->s, cudaStreamNonBlocking);
    if (e != cudaSuccess) return bail(bfail(e, "cudaStreamCreate"));
    b->own_stream = true;
  }
  std::vector<double> h;
  for (int r = 0; r < ngrids; r++) {
    const cans_run_desc &d = descs[r];
    auto &G = b->g[r];
    G.ix = d.ix;
    G.stop_on_bad = d.stop_on_bad ? 1 : 0;
    G.jx = d.jx;
    G.n = (size_t)d.ix * d.jx;
    G.ph = make_phys(d.gm, d.qav);
    G.bc.margin = d.margin;
    for (int v = 0; v < kMaxVar; v++)
      for (int f = 0; f < 6; f++) {
        G.bc.kind[v][f] = BD_NONE;
        G.bc.q0[v][f] = 0.0;
      }
    for (int k = 0; k < 2; k++) {
      e = cudaMalloc(&G.buf[k], sizeof(double) * G.n * b->nvar);
      if (e != cudaSuccess) return bail(bfail(e, "cudaMalloc(state)"));
      e = cudaMemsetAsync(G.buf[k], 0, sizeof(double) * G.n * b->nvar, b->s);
      if (e != cudaSuccess) return bail(bfail(e, "cudaMemset(state)"));
    }
    const size_t nmx = kAxisArrays * (size_t)d.ix, nm = nmx + kAxisArrays * (size_t)d.jx;
    e = cudaMalloc(&G.metrics, sizeof(double) * nm);
    if (e != cudaSuccess) return bail(bfail(e, "cudaMalloc(metrics)"));
    h.assign(nm, 0.0);
    place_axis(G.ax, G.metrics, d.ix);
    place_axis(G.ay, G.metrics + nmx, d.jx);
    G.ax.uniform = build_axis_host(d.ix, d.dx, d.dxm, h.data());
    G.ay.uniform = build_axis_host(d.jx, d.dy, d.dym, h.data() + nmx);
    e = cudaMemcpyAsync(G.metrics, h.data(), sizeof(double) * nm, cudaMemcpyHostToDevice, b->s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->s);
    if (e != cudaSuccess) return bail(bfail(e, "cudaMemcpy(metrics)"));
    e = cudaMalloc(&G.ctl, sizeof(Ctl));
    if (e != cudaSuccess) return bail(bfail(e, "cudaMalloc(ctl)"));
    Ctl c;
    std::memset(&c, 0, sizeof c);
    c.done = 1;
    c.buf[0] = G.buf[0];
    c.buf[1] = G.buf[1];
    e = cudaMemcpyAsync(G.ctl, &c, sizeof c, cudaMemcpyHostToDevice, b->s);
    if (e != cudaSuccess) return bail(bfail(e, "cudaMemcpy(ctl)"));
  }
  e = cudaMalloc(&b->d_grids, sizeof(BatchGrid) * ngrids);
  if (e == cudaSuccess) e = cudaMalloc(&b->d_bc, sizeof(BcTable) * ngrids);
  if (e == cudaSuccess) e = cudaMalloc(&b->d_queue, kQueues * sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaMemsetAsync(b->d_queue, 0, kQueues * sizeof(unsigned int), b->s);
  if (e != cudaSuccess) return bail(bfail(e, "cudaMalloc(batch tables)"));
  int rc = sync_tables(b);
  if (rc) return bail(rc);
  *out = b;
  return CANS_OK;
}

extern "C" int cans_batch_set_bc(cans_batch *b, int grid, int var, int face, int kind,
                                 double q0) {
  if (!b || grid < 0 || grid >= b->ngrids || var < 0 || var >= b->nvar || face < 0 ||
      face >= 4 || kind < CANS_BD_NONE || kind > CANS_BD_FRD)
    return CANS_ERR_ARG;
  b->g[grid].bc.kind[var][face] = kind;
  b->g[grid].bc.q0[var][face] = q0;
  return sync_tables(b);
}

extern "C" int cans_batch_push(cans_batch *b, int grid, double *const *host) {
  if (!b || grid < 0 || grid >= b->ngrids || !host) return CANS_ERR_ARG;
  Ctl c;
  int rc = read_ctl(b, grid, &c);
  if (rc) return rc;
  auto &G = b->g[grid];
  for (int v = 0; v < b->nvar; v++)
    BK(cudaMemcpyAsync(G.buf[c.cur] + v * G.n, host[v], sizeof(double) * G.n,
                       cudaMemcpyHostToDevice, b->s));
  BK(cudaStreamSynchronize(b->s));
  return CANS_OK;
}

extern "C" int cans_batch_pull(cans_batch *b, int grid, double *const *host) {
  if (!b || grid < 0 || grid >= b->ngrids || !host) return CANS_ERR_ARG;
  Ctl c;
  int rc = read_ctl(b, grid, &c);
  if (rc) return rc;
  auto &G = b->g[grid];
  for (int v = 0; v < b->nvar; v++)
    BK(cudaMemcpyAsync(host[v], G.buf[c.cur] + v * G.n, sizeof(double) * G.n,
                       cudaMemcpyDeviceToHost, b->s));
  BK(cudaStreamSynchronize(b->s));
  return CANS_OK;
}

extern "C" int cans_batch_start(cans_batch *b, double t0, double tend, long long nstop,
                                double safety, double dtmin) {
  NvtxRange nvtx("cans_batch_start");
  if (!b) return CANS_ERR_ARG;
  for (int r = 0; r < b->ngrids; r++) {
    auto &G = b->g[r];
    Ctl c;
    int rc = read_ctl(b, r, &c);
    if (rc) return rc;
    c.t = t0;
    c.tp = t0;
    c.tend = tend;
    c.nstop = nstop;
    c.safety = safety;
    c.dtmin = dtmin;
    c.dtout = 0.0;
    c.pause_on_output = 0;
    c.ns = 0;
    c.nexec = 0;
    c.merr = 0;
    c.done = 0;
    c.pause = 0;
    c.frame_blocks_done = 0;
    c.nonfinite = 0;
    c.nfloor = 0;
    c.stop_on_bad = G.stop_on_bad;
    c.cfl_bits = r4_1e20();
    BK(cudaMemcpyAsync(G.ctl, &c, sizeof c, cudaMemcpyHostToDevice, b->s));
    BK(launch_cfl2d_full(b->solver, b->exact != 0, G.buf[c.cur], G.ix, G.jx, G.ax, G.ay,
                         G.ph, safety, &G.ctl->cfl_bits, b->s));
  }
  k_prepare_batch<<<(b->ngrids + 127) / 128, 128, 0, b->s>>>(b->d_grids, b->ngrids);
  count_launch();
  BK(cudaGetLastError());
  BK(cudaMemsetAsync(b->d_queue, 0, kQueues * sizeof(unsigned int), b->s));
  BK(cudaStreamSynchronize(b->s));
  return CANS_OK;
}

extern "C" int cans_batch_advance(cans_batch *b, int iters, int use_graph) {
  NvtxRange nvtx("cans_batch_advance");
  if (!b || iters < 0) return CANS_ERR_ARG;
  if (!use_graph) {
    for (int k = 0; k < iters; k++) {
      int rc = enqueue_batch_iteration(b);
      if (rc) return rc;
    }
    return CANS_OK;
  }
  const int chunk = iters < 16 ? iters : 16;
  if (chunk == 0) return CANS_OK;
  if (!b->graph || b->graph_iters != chunk) {
    drop_graph(b);
    cudaGraph_t g = nullptr;
    const unsigned long long before = launch_count();
    BK(cudaStreamBeginCapture(b->s, cudaStreamCaptureModeThreadLocal));
    int rc = CANS_OK;
    for (int k = 0; k < chunk && rc == CANS_OK; k++) rc = enqueue_batch_iteration(b);
    cudaError_t e = cudaStreamEndCapture(b->s, &g);
    count_launch(-(int)(launch_count() - before));  // counted at replay
    if (rc) {
      if (g) cudaGraphDestroy(g);
      return rc;
    }
    if (e != cudaSuccess) return bfail(e, "cudaStreamEndCapture");
    size_t nn = 0;
    cudaGraphGetNodes(g, nullptr, &nn);
    e = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return bfail(e, "cudaGraphInstantiate");
    b->graph_iters = chunk;
    b->graph_nodes = (int)nn;
  }
  int done = 0;
  while (done + chunk <= iters) {
    BK(cudaGraphLaunch(b->graph, b->s));
    count_launch(b->graph_nodes);
    done += chunk;
  }
  for (; done < iters; done++) {
    int rc = enqueue_batch_iteration(b);
    if (rc) return rc;
  }
  return CANS_OK;
}

extern "C" int cans_batch_query(cans_batch *b, int grid, cans_run_state *st) {
  if (!b || grid < 0 || grid >= b->ngrids || !st) return CANS_ERR_ARG;
  Ctl c;
  int rc = read_ctl(b, grid, &c);
  if (rc) return rc;
  st->t = c.t;
  st->dt = c.dt;
  st->ns = c.ns;
  st->nexec = c.nexec;
  st->merr = c.merr;
  st->done = c.done;
  st->pause = c.pause;
  st->n_floor = 0;
  st->n_bad = c.nonfinite;
  return CANS_OK;
}

extern "C" int cans_batch_configs(void) { return kNumConfigs; }

extern "C" int cans_batch_set_config(cans_batch *b, int config) {
  if (!b || config < 0 || config >= kNumConfigs) return CANS_ERR_ARG;
  b->config = config;
  return sync_tables(b);
}

extern "C" int cans_batch_autotune(cans_batch *b, int trial_steps, int *config) {
  if (!b || trial_steps < 1) return CANS_ERR_ARG;
  // Time the step kernel alone: it writes only each run's other buffer and
  // leaves the current states, times and dt unchanged.  Call after
  // cans_batch_start.
  cudaEvent_t e0, e1;
  BK(cudaEventCreate(&e0));
  BK(cudaEventCreate(&e1));
  float best = 1e30f;
  int best_cfg = b->config;
  for (int c = 0; c < kNumConfigs; c++) {
    b->config = c;
    int rc = sync_tables(b);
    if (rc) return rc;
    BK(cudaMemsetAsync(b->d_queue, 0, kQueues * sizeof(unsigned int), b->s));
    if ((rc = step_launch(b, c))) return rc;  // warm-up
    BK(cudaMemsetAsync(b->d_queue, 0, kQueues * sizeof(unsigned int), b->s));
    BK(cudaEventRecord(e0, b->s));
    for (int k = 0; k < trial_steps; k++) {
      if ((rc = step_launch(b, c))) return rc;
      BK(cudaMemsetAsync(b->d_queue, 0, kQueues * sizeof(unsigned int), b->s));
    }
    BK(cudaEventRecord(e1, b->s));
    BK(cudaEventSynchronize(e1));
    float ms = 0.f;
    BK(cudaEventElapsedTime(&ms, e0, e1));
    if (ms < best) {
      best = ms;
      best_cfg = c;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // the trial steps reduced the CFL of the state they wrote, which is the
  // state the first real step writes again: the minimum is unchanged
  b->config = best_cfg;
  int rc = sync_tables(b);
  if (rc) return rc;
  if (config) *config = best_cfg;
  return CANS_OK;
}
