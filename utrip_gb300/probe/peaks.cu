// Arithmetic peaks of the device for the benchmark's rooflines: the FP64
// and FP32 fused-multiply-add throughput.  Built into its own library,
// libcansprobe.so, beside libcansgpu.so: it is measurement tooling for
// bench.py, not part of the C ABI of the solver.  It also evaluates the FP64
// functions of fd64.cuh and the sums of isum.cuh on arrays, and host rules of the
// launchers, for their tests.
#include <cuda_runtime.h>

#include "balance2d.h"
#include "cans_internal.h"
#include "fd64.cuh"
#include "host_range.h"
#include "isum.cuh"

namespace {

// Eight independent FMA chains per thread; `iters` rounds.  The result is
// written so the compiler keeps every operation.
template <class T>
__global__ void k_fma_chains(T *out, int iters, T a, T b) {
  T x[8];
#pragma unroll
  for (int k = 0; k < 8; k++) x[k] = (T)(threadIdx.x * 1e-3 + k);
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = fma(x[k], a, b);
  }
  T s = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) s += x[k];
  if (s == (T)1234.5678) out[0] = s;  // practically never taken
}

template <class T>
int measure(double *tflops, int iters, T a, T b) {
  if (!tflops) return 1;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 2;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 2;
  T *out = nullptr;
  if (cudaMalloc(&out, sizeof(T)) != cudaSuccess) return 2;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int blocks = sms * 8, threads = 256;
  k_fma_chains<T><<<blocks, threads>>>(out, 64, a, b);  // warm-up
  cudaEventRecord(e0);
  k_fma_chains<T><<<blocks, threads>>>(out, iters, a, b);
  cudaEventRecord(e1);
  cudaError_t err = cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (err != cudaSuccess) return 2;
  const double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
  *tflops = flops / (ms * 1e-3) / 1e12;
  return 0;
}

}  // namespace

// Measured FMA rates in TFLOP/s (2 flops per FMA), on the default stream.
// Synchronous; 0 on success.
extern "C" int cans_probe_fp64_tflops(double *tflops) {
  return measure<double>(tflops, 4096, 0.999999, 1e-7);
}
extern "C" int cans_probe_fp32_tflops(double *tflops) {
  return measure<float>(tflops, 65536, 0.999999f, 1e-7f);
}

namespace {
// op 0 rcp, 1 sqrt, 2 rsqrt, 3 and 4 the two results of sqrt_rsqrt, 5 lt(x, w),
// 6 max(x, w), 7 the positive part
__global__ void k_fd64(int op, const double *x, const double *w, double *y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = w[i];
  double s = 0.0, r = 0.0;
  switch (op) {
    case 0: r = cans::fd::rcp(a); break;
    case 1: r = cans::fd::sqrt_(a); break;
    case 2: r = cans::fd::rsqrt_(a); break;
    case 3: cans::fd::sqrt_rsqrt(a, r, s); break;
    case 4: cans::fd::sqrt_rsqrt(a, s, r); break;
    case 5: r = cans::fd::lt(a, b) ? 1.0 : 0.0; break;
    case 6: r = cans::fd::max_(a, b); break;
    default: r = cans::fd::pos_part(a); break;
  }
  y[i] = r;
}
}  // namespace

// y[i] = the function `op` of fd64.cuh of x[i] (and w[i]); host arrays.
// Synchronous; 0 on success.
extern "C" int cans_probe_fd64(int op, const double *x, const double *w, double *y, int n) {
  if (n < 1 || !x || !w || !y || op < 0 || op > 7) return 1;
  double *d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 3 * b) != cudaSuccess) return 2;
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, w, b, cudaMemcpyHostToDevice);
  k_fd64<<<(n + 255) / 256, 256>>>(op, d, d + n, d + 2 * (size_t)n, n);
  const cudaError_t e = cudaMemcpy(y, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}

namespace {
// y[2i] = the sum, y[2i+1] = (b - a) + (c - d) of the operands a, b, c, d =
// x[4i .. 4i+3]; f[i] = 1 where they must be formed in FP64
__global__ void k_isum(const double *x, double *y, int *f, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool sp = false;
  const cans::isum::Four q =
      cans::isum::four(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3], sp);
  y[2 * i] = cans::isum::out<8>((q.a + q.b) + (q.c + q.d), q.E);
  y[2 * i + 1] = cans::isum::out<8>((q.b - q.a) + (q.c - q.d), q.E);
  f[i] = sp ? 1 : 0;
}
}  // namespace

// Host arrays of 4 n, 2 n and n values.  Synchronous; 0 on success.
extern "C" int cans_probe_isum(const double *x, double *y, int *f, int n) {
  if (n < 1 || !x || !y || !f) return 1;
  double *d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 7 * b) != cudaSuccess) return 2;
  int *df = reinterpret_cast<int *>(d + 6 * (size_t)n);
  cudaMemcpy(d, x, 4 * b, cudaMemcpyHostToDevice);
  k_isum<<<(n + 255) / 256, 256>>>(d, d + 4 * (size_t)n, df, n);
  cudaMemcpy(y, d + 4 * (size_t)n, 2 * b, cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaMemcpy(f, df, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}

namespace {
// z = x + y by isum::add2; f = 1 where it must be formed in FP64
__global__ void k_add2(const double *x, const double *y, double *z, int *f, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool sp = false;
  z[i] = cans::isum::add2(x[i], y[i], sp);
  f[i] = sp ? 1 : 0;
}
// the face states of cells x[4i .. 4i+3]: y[2i], y[2i+1]
__global__ void k_muscl(const double *x, double *y, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n)
    cans::isum::muscl(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3], y[2 * i], y[2 * i + 1]);
}
}  // namespace

// Host arrays of n values each.  Synchronous; 0 on success.
extern "C" int cans_probe_add2(const double *x, const double *y, double *z, int *f, int n) {
  if (n < 1 || !x || !y || !z || !f) return 1;
  double *d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 4 * b) != cudaSuccess) return 2;
  int *df = reinterpret_cast<int *>(d + 3 * (size_t)n);
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
  k_add2<<<(n + 255) / 256, 256>>>(d, d + n, d + 2 * (size_t)n, df, n);
  cudaMemcpy(z, d + 2 * (size_t)n, b, cudaMemcpyDeviceToHost);
  const cudaError_t e = cudaMemcpy(f, df, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}

// Host arrays of 4 n and 2 n values.  Synchronous; 0 on success.
extern "C" int cans_probe_muscl(const double *x, double *y, int n) {
  if (n < 1 || !x || !y) return 1;
  double *d = nullptr;
  const size_t b = sizeof(double) * (size_t)n;
  if (cudaMalloc(&d, 6 * b) != cudaSuccess) return 2;
  cudaMemcpy(d, x, 4 * b, cudaMemcpyHostToDevice);
  k_muscl<<<(n + 255) / 256, 256>>>(d, d + 4 * (size_t)n, n);
  const cudaError_t e = cudaMemcpy(y, d + 4 * (size_t)n, 2 * b, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}

// May the rules kind[0..3] (x lower and upper face, y lower and upper) of a variable be
// applied in one pass (bc_one_pass)?  Host only.
extern "C" int cans_probe_bc_one_pass(int margin, int ix, int jx, const int *kind) {
  cans::BcTable bc{};
  bc.margin = margin;
  for (auto &row : bc.kind)
    for (int f = 0; f < 6; f++) row[f] = cans::BD_NONE;
  for (int f = 0; f < 4; f++) bc.kind[cans::kMaxVar - 1][f] = kind[f];
  return cans::bc_one_pass(bc, ix, jx) ? 1 : 0;
}

// Does one of the rules lo and hi of a line's faces read what the other changes
// (bc_faces_meet)?  Host only.
extern "C" int cans_probe_bc_faces_meet(int margin, int n, int lo, int hi) {
  return cans::bc_faces_meet(lo, hi, margin, n) ? 1 : 0;
}

// Would the array of n doubles at address p pass as page-locked (mapped_range) with the
// nseg registrations [lo, hi) at seg[2i], seg[2i+1] of whole pages, the device address
// being that of the host plus shift[i]?  No memory is touched.
extern "C" int cans_probe_mapped_range(unsigned long long p, unsigned long long n,
                                       unsigned long long page, const unsigned long long *seg,
                                       const unsigned long long *shift, int nseg) {
  return cans::mapped_range((double *)(uintptr_t)p, n, page,
                            [=](void *q) -> void * {
                              const uintptr_t a = (uintptr_t)q;
                              for (int i = 0; i < nseg; i++)
                                if (a >= seg[2 * i] && a < seg[2 * i + 1])
                                  return (void *)(a + shift[i]);
                              return nullptr;
                            }) != nullptr;
}

// Rows of a segment as the marching steps choose them (balance_seg).  Host only.
extern "C" int cans_probe_balance_seg(int strips, int rows, int ch, int sms) {
  return cans::balance_seg(strips, rows, ch, sms);
}
