// Shared types and helpers for the DEReK GB300 library.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "derek_gpu.h"

namespace derek {

// Complex element type per precision: float2 (FP32 path) or double2 (FP64).
template <typename R> struct CT;
template <> struct CT<float>  { using T = float2; };
template <> struct CT<double> { using T = double2; };
template <typename R> using cplx = typename CT<R>::T;

template <typename R> __host__ __device__ __forceinline__ cplx<R> mk(R x, R y) {
  cplx<R> c; c.x = x; c.y = y; return c;
}
template <typename R> __host__ __device__ __forceinline__ cplx<R> cadd(cplx<R> a, cplx<R> b) {
  return mk<R>(a.x + b.x, a.y + b.y);
}
template <typename R> __host__ __device__ __forceinline__ cplx<R> csub(cplx<R> a, cplx<R> b) {
  return mk<R>(a.x - b.x, a.y - b.y);
}
template <typename R> __host__ __device__ __forceinline__ cplx<R> cmul(cplx<R> a, cplx<R> b) {
  return mk<R>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
template <typename R> __host__ __device__ __forceinline__ cplx<R> cmulc(cplx<R> a, cplx<R> b) {
  return mk<R>(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
template <typename R> __host__ __device__ __forceinline__ cplx<R> cscale(cplx<R> a, R s) {
  return mk<R>(a.x * s, a.y * s);
}
// a s + b (real s), fused
template <typename R> __device__ __forceinline__ cplx<R> caxpy(cplx<R> a, R s, cplx<R> b);
template <> __device__ __forceinline__ double2 caxpy<double>(double2 a, double s, double2 b) {
  return make_double2(fma(a.x, s, b.x), fma(a.y, s, b.y));
}
// SIGN i (a - b)
template <typename R, int SIGN> __device__ __forceinline__ cplx<R> csub_si(cplx<R> a, cplx<R> b) {
  return SIGN > 0 ? mk<R>(b.y - a.y, a.x - b.x) : mk<R>(a.y - b.y, b.x - a.x);
}

// Complex FP32 additions and real multiples as packed pairs: one issue slot
// instead of two (the multiply-add pipe's rate is the same).  The register-line
// transforms are bound by issue, and their values sit in aligned register pairs
// anyway.  Each half rounds as the scalar operation does.  Multiplications by
// +-i swap the halves, so they stay two scalar operations (csub_si).
#ifdef __CUDA_ARCH__
__device__ __forceinline__ unsigned long long pack2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
template <> __device__ __forceinline__ float2 cadd<float>(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(r);
}
template <> __device__ __forceinline__ float2 csub<float>(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(r);
}
#endif
template <> __device__ __forceinline__ float2 caxpy<float>(float2 a, float s, float2 b) {
#ifdef __CUDA_ARCH__
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(make_float2(s, s))), "l"(pack2(b)));
  return unpack2(r);
#else
  return make_float2(a.x * s + b.x, a.y * s + b.y);
#endif
}

constexpr int kMaxRadices = 8;
constexpr int kMaxDim = 128;       // largest FFT length along one axis

// Radix plan of one FFT length (product of radices == n).
struct FftPlan {
  int n;
  int nstages;
  int radix[kMaxRadices];
  long long tw_off;   // offset of this length's twiddle table (n entries)
};

// Factorisation of one transform length for the shared-memory line kernels
// (fft4.cuh): n = a * b with a, b <= 16.
struct LinePlan {
  int n, a, b;
  int pfa;                 // a, b coprime: prime-factor index maps, no twiddles
  int inv;                 // pfa: inverse of a + b modulo n
  long long tw_off;        // twiddle table exp(-2 pi i t / n), t < n
};

inline void set_line_split(LinePlan &p, int a, int b) {
  p.a = a;
  p.b = b;
  int x = a, y = b;
  while (y) {
    const int t = x % y;
    x = y;
    y = t;
  }
  p.pfa = x == 1;
  p.inv = 1;
  if (p.pfa)
    while ((long long)p.inv * (a + b) % p.n != 1 % p.n) ++p.inv;
}

// One independent Kohn-Sham system of a batch.
struct SysDev {
  int n[3];
  int nr;
  int nk;
  int nb;                  // bands carried (requested + buffer), x nspinor
  int nbr;                 // bands requested and reported, x nspinor
  int ks0;                 // first k-set index of this system
  int active;              // 0 once converged (work items exit early)
  int nspinor;             // 1, or 2: band b is items 2b (up) and 2b + 1 (down)
  double volume;
  double B[9];             // inv_cell, row-major: G_i = sum_j B[i*3+j] m_j
  double ecut;
  double nelec;
  double kT;
  long long grid_off;      // offset of this system's grids (nr entries)
  FftPlan plan[3];         // Stockham plans (full-grid transforms)
  LinePlan lp[3];          // line splits (H.psi and density)
};

// One (system, k-point) pair: its plane-wave sphere and buffers.  The
// sphere's coefficients are stored in column order: the ncol (y,z) columns
// the sphere occupies, each a contiguous run of increasing Miller x.
struct KSetDev {
  int sys;
  int kidx;
  int npw;
  int npw_pad;
  int nb;                  // bands carried (requested + buffer), x nspinor
  int nbr;                 // bands requested and reported, x nspinor
  int ncol;                // (y,z) columns of the sphere
  int ncol_pad;
  int nrow;                // distinct y rows holding columns
  int item0;               // first (k-set, band) item of this k-set
  long long psi_off;       // element offset of band 0 in psi-shaped buffers
  long long ent_off;       // offset into per-sphere-entry tables
  long long col_off;       // offset into per-column tables (ncol + 1 entries)
  long long row_off;       // offset into the active-row lists
  long long a_off;         // element offset in the x-line buffer (nb * n1 * ncol_pad)
  double wk;
  double kfrac[3];
};

// One unit of the density pass: bands g, g + ng, ... of a k-set, summed into a
// partial grid of its own (spinor systems: four grids n, mx, my, mz).
struct DensityUnit {
  int ks, g, ng;
  long long off;           // element offset of the partial grid
};

// Host-side count of kernel launches issued by the library (every launch
// site calls note_launch; a CUDA graph replay adds its captured kernel count).
void note_launch(long long n = 1);
unsigned long long launch_total();

// Programmatic dependent launch.  Every kernel begins with grid_dependency():
// it lets the stream's next kernel become resident as soon as the last of this
// one's blocks has started, and then waits until the previous kernel has
// completed and its writes are visible.  Nothing runs ahead of the wait, so the
// order of work is the stream's; what goes is the launch gap between kernels.
// Only for grids of at most a block per SM (the grid FFTs' short blocks: eight),
// straight into a stream (the adjoint
// gradient's thousands of small kernels 138 -> 119 ms, a Gamma SCF's first pass 6.4 ->
// 6.1 ms in all).  Larger grids start unevenly around
// the waiting predecessor's blocks (band structure 23.4 against 25.1 ms, spinor
// SCF 21.6 against 22.7 ms), and a graph's own edges are faster than programmatic
// ones (Gamma SCF 6.4 against 6.9 ms, 64 k-points 320 against 327 ms).  Launched
// plainly, grid_dependency() does nothing.
__device__ __forceinline__ void grid_dependency() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
inline int sm_count() {
  static int n = [] {
    int dev = 0, c = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c > 0 ? c : 1;
  }();
  return n;
}

// per_sm: blocks per SM up to which a grid counts as small
inline bool programmatic_launch(dim3 grid, cudaStream_t stream, int per_sm = 1) {
  if ((long long)grid.x * grid.y * grid.z > per_sm * sm_count()) return false;
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(stream, &c) == cudaSuccess && c == cudaStreamCaptureStatusNone;
}
template <typename... P, typename... A>
void launch_with(bool programmatic, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                 A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = programmatic ? 1 : 0;
  note_launch();
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
  launch_with(programmatic_launch(grid, stream), kernel, grid, block, smem, stream, args...);
}
// Long FP64 solves want an SM to each block, which the scheduler gives them once
// the predecessor has left (a band structure of 40 k-points, whose solves doubled
// up on SMs otherwise: 23.4 against 29.1 ms)
template <typename... P, typename... A>
void launch_plain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
  launch_with(false, kernel, grid, block, smem, stream, args...);
}

// Error codes mirrored from the C ABI.
enum Status : int {
  OK = DEREK_OK,
  BAD_ARG = DEREK_ERR_BAD_ARG,
  OOM = DEREK_ERR_OOM,
  CUDA = DEREK_ERR_CUDA,
  NOT_CONVERGED = DEREK_ERR_NOT_CONVERGED,
  CHOLESKY = DEREK_ERR_CHOLESKY,
  NAN_DETECTED = DEREK_ERR_NAN,
  TIMEOUT = DEREK_ERR_TIMEOUT,
  UNSUPPORTED = DEREK_ERR_UNSUPPORTED,
};

}  // namespace derek
