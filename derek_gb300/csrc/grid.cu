// Fine-grid kernels: full 3D FFT of density-like grids and the LDA
// exchange-correlation evaluation.
#include "fft_smem.cuh"
#include "kernels.cuh"
#include "metric.cuh"
#include "xc.cuh"

namespace derek {

// A 3D transform is three passes of one axis each, over tiles of lines small
// enough that every pass of one small grid has more blocks than the GPU has
// SMs (a block per (y,z) plane and one per (x,z) plane kept 32 SMs busy on 32^3).
// Real grids go through half spectra, kz <= n3/2 at its own place in the grid's
// storage: two real rows share one complex z transform, and the y and x passes
// see half the columns.  The x pass of a convolution transforms forward,
// multiplies and transforms back without leaving the block.
// Bound by FP64 issue.  Measured: V_H[n] (both directions) of 32^3 71 -> 53 us, of 24
// systems up to 72^3 1.67 -> 0.88 ms; complex 3D transform of 32^3 33 -> 27 us.
constexpr int kGridThreads = 128;
constexpr int kRowTile = 4;   // z transforms of a block

__device__ __forceinline__ void load_plan_tw(double2 *tw, const Tables &t, const FftPlan &p) {
  for (int i = threadIdx.x; i < p.n; i += blockDim.x) tw[i] = t.tw64[p.tw_off + i];
}

// z pass, complex rows in place
template <int SIGN>
__global__ void __launch_bounds__(kGridThreads) k_rows(Tables t, int sys_begin, double2 *__restrict__ data) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SysDev &S = t.sys[sys_begin + blockIdx.y];
  const int n3 = S.n[2], rows = S.n[0] * S.n[1], l0 = blockIdx.x * kRowTile;
  if (l0 >= rows) return;
  const int nl = min(kRowTile, rows - l0), ld = n3 | 1;
  double2 *bufA = reinterpret_cast<double2 *>(smem_raw), *bufB = bufA + kRowTile * ld, *tw = bufB + kRowTile * ld;
  load_plan_tw(tw, t, S.plan[2]);
  double2 *g = data + S.grid_off + (long long)l0 * n3;
  for (int i = threadIdx.x; i < nl * n3; i += blockDim.x) bufA[(i / n3) * ld + i % n3] = g[i];
  __syncthreads();
  const double2 *res = fft_lines<double, SIGN, false>(bufA, bufB, S.plan[2], nl, ld, 1, tw, nullptr);
  for (int i = threadIdx.x; i < nl * n3; i += blockDim.x) g[i] = res[(i / n3) * ld + i % n3];
}

// z pass of a real grid, forward: rows 2 l and 2 l + 1 as one complex row
// Z = A + i B; A(k) = (Z(k) + conj Z(-k)) / 2, B(k) = (Z(k) - conj Z(-k)) / 2i
__global__ void __launch_bounds__(kGridThreads) k_rows_r2c(Tables t, const double *__restrict__ rho,
                                                           double2 *__restrict__ data, int all) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SysDev &S = t.sys[blockIdx.y];
  if (!all && !S.active) return;
  const int n3 = S.n[2], rows = S.n[0] * S.n[1], l0 = blockIdx.x * kRowTile, pairs = (rows + 1) / 2;
  if (l0 >= pairs) return;
  const int nl = min(kRowTile, pairs - l0), ld = n3 | 1, nh = n3 / 2 + 1;
  double2 *bufA = reinterpret_cast<double2 *>(smem_raw), *bufB = bufA + kRowTile * ld, *tw = bufB + kRowTile * ld;
  load_plan_tw(tw, t, S.plan[2]);
  const double *src = rho + S.grid_off;
  for (int i = threadIdx.x; i < nl * n3; i += blockDim.x) {
    const int l = i / n3, z = i - l * n3, r = 2 * (l0 + l);
    bufA[l * ld + z] = make_double2(src[(long long)r * n3 + z], r + 1 < rows ? src[(long long)(r + 1) * n3 + z] : 0.0);
  }
  __syncthreads();
  const double2 *res = fft_lines<double, -1, false>(bufA, bufB, S.plan[2], nl, ld, 1, tw, nullptr);
  double2 *g = data + S.grid_off;
  for (int i = threadIdx.x; i < nl * nh; i += blockDim.x) {
    const int l = i / nh, k = i - l * nh, r = 2 * (l0 + l);
    const double2 p = res[l * ld + k], q = res[l * ld + (k ? n3 - k : 0)];
    g[(long long)r * n3 + k] = make_double2(0.5 * (p.x + q.x), 0.5 * (p.y - q.y));
    if (r + 1 < rows) g[(long long)(r + 1) * n3 + k] = make_double2(0.5 * (p.y + q.y), 0.5 * (q.x - p.x));
  }
}

// z pass back to a real grid: Z(k) = A(k) + i B(k), Z(-k) = conj A(k) + i conj B(k);
// the self-conjugate k (0, n3/2) contribute their real parts.  ADD: out += it.
template <bool ADD>
__global__ void __launch_bounds__(kGridThreads) k_rows_c2r(Tables t, const double2 *__restrict__ data,
                                                           double *__restrict__ out, int all) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SysDev &S = t.sys[blockIdx.y];
  if (!all && !S.active) return;
  const int n3 = S.n[2], rows = S.n[0] * S.n[1], l0 = blockIdx.x * kRowTile, pairs = (rows + 1) / 2;
  if (l0 >= pairs) return;
  const int nl = min(kRowTile, pairs - l0), ld = n3 | 1, nh = n3 / 2 + 1;
  double2 *bufA = reinterpret_cast<double2 *>(smem_raw), *bufB = bufA + kRowTile * ld, *tw = bufB + kRowTile * ld;
  load_plan_tw(tw, t, S.plan[2]);
  const double2 *g = data + S.grid_off;
  for (int i = threadIdx.x; i < nl * nh; i += blockDim.x) {
    const int l = i / nh, k = i - l * nh, r = 2 * (l0 + l);
    double2 p = g[(long long)r * n3 + k], q = make_double2(0.0, 0.0);
    if (r + 1 < rows) q = g[(long long)(r + 1) * n3 + k];
    if (k == 0 || 2 * k == n3) {
      bufA[l * ld + k] = make_double2(p.x, q.x);
    } else {
      bufA[l * ld + k] = make_double2(p.x - q.y, p.y + q.x);
      bufA[l * ld + n3 - k] = make_double2(p.x + q.y, q.x - p.y);
    }
  }
  __syncthreads();
  const double2 *res = fft_lines<double, +1, false>(bufA, bufB, S.plan[2], nl, ld, 1, tw, nullptr);
  double *dst = out + S.grid_off;
  for (int i = threadIdx.x; i < nl * n3; i += blockDim.x) {
    const int l = i / n3, z = i - l * n3, r = 2 * (l0 + l);
    const double2 v = res[l * ld + z];
    double *d = dst + (long long)r * n3 + z;
    d[0] = ADD ? d[0] + v.x : v.x;
    if (r + 1 < rows) d[n3] = ADD ? d[n3] + v.y : v.y;
  }
}

// y pass: columns z0 .. z0 + tz of plane x (half: of the kz <= n3/2 half)
template <int SIGN>
__global__ void __launch_bounds__(kGridThreads) k_cols_y(Tables t, int sys_begin, double2 *__restrict__ data, int tz,
                                                         int half, int all) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SysDev &S = t.sys[sys_begin + blockIdx.z];
  const int n2 = S.n[1], n3 = S.n[2], nz = half ? n3 / 2 + 1 : n3, x = blockIdx.y, z0 = blockIdx.x * tz;
  if ((!all && !S.active) || x >= S.n[0] || z0 >= nz) return;
  const int nl = min(tz, nz - z0);
  double2 *bufA = reinterpret_cast<double2 *>(smem_raw), *bufB = bufA + n2 * tz, *tw = bufB + n2 * tz;
  load_plan_tw(tw, t, S.plan[1]);
  double2 *g = data + S.grid_off + (long long)x * n2 * n3 + z0;
  for (int i = threadIdx.x; i < n2 * nl; i += blockDim.x) bufA[(i / nl) * tz + i % nl] = g[(long long)(i / nl) * n3 + i % nl];
  __syncthreads();
  const double2 *res = fft_lines<double, SIGN, true>(bufA, bufB, S.plan[1], nl, 1, tz, tw, nullptr);
  for (int i = threadIdx.x; i < n2 * nl; i += blockDim.x) g[(long long)(i / nl) * n3 + i % nl] = res[(i / nl) * tz + i % nl];
}

// x pass: columns z0 .. of row y.  MODE 0: one direction; kHartree and kKerker:
// forward, times the factor of G, backward (half spectra).  A real result's
// factor is the mean over G and its conjugate partner: the two differ where a
// component sits at the Nyquist index of a sheared cell.
enum { kPlain = 0, kHartree = 1, kKerker = 2 };
template <int SIGN, int MODE>
__global__ void __launch_bounds__(kGridThreads) k_cols_x(Tables t, int sys_begin, double2 *__restrict__ data, int tz,
                                                         int half, int all, double alpha, double q0) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SysDev &S = t.sys[sys_begin + blockIdx.z];
  const int n1 = S.n[0], n2 = S.n[1], n3 = S.n[2], nz = half ? n3 / 2 + 1 : n3, y = blockIdx.y, z0 = blockIdx.x * tz;
  if ((!all && !S.active) || y >= n2 || z0 >= nz) return;
  const int nl = min(tz, nz - z0);
  double2 *bufA = reinterpret_cast<double2 *>(smem_raw), *bufB = bufA + n1 * tz, *tw = bufB + n1 * tz;
  load_plan_tw(tw, t, S.plan[0]);
  const long long xs = (long long)n2 * n3;
  double2 *g = data + S.grid_off + (long long)y * n3 + z0;
  for (int i = threadIdx.x; i < n1 * nl; i += blockDim.x) bufA[(i / nl) * tz + i % nl] = g[(i / nl) * xs + i % nl];
  __syncthreads();
  double2 *res = fft_lines<double, SIGN, true>(bufA, bufB, S.plan[0], nl, 1, tz, tw, nullptr);
  if constexpr (MODE != kPlain) {
    const Metric metric(S);
    const double invn = 1.0 / S.nr;
    for (int i = threadIdx.x; i < n1 * nl; i += blockDim.x) {
      const int x = i / nl, k = z0 + i % nl;
      auto factor = [&](int ix, int iy, int iz) {
        const double g2 = metric.gsq(S, ix, iy, iz);
        if constexpr (MODE == kHartree) return g2 > 0 ? 12.566370614359172953850573533118 * invn / g2 : 0.0;
        return alpha * g2 / (g2 + q0 * q0) * invn;
      };
      double f = factor(x, y, k);
      if (2 * x == n1 || 2 * y == n2 || 2 * k == n3)
        f = 0.5 * (f + factor(x ? n1 - x : 0, y ? n2 - y : 0, k ? n3 - k : 0));
      double2 &c = res[(i / nl) * tz + i % nl];
      c.x *= f;
      c.y *= f;
    }
    __syncthreads();
    res = fft_lines<double, -SIGN, true>(res, res == bufA ? bufB : bufA, S.plan[0], nl, 1, tz, tw, nullptr);
  }
  for (int i = threadIdx.x; i < n1 * nl; i += blockDim.x) g[(i / nl) * xs + i % nl] = res[(i / nl) * tz + i % nl];
}

namespace {

// launch shape of the passes over systems [.., nsys) with axes up to max_n
struct GridShape {
  int tz, nsys, max_n;
  size_t cols, rows;
  dim3 col_grid(int half) const { return dim3(((half ? max_n / 2 + 1 : max_n) + tz - 1) / tz, max_n, nsys); }
  dim3 row_grid(int real) const {
    const int lines = real ? (max_n * max_n + 1) / 2 : max_n * max_n;
    return dim3((lines + kRowTile - 1) / kRowTile, nsys);
  }
  GridShape(int ns, int n) : nsys(ns), max_n(n) {
    // 128-byte runs of a column tile, 64-byte ones where the wider tile would
    // leave SMs without a block
    tz = (long long)ns * n * ((n + 7) / 8) >= 4 * sm_count() ? 8 : 4;
    cols = (2 * (size_t)n * tz + n) * sizeof(double2);
    rows = (2 * (size_t)kRowTile * (n | 1) + n) * sizeof(double2);
  }
};

// The passes are a chain of short kernels with all their blocks resident at once
// up to 8 per SM, so each starts beside its predecessor (common.cuh): a 32^3 grid
// forward and back through the ABI 178 -> 174 us.  The shared-memory limit is raised
// only for lines that need it (the call is host time before every launch).
template <typename... P, typename... A>
void grid_pass(void (*kernel)(P...), dim3 grid, size_t smem, cudaStream_t st, A &&...args) {
  if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  derek::launch_with(derek::programmatic_launch(grid, st, 8), kernel, grid, kGridThreads, smem, st, args...);
}

template <int SIGN> void cols_y(const GridShape &g, const Tables &t, int s0, double2 *data, int half, int all, cudaStream_t st) {
  grid_pass(k_cols_y<SIGN>, g.col_grid(half), g.cols, st, t, s0, data, g.tz, half, all);
}
template <int SIGN, int MODE>
void cols_x(const GridShape &g, const Tables &t, int s0, double2 *data, int half, int all, double alpha, double q0,
            cudaStream_t st) {
  grid_pass(k_cols_x<SIGN, MODE>, g.col_grid(half), g.cols, st, t, s0, data, g.tz, half,
                                                                                            all, alpha, q0);
}
void rows_r2c(const GridShape &g, const Tables &t, const double *rho, double2 *data, int all, cudaStream_t st) {
  grid_pass(k_rows_r2c, g.row_grid(1), g.rows, st, t, rho, data, all);
}
template <bool ADD> void rows_c2r(const GridShape &g, const Tables &t, const double2 *data, double *out, int all, cudaStream_t st) {
  grid_pass(k_rows_c2r<ADD>, g.row_grid(1), g.rows, st, t, data, out, all);
}

}  // namespace

void launch_fft3d_grid(const Tables &t, int sys_begin, int nsys, int max_n, double2 *data, int sign,
                       cudaStream_t st) {
  if (nsys <= 0) return;
  const GridShape g(nsys, max_n);
  if (sign < 0) {
    grid_pass(k_rows<-1>, g.row_grid(0), g.rows, st, t, sys_begin, data);
    cols_y<-1>(g, t, sys_begin, data, 0, 1, st);
    cols_x<-1, kPlain>(g, t, sys_begin, data, 0, 1, 0.0, 0.0, st);
  } else {
    grid_pass(k_rows<1>, g.row_grid(0), g.rows, st, t, sys_begin, data);
    cols_y<1>(g, t, sys_begin, data, 0, 1, st);
    cols_x<1, kPlain>(g, t, sys_begin, data, 0, 1, 0.0, 0.0, st);
  }
}

void launch_real_spectrum(const Tables &t, int nsys, int max_n, const double *rho, double2 *work, cudaStream_t st) {
  if (nsys <= 0) return;
  const GridShape g(nsys, max_n);
  rows_r2c(g, t, rho, work, 0, st);
  cols_y<-1>(g, t, 0, work, 1, 0, st);
  cols_x<-1, kPlain>(g, t, 0, work, 1, 0, 0.0, 0.0, st);
}

void launch_hartree(const Tables &t, int nsys, int max_n, const double *rho, double2 *work, double *vh, int all,
                    cudaStream_t st) {
  if (nsys <= 0) return;
  const GridShape g(nsys, max_n);
  rows_r2c(g, t, rho, work, all, st);
  cols_y<-1>(g, t, 0, work, 1, all, st);
  cols_x<-1, kHartree>(g, t, 0, work, 1, all, 0.0, 0.0, st);
  cols_y<1>(g, t, 0, work, 1, all, st);
  rows_c2r<false>(g, t, work, vh, all, st);
}

void launch_kerker_add(const Tables &t, int nsys, int max_n, const double *res, double2 *work, double alpha, double q0,
                       double *rho, cudaStream_t st) {
  if (nsys <= 0) return;
  const GridShape g(nsys, max_n);
  rows_r2c(g, t, res, work, 0, st);
  cols_y<-1>(g, t, 0, work, 1, 0, st);
  cols_x<-1, kKerker>(g, t, 0, work, 1, 0, alpha, q0, st);
  cols_y<1>(g, t, 0, work, 1, 0, st);
  rows_c2r<true>(g, t, work, rho, 0, st);
}

__global__ void k_lda(long n, const double *__restrict__ rho, double *__restrict__ exc,
                      double *__restrict__ vxc) {
  grid_dependency();
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double e, v;
    lda_point(rho[i], e, v);
    if (exc) exc[i] = e;
    if (vxc) vxc[i] = v;
  }
}

void launch_lda(long n, const double *rho, double *exc, double *vxc, cudaStream_t st) {
  if (n <= 0) return;
  long blocks = (n + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  derek::launch(k_lda, (int)blocks, 256, 0, st, n, rho, exc, vxc);
}

}  // namespace derek
