// Wavefunction slices between the caller's layout and the library's.
//
// The caller holds complex128 [nspinor][bands][npw] in the reference's G order
// (coeff(gvec, band, spinor) of one k-point); the device holds padded rows in
// column order, in the handle's precision, band b's spinor s at row
// nspinor b + s.  The caller's rows cross as they are (the link moves them at
// about 170 GB/s, from pageable memory too) and the reordering and conversion
// run here: on the host they took far longer than the copy (80 bands x 17,529
// plane waves: set_wfn + apply_h 2.9 ms, now 0.42 ms with 0.15 ms of H.psi).
#include "kernels.cuh"

namespace derek {

// device row of the caller's row r
__device__ __forceinline__ int device_row(int r, int nrows, int nsp) {
  const int nb = nrows / nsp;
  return nsp == 1 ? r : 2 * (r % nb) + r / nb;
}

// the caller's rows [row0, row0 + gridDim.y) of a slice of nrows, held at src
template <typename R>
__global__ void __launch_bounds__(256) k_wfn_in(const double2 *__restrict__ src, const int *__restrict__ perm, int npw,
                                                int npw_pad, int row0, int nrows, int nsp, cplx<R> *__restrict__ dst) {
  grid_dependency();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= npw_pad) return;
  cplx<R> v = mk<R>(0, 0);
  if (g < npw) {
    const double2 s = src[(long long)blockIdx.y * npw + perm[g]];
    v = mk<R>((R)s.x, (R)s.y);
  }
  dst[(long long)device_row(row0 + blockIdx.y, nrows, nsp) * npw_pad + g] = v;
}

template <typename R>
__global__ void __launch_bounds__(256) k_wfn_out(const cplx<R> *__restrict__ src, const int *__restrict__ perm,
                                                 int npw, int npw_pad, int row0, int nrows, int nsp,
                                                 double2 *__restrict__ dst) {
  grid_dependency();
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= npw) return;
  const cplx<R> s = src[(long long)device_row(row0 + blockIdx.y, nrows, nsp) * npw_pad + g];
  dst[(long long)blockIdx.y * npw + perm[g]] = make_double2((double)s.x, (double)s.y);
}

void launch_wfn_in(int fp64, const double2 *src, const int *perm, const KSetDev &K, int nsp, int row0, int count,
                   void *dst, cudaStream_t st) {
  const dim3 grid((K.npw_pad + 255) / 256, count);
  if (fp64)
    derek::launch(k_wfn_in<double>, grid, 256, 0, st, src, perm, K.npw, K.npw_pad, row0, K.nbr, nsp, (double2 *)dst);
  else
    derek::launch(k_wfn_in<float>, grid, 256, 0, st, src, perm, K.npw, K.npw_pad, row0, K.nbr, nsp, (float2 *)dst);
}

void launch_wfn_out(int fp64, const void *src, const int *perm, const KSetDev &K, int nsp, int row0, int count,
                    double2 *dst, cudaStream_t st) {
  const dim3 grid((K.npw + 255) / 256, count);
  if (fp64)
    derek::launch(k_wfn_out<double>, grid, 256, 0, st, (const double2 *)src, perm, K.npw, K.npw_pad, row0, K.nbr, nsp, dst);
  else
    derek::launch(k_wfn_out<float>, grid, 256, 0, st, (const float2 *)src, perm, K.npw, K.npw_pad, row0, K.nbr, nsp, dst);
}

}  // namespace derek
