// Non-collinear spinor H.psi and density.
//
// The reference's wavefunction always carries two spinor components,
// coeff(gvec, kpt, band, 1:2) (Source/wave.f90:30,164), and its potential a
// 2x2 matrix per fine-grid point, nc_pot(:, 2, 2) (Source/pot.f90:33,88),
// whose V / B decomposition Source/xsf.f90:44-51 writes as
//   nc_pot = V I + mu_B (Bx sigma_x + By sigma_y + Bz sigma_z),  mu_B = 1/2.
// Its density holds the charge and a three-component spin density,
// den%charge(nr) and den%spin(nr, 3) (Source/density.f90:63-64).  The
// products themselves are empty stubs (pot_apply_wfn, Source/pot.f90:344-382;
// density_calculate, Source/density.f90:101-130); this file defines them:
//   (H psi)_s(G) = 1/2|k+G|^2 psi_s(G) + (1/N) F[ sum_s' V_ss'(r) psi_s'(r) ](G)
//   n(r)  = sum_b w_b (|u_b|^2 + |d_b|^2)
//   m(r)  = sum_b w_b psi_b^H sigma psi_b
//         = sum_b w_b (2 Re u* d, 2 Im u* d, |u|^2 - |d|^2)
// with psi_b(r) = (u_b(r), d_b(r)) = F^-1 of the two coefficient sets.
//
// Layout: band b of a spinor system is two consecutive items, 2b (up) and
// 2b + 1 (down), with coefficient rows 2b and 2b + 1 of the k-set.  A band's
// vector is therefore one contiguous run of 2 npw_pad coefficients, so
// overlaps and rotations see a spinor band as a longer scalar band.  The
// x-line passes of hpsi4.cu run per item unchanged; only the (y,z)-plane
// pass couples the two components, so this file holds that pass (both
// components' planes in shared memory, the 2x2 product in place) and the
// density pass that accumulates n and m.
#include "fft4.cuh"
#include "kernels.cuh"

namespace derek {

// Three blocks of 192 threads per SM as in the scalar line passes (hpsi4.cu), so
// that one's transforms run beside another's products; one of 512 where two do
// not fit the shared memory.  SCF, 3 x 192 against 512 threads: FP32 35^3 11.6 /
// 17.9 ms, FP64 32^3 34.7 / 44.9 ms, 44^3 119 / 132 ms, 64^3 327 / 280 ms.
constexpr int kSpinorThreads = 192;
inline bool spinor_small(size_t smem) { return 2 * smem <= 226 * 1024; }

size_t spinor_plane_smem(int n2, int n3, size_t elem) {
  return (2 * (size_t)n2 * (n3 | 1) + (size_t)n2 + n3) * elem;
}

template <typename R>
__device__ __forceinline__ void load_lines_tw(cplx<R> *dst, const cplx<R> *src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

// Scatter the sphere columns of both components at plane x into the zeroed
// planes P0 (up) and P1 (down), then backward z (rows holding columns) and
// backward y (every column) on both.
template <typename R>
__device__ __forceinline__ void spinor_planes_backward(const Tables &t, const KSetDev &K, const SysDev &S,
                                                       const cplx<R> *a0, const cplx<R> *a1, cplx<R> *P0,
                                                       cplx<R> *P1, const cplx<R> *twy, const cplx<R> *twz) {
  const int n2 = S.n[1], n3 = S.n[2], pz = n3 | 1;
  for (int i = threadIdx.x; i < 2 * n2 * pz; i += blockDim.x) P0[i] = mk<R>(0, 0);
  __syncthreads();
  const short *cy = t.col_y + K.col_off;
  const short *cz = t.col_z + K.col_off;
  for (int c = threadIdx.x; c < K.ncol; c += blockDim.x) {
    const int o = cy[c] * pz + cz[c];
    P0[o] = a0[c];
    P1[o] = a1[c];
  }
  __syncthreads();
  const short *rows = t.rows + K.row_off;
  fft4_lines<R, +1>(P0, S.lp[2], K.nrow, pz, 1, rows, twz);
  fft4_lines<R, +1>(P1, S.lp[2], K.nrow, pz, 1, rows, twz);
  fft4_lines<R, +1>(P0, S.lp[1], n3, 1, pz, nullptr, twy);
  fft4_lines<R, +1>(P1, S.lp[1], n3, 1, pz, nullptr, twy);
}

// (y,z)-plane pass of one band (items 2q, 2q + 1 of the launch) at x-plane
// blockIdx.y: backward yz of both components, the 2x2 product, forward yz,
// columns written back in place.
template <typename R, int NT>
__global__ void __launch_bounds__(NT, NT == kSpinorThreads ? 3 : 1) k_plane_spinor(Tables t, int item_begin, cplx<R> *__restrict__ abuf,
                                                      const cplx<R> *__restrict__ vnc) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slot = 2 * blockIdx.x;
  const int item = t.item_list ? t.item_list[slot] : item_begin + slot;
  const int x = blockIdx.y;
  const KSetDev &K = t.ks[t.item_ks[item]];
  const SysDev &S = t.sys[K.sys];
  if (!S.active) return;
  const int n1 = S.n[0], n2 = S.n[1], n3 = S.n[2];
  const int b = t.item_band[item];
  if (x >= n1 || (b & 1)) return;   // b is the up component; b + 1 < K.nb is the down one
  const int pz = n3 | 1;
  cplx<R> *P0 = reinterpret_cast<cplx<R> *>(smem_raw);
  cplx<R> *P1 = P0 + n2 * pz;
  cplx<R> *twy = P1 + n2 * pz;
  cplx<R> *twz = twy + n2;
  load_lines_tw<R>(twy, twtab<R>(t) + S.lp[1].tw_off, n2);
  load_lines_tw<R>(twz, twtab<R>(t) + S.lp[2].tw_off, n3);
  const long long plane = (long long)n1 * K.ncol_pad;
  cplx<R> *a0 = abuf + K.a_off + (long long)b * plane + (long long)x * K.ncol_pad;
  cplx<R> *a1 = a0 + plane;
  spinor_planes_backward<R>(t, K, S, a0, a1, P0, P1, twy, twz);
  const cplx<R> *v = vnc + 4 * (S.grid_off + (long long)x * n2 * n3);
  // a warp per real-space row; the backward transforms left it in slot order
  for (int y = threadIdx.x >> 5; y < n2; y += blockDim.x >> 5) {
    const int sy = line_slot_of(S.lp[1], y) * pz;
    for (int z = threadIdx.x & 31; z < n3; z += 32) {
      const int o = sy + line_slot_of(S.lp[2], z);
      const cplx<R> *w = v + 4 * (y * n3 + z);
      const cplx<R> u = P0[o], d = P1[o];
      const cplx<R> v11 = w[0], v21 = w[1], v12 = w[2], v22 = w[3];
      P0[o] = cadd<R>(cmul<R>(v11, u), cmul<R>(v12, d));
      P1[o] = cadd<R>(cmul<R>(v21, u), cmul<R>(v22, d));
    }
  }
  __syncthreads();
  const short *rows = t.rows + K.row_off;
  fft4_lines<R, -1>(P0, S.lp[1], n3, 1, pz, nullptr, twy);
  fft4_lines<R, -1>(P1, S.lp[1], n3, 1, pz, nullptr, twy);
  fft4_lines<R, -1>(P0, S.lp[2], K.nrow, pz, 1, rows, twz);
  fft4_lines<R, -1>(P1, S.lp[2], K.nrow, pz, 1, rows, twz);
  const short *cy = t.col_y + K.col_off;
  const short *cz = t.col_z + K.col_off;
  for (int c = threadIdx.x; c < K.ncol; c += blockDim.x) {
    const int o = cy[c] * pz + cz[c];
    a0[c] = P0[o];
    a1[c] = P1[o];
  }
}

// Density pass per (unit, x-plane): n, mx, my, mz of the unit's bands
// with per-item weights occ (equal on both items of a band), written as four
// planes of nr values at the unit's partial grids.  Each thread owns the
// same grid points in every band, so the sums need no synchronisation.
template <typename R, int NT>
__global__ void __launch_bounds__(NT, NT == kSpinorThreads ? 3 : 1) k_density_spinor(Tables t, const DensityUnit *__restrict__ units,
                                                        const cplx<R> *__restrict__ abuf,
                                                        const double *__restrict__ occ,
                                                        double *__restrict__ partial) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const DensityUnit U = units[blockIdx.x];
  const int x = blockIdx.y;
  const KSetDev &K = t.ks[U.ks];
  const SysDev &S = t.sys[K.sys];
  if (!S.active || S.nspinor != 2) return;
  const int n1 = S.n[0], n2 = S.n[1], n3 = S.n[2];
  if (x >= n1) return;
  const int pz = n3 | 1;
  cplx<R> *P0 = reinterpret_cast<cplx<R> *>(smem_raw);
  cplx<R> *P1 = P0 + n2 * pz;
  cplx<R> *twy = P1 + n2 * pz;
  cplx<R> *twz = twy + n2;
  load_lines_tw<R>(twy, twtab<R>(t) + S.lp[1].tw_off, n2);
  load_lines_tw<R>(twz, twtab<R>(t) + S.lp[2].tw_off, n3);
  const long long nr = S.nr;
  double *dst = partial + U.off + (long long)x * n2 * n3;
  for (int i = threadIdx.x; i < n2 * n3; i += blockDim.x) {
    dst[i] = 0.0;
    dst[nr + i] = 0.0;
    dst[2 * nr + i] = 0.0;
    dst[3 * nr + i] = 0.0;
  }
  const long long plane = (long long)n1 * K.ncol_pad;
  for (int b = 2 * U.g; b + 1 < K.nb; b += 2 * U.ng) {
    const double w = occ[K.item0 + b];
    if (w == 0.0) continue;
    __syncthreads();   // the previous band's planes are read to the end
    const cplx<R> *a0 = abuf + K.a_off + (long long)b * plane + (long long)x * K.ncol_pad;
    spinor_planes_backward<R>(t, K, S, a0, a0 + plane, P0, P1, twy, twz);
    for (int i = threadIdx.x; i < n2 * n3; i += blockDim.x) {
      const int y = i / n3, z = i - y * n3;
      const int o = line_slot_of(S.lp[1], y) * pz + line_slot_of(S.lp[2], z);
      const cplx<R> u = P0[o], d = P1[o];
      const double ux = u.x, uy = u.y, dx = d.x, dy = d.y;
      const double uu = ux * ux + uy * uy, dd = dx * dx + dy * dy;
      dst[i] += w * (uu + dd);
      dst[nr + i] += 2.0 * w * (ux * dx + uy * dy);
      dst[2 * nr + i] += 2.0 * w * (ux * dy - uy * dx);
      dst[3 * nr + i] += w * (uu - dd);
    }
  }
}

template <typename R>
void launch_plane_spinor(const Tables &t, int item_begin, int nitems, const int n[3], int max_m, cplx<R> *abuf,
                         const cplx<R> *vnc, cudaStream_t st) {
  if (nitems <= 1) return;
  if constexpr (std::is_same<R, float>::value) {
    if (launch_plane_spinor_reg(t, item_begin, nitems, n, max_m, abuf, vnc, st)) return;
  }
  const size_t sm = spinor_plane_smem(n[1], n[2], sizeof(cplx<R>));
  auto go = [&](auto kern, int threads) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    derek::launch(kern, dim3(nitems / 2, n[0]), threads, sm, st, t, item_begin, abuf, vnc);
  };
  if (spinor_small(sm))
    go(k_plane_spinor<R, kSpinorThreads>, kSpinorThreads);
  else
    go(k_plane_spinor<R, 512>, 512);
}

template <typename R>
void launch_density_spinor(const Tables &t, const DensityUnit *units, int nunits, const int n[3],
                           const cplx<R> *abuf, const double *occ, double *partial, cudaStream_t st) {
  if (nunits <= 0) return;
  const size_t sm = spinor_plane_smem(n[1], n[2], sizeof(cplx<R>));
  auto go = [&](auto kern, int threads) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    derek::launch(kern, dim3(nunits, n[0]), threads, sm, st, t, units, abuf, occ, partial);
  };
  if (spinor_small(sm))
    go(k_density_spinor<R, kSpinorThreads>, kSpinorThreads);
  else
    go(k_density_spinor<R, 512>, 512);
}

#define DEREK_INST(R)                                                                                  \
  template void launch_plane_spinor<R>(const Tables &, int, int, const int *, int, cplx<R> *, const cplx<R> *, \
                                       cudaStream_t);                                                  \
  template void launch_density_spinor<R>(const Tables &, const DensityUnit *, int, const int *,        \
                                         const cplx<R> *, const double *, double *, cudaStream_t);
DEREK_INST(float)
DEREK_INST(double)
#undef DEREK_INST

}  // namespace derek
