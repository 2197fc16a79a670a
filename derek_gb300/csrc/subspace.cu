// Subspace kernels of the Chebyshev-filtered subspace iteration:
//   overlaps  A^H B (split-K, batched over k-sets)        -> FP64 matrices
//   rotation  X <- X C (in place, batched over k-sets)
//   Cholesky of the overlap and the inverse factor C = L^-H (FP64)
//   Hermitian Jacobi eigensolver of the projected Hamiltonian (FP64)
// These replace the empty wave_dot_* routines (Source/wave.f90:929-1036)
// with the full matrices a Rayleigh-Ritz step needs.
#include <algorithm>
#include <cstdio>

#include "subspace.cuh"

#include <cooperative_groups.h>

namespace derek {

// acc += a b as four fused multiply-adds.  (acc.x += a.x b.x - a.y b.y compiles
// to a product, a fused multiply-add and an addition: three slots of the pipe
// per component instead of two.)
__device__ __forceinline__ double fmadd(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fmadd(float a, float b, float c) { return fmaf(a, b, c); }
template <typename R> __device__ __forceinline__ void cmac(cplx<R> &acc, cplx<R> a, cplx<R> b) {
  acc.x = fmadd(a.x, b.x, acc.x);
  acc.y = fmadd(a.x, b.y, acc.y);
  acc.x = fmadd(-a.y, b.y, acc.x);
  acc.y = fmadd(a.y, b.x, acc.y);
}

// ---------------------------------------------------------------------------
// Overlap: part[ks][split] = sum_{G in split} conj(A_i(G)) B_j(G)
//
// Bound by the FP64 pipe (GB300: 2 lanes per clock and SM, and a warp
// instruction costs its 16 clocks however few of its lanes are active) or, in
// FP32, by shared-memory loads.  So the unit of work is one MT x MT tile of
// band pairs and the tiles of a k-set are numbered one after another and dealt
// to the threads (P per thread): no lane idles on a band count that is no
// multiple of a tile, and A = B computes the upper triangle only (the lower
// one is its exact conjugate).  Every block stages OKC coefficients of all
// bands.  The split along G is as fine as it takes to give every SM blocks
// (launch_overlap).  Measured, FP64: 12 bands x 1,510 plane waves 716 -> 12 us
// (A = B) and 15 us; 84 bands x 17,529 on 4 k-points 8.2 -> 1.7 ms (A = B) and
// 3.7 ms (1.0 and 2.0 x 10^9 multiply-adds at the pipe's rate: 1.6 and 3.2 ms).
// ---------------------------------------------------------------------------
template <typename R> struct OverlapShape;
// FP64: one pair per tile, its four fused multiply-adds hide both loads
template <> struct OverlapShape<double> {
  static constexpr int MT = 1, OKC = 16, PMAX = 8;
};
// FP32: 2 x 2 pairs, half the shared loads per multiply-add; short chunks, whose
// sums are rounded on their own (an SCF's free energy at its FP32 noise floor
// moves by 1.9e-7 Ha per iteration, 3.8e-7 with one running sum)
template <> struct OverlapShape<float> {
  static constexpr int MT = 2, OKC = 16, PMAX = 4;
};

template <typename R, int P, bool SAME>
__global__ void __launch_bounds__(256) k_overlap_pairs(const Tables t, int ks_begin,
                                                       const cplx<R> *__restrict__ A,
                                                       const cplx<R> *__restrict__ B,
                                                       double2 *__restrict__ part,
                                                       const long long *__restrict__ part_off,
                                                       int ksplit) {
  grid_dependency();
  constexpr int MT = OverlapShape<R>::MT, OKC = OverlapShape<R>::OKC, LD = OKC + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ksi = ks_begin + blockIdx.z;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;
  const int nb = K.nb;
  const int nt = (nb + MT - 1) / MT, rows = nt * MT;
  const int np = SAME ? nt * (nt + 1) / 2 : nt * nt;
  const int p0 = blockIdx.x * blockDim.x * P;
  const int g0 = blockIdx.y * ksplit;
  if (p0 >= np || g0 >= K.npw) return;
  const int g1 = min(K.npw, g0 + ksplit);
  cplx<R> *As = reinterpret_cast<cplx<R> *>(smem_raw);   // [rows][LD]
  cplx<R> *Bs = SAME ? As : As + rows * LD;
  const cplx<R> *Ab = A + K.psi_off;
  const cplx<R> *Bb = B + K.psi_off;
  int oi[P], oj[P];   // shared rows of the thread's tiles (-1: none)
  cplx<R> acc[P][MT][MT];
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const int p = p0 + (int)threadIdx.x + q * (int)blockDim.x;
    oi[q] = oj[q] = -1;
    if (p < np) {
      int i, j;
      if (SAME) {
        // row i of the upper triangle starts at i nt - i (i - 1) / 2
        const float w = 2.f * nt + 1.f;
        i = min(nt - 1, max(0, (int)(0.5f * (w - sqrtf(fmaxf(w * w - 8.f * p, 0.f))))));
        while (i * nt - i * (i - 1) / 2 > p) --i;
        while ((i + 1) * nt - (i + 1) * i / 2 <= p) ++i;
        j = i + p - (i * nt - i * (i - 1) / 2);
      } else {
        i = p / nt;
        j = p - i * nt;
      }
      oi[q] = i * MT * LD;
      oj[q] = j * MT * LD;
    }
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
      for (int b = 0; b < MT; ++b) acc[q][a][b] = mk<R>(0, 0);
  }
  for (int k0 = g0; k0 < g1; k0 += OKC) {
    for (int e = threadIdx.x; e < rows * OKC; e += blockDim.x) {
      const int r = e / OKC, c = e % OKC;
      const int g = k0 + c;
      const bool in = r < nb && g < g1;
      As[r * LD + c] = in ? Ab[(long long)r * K.npw_pad + g] : mk<R>(0, 0);
      if (!SAME) Bs[r * LD + c] = in ? Bb[(long long)r * K.npw_pad + g] : mk<R>(0, 0);
    }
    __syncthreads();
    // FP32 sums in two levels, the chunk's products first: the rounding of a
    // long running sum is what the Ritz values' noise comes from
    cplx<R> sum[P][MT][MT];
#pragma unroll
    for (int q = 0; q < P; ++q)
#pragma unroll
      for (int u = 0; u < MT; ++u)
#pragma unroll
        for (int v = 0; v < MT; ++v) sum[q][u][v] = std::is_same<R, float>::value ? mk<R>(0, 0) : acc[q][u][v];
#pragma unroll 2
    for (int c = 0; c < OKC; ++c) {
#pragma unroll
      for (int q = 0; q < P; ++q) {
        if (oi[q] < 0) continue;
        cplx<R> a[MT], b[MT];
#pragma unroll
        for (int u = 0; u < MT; ++u) {
          a[u] = As[oi[q] + u * LD + c];
          b[u] = Bs[oj[q] + u * LD + c];
        }
#pragma unroll
        for (int u = 0; u < MT; ++u)
#pragma unroll
          for (int v = 0; v < MT; ++v) {
            // conj(a) b: conjugate of a on the left factor
            cmac<R>(sum[q][u][v], mk<R>(a[u].x, -a[u].y), b[v]);
          }
      }
    }
#pragma unroll
    for (int q = 0; q < P; ++q)
#pragma unroll
      for (int u = 0; u < MT; ++u)
#pragma unroll
        for (int v = 0; v < MT; ++v)
          acc[q][u][v] = std::is_same<R, float>::value ? cadd<R>(acc[q][u][v], sum[q][u][v]) : sum[q][u][v];
    __syncthreads();
  }
  double2 *dst = part + part_off[ksi] + (long long)blockIdx.y * nb * nb;
#pragma unroll
  for (int q = 0; q < P; ++q) {
    if (oi[q] < 0) continue;
    const int i0 = oi[q] / LD, j0 = oj[q] / LD;
#pragma unroll
    for (int u = 0; u < MT; ++u)
#pragma unroll
      for (int v = 0; v < MT; ++v)
        if (i0 + u < nb && j0 + v < nb)
          dst[(i0 + u) * nb + j0 + v] = make_double2((double)acc[q][u][v].x, (double)acc[q][u][v].y);
  }
}

// Sum of the splits, one pair (i, j), i <= j, by kReduceLanes lanes: each adds
// every kReduceLanes-th split, then a fixed shuffle tree (one thread per pair
// waited on a chain of up to ~50 dependent FP64 additions, 23 us at 12 bands).
// half: only the upper triangle was computed, the matrix is Hermitian by
// construction; hermitize: the mean of the two triangles.
constexpr int kReduceLanes = 8;
__global__ void __launch_bounds__(256) k_overlap_reduce(const Tables t, int ks_begin, const double2 *__restrict__ part,
                                                        const long long *__restrict__ part_off, int ksplit,
                                                        double2 *__restrict__ out,
                                                        const long long *__restrict__ mat_off, int hermitize,
                                                        int half) {
  grid_dependency();
  const int ksi = ks_begin + blockIdx.x;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;
  const int nb = K.nb;
  const int lane = threadIdx.x % kReduceLanes;
  const int e = (blockIdx.y * blockDim.x + threadIdx.x) / kReduceLanes;
  const int i = e / nb, j = e - i * nb;
  const bool on = e < nb * nb && i <= j;
  const int nsplit = (K.npw + ksplit - 1) / ksplit;
  const double2 *src = part + part_off[ksi];
  const int f = j * nb + i;
  const bool lower = on && !half && i < j;
  double2 u = make_double2(0, 0), l = make_double2(0, 0);
#pragma unroll 4
  for (int s = lane; s < (on ? nsplit : 0); s += kReduceLanes) {
    const double2 v = src[(long long)s * nb * nb + e];
    u.x += v.x;
    u.y += v.y;
    if (lower) {
      const double2 w = src[(long long)s * nb * nb + f];
      l.x += w.x;
      l.y += w.y;
    }
  }
#pragma unroll
  for (int w = kReduceLanes / 2; w > 0; w >>= 1) {
    u.x += __shfl_down_sync(0xffffffffu, u.x, w, kReduceLanes);
    u.y += __shfl_down_sync(0xffffffffu, u.y, w, kReduceLanes);
    l.x += __shfl_down_sync(0xffffffffu, l.x, w, kReduceLanes);
    l.y += __shfl_down_sync(0xffffffffu, l.y, w, kReduceLanes);
  }
  if (!on || lane) return;
  double2 *M = out + mat_off[ksi];
  if (i == j) {
    M[e] = make_double2(u.x, hermitize || half ? 0.0 : u.y);
  } else if (half) {
    M[e] = u;
    M[f] = make_double2(u.x, -u.y);
  } else if (hermitize) {
    const double2 h = make_double2(0.5 * (u.x + l.x), 0.5 * (u.y - l.y));
    M[e] = h;
    M[f] = make_double2(h.x, -h.y);
  } else {
    M[e] = u;
    M[f] = l;
  }
}

// ---------------------------------------------------------------------------
// Rotation: X[:, j] <- sum_i X[:, i] C[i][j], in place per G tile.  upper: C is
// upper triangular (the Cholesky factor L^-H), rows i > j are left out.
// A lane holds a G, a warp a set of output bands j, so C is read as a
// broadcast.  JQ is the number of bands per thread the widest subspace needs:
// with room for 128 bands whatever the subspace, predicated-off multiply-adds
// of the missing bands cost as much of the pipe as real ones.
// ---------------------------------------------------------------------------
constexpr int RG = 32;      // G columns per tile
constexpr int RWARPS = 8;
constexpr int RROWS = 8;    // rows of C staged at a time (FP64), skip unit of upper

// FP64: bound by the FP64 pipe.  The whole X tile sits in shared memory, C
// passes through it in chunks of RROWS rows; warp w holds bands w, w + 8, ...
// Measured, 84 bands x 17,529 on 4 k-points: 8.6 -> 3.3 ms full, 1.8 ms upper
// (pipe time 3.2 and 1.6 ms).
template <int JQ>
__global__ void __launch_bounds__(256, 2) k_rotate64(const Tables t, int ks_begin, double2 *__restrict__ X,
                                                     const double2 *__restrict__ C,
                                                     const long long *__restrict__ mat_off, int upper) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ksi = ks_begin + blockIdx.y;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;
  const int g0 = blockIdx.x * RG, npw = K.npw, nb = K.nb;
  if (g0 >= npw) return;
  double2 *Xs = reinterpret_cast<double2 *>(smem_raw);   // [nb][RG]
  double2 *Cs = Xs + nb * RG;                            // [RROWS][nb]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double2 *Xb = X + K.psi_off;
  const double2 *Cb = C + mat_off[ksi];
  for (int r = w; r < nb; r += RWARPS)
    Xs[r * RG + lane] = g0 + lane < npw ? Xb[(long long)r * K.npw_pad + g0 + lane] : make_double2(0.0, 0.0);
  double2 acc[JQ];
#pragma unroll
  for (int q = 0; q < JQ; ++q) acc[q] = make_double2(0.0, 0.0);
  for (int r0 = 0; r0 < nb; r0 += RROWS) {
    const int nr = min(RROWS, nb - r0);
    for (int e = threadIdx.x; e < nr * nb; e += blockDim.x) Cs[e] = Cb[(long long)r0 * nb + e];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < JQ; ++q) {
      const int j = w + RWARPS * q;
      if (j >= nb || (upper && j < r0)) continue;
      for (int r = 0; r < nr; ++r) {
        const double2 x = Xs[(r0 + r) * RG + lane], c = Cs[r * nb + j];
        cmac<double>(acc[q], x, c);
      }
    }
    __syncthreads();
  }
  if (g0 + lane < npw) {
#pragma unroll
    for (int q = 0; q < JQ; ++q) {
      const int j = w + RWARPS * q;
      if (j < nb) Xb[(long long)j * K.npw_pad + g0 + lane] = acc[q];
    }
  }
}

// FP32, bound by shared-memory loads and multiply-adds alike: C is converted once per block into shared memory (FP64-to-FP32
// conversions run on the FP64 pipe; per 32 columns they took as long as the
// product itself) and the block walks G tiles of 64.  A thread holds two G and
// the band pairs 2 (w + 8 q) + {0, 1}: one 16-byte broadcast of C per four
// complex products.
template <int JQ>
__global__ void __launch_bounds__(256, 2) k_rotate32(const Tables t, int ks_begin, float2 *__restrict__ X,
                                                     const double2 *__restrict__ C,
                                                     const long long *__restrict__ mat_off, int upper) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ksi = ks_begin + blockIdx.y;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;
  constexpr int TG = 2 * RG;
  const int npw = K.npw, nb = K.nb, ldc = (nb + 1) & ~1;
  if ((int)blockIdx.x * TG >= npw) return;
  float2 *Cs = reinterpret_cast<float2 *>(smem_raw);   // [nb][ldc]
  float2 *Xs = Cs + nb * ldc;                          // [nb][TG]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  float2 *Xb = X + K.psi_off;
  const double2 *Cb = C + mat_off[ksi];
  for (int r = w; r < nb; r += RWARPS)
    for (int c = lane; c < ldc; c += 32) {
      const double2 v = c < nb ? Cb[(long long)r * nb + c] : make_double2(0.0, 0.0);
      Cs[r * ldc + c] = make_float2((float)v.x, (float)v.y);
    }
  for (int g0 = blockIdx.x * TG; g0 < npw; g0 += gridDim.x * TG) {
    __syncthreads();   // C staged; the previous tile's reads done
    for (int r = w; r < nb; r += RWARPS)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int g = g0 + lane + 32 * u;
        Xs[r * TG + lane + 32 * u] = g < npw ? Xb[(long long)r * K.npw_pad + g] : make_float2(0.f, 0.f);
      }
    __syncthreads();
    float2 acc[JQ][2][2];
#pragma unroll
    for (int q = 0; q < JQ; ++q)
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int u = 0; u < 2; ++u) acc[q][v][u] = make_float2(0.f, 0.f);
    for (int r0 = 0; r0 < nb; r0 += RROWS) {
      const int r1 = min(nb, r0 + RROWS);
      // the first pair this chunk of rows reaches
      const int q0 = upper ? max(0, (r0 / 2 - w + RWARPS - 1) / RWARPS) : 0;
      for (int r = r0; r < r1; ++r) {
        const float2 x0 = Xs[r * TG + lane], x1 = Xs[r * TG + lane + 32];
#pragma unroll
        for (int q = 0; q < JQ; ++q) {
          const int j = 2 * (w + RWARPS * q);
          if (j >= nb || q < q0) continue;
          const float4 c = *reinterpret_cast<const float4 *>(&Cs[r * ldc + j]);
          const float2 ca = make_float2(c.x, c.y), cb = make_float2(c.z, c.w);
          cmac<float>(acc[q][0][0], x0, ca);
          cmac<float>(acc[q][0][1], x1, ca);
          cmac<float>(acc[q][1][0], x0, cb);
          cmac<float>(acc[q][1][1], x1, cb);
        }
      }
    }
#pragma unroll
    for (int q = 0; q < JQ; ++q)
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = 2 * (w + RWARPS * q) + v, g = g0 + lane + 32 * u;
          if (j < nb && g < npw) Xb[(long long)j * K.npw_pad + g] = acc[q][v][u];
        }
  }
}

// neg ? -x : x on the sign bit (a negation by itself is an FP64 operation)
__device__ __forceinline__ double flip(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}

// ---------------------------------------------------------------------------
// Cholesky S = L L^H and C = L^-H (upper triangular), one block per k-set.
// Worked as S = (Lu) D (Lu)^H with Lu unit lower triangular: step j subtracts
// (m_ij / d_j) times the pivot row from every row i > j, of the trailing matrix
// and of the inverse that grows beside it (Y = Lu^-1), so a step is one
// division, one pass over independent elements and one barrier; the roots
// come at the end, L^-1 = D^-1/2 Y.  Y shares the square with the matrix (its
// row i, stored as column i of the upper triangle), which keeps up to 118 bands in
// shared memory.  Before, a root, a division and three barriers a step, the
// inverse by one thread per column and 81 bands and more in global memory: 12
// bands 35 -> 13 us, 24 bands 102 -> 33 us, 84 bands 1,140 -> 540 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zmulc(double2 a, double2 b) {  // a * conj(b)
  return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

__global__ void __launch_bounds__(256) k_cholesky_inv(const Tables t, int ks_begin,
                                                      const double2 *__restrict__ S,
                                                      double2 *__restrict__ Cout,
                                                      const long long *__restrict__ mat_off,
                                                      double2 *__restrict__ scratch,
                                                      int *__restrict__ status, int use_smem) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ksi = ks_begin + blockIdx.x;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;
  const int n = K.nb, ld = n | 1;   // odd pitch: columns are walked too
  // M[i][k], i >= k: the matrix (its diagonal ends as D); M[c][i], c < i: Y[i][c]
  double2 *M = use_smem ? reinterpret_cast<double2 *>(smem_raw) : scratch + 2 * mat_off[ksi];
  const double2 *Sb = S + mat_off[ksi];
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) M[(e / n) * ld + e % n] = e / n >= e % n ? Sb[e] : make_double2(0, 0);
  __syncthreads();
  // failure threshold relative to the largest diagonal element
  double dmax = 0.0;
  for (int i = 0; i < n; i += 32) {
    const double v = i + (threadIdx.x & 31) < n ? M[(i + (threadIdx.x & 31)) * (ld + 1)].x : 0.0;
    dmax = fmax(dmax, v);
  }
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, w));
  const double thr = 1e-13 * dmax;
  bool fail = false;
  for (int j = 0; j < n; ++j) {
    // every thread reads the pivot: the previous step's barrier published it
    const double d = M[j * ld + j].x;
    const bool low = !(d > thr);
    fail |= low;
    const double w = 1.0 / (low ? thr : d);
    const int rows = n - 1 - j;
    for (int e = threadIdx.x; e < rows * n; e += blockDim.x) {
      const int i = j + 1 + e / n, k = e - (e / n) * n;
      if (k > i) continue;
      const double2 m = M[i * ld + j], f = make_double2(m.x * w, m.y * w);
      // trailing matrix (k > j): M[i][k] -= m_ij / d conj(m_kj); inverse (k <= j):
      // Y[i][k] -= m_ij / d Y[j][k] with Y[j][j] = 1, without a branch between them
      double2 z = M[k * ld + j];
      z = make_double2(k == j ? 1.0 : z.x, k == j ? 0.0 : flip(z.y, k > j));
      double2 &dst = M[k > j ? i * ld + k : k * ld + i];
      double2 v = dst;
      cmac<double>(v, make_double2(-f.x, -f.y), z);
      dst = make_double2(v.x, k == i ? 0.0 : v.y);
    }
    __syncthreads();
  }
  // C[i][j] = conj(Linv[j][i]), Linv[j][i] = Y[j][i] / sqrt(d_j)
  double2 *Cb = Cout + mat_off[ksi];
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e % n;
    const double d = M[j * ld + j].x;
    const double r = rsqrt(d > thr ? d : thr);
    double2 v = make_double2(0.0, 0.0);
    if (i < j) v = M[i * ld + j];
    if (i == j) v.x = 1.0;
    Cb[e] = make_double2(v.x * r, -v.y * r);
  }
  // keep an earlier failure of this k-set (a timed-out overlap wait)
  if (threadIdx.x == 0 && fail && status[ksi] == 0) status[ksi] = DEREK_ERR_CHOLESKY;
}

// ---------------------------------------------------------------------------
// Hermitian Jacobi eigensolver (parallel cyclic, round-robin pair ordering).
// Each round rotates np = ne/2 disjoint index pairs (p, q) at once:
//   A <- U^H A U,  V <- V U,  U = diag(1, e^{-i phi}) [[c, s], [-s, c]] per pair.
// Entry (i, j) of U^H A U depends only on the 2x2 block of A at the pairs
// holding i and j, so a round is one pass over the blocks (a <= b) of pairs:
// A'_ab = U_a^H A_ab U_b, with A'_ba = A'_ab^H written by the same thread.
// All arithmetic on A and on the eigenvectors, stored one per row, is FP64.
// Eigenvalues ascending go to eig[item0 + j]; eigenvectors (columns) to C.
//
// Bound by FP64 issue: an FP64 operation of one warp takes 64 clocks of its
// quarter of the SM, dependent or not, so what counts is operations per warp
// on the fullest quarter.
//   Rotations: the angle and the phase come from FP32 (their error leaves
//   1e-7 of an off-diagonal element for the next sweep, which squares it), and
//   (c, s) and the phase are then brought to unit length in FP64 by two terms
//   of 1/sqrt(1 + d), d ~ 1e-7.  12 FP64 operations instead of two reciprocal
//   roots, a root and a division in a chain of ~2,700 clocks.
//   Blocks: one per thread (LPB = 1) or, where a CTA has few, one element per
//   lane (LPB = 4).
//   A cluster of CS CTAs shares a k-set: each CTA keeps a full copy of A,
//   computes every rotation (equal copies, equal decisions), updates its share
//   of the blocks in all copies through distributed shared memory, and its
//   slice of the eigenvector rows.
// Two cluster barriers a round, both split so that work covers them: B1, every
// CTA has read this round's pivots, before remote copies are written (the
// first block is computed between arrival and wait); B2, every block is
// written, with the eigenvector update in between.
// Measured per solve, mean over an SCF, against two CTAs with exact angles: n =
// 12, 178 -> 98 us; n = 24, 8 k-sets, 560 -> 340 us, 40 k-sets 542 -> 363 us; n =
// 84, 4 k-sets, 9.6 -> 4.4 ms; 64 k-sets 7.8 ms either way (two CTAs, all of it
// FP64 issue).
// ---------------------------------------------------------------------------
__host__ __device__ constexpr size_t jacobi_round_bytes(size_t np) {
  return (np * (sizeof(double2) + 2 * sizeof(double) + 3 * sizeof(int)) + 15) / 16 * 16;
}
struct JacobiTables {   // of one round, in shared memory
  double2 *ph;
  double *c, *s;
  int *pp, *pq, *act;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// pair k of round r in the circle schedule over ne positions (position 0
// fixed, the others advance one place per round)
__device__ __forceinline__ void rr_pair(int k, int r, int ne, int &p, int &q) {
  const int m = ne - 1;
  int a = k - 1 + r, b = ne - 2 - k + r;
  if (a >= m) a -= m;
  if (b >= m) b -= m;
  a = k == 0 ? 0 : 1 + a;
  b += 1;
  p = min(a, b);
  q = max(a, b);
}

// x + y i scaled to unit length, x^2 + y^2 = 1 + d with |d| ~ 1e-7
__device__ __forceinline__ void unit_length(double &x, double &y) {
  const double d = fma(x, x, fma(y, y, -1.0));
  const double k = fma(d, fma(d, 0.375, -0.5), 1.0);
  x *= k;
  y *= k;
}

template <int CS, int LPB>
__global__ void __launch_bounds__(256) k_jacobi(const Tables t, int ks_begin, const double2 *__restrict__ Hs,
                                                double2 *__restrict__ Cout, const long long *__restrict__ mat_off,
                                                double *__restrict__ eig, int max_sweeps, double tol,
                                                int *__restrict__ sweeps_out) {
  grid_dependency();
  namespace cg = cooperative_groups;
  constexpr int NT = 256;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int crank = blockIdx.x % CS;
  const int ksi = ks_begin + blockIdx.x / CS;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;   // the whole cluster leaves together
  const int tid = threadIdx.x;
  const int n = K.nb;
  const int ne = n + (n & 1);   // even count for the tournament; index n is a dummy
  const int np = ne / 2;
  const int nblk = np * (np + 1) / 2;
  const int hv = (n + CS - 1) / CS;   // eigenvector rows of a CTA
  const int v0 = min(n, crank * hv), nv = min(n, v0 + hv) - v0;
  double2 *A = reinterpret_cast<double2 *>(smem_raw);
  double2 *Vt = A + n * n;                  // [n][hv]: eigenvector i, rows v0 ...
  unsigned char *sp = reinterpret_cast<unsigned char *>(Vt + n * hv);
  // two rounds' tables: a round's eigenvector update overlaps the next round's
  // rotations
  auto tables = [sp, np](int i) {
    JacobiTables T;
    T.ph = reinterpret_cast<double2 *>(sp + i * jacobi_round_bytes(np));
    T.c = reinterpret_cast<double *>(T.ph + np);
    T.s = T.c + np;
    T.pp = reinterpret_cast<int *>(T.s + np);
    T.pq = T.pp + np;
    T.act = T.pq + np;
    return T;
  };
  short2 *blk = reinterpret_cast<short2 *>(sp + 2 * jacobi_round_bytes(np));   // [nblk]: (a, b), a <= b
  __shared__ float red[2][NT / 32];
  double2 *copy[CS];   // A of every CTA, the own one first
  copy[0] = A;
  if constexpr (CS > 1) {
    cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
    for (int r = 1; r < CS; ++r) copy[r] = cluster.map_shared_rank(A, (crank + r) % CS);
  }
  const double2 *Hb = Hs + mat_off[ksi];
  for (int e = tid; e < n * n; e += NT) A[e] = Hb[e];
  for (int e = tid; e < n * hv; e += NT) Vt[e] = make_double2(e / hv == v0 + e % hv ? 1.0 : 0.0, 0.0);
  for (int w = tid; w < nblk; w += NT) {
    // w -> (a, b) with a <= b, rows of the upper triangle in order
    int a = 0, rem = w;
    while (rem >= np - a) {
      rem -= np - a;
      ++a;
    }
    blk[w] = make_short2((short)a, (short)(a + rem));
  }
  if constexpr (CS > 1) {   // every CTA running and initialised before a remote write
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  // A lives in its upper triangle: half the stores to the other copies, whose
  // 16-byte packets bound large clusters (5.6 -> 4.4 ms at 84 bands, CS = 8)
  auto get = [&](int r, int c) {
    const double2 v = A[min(r, c) * n + max(r, c)];
    return make_double2(v.x, flip(v.y, r > c));
  };
  auto put = [&](int r, int c, double2 v) {
    const int idx = min(r, c) * n + max(r, c);
    const double2 w = make_double2(v.x, r == c ? 0.0 : flip(v.y, r > c));
#pragma unroll
    for (int k = 0; k < CS; ++k) copy[k][idx] = w;
  };
  // FP32 arithmetic runs on entries divided by the largest one
  float big = 0.f;
  for (int e = tid; e < n * n; e += NT) big = fmaxf(big, fmaxf(fabsf((float)A[e].x), fabsf((float)A[e].y)));
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, w));
  if ((tid & 31) == 0) red[0][tid >> 5] = big;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) big = fmaxf(big, red[0][w]);
  const float scale = big > 0.f ? 1.f / big : 1.f;
  __syncthreads();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    // convergence: sum of |offdiag|^2 against sum of |A|^2; FP32 sums decide as
    // well as FP64 ones
    float off = 0.f, dia = 0.f;
    for (int e = tid; e < n * n; e += NT) {
      const float x = (float)A[e].x * scale, y = (float)A[e].y * scale;
      const int i = e / n, j = e - i * n;
      if (i == j)
        dia = fmaf(x, x, dia);
      else if (i < j)
        off = fmaf(x, x, fmaf(y, y, off));
    }
    off *= 2.f;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, w);
      dia += __shfl_xor_sync(0xffffffffu, dia, w);
    }
    if ((tid & 31) == 0) {
      red[0][tid >> 5] = off;
      red[1][tid >> 5] = dia;
    }
    __syncthreads();
    off = dia = 0.f;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
      off += red[0][w];
      dia += red[1][w];
    }
    const float tot = off + dia, ftol = (float)tol;
    __syncthreads();
    if (!(off > ftol * ftol * tot)) break;
    // rotations of elements below tol ||A||_F / (4 n) cannot matter for the
    // test and are skipped
    const float skip = ftol / (4.f * n), skip2 = skip * skip * tot;
    for (int round = 0; round < ne - 1; ++round) {
      const JacobiTables T = tables(round & 1);
      // threads 0 .. np-1: phases; threads 128 ..: (c, s) of the same pairs, on
      // warps of other quarters of the SM
      const int half = tid >> 7, k = tid & 127;
      if (k < np) {
        int p, q;
        rr_pair(k, round, ne, p, q);
        double u = 1.0, v = 0.0;
        int on = 0;
        if (q < n) {
          const double2 b = A[p * n + q];
          const float bx = (float)b.x * scale, by = (float)b.y * scale;
          const float e2 = bx * bx + by * by;
          on = e2 > skip2;
          if (on) {
            const float ie = rsqrtf(e2);
            float fu = bx * ie, fv = by * ie;
            if (half) {
              const float d = (float)(A[q * n + q].x - A[p * n + p].x) * scale;
              const float tau = d * (0.5f * ie);
              const float tt = copysignf(1.f, tau) / (fabsf(tau) + sqrtf(fmaf(tau, tau, 1.f)));
              fu = rsqrtf(fmaf(tt, tt, 1.f));
              fv = tt * fu;
            }
            u = fu;
            v = fv;
            unit_length(u, v);
          }
        }
        if (half) {
          T.c[k] = u;
          T.s[k] = v;
          T.pp[k] = p;
          T.pq[k] = q;
        } else {
          T.ph[k] = make_double2(u, v);
          T.act[k] = on;
        }
      }
      __syncthreads();
      if constexpr (CS > 1) cluster_arrive();   // B1: this CTA has read its pivots
      bool waited = CS == 1;
      // blocks of A: left by U_a^H (new row p = c A_p - s ph A_q, new row
      // q = s A_p + c ph A_q), right by U_b (new col p = c X_p - s conj(ph) X_q,
      // new col q = s X_p + c conj(ph) X_q)
      if constexpr (LPB == 4) {
        const int i = (tid >> 1) & 1, j = tid & 1;
        const int per = (nblk * 4 + CS - 1) / CS;   // items of a CTA
        for (int base = 0; base < per; base += NT) {
          const int w = (base + tid) / 4 * CS + crank;
          const bool in = w < nblk;
          const short2 ab = in ? blk[w] : make_short2(0, 0);
          const int ia = ab.x, ib = ab.y;
          const bool on = in && (T.act[ia] | T.act[ib]);
          const int row = i ? T.pq[ia] : T.pp[ia], col = j ? T.pq[ib] : T.pp[ib];
          const bool ok = on && row < n && col < n;
          double2 x = ok ? get(row, col) : make_double2(0.0, 0.0);
          double2 y;
          {
            y.x = __shfl_xor_sync(0xffffffffu, x.x, 2);
            y.y = __shfl_xor_sync(0xffffffffu, x.y, 2);
            const double2 ph = T.ph[ia];
            const double2 z = zmul(ph, i ? x : y);
            const double2 o = i ? y : x;
            const double c = T.c[ia], sn = T.s[ia];
            const double al = i ? sn : c, be = flip(i ? c : sn, !i);
            x = make_double2(fma(be, z.x, al * o.x), fma(be, z.y, al * o.y));
          }
          {
            y.x = __shfl_xor_sync(0xffffffffu, x.x, 1);
            y.y = __shfl_xor_sync(0xffffffffu, x.y, 1);
            const double2 ph = T.ph[ib];
            const double2 z = zmul(make_double2(ph.x, -ph.y), j ? x : y);
            const double2 o = j ? y : x;
            const double c = T.c[ib], sn = T.s[ib];
            const double al = j ? sn : c, be = flip(j ? c : sn, !j);
            x = make_double2(fma(be, z.x, al * o.x), fma(be, z.y, al * o.y));
          }
          if constexpr (CS > 1) {
            if (!waited) {
              __syncwarp();
              cluster_wait();
              waited = true;
            }
          }
          if (ok && (ia != ib || j >= i)) put(row, col, x);
        }
      } else {
        for (int base = 0; base < nblk; base += CS * NT) {
          const int w = base + tid * CS + crank;
          const bool in = w < nblk;
          const short2 ab = in ? blk[w] : make_short2(0, 0);
          const int ia = ab.x, ib = ab.y;
          const int on_a = in ? T.act[ia] : 0, on_b = in ? T.act[ib] : 0;
          const int pa = T.pp[ia], qa = T.pq[ia], pb = T.pp[ib], qb = T.pq[ib];
          const bool qa_ok = qa < n, qb_ok = qb < n;
          const double2 z = make_double2(0.0, 0.0);
          double2 x00 = z, x01 = z, x10 = z, x11 = z;
          if (on_a | on_b) {
            x00 = get(pa, pb);
            if (qb_ok) x01 = get(pa, qb);
            if (qa_ok) x10 = get(qa, pb);
            if (qa_ok && qb_ok) x11 = get(qa, qb);
          }
          if (on_a) {
            const double c = T.c[ia], sn = T.s[ia];
            const double2 ph = T.ph[ia];
            const double2 t0 = zmul(ph, x10), t1 = zmul(ph, x11);
            const double2 n00 = make_double2(fma(-sn, t0.x, c * x00.x), fma(-sn, t0.y, c * x00.y));
            const double2 n01 = make_double2(fma(-sn, t1.x, c * x01.x), fma(-sn, t1.y, c * x01.y));
            x10 = make_double2(fma(c, t0.x, sn * x00.x), fma(c, t0.y, sn * x00.y));
            x11 = make_double2(fma(c, t1.x, sn * x01.x), fma(c, t1.y, sn * x01.y));
            x00 = n00;
            x01 = n01;
          }
          if (on_b) {
            const double c = T.c[ib], sn = T.s[ib];
            const double2 ph = T.ph[ib], phc = make_double2(ph.x, -ph.y);
            const double2 t0 = zmul(phc, x01), t1 = zmul(phc, x11);
            const double2 n00 = make_double2(fma(-sn, t0.x, c * x00.x), fma(-sn, t0.y, c * x00.y));
            const double2 n10 = make_double2(fma(-sn, t1.x, c * x10.x), fma(-sn, t1.y, c * x10.y));
            x01 = make_double2(fma(c, t0.x, sn * x00.x), fma(c, t0.y, sn * x00.y));
            x11 = make_double2(fma(c, t1.x, sn * x10.x), fma(c, t1.y, sn * x10.y));
            x00 = n00;
            x10 = n10;
          }
          if constexpr (CS > 1) {
            if (!waited) {
              __syncwarp();
              cluster_wait();
              waited = true;
            }
          }
          if (!(on_a | on_b)) continue;
          put(pa, pb, x00);
          if (qb_ok) put(pa, qb, x01);
          if (qa_ok && ia != ib) put(qa, pb, x10);   // a pair's own block: the mirror of x01
          if (qa_ok && qb_ok) put(qa, qb, x11);
        }
      }
      if constexpr (CS > 1) {
        if (!waited) cluster_wait();
        __syncwarp();
        cluster_arrive();   // B2: this CTA's blocks are written everywhere
      }
      // eigenvectors: Vt[col][row], new col p = c X_p - s conj(ph) X_q,
      // new col q = s X_p + c conj(ph) X_q; last threads first, the blocks
      // fill the first ones
      for (int w = NT - 1 - tid; w < np * nv; w += NT) {
        const int kk = w / nv, row = w - kk * nv;
        if (!T.act[kk]) continue;
        const double c = T.c[kk], sn = T.s[kk];
        const double2 ph = T.ph[kk];
        double2 &xp = Vt[T.pp[kk] * hv + row];
        double2 &xq = Vt[T.pq[kk] * hv + row];
        const double2 a = xp, tq = zmul(make_double2(ph.x, -ph.y), xq);
        xp = make_double2(fma(-sn, tq.x, c * a.x), fma(-sn, tq.y, c * a.y));
        xq = make_double2(fma(c, tq.x, sn * a.x), fma(c, tq.y, sn * a.y));
      }
      if constexpr (CS > 1) {
        __syncwarp();
        cluster_wait();
      } else {
        __syncthreads();
      }
    }
    __syncthreads();   // the eigenvector update of the last round
  }
  if (tid == 0 && crank == 0 && sweeps_out) sweeps_out[ksi] = sweep;
  // ascending order by rank (ties by index) on order-preserving integer keys
  long long *key = reinterpret_cast<long long *>(tables(0).ph);
  int *rank = reinterpret_cast<int *>(tables(1).ph);
  __syncthreads();
  for (int i = tid; i < n; i += NT) {
    const long long v = __double_as_longlong(A[i * n + i].x);
    key[i] = v < 0 ? ~v ^ (long long)0x8000000000000000ull : v;
  }
  __syncthreads();
  for (int i = tid; i < n; i += NT) {
    const long long vi = key[i];
    int r = 0;
    for (int j = 0; j < n; ++j) r += key[j] < vi || (key[j] == vi && j < i);
    rank[i] = r;
    if (crank == 0) eig[K.item0 + r] = A[i * n + i].x;
  }
  __syncthreads();
  double2 *Cb = Cout + mat_off[ksi];
  for (int e = tid; e < n * nv; e += NT) {
    const int r = e / n, i = e - r * n;
    Cb[(v0 + r) * n + rank[i]] = Vt[i * hv + r];
  }
  if constexpr (CS > 1) {   // no CTA leaves while a partner could still address it
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
}

// The same solve with A and the eigenvectors in global scratch, for subspaces
// whose A does not fit the shared memory (from about 116 bands).
// Rotation that zeroes the Hermitian 2x2 block [[a, b], [conj(b), d]]: the
// phase ph = b / |b|, then the real symmetric rotation (c, s) of
// [[a, |b|], [|b|, d]] with t = sign(tau) / (|tau| + sqrt(1 + tau^2)),
// tau = (d - a) / (2 |b|), c = 1 / sqrt(1 + t^2), s = t c (Rutishauser).
// Written as two reciprocal square roots, one square root and one division:
// the dependent FP64 chain every Jacobi round waits on.  The entries are bounded by the matrix norm, so |b| needs
// no hypot scaling.  False (no rotation) when |b| <= skip.
__device__ __forceinline__ bool jacobi_rotation(double a, double d, double2 b, double skip, double &c,
                                                double &s, double2 &ph) {
  const double e2 = b.x * b.x + b.y * b.y;
  if (!(e2 > skip * skip)) return false;
  const double ie = rsqrt(e2);
  ph = make_double2(b.x * ie, b.y * ie);
  const double tau = (d - a) * (0.5 * ie);
  const double tt = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
  c = rsqrt(1.0 + tt * tt);
  s = tt * c;
  return true;
}


__global__ void __launch_bounds__(256) k_jacobi_global(const Tables t, int ks_begin,
                                                const double2 *__restrict__ Hs,
                                                double2 *__restrict__ Cout,
                                                const long long *__restrict__ mat_off,
                                                double *__restrict__ eig,
                                                double2 *__restrict__ scratch, int max_sweeps,
                                                double tol, int *__restrict__ sweeps_out) {
  grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ksi = ks_begin + blockIdx.x;
  const KSetDev &K = t.ks[ksi];
  if (!t.sys[K.sys].active) return;
  const int n = K.nb;
  const int ne = n + (n & 1);  // even count for the tournament; index n is a dummy
  const int np = ne / 2;
  const int nblk = np * (np + 1) / 2;
  double2 *Vt = scratch + 2 * mat_off[ksi], *A = Vt + (long long)n * n;
  double2 *rph = reinterpret_cast<double2 *>(smem_raw);  // [np]
  double *rc = reinterpret_cast<double *>(rph + np);
  double *rs = rc + np;
  int *pp = reinterpret_cast<int *>(rs + np);
  int *pq = pp + np;
  int *act = pq + np;
  short2 *blk = reinterpret_cast<short2 *>(act + np);  // [nblk]: (a, b), a <= b
  __shared__ double red[256];
  __shared__ double red2[256];
  const double2 *Hb = Hs + mat_off[ksi];
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    A[e] = Hb[e];
    const int i = e / n, j = e % n;
    Vt[e] = make_double2(i == j ? 1.0 : 0.0, 0.0);
  }
  for (int w = threadIdx.x; w < nblk; w += blockDim.x) {
    // w -> (a, b) with a <= b, rows of the upper triangle in order
    int a = 0, rem = w;
    while (rem >= np - a) {
      rem -= np - a;
      ++a;
    }
    blk[w] = make_short2((short)a, (short)(a + rem));
  }
  __syncthreads();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    // convergence: sum of |offdiag|^2 vs sum of |A|^2, both summed directly
    double off = 0, tot = 0;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
      const double m2 = A[e].x * A[e].x + A[e].y * A[e].y;
      tot += m2;
      if (e / n != e % n) off += m2;
    }
    red[threadIdx.x] = off;
    red2[threadIdx.x] = tot;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) {
        red[threadIdx.x] += red[threadIdx.x + s];
        red2[threadIdx.x] += red2[threadIdx.x + s];
      }
      __syncthreads();
    }
    const bool done = red[0] <= tol * tol * red2[0];
    // skip rotations whose element cannot matter for the convergence test
    // (threshold Jacobi): |a_pq| below tol * ||A||_F / (4 n)
    const double skip = tol * sqrt(red2[0]) / (4.0 * n);
    __syncthreads();
    if (done) break;
    for (int round = 0; round < ne - 1; ++round) {
      for (int k = threadIdx.x; k < np; k += blockDim.x) {
        int p, q;
        rr_pair(k, round, ne, p, q);
        pp[k] = p;
        pq[k] = q;
        double c = 1.0, s = 0.0;
        double2 ph = make_double2(1.0, 0.0);
        int on = 0;
        if (q < n) {
          on = jacobi_rotation(A[p * n + p].x, A[q * n + q].x, A[p * n + q], skip, c, s, ph) ? 1 : 0;
        }
        rc[k] = c;
        rs[k] = s;
        rph[k] = ph;
        act[k] = on;
      }
      __syncthreads();
      // blocks of A: left by U_a^H (new row p = c A_p - s ph A_q, new row
      // q = s A_p + c ph A_q), right by U_b (new col p = c X_p - s conj(ph) X_q,
      // new col q = s X_p + c conj(ph) X_q)
      for (int w = threadIdx.x; w < nblk; w += blockDim.x) {
        const short2 ab = blk[w];
        const int ia = ab.x, ib = ab.y;
        const int on_a = act[ia], on_b = act[ib];
        if (!on_a && !on_b) continue;
        const int pa = pp[ia], qa = pq[ia], pb = pp[ib], qb = pq[ib];
        const bool qa_ok = qa < n, qb_ok = qb < n;
        const double2 z = make_double2(0.0, 0.0);
        double2 x00 = A[pa * n + pb];
        double2 x01 = qb_ok ? A[pa * n + qb] : z;
        double2 x10 = qa_ok ? A[qa * n + pb] : z;
        double2 x11 = (qa_ok && qb_ok) ? A[qa * n + qb] : z;
        if (on_a) {
          const double c = rc[ia], s = rs[ia];
          const double2 ph = rph[ia];
          const double2 t0 = zmul(ph, x10), t1 = zmul(ph, x11);
          const double2 n00 = make_double2(c * x00.x - s * t0.x, c * x00.y - s * t0.y);
          const double2 n01 = make_double2(c * x01.x - s * t1.x, c * x01.y - s * t1.y);
          x10 = make_double2(s * x00.x + c * t0.x, s * x00.y + c * t0.y);
          x11 = make_double2(s * x01.x + c * t1.x, s * x01.y + c * t1.y);
          x00 = n00;
          x01 = n01;
        }
        if (on_b) {
          const double c = rc[ib], s = rs[ib];
          const double2 phc = make_double2(rph[ib].x, -rph[ib].y);
          const double2 t0 = zmul(phc, x01), t1 = zmul(phc, x11);
          const double2 n00 = make_double2(c * x00.x - s * t0.x, c * x00.y - s * t0.y);
          const double2 n10 = make_double2(c * x10.x - s * t1.x, c * x10.y - s * t1.y);
          x01 = make_double2(s * x00.x + c * t0.x, s * x00.y + c * t0.y);
          x11 = make_double2(s * x10.x + c * t1.x, s * x10.y + c * t1.y);
          x00 = n00;
          x10 = n10;
        }
        if (ia == ib) {
          // the pair's own 2x2 block is now diagonal and real
          A[pa * n + pa] = make_double2(x00.x, 0.0);
          A[qa * n + qa] = make_double2(x11.x, 0.0);
          A[pa * n + qa] = z;
          A[qa * n + pa] = z;
          continue;
        }
        A[pa * n + pb] = x00;
        A[pb * n + pa] = make_double2(x00.x, -x00.y);
        if (qb_ok) {
          A[pa * n + qb] = x01;
          A[qb * n + pa] = make_double2(x01.x, -x01.y);
        }
        if (qa_ok) {
          A[qa * n + pb] = x10;
          A[pb * n + qa] = make_double2(x10.x, -x10.y);
        }
        if (qa_ok && qb_ok) {
          A[qa * n + qb] = x11;
          A[qb * n + qa] = make_double2(x11.x, -x11.y);
        }
      }
      // eigenvectors: Vt[col][row], new col p = c X_p - s conj(ph) X_q,
      // new col q = s X_p + c conj(ph) X_q
      for (int w = threadIdx.x; w < np * n; w += blockDim.x) {
        const int k = w / n, row = w - (w / n) * n;
        if (!act[k]) continue;
        const double c = rc[k], s = rs[k];
        const double phx = rph[k].x, phy = -rph[k].y;
        double2 &xp = Vt[pp[k] * n + row];
        double2 &xq = Vt[pq[k] * n + row];
        const double2 a = xp, b = xq;
        const double tx = phx * b.x - phy * b.y, ty = phx * b.y + phy * b.x;
        xp.x = c * a.x - s * tx;
        xp.y = c * a.y - s * ty;
        xq.x = s * a.x + c * tx;
        xq.y = s * a.y + c * ty;
      }
      __syncthreads();
    }
  }
  if (threadIdx.x == 0 && sweeps_out) sweeps_out[ksi] = sweep;
  // sort eigenvalues ascending (selection by rank; ties broken by index)
  double *ev = rc;  // reuse: np * 2 >= n entries (rc and rs are adjacent)
  for (int i = threadIdx.x; i < n; i += blockDim.x) ev[i] = A[i * n + i].x;
  __syncthreads();
  double2 *Cb = Cout + mat_off[ksi];
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double vi = ev[i];
    int rank = 0;
    for (int j = 0; j < n; ++j) rank += (ev[j] < vi) || (ev[j] == vi && j < i);
    eig[K.item0 + rank] = vi;
    for (int r = 0; r < n; ++r) {
      Cb[r * n + rank] = Vt[i * n + r];
    }
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
int overlap_split_min(long long total_npw) {
  const long long s = (total_npw / (4 * sm_count()) + 31) / 32 * 32;
  return (int)std::max<long long>(32, std::min<long long>(kOverlapSplitMin, s));
}

template <typename R, bool SAME>
static void overlap_go(const Tables &t, int ks_begin, int nks, int max_nb, int max_npw, int ksplit, int split_min,
                       const cplx<R> *A, const cplx<R> *B, double2 *part, const long long *part_off, double2 *out,
                       const long long *mat_off, int hermitize, cudaStream_t st) {
  using Sh = OverlapShape<R>;
  const int nt = (max_nb + Sh::MT - 1) / Sh::MT;
  const int np = SAME ? nt * (nt + 1) / 2 : nt * nt;
  int P = 1;
  while (P < Sh::PMAX && P * 256 < np) P *= 2;
  const int groups = (np + 256 * P - 1) / (256 * P);
  const int threads = ((np + groups * P - 1) / (groups * P) + 31) / 32 * 32;
  // four blocks per SM where the buffers of the partial sums allow it, never
  // longer than the planned split
  const int want = std::max(1, (4 * sm_count() + groups * nks - 1) / (groups * nks));
  const int fill = ((max_npw + want - 1) / want + Sh::OKC - 1) / Sh::OKC * Sh::OKC;
  ksplit = std::min(ksplit, std::max(split_min, fill));
  const size_t sm = (size_t)nt * Sh::MT * (Sh::OKC + 1) * sizeof(cplx<R>) * (SAME ? 1 : 2);
  const dim3 grid(groups, (max_npw + ksplit - 1) / ksplit, nks);
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    derek::launch(kern, grid, threads, sm, st, t, ks_begin, A, B, part, part_off, ksplit);
  };
  switch (P) {
    case 1: go(k_overlap_pairs<R, 1, SAME>); break;
    case 2: go(k_overlap_pairs<R, 2, SAME>); break;
    case 4: go(k_overlap_pairs<R, 4, SAME>); break;
    default: go(k_overlap_pairs<R, Sh::PMAX, SAME>); break;
  }
  launch_overlap_reduce(t, ks_begin, nks, max_nb, part, part_off, ksplit, out, mat_off, hermitize, SAME, st);
}

template <typename R>
void launch_overlap(const Tables &t, int ks_begin, int nks, int max_nb, int max_npw, int ksplit, int split_min,
                    const cplx<R> *A, const cplx<R> *B, double2 *part, const long long *part_off,
                    double2 *out, const long long *mat_off, int hermitize, cudaStream_t st) {
  if (nks <= 0) return;
  if (A == B)
    overlap_go<R, true>(t, ks_begin, nks, max_nb, max_npw, ksplit, split_min, A, B, part, part_off, out, mat_off,
                        hermitize, st);
  else
    overlap_go<R, false>(t, ks_begin, nks, max_nb, max_npw, ksplit, split_min, A, B, part, part_off, out, mat_off,
                         hermitize, st);
}

void launch_overlap_reduce(const Tables &t, int ks_begin, int nks, int max_nb, const double2 *part,
                           const long long *part_off, int ksplit, double2 *out,
                           const long long *mat_off, int hermitize, int half, cudaStream_t st) {
  const dim3 grid(nks, (max_nb * max_nb * kReduceLanes + 255) / 256);
  derek::launch(k_overlap_reduce, grid, 256, 0, st, t, ks_begin, part, part_off, ksplit, out, mat_off, hermitize, half);
}

template <typename R>
void launch_rotate(const Tables &t, int ks_begin, int nks, int max_nb, int max_npw, cplx<R> *X,
                   const double2 *C, const long long *mat_off, int upper, cudaStream_t st) {
  if (nks <= 0) return;
  constexpr bool F64 = std::is_same<R, double>::value;
  const int ldc = (max_nb + 1) & ~1;
  const size_t sm = F64 ? (size_t)max_nb * (RG + RROWS) * sizeof(cplx<R>)
                        : (size_t)max_nb * (ldc + 2 * RG) * sizeof(cplx<R>);
  const int tiles = (max_npw + (F64 ? RG : 2 * RG) - 1) / (F64 ? RG : 2 * RG);
  // FP32 blocks keep their converted C over several tiles once that leaves
  // four blocks per SM
  const int gx = F64 ? tiles : std::min(tiles, std::max(1, (4 * sm_count() + nks - 1) / nks));
  auto go = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    derek::launch(kern, dim3(gx, nks), 256, sm, st, t, ks_begin, X, C, mat_off, upper);
  };
  if constexpr (F64) {
    switch ((max_nb + RWARPS - 1) / RWARPS) {
      case 1: go(k_rotate64<1>); break;
      case 2: go(k_rotate64<2>); break;
      case 3: go(k_rotate64<3>); break;
      case 4: go(k_rotate64<4>); break;
      case 5: case 6: go(k_rotate64<6>); break;
      case 7: case 8: go(k_rotate64<8>); break;
      case 9: case 10: case 11: case 12: go(k_rotate64<12>); break;
      default: go(k_rotate64<16>); break;
    }
  } else {
    switch ((max_nb + 2 * RWARPS - 1) / (2 * RWARPS)) {
      case 1: go(k_rotate32<1>); break;
      case 2: go(k_rotate32<2>); break;
      case 3: go(k_rotate32<3>); break;
      case 4: go(k_rotate32<4>); break;
      case 5: case 6: go(k_rotate32<6>); break;
      default: go(k_rotate32<8>); break;
    }
  }
}

static bool cholesky_fits_smem(int max_nb) { return (size_t)max_nb * (max_nb | 1) * sizeof(double2) <= 226 * 1024; }
void launch_cholesky_inv(const Tables &t, int ks_begin, int nks, int max_nb, const double2 *S,
                         double2 *C, const long long *mat_off, double2 *scratch, int *status,
                         cudaStream_t st) {
  if (nks <= 0) return;
  const int use_smem = cholesky_fits_smem(max_nb);
  const size_t sm = use_smem ? (size_t)max_nb * (max_nb | 1) * sizeof(double2) : 0;
  cudaFuncSetAttribute(k_cholesky_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  derek::launch_plain(k_cholesky_inv, nks, 256, sm, st, t, ks_begin, S, C, mat_off, scratch, status, use_smem);
}

// tables of the Jacobi kernels: two rounds' rotations and the block list
static size_t jacobi_tables(int max_nb) {
  const size_t np = (size_t)(max_nb + 1) / 2;
  return 2 * jacobi_round_bytes(np) + np * (np + 1) / 2 * sizeof(short2);
}
static size_t jacobi_smem(int max_nb, int cs) {
  const size_t hv = (size_t)(max_nb + cs - 1) / cs;
  return (size_t)max_nb * (max_nb + hv) * sizeof(double2) + jacobi_tables(max_nb);
}
constexpr size_t kJacobiSmem = 227 * 1024 - 1024;   // beside the static reduction arrays

template <int CS, int LPB, typename... Args>
static void jacobi_go(int nks, size_t sm, cudaStream_t st, Args... args) {
  auto kern = k_jacobi<CS, LPB>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CS * nks);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  derek::note_launch();
  cudaLaunchKernelEx(&cfg, kern, args...);
}

void launch_jacobi(const Tables &t, int ks_begin, int nks, int max_nb, const double2 *Hs,
                   double2 *C, const long long *mat_off, double *eig, double2 *scratch,
                   int max_sweeps, double tol, int *sweeps_out, cudaStream_t st, int single) {
  if (nks <= 0) return;
  const int np = (max_nb + 1) / 2, nblk = np * (np + 1) / 2;
  // CTAs per k-set: as many as leave each its own SM (128 of them: clusters
  // do not fill every SM) and 16 blocks of a round; at least as many as make
  // A and a slice of the eigenvectors fit
  int cs = 1;
  while (!single && cs < 8 && 2 * cs * nks <= 128 && nblk >= 32 * cs) cs *= 2;
  while (cs < 8 && jacobi_smem(max_nb, cs) > kJacobiSmem) cs *= 2;
  const size_t sm = jacobi_smem(max_nb, cs);
  if (sm > kJacobiSmem) {
    const size_t tab = jacobi_tables(max_nb);
    derek::launch(k_jacobi_global, nks, 256, tab, st, t, ks_begin, Hs, C, mat_off, eig, scratch, max_sweeps,
                                                                 tol, sweeps_out);
    return;
  }
  // one element per lane (16 FP64 operations) or one block per thread (48):
  // whichever leaves the fullest quarter of the SM fewer
  auto quarter = [&](int lanes) { return ((lanes + 31) / 32 + 3) / 4; };
  const bool fine = quarter((4 * nblk + cs - 1) / cs) * 16 < quarter((nblk + cs - 1) / cs) * 48;
  auto go = [&](auto csc, auto lc) {
    jacobi_go<decltype(csc)::value, decltype(lc)::value>(nks, sm, st, t, ks_begin, Hs, C, mat_off, eig, max_sweeps, tol,
                                                        sweeps_out);
  };
  auto pick = [&](auto csc) {
    if (fine)
      go(csc, std::integral_constant<int, 4>{});
    else
      go(csc, std::integral_constant<int, 1>{});
  };
  switch (cs) {
    case 1: pick(std::integral_constant<int, 1>{}); break;
    case 2: pick(std::integral_constant<int, 2>{}); break;
    case 4: pick(std::integral_constant<int, 4>{}); break;
    default: pick(std::integral_constant<int, 8>{}); break;
  }
}

#define DEREK_INST(R)                                                                          \
  template void launch_overlap<R>(const Tables &, int, int, int, int, int, int, const cplx<R> *, \
                                  const cplx<R> *, double2 *, const long long *, double2 *,   \
                                  const long long *, int, cudaStream_t);                      \
  template void launch_rotate<R>(const Tables &, int, int, int, int, cplx<R> *,               \
                                 const double2 *, const long long *, int, cudaStream_t);
DEREK_INST(float)
DEREK_INST(double)
#undef DEREK_INST

}  // namespace derek
