// FP32 spinor (y,z)-plane pass with every line transform in one thread's
// registers (regfft.cuh), for the compiled cubic-plane lengths.
//
// A block holds XP x-planes of one band, both components.  The columns of both
// are gathered, the rows holding columns transformed along z, and then one
// thread per (plane, z) walks its column of both components without a barrier:
//   up:    kept rows -> backward y in registers -> all N rows of P0
//   down:  kept rows -> backward y in registers, kept there
//   per y: the 2x2 product of the up value in P0 and the down one in a register
//   down:  forward y -> kept rows of P1;  up: P0 -> forward y -> kept rows of P0
// so only the up plane is stored with all N rows, the down one with the
// sphere's rows (planes.cuh).  V is read once per point and band, 32 bytes,
// from L2.  As many planes as half of the shared memory holds, so that two
// blocks of an SM overlap their barriers.
// Bound by FP32 issue, as the scalar pass.  Measured at 48^3, 192 items (96
// spinor bands): 932 us with shared-memory lines of 512 threads, 182 us here.
#include <algorithm>

#include "planes.cuh"

namespace derek {
namespace {

template <int N, int RY, int XP, int NT, int BLOCKS>
__global__ void __launch_bounds__(NT, BLOCKS) k_plane_spinor_reg(Tables t, int item_begin, float2 *__restrict__ abuf,
                                                         const float4 *__restrict__ vnc) {
  grid_dependency();
  using Lay = RowsLayout<N, RY>;
  constexpr int PZ = Lay::PZ, PP1 = Lay::PP, PP0 = PlaneLayout<N>::PP;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int slot = 2 * blockIdx.x;
  const int item = t.item_list ? t.item_list[slot] : item_begin + slot;
  const KSetDev &K = t.ks[t.item_ks[item]];
  const SysDev &S = t.sys[K.sys];
  const int n1 = S.n[0], b = t.item_band[item], x0 = blockIdx.y * XP;
  if (!S.active || x0 >= n1 || (b & 1)) return;
  const int np = min(XP, n1 - x0);
  float2 *P0 = reinterpret_cast<float2 *>(smem_raw);   // up: row y at y PZ
  float2 *P1 = P0 + XP * PP0;                          // down: row my + RY
  const int tid = threadIdx.x;
  // the rows the backward y transforms read
  for (int i = tid; i < XP * Lay::NRW * PZ; i += NT) {
    const int p = i / (Lay::NRW * PZ), r = i - p * (Lay::NRW * PZ);
    const int my = r / PZ - RY, z = r % PZ;
    P0[p * PP0 + (my < 0 ? my + N : my) * PZ + z] = make_float2(0.f, 0.f);
    P1[p * PP1 + r] = make_float2(0.f, 0.f);
  }
  __syncthreads();
  const long long ld = K.ncol_pad, band = (long long)n1 * ld;
  float2 *a0 = abuf + K.a_off + (long long)b * band + (long long)x0 * ld, *a1 = a0 + band;
  const short *cy = t.col_y + K.col_off, *cz = t.col_z + K.col_off;
  const int ncol = K.ncol, nrow = K.nrow;
  for (int c = tid; c < ncol; c += NT) {
    const int y = cy[c], o0 = y * PZ + cz[c], o1 = Lay::row_of(y) * PZ + cz[c];
#pragma unroll
    for (int p = 0; p < XP; ++p)
      if (p < np) {
        P0[p * PP0 + o0] = a0[p * ld + c];
        P1[p * PP1 + o1] = a1[p * ld + c];
      }
  }
  __syncthreads();
  const short *rows = t.rows + K.row_off;
  const int nz = 2 * np * nrow;
  auto z_line = [&](int i) -> float2 * {
    const int c = i / (np * nrow), q = i - c * (np * nrow), p = q / nrow;
    const int y = rows[q - p * nrow];
    return c == 0 ? P0 + p * PP0 + y * PZ : P1 + p * PP1 + Lay::row_of(y) * PZ;
  };
  for (int i = tid; i < nz; i += NT) {
    float2 *line = z_line(i);
    float2 v[N];
    static_for<0, N>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      if constexpr (Lay::kept(j))
        v[j] = line[j];
      else
        v[j] = make_float2(0.f, 0.f);
    });
    reg_fft<N, +1, 0, Lay>(v);
    store_line<N, 1>(v, line, 1);
  }
  __syncthreads();
  if (tid < np * N) {
    const int p = tid / N, z = tid - p * N;
    float2 *up = P0 + p * PP0 + z, *dn = P1 + p * PP1 + z;
    const float4 *vz = vnc + 2 * (S.grid_off + (long long)(x0 + p) * N * N + z);
    float2 v[N];
    static_for<0, N>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      if constexpr (Lay::kept(j))
        v[j] = up[j * PZ];
      else
        v[j] = make_float2(0.f, 0.f);
    });
    reg_fft<N, +1, 0, Lay>(v);
    store_line<N, 1>(v, up, PZ);
    load_column<N, RY>(v, dn);
    reg_fft<N, +1, 0, Lay>(v);
    static_for<0, N>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      const float4 c1 = vz[2 * m * N], c2 = vz[2 * m * N + 1];   // V11, V21 and V12, V22
      const float2 u = up[m * PZ];
      float2 &d = v[line_slot<N>(m, 1)];
      up[m * PZ] = cadd<float>(cmul<float>(make_float2(c1.x, c1.y), u), cmul<float>(make_float2(c2.x, c2.y), d));
      d = cadd<float>(cmul<float>(make_float2(c1.z, c1.w), u), cmul<float>(make_float2(c2.z, c2.w), d));
      // at most four points' V in registers beside the line
      if constexpr (m % 4 == 3) asm volatile("" ::: "memory");
    });
    reg_fft<N, -1, 1>(v);
    static_for<0, N>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      if constexpr (Lay::kept(m)) dn[Lay::row_of(m) * PZ] = v[line_slot<N>(m, 2)];
    });
    load_line<N>(v, up, PZ);
    reg_fft<N, -1, 0>(v);
    static_for<0, N>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      if constexpr (Lay::kept(m)) up[m * PZ] = v[line_slot<N>(m, 1)];
    });
  }
  __syncthreads();
  for (int i = tid; i < nz; i += NT) {
    float2 *line = z_line(i);
    float2 v[N];
    load_line<N>(v, line, 1);
    reg_fft<N, -1, 0>(v);
    static_for<0, N>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      if constexpr (Lay::kept(m)) line[m] = v[line_slot<N>(m, 1)];
    });
  }
  __syncthreads();
  for (int c = tid; c < ncol; c += NT) {
    const int y = cy[c], o0 = y * PZ + cz[c], o1 = Lay::row_of(y) * PZ + cz[c];
#pragma unroll
    for (int p = 0; p < XP; ++p)
      if (p < np) {
        a0[p * ld + c] = P0[p * PP0 + o0];
        a1[p * ld + c] = P1[p * PP1 + o1];
      }
  }
}

template <int N, int RY>
void spinor_go(const Tables &t, int item_begin, int nitems, int n1, float2 *abuf, const float2 *vnc, cudaStream_t st) {
  constexpr int PLANE = (PlaneLayout<N>::PP + RowsLayout<N, RY>::PP) * 8;
  constexpr int HALF = (kSmemMax / 2 - 1024) / PLANE, ALL = kSmemMax / PLANE;
  constexpr int FIT = HALF >= 2 ? HALF : ALL;
  constexpr int XP = FIT < kThreadsMax / N ? FIT : kThreadsMax / N;
  static_assert(XP >= 1, "a plane pair fits the shared memory");
  constexpr int NT = (N * XP + 31) / 32 * 32;
  auto kern = k_plane_spinor_reg<N, RY, XP, NT, HALF >= 2 ? 2 : 1>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, XP * PLANE);
  derek::launch(kern, dim3(nitems / 2, (n1 + XP - 1) / XP), NT, XP * PLANE, st, t, item_begin, abuf, reinterpret_cast<const float4 *>(vnc));
}

template <int N>
void spinor_n(const Tables &t, int item_begin, int nitems, int n1, int max_m, float2 *abuf, const float2 *vnc,
              cudaStream_t st) {
  if constexpr (tight_ry<N>() > 0) {
    if (max_m <= tight_ry<N>()) return spinor_go<N, tight_ry<N>()>(t, item_begin, nitems, n1, abuf, vnc, st);
  }
  if (max_m <= compact_ry<N>())
    spinor_go<N, compact_ry<N>()>(t, item_begin, nitems, n1, abuf, vnc, st);
  else
    spinor_go<N, N / 2>(t, item_begin, nitems, n1, abuf, vnc, st);
}

}  // namespace

bool launch_plane_spinor_reg(const Tables &t, int item_begin, int nitems, const int n[3], int max_m, float2 *abuf,
                             const float2 *vnc, cudaStream_t st) {
  if (n[1] != n[2]) return false;
  switch (n[1]) {
    case 72: spinor_n<72>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 64: spinor_n<64>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 54: spinor_n<54>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 48: spinor_n<48>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 36: spinor_n<36>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 32: spinor_n<32>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 27: spinor_n<27>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    case 24: spinor_n<24>(t, item_begin, nitems, n[0], max_m, abuf, vnc, st); return true;
    default: return false;
  }
}

}  // namespace derek
