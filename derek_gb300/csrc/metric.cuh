// |G|^2 on the fine grid.
#pragma once

#include "common.cuh"

namespace derek {

// |G|^2 = m^T W m of a grid point, W = B^T B.  Exactly zero at G = 0.
struct Metric {
  double w00, w01, w02, w11, w12, w22;
  __device__ __forceinline__ explicit Metric(const SysDev &S) {
    w00 = w01 = w02 = w11 = w12 = w22 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double x = S.B[3 * i], y = S.B[3 * i + 1], z = S.B[3 * i + 2];
      w00 += x * x;
      w01 += 2.0 * x * y;
      w02 += 2.0 * x * z;
      w11 += y * y;
      w12 += 2.0 * y * z;
      w22 += z * z;
    }
  }
  // of the FFT indices (ix, iy, iz)
  __device__ __forceinline__ double gsq(const SysDev &S, int ix, int iy, int iz) const {
    const int n1 = S.n[0], n2 = S.n[1], n3 = S.n[2];
    const double m0 = ix < n1 - n1 / 2 ? ix : ix - n1;
    const double m1 = iy < n2 - n2 / 2 ? iy : iy - n2;
    const double m2 = iz < n3 - n3 / 2 ? iz : iz - n3;
    return m0 * (w00 * m0 + w01 * m1 + w02 * m2) + m1 * (w11 * m1 + w12 * m2) + w22 * m2 * m2;
  }
};

}  // namespace derek
