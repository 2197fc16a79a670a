// Line DFTs over shared memory: two digit steps, every lane busy.
//
// A line of n = a b points (a, b <= 16) is an a x b array of digits.  Backward:
// radix-a transforms over the first digit, then radix-b ones over the second;
// forward: the same two steps in the other order.  Both work in place on the
// slots of the line, so after the backward transform element m sits in slot
// line_slot_of(m), and a forward transform takes it from there back to the
// natural order: the passes multiply by V(r) or sum densities at permuted
// slots and never move data to undo the permutation.
//   Coprime a, b: prime-factor maps (Good-Thomas), slot (b n1 + a n2) mod n and
//   slot(m) = (a + b) m mod n; no twiddles.
//   Otherwise Cooley-Tukey: slot b n1 + n2, slot(m) = b (m mod a) + m div a,
//   twiddles W_n^{n2 k1} after the first step of either direction.
// The unit of work is one radix transform of one line, and the units of all
// lines of a pass are dealt to the block's threads one after another (lines
// fastest), with a block barrier per step.  GB300's FP64 pipe takes 16 clocks
// of an SM per warp instruction however few of its lanes are active, so the
// earlier form (a warp per group of floor(32 / max(a, b)) whole lines, 27 and
// 24 of 32 lanes at n = 72) lost a fifth of the pipe.  With the leaner radix
// transforms (fft_smem.cuh) and two blocks per SM the FP64 plane pass went from
// 18.5 to 11.8 ms (72^3, 336 items; 9.9 ms of pipe time), an FP64 SCF on 44^3
// (radix 11) from 525 to 59 ms.
// SIGN = -1 is the forward transform (exponent -i, FFTW_FORWARD), +1 the
// backward one; neither is normalised (Source/fft.f90:204-212).
#pragma once

#include "fft_smem.cuh"

namespace derek {

// slot that holds element m after a backward transform, and the element a
// slot holds
__device__ __forceinline__ int line_slot_of(const LinePlan &p, int m) {
  return p.pfa ? (m * (p.a + p.b)) % p.n : p.b * (m % p.a) + m / p.a;
}
__device__ __forceinline__ int line_elem_of(const LinePlan &p, int s) {
  return p.pfa ? (s * p.inv) % p.n : s / p.b + p.a * (s % p.b);
}

// The steps are separate functions (one per radix), so they take offsets into
// the block's dynamic shared memory instead of pointers: their accesses stay
// shared-memory instructions.
template <typename R_> __device__ __forceinline__ int smem_offset(const cplx<R_> *p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return (int)(reinterpret_cast<const unsigned char *>(p) - smem_raw);
}
template <typename R_> __device__ __forceinline__ cplx<R_> *smem_at(int off) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  return reinterpret_cast<cplx<R_> *>(smem_raw + off);
}
// i / d for 0 <= i < 2^13, 1 <= d <= 128 as (i * line_magic(d)) >> 20: the
// magic number exceeds 2^20 / d by less than 1, so the quotient is exact while
// i d < 2^20
__device__ __forceinline__ unsigned line_magic(int d) { return ((1u << 20) + d - 1) / d; }

// One digit step of a line set: units u < nu of every line, unit u's elements
// at slots u start + k inc (mod n), k < R.  tw: twiddles W_n^{u k} after the
// transform (offset, or -1 for none).
template <typename R_, int SIGN, int R>
__device__ __noinline__ void line_step(int buf_off, int nlines, int ldist, int es, const short *lines, int n, int nu,
                                       int start, int inc, int tw_off) {
  cplx<R_> *buf = smem_at<R_>(buf_off);
  const int total = nlines * nu;
  const unsigned magic = line_magic(nlines);
  const int ne = n * es;
  start *= es;
  inc *= es;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int u = (i * magic) >> 20, l = i - u * nlines;
    cplx<R_> *line = buf + (lines ? (int)lines[l] : l) * ldist;
    int o[R];
    int s = u * start;
    cplx<R_> v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      o[k] = s;
      v[k] = line[s];
      s += inc;
      if (s >= ne) s -= ne;
    }
    Dft<R_, R, SIGN>::run(v);
    if (tw_off >= 0) {
      const cplx<R_> *tw = smem_at<R_>(tw_off);
      int idx = 0;
#pragma unroll
      for (int k = 1; k < R; ++k) {
        idx += u;
        if (idx >= n) idx -= n;
        cplx<R_> w = tw[idx];
        if (SIGN > 0) w.y = -w.y;
        v[k] = cmul<R_>(v[k], w);
      }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) line[o[k]] = v[k];
  }
}

// Last backward step, times V, first forward step, over the second digit:
// both transforms of a unit touch the same slots, so V(r) is applied in
// registers.  Line l's element m multiplies with v[m vstride + line_elem_of(pl, l)].
template <typename R_, int R>
__device__ __noinline__ void line_step_v(int buf_off, int nlines, int es, const LinePlan &p, const LinePlan &pl,
                                         const R_ *__restrict__ v, int vstride, int tw_off) {
  cplx<R_> *buf = smem_at<R_>(buf_off);
  const int n = p.n, total = nlines * p.a, pfa = p.pfa;
  const unsigned magic = line_magic(nlines);
  const int ne = n * es;
  const int inc = (pfa ? p.a : 1) * es;
  const int minc = pfa ? (p.a * p.inv) % n : p.a;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int u = (i * magic) >> 20, l = i - u * nlines;
    cplx<R_> *line = buf + l;
    int m = line_elem_of(p, p.b * u);
    int s = p.b * u * es;
    const R_ *vl = v + line_elem_of(pl, l);
    int o[R];
    R_ w[R];
    cplx<R_> x[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      o[k] = s;
      w[k] = vl[m * vstride];
      x[k] = line[s];
      s += inc;
      if (s >= ne) s -= ne;
      m += minc;
      if (m >= n) m -= n;
    }
    Dft<R_, R, +1>::run(x);
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = cscale<R_>(x[k], w[k]);
    Dft<R_, R, -1>::run(x);
    if (!pfa) {
      const cplx<R_> *tw = smem_at<R_>(tw_off);
      int idx = 0;
#pragma unroll
      for (int k = 1; k < R; ++k) {
        idx += u;
        if (idx >= n) idx -= n;
        x[k] = cmul<R_>(x[k], tw[idx]);
      }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) line[o[k]] = x[k];
  }
}

#define DEREK_RADIX_SWITCH(r, F) \
  switch (r) {                   \
    case 2: F(2); break;         \
    case 3: F(3); break;         \
    case 4: F(4); break;         \
    case 5: F(5); break;         \
    case 6: F(6); break;         \
    case 7: F(7); break;         \
    case 8: F(8); break;         \
    case 9: F(9); break;         \
    case 10: F(10); break;       \
    case 11: F(11); break;       \
    case 12: F(12); break;       \
    case 13: F(13); break;       \
    case 14: F(14); break;       \
    case 15: F(15); break;       \
    case 16: F(16); break;       \
    default: break;              \
  }

// the step over the first digit (a points) or the second one (b points)
template <typename R_, int SIGN>
__device__ __forceinline__ void line_step_a(cplx<R_> *buf, const LinePlan &p, int nlines, int ldist, int es,
                                            const short *lines, const cplx<R_> *tw) {
  const int off = smem_offset<R_>(buf), tw_off = tw ? smem_offset<R_>(tw) : -1;
#define F(r) line_step<R_, SIGN, r>(off, nlines, ldist, es, lines, p.n, p.b, p.pfa ? p.a : 1, p.b, tw_off)
  DEREK_RADIX_SWITCH(p.a, F)
#undef F
}
template <typename R_, int SIGN>
__device__ __forceinline__ void line_step_b(cplx<R_> *buf, const LinePlan &p, int nlines, int ldist, int es,
                                            const short *lines, const cplx<R_> *tw) {
  const int off = smem_offset<R_>(buf), tw_off = tw ? smem_offset<R_>(tw) : -1;
#define F(r) line_step<R_, SIGN, r>(off, nlines, ldist, es, lines, p.n, p.a, p.b, p.pfa ? p.a : 1, tw_off)
  DEREK_RADIX_SWITCH(p.b, F)
#undef F
}

// In-place transform of `nlines` lines held in shared memory: line l (or
// lines[l] when a list is given) starts at buf + line * ldist, slot i at
// + i * es.  Backward: natural order in, slot order out; forward: slot order
// in, natural order out.  All threads of the block call it; it ends with
// __syncthreads().
template <typename R_, int SIGN>
__device__ void fft4_lines(cplx<R_> *buf, const LinePlan &p, int nlines, int ldist, int es,
                           const short *lines, const cplx<R_> *__restrict__ tw) {
  const cplx<R_> *w = p.pfa ? nullptr : tw;
  if (SIGN > 0) {
    line_step_a<R_, SIGN>(buf, p, nlines, ldist, es, lines, w);
    __syncthreads();
    line_step_b<R_, SIGN>(buf, p, nlines, ldist, es, lines, nullptr);
  } else {
    line_step_b<R_, SIGN>(buf, p, nlines, ldist, es, lines, w);
    __syncthreads();
    line_step_a<R_, SIGN>(buf, p, nlines, ldist, es, lines, nullptr);
  }
  __syncthreads();
}

// The backward and forward transforms of a plane's columns around V(r): column
// l (slot l of plan pl's lines) at buf + l, slots es apart; the three steps
// are a-radix, b-radix times V times b-radix, a-radix.
template <typename R_>
__device__ void fft4_columns_v(cplx<R_> *buf, const LinePlan &p, const LinePlan &pl, int ncols, int es,
                               const R_ *__restrict__ v, int vstride, const cplx<R_> *__restrict__ tw) {
  line_step_a<R_, +1>(buf, p, ncols, 1, es, nullptr, p.pfa ? nullptr : tw);
  __syncthreads();
  const int off = smem_offset<R_>(buf), tw_off = smem_offset<R_>(tw);
#define F(r) line_step_v<R_, r>(off, ncols, es, p, pl, v, vstride, tw_off)
  if (p.b > 1) {
    DEREK_RADIX_SWITCH(p.b, F)
  } else {
    line_step_v<R_, 1>(off, ncols, es, p, pl, v, vstride, tw_off);
  }
#undef F
  __syncthreads();
  line_step_a<R_, -1>(buf, p, ncols, 1, es, nullptr, nullptr);
  __syncthreads();
}

constexpr int plan_a(int n) {
  int best = 0, span = 1 << 30, p2 = 0;
  for (int x = 1; x <= 16; ++x) {
    if (n % x) continue;
    const int y = n / x;
    if (y > 16) continue;
    const int s = x > y ? x : y;
    const int q = ((x & (x - 1)) == 0 && x > 1) ? 1 : 0;
    if (s < span || (s == span && q > p2)) {
      best = x;
      span = s;
      p2 = q;
    }
  }
  return best;
}

}  // namespace derek
