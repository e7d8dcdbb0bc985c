// Device helpers shared by the Krylov and multigrid kernels.
#pragma once

#include "kernels.cuh"

namespace anb {

template <class T>
__device__ __forceinline__ double ld(const T* p) {
  return (double)__ldg(p);
}

// Row r's slots in registers, for a compile-time bound WM on the slice width: every column and
// value load of the row is issued before the first gather, so a row costs two dependent memory
// round trips instead of two per unrolled group.  Slots past the row's slice width are
// (column r, value 0) and read nothing.
template <int WM, class T>
__device__ __forceinline__ void sell_regs(const int* sliceOff, const int* col, const T* val, int r, int (&c)[WM],
                                          double (&v)[WM]) {
  const int s = r >> 5;
  const int b0 = __ldg(&sliceOff[s]);
  const int W = (__ldg(&sliceOff[s + 1]) - b0) >> 5;
  const int b = b0 + (r & 31);
#pragma unroll
  for (int k = 0; k < WM; ++k) {
    c[k] = r;
    v[k] = 0.0;
    if (k < W) {
      c[k] = __ldg(&col[b + (k << 5)]);
      v[k] = ld(&val[b + (k << 5)]);
    }
  }
}

// Iteration count and convergence test on |r|^2 = rr (last block, thread 0).
template <class T>
__device__ __forceinline__ void pcg_converged(const PcgArgsT<T>& a, double rr) {
  a.sc[4] = rr;
  a.fl[1] += 1;
  if (sqrt(rr) <= a.sc[3]) {
    a.fl[0] = 1;
    a.fl[2] = 1;
  } else if (a.fl[1] >= a.maxit || a.sc[5] == 0.0) {
    a.fl[0] = 1;
    a.fl[2] = 0;
  }
}

// Sum over G consecutive lanes, valid in the first.
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o, G);
  return v;
}

}  // namespace anb
