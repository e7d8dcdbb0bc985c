// Smoothed-aggregation V(1,1)-cycle of the pressure CG and the refresh of its values (sm_100a),
// standing in for the reference's BoomerAMG (main.cu:2224-2273).
//
// With one weighted-Jacobi sweep before and after the coarse correction, the cycle of a level is
//   M^-1 b = w (b + r1) + Q A_c^-1 P^T r1,   r1 = b - A w b,   Q = (I - w A) P,   P^T r1 = Q^T b:
// the post-smoothing is part of Q, which is stored, so no second product with A is needed.  Level 0
// computes r1 (fused with the update of the PCG iteration) and restricts it with P^T (3.6 entries a
// row on hexes against 8.6 of Q); the coarser levels, where a launch costs more than the bytes,
// restrict b with Q^T and compute r1 in the up sweep: two launches a level.
//
// The weights are w = omega / a_ii on the finest level, whose rows are diagonally dominant.  The coarse
// matrices have positive off-diagonals too and no such bound (the largest eigenvalue of D^-1 A reaches 2.4
// where the coefficients spread over 1e6), so there w = min(omega / a_ii, 1.99 / sum_j |a_ij|): the matrix
// of row sums minus A is positive semidefinite, hence w A < 2 and the cycle stays positive definite
// whatever the coefficients.  Where the bound does not bind the weights are those of omega alone;
// on isotropic grids the iterations are the same.
//
// Against the plain aggregation with over-correction (kernels_krylov.cu) the CG needs half the
// iterations (143 -> 66 per SIMPLE step on 970k hexes, 151 -> 80 on 334k tets, both to 1e-15) with
// 11 launches each instead of 17; a step took 30.2 -> 17.5 ms and 13.4 -> 8.7 ms.  An iteration moves
// 0.5 GB at 970k cells (A twice, Q, P^T, the level-1 matrices) in 170 us: the level-0 kernels run at
// 3.5-4 TB/s like the other SELL kernels, the levels below 5,000 rows at launch latency.
#include <algorithm>

#include <cooperative_groups.h>

#include "krylov_dev.cuh"

namespace anb {
namespace {

namespace cg = cooperative_groups;

// ---------------------------------------------------------------- solve

// k_amg_resid0 without the pre-smoothed iterate, which the up sweep forms again from r and r1:
// r_new = r - alpha q, x += alpha p, |r_new|^2 with the convergence test, r1 = r_new - A w r_new.
template <class T, int WM>
__global__ void __launch_bounds__(kBlock) k_sa_resid0(PcgArgsT<T> a, AmgLevelDevT<T> f, const T* rIn, T* rOut,
                                                      const T* p) {
  __shared__ double sm[32];
  if (a.fl[0]) return;
  const bool upd = a.fl[3] == 0;
  const double al = upd ? a.sc[1] : 0.0;
  double acc[1] = {0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += gridDim.x * blockDim.x) {
    double ri;
    if (upd) {
      const double rr = __fma_rn(-al, ld(&a.q[i]), ld(&rIn[i]));
      acc[0] += rr * rr;
      ri = (double)(T)rr;
      a.x[i] = (T)__fma_rn(al, (double)p[i], (double)a.x[i]);
    } else {
      ri = ld(&rIn[i]);
    }
    rOut[i] = (T)ri;
    double ax = ld(&f.diag[i]) * (ld(&f.wdinv[i]) * ri);
    auto add = [&](int j, double v) {
      const double rj = upd ? (double)(T)__fma_rn(-al, ld(&a.q[j]), ld(&rIn[j])) : ld(&rIn[j]);
      ax += v * (ld(&f.wdinv[j]) * rj);
    };
    if constexpr (WM == 0) {
      const int s = i >> 5;
      const int b = __ldg(&f.sliceOff[s]) + (i & 31);
      const int W = (__ldg(&f.sliceOff[s + 1]) - __ldg(&f.sliceOff[s])) >> 5;
#pragma unroll 4
      for (int k = 0; k < W; ++k) add(__ldg(&f.col[b + (k << 5)]), ld(&f.val[b + (k << 5)]));
    } else {
      int c[WM];
      double v[WM];
      sell_regs<WM>(f.sliceOff, f.col, f.val, i, c, v);
#pragma unroll
      for (int k = 0; k < WM; ++k) add(c[k], v[k]);
    }
    f.x2[i] = (T)(ri - ax);
  }
  if (!upd) return;  // uniform over the grid
  if (grid_reduce<1>(acc, 0u, a.red, sm) && threadIdx.x == 0) pcg_converged(a, acc[0]);
}

// Restriction: b_next = R x (R = P^T or Q^T by coarse rows), G lanes a row; with w given also the
// pre-smoothed iterate w b_next, which the up sweep of that level gathers.
template <int G, class T>
__global__ void __launch_bounds__(kBlock) k_sa_restrict(const int* done, int n, const int* off, const int* col,
                                                        const T* val, const T* x, T* bNext, const T* w, T* xNext) {
  if (*done) return;
  const int lane = threadIdx.x & 31, sub = lane % G;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nWarps = (gridDim.x * blockDim.x) >> 5;
  for (int base = warp * (32 / G); base < n; base += nWarps * (32 / G)) {
    const int i = base + lane / G;
    double acc = 0.0;
    if (i < n) {
      const int k1 = __ldg(&off[i + 1]);
#pragma unroll 8
      for (int k = __ldg(&off[i]) + sub; k < k1; k += G) acc += ld(&val[k]) * ld(&x[__ldg(&col[k])]);
    }
    acc = group_sum<G>(acc);
    if (i < n && sub == 0) {
      const T b = (T)acc;
      bNext[i] = b;
      if (w) xNext[i] = (T)(ld(&w[i]) * (double)b);
    }
  }
}

// The same with a block a row, for the few long rows of the deep levels (500 rows of 400 entries: a
// warp a row walks them in 13 dependent steps, 18 us).
template <class T>
__global__ void __launch_bounds__(kBlock) k_sa_restrict_block(const int* done, const int* off, const int* col,
                                                              const T* val, const T* x, T* bNext, const T* w, T* xNext) {
  __shared__ double sm[32];
  if (*done) return;
  const int i = blockIdx.x, k1 = __ldg(&off[i + 1]);
  double acc[1] = {0.0};
#pragma unroll 4
  for (int k = __ldg(&off[i]) + threadIdx.x; k < k1; k += kBlock) acc[0] += ld(&val[k]) * ld(&x[__ldg(&col[k])]);
  block_reduce<1>(acc, 0u, sm);
  if (threadIdx.x == 0) {
    const T b = (T)acc[0];
    bNext[i] = b;
    if (w) xNext[i] = (T)(ld(&w[i]) * (double)b);
  }
}

// Up sweep of a coarse level: out = x + w r1 + Q e with x = w b and r1 = b - A x, i.e.
// (2 - w_i a_ii) x_i + sum of the row [-w_i A_offdiag | Q] times [x | e].  The two matrices are stored as
// one CSR and the two vectors as one array, so a row is a single gather sum; G lanes a row.
template <int G, class T>
__global__ void __launch_bounds__(kBlock) k_sa_up(const int* done, AmgLevelDevT<T> f, T* out) {
  if (*done) return;
  const int lane = threadIdx.x & 31, sub = lane % G;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nWarps = (gridDim.x * blockDim.x) >> 5;
  for (int base = warp * (32 / G); base < f.n; base += nWarps * (32 / G)) {
    const int i = base + lane / G;
    double y = 0.0;
    if (i < f.n) {
      if (sub == 0) y = (2.0 - ld(&f.wdinv[i]) * ld(&f.diag[i])) * ld(&f.x[i]);
      const int k1 = __ldg(&f.mOff[i + 1]);
#pragma unroll 8
      for (int k = __ldg(&f.mOff[i]) + sub; k < k1; k += G) y += ld(&f.mVal[k]) * ld(&f.x[__ldg(&f.mCol[k])]);
    }
    y = group_sum<G>(y);
    if (i < f.n && sub == 0) out[i] = (T)y;
  }
}

// Up sweep of level 0: z = w (r + r1) + Q e, thread a row over the SELL-32 Q (rows of at most
// kQChunk entries issue all their loads before the first use), with r.z and beta of the PCG.
constexpr int kQChunk = 12;
template <class T>
__global__ void __launch_bounds__(kBlock) k_sa_up0(AmgLevelDevT<T> f, const T* e, PcgArgsT<T> a) {
  __shared__ double sm[32];
  if (a.fl[0]) return;
  double acc[1] = {0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < f.n; i += gridDim.x * blockDim.x) {
    const int len = __ldg(&f.qOff[i + 1]) - __ldg(&f.qOff[i]);
    const int b = __ldg(&f.qSlice[i >> 5]) + (i & 31);
    const double r = ld(&f.b[i]);
    double z = ld(&f.wdinv[i]) * (r + ld(&f.x2[i]));
    for (int k0 = 0; k0 < len; k0 += kQChunk) {
      int c[kQChunk];
      double v[kQChunk];
#pragma unroll
      for (int k = 0; k < kQChunk; ++k) {
        c[k] = 0;
        v[k] = 0.0;
        if (k0 + k < len) {
          c[k] = __ldg(&f.qColS[b + ((k0 + k) << 5)]);
          v[k] = ld(&f.qVal[b + ((k0 + k) << 5)]);
        }
      }
#pragma unroll
      for (int k = 0; k < kQChunk; ++k)
        if (k0 + k < len) z += v[k] * ld(&e[c[k]]);
    }
    const T zn = (T)z;
    a.z[i] = zn;
    acc[0] += r * (double)zn;
  }
  if (grid_reduce<1>(acc, 0u, a.red, sm) && threadIdx.x == 0) {
    const double rzOld = a.sc[0];
    a.sc[2] = a.fl[3] ? 0.0 : acc[0] / rzOld;
    a.sc[0] = acc[0];
  }
}

// Coarsest level: x = A^-1 b with the stored inverse, a warp a row.
template <class T>
__global__ void __launch_bounds__(kBlock) k_sa_dense(const int* done, int n, const double* inv, const T* b, T* x) {
  if (*done) return;
  const int lane = threadIdx.x & 31;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  double s = 0.0;
#pragma unroll 5
  for (int j = lane; j < n; j += 32) s += __ldg(&inv[(size_t)i * n + j]) * ld(&b[j]);
  s = warp_sum(s);
  if (lane == 0) x[i] = (T)s;
}

// The small levels in one launch: restriction down to the dense level, its solve and the up sweeps, on
// one thread-block cluster whose barriers order the phases.  Vectors written inside the launch are
// read through L2; all CTAs take the same barriers (uniform loop bounds and done flag).
constexpr int kTailThreads = 1024;
constexpr int kTailMaxLevels = 6;
template <class T>
struct SaTailArgs {
  int nLev;
  AmgLevelDevT<T> lv[kTailMaxLevels];
  const double* dense;
};

// Rows of the cluster's CTAs in turn, a team of TS threads of one CTA a row.
template <int TS, class T>
__device__ __forceinline__ void tail_restrict(const AmgLevelDevT<T>& f, const AmgLevelDevT<T>& c, bool last, int rank,
                                              int nCta, double (&sm)[kTailThreads / 32]) {
  constexpr int kTeams = kTailThreads / TS;
  const int team = threadIdx.x / TS, tt = threadIdx.x % TS, lane = threadIdx.x & 31;
  for (int r0 = 0; r0 < c.n; r0 += nCta * kTeams) {  // uniform over the cluster
    const int i = r0 + team * nCta + rank;
    double acc = 0.0;
    if (i < c.n) {
      const int k1 = __ldg(&f.tOff[i + 1]);
#pragma unroll 4
      for (int k = __ldg(&f.tOff[i]) + tt; k < k1; k += TS)
        acc += ld(&f.tVal[k]) * (double)__ldcg(&f.b[__ldg(&f.tCol[k])]);
    }
    acc = warp_sum(acc);
    if constexpr (TS > 32) {
      if (lane == 0) sm[threadIdx.x >> 5] = acc;
      __syncthreads();
      if (tt == 0) {
        acc = 0.0;
#pragma unroll
        for (int u = 0; u < TS / 32; ++u) acc += sm[(threadIdx.x >> 5) + u];
      }
      __syncthreads();
    }
    if (i < c.n && tt == 0) {
      const T b = (T)acc;
      c.b[i] = b;
      if (!last) c.x[i] = (T)(ld(&c.wdinv[i]) * (double)b);
    }
  }
}

template <int G, class T>
__device__ __forceinline__ void tail_up(const AmgLevelDevT<T>& f, int warp, int nWarps) {
  const int lane = threadIdx.x & 31, sub = lane % G;
  for (int base = warp * (32 / G); base < f.n; base += nWarps * (32 / G)) {
    const int i = base + lane / G;
    double y = 0.0;
    if (i < f.n) {
      if (sub == 0) y = (2.0 - ld(&f.wdinv[i]) * ld(&f.diag[i])) * (double)__ldcg(&f.x[i]);
      const int k1 = __ldg(&f.mOff[i + 1]);
#pragma unroll 8
      for (int k = __ldg(&f.mOff[i]) + sub; k < k1; k += G)
        y += ld(&f.mVal[k]) * (double)__ldcg(&f.x[__ldg(&f.mCol[k])]);
    }
    y = group_sum<G>(y);
    if (i < f.n && sub == 0) f.x2[i] = (T)y;
  }
}

template <class T>
__global__ void __launch_bounds__(kTailThreads, 1) k_sa_tail(const int* done, const __grid_constant__ SaTailArgs<T> a) {
  if (*done) return;
  cg::cluster_group cl = cg::this_cluster();
  __shared__ double sm[kTailThreads / 32];
  const int rank = (int)cl.block_rank(), nCta = (int)cl.num_blocks();
  const int t = rank * blockDim.x + threadIdx.x;
  const int warp = t >> 5, nWarps = (nCta * blockDim.x) >> 5;
  const int L = a.nLev;
  for (int l = 0; l + 1 < L; ++l) {
    const bool last = l + 2 == L;
    if (a.lv[l + 1].n > 8 * nCta) tail_restrict<32>(a.lv[l], a.lv[l + 1], last, rank, nCta, sm);
    else tail_restrict<128>(a.lv[l], a.lv[l + 1], last, rank, nCta, sm);
    cl.sync();
  }
  const AmgLevelDevT<T>& d = a.lv[L - 1];
  for (int i = warp; i < d.n; i += nWarps) {
    const int lane = threadIdx.x & 31;
    double s = 0.0;
#pragma unroll 4
    for (int j = lane; j < d.n; j += 32) s += __ldg(&a.dense[(size_t)i * d.n + j]) * (double)__ldcg(&d.b[j]);
    s = warp_sum(s);
    if (lane == 0) d.x2[i] = (T)s;
  }
  for (int l = L - 2; l >= 0; --l) {
    cl.sync();
    if (a.lv[l].n > 32 * nCta) tail_up<16>(a.lv[l], warp, nWarps);
    else tail_up<32>(a.lv[l], warp, nWarps);
  }
}

cudaLaunchConfig_t tail_config(cudaStream_t s, int cluster, cudaLaunchAttribute* at) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(cluster);
  cfg.blockDim = dim3(kTailThreads);
  cfg.stream = s;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// ---------------------------------------------------------------- refresh
// All sums in double and in a fixed order: the values do not depend on the launch shape.

// First entry, count and stride of row i's off-diagonals (SELL-32 or CSR).
template <class T>
__device__ __forceinline__ void row_entries(const AmgLevelDevT<T>& f, int i, int& b, int& cnt, int& stride) {
  if (f.sliceOff) {
    const int s = i >> 5, o = __ldg(&f.sliceOff[s]);
    b = o + (i & 31);
    cnt = (__ldg(&f.sliceOff[s + 1]) - o) >> 5;
    stride = 32;
  } else {
    b = __ldg(&f.rowOff[i]);
    cnt = __ldg(&f.rowOff[i + 1]) - b;
    stride = 1;
  }
}

// P = (I - omegaP D^-1 A) P0: G lanes a row, which sum each entry of P over the row's matrix entries
// in turn (padding slots hold value 0).  With omegaP = 0 the only entry, of the own aggregate, is 1.
template <int G, class T>
__global__ void __launch_bounds__(kBlock) k_sa_p(AmgLevelDevT<T> f) {
  const int lane = threadIdx.x & 31, sub = lane % G;
  const int base = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32 / G);
  const int i = base + lane / G;
  int b = 0, cnt = 0, st = 1, k0 = 0, nk = 0, own = -1;
  double d = 1.0;
  if (i < f.n) {
    row_entries(f, i, b, cnt, st);
    d = ld(&f.diag[i]);
    own = __ldg(&f.agg[i]);
    k0 = __ldg(&f.pOff[i]);
    nk = __ldg(&f.pOff[i + 1]) - k0;
  }
  const double s = d != 0.0 ? f.omegaP / d : 0.0;
  int most = nk;  // the rows of a warp run the same number of sums: group_sum needs every lane
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
  for (int k = 0; k < most; ++k) {
    const int I = k < nk ? __ldg(&f.pCol[k0 + k]) : -1;
    double acc = (I == own && sub == 0) ? d : 0.0;
    if (I >= 0) {
#pragma unroll 4
      for (int e = sub; e < cnt; e += G)
        if (__ldg(&f.agg[__ldg(&f.col[b + e * st])]) == I) acc += ld(&f.val[b + e * st]);
    }
    acc = group_sum<G>(acc);
    if (I >= 0 && sub == 0) f.pVal[k0 + k] = (T)((I == own ? 1.0 : 0.0) - s * acc);
  }
}

// A sparse product by rows, C = sum over e of coef_e B_row(e), on a fixed pattern of C.  A team of TS
// threads takes a row of C; its groups of G lanes take the terms e in turn and add the (distinct)
// columns of one row of B to the group's own copy of the row of C in shared memory, the position found
// by bisection of C's sorted columns; the copies are summed in group order, so the result does not
// depend on timing.  kAP: C = A P by fine rows (written as A P and Q = P - w A P); otherwise the
// next level's matrix P^T (A P) with its diagonal apart.  cap: longest row of C (+ 1).
template <int G, int TS, bool kAP, class T>
__global__ void __launch_bounds__(kBlock) k_sa_product(AmgLevelDevT<T> f, AmgLevelDevT<T> c, double omega, int cap) {
  extern __shared__ double sh[];
  constexpr int NG = TS / G, kTeams = kBlock / TS;
  const int team = threadIdx.x / TS, tt = threadIdx.x % TS, grp = tt / G, sub = tt % G;
  double* acc = sh + (size_t)team * NG * cap;
  int* cols = reinterpret_cast<int*>(sh + (size_t)kTeams * NG * cap) + (size_t)team * cap;
  const unsigned mask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << ((threadIdx.x & 31) / G * G);
  const int r = blockIdx.x * kTeams + team;  // one row a team: grid covers the rows
  const int rows = kAP ? f.n : c.n;
  const bool live = r < rows;
  auto sync = [] {
    if constexpr (TS > 32) __syncthreads();
    else __syncwarp();
  };
  int c0 = 0, nc = 0, e0 = 0, ne = 0, st = 1;
  if (live) {
    const int* off = kAP ? f.qOff : c.rowOff;
    c0 = __ldg(&off[r]);
    nc = __ldg(&off[r + 1]) - c0;
    if (kAP) {
      row_entries(f, r, e0, ne, st);
      ++ne;  // the diagonal first
    } else {
      e0 = __ldg(&f.ptOff[r]);
      ne = __ldg(&f.ptOff[r + 1]) - e0;
    }
    const int* cc = kAP ? f.qCol : c.col;
    for (int s = tt; s < nc; s += TS) cols[s] = __ldg(&cc[c0 + s]);
    for (int s = sub; s <= nc && s < cap; s += G) acc[grp * cap + s] = 0.0;
  }
  sync();
  if (live) {
    for (int e = grp; e < ne; e += NG) {
      int b;
      double a;
      if (kAP) {
        b = e == 0 ? r : __ldg(&f.col[e0 + (e - 1) * st]);
        a = e == 0 ? ld(&f.diag[r]) : ld(&f.val[e0 + (e - 1) * st]);
      } else {
        b = __ldg(&f.ptCol[e0 + e]);
        a = ld(&f.pVal[__ldg(&f.ptSrc[e0 + e])]);
      }
      const int* bOff = kAP ? f.pOff : f.qOff;
      const int* bCol = kAP ? f.pCol : f.qCol;
      const T* bVal = kAP ? f.pVal : f.apVal;
      const int k1 = __ldg(&bOff[b + 1]);
      for (int k = __ldg(&bOff[b]) + sub; k < k1; k += G) {
        const int J = __ldg(&bCol[k]);
        const double v = ld(&bVal[k]);
        int lo = 0;
        if (!kAP && J == r) {
          lo = nc;
        } else {
          int hi = nc;  // the first column >= J, which is J: the pattern holds every product
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (cols[mid] < J) lo = mid + 1;
            else hi = mid;
          }
        }
        acc[grp * cap + lo] += a * v;
      }
      __syncwarp(mask);
    }
  }
  sync();
  if (!live) return;
  double size = 0.0, diag = 0.0;  // sum of |a| over the row; the diagonal in the thread that has it
  for (int s = tt; s < nc + (kAP ? 0 : 1); s += TS) {
    double sum = 0.0;
#pragma unroll 4
    for (int g = 0; g < NG; ++g) sum += acc[g * cap + s];
    size += fabs(sum);
    if (kAP) {
      f.apVal[c0 + s] = (T)sum;
      const int J = cols[s];
      double p = 0.0;
      for (int k = __ldg(&f.pOff[r]); k < __ldg(&f.pOff[r + 1]); ++k)
        if (__ldg(&f.pCol[k]) == J) p = ld(&f.pVal[k]);
      const T q = (T)(p - ld(&f.wdinv[r]) * sum);
      if (f.qSlice) f.qVal[__ldg(&f.qSlice[r >> 5]) + (s << 5) + (r & 31)] = q;
      else f.mVal[__ldg(&f.rowOff[r + 1]) + c0 + s] = q;  // behind the row's -w A
    } else if (s < nc) {
      c.val[c0 + s] = (T)sum;
    } else {
      c.diag[r] = (T)sum;
      diag = sum;
    }
  }
  if constexpr (!kAP) {
    if constexpr (TS > 32) {
      __shared__ double sm[TS / 32];
      size = warp_sum(size);
      if ((tt & 31) == 0) sm[tt >> 5] = size;
      __syncthreads();
      size = 0.0;
#pragma unroll
      for (int u = 0; u < TS / 32; ++u) size += sm[u];
    } else {
      size = __shfl_sync(0xffffffffu, warp_sum(size), 0);
    }
    if (tt == nc % TS) c.wdinv[r] = (T)fmin(omega / diag, kSaWeight / size);
  }
}

__global__ void __launch_bounds__(kBlock) k_sa_sell_cols(int n, const int* off, const int* col, const int* slice,
                                                         int* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int k0 = off[i], k1 = off[i + 1], b = slice[i >> 5] + (i & 31);
    for (int k = k0; k < k1; ++k) out[b + ((k - k0) << 5)] = col[k];
  }
}

// The -w A part of the merged rows of a coarse level, G lanes a row.
template <int G, class T>
__global__ void __launch_bounds__(kBlock) k_sa_scale(AmgLevelDevT<T> f) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = t / G, sub = t % G;
  if (i >= f.n) return;
  const double w = ld(&f.wdinv[i]);
  const int k0 = __ldg(&f.rowOff[i]), k1 = __ldg(&f.rowOff[i + 1]), m0 = __ldg(&f.mOff[i]);
  for (int k = k0 + sub; k < k1; k += G) f.mVal[m0 + k - k0] = (T)(-w * ld(&f.val[k]));
}

template <class T>
__global__ void __launch_bounds__(kBlock) k_sa_gather(int n, const int* src, const T* v, T* out) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) out[e] = v[src[e]];
}

// A P and Q of the finest level: a thread a row, its row of A P in a column of shared memory (25
// products and 9 positions a row on hexes: too little for a warp; 500 us at 970k cells with a warp a
// row).  The matrix and the columns of Q are SELL-32, so a warp reads them coalesced.
constexpr int kApThreads = 128;
template <class T>
__global__ void __launch_bounds__(kApThreads) k_sa_ap0(AmgLevelDevT<T> f, int cap) {
  extern __shared__ double sh[];
  double* acc = sh + threadIdx.x;
  int* cols = reinterpret_cast<int*>(sh + (size_t)cap * kApThreads) + threadIdx.x;
  const int i = blockIdx.x * kApThreads + threadIdx.x;
  if (i >= f.n) return;
  const int q0 = __ldg(&f.qOff[i]), nq = __ldg(&f.qOff[i + 1]) - q0;
  const int qb = __ldg(&f.qSlice[i >> 5]) + (i & 31);
  for (int s = 0; s < nq; ++s) {
    cols[s * kApThreads] = __ldg(&f.qColS[qb + (s << 5)]);
    acc[s * kApThreads] = 0.0;
  }
  int b, cnt, st;
  row_entries(f, i, b, cnt, st);
  auto add = [&](int j, double a) {
    const int k1 = __ldg(&f.pOff[j + 1]);
    for (int k = __ldg(&f.pOff[j]); k < k1; ++k) {
      const int J = __ldg(&f.pCol[k]);
      int lo = 0, hi = nq;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cols[mid * kApThreads] < J) lo = mid + 1;
        else hi = mid;
      }
      acc[lo * kApThreads] += a * ld(&f.pVal[k]);
    }
  };
  add(i, ld(&f.diag[i]));
  for (int e = 0; e < cnt; ++e) {
    const int j = __ldg(&f.col[b + e * st]);
    if (j != i) add(j, ld(&f.val[b + e * st]));  // padding slots name the row itself
  }
  const double w = ld(&f.wdinv[i]);
  for (int s = 0; s < nq; ++s) {
    const double v = acc[s * kApThreads];
    f.apVal[q0 + s] = (T)v;
    acc[s * kApThreads] = -w * v;
  }
  add(i, 1.0);  // + P
  for (int s = 0; s < nq; ++s) f.qVal[qb + (s << 5)] = (T)acc[s * kApThreads];
}

int grid_for(long long threads, int cap) {
  return (int)std::max<long long>(1, std::min<long long>(cap, (threads + kBlock - 1) / kBlock));
}

template <class F>
void with_lanes(int g, F&& fn) {
  switch (g) {
    case 4: fn(std::integral_constant<int, 4>{}); break;
    case 8: fn(std::integral_constant<int, 8>{}); break;
    case 16: fn(std::integral_constant<int, 16>{}); break;
    default: fn(std::integral_constant<int, 32>{}); break;
  }
}

}  // namespace

void launch_sa_sell_cols(const LaunchCfg& lc, int n, const int* off, const int* col, const int* slice, int* out) {
  g_launches += 1;
  k_sa_sell_cols<<<grid_for(n, 1 << 30), kBlock, 0, lc.stream>>>(n, off, col, slice, out);
}

template <int G, int TS, bool kAP, class T>
static void launch_product(const LaunchCfg& lc, const AmgLevelDevT<T>& f, const AmgLevelDevT<T>& c, double omega,
                           int cap) {
  const size_t smem = sa_product_smem(G, TS, cap);
  auto kern = k_sa_product<G, TS, kAP, T>;
  if (smem > 48 * 1024 && allow_smem<kSaSmemMax>(kern) != cudaSuccess) return;  // cudaGetLastError reports it
  constexpr int kTeams = kBlock / TS;
  const int rows = kAP ? f.n : c.n;
  kern<<<(rows + kTeams - 1) / kTeams, kBlock, smem, lc.stream>>>(f, c, omega, cap);
}

// A P and Q of level l from the stored P
template <class T>
static void refresh_q(const LaunchCfg& lc, AmgDevT<T>& amg, int l) {
  AmgLevelDevT<T>& f = amg.lv[l];
  AmgLevelDevT<T>& c = amg.lv[l + 1];
  // a warp a row while there are rows enough to fill the GPU with warps, else a block a row
  const size_t smem0 = (size_t)f.capQ * kApThreads * (sizeof(double) + sizeof(int));
  constexpr size_t kAp0Smem = 96 * 1024;
  if (l == 0 && smem0 <= kAp0Smem) {
    if (smem0 > 48 * 1024 && allow_smem<kAp0Smem>(k_sa_ap0<T>) != cudaSuccess) return;
    k_sa_ap0<T><<<(f.n + kApThreads - 1) / kApThreads, kApThreads, smem0, lc.stream>>>(f, f.capQ);
  } else if (sa_small_team(f.n, f.capQ)) {
    launch_product<8, 32, true>(lc, f, c, amg.omega, f.capQ);
  } else {
    launch_product<8, 256, true>(lc, f, c, amg.omega, f.capQ);
  }
}

template <class T>
void sa_refresh_level(const LaunchCfg& lc, AmgDevT<T>& amg, int l) {
  AmgLevelDevT<T>& f = amg.lv[l];
  AmgLevelDevT<T>& c = amg.lv[l + 1];
  g_launches += 4;
  if (l == 0) k_sa_p<1, T><<<(f.n + kBlock - 1) / kBlock, kBlock, 0, lc.stream>>>(f);
  else with_lanes(f.lanesUp, [&](auto G) {
    k_sa_p<G.value, T><<<grid_for((long long)G.value * f.n, 1 << 30), kBlock, 0, lc.stream>>>(f);
  });
  refresh_q(lc, amg, l);
  k_sa_gather<T><<<grid_for(f.nT, 1 << 30), kBlock, 0, lc.stream>>>(f.nT, f.tSrc, l == 0 ? f.pVal : f.mVal, f.tVal);
  if (l > 0) {
    g_launches += 1;
    k_sa_scale<8, T><<<grid_for(8LL * f.n, 1 << 30), kBlock, 0, lc.stream>>>(f);
  }
  if (sa_small_team(c.n, f.capC)) launch_product<8, 32, false>(lc, f, c, amg.omega, f.capC);
  else launch_product<16, 256, false>(lc, f, c, amg.omega, f.capC);
}

// With a stale hierarchy (p_amg_rebuild_every > 1) the finest Q still has to belong to the current matrix:
// the restriction goes through the current residual, and with an older Q the preconditioner would lose its
// symmetry.  P and the coarse levels stay as they are.
template <class T>
void sa_refresh_fine(const LaunchCfg& lc, AmgDevT<T>& amg) {
  g_launches += 1;
  refresh_q(lc, amg, 0);
}

template <class T>
void sa_refresh(const LaunchCfg& lc, AmgDevT<T>& amg) {
  for (int l = 0; l + 1 < amg.nLevels; ++l) sa_refresh_level(lc, amg, l);
  amg_dense_factor(lc, amg.lv[amg.nLevels - 1], amg.dense);
}

template <class T>
void sa_vcycle(const LaunchCfg& lc, const PcgArgsT<T>& a, const AmgDevT<T>* amg, int v) {
  const int L = amg->nLevels;
  const T* rIn = v ? a.r2 : a.r;
  T* rOut = v ? a.r : a.r2;
  const T* p = v ? a.p1 : a.p0;
  AmgLevelDevT<T> f0 = amg->lv[0];
  f0.b = rOut;
  const int cap = 1 << 20;
  auto restrict_to = [&](const AmgLevelDevT<T>& f, const T* x, int l) {
    const AmgLevelDevT<T>& c = amg->lv[l];
    const bool last = l == L - 1;
    if (f.lanesDown > 32) {
      k_sa_restrict_block<T><<<c.n, kBlock, 0, lc.stream>>>(a.fl, f.tOff, f.tCol, f.tVal, x, c.b,
                                                            last ? nullptr : c.wdinv, c.x);
      return;
    }
    with_lanes(f.lanesDown, [&](auto G) {
      k_sa_restrict<G.value, T><<<grid_for((long long)G.value * c.n, cap), kBlock, 0, lc.stream>>>(
          a.fl, c.n, f.tOff, f.tCol, f.tVal, x, c.b, last ? nullptr : c.wdinv, c.x);
    });
  };
  {
    ProfScope ps(lc, kKfAmgResid0, 0.0, 2);
    with_width(f0.maxW, [&](auto W) { launch_rows(lc, lc.rowBlocks, k_sa_resid0<T, W.value>, a, f0, rIn, rOut, p); });
    restrict_to(f0, f0.x2, 1);
  }
  {
    // first level of the cluster tail (L - 1: the dense level on its own)
    int t0 = L - 1;
    while (amg->tailCluster > 0 && t0 > 1 && amg->lv[t0 - 1].n <= amg->tailRows && L - (t0 - 1) <= kTailMaxLevels) --t0;
    ProfScope ps(lc, kKfAmgCoarse, 0.0, 2 * (t0 - 1) + 1);
    for (int l = 1; l < t0; ++l) restrict_to(amg->lv[l], amg->lv[l].b, l + 1);
    if (t0 < L - 1) {
      SaTailArgs<T> ta{};
      ta.nLev = L - t0;
      for (int l = 0; l < ta.nLev; ++l) ta.lv[l] = amg->lv[t0 + l];
      ta.dense = amg->dense;
      cudaLaunchAttribute at[1];
      const cudaLaunchConfig_t cfg = tail_config(lc.stream, amg->tailCluster, at);
      cudaLaunchKernelEx(&cfg, k_sa_tail<T>, (const int*)a.fl, ta);
    } else {
      const AmgLevelDevT<T>& c = amg->lv[L - 1];
      k_sa_dense<T><<<grid_for(32LL * c.n, cap), kBlock, 0, lc.stream>>>(a.fl, c.n, amg->dense, c.b, c.x2);
    }
    for (int l = t0 - 1; l >= 1; --l) {
      const AmgLevelDevT<T>& f = amg->lv[l];
      with_lanes(f.lanesUp, [&](auto G) {
        k_sa_up<G.value, T><<<grid_for((long long)G.value * f.n, cap), kBlock, 0, lc.stream>>>(a.fl, f, f.x2);
      });
    }
  }
  {
    ProfScope ps(lc, kKfAmgUp0, 0.0);
    launch_rows(lc, lc.rowBlocks, k_sa_up0<T>, f0, (const T*)amg->lv[1].x2, a);
  }
}

// Cluster size of the tail: 16 CTAs (a non-portable size) when the device can co-schedule them,
// else 8, else none.
template <class T>
void sa_configure_tail(AmgDevT<T>& amg, int tailRows, cudaStream_t s) {
  amg.tailRows = tailRows;
  amg.tailCluster = 0;
  if (tailRows <= 0) return;
  cudaFuncSetAttribute(k_sa_tail<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  for (int cs : {16, 8}) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = tail_config(s, cs, at);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_sa_tail<T>, &cfg) == cudaSuccess && n > 0) {
      amg.tailCluster = cs;
      return;
    }
    cudaGetLastError();
  }
}

#define ANB_INSTANTIATE(T)                                                          \
  template void sa_refresh_level<T>(const LaunchCfg&, AmgDevT<T>&, int);            \
  template void sa_refresh<T>(const LaunchCfg&, AmgDevT<T>&);                       \
  template void sa_refresh_fine<T>(const LaunchCfg&, AmgDevT<T>&);                  \
  template void sa_configure_tail<T>(AmgDevT<T>&, int, cudaStream_t);               \
  template void sa_vcycle<T>(const LaunchCfg&, const PcgArgsT<T>&, const AmgDevT<T>*, int);
ANB_INSTANTIATE(double)
ANB_INSTANTIATE(float)
#undef ANB_INSTANTIATE

}  // namespace anb
