// The whole Jacobi-BiCGSTAB solve of a small system as one cooperative kernel (sm_100a), standing in
// for the reference's BiCGSTAB + DiagScale (main.cu:2553-2576) as kernels_krylov.cu does.
//
// Up to a few hundred thousand unknowns the five kernels of an iteration move data that stays in L2
// and cost their launches and the fence-ticket-read chains of their reductions: 27 us an iteration
// for 3 x 16k unknowns.  Here every thread keeps its rows' vectors in registers and its rows of the
// matrix in registers or shared memory for the whole solve; only D^-1 p and D^-1 s go through memory,
// because the products gather them, and an iteration is four grid barriers (about 10 us in all), each of
// which carries the block partials of the sums due there.  All blocks add the partials in the same order,
// so they take the same branches and the result does not depend on timing.  The grid is one block per SM
// (cooperative launch); a barrier that is not reached within kSpinLimit polls sets the fail flag and every
// block returns.
//
// rho of the next step is rh.s - omega rh.t, whose sums are due with those of t, where the five kernels sum rh.r
// of the new residual at a barrier of its own: a rounding of eps |rh| |s| in place of eps |rh| |r|, with |s| / |r|
// one half step's reduction.  It enters beta alone, so the search directions and never the recurrences of x and r;
// the iterations are the five kernels' to a few per cent.
//
// Measured (ms per pass, five kernels -> one): SIMPLE steps on 16k hexes 21.4 -> 15.5, 36k with all
// correctors 22.9 -> 18.0, scalar transport on 262k cells 44 -> 24, force gradient at 36k 88 -> 70; with
// the matrix of four rows a thread in shared memory instead of L2, and no fences beyond the release and
// acquire of the barriers, transport 14.0 -> 10.8.  The line is drawn at four rows a thread (303k
// unknowns), the last size measured faster (3 x 91k 4.6 -> 4.2 ms a step); beyond it the vectors outgrow
// the registers.
#include <algorithm>

#include "krylov_dev.cuh"

namespace anb {
namespace {

constexpr int kCoopThreads = 512;
constexpr int kCoopWarps = kCoopThreads / 32;
constexpr int kMaxQ = 4;                       // sums per component at one barrier
constexpr unsigned kSpinLimit = 4000000;       // polls of about half a microsecond

struct CoopBar {
  unsigned* count;   // arrivals, 0 at launch
  int* fail;
  double* part;      // 2 buffers x (3 kMaxQ) sums x gridDim.x blocks
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(unsigned* p) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// Recurrence scalars and flags of a component, kept by every block (one thread updates them).
struct CoopState {
  double eps, rn, bn, rhoN, rho, al, om;
  int done, half, its, conv;
};

struct CoopShared {
  double warp[kCoopWarps][kMaxQ];
  double sum[3 * kMaxQ];
  CoopState st[3];
  int bad;
};

// Grid barrier that also sums Q values per component over the grid (warp w works for component
// (first warp of the block + w) % nc) and then lets one thread per component run update(c, sums).
// Everything the block wrote before is visible to every block after it.  False: timed out.
template <int Q, class F>
__device__ __forceinline__ bool grid_sum(const CoopBar& bar, CoopShared& sh, unsigned& epoch, int nc, double (&v)[Q],
                                         F&& update) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nb = gridDim.x;
#pragma unroll
  for (int q = 0; q < Q; ++q) v[q] = warp_sum(v[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < Q; ++q) sh.warp[w][q] = v[q];
  __syncthreads();
  double* part = bar.part + (size_t)(epoch & 1u) * 3 * kMaxQ * nb;
  if ((int)threadIdx.x < nc * Q) {
    const int c = threadIdx.x / Q, q = threadIdx.x % Q;
    double s = 0.0;
    for (int u = 0; u < kCoopWarps; ++u)
      if (((int)blockIdx.x * kCoopWarps + u) % nc == c) s += sh.warp[u][q];
    __stcg(&part[(size_t)threadIdx.x * nb + blockIdx.x], s);
  }
  ++epoch;
  __syncthreads();
  if (threadIdx.x == 0) {
    // release and acquire order the whole block's accesses: the block barriers around them are cumulative
    add_release(bar.count);
    const unsigned want = epoch * (unsigned)nb;
    unsigned n = 0;
    while (ld_acquire(bar.count) < want && n < kSpinLimit) ++n;
    sh.bad = n >= kSpinLimit;
  }
  __syncthreads();
  if (sh.bad) {
    if (threadIdx.x == 0) *bar.fail = 1;
    return false;
  }
  if (w < nc * Q) {
    double s = 0.0;
    for (int b = lane; b < nb; b += 32) s += __ldcg(&part[(size_t)w * nb + b]);
    s = warp_sum(s);
    if (lane == 0) sh.sum[w] = s;
  }
  __syncthreads();
  if ((int)threadIdx.x < nc) update(sh.st[threadIdx.x], &sh.sum[threadIdx.x * Q]);
  __syncthreads();
  return true;
}

// Where a thread keeps its rows of the matrix for the whole solve: one row of registers, shared memory
// for two and four (12 bytes a slot: at most 196 KB for four rows of eight), memory for wider rows.
enum class Keep { kRegisters, kShared, kMemory };
constexpr size_t coop_smem(Keep keep, int R, int WM) {
  return keep == Keep::kShared ? (size_t)R * WM * kCoopThreads * (sizeof(double) + sizeof(int)) : 0;
}

// R rows a thread; WM: bound on the row width (0: any).
template <int R, int WM, Keep kKeep>
__global__ void __launch_bounds__(kCoopThreads, 1) k_bicg_coop(BicgArgs a, int mask, CoopBar bar) {
  constexpr bool kReg = kKeep == Keep::kRegisters;
  __shared__ CoopShared sh;
  extern __shared__ double keep[];  // values [slot][thread], then columns
  double* sVal = keep + threadIdx.x;
  int* sCol = reinterpret_cast<int*>(keep + (size_t)R * WM * kCoopThreads) + threadIdx.x;
  const int n = a.A.n, nc = a.nc, lane = threadIdx.x & 31;
  // warps take the components in turn, so that the warps of a block read the same matrix rows
  const int gw = blockIdx.x * kCoopWarps + (threadIdx.x >> 5);
  const int groups = (int)gridDim.x * kCoopWarps / nc;
  const int comp = gw % nc, group = gw / nc;
  const bool worker = group < groups;
  unsigned epoch = 0;
  int row[R] = {};
  double x[R], r[R], rh[R], p[R], v[R], s[R], dinv[R], dg[R] = {};
  int col[kReg ? R : 1][kReg ? WM : 1];
  double val[kReg ? R : 1][kReg ? WM : 1];
  const size_t o = (size_t)comp * n;

  // y = (A z)_row of item k, z through L2 (other blocks write it between the barriers)
  auto product = [&](int k, const double* z, double own) {
    double y = dg[k] * own;
    if constexpr (kReg) {
      double g[WM];
#pragma unroll
      for (int e = 0; e < WM; ++e) g[e] = __ldcg(&z[col[k][e]]);
#pragma unroll
      for (int e = 0; e < WM; ++e) y += val[k][e] * g[e];
    } else if constexpr (kKeep == Keep::kShared) {
      double g[WM];
#pragma unroll
      for (int e = 0; e < WM; ++e) g[e] = __ldcg(&z[sCol[(k * WM + e) * kCoopThreads]]);
#pragma unroll
      for (int e = 0; e < WM; ++e) y += sVal[(k * WM + e) * kCoopThreads] * g[e];
    } else {
      const int b = __ldg(&a.A.sliceOff[row[k] >> 5]) + (row[k] & 31);
      const int W = (__ldg(&a.A.sliceOff[(row[k] >> 5) + 1]) - __ldg(&a.A.sliceOff[row[k] >> 5])) >> 5;
#pragma unroll 4
      for (int e = 0; e < W; ++e)
        y += ld(&a.A.val[b + (e << 5)]) * __ldcg(&z[__ldg(&a.A.col[b + (e << 5)])]);
    }
    return y;
  };

  double q2[2] = {0.0, 0.0};
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const int i = (group + k * groups) * 32 + lane;
    row[k] = worker && i < n ? i : -1;
    x[k] = r[k] = rh[k] = p[k] = v[k] = s[k] = dinv[k] = dg[k] = 0.0;
    if constexpr (kReg) {
#pragma unroll
      for (int e = 0; e < WM; ++e) {
        col[k][e] = 0;
        val[k][e] = 0.0;
      }
    }
    if (row[k] < 0) continue;
    if constexpr (kReg) sell_regs<WM>(a.A.sliceOff, a.A.col, a.A.val, i, col[k], val[k]);
    if constexpr (kKeep == Keep::kShared) {
      int c[WM];
      double m[WM];
      sell_regs<WM>(a.A.sliceOff, a.A.col, a.A.val, i, c, m);
#pragma unroll
      for (int e = 0; e < WM; ++e) {
        sCol[(k * WM + e) * kCoopThreads] = c[e];
        sVal[(k * WM + e) * kCoopThreads] = m[e];
      }
    }
    dg[k] = ld(&a.A.diag[i]);
    dinv[k] = 1.0 / dg[k];
    x[k] = a.x[o + i];
    const double b = ld(&a.b[o + i]);
    r[k] = rh[k] = b - product(k, a.x + o, x[k]);
    q2[0] += r[k] * r[k];
    q2[1] += b * b;
  }
  if (!grid_sum<2>(bar, sh, epoch, nc, q2, [&](CoopState& c, const double* sum) {
        c.bn = sqrt(sum[1]);
        c.eps = fmax(a.atol, a.rtol * c.bn);
        c.rn = sqrt(sum[0]);
        c.rhoN = sum[0];
        c.rho = c.al = c.om = 1.0;
        c.half = c.its = 0;
        c.done = !((mask >> threadIdx.x) & 1) || c.rn <= c.eps;
        c.conv = c.done;
      }))
    return;
  auto all_finished = [&] {
    bool f = true;
    for (int c = 0; c < nc; ++c) f = f && sh.st[c].done;
    return f;
  };
  const CoopState& me = sh.st[comp];
  double* ph = a.ph + o;
  double* shv = a.sh + o;
  bool first = true;
  while (!all_finished()) {
    // p = r + beta (p - omega v), with |r|^2 of the iteration before
    double q1[1] = {0.0};
    if (!me.done) {
      const double beta = (me.rhoN / me.rho) * (me.al / me.om), w = me.om;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (row[k] < 0) continue;
        q1[0] += r[k] * r[k];
        p[k] = r[k] + beta * (p[k] - w * v[k]);
        __stcg(&ph[row[k]], dinv[k] * p[k]);
      }
    }
    if (!grid_sum<1>(bar, sh, epoch, nc, q1, [&](CoopState& c, const double* sum) {
          if (first || c.done) return;
          c.rn = sqrt(sum[0]);
          if (c.rn <= c.eps) c.done = c.conv = 1;
          else if (c.its >= a.maxit || c.om == 0.0) c.done = 1;
        }))
      return;
    if (all_finished()) break;
    first = false;
    // v = A D^-1 p, alpha = rho / (rh . v)
    q1[0] = 0.0;
    if (!me.done) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (row[k] < 0) continue;
        v[k] = product(k, ph, dinv[k] * p[k]);
        q1[0] += rh[k] * v[k];
      }
    }
    if (!grid_sum<1>(bar, sh, epoch, nc, q1, [&](CoopState& c, const double* sum) {
          if (c.done) return;
          c.al = sum[0] != 0.0 ? c.rhoN / sum[0] : 0.0;
          c.rho = c.rhoN;
          if (sum[0] == 0.0) c.done = 1;  // breakdown: stop this component
        }))
      return;
    // s = r - alpha v, half step when |s| is small enough
    q1[0] = 0.0;
    if (!me.done) {
      const double al = me.al;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (row[k] < 0) continue;
        s[k] = r[k] - al * v[k];
        __stcg(&shv[row[k]], dinv[k] * s[k]);
        q1[0] += s[k] * s[k];
      }
    }
    if (!grid_sum<1>(bar, sh, epoch, nc, q1, [&](CoopState& c, const double* sum) {
          if (!c.done) c.half = sqrt(sum[0]) <= c.eps;
        }))
      return;
    // t = A D^-1 s, omega = (t.s)/(t.t); rh.r of the new residual from rh.s and rh.t
    double q4[4] = {0.0, 0.0, 0.0, 0.0}, t[R];
    const bool act = !me.done, hf = me.half;
#pragma unroll
    for (int k = 0; k < R; ++k) {
      t[k] = 0.0;
      if (row[k] < 0 || !act || hf) continue;
      t[k] = product(k, shv, dinv[k] * s[k]);
      q4[0] += t[k] * s[k];
      q4[1] += t[k] * t[k];
      q4[2] += rh[k] * s[k];
      q4[3] += rh[k] * t[k];
    }
    if (!grid_sum<4>(bar, sh, epoch, nc, q4, [&](CoopState& c, const double* sum) {
          if (c.done) return;
          c.its += 1;
          if (c.half) {
            c.done = c.conv = 1;
            return;
          }
          c.om = sum[1] > 0.0 ? sum[0] / sum[1] : 0.0;
          c.rhoN = sum[2] - c.om * sum[3];
        }))
      return;
    if (act) {
      const double al = me.al, om = me.om;
#pragma unroll
      for (int k = 0; k < R; ++k) {
        if (row[k] < 0) continue;
        x[k] += al * (dinv[k] * p[k]);
        if (hf) continue;
        x[k] += om * (dinv[k] * s[k]);
        r[k] = s[k] - om * t[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < R; ++k)
    if (row[k] >= 0) a.x[o + row[k]] = x[k];
  if (blockIdx.x == 0 && (int)threadIdx.x < nc) {
    const CoopState& c = sh.st[threadIdx.x];
    a.sc[8 * threadIdx.x + 4] = c.eps;
    a.sc[8 * threadIdx.x + 5] = c.rn;
    a.sc[8 * threadIdx.x + 6] = c.bn;
    int* f = a.fl + 4 * threadIdx.x;
    f[0] = 1;
    f[1] = c.half;
    f[2] = c.its;
    f[3] = c.conv;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) a.fl[12] = 0;
}

template <int R, int WM, Keep kKeep>
bool launch_one(cudaStream_t s, int blocks, const BicgArgs& a, int mask, const CoopBar& bar) {
  auto kern = k_bicg_coop<R, WM, kKeep>;
  constexpr size_t smem = coop_smem(kKeep, R, WM);
  BicgArgs aa = a;
  int m = mask;
  CoopBar b = bar;
  void* args[] = {&aa, &m, &b};
  if ((smem == 0 || allow_smem<smem>(kern) == cudaSuccess) &&
      cudaLaunchCooperativeKernel((const void*)kern, dim3(blocks), dim3(kCoopThreads), args, smem, s) == cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}

template <int WM>
bool launch_width(cudaStream_t s, int blocks, int rows, const BicgArgs& a, int mask, const CoopBar& bar) {
  if constexpr (WM == 0) {
    if (rows <= 1) return launch_one<1, 0, Keep::kMemory>(s, blocks, a, mask, bar);
    if (rows <= 2) return launch_one<2, 0, Keep::kMemory>(s, blocks, a, mask, bar);
    return launch_one<4, 0, Keep::kMemory>(s, blocks, a, mask, bar);
  } else {
    if (rows <= 1) return launch_one<1, WM, Keep::kRegisters>(s, blocks, a, mask, bar);
    if (rows <= 2) return launch_one<2, WM, Keep::kShared>(s, blocks, a, mask, bar);
    return launch_one<4, WM, Keep::kShared>(s, blocks, a, mask, bar);
  }
}

}  // namespace

int bicg_coop_partials(int nSM) { return 2 * 3 * kMaxQ * nSM; }

bool bicg_coop_fits(int n, int nc, int nSM) {
  if (nSM <= 0 || nc < 1 || nc > 3) return false;
  const long long perPass = (long long)nSM * kCoopWarps / nc * 32;
  return n <= kCoopRows * perPass;
}

bool bicg_coop_solve(const LaunchCfg& lc, const BicgArgs& a, int mask, int nSM, double* partials) {
  if (a.precond || !bicg_coop_fits(a.A.n, a.nc, nSM)) return false;
  const long long perPass = (long long)nSM * kCoopWarps / a.nc * 32;
  const int rows = (int)((a.A.n + perPass - 1) / perPass);
  CoopBar bar{reinterpret_cast<unsigned*>(a.fl + 14), a.fl + 13, partials};
  if (cudaMemsetAsync(a.fl + 13, 0, 2 * sizeof(int), lc.stream) != cudaSuccess) return false;
  bool ok = false;
  with_width(a.A.maxW, [&](auto W) { ok = launch_width<W.value>(lc.stream, nSM, rows, a, mask, bar); });
  if (ok) g_launches += 1;
  return ok;
}

}  // namespace anb
