// Patterns of a smoothed-aggregation level step on the device (sm_100a): P, A P, their transposes and
// P^T A P from the matrix pattern and the aggregates (sa_setup.hpp states the rules; the host form there
// gives the same patterns and serves the rows that do not fit a table here).
//
// A row's columns are collected in a hash table in shared memory, one team (a warp or a block) a row,
// one thread a term; a first pass counts them, a scan makes the offsets, and a second pass collects them
// again and writes them in ascending order (each entry's place is the number of smaller ones).  The
// results do not depend on the order of insertion.  A Poisson solve on 110k cells builds its hierarchy
// anew; the patterns took 18 of its 34 ms on 16 host threads with their transfers.
#include <algorithm>

#include "kernels.cuh"

namespace anb {
namespace {

struct PatTerm {  // rows of the product and their terms
  int rows;
  const int *sliceOff, *rowOff, *col;  // matrix pattern (SELL-32 or CSR): modes 0, 1
  const int* agg;
  int smooth;                          // mode 0: with the neighbours
  const int *bOff, *bCol;              // rows of B: P (mode 1), A P (mode 2)
  const int *tOff, *tCol;              // P^T: mode 2
};

// Mode 0: P, the aggregates of a row and its neighbours; 1: A P, the rows of P of the same; 2: off-diagonals
// of P^T A P, the rows of A P of the rows of an aggregate's P^T.  FILL: write the sorted columns at off[row],
// else their number to cnt[row].  H (a power of two): table size; a row that overflows it sets *flag.
template <int TS, int MODE, bool FILL>
__global__ void __launch_bounds__(kBlock) k_pattern(PatTerm a, int H, int* cnt, const int* off, int* out, int* flag) {
  extern __shared__ int smi[];
  __shared__ int count[kBlock / TS], cursor[kBlock / TS];
  constexpr int kTeams = kBlock / TS;
  const int team = threadIdx.x / TS, tt = threadIdx.x % TS;
  int* table = smi + (size_t)team * 2 * H;
  int* list = table + H;
  const int row = blockIdx.x * kTeams + team;
  const bool live = row < a.rows;
  auto sync = [] {
    if constexpr (TS > 32) __syncthreads();
    else __syncwarp();
  };
  for (int s = tt; s < H; s += TS) table[s] = -1;
  if (tt == 0) count[team] = cursor[team] = 0;
  sync();
  if (live) {
    auto insert = [&](int J) {
      unsigned h = ((unsigned)J * 2654435761u) >> 12;
      for (int t = 0; t < H; ++t, ++h) {
        const int old = atomicCAS(&table[h & (H - 1)], -1, J);
        if (old == -1) atomicAdd(&count[team], 1);
        if (old == -1 || old == J) return;
      }
      *flag = 1;
    };
    if constexpr (MODE == 2) {
      const int e1 = a.tOff[row + 1];
      for (int e = a.tOff[row] + tt; e < e1; e += TS) {
        const int i = a.tCol[e], k1 = a.bOff[i + 1];
        for (int k = a.bOff[i]; k < k1; ++k)
          if (a.bCol[k] != row) insert(a.bCol[k]);
      }
    } else {
      int b, n, st;
      if (a.sliceOff) {
        b = a.sliceOff[row >> 5] + (row & 31);
        n = (a.sliceOff[(row >> 5) + 1] - a.sliceOff[row >> 5]) >> 5;
        st = 32;
      } else {
        b = a.rowOff[row];
        n = a.rowOff[row + 1] - b;
        st = 1;
      }
      if (MODE == 0 && !a.smooth) n = 0;
      for (int e = tt - 1; e < n; e += TS) {  // term -1: the row itself
        const int j = e < 0 ? row : a.col[b + e * st];
        if constexpr (MODE == 0) {
          insert(a.agg[j]);
        } else {
          const int k1 = a.bOff[j + 1];
          for (int k = a.bOff[j]; k < k1; ++k) insert(a.bCol[k]);
        }
      }
    }
  }
  sync();
  if constexpr (!FILL) {
    if (live && tt == 0) cnt[row] = count[team];
  } else {
    for (int s = tt; s < H; s += TS)
      if (table[s] >= 0) list[atomicAdd(&cursor[team], 1)] = table[s];
    sync();
    if (!live) return;
    const int n = cursor[team], o = off[row];
    for (int s = tt; s < n; s += TS) {
      const int J = list[s];
      int rank = 0;
      for (int u = 0; u < n; ++u) rank += list[u] < J;
      out[o + rank] = J;
    }
  }
}

// off = exclusive scan of cnt (n entries, off[n] the total); info[0] = the total, info[1] = the largest.
// One block, contiguous pieces: set-up only, 0.2 ms for a million entries.
__global__ void __launch_bounds__(1024) k_scan(int n, const int* cnt, int* off, int* info) {
  __shared__ int part[1024], big[1024];
  const int t = threadIdx.x, per = (n + 1023) / 1024, lo = min(n, t * per), hi = min(n, lo + per);
  int s = 0, m = 0;
  for (int i = lo; i < hi; ++i) {
    s += cnt[i];
    m = max(m, cnt[i]);
  }
  part[t] = s;
  big[t] = m;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int p = t >= d ? part[t - d] : 0, b = t >= d ? big[t - d] : 0;
    __syncthreads();
    part[t] += p;
    big[t] = max(big[t], b);
    __syncthreads();
  }
  int o = t > 0 ? part[t - 1] : 0;
  for (int i = lo; i < hi; ++i) {
    off[i] = o;
    o += cnt[i];
  }
  if (t == 1023) {
    off[n] = part[t];
    info[0] = part[t];
    info[1] = big[t];
  }
}

__global__ void __launch_bounds__(kBlock) k_count_cols(int n, const int* col, int* cnt) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) atomicAdd(&cnt[col[e]], 1);
}

// Entries of the transpose in any order (cursor: a copy of its offsets), then each row sorted.
__global__ void __launch_bounds__(kBlock) k_transpose_fill(int n, const int* off, const int* col, int* cursor, int* tCol,
                                                           int* tSrc) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = off[i]; k < off[i + 1]; ++k) {
      const int s = atomicAdd(&cursor[col[k]], 1);
      tCol[s] = i;
      tSrc[s] = k;
    }
}
template <int TS>
__global__ void __launch_bounds__(kBlock) k_transpose_sort(int rows, int cap, const int* tOff, int* tCol, int* tSrc) {
  extern __shared__ int smi[];
  const int team = threadIdx.x / TS, tt = threadIdx.x % TS, row = blockIdx.x * (kBlock / TS) + team;
  int* src = smi + (size_t)team * 2 * cap;
  int* fine = src + cap;
  const int o = row < rows ? tOff[row] : 0, n = row < rows ? tOff[row + 1] - o : 0;
  for (int s = tt; s < n; s += TS) {
    src[s] = tSrc[o + s];
    fine[s] = tCol[o + s];
  }
  if constexpr (TS > 32) __syncthreads();
  else __syncwarp();
  for (int s = tt; s < n; s += TS) {
    const int k = src[s];
    int rank = 0;
    for (int u = 0; u < n; ++u) rank += src[u] < k;
    tSrc[o + rank] = k;
    tCol[o + rank] = fine[s];
  }
}

// Slots (times 32) of every SELL-32 slice of a CSR pattern.
__global__ void __launch_bounds__(kBlock) k_slice_width(int n, const int* off, int* cnt) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= (n + 31) / 32) return;
  int w = 0;
  for (int i = 32 * s; i < min(n, 32 * s + 32); ++i) w = max(w, off[i + 1] - off[i]);
  cnt[s] = 32 * w;
}

// Merged rows [A | Q] (columns n + J for Q) and the places of Q^T's entries in them.
__global__ void __launch_bounds__(kBlock) k_merge_cols(int n, const int* rowOff, const int* col, const int* qOff,
                                                       const int* qCol, int* mOff, int* mCol) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
    int o = rowOff[i] + qOff[i];
    mOff[i] = o;
    if (i == n) continue;
    for (int e = rowOff[i]; e < rowOff[i + 1]; ++e) mCol[o++] = col[e];
    for (int e = qOff[i]; e < qOff[i + 1]; ++e) mCol[o++] = n + qCol[e];
  }
}
__global__ void __launch_bounds__(kBlock) k_shift_src(int n, const int* rowOff, const int* tCol, int* tSrc) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    tSrc[e] += rowOff[tCol[e] + 1];
}

int grid_for(long long threads) { return (int)std::max<long long>(1, (threads + kBlock - 1) / kBlock); }

template <int TS, int MODE>
void launch_pattern(cudaStream_t s, const PatTerm& a, int H, int* cnt, const int* off, int* out, int* flag) {
  const size_t smem = (size_t)(kBlock / TS) * 2 * H * sizeof(int);  // at most 32 KB
  const int grid = (a.rows + kBlock / TS - 1) / (kBlock / TS);
  if (out) k_pattern<TS, MODE, true><<<grid, kBlock, smem, s>>>(a, H, cnt, off, out, flag);
  else k_pattern<TS, MODE, false><<<grid, kBlock, smem, s>>>(a, H, cnt, off, out, flag);
  g_launches += 1;
}

}  // namespace

void sa_pattern_rows(const LaunchCfg& lc, const SaDevPattern& p, int mode, bool fill, int* cnt, int* flag) {
  PatTerm a{};
  a.rows = mode == 2 ? p.nc : p.n;
  a.sliceOff = p.sliceOff;
  a.rowOff = p.rowOff;
  a.col = p.col;
  a.agg = p.agg;
  a.smooth = p.smooth;
  a.bOff = mode == 1 ? p.pOff : p.qOff;
  a.bCol = mode == 1 ? p.pCol : p.qCol;
  a.tOff = p.ptOff;
  a.tCol = p.ptCol;
  const bool fine = p.sliceOff != nullptr;  // the finest level's short rows
  if (mode == 0) launch_pattern<32, 0>(lc.stream, a, fine ? 64 : 256, cnt, p.pOff, fill ? p.pCol : nullptr, flag);
  else if (mode == 1) launch_pattern<32, 1>(lc.stream, a, fine ? 128 : 512, cnt, p.qOff, fill ? p.qCol : nullptr, flag);
  else if (fine) launch_pattern<32, 2>(lc.stream, a, 256, cnt, p.cOff, fill ? p.cCol : nullptr, flag);
  else launch_pattern<256, 2>(lc.stream, a, 2048, cnt, p.cOff, fill ? p.cCol : nullptr, flag);
}

void sa_scan(const LaunchCfg& lc, int n, const int* cnt, int* off, int* info) {
  g_launches += 1;
  k_scan<<<1, 1024, 0, lc.stream>>>(n, cnt, off, info);
}

void sa_count_cols(const LaunchCfg& lc, int entries, const int* col, int* cnt) {
  g_launches += 1;
  k_count_cols<<<grid_for(entries), kBlock, 0, lc.stream>>>(entries, col, cnt);
}

bool sa_transpose(const LaunchCfg& lc, int n, int nc, int longest, const int* off, const int* col, const int* tOff,
                  int* cursor, int* tCol, int* tSrc) {
  if (longest > 4096) return false;
  if (cudaMemcpyAsync(cursor, tOff, sizeof(int) * nc, cudaMemcpyDeviceToDevice, lc.stream) != cudaSuccess) return false;
  g_launches += 2;
  k_transpose_fill<<<grid_for(n), kBlock, 0, lc.stream>>>(n, off, col, cursor, tCol, tSrc);
  if (longest <= 512)
    k_transpose_sort<32><<<(nc + 7) / 8, kBlock, 8 * 2 * longest * sizeof(int), lc.stream>>>(nc, longest, tOff, tCol, tSrc);
  else
    k_transpose_sort<kBlock><<<nc, kBlock, 2 * longest * sizeof(int), lc.stream>>>(nc, longest, tOff, tCol, tSrc);
  return true;
}

void sa_slice_widths(const LaunchCfg& lc, int n, const int* off, int* cnt) {
  g_launches += 1;
  k_slice_width<<<grid_for((n + 31) / 32), kBlock, 0, lc.stream>>>(n, off, cnt);
}

void sa_merge(const LaunchCfg& lc, const SaDevPattern& p, int* mOff, int* mCol) {
  g_launches += 2;
  k_merge_cols<<<grid_for(p.n + 1), kBlock, 0, lc.stream>>>(p.n, p.rowOff, p.col, p.qOff, p.qCol, mOff, mCol);
  k_shift_src<<<grid_for(p.nQ), kBlock, 0, lc.stream>>>(p.nQ, p.rowOff, p.qtCol, p.qtSrc);
}

}  // namespace anb
