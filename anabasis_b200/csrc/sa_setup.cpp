// Smoothed-aggregation structure set-up (host).
#include "sa_setup.hpp"

#include <algorithm>
#include <cmath>
#include <utility>

#include <omp.h>

namespace anb {
namespace {

// CSR rows built in parallel: emit(i, out) appends row i's columns.  Threads take contiguous row
// ranges, so the result does not depend on their number.
template <class F>
void build_rows(int n, int marks, std::vector<int>& off, std::vector<int>& col, F&& emit) {
  off.assign((size_t)n + 1, 0);
  std::vector<std::vector<int>> part(omp_get_max_threads());
  std::vector<int> first(part.size() + 1, 0);
  int used = 1;
#pragma omp parallel
  {
    const int t = omp_get_thread_num(), T = omp_get_num_threads();
#pragma omp single
    used = T;
    const int lo = (int)((long long)n * t / T), hi = (int)((long long)n * (t + 1) / T);
    std::vector<int>& out = part[t];
    std::vector<int> mark(marks, -1);
    for (int i = lo; i < hi; ++i) {
      const size_t before = out.size();
      emit(i, out, mark);
      std::sort(out.begin() + before, out.end());
      off[i + 1] = (int)(out.size() - before);
    }
  }
  for (int i = 0; i < n; ++i) off[i + 1] += off[i];
  col.resize(off[n]);
#pragma omp parallel for schedule(static, 1)
  for (int t = 0; t < used; ++t) {
    const int lo = (int)((long long)n * t / used);
    std::copy(part[t].begin(), part[t].end(), col.begin() + off[lo]);
  }
}

// Rows of the transpose (nc rows), each in ascending order of the original row.  Threads count and
// then place contiguous row ranges, one after the other within every row of the transpose.
void transpose(int n, int nc, const std::vector<int>& off, const std::vector<int>& col, std::vector<int>& tOff,
               std::vector<int>& tCol, std::vector<int>& tSrc) {
  tOff.assign((size_t)nc + 1, 0);
  tCol.resize(col.size());
  tSrc.resize(col.size());
  const int most = std::max(1, std::min(omp_get_max_threads(), n / 4096));
  std::vector<std::vector<int>> cnt(most);
#pragma omp parallel num_threads(most)
  {
    const int t = omp_get_thread_num(), T = omp_get_num_threads();
    const int lo = (int)((long long)n * t / T), hi = (int)((long long)n * (t + 1) / T);
    std::vector<int>& c = cnt[t];
    c.assign(nc, 0);
    for (int k = off[lo]; k < off[hi]; ++k) c[col[k]]++;
#pragma omp barrier
#pragma omp for schedule(static)
    for (int I = 0; I < nc; ++I) {
      int s = 0;
      for (int u = 0; u < T; ++u) {
        const int here = cnt[u][I];
        cnt[u][I] = s;  // entries of the threads before
        s += here;
      }
      tOff[I + 1] = s;
    }
#pragma omp single
    for (int I = 0; I < nc; ++I) tOff[I + 1] += tOff[I];
    for (int i = lo; i < hi; ++i)
      for (int k = off[i]; k < off[i + 1]; ++k) {
        const int s = tOff[col[k]] + c[col[k]]++;
        tCol[s] = i;
        tSrc[s] = k;
      }
  }
}

// Aggregates numbered by their first row.
std::vector<int> renumber(std::vector<int> agg, int nc) {
  std::vector<int> ren(nc, -1);
  int next = 0;
  for (int& a : agg) {
    if (ren[a] < 0) ren[a] = next++;
    a = ren[a];
  }
  return agg;
}

}  // namespace

std::vector<int> sa_aggregate(const SaMatrix& A, double theta, int& nc) {
  const int n = A.n;
  const double t2 = theta * theta;
  auto strong = [&](int i, int k) {
    const double a = A.val[k];
    return a < 0.0 && a * a > t2 * A.diag[i] * A.diag[A.col[k]];
  };
  std::vector<int> agg(n, -1);
  nc = 0;
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    bool free = true;
    for (int k = A.off[i]; k < A.off[i + 1] && free; ++k) free = !strong(i, k) || agg[A.col[k]] < 0;
    if (!free) continue;
    agg[i] = nc;
    for (int k = A.off[i]; k < A.off[i + 1]; ++k)
      if (strong(i, k)) agg[A.col[k]] = nc;
    ++nc;
  }
  std::vector<int> join(agg);
#pragma omp parallel for schedule(static)
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    double best = 0.0;
    for (int k = A.off[i]; k < A.off[i + 1]; ++k) {
      const int j = A.col[k];
      if (agg[j] < 0 || !strong(i, k)) continue;
      const double s = A.val[k] * A.val[k] / (A.diag[i] * A.diag[j]);
      if (s > best) {
        best = s;
        join[i] = agg[j];
      }
    }
  }
  agg.swap(join);
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    agg[i] = nc;
    for (int k = A.off[i]; k < A.off[i + 1]; ++k)
      if (agg[A.col[k]] < 0 && strong(i, k)) agg[A.col[k]] = nc;
    ++nc;
  }
  return renumber(std::move(agg), nc);
}

double sa_next_entries(const SaMatrix& A, const std::vector<int>& agg, int nc) {
  const int n = A.n;
  constexpr int kStep = 16;
  std::vector<int> mOff((size_t)nc + 1, 0), mem(n);
  for (int i = 0; i < n; ++i) mOff[agg[i] + 1]++;
  for (int I = 0; I < nc; ++I) mOff[I + 1] += mOff[I];
  {
    std::vector<int> fill(mOff.begin(), mOff.end() - 1);
    for (int i = 0; i < n; ++i) mem[fill[agg[i]]++] = i;
  }
  // row I of P^T A P reaches the aggregates of every row within three steps of I's rows
  long long sum = 0;
  const int rows = (nc + kStep - 1) / kStep;
#pragma omp parallel reduction(+ : sum)
  {
    std::vector<char> seen(n, 0);
    std::vector<int> met(nc, -1), q;
#pragma omp for schedule(static)
    for (int u = 0; u < rows; ++u) {
      const int I = u * kStep;
      q.assign(mem.begin() + mOff[I], mem.begin() + mOff[I + 1]);
      for (int i : q) seen[i] = 1;
      size_t from = 0;
      for (int d = 0; d < 3; ++d) {
        const size_t to = q.size();
        for (; from < to; ++from)
          for (int k = A.off[q[from]]; k < A.off[q[from] + 1]; ++k)
            if (!seen[A.col[k]]) {
              seen[A.col[k]] = 1;
              q.push_back(A.col[k]);
            }
      }
      for (int i : q) {
        seen[i] = 0;
        if (met[agg[i]] != I) {
          met[agg[i]] = I;
          ++sum;
        }
      }
      --sum;  // the diagonal
    }
  }
  return (double)sum / rows * nc;
}

std::vector<int> sa_groups(const SaMatrix& A, int size, int& nc) {
  const int n = A.n;
  // strength |a_ij| / sqrt(a_ii a_jj), squared and without the row's own factor
  auto strength = [&](int k) { return A.val[k] < 0.0 ? A.val[k] * A.val[k] / A.diag[A.col[k]] : 0.0; };
  std::vector<int> agg(n, -1);
  std::vector<std::pair<double, int>> near;
  nc = 0;
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    near.clear();
    for (int k = A.off[i]; k < A.off[i + 1]; ++k)
      if (agg[A.col[k]] < 0 && strength(k) > 0.0) near.push_back({strength(k), A.col[k]});
    if (near.empty()) continue;
    const size_t m = std::min(near.size(), (size_t)size - 1);
    std::partial_sort(near.begin(), near.begin() + m, near.end(), [](const auto& x, const auto& y) {
      return x.first != y.first ? x.first > y.first : x.second < y.second;
    });
    agg[i] = nc;
    for (size_t q = 0; q < m; ++q) agg[near[q].second] = nc;
    ++nc;
  }
  std::vector<int> join(agg);
  for (int i = 0; i < n; ++i) {
    if (agg[i] >= 0) continue;
    double best = 0.0;
    for (int k = A.off[i]; k < A.off[i + 1]; ++k)
      if (agg[A.col[k]] >= 0 && strength(k) > best) {
        best = strength(k);
        join[i] = agg[A.col[k]];
      }
    if (join[i] < 0) join[i] = nc++;
  }
  return renumber(std::move(join), nc);
}

bool sa_coarsen(const SaMatrix& A, int level, int maxRowLen, bool groups, SaStep& step) {
  step = SaStep{};
  if (!groups) {
    const double most = 1.25 * (double)A.col.size();
    double theta = sa_theta(level, A.n, maxRowLen), next = 0.0;
    for (int left = 3;; --left, theta *= 0.5) {
      step.agg = sa_aggregate(A, theta, step.nc);
      next = sa_next_entries(A, step.agg, step.nc);
      if (left == 0 || next <= most || (level == 0 && theta < 2 * kSaLeastTheta)) break;
    }
    const bool slow = step.nc > A.n / 2, dense = level > 0 ? next > most : A.n > kSaDenseRows && next > 10.0 * A.n;
    if (!slow && !dense) return true;
  }
  if (!sa_groupable(A, level)) return false;
  step.smooth = false;
  step.agg = sa_groups(A, kSaGroupSize, step.nc);
  return step.nc <= A.n / 2;
}

SaPattern sa_pattern(const SaMatrix& A, std::vector<int> aggIn, int nc, bool wantQT, bool smooth) {
  SaPattern S;
  S.n = A.n;
  S.nc = nc;
  S.agg = std::move(aggIn);
  const int n = A.n;
  build_rows(n, nc, S.pOff, S.pCol, [&](int i, std::vector<int>& out, std::vector<int>& mark) {
    auto add = [&](int I) {
      if (mark[I] == i) return;
      mark[I] = i;
      out.push_back(I);
    };
    add(S.agg[i]);
    for (int k = A.off[i]; smooth && k < A.off[i + 1]; ++k) add(S.agg[A.col[k]]);
  });
  build_rows(n, nc, S.qOff, S.qCol, [&](int i, std::vector<int>& out, std::vector<int>& mark) {
    auto add = [&](int j) {
      for (int k = S.pOff[j]; k < S.pOff[j + 1]; ++k) {
        const int I = S.pCol[k];
        if (mark[I] == i) continue;
        mark[I] = i;
        out.push_back(I);
      }
    };
    add(i);
    for (int k = A.off[i]; k < A.off[i + 1]; ++k) add(A.col[k]);
  });
  transpose(n, nc, S.pOff, S.pCol, S.ptOff, S.ptCol, S.ptSrc);
  if (wantQT) transpose(n, nc, S.qOff, S.qCol, S.qtOff, S.qtCol, S.qtSrc);
  build_rows(nc, nc, S.cOff, S.cCol, [&](int I, std::vector<int>& out, std::vector<int>& mark) {
    mark[I] = I;  // the diagonal is apart
    for (int e = S.ptOff[I]; e < S.ptOff[I + 1]; ++e) {
      const int i = S.ptCol[e];
      for (int k = S.qOff[i]; k < S.qOff[i + 1]; ++k) {
        const int J = S.qCol[k];
        if (mark[J] == I) continue;
        mark[J] = I;
        out.push_back(J);
      }
    }
  });
  return S;
}

SaMatrix sa_fine_matrix(const Layout& L, const std::vector<double>& vals, const std::vector<double>& diag) {
  SaMatrix A;
  A.n = L.nCells;
  A.off.assign((size_t)A.n + 1, 0);
  for (int r = 0; r < A.n; ++r) A.off[r + 1] = A.off[r] + L.rowLen[r];
  A.col.resize(A.off[A.n]);
  A.val.resize(A.off[A.n]);
  A.diag = diag;
#pragma omp parallel for schedule(static)
  for (int r = 0; r < A.n; ++r)
    for (int k = 0; k < L.rowLen[r]; ++k) {
      const int e = L.sliceOff[r / kSlice] + k * kSlice + r % kSlice;
      A.col[A.off[r] + k] = L.col[e];
      A.val[A.off[r] + k] = vals[e];
    }
  return A;
}

}  // namespace anb
