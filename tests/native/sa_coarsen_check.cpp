// CPU replay of the smoothed-aggregation level steps (csrc/sa_setup.cpp) with values computed on the host:
// 7-point grids of spacings hx, hy, hz and cell coefficients spread over a factor.  Prints "refused at <level>"
// or "levels <count>" after checking that every step halves the rows at least, that a refusal comes on the
// two finest levels or above the rows that can be grouped, and that the last level fits the dense inverse.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "../../anabasis_b200/csrc/sa_setup.hpp"

using namespace anb;

struct Csr {
  int n = 0, m = 0;
  std::vector<int> off{0}, col;
  std::vector<double> val;
};

static Csr multiply(const Csr& a, const Csr& b) {
  Csr c;
  c.n = a.n;
  c.m = b.m;
  std::vector<double> acc(b.m, 0.0);
  std::vector<int> mark(b.m, -1), cols;
  for (int i = 0; i < a.n; ++i) {
    cols.clear();
    for (int k = a.off[i]; k < a.off[i + 1]; ++k)
      for (int q = b.off[a.col[k]]; q < b.off[a.col[k] + 1]; ++q) {
        const int j = b.col[q];
        if (mark[j] != i) {
          mark[j] = i;
          acc[j] = 0.0;
          cols.push_back(j);
        }
        acc[j] += a.val[k] * b.val[q];
      }
    std::sort(cols.begin(), cols.end());
    for (int j : cols) {
      c.col.push_back(j);
      c.val.push_back(acc[j]);
    }
    c.off.push_back((int)c.col.size());
  }
  return c;
}

static Csr transpose(const Csr& a) {
  Csr t;
  t.n = a.m;
  t.m = a.n;
  t.off.assign(t.n + 1, 0);
  t.col.resize(a.col.size());
  t.val.resize(a.col.size());
  for (int j : a.col) t.off[j + 1]++;
  for (int j = 0; j < t.n; ++j) t.off[j + 1] += t.off[j];
  std::vector<int> fill(t.off.begin(), t.off.end() - 1);
  for (int i = 0; i < a.n; ++i)
    for (int k = a.off[i]; k < a.off[i + 1]; ++k) {
      const int s = fill[a.col[k]]++;
      t.col[s] = i;
      t.val[s] = a.val[k];
    }
  return t;
}

static int fail(const char* what, int level) {
  std::printf("%s on level %d\n", what, level);
  return 1;
}

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  const int N = std::atoi(argv[1]);
  const double h[3] = {std::atof(argv[2]), std::atof(argv[3]), std::atof(argv[4])}, spread = std::atof(argv[5]);
  SaMatrix A;
  A.n = N * N * N;
  A.off.push_back(0);
  A.diag.assign(A.n, 0.0);
  unsigned s = 1;
  std::vector<double> kappa(A.n);
  for (double& k : kappa) k = std::pow(spread, ((s = s * 1664525u + 1013904223u) >> 8) / 16777216.0);
  for (int r = 0; r < A.n; ++r) {
    const int x[3] = {r % N, r / N % N, r / N / N}, step[3] = {1, N, N * N};
    for (int q : {2, 1, 0, 3, 4, 5}) {  // columns in ascending order: -z -y -x +x +y +z
      const int a = q % 3, to = x[a] + (q < 3 ? -1 : 1);
      const double c = 1.0 / (h[a] * h[a]);
      if (to < 0 || to >= N) {
        A.diag[r] += 2.0 * c * kappa[r];
        continue;
      }
      const int j = r + (q < 3 ? -step[a] : step[a]);
      const double v = 2.0 * c * kappa[r] * kappa[j] / (kappa[r] + kappa[j]);
      A.col.push_back(j);
      A.val.push_back(-v);
      A.diag[r] += v;
    }
    A.off.push_back((int)A.col.size());
  }
  int level = 0;
  for (; A.n > 128; ++level) {
    if (level + 1 >= kSaMaxLevels) return fail("too many levels", level);
    SaStep step;
    if (!sa_coarsen(A, level, 6, false, step)) {
      if (level > 1 && A.n <= kSaGroupRows) return fail("a level that can be grouped was refused", level);
      std::printf("refused at %d\n", level);
      return 0;
    }
    if (2 * step.nc > A.n) return fail("slow step", level);
    // A as CSR, P, and the next matrix
    Csr full, p0;
    full.n = full.m = p0.n = A.n;
    p0.m = step.nc;
    for (int i = 0; i < A.n; ++i) {
      full.col.push_back(i);
      full.val.push_back(A.diag[i]);
      for (int k = A.off[i]; k < A.off[i + 1]; ++k) {
        full.col.push_back(A.col[k]);
        full.val.push_back(A.val[k]);
      }
      full.off.push_back((int)full.col.size());
      p0.col.push_back(step.agg[i]);
      p0.val.push_back(1.0);
      p0.off.push_back(i + 1);
    }
    Csr p = p0;
    if (step.smooth) {
      Csr m = full;
      for (int i = 0; i < m.n; ++i)
        for (int k = m.off[i]; k < m.off[i + 1]; ++k)
          m.val[k] = (m.col[k] == i ? 1.0 : 0.0) - 2.0 / 3.0 / A.diag[i] * m.val[k];
      p = multiply(m, p0);
    }
    const Csr next = multiply(transpose(p), multiply(full, p));
    // the estimate looks at every 16th row: half as much again covers its scatter on the small levels
    if (step.smooth && level > 0 && (double)next.col.size() > 1.5 * 1.25 * (A.col.size() + A.n))
      return fail("the next matrix is denser than asked for", level);
    if (!step.smooth && next.col.size() > full.col.size()) return fail("groups filled in", level);
    SaMatrix c;
    c.n = next.n;
    c.off.push_back(0);
    c.diag.assign(c.n, 0.0);
    for (int i = 0; i < c.n; ++i) {
      for (int k = next.off[i]; k < next.off[i + 1]; ++k) {
        if (next.col[k] == i) {
          c.diag[i] = next.val[k];
        } else {
          c.col.push_back(next.col[k]);
          c.val.push_back(next.val[k]);
        }
      }
      c.off.push_back((int)c.col.size());
    }
    A = std::move(c);
  }
  std::printf("levels %d\n", level + 1);
  return 0;
}
