// CPU check of the host patterns of the smoothed-aggregation set-up (csrc/sa_setup.cpp) against sets built
// from their definitions, on 7-point grids; prints "ok" or the number of rows that differ.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "../../anabasis_b200/csrc/sa_setup.hpp"

using namespace anb;

static std::set<int> row(const std::vector<int>& off, const std::vector<int>& col, int i) {
  return std::set<int>(col.begin() + off[i], col.begin() + off[i + 1]);
}

int main(int argc, char** argv) {
  if (argc < 5) return 2;
  const int nx = std::atoi(argv[1]), ny = std::atoi(argv[2]), nz = std::atoi(argv[3]);
  const double theta = std::atof(argv[4]);
  SaMatrix A;
  A.n = nx * ny * nz;
  A.off.push_back(0);
  A.diag.assign(A.n, 0.1);
  unsigned s = 1;
  auto rnd = [&] { return ((s = s * 1664525u + 1013904223u) >> 8) / 16777216.0; };
  for (int k = 0; k < nz; ++k)
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i) {
        const int r = (k * ny + j) * nx + i;
        auto add = [&](int a, int b, int c, double w) {
          if (a < 0 || b < 0 || c < 0 || a >= nx || b >= ny || c >= nz) return;
          const double v = w * (1 + 0.3 * rnd());
          A.col.push_back((c * ny + b) * nx + a);
          A.val.push_back(-v);
          A.diag[r] += v;
        };
        add(i, j, k - 1, 4.5), add(i, j - 1, k, 4.5), add(i - 1, j, k, 1.0);
        add(i + 1, j, k, 1.0), add(i, j + 1, k, 4.5), add(i, j, k + 1, 4.5);
        A.off.push_back((int)A.col.size());
      }
  int nc = 0, bad = 0;
  const std::vector<int> agg = sa_aggregate(A, theta, nc);
  const double guess = sa_next_entries(A, agg, nc);
  const SaPattern S = sa_pattern(A, agg, nc, true);
  std::set<int> used(agg.begin(), agg.end());
  bad += (int)used.size() != nc || *used.begin() != 0 || *used.rbegin() != nc - 1;
  for (int i = 0; i < A.n; ++i) {
    std::set<int> p, q;
    p.insert(agg[i]);
    for (int j : row(A.off, A.col, i)) p.insert(agg[j]);
    q = row(S.pOff, S.pCol, i);
    bad += p != q || (int)q.size() != S.pOff[i + 1] - S.pOff[i];
    for (int j : row(A.off, A.col, i))
      for (int I : row(S.pOff, S.pCol, j)) q.insert(I);
    bad += q != row(S.qOff, S.qCol, i) || (int)q.size() != S.qOff[i + 1] - S.qOff[i];
  }
  for (int I = 0; I < nc; ++I) {
    std::set<int> c;
    for (int e = S.ptOff[I]; e < S.ptOff[I + 1]; ++e) {
      const int i = S.ptCol[e], k = S.ptSrc[e];
      bad += k < S.pOff[i] || k >= S.pOff[i + 1] || S.pCol[k] != I || (e > S.ptOff[I] && S.ptCol[e - 1] >= i);
      for (int J : row(S.qOff, S.qCol, i)) c.insert(J);
    }
    c.erase(I);
    bad += c != row(S.cOff, S.cCol, I) || (int)c.size() != S.cOff[I + 1] - S.cOff[I];
    for (int e = S.qtOff[I]; e < S.qtOff[I + 1]; ++e) {
      const int i = S.qtCol[e], k = S.qtSrc[e];
      bad += k < S.qOff[i] || k >= S.qOff[i + 1] || S.qCol[k] != I;
    }
  }
  bad += S.ptCol.size() != S.pCol.size() || S.qtCol.size() != S.qCol.size();
  if (A.n >= 5000) bad += guess < 0.7 * S.cCol.size() || guess > 1.4 * S.cCol.size();
  if (bad) std::printf("%d rows differ\n", bad);
  else std::printf("ok\n");
  return bad != 0;
}
