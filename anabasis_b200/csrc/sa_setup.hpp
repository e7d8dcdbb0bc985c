// Host side of the set-up of the smoothed-aggregation hierarchy that preconditions the pressure CG.
//
// One level step: strong couplings (a_ij < 0, a_ij^2 > theta^2 a_ii a_jj) give star aggregates (a
// root with all its strong neighbours where all of them are free; the rows left over join the
// aggregate of their strongest aggregated neighbour, what remains forms aggregates of its own).  The
// prolongator is P = (I - omegaP D^-1 A) P0 with P0 piecewise constant.  Only patterns are made here:
// they follow the matrix pattern and the aggregates, never the values, so the device can refresh every
// value in place when the matrix changes (sa_refresh).
#pragma once

#include <vector>

#include "layout.hpp"

namespace anb {

// Off-diagonal CSR with the diagonal apart.
struct SaMatrix {
  int n = 0;
  std::vector<int> off, col;
  std::vector<double> val, diag;
};

struct SaPattern {
  int n = 0, nc = 0;
  std::vector<int> agg;                 // n
  std::vector<int> pOff, pCol;          // P by rows: the aggregates of the row and its neighbours
  std::vector<int> qOff, qCol;          // A P by rows (the pattern of P is part of it)
  std::vector<int> ptOff, ptCol, ptSrc; // P^T by rows: fine row and entry of P
  std::vector<int> qtOff, qtCol, qtSrc; // Q^T by rows: fine row and entry of Q (only on request)
  std::vector<int> cOff, cCol;          // off-diagonals of the next level's matrix P^T A P
};

constexpr int kSaMaxLevels = 12;
// Threshold of the strong couplings.  On the finest level 0.02 keeps every face of a mildly stretched
// hex grid strong (level 1: n / 8 rows of 30 entries), 0.1 coarsens along the strong directions only
// (n / 5.6 rows of 38): fewer iterations of a dearer cycle, which pays where launches and not bytes
// set the cycle's time (ms per SIMPLE step, 0.1 / 0.02: 16k hexes 2.00 / 2.24, 36k 5.5 / 6.1, 250k
// 6.3 / 5.65, 970k 20.4 / 18.4) and on tetrahedra, whose rows stay short (334k 9.7 / 10.3).  Below,
// 0.04 (0.02: 82 iterations a step at 970k cells instead of 65; 0.06: matrices too dense).
inline double sa_theta(int level, int n, int maxRowLen) {
  if (level > 0) return 0.04;
  return n <= 100000 || maxRowLen <= 4 ? 0.1 : 0.02;
}

// Aggregate of every row; nc receives the count.  Aggregates are numbered by their first row.
std::vector<int> sa_aggregate(const SaMatrix& A, double theta, int& nc);
// Estimate of the next matrix's off-diagonal entries for these aggregates, from every 16th of its rows.
double sa_next_entries(const SaMatrix& A, const std::vector<int>& agg, int nc);
// Aggregates of up to `size` rows, each a row with its strongest free neighbours (rows left over join their
// strongest neighbour's), whatever the threshold: a full matrix shrinks by about that factor.
std::vector<int> sa_groups(const SaMatrix& A, int size, int& nc);

// One level step.  The threshold is halved, at most three times, while the next matrix would hold more than
// 1.25 times this one's entries: fewer weak couplings, larger aggregates.  It is the first sign of trouble
// when that does not help, or when less than half of the rows go (weak couplings throughout: spread
// coefficients, or a level that is nearly full).  Then
//  - a deep level (the third of the hierarchy or lower, up to kSaGroupRows rows) or a second one that is a
//    quarter full is grouped by eight with a piecewise constant P (smooth = false): the next matrix has no
//    more entries a row than this one;
//  - otherwise the step is refused, and the plain aggregation serves, before another level has been built.
// On the finest level the threshold stays at kSaLeastTheta or more, which keeps the weak directions of a
// stretched grid weak.  Flat cells (two weak directions) are then joined to lines of three and the second level
// is dense, 16 entries for every finest row of a hex grid and 8 on tets.  It coarsens well again up to 16:1,
// and pays where launches set the time of a cycle: ms a step, taken / refused, 36k hexes of 10:1 3.1 / 5.4,
// 97k 5.2 / 6.3, 246k 9.2 / 10.0, 980k 39.4 / 23.8; 691k tets 19.5 / 28.2.  It is refused above kSaDenseRows
// rows with more than 10 entries for each.  groups: go to the groups at once (the caller found a row too
// long for the device's products).
struct SaStep {
  std::vector<int> agg;
  int nc = 0;
  bool smooth = true;
};
constexpr double kSaLeastTheta = 0.01;
constexpr int kSaDenseRows = 250000;
constexpr int kSaGroupRows = 16384;
constexpr int kSaGroupSize = 8;
inline bool sa_groupable(const SaMatrix& A, int level) {
  return level > 1 ? A.n <= kSaGroupRows : level == 1 && 4.0 * A.col.size() > (double)A.n * A.n;
}
bool sa_coarsen(const SaMatrix& A, int level, int maxRowLen, bool groups, SaStep& step);

// All patterns of one level step for the given aggregates; P is piecewise constant without smooth.
SaPattern sa_pattern(const SaMatrix& A, std::vector<int> agg, int nc, bool wantQT, bool smooth = true);
// The level-0 matrix as CSR; vals in the layout's SELL-32 storage.
SaMatrix sa_fine_matrix(const Layout& L, const std::vector<double>& vals, const std::vector<double>& diag);

}  // namespace anb
