// Band plans of the on-chip FP32 sweep (host only).
#include "x2g_columns_plan.h"

#include <algorithm>

namespace x2g {

namespace {

constexpr int kFirst = 5;  // first interior row
constexpr int kSide = 5;   // fewest rows a thread has below the row seam, if it lies in its rows
constexpr int kAbove = 10;  // and above it
constexpr int kBand = 8;   // fewest rows of a band
constexpr int kEnd = 4;    // fewest rows of a group of threads: a halo's

int slots(int rows) { return (rows + 4) / 5; }

// The cut of a band with the row seam after its first p rows and q rows above
// it, so that no thread has more than m slots; -1: there is none.  One group:
// the band's height.
int seam_cut(int p, int q, int m, int groups) {
  if (p < kSide || q < kAbove) return -1;
  if (groups == 1) return slots(p) + slots(q) <= m ? p + q : -1;
  // the seam in the first group's rows: x upper rows with the p lower ones
  int x = std::min(5 * (m - slots(p)), q - kEnd);
  if (x >= kAbove && q - x <= 5 * m) return p + std::max(kAbove, std::min(x, (p + q + 1) / 2 - p));
  // or in the second's: x lower rows with the q upper ones
  x = std::min(5 * (m - slots(q)), p - kEnd);
  if (x >= kSide && p - x <= 5 * m) return p - std::max(kSide, std::min(x, (p + q + 1) / 2 - q));
  return -1;
}

// what k_columns relies on
bool holds(const ColPlan &p, int nmu, int seam) {
  if (p.row0[0] != kFirst || p.row0[p.size] != nmu) return false;
  for (int k = 0; k < p.size; ++k) {
    const int n = p.row0[k + 1] - p.row0[k];
    // halos come from the next band alone, a halo's rows from one group
    if (n < kBand || n > p.maxrows || (p.groups == 2 && (p.cut[k] < kEnd || p.cut[k] > n - kEnd))) return false;
    for (int g = 0; g < p.groups; ++g) {
      const int a = p.row0[k] + (g ? p.cut[k] : 0), b = g + 1 < p.groups ? p.row0[k] + p.cut[k] : p.row0[k + 1];
      if (a < seam && b > seam) {
        if (seam - a < kSide || b - seam < kAbove || slots(seam - a) + slots(b - seam) > p.slots) return false;
      } else if (a == seam || b == seam || slots(b - a) > p.slots) {
        return false;
      }
    }
  }
  return true;
}

}  // namespace

// kl bands of nearly equal height below the seam's band, size - 1 - kl above
// it.  The least slots m with which the rows can be placed, then the least
// height of the tallest band.
bool column_plan(int nni, int nmu, int size, int groups, ColPlan &plan) {
  const int seam = (nmu + 7) / 2, lower = seam - kFirst, upper = nmu - seam;
  if (size < 1 || size > kMaxCluster) return false;
  for (int m = std::max(1, slots(lower + upper) / (size * groups)); m <= slots(lower) + slots(upper); ++m) {
    const int cap = 5 * m * groups;
    int best = 1 << 30, bp = 0, bq = 0, bk = -1;
    for (int kl = 0; kl < size; ++kl) {
      const int ku = size - 1 - kl;
      const int p0 = kl ? std::max(kSide, lower - cap * kl) : lower, p1 = kl ? std::min(cap, lower - kBand * kl) : lower;
      const int q0 = ku ? std::max(kAbove, upper - cap * ku) : upper, q1 = ku ? std::min(cap, upper - kBand * ku) : upper;
      for (int p = p0; p <= p1; ++p)
        for (int q = q0; q <= q1; ++q) {
          const int hl = kl ? (lower - p + kl - 1) / kl : 0, hu = ku ? (upper - q + ku - 1) / ku : 0;
          const int tallest = std::max(std::max(hl, hu), p + q);
          if (tallest < best && p + q >= kBand && seam_cut(p, q, m, groups) > 0) {
            best = tallest;
            bp = p;
            bq = q;
            bk = kl;
          }
        }
    }
    if (bk < 0) continue;
    plan.size = size;
    plan.groups = groups;
    plan.slots = m;
    plan.maxrows = best;
    int at = 0;
    auto share = [&](int from, int rows, int k) {
      for (int i = 0; i < k; ++i) plan.row0[at++] = from + rows * i / k;
    };
    share(kFirst, lower - bp, bk);
    plan.row0[at++] = seam - bp;
    share(seam + bq, upper - bq, size - 1 - bk);
    for (int k = size; k <= kMaxCluster; ++k) plan.row0[k] = nmu;
    for (int k = 0; k < kMaxCluster; ++k) {
      const int n = k < size ? plan.row0[k + 1] - plan.row0[k] : 0;
      plan.cut[k] = k == bk ? seam_cut(bp, bq, m, groups) : groups == 2 ? (n + 1) / 2 : n;
    }
    plan.pitch = (nni + 8 + 31) / 32 * 32;
    // the seam's columns nnix - 2 .. nnix + 2 in one warp
    const int nnix = (nni + 7) / 2;
    plan.shift = 0;
    while ((nnix - 7 + plan.shift) % 32 > 27) ++plan.shift;
    plan.warps = (nni - 2 + plan.shift + 31) / 32;
    if (holds(plan, nmu, seam)) return true;
  }
  return false;
}

}  // namespace x2g
