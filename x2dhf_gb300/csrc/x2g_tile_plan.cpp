// Plan of whole schedule tiles for one cluster per relaxation job, made when it
// is asked for (host only, for inspection: no kernel reads it; the on-chip
// sweep's plans are those of x2g_columns_plan.cpp).
#include <algorithm>
#include <utility>

#include "x2g_internal.h"

namespace x2g {

namespace {

struct TilePlan {
  int size = 0, maxrows = 0;  // CTAs per job (0: the grid needs more than one cluster)
  size_t smem = 0;
  std::vector<int> row0;  // CTA k owns ext rows [row0[k], row0[k+1])
  // the CTAs' points regrouped [cta][colour][segment] as chunks, with
  // size * 5 * segments + 1 offsets: with the schedule's colours and levels,
  // and with the seam-free colouring
  std::vector<int> pts, off, free_pts, free_off;
};

// Chunks of one segment appended to `chunks`: the segment's points (ext
// row, col) of one CTA band starting at ext row r0 grouped into runs of up to
// 4 points of one row at stride 5, packed (band row << 19) | (col << 2) |
// (count - 1), and dealt round-robin over buckets of the shared-memory bank
// of their first correction value, so that a warp's 32 chunks start on
// distinct banks where the buckets allow.
static void append_chunks(std::vector<std::pair<int, int>> &pts, int r0, int n8, std::vector<int> &chunks) {
  std::sort(pts.begin(), pts.end());
  std::vector<std::vector<int>> bank(32);
  for (size_t i = 0; i < pts.size();) {
    size_t n = 1;
    while (n < 4 && i + n < pts.size() && pts[i + n].first == pts[i].first &&
           pts[i + n].second == pts[i + n - 1].second + 5)
      ++n;
    const int lr = pts[i].first - r0;
    bank[((lr + 4) * n8 + pts[i].second) % 32].push_back(
        int((unsigned(lr) << 19) | (unsigned(pts[i].second) << 2) | unsigned(n - 1)));
    i += n;
  }
  for (size_t depth = 0, left = 1; left;) {
    left = 0;
    for (auto &bk : bank)
      if (depth < bk.size()) {
        chunks.push_back(bk[depth]);
        left = 1;
      }
    ++depth;
  }
}

// The segments of the seam-free colouring on the CTA bands r0: colour (col -
// row) mod 5 of the ext point, so the stencil's neighbours at distance 1..4
// along a row or a column always have another colour and the points of one
// colour are independent.  Per (CTA, colour) segment A (no halo read or write),
// B (within 4 rows of a shared band edge), and an empty seam segment.
void free_chunks(const Schedule &g, const std::vector<int> &r0, TilePlan &plan) {
  const int C = int(r0.size()) - 1;
  plan.free_off.push_back(0);
  for (int k = 0; k < C; ++k) {
    auto edge = [&](int row) { return (k > 0 && row < r0[k] + 4) || (k < C - 1 && row >= r0[k + 1] - 4); };
    const int ra = std::max(r0[k], 5), rb = std::min(r0[k + 1], g.nmu);
    for (int c = 0; c < 5; ++c)
      for (int seg = 0; seg < 3; ++seg) {
        std::vector<std::pair<int, int>> pts;
        for (int row = ra; row < rb && seg < 2; ++row) {
          if (edge(row) != (seg == 1)) continue;
          for (int col = 5; col <= g.nni + 2; ++col)
            if (((col - row) % 5 + 5) % 5 == c) pts.push_back({row, col});
        }
        append_chunks(pts, r0[k], g.n8, plan.free_pts);
        plan.free_off.push_back(int(plan.free_pts.size()));
      }
  }
}

// Contiguous tile ranges, ~30 rows per CTA, 2..16 CTAs of at least 4 rows
// (halos come from the next CTA only); shared memory per CTA for (residual,
// omega/lhs) pairs, the correction band with 4-row halos, b(mu) of the band's
// rows, d(nu) by column, the segment offsets and the CTA's chunks.
TilePlan tile_plan(const Schedule &g) {
  TilePlan plan;
  const int rows = g.nmu - 4, C = std::min(std::max(2, std::min(16, (rows + 29) / 30)), g.ntiles);
  if (C < 2) return plan;
  std::vector<int> t0(C + 1), r0(C + 1);
  int t = 0;
  t0[0] = 0;
  for (int k = 1; k < C; ++k) {
    const int target = 4 + (rows * k + C / 2) / C;
    while (t < g.ntiles - (C - k) && g.tile_row1[t] <= target) ++t;
    if (t <= t0[k - 1]) t = t0[k - 1] + 1;
    t0[k] = t;
  }
  t0[C] = g.ntiles;
  for (int k = 0; k < C; ++k) {
    if (t0[k + 1] <= t0[k]) return TilePlan();
    r0[k] = g.tile_row0[t0[k]];
    plan.maxrows = std::max(plan.maxrows, g.tile_row1[t0[k + 1] - 1] - g.tile_row0[t0[k]]);
  }
  r0[C] = g.nmu;
  for (int k = 0; k < C; ++k)
    if (r0[k + 1] - r0[k] < 4) return TilePlan();
  // colour and level of every point; a seam point is a level-0 point with a
  // neighbour of its colour (which then has a higher level)
  std::vector<signed char> colour(g.next, -1), level(g.next, 0);
  for (int b = 0; b < g.ntiles * 5 * g.nlev; ++b)
    for (int q = g.off[b]; q < g.off[b + 1]; ++q) {
      colour[g.pts[q]] = (signed char)(b / g.nlev % 5);
      level[g.pts[q]] = (signed char)(b % g.nlev);
    }
  auto seam = [&](int ij) {
    for (int k = 1; k <= 4; ++k)
      for (int o : {k, -k, k * g.n8, -k * g.n8})
        if (colour[ij + o] == colour[ij] && level[ij + o] > 0) return true;
    return false;
  };
  // per (CTA, colour) the level-0 points off the shared band edges, those within
  // 4 rows of one, the level-0 seam points, then the levels 1..nlev-1
  const int S = g.nlev + 2;
  int maxchunks = 0;
  plan.off.push_back(0);
  for (int k = 0; k < C; ++k) {
    const int first = int(plan.pts.size());
    auto edge = [&](int row) { return (k > 0 && row < r0[k] + 4) || (k < C - 1 && row >= r0[k + 1] - 4); };
    for (int c = 0; c < 5; ++c)
      for (int seg = 0; seg < S; ++seg) {
        const int l = (seg < 2) ? 0 : seg - 2;
        std::vector<std::pair<int, int>> pts;
        for (int u = t0[k]; u < t0[k + 1]; ++u) {
          const int o = (u * 5 + c) * g.nlev + l;
          for (int q = g.off[o]; q < g.off[o + 1]; ++q) {
            const int ij = g.pts[q], row = ij / g.n8, col = ij % g.n8;
            if (seg < 3) {
              const bool s0 = seam(ij);
              if (seg == 2 ? !s0 : (s0 || edge(row) != (seg == 1))) continue;
            }
            pts.push_back({row, col});
          }
        }
        append_chunks(pts, r0[k], g.n8, plan.pts);
        plan.off.push_back(int(plan.pts.size()));
      }
    maxchunks = std::max(maxchunks, int(plan.pts.size()) - first);
  }
  plan.smem = 2 * size_t(plan.maxrows) * g.n8 * sizeof(float) + size_t(plan.maxrows + 8) * g.n8 * sizeof(float) +
              size_t(plan.maxrows + g.n8) * sizeof(float) + size_t(5 * S + 1) * sizeof(int) +
              size_t(maxchunks) * sizeof(int);
  if (plan.maxrows >= 4096 || g.n8 >= (1 << 17) || plan.smem > 200 * 1024) return TilePlan();
  plan.size = C;
  plan.row0 = r0;
  free_chunks(g, r0, plan);
  return plan;
}

int host_tile_plan(int nnu, int nmu, TilePlan &plan) {
  HostGrid g;
  if (!build_host_grid(g, nnu, nmu, 2.0, 40.0, 1.0, 1.0, 4).empty()) return X2G_ERR_SCHEDULE;
  plan = tile_plan(*g.s);
  return X2G_OK;
}

int copy_chunks(const std::vector<int> &pts, const std::vector<int> &offsets, int *nchunks, int *noff, int *chunks, int *off) {
  if (nchunks) *nchunks = int(pts.size());
  if (noff) *noff = int(offsets.size());
  if (chunks) std::copy(pts.begin(), pts.end(), chunks);
  if (off) std::copy(offsets.begin(), offsets.end(), off);
  return X2G_OK;
}

}  // namespace
}  // namespace x2g

// CTAs per job, rows per CTA, shared memory bytes; row0[C+1] when non-NULL.
extern "C" int x2g_host_cluster_plan(int nnu, int nmu, int *csize, int *maxrows, long *smem, int *row0) {
  x2g::TilePlan plan;
  const int rc = x2g::host_tile_plan(nnu, nmu, plan);
  if (rc != X2G_OK) return rc;
  if (csize) *csize = plan.size;
  if (maxrows) *maxrows = plan.maxrows;
  if (smem) *smem = long(plan.smem);
  if (row0) std::copy(plan.row0.begin(), plan.row0.end(), row0);
  return X2G_OK;
}

// Packed chunks and segment offsets (CTA-major, 5 colours x (nlevels + 2)
// segments per CTA, plus the end).  Null arrays: the counts.
extern "C" int x2g_host_cluster_chunks(int nnu, int nmu, int *nchunks, int *noff, int *chunks, int *off) {
  x2g::TilePlan plan;
  const int rc = x2g::host_tile_plan(nnu, nmu, plan);
  return rc != X2G_OK ? rc : x2g::copy_chunks(plan.pts, plan.off, nchunks, noff, chunks, off);
}

// The same for the seam-free colouring.
extern "C" int x2g_host_free_chunks(int nnu, int nmu, int *nchunks, int *noff, int *chunks, int *off) {
  x2g::TilePlan plan;
  const int rc = x2g::host_tile_plan(nnu, nmu, plan);
  return rc != X2G_OK ? rc : x2g::copy_chunks(plan.free_pts, plan.free_off, nchunks, noff, chunks, off);
}
