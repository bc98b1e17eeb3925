// Host-side construction of the grid, operator tables and the GPU sweep
// schedule.  The formulas are those of x2dhf's src/initCBAllocArrays.F90
// (initCBlocks:813-858, initSuppl:1636-2051, initLP:1517-1560, mesh:2503-2544)
// written out in 0-based C++; the schedule (row bands, colour levels) is this
// library's own.
#include <algorithm>
#include <memory>
#include <mutex>
#include <cmath>
#include <cstdio>
#include <numeric>

#include "x2g_columns_plan.h"
#include "x2g_internal.h"

namespace x2g {

namespace {

// 7-point Newton-Cotes weights on n = 1 (mod 6) points (initSuppl:1917-1955)
std::vector<double> newton_cotes(int n, double h) {
  std::vector<double> w(n + 6, 0.0);
  double w1 = h / 140.0;
  w[0] = 0.0 + w1 * 41.0;
  for (int i = 1; i < n; i += 6) {
    w[i] = w1 * 216.0;
    w[i + 1] = w1 * 27.0;
    w[i + 2] = w1 * 272.0;
    w[i + 3] = w1 * 27.0;
    w[i + 4] = w1 * 216.0;
    w[i + 5] = (i + 5 == n - 1) ? w1 * 41.0 : 2.0 * w1 * 41.0;
  }
  w.resize(n);
  return w;
}

// Sweeps over a list as a pipelined wavefront: list-order SOR over the
// "middle" list, MCSOR over the same list colour after colour (mcsor's loops
// i = c, ngrid, 5 one after the other).  A sequential sweep over the list
// (sormcsor.F90:41-74, 170-386) followed by the axis extrapolation
// (:94-129) after every sweep is reproduced exactly when every point update
// and every axis extrapolation of sweep s runs at step level + s * delta and
// the updates of one step run in any order: a point reads the new values of
// its neighbours earlier in the list (lower levels, this sweep), the previous
// sweep's values of those later in the list and of the axis, and delta makes
// every such previous-sweep value final before it is read and not yet
// overwritten.  The ghost cells and the mu >= nmu-3 rows stay fixed during a
// relaxation call.
//
// One pass over the list: a point's neighbours earlier in it are those that have
// a level already.  Its level is above theirs, so that it reads their new values
// and they its old one, if delta exceeds the difference; the same holds for an
// axis point and the five it reads, among which are the only points that read
// it.
std::string build_wave_schedule(const Schedule &g, const std::vector<int> &order, const std::vector<int> &packed,
                                const int *offs, WaveHost &w) {
  const int npts = int(order.size()), n8 = g.n8, nni = g.nni, nmu = g.nmu;
  std::vector<int> level(g.next, -1), mask(npts);  // level by ext index
  int nlev = 0, delta = 1;
  for (int p = 0; p < npts; ++p) {
    // an interior point's 16 neighbours all lie in the extended array
    const int *at = level.data() + order[p];
    int most = -1;
    unsigned least = ~0u, m = 0;
    for (int k = 0; k < 16; ++k) {
      const int l = at[offs[k]];
      most = std::max(most, l);
      least = std::min(least, unsigned(l));
      m |= unsigned(l >= 0) << k;
    }
    if (m) delta = std::max(delta, most + 1 - int(least) + 1);  // the earlier one's old value
    level[order[p]] = most + 1;
    mask[p] = int(m);
    nlev = std::max(nlev, most + 2);
  }
  // axis points (sormcsor.F90:94-129, lists of mesh:2823-2842): the mu=1
  // row (ext row 4, cols 5..nni+2) from rows 5..9, then the nu=1 and nu=nni
  // columns (ext rows 4..nmu-1, cols 4 and nni+3) from the 5 columns inward;
  // their row-4 corners read the mu=1 row
  struct Axis {
    int ij, st;
  };
  std::vector<Axis> ax;
  for (int c = 5; c <= nni + 2; ++c) ax.push_back({4 * n8 + c, n8});
  for (int r = 4; r < nmu; ++r) {
    ax.push_back({r * n8 + 4, 1});
    ax.push_back({r * n8 + nni + 3, -1});
  }
  int nblev = 0;
  for (const Axis &a : ax) {
    int most = -1, least = 0x7fffffff;
    for (int k = 1; k <= 5; ++k) {
      const int l = level[a.ij + k * a.st];
      if (l < 0) return "schedule: an axis point reads neither an interior nor an axis point";
      most = std::max(most, l);
      least = std::min(least, l);
    }
    level[a.ij] = most + 1;
    delta = std::max(delta, most + 1 - least + 1);  // read before the next sweep overwrites it
    nblev = std::max(nblev, most + 2);
  }
  w.nlev = nlev;
  w.nblev = nblev;
  w.delta = delta;
  w.off.assign(nlev + 1, 0);
  for (int p = 0; p < npts; ++p) w.off[level[order[p]] + 1]++;
  for (int l = 0; l < nlev; ++l) w.off[l + 1] += w.off[l];
  w.pts.resize(size_t(npts) * 2);
  {
    std::vector<int> fill(w.off.begin(), w.off.end() - 1);
    for (int p = 0; p < npts; ++p) {
      const int at = fill[level[order[p]]]++, rc = packed[p], row = rc >> 16, col = rc & 0xffff;
      w.pts[2 * size_t(at)] = rc;
      // and whether it is the fifth point of an axis extrapolation
      w.pts[2 * size_t(at) + 1] = mask[p] | (row == 9) << 16 | (col == 9) << 17 | (col == nni - 2) << 18;
    }
  }
  w.boff.assign(nblev + 1, 0);
  for (const Axis &a : ax) w.boff[level[a.ij] + 1]++;
  for (int l = 0; l < nblev; ++l) w.boff[l + 1] += w.boff[l];
  w.bpts.assign(ax.size(), 0);
  {
    std::vector<int> fill(w.boff.begin(), w.boff.end() - 1);
    for (const Axis &a : ax) w.bpts[fill[level[a.ij]]++] = ((a.ij / n8) << 16) | (a.ij % n8);
  }
  return "";
}

// SOR's points by row and side, from the wavefront schedule (whose entries are
// sorted by level, so every row and side is in list order).
void build_march(Schedule &g) {
  const int sides = (g.nmu - 4) * 2, n8 = g.n8, last = g.nni + 3, middle = (g.n8 - 1) / 2 - 1;  // last column of the first half
  const int npts = int(g.sor.pts.size() / 2), naxis = int(g.sor.bpts.size());
  auto side = [&](int rc) { return ((rc >> 16) - 4) * 2 + ((rc & 0xffff) > middle); };
  g.march_off.assign(sides + 1, 0);
  for (int k = 0; k < npts; ++k) g.march_off[side(g.sor.pts[2 * size_t(k)]) + 1]++;
  for (int k = 0; k < naxis; ++k) g.march_off[side(g.sor.bpts[k]) + 1]++;
  for (int k = 0; k < sides; ++k) g.march_off[k + 1] += g.march_off[k];
  g.march_pts.resize(size_t(npts + naxis) * 2);
  std::vector<int> fill(g.march_off.begin(), g.march_off.end() - 1);
  auto add = [&](int rc, int mask) {
    const size_t at = size_t(fill[side(rc)]++) * 2;
    g.march_pts[at] = (rc >> 16) * n8 + (rc & 0xffff);
    g.march_pts[at + 1] = mask;
  };
  for (int k = 0; k < npts; ++k) add(g.sor.pts[2 * size_t(k)], g.sor.pts[2 * size_t(k) + 1]);
  for (int k = 0; k < naxis; ++k) {
    const int col = g.sor.bpts[k] & 0xffff;
    add(g.sor.bpts[k], int(col == 4 ? kMarchAxisUp : col == last ? kMarchAxisDown : kMarchAxisMu));
  }
}

}  // namespace

std::string attach_schedule(HostGrid &g);

std::string build_host_grid(HostGrid &g, int nni, int nmu, double r, double rinf, double z1, double z2,
                            int mpole) {
  if (nni < 13 || nmu < 13 || (nni - 1) % 6 || (nmu - 1) % 6 || (nni - 6) % 5 || (nmu - 6) % 5)
    return "grid sizes must be >= 13 and satisfy n = 1 (mod 6), n - 6 = 0 (mod 5)";
  if (!(r > 0) || !(rinf > r / 2)) return "bond length must be > 0 and R_inf > R/2";
  if (mpole < 2 || mpole > 8) return "mpole must be in [2,8]";
  g.nni = nni;
  g.nmu = nmu;
  g.n8 = nni + 8;
  g.m8 = nmu + 8;
  g.next = g.n8 * g.m8;
  g.mxsize = nni * nmu;
  g.r = r;
  g.r2 = r / 2.0;
  g.z1 = z1;
  g.z2 = z2;
  g.mpole = mpole;
  // grid steps (initCBlocks:813-858)
  g.hni = kPi / double(nni - 1);
  double xmi0 = 2.0 * rinf / r;
  xmi0 = std::log(xmi0 + std::sqrt(xmi0 * xmi0 - 1.0));
  g.hmu = xmi0 / double(nmu - 1);
  g.vxi.assign(nmu, 0);
  g.vxisq.assign(nmu, 0);
  g.vxi1.assign(nmu, 0);
  g.vxi2.assign(nmu, 0);
  double vmu = 0.0;
  for (int i = 0; i < nmu; i++) {
    if (i > 0) vmu = vmu + g.hmu;
    g.vxi[i] = std::cosh(vmu);
    g.vxisq[i] = g.vxi[i] * g.vxi[i];
    g.vxi1[i] = std::sqrt(g.vxi[i] * g.vxi[i] - 1.0);
    g.vxi2[i] = (i == 0) ? 0.0 : g.vxi[i] / g.vxi1[i];
  }
  g.veta.assign(nni, 0);
  g.vetasq.assign(nni, 0);
  g.veta1.assign(nni, 0);
  g.veta2.assign(nni, 0);
  for (int j = 0; j < nni; j++) {
    double vni = double(j) * g.hni;
    g.veta[j] = std::cos(vni);
    g.vetasq[j] = g.veta[j] * g.veta[j];
    g.veta1[j] = std::sqrt(1.0 - g.veta[j] * g.veta[j]);
    g.veta2[j] = (g.veta1[j] < kPrecis) ? 0.0 : g.veta[j] / g.veta1[j];
  }
  g.rinf = r * g.vxi[nmu - 1] / 2.0;
  // supplementary arrays (initSuppl:1759-1911), Coulomb nuclei
  const int mx = g.mxsize;
  g.e.assign(mx, 0);
  g.f0.assign(mx, 0);
  g.f1.assign(mx, 0);
  g.f2.assign(mx, 0);
  g.f4.assign(mx, 0);
  g.g.assign(mx, 0);
  g.wgt1.assign(mx, 0);
  g.wgt2.assign(mx, 0);
  g.borb_mu.assign(nmu, 0);
  g.bpot_mu.assign(nmu, 0);
  g.f3_mu.assign(nmu, 0);
  g.e_mu.assign(nmu, 0);
  g.e_nu.assign(nni, 0);
  g.d_nu = g.veta2;
  g.diag = -14350.0 / (5040.0) * (1.0 / (g.hmu * g.hmu) + 1.0 / (g.hni * g.hni));
  std::vector<double> wjac1(mx), wjac2(mx);
  const double wj1 = -r * kPi / 2.0, wj2 = r * r * kPi / 2.0, xrr = 0.5 * r;
  for (int i = 0; i < nmu; i++) {
    double w1 = g.vxi1[i], w2 = g.vxi[i] * g.vxi[i], w9 = xrr * g.vxi[i], w4 = g.vxi2[i];
    double w5 = 0.0, w6 = 0.0;
    if (i > 0) {
      w5 = g.vxi[i] / g.vxi1[i] - 2.0 * g.vxi1[i] / g.vxi[i];
      w6 = 1.0 / (g.vxi1[i] * g.vxi1[i]);
    }
    double w8 = -r * r * r * kPi * g.vxi[i] / 2.0;
    g.borb_mu[i] = w4;
    g.bpot_mu[i] = w5;
    g.f3_mu[i] = -2.0 / w2 + g.diag;
    g.e_mu[i] = -w6;
    for (int j = 0; j < nni; j++) {
      int ij = i * nni + j;
      double w10 = g.veta1[j];
      g.e[ij] = (w10 < kPrecis) ? 0.0 : (-w6 - 1.0 / (w10 * w10));
      if (i == 0) g.e_nu[j] = (w10 < kPrecis) ? 0.0 : 1.0 / (w10 * w10);
      double w7 = w2 - g.veta[j] * g.veta[j];
      g.f1[ij] = r * r * w7 / 2.0;
      g.f0[ij] = r * (g.vxi[i] * (z1 + z2) + g.veta[j] * (z2 - z1));
      g.f2[ij] = (i == 0) ? 0.0 : -r * w7 / g.vxi[i];
      g.g[ij] = w8 * w7;
      g.f4[ij] = w9;
      wjac1[ij] = wj1 * w1 * w10;
      wjac2[ij] = wj2 * w1 * w10 * (w1 * w1 + w10 * w10) / g.vxi[i];
    }
  }
  g.wmu = newton_cotes(nmu, g.hmu);
  g.wni = newton_cotes(nni, g.hni);
  for (int i = 0; i < nmu; i++)
    for (int j = 0; j < nni; j++) {
      int ij = i * nni + j;
      wjac1[ij] = g.wmu[i] * wjac1[ij];
      wjac2[ij] = g.wmu[i] * wjac2[ij];
      g.wgt1[ij] = g.wni[j] * wjac1[ij];
      g.wgt2[ij] = g.wni[j] * wjac2[ij];
    }
  // 8th-order Stirling coefficients (initSuppl:1680-1683, 1979-2001)
  static const double aa1[9] = {3.0, -32.0, 168.0, -672.0, 0.0, 672.0, -168.0, 32.0, -3.0};
  static const double aa2[9] = {-9.0, 128.0, -1008.0, 8064.0, -14350.0, 8064.0, -1008.0, 128.0, -9.0};
  const double c1 = 1.0 / (840.0), c2 = 1.0 / (5040.0);
  for (int k = 0; k < 4; k++) {
    g.dmu2[k] = c2 * aa2[k] / (g.hmu * g.hmu);
    g.dmu1[k] = c1 * aa1[k] / g.hmu;
    g.dni2[k] = c2 * aa2[k] / (g.hni * g.hni);
    g.dni1[k] = c1 * aa1[k] / g.hni;
  }
  g.dmu9.assign(9 * nmu, 0);
  g.dni9.assign(9 * nni, 0);
  for (int i = 0; i < nmu; i++)
    for (int k = 0; k < 9; k++) {
      double a2 = c2 * aa2[k] / (g.hmu * g.hmu), a1 = c1 * aa1[k] / g.hmu;
      g.dmu9[9 * i + k] = a2 + g.borb_mu[i] * a1;
    }
  for (int j = 0; j < nni; j++)
    for (int k = 0; k < 9; k++) {
      double a2 = c2 * aa2[k] / (g.hni * g.hni), a1 = c1 * aa1[k] / g.hni;
      g.dni9[9 * j + k] = a2 + g.d_nu[j] * a1;
    }
  g.exeven[0] = 210.0 / 126.0;
  g.exeven[1] = -120.0 / 126.0;
  g.exeven[2] = 45.0 / 126.0;
  g.exeven[3] = -10.0 / 126.0;
  g.exeven[4] = 1.0 / 126.0;
  // Legendre polynomials times (R/2 r)^k (initLP:1531-1589)
  g.leg.assign(size_t(mpole) * mx, 0.0);
  for (int i = 0; i < nmu; i++)
    for (int j = 0; j < nni; j++) {
      int ij = i * nni + j;
      double rr = std::sqrt(g.vxisq[i] + g.vetasq[j] - 1.0);
      double xr = g.r2 * rr;
      double costh = (std::fabs(rr) < kPrecis) ? 0.0 : g.vxi[i] * g.veta[j] / rr;
      double dome[10];
      dome[1] = costh;
      dome[2] = (3.0 * costh * costh - 1.0) * 0.50;
      for (int n = 2; n <= mpole - 1; n++)
        dome[n + 1] = (double(2 * n + 1) * costh * dome[n] - double(n) * dome[n - 1]) / double(n + 1);
      double xw = xr;
      g.leg[ij] = dome[1] * xw;
      for (int k = 2; k <= mpole; k++) {
        xw = xw * xr;
        g.leg[size_t(k - 1) * mx + ij] = dome[k] * xw;
      }
    }

  return attach_schedule(g);
}

// The sweep schedules of a grid -- "middle" ordering, colour levels, tiles,
// band plans, persistent-band and wavefront schedules -- depend on N_nu and
// N_mu only.  build_schedule makes them; attach_schedule takes them from a
// process-wide cache of the most recent grid sizes (they take tens of
// milliseconds to build; a serving loop or repeated solves on one grid size
// build them once, and the grids of a size share them).
static std::string build_schedule(Schedule &g) {
  const int nni = g.nni, nmu = g.nmu;
  // ------------------------------------------------------------------
  // "middle" ordering of the interior points (mesh:2503-2544), 1-based
  // ext rows ii in 6..nmu, cols jj in 6..nni+3, middle-outward.
  // ------------------------------------------------------------------
  const int n8 = g.n8 = nni + 8, m8 = nmu + 8, nmux = (m8 - 1) / 2, nnix = (n8 - 1) / 2;
  g.next = n8 * m8;
  const int npts = (nni - 2) * (nmu - 5);
  g.order.resize(npts);
  std::vector<int> packed(npts);  // the same points as (ext row << 16) | ext col
  std::vector<signed char> colour(g.next, -1);  // list position mod 5 (mcsor loops i=c,ngrid1,5)
  for (int i = 6, p = 0; i <= nmu; i++) {
    const int row = ((i <= nmux) ? nmux - i + 6 : i) - 1;
    for (int j = 6; j <= nni + 3; j++, p++) {
      const int col = ((j <= nnix) ? nnix - j + 6 : j) - 1;
      g.order[p] = row * n8 + col;
      packed[p] = (row << 16) | col;
      colour[row * n8 + col] = (signed char)(p % 5);
    }
  }
  // colour level: a point waits for every same-colour stencil neighbour
  // earlier in the list (new value read) and, by symmetry, is waited on by
  // every same-colour neighbour later in the list (old value read).
  std::vector<signed char> lev(g.next, -1);  // by ext index
  std::vector<std::pair<int, int>> deps;     // ext indices
  int offs[16];
  for (int k = 1; k <= 4; k++) {
    offs[4 * (k - 1) + 0] = -k;
    offs[4 * (k - 1) + 1] = k;
    offs[4 * (k - 1) + 2] = -k * n8;
    offs[4 * (k - 1) + 3] = k * n8;
  }
  int maxlev = 0;
  for (int p = 0; p < npts; p++) {
    const int ij = g.order[p], c = colour[ij];
    int L = 0;
    for (int o : offs) {
      const int q = ij + o;
      if (colour[q] != c || lev[q] < 0) continue;
      L = std::max(L, lev[q] + 1);
      deps.push_back({q, ij});
    }
    if (L >= kMaxLevels) return "colour level depth exceeds the schedule limit";
    lev[ij] = (signed char)L;
    maxlev = std::max(maxlev, L);
  }
  g.nlev = maxlev + 1;
  // row bands: 0-based ext rows [4, nmu); band 0 must hold rows 4..9 (the
  // mu=1 extrapolation reads rows 5..9), ~4 rows each, merged until every
  // same-colour dependency lies inside one band.
  const int H = 4;
  std::vector<int> bounds;
  bounds.push_back(4);
  int b = 10;
  while (b < nmu) {
    bounds.push_back(b);
    b += H;
  }
  bounds.push_back(nmu);
  // a band narrower than 2 rows at the end is merged into its neighbour
  if (bounds.size() > 2 && bounds[bounds.size() - 1] - bounds[bounds.size() - 2] < 2)
    bounds.erase(bounds.end() - 2);
  auto band_of = [&](int row) {
    return int(std::upper_bound(bounds.begin(), bounds.end(), row) - bounds.begin()) - 1;
  };
  for (bool changed = true; changed;) {
    changed = false;
    for (auto &d : deps) {
      int ra = d.first / n8, rb = d.second / n8;
      int ta = band_of(ra), tb = band_of(rb);
      if (ta != tb) {
        int lo = std::min(ta, tb), hi = std::max(ta, tb);
        bounds.erase(bounds.begin() + lo + 1, bounds.begin() + hi + 1);
        changed = true;
        break;
      }
    }
  }
  g.ntiles = int(bounds.size()) - 1;
  g.tile_row0.assign(bounds.begin(), bounds.end() - 1);
  g.tile_row1.assign(bounds.begin() + 1, bounds.end());
  // bucket points by (tile, colour, level), list order inside each bucket
  std::vector<int> tile(nmu);  // by ext row
  for (int row = 4; row < nmu; ++row) tile[row] = band_of(row);
  auto bucket = [&](int p) { return (tile[packed[p] >> 16] * 5 + colour[g.order[p]]) * g.nlev + lev[g.order[p]]; };
  const int nb = g.ntiles * 5 * g.nlev;
  g.off.assign(nb + 1, 0);
  for (int p = 0; p < npts; p++) g.off[bucket(p) + 1]++;
  for (int k = 0; k < nb; k++) g.off[k + 1] += g.off[k];
  g.pts.resize(npts);
  std::vector<int> rc(npts), fill(g.off.begin(), g.off.end() - 1);
  for (int p = 0; p < npts; p++) {
    const int at = fill[bucket(p)]++;
    g.pts[at] = g.order[p];
    rc[at] = packed[p];
  }
  g.st_pts.reserve(npts);
  g.st_place.resize(npts);
  g.st_off.assign(size_t(5) * g.nlev * (g.ntiles + 1), 0);
  for (int c = 0; c < 5; ++c)
    for (int l = 0; l < g.nlev; ++l) {
      int *so = &g.st_off[size_t(c * g.nlev + l) * (g.ntiles + 1)];
      for (int t = 0; t < g.ntiles; ++t) {
        so[t] = int(g.st_pts.size());
        const int o = (t * 5 + c) * g.nlev + l;
        for (int k = g.off[o]; k < g.off[o + 1]; ++k) {
          g.st_place[((rc[k] >> 16) - 5) * (nni - 2) + (rc[k] & 0xffff) - 5] = int(g.st_pts.size());
          g.st_pts.push_back(rc[k]);
        }
      }
      so[g.ntiles] = int(g.st_pts.size());
    }
  for (int G = 1; G <= Schedule::kBandRuns; ++G) {
    int most = 0;
    for (int t0 = 0; t0 < g.ntiles; t0 += G) {
      const int t1 = std::min(t0 + G, g.ntiles);
      most = std::max(most, g.tile_row1[t1 - 1] - g.tile_row0[t0]);
    }
    g.st_rows[G] = most + 8;
  }
  // final check: no two points of one (tile,colour,level) bucket interact,
  // and every dependency is inside a tile with a strictly larger level
  for (auto &d : deps) {
    int ra = d.first / n8, rb = d.second / n8;
    if (band_of(ra) != band_of(rb)) return "schedule check: dependency crosses a tile";
    if (!(lev[d.second] > lev[d.first])) return "schedule check: level order violated";
  }
  for (int size = 1; size <= kMaxCluster; ++size)
    for (int groups = 1; groups <= 2; ++groups) {
      ColPlan cp;
      if (column_plan(nni, nmu, size, groups, cp)) g.columns.push_back(cp);
    }
  std::string msg = build_wave_schedule(g, g.order, packed, offs, g.sor);
  if (!msg.empty()) return msg;
  build_march(g);
  std::vector<int> order, at;
  order.reserve(npts);
  at.reserve(npts);
  for (int c = 0; c < 5; ++c)
    for (int p = c; p < npts; p += 5) {
      order.push_back(g.order[p]);
      at.push_back(packed[p]);
    }
  return build_wave_schedule(g, order, at, offs, g.mcsor);
}


namespace {
struct ScheduleCache {
  std::mutex m;
  std::vector<std::shared_ptr<const Schedule>> entries;  // most recent last
};
ScheduleCache &schedule_cache() {
  static ScheduleCache c;
  return c;
}
constexpr size_t kScheduleCacheEntries = 8;
}  // namespace

std::string attach_schedule(HostGrid &g) {
  ScheduleCache &c = schedule_cache();
  {
    std::lock_guard<std::mutex> lock(c.m);
    for (auto &e : c.entries)
      if (e->nni == g.nni && e->nmu == g.nmu) {
        g.s = e;
        return "";
      }
  }
  auto made = std::make_shared<Schedule>();
  made->nni = g.nni;
  made->nmu = g.nmu;
  std::string msg = build_schedule(*made);
  if (!msg.empty()) return msg;
  g.s = made;
  std::lock_guard<std::mutex> lock(c.m);
  c.entries.push_back(std::move(made));
  if (c.entries.size() > kScheduleCacheEntries) c.entries.erase(c.entries.begin());
  return "";
}

}  // namespace x2g

// ---------------------------------------------------------------------
// CUDA-free access to the host-side tables (used by CPU tests)
// ---------------------------------------------------------------------
extern "C" int x2g_host_table(int nnu, int nmu, double r, double rinf, double z1, double z2, int which,
                              double *out) {
  x2g::HostGrid g;
  std::string msg = x2g::build_host_grid(g, nnu, nmu, r, rinf, z1, z2, 4);
  if (!msg.empty()) return X2G_ERR_ARG;
  for (int i = 0; i < nmu; ++i)
    for (int j = 0; j < nnu; ++j) {
      const int k = i * nnu + j;
      double v;
      switch (which) {
        case 0: v = g.borb_mu[i]; break;
        case 1: v = g.bpot_mu[i]; break;
        case 2: v = g.d_nu[j]; break;
        case 3: v = g.e[k]; break;
        case 4: v = g.f0[k]; break;
        case 5: v = g.f1[k]; break;
        case 6: v = g.f2[k]; break;
        case 7: v = g.f3_mu[i]; break;
        case 8: v = g.f4[k]; break;
        case 9: v = g.g[k]; break;
        case 10: v = g.wgt1[k]; break;
        case 11: v = g.wgt2[k]; break;
        default: return X2G_ERR_ARG;
      }
      out[k] = v;
    }
  return X2G_OK;
}

// Sweep order and schedule of the host grid: order[npoints] (ext indices,
// 0-based, reference list order), tile/colour/level of every point.
extern "C" int x2g_host_schedule(int nnu, int nmu, int *npoints, int *ntiles, int *nlevels, int *order,
                                 int *tile, int *colour, int *level) {
  x2g::HostGrid grid;
  std::string msg = x2g::build_host_grid(grid, nnu, nmu, 2.0, 40.0, 1.0, 1.0, 4);
  if (!msg.empty()) return X2G_ERR_SCHEDULE;
  const x2g::Schedule &g = *grid.s;
  if (npoints) *npoints = int(g.order.size());
  if (ntiles) *ntiles = g.ntiles;
  if (nlevels) *nlevels = g.nlev;
  if (order) std::copy(g.order.begin(), g.order.end(), order);
  if (tile && colour && level) {
    for (int t = 0; t < g.ntiles; ++t)
      for (int c = 0; c < 5; ++c)
        for (int l = 0; l < g.nlev; ++l) {
          const int o = (t * 5 + c) * g.nlev + l;
          for (int k = g.off[o]; k < g.off[o + 1]; ++k) {
            tile[k] = t;
            colour[k] = c;
            level[k] = l;
            order[k] = g.pts[k];
          }
        }
  }
  return X2G_OK;
}

extern "C" int x2g_host_band_schedule(int nnu, int nmu, int *npoints, int *ntiles, int *nlevels, int *pts, int *off,
                                      int *rows, int *tile_row0, int *tile_row1) {
  x2g::HostGrid grid;
  std::string msg = x2g::build_host_grid(grid, nnu, nmu, 2.0, 40.0, 1.0, 1.0, 4);
  if (!msg.empty()) return X2G_ERR_SCHEDULE;
  const x2g::Schedule &g = *grid.s;
  if (npoints) *npoints = int(g.st_pts.size());
  if (ntiles) *ntiles = g.ntiles;
  if (nlevels) *nlevels = g.nlev;
  if (pts) std::copy(g.st_pts.begin(), g.st_pts.end(), pts);
  if (off) std::copy(g.st_off.begin(), g.st_off.end(), off);
  if (rows) std::copy(g.st_rows, g.st_rows + x2g::Schedule::kBandRuns + 1, rows);
  if (tile_row0) std::copy(g.tile_row0.begin(), g.tile_row0.end(), tile_row0);
  if (tile_row1) std::copy(g.tile_row1.begin(), g.tile_row1.end(), tile_row1);
  return X2G_OK;
}

// Schedule of the list-order SOR wavefront (host only): interior points by
// SOR level, packed (ext row << 16) | ext col (pts, npoints values; off,
// nlev + 1 offsets), axis points by the level their extrapolation follows
// (bpts; boff, nblev + 1 offsets), and the level shift between sweeps.
// Null arrays: counts only.
extern "C" int x2g_host_sor_schedule(int nnu, int nmu, int *npoints, int *nlev, int *nblev, int *delta, int *pts,
                                     int *off, int *bpts, int *boff) {
  x2g::HostGrid grid;
  std::string msg = x2g::build_host_grid(grid, nnu, nmu, 2.0, 40.0, 1.0, 1.0, 4);
  if (!msg.empty()) return X2G_ERR_SCHEDULE;
  const x2g::Schedule &g = *grid.s;
  if (npoints) *npoints = int(g.sor.pts.size() / 2);
  if (nlev) *nlev = g.sor.nlev;
  if (nblev) *nblev = g.sor.nblev;
  if (delta) *delta = g.sor.delta;
  for (size_t k = 0; pts && k < g.sor.pts.size() / 2; ++k) pts[k] = g.sor.pts[2 * k];
  if (off) std::copy(g.sor.off.begin(), g.sor.off.end(), off);
  if (bpts) std::copy(g.sor.bpts.begin(), g.sor.bpts.end(), bpts);
  if (boff) std::copy(g.sor.boff.begin(), g.sor.boff.end(), boff);
  return X2G_OK;
}
