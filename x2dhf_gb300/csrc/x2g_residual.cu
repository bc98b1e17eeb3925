// FP64 residuals of the mixed form.
#include "x2g_device.cuh"
#include "x2g_kernels.cuh"

namespace x2g {

namespace {

constexpr int kThreads = 256;

// r = rhs - A u of an interior point in FP64, and its lhs; the stencil uses the
// grid's separable weights (one FMA per neighbour) and reads the ghost cells as
// mirrored interior values, so u needs no ghost refresh first
__device__ __forceinline__ double residual_at(const GridDev &g, const JobDev &J, int mu, int nu, double &lhs) {
  const int n8 = g.n8, ik = mu * g.nni + nu, ij = (mu + 4) * n8 + nu + 4;
  const double *u = J.u;
  double rhs;
  if (J.kind == 1) {
    rhs = (J.psa[ij] * J.psb[ij]) * g.g[ik];
    lhs = (J.idel2 == 0.0) ? g.f3_mu[mu] : fma(J.idel2, g.e[ik], g.f3_mu[mu]);
  } else {
    rhs = J.rhs[ik];
    lhs = J.lhs[ik];
  }
  const double *cm = (J.kind == 0 ? g.cmu_orb : g.cmu_pot) + mu * 8, *cn = g.cnu + nu * 8;
  double cc = lhs * u[ij];
  if (mu >= 4 && nu >= 4 && nu <= g.nni - 5) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int dm = (4 - q) * n8, dn = 4 - q;
      cc = fma(cm[q], u[ij - dm], cc);
      cc = fma(cm[4 + q], u[ij + dm], cc);
      cc = fma(cn[q], u[ij - dn], cc);
      cc = fma(cn[4 + q], u[ij + dn], cc);
    }
  } else {
    // the stencil reaches the putin ghosts
    const int row = mu + 4, col = nu + 4;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int d = 4 - q;
      cc = fma(cm[q], ghost_read(g, u, row - d, col, J.isym), cc);
      cc = fma(cm[4 + q], u[ij + d * n8], cc);
      cc = fma(cn[q], ghost_read(g, u, row, col - d, J.isym), cc);
      cc = fma(cn[4 + q], ghost_read(g, u, row, col + d, J.isym), cc);
    }
  }
  return rhs - cc;
}

// Mixed form residual over the interior, stored as FP32 with omega / lhs.
// kPacked: the points are taken in st_pts order and stored as (r, w) pairs in
// that order (persistent-band sweep); otherwise r32 / w32 are plain nni x nmu
// arrays (cluster sweep; need_w 0: the potentials' cluster sweep forms omega /
// lhs itself, only r32 is stored).
template <bool kPacked>
__global__ void k_residual(GridDev g, const __grid_constant__ JobTable jobs, int zero_e, int need_w) {
  const JobDev &J = jobs.j[blockIdx.y];
  const int nint = (g.nni - 2) * (g.nmu - 5);
  if (zero_e)
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.next; k += gridDim.x * blockDim.x) J.e32[k] = 0.0f;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nint; k += gridDim.x * blockDim.x) {
    int mu, nu;
    if (kPacked) {
      const int rc = g.st_pts[k];
      mu = (rc >> 16) - 4;
      nu = (rc & 0xffff) - 4;
    } else {
      mu = 1 + k / (g.nni - 2);
      nu = 1 + k % (g.nni - 2);
    }
    double lhs;
    const double r = residual_at(g, J, mu, nu, lhs);
    if (kPacked) {
      J.rw[k] = make_float2(narrow_f64(r), J.omegaf / narrow_f64(lhs));
    } else {
      const int ik = mu * g.nni + nu;
      J.r32[ik] = narrow_f64(r);
      if (need_w) J.w32[ik] = J.omegaf / narrow_f64(lhs);
    }
  }
}

// The residual of potentials built from orbitals with its stencil sum in fixed
// point on the integer pipes: a warp's FP64 instruction takes the SM 19 cycles,
// a 32-bit product with a 64-bit sum one, and 16 of a point's 20 FP64
// operations are the neighbours' FMAs.
//
// A block takes a tile of 32 x 32 points.  Its values of u become whole numbers
// of 60 bits in units of the largest one's last bits, two signed halves each
// (mirrored and negated where they are ghosts), the weights are halves of 58
// bits from the host; a product is high x high and the two mixed products, each
// summed exactly in 64 bits (what the two low halves would add is 2^-57 of the
// largest product).  rhs - lhs u, formed in FP64, is rounded to the sum's
// units, and their difference rounded once, to FP32.  Every rounding is to
// nearest: truncated values shift the sums by a constant sign, and SCFs then
// stall at their noise floor.
//
// All of this is in units of the tile's largest value and of the grid's largest
// weight, W (about 2^-58 of their product in all), where the FMAs round to 53
// bits of what a point's own terms come to.  So a point keeps the sum where its
// term lhs u alone is within 2^-4 of W times the tile's largest value (|lhs| is
// never below the diagonal's, so that u's exponent tells): there the error is no
// larger than the FMAs', root mean square and worst, in terms of the point's
// largest product (smooth potentials 4.7e-17 and 2e-16 against 1.8e-16 and
// 9e-16, points at the limit 9e-17 against 1.8e-16).  The others, values that do
// not fit the units, and tiles at the ends of the exponent range are collected
// and summed by FMAs, 32 at a time, the same as k_residual's bits (smooth
// potentials of sigma pairs: none; of pi pairs, small near the axis, 4 % of the
// points of 331 x 481 and 15 % of 151 x 241, that lie in 20 and 44 % of a warp's
// rows).
//
// What bounds it: waiting (issue in two cycles of five, the FP64 pipe 39 % busy):
// for the tile and the orbitals, then for the products one after the other, about
// 300 instructions a point of which 96 are the products (two each); 8 rows per
// warp share the column's weights and its values.  22 potentials of 331 x 481: 75
// us in an SCF, 90 with a third of them of azimuthal number 2; with FMAs 149.
constexpr int kTile = 32;           // columns and rows of a block's tile
constexpr int kSpan = kTile + 8;    // with the stencil's four on each side
constexpr int kRowsPerWarp = 8;
constexpr int kThreadsRes = kTile / kRowsPerWarp * 32;
constexpr int kBlocksRes = 5;
constexpr int kWarpSpan = kSpan / (kThreadsRes / 32);        // rows of the tile that a warp loads
constexpr int kValues = kWarpSpan + (kWarpSpan + 3) / 4;  // values that a thread loads

// x 2^(1081 - top), rounded, as .x 2^29 + .y with |.x| <= 2^30, |.y| <= 2^28;
// top: the largest exponent field of the tile; flip: sign bit to change
__device__ __forceinline__ int2 to_fixed(double x, int top, unsigned flip) {
  const unsigned hi = unsigned(__double2hiint(x)), lo = unsigned(__double2loint(x));
  const int ex = int((hi >> 20) & 0x7ffu), s = top - ex;
  // one bit more than is kept
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 7;
  m >>= min(s, 63);  // (no such bits are left: zeros and subnormals are far below the tile's largest)
  const int h = int((m + (1ull << 29)) >> 30), l = int(unsigned(m) - (unsigned(h) << 30) + 1) >> 1;
  return int(hi ^ flip) < 0 ? make_int2(-h, -l) : make_int2(h, l);
}

// x / 2^(unit - 1075), rounded to a whole number, |x| < 2^(unit - 1014)
__device__ __forceinline__ long long to_units(double x, int unit) {
  const unsigned hi = unsigned(__double2hiint(x)), lo = unsigned(__double2loint(x));
  const int ex = int((hi >> 20) & 0x7ffu), s = unit + 10 - ex;
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;
  m = ((m >> min(max(s - 1, 0), 63)) + 1) >> 1;
  return (int(hi) < 0) ? -(long long)m : (long long)m;
}

// v 2^(unit - 1075) as a float, rounded to nearest even; infinite above its
// range, zero below its normal range
__device__ __forceinline__ float from_units(long long v, int unit) {
  const unsigned long long a = v < 0 ? (unsigned long long)-v : (unsigned long long)v;
  const int lz = __clzll((long long)a) & 63;
  const unsigned long long m = a << lz;  // the top bit set
  const unsigned top = unsigned(m >> 32), low = unsigned(m) != 0;
  // 24 bits and the eight below them, the last one sticky
  const unsigned f = (top >> 8) + (((top & 0xffu) | low) + ((top >> 8) & 1u) > 0x80u ? 1u : 0u);
  const int ex = unit - 1075 + 63 - lz + 127;  // biased
  unsigned bits = (unsigned(ex - 1) << 23) + f;
  bits = ex >= 255 ? 0x7f800000u : bits;
  bits = (ex < 1 || a == 0) ? 0u : bits;
  return __uint_as_float(bits | (unsigned(v >> 32) & 0x80000000u));
}

struct Acc {
  long long a, b;  // sums of products high x high, and high x low
  __device__ __forceinline__ void add(int2 w, int2 u) {
    a += (long long)w.x * u.x;
    b += (long long)w.x * u.y;
    b += (long long)w.y * u.x;
  }
};

__device__ __noinline__ float residual_fma(const GridDev &g, const JobDev &J, int mu, int nu) {
  double lhs;
  return narrow_f64(residual_at(g, J, mu, nu, lhs));
}

// x at a byte offset: one 32-bit offset serves arrays of one layout
template <class T>
__device__ __forceinline__ T at(const T *x, unsigned bytes) {
  return __ldg(reinterpret_cast<const T *>(reinterpret_cast<const char *>(x) + bytes));
}

template <bool kPacked>
__global__ void __launch_bounds__(kThreadsRes, kBlocksRes)
    k_residual_fixed(GridDev g, const __grid_constant__ JobTable jobs, int across, int need_w) {
  const JobDev &J = jobs.j[blockIdx.y];
  __shared__ int2 tile[kSpan * kSpan];
  __shared__ int4 s_wmu[kTile * 4];
  __shared__ unsigned s_near[kSpan];
  __shared__ int s_top[kThreadsRes / 32];
  __shared__ unsigned char s_rest[kThreadsRes / 32][kRowsPerWarp * 32];  // a warp's points that are left to FMAs
  const int tid = int(threadIdx.x), lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int down = int(blockIdx.x) / across;
  const int mu0 = down * kTile + 1, nu0 = (int(blockIdx.x) - down * across) * kTile + 1;
  const int n8 = g.n8, nni = g.nni, isym = J.isym;
  const double *const __restrict__ u = J.u;
  if (kPacked)
    for (int k = blockIdx.x * kThreadsRes + tid; k < g.next; k += gridDim.x * kThreadsRes) J.e32[k] = 0.0f;
  // the tile: rows mu0 - 4 .. mu0 + 35, columns nu0 - 4 .. nu0 + 35; a warp
  // takes ten rows, lanes 32 columns and then the last eight of four rows at a
  // time (beyond the array the last row or column again: no point reads them)
  auto column = [&](int col, unsigned &flip) {
    col = min(col, nni + 6);
    const bool mirror = col < 4 || col > nni + 3;
    flip = mirror && isym != 1 ? 0x80000000u : 0u;
    return col < 4 ? 8 - col : col > nni + 3 ? 2 * nni + 6 - col : col;
  };
  auto row = [&](int r, unsigned &flip) {
    r = min(r, g.nmu + 3);
    flip = r < 4 && isym != 1 ? 0x80000000u : 0u;
    return r < 4 ? 8 - r : r;
  };
  unsigned flip_a, flip_b;
  const int col_a = column(nu0 + lane, flip_a), col_b = column(nu0 + 32 + (lane & 7), flip_b);
  double x[kValues];
#pragma unroll
  for (int q = 0; q < kValues; ++q) {
    const int i = q < kWarpSpan ? q : min((lane >> 3) + 4 * (q - kWarpSpan), kWarpSpan - 1);
    unsigned f;
    x[q] = at(u, 8u * unsigned(row(mu0 + warp * kWarpSpan + i, f) * n8 + (q < kWarpSpan ? col_a : col_b)));
  }
  // rhs - lhs u of the warp's points
  const int nu = nu0 + lane, mu1 = mu0 + warp * kRowsPerWarp, rows = min(kRowsPerWarp, g.nmu - 4 - mu1);
  const bool in = nu <= nni - 2;
  const int nuc = in ? nu : nni - 2;
  const unsigned at_ext = 8u * unsigned((mu1 + 4) * n8 + nuc + 4), at_int = 8u * unsigned(mu1 * nni + nuc);
  double rest[kRowsPerWarp];
  float w32[kRowsPerWarp];  // kPacked: omega / lhs
  {
    const double idel2 = J.idel2;
    const bool plain = __double2hiint(idel2) == 0;
    const double *const __restrict__ psa = J.psa, *const __restrict__ psb = J.psb;
#pragma unroll
    for (int q = 0; q < kRowsPerWarp; ++q) {
      // (a short warp's last rows again)
      const int qr = min(q, rows - 1);
      const unsigned e = at_ext + unsigned(qr * 8) * n8, k = at_int + unsigned(qr * 8) * nni;
      double lhs = rows > 0 ? __ldg(g.f3_mu + mu1 + qr) : 0.0;
      if (rows > 0) {
        if (!plain) lhs = fma(idel2, at(g.e, k), lhs);
        rest[q] = fma(-lhs, at(u, e), (at(psa, e) * at(psb, e)) * at(g.g, k));
        if (kPacked)
          w32[q] = J.omegaf / narrow_f64(lhs);
        else if (need_w && in && q < rows)
          J.w32[(mu1 + q) * nni + nu] = J.omegaf / narrow_f64(lhs);
      }
    }
  }
  s_wmu[tid] = __ldg(reinterpret_cast<const int4 *>(g.wmu_pot) + min(mu0 * 4 + tid, g.nmu * 4 - 1));
  int top = 0;
#pragma unroll
  for (int q = 0; q < kValues; ++q) top = max(top, __double2hiint(x[q]) & 0x7fffffff);
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) s_top[warp] = top;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreadsRes / 32; ++w) top = max(top, s_top[w]);
  const bool zero = top == 0;
  top >>= 20;
  // out of reach of the fixed point's exponents: infinities, NaNs and tiles
  // at the ends of the range go point by point
  const bool far = top < 256 || top > 1792;
  const int low = far ? 0x7fffffff : (top - g.near) << 20;
  unsigned near = 0, edge = 0;
#pragma unroll
  for (int q = 0; q < kValues; ++q) {
    const int i = q < kWarpSpan ? q : min((lane >> 3) + 4 * (q - kWarpSpan), kWarpSpan - 1);
    unsigned f;
    row(mu0 + warp * kWarpSpan + i, f);
    f |= q < kWarpSpan ? flip_a : flip_b;
    tile[(warp * kWarpSpan + i) * kSpan + (q < kWarpSpan ? lane : 32 + (lane & 7))] = to_fixed(x[q], top, f);
    const unsigned w = __ballot_sync(0xffffffffu, (__double2hiint(x[q]) & 0x7fffffff) >= low);
    if (q < kWarpSpan)
      near = lane == q ? w : near;
    else
      edge = (lane >> 2) == q - kWarpSpan ? w >> 8 * (lane & 3) & 0xffu : edge;
  }
  // lane i's row of the tile: near values in columns 4..35
  if (lane < kWarpSpan) s_near[warp * kWarpSpan + lane] = __funnelshift_r(near, edge, 4);
  __syncthreads();
  if (rows <= 0) return;
  int left = 0;
  int2 wn[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) wn[q] = at(g.wnu, unsigned(nuc * 64 + q * 8));
  const int2 *const t = tile + warp * kRowsPerWarp * kSpan + lane + 4;
  const int unit = top - g.wscale + 52;  // a unit of the products' sum is 2^(unit - 1075)
  int2 c[kRowsPerWarp + 8];              // the column's values
#pragma unroll
  for (int q = 0; q < 8; ++q) c[q] = t[q * kSpan];
#pragma unroll
  for (int q = 0; q < kRowsPerWarp; ++q) {
    c[q + 8] = t[(q + 8) * kSpan];
    const int2 *const h = t + (q + 4) * kSpan;
    Acc s{0, 0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      // wmu: distances 4, 3, 2, 1 before the point, then 4, 3, 2, 1 after it
      const int4 w = s_wmu[(warp * kRowsPerWarp + q) * 4 + k];
      s.add(make_int2(w.x, w.y), c[q + (k < 2 ? 2 * k : 12 - 2 * k)]);
      s.add(make_int2(w.z, w.w), c[q + (k < 2 ? 2 * k + 1 : 11 - 2 * k)]);
      s.add(wn[k], h[k - 4]);
      s.add(wn[4 + k], h[4 - k]);
    }
    const long long sum = s.a + ((s.b + (1ll << 28)) >> 29);
    float r = from_units(to_units(rest[q], unit) - sum, unit);
    if (zero) r = narrow_f64(rest[q]);
    // rest beyond the tile's units
    const bool large = ((unsigned(__double2hiint(rest[q])) >> 20) & 0x7ffu) > unsigned(unit + 8);
    const bool keep = zero || ((s_near[warp * kRowsPerWarp + q + 4] >> lane & 1u) != 0 && !large), on = in && q < rows;
    const unsigned others = __ballot_sync(0xffffffffu, on && !keep);
    if (others >> lane & 1u) s_rest[warp][left + __popc(others & ((1u << lane) - 1))] = (unsigned char)(q * 32 + lane);
    left += __popc(others);
    if (kPacked) {
      float2 *const to = J.rw + __ldg(g.st_place + (mu1 + min(q, rows - 1) - 1) * (nni - 2) + nuc - 1);
      if (on && keep) *to = make_float2(r, w32[q]);
      if (on && !keep) to->y = w32[q];
    } else if (on && keep) {
      J.r32[(mu1 + q) * nni + nu] = r;
    }
  }
  __syncwarp();
  for (int k = lane; k < left; k += 32) {
    const int id = s_rest[warp][k], mu = mu1 + id / 32, at_nu = nu0 + id % 32;
    const float r = residual_fma(g, J, mu, at_nu);
    if (kPacked)
      J.rw[__ldg(g.st_place + (mu - 1) * (nni - 2) + at_nu - 1)].x = r;
    else
      J.r32[mu * nni + at_nu] = r;
  }
}

}  // namespace

void launch_residual(const GridDev &g, const JobTable &jobs, int njobs, bool fixed, bool packed, bool need_w,
                     cudaStream_t s) {
  if (!fixed) {
    const int want = ((g.nni - 2) * (g.nmu - 5) + kThreads - 1) / kThreads;
    const dim3 grid(unsigned(want < 1184 ? want : 1184), unsigned(njobs));
    if (packed)
      k_residual<true><<<grid, kThreads, 0, s>>>(g, jobs, 1, 1);
    else
      k_residual<false><<<grid, kThreads, 0, s>>>(g, jobs, 0, need_w);
    return;
  }
  const int across = (g.nni - 2 + kTile - 1) / kTile, down = (g.nmu - 5 + kTile - 1) / kTile;
  const dim3 grid(unsigned(across * down), unsigned(njobs));
  if (packed)
    k_residual_fixed<true><<<grid, kThreadsRes, 0, s>>>(g, jobs, across, 1);
  else
    k_residual_fixed<false><<<grid, kThreadsRes, 0, s>>>(g, jobs, across, need_w);
}

}  // namespace x2g
