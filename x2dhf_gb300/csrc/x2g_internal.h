// Internal structures of the x2dhf GB300 relaxation library.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <memory>
#include <mutex>
#include <vector>

#include "../../include/x2dhf_gpu.h"

#include "x2g_pairs.cuh"

namespace x2g {

constexpr double kPrecis = 2.220446049250313080847263336181640625e-16;  // epsilon(1d0), initVariables.F90:397
constexpr double kPi = 3.14159265358979323846264338327950;                // params.F90:94
constexpr int kMaxLevels = 8;
// device words of a context's barrier state: [0] arrivals, [1] generation,
// [2] error word, [3] reduction ticket, then the tickets of the batched
// moment reductions from word 288 (kMomentItems), then the persistent
// sweep's per-block phase counts from word kPhaseWords (kPhaseBlocks, one
// 128-byte line each)
constexpr int kMomentTickets = 288;
constexpr int kPhaseWords = 352, kPhaseBlocks = 320, kPhaseStride = 32;
constexpr int kBarWords = kPhaseWords + kPhaseBlocks * kPhaseStride;

// ----------------------------------------------------------------------
// A sequential sweep over a list of points as a pipelined wavefront: an
// interior point's level is 1 + the largest level of its stencil neighbours
// earlier in the list (their new values are read), an axis point's level 1 +
// the largest level of the points its extrapolation reads (the corners read
// the mu=1 row); sweep s of a point runs at step level + s * delta.  pts /
// bpts hold the interior / axis points by level, packed (ext row << 16) | ext
// col, with offsets off[nlev + 1] / boff[nblev + 1].
// ----------------------------------------------------------------------
struct WaveHost {
  int nlev = 0, nblev = 0, delta = 0;
  // pts: interior points as pairs (packed point, mask); mask: the stencil
  // neighbours earlier in the list, bit 4 (k-1) + {0: -k, 1: +k, 2: -k rows, 3:
  // +k rows}; bits 16..18: the point is the fifth of the extrapolation of the
  // mu=1 row, nu=1 or nu=nni column
  std::vector<int> pts, off, bpts, boff;
};

// ----------------------------------------------------------------------
// Bands of the on-chip FP32 sweep (k_columns) for clusters of `size` CTAs:
// CTA k owns ext rows [row0[k], row0[k+1]) of the interior rows 5..nmu-1.
// With two threads per column (groups 2) a band is cut before its row cut[k].
// The row seam lies inside one thread's rows; slots is the most points of one
// colour in a thread's rows, pitch the row pitch in words (a multiple of 32),
// warps those of a group, shift the lanes before the first column that keep
// the column seam inside one warp.
// ----------------------------------------------------------------------
constexpr int kMaxCluster = 16;
struct ColPlan {
  int size, groups, maxrows, slots, pitch, warps, shift;
  // set for the launch: the rows the kernel's arrays hold, the FP32 stencil
  // weights as (mu, nu) pairs, (-1, -1), and those along mu as (dmu1, -dmu1)
  // and (dmu2, dmu2)
  int rows;
  float2 c2[4], c1[4], neg, m1[4], m2[4];
  int row0[kMaxCluster + 1], cut[kMaxCluster];
};

// ----------------------------------------------------------------------
// What the sweeps of a grid size follow: depends on N_nu and N_mu only, and is
// shared by the grids of a size (attach_schedule).
// ----------------------------------------------------------------------
struct Schedule {
  int nni = 0, nmu = 0, n8 = 0, next = 0;
  // "middle" ordering of interior points (ext indices, reference list order)
  std::vector<int> order;
  // sweep schedule: tiles = bands of ext rows [row0,row1)
  int ntiles = 0, nlev = 0;
  std::vector<int> tile_row0, tile_row1;
  std::vector<int> pts;  // ext indices grouped [tile][colour][level]
  std::vector<int> off;  // (ntiles*5*nlev + 1) offsets into pts
  // persistent-band FP32 sweep of grids beyond one cluster: the same points
  // regrouped [colour][level][tile] (st_pts, packed (ext row << 16) | ext
  // col), so that the points of one colour and level in any run of
  // consecutive tiles are one contiguous range; st_off[(c * nlev + l) *
  // (ntiles + 1) + t] is the start of tile t.  st_rows[G] = most rows of any
  // run of G consecutive tiles plus the 4-row halos on both sides (G =
  // 1..kBandRuns)
  static constexpr int kBandRuns = 16;
  std::vector<int> st_pts, st_off;
  // the place of interior point (mu, nu) in st_pts, (nni - 2) (mu - 1) + nu - 1
  std::vector<int> st_place;
  int st_rows[kBandRuns + 1] = {};
  // bands of the on-chip FP32 sweep, by cluster size and threads per column
  std::vector<ColPlan> columns;
  // SOR's points of ext rows 4..nmu-1 (4: the mu=1 axis) by row and side of
  // the middle column, in list order: row r's left (right) points are entries
  // [march_off[2(r-4)], march_off[2(r-4)+1]) (then up to march_off[2(r-4)+2])
  // of march_pts, pairs of the ext index and a mask (sor's, kMarchAxis... for
  // axis points and the stride to what they read); a side ends with its axis
  // point
  std::vector<int> march_pts, march_off;
  // the FP64 sweeps' wavefront schedules (build_wave_schedule): list-order
  // SOR over the "middle" list (sor, sormcsor.F90:20-132), and MCSOR as the
  // same sweep over the list colour after colour (mcsor, :143-386)
  WaveHost sor, mcsor;
};

// ----------------------------------------------------------------------
// Host-side grid: every table the relaxation path reads, built with the
// reference's formulas (initCBAllocArrays.F90 initCBlocks:813-858,
// initSuppl:1636-2051).  Indices are 0-based: nu j in [0,nni), mu i in
// [0,nmu); plain index i*nni+j; extended index (i+4)*n8+(j+4).
// ----------------------------------------------------------------------
struct HostGrid {
  int nni = 0, nmu = 0, n8 = 0, m8 = 0, next = 0, mxsize = 0, mpole = 4;
  double r = 0, r2 = 0, z1 = 0, z2 = 0, rinf = 0, hni = 0, hmu = 0, diag = 0;
  std::vector<double> vxi, vxisq, vxi1, vxi2, veta, vetasq, veta1, veta2, wmu, wni;
  double dmu1[4], dmu2[4], dni1[4], dni2[4], exeven[5];
  std::vector<double> dmu9, dni9;              // 9-point derivative weights (diffmu/diffnu)
  std::vector<double> borb_mu, bpot_mu, f3_mu;  // mu-only coefficient tables
  // the two axis terms of e = e_mu(mu) - e_nu(nu) (e_mu = -1/(xi^2-1),
  // e_nu = 1/(1-eta^2), 0 on the nu axis points, where e is 0)
  std::vector<double> e_mu, e_nu;
  std::vector<double> d_nu;                     // nu-only
  std::vector<double> e, f0, f1, f2, f4, g, wgt1, wgt2;  // plain 2-D tables
  std::vector<double> leg;                      // mpole tables P_k(cos th) r^k, plain
  std::shared_ptr<const Schedule> s;            // of this grid size
};

std::string build_host_grid(HostGrid &g, int nni, int nmu, double r, double rinf, double z1, double z2, int mpole);

// ----------------------------------------------------------------------
// Wavefront schedule on the device: interior points by level ((ext row << 16)
// | ext col, and the bits of the neighbours earlier in the list) and axis
// points by level, with their offsets.
// ----------------------------------------------------------------------
struct WaveDev {
  const int2 *pts;
  const int *off, *bpts, *boff;
  int nlev, nblev, delta;
};

// SOR's points by row and side (Schedule::march_pts): (ext index, mask)
struct MarchDev {
  const int2 *pts;
  const int *off;
};
constexpr unsigned kMarchAxisMu = 1u << 20, kMarchAxisUp = 1u << 21, kMarchAxisDown = 1u << 22;
constexpr unsigned kMarchAxis = kMarchAxisMu | kMarchAxisUp | kMarchAxisDown;

// ----------------------------------------------------------------------
// Device view of a grid, passed by value to kernels.
// ----------------------------------------------------------------------
struct GridDev {
  int nni, nmu, n8, m8, next, mxsize, ntiles, nlev, mpole;
  double r2;
  double dmu1[4], dmu2[4], dni1[4], dni2[4], exeven[5], diag;
  PairCoef pmu2[4], pmu1[4], pnu2[4], pnu1[4];  // dmu2, dmu1, dni2, dni1 as factors of pair_products
  bool pairs;                                   // all of them are of moderate size
  const double *borb_mu, *bpot_mu, *f3_mu, *d_nu;
  const double *e, *f0, *f1, *f2, *f4, *g, *wgt1, *wgt2, *leg;
  const double *wf;  // wgt2 f4: the weight of the orbital inner products (Gram-matrix orthonormalisation)
  const double *dmu9, *dni9;
  const double *vxi, *vxisq, *veta, *vetasq;
  const int *tile_row0, *tile_row1, *pts, *off;
  const int *st_pts, *st_off;
  int st_rows[17];
  WaveDev sor, mcsor;
  MarchDev march;
  // FP32 copies of the coefficient tables for the mixed form
  const float *borb_mu32, *bpot_mu32, *d_nu32;
  const double *e_mu, *e_nu;
  // separable stencil weights of the mixed form's FP64 residual: for the
  // neighbours at distance 4,3,2,1 before and after the point, cmu_*[mu * 8 +
  // q] = dmu2 + b dmu1 (q < 4, before) and dmu2 - b dmu1 (q >= 4, after) with
  // b = borb or bpot; cnu[nu * 8 + q] likewise with dni2, d(nu), dni1
  const double *cmu_orb, *cmu_pot, *cnu;
  // the same as fixed-point numbers w 2^wscale = .x 2^29 + .y with |.x| <=
  // 2^28, |.y| <= 2^28, and the place of interior point (mu, nu) in st_pts
  // (potentials)
  const int2 *wmu_pot, *wnu;
  int wscale;
  // a value of u whose exponent is at most this far below its tile's largest
  // makes lhs u at least 2^-4 of the largest weight times that value
  int near;
  const int *st_place;
  // per-grid moment tables (built on the device at grid creation):
  // exm[(idel * 8 + q) * mxsize + k] = wgt2 f4 P_{q+1}^idel(cos th) (r2 r)^(q+1)
  // for idel 0..4, q < mpole; asy[slot * 4 nni + p] on the 4 boundary rows
  // (p = row * nni + nu): slot 0 r2 xi, 1 1/(r2 r), 2+m-1 P_m(cos th)
  // (r2 r)^-(m+1) for m = 1..8, 10 + idel * 8 + m-1 the exchange functions
  // P_m^idel(cos th) (r2 r)^-(m+1), 50 orbAsymptGet's raiq(mu-1) - raiq(mu)
  const double *exm, *asy;
  // FP32 stencil weights, rounded on the host: GB300 issues double->float
  // conversions on its narrow FP64 pipe, so the FP32 kernels never convert
  float dmu1f[4], dmu2f[4], dni1f[4], dni2f[4], exevenf[5];
};

// Device job (one function to relax), built from x2g_job.
struct JobDev {
  double *u;
  const double *lhs;
  const double *rhs;
  const double *psa, *psb;
  union {
    double *rhs_buf;  // FP64: materialised rhs of a potential
    double *pairs;    // wavefront: (lhs, rhs) by plain index
  };
  union {
    float *e32;          // mixed: FP32 extended correction
    ulonglong2 *tagged;  // wavefront: (value, sweeps done) by ext index
  };
  float *r32, *w32; // mixed: FP32 residual and omega / diagonal
  float2 *rw;       // mixed, persistent-band sweep: (residual, omega / diagonal) in st_pts order
  double omega;
  double idel2;
  float omegaf, omega1f;  // omega and 1 - omega rounded to FP32 on the host
  int isym, kind;
};

// Jobs of one relaxation launch, passed by value as a kernel parameter
// (__grid_constant__): no host-to-device copy per call.  Larger batches are
// split into launches of kParamJobs.
constexpr int kParamJobs = 32;
struct JobTable {
  JobDev j[kParamJobs];
};

// Grid barrier state in device memory.  The error word is sticky: a
// launch that finds it set leaves at its first wait, and only the host's
// readback (x2g_synchronize) clears it, so an error of one launch of a
// multi-launch call survives the launches after it.
struct BarrierDev {
  unsigned int *count;
  unsigned int *gen;
  int *err;                     // first error code (0 = none)
  unsigned long long limit_ns;  // longest wait of one block; 0: a wait not met at its first check fails
};

constexpr unsigned long long kDefaultWaitLimitNs = 2000000000ull;  // 2 s

}  // namespace x2g

struct x2g_ctx {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;  // highest priority
  cudaStream_t aux = nullptr;     // lowest priority, joined back into stream by events
  cudaEvent_t ev_split[2] = {nullptr, nullptr};
  int residual_overlap = 1;       // potential batches in two waves: the second wave's residual under the first's sweep
  // barrier words + error flag (4 ints)
  unsigned int *bar = nullptr;
  // reusable device workspace
  void *work = nullptr;
  size_t work_bytes = 0;
  std::mutex host_call;         // held by a call on host arrays, which shares the next two
  void *host_arrays = nullptr;  // device copies of a host call's arrays
  size_t host_arrays_bytes = 0;
  void *red = nullptr;  // reduction partials
  size_t red_bytes = 0;
  double *host_red = nullptr;  // pinned host buffer for small readbacks
  long long h2d_bytes = 0, d2h_bytes = 0;  // host<->device bytes copied by the library
  long launches = 0;
  int cluster_smem = -1;        // largest dynamic shared memory of a cluster sweep CTA (0: none)
  int no_cluster = 0;           // 1: mixed form uses the persistent-band FP32 kernel
  int auto_band = 0;            // 1: batches beyond the co-resident clusters take the persistent-band kernel
  int pot_clusters = 2;         // potentials' cluster variant: 0 never, 1 always, 2 batches beyond the plain kernel's clusters
  int mixed_free = 0;           // cluster sweep colouring: 0 the reference's list order mod 5, 1 seam-free
  // kernels of the cluster sweep that run a grid size's band plans here
  struct ColumnShape {
    int plan;  // place in Schedule::columns
    const void *fn;
    bool sep;
    int rows;
    size_t smem;
    int active;  // co-resident clusters
  };
  struct ColumnShapes {
    int nni, nmu;
    std::vector<ColumnShape> shapes;
  };
  std::vector<ColumnShapes> columns;
  int band_attr = 0;            // shared memory cap granted to the persistent-band sweep
  long band_key = -1;           // shared bytes of its last occupancy query
  int band_blocks = 0;          // co-resident blocks for that size
  int band_sm_smem = 0;         // shared memory per SM
  int f64_blocks = -1;          // co-resident blocks of the cooperative FP64 sweep on this device
  int march_smem = -1;          // shared memory that a block of the marching SOR sweep may have (0: it cannot run)
  int wave_ok = -1;             // the wavefront kernels can be co-resident, one block per SM
  int ortho_blocks = -1;        // co-resident blocks of the one-launch orthonormalisation
  int gram_blocks = -1;         // co-resident blocks of its Gram-matrix form
  int gram_ortho = 0;           // batch mode 2: orthonormalise in rounds (0) or through the Gram matrix (1)
  unsigned long long wait_limit_ns = x2g::kDefaultWaitLimitNs;  // device-side wait limit (x2g_set_wait_limit)
  // optional per-launch timing of the sweep kernels (CUDA events on stream)
  int profiling = 0;
  struct Pending {
    cudaEvent_t a, b;
    int precision;
    double points;  // point-updates performed by the launch
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> event_pool;
  double prof_ms[2] = {0, 0};      // FP64, mixed (FP32 sweep kernel only)
  double prof_points[2] = {0, 0};
  long prof_launches[2] = {0, 0};
};

struct x2g_grid {
  x2g_ctx *ctx = nullptr;
  x2g::HostGrid h;
  x2g::GridDev d{};
  std::vector<void *> allocs;
};

namespace x2g {
// status helpers (x2g_capi.cu)
int set_status(int code, const std::string &msg);
int cuda_status(cudaError_t e, const char *where);
void *ctx_workspace(x2g_ctx *ctx, size_t bytes);
inline void count_copy(x2g_ctx *ctx, size_t h2d, size_t d2h) {
  if (ctx) {
    ctx->h2d_bytes += (long long)h2d;
    ctx->d2h_bytes += (long long)d2h;
  }
}
}  // namespace x2g
