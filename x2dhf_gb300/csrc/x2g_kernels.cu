// CUDA kernels of the x2dhf GB300 relaxation library (sm_103a).
//
// Layout: every function lives in the reference's extended layout
// ((nni+8) x (nmu+8) doubles, nu fastest), so putin reduces to a ghost
// refresh and putout to nothing.  Plain 2-D tables are nni x nmu.
//
// FP64 arithmetic that must reproduce the reference bit for bit is written
// with __dadd_rn/__dmul_rn/__ddiv_rn, which the compiler never contracts
// into FMAs (the reference was built without FMA contraction).
#include <algorithm>
#include <cooperative_groups.h>
#include <cstdio>
#include <vector>

#include "x2g_columns.cuh"
#include "x2g_columns_plan.h"
#include "x2g_pairs.cuh"

namespace x2g {

namespace {

constexpr int kThreads = 256;
constexpr int kBandThreads = 512;

__device__ __forceinline__ double A(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double S(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double M(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double D(double a, double b) { return __ddiv_rn(a, b); }

template <typename T>
__device__ __forceinline__ T ldcg(const T *p) {
  return __ldcg(p);
}

// Whether a wait that started at t0 has run out: checked every 256 spins,
// or at every spin when the limit is 0 (a wait not met at once fails).
__device__ __forceinline__ bool wait_expired(const BarrierDev &b, unsigned spins, unsigned long long t0) {
  return (b.limit_ns == 0 || (spins & 255u) == 0) && globaltimer() - t0 >= b.limit_ns;
}

// Grid-wide barrier for a cooperative launch.  Every wait is bounded: after
// b.limit_ns the block records X2G_ERR_TIMEOUT and all blocks leave the
// kernel at their next barrier; a launch that finds the error word already
// set leaves at its first barrier.  Returns false when the kernel must stop.
__device__ bool grid_barrier(const BarrierDev &b, unsigned nblocks) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    volatile unsigned *vgen = b.gen;
    volatile int *verr = b.err;
    const unsigned g0 = *vgen;
    __threadfence();
    const unsigned arrived = atomicAdd(b.count, 1u);
    if (arrived == nblocks - 1) {
      atomicExch(b.count, 0u);
      __threadfence();
      atomicAdd(b.gen, 1u);
    } else {
      const unsigned long long t0 = globaltimer();
      unsigned spins = 0;
      while (*vgen == g0) {
        if (*verr) {
          ok = 0;
          break;
        }
        if (wait_expired(b, ++spins, t0)) {
          atomicCAS(b.err, 0, X2G_ERR_TIMEOUT);
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
    if (*verr) ok = 0;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Neighbour wait of the persistent-band sweep: block b publishes in
// phase[b] how many colour phases it has finished (release store after its
// writes), and before reloading its halos for phase k waits until every
// block whose rows lie within 4 rows of its band (nb[0..5], -1 = none) has
// finished k phases (acquire loads by lanes 0..5 of warp 0), while lane 6
// reads the error word once, so that a launch started after an error leaves
// at its first wait.  The wait is bounded as in grid_barrier.
__device__ __forceinline__ void st_release(unsigned *p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ bool wait_neighbours(const BarrierDev &b, const unsigned *phase, int nbq, unsigned k) {
  __shared__ int s_ok;
  if (threadIdx.x < 32) {
    int ok = 1;
    volatile int *verr = b.err;
    if (threadIdx.x == 6) {
      if (*verr) ok = 0;
    } else if (nbq >= 0) {
      const unsigned long long t0 = globaltimer();
      unsigned spins = 0;
      while (ld_acquire(phase + size_t(nbq) * kPhaseStride) < k) {
        if (*verr) {
          ok = 0;
          break;
        }
        if (wait_expired(b, ++spins, t0)) {
          atomicCAS(b.err, 0, X2G_ERR_TIMEOUT);
          ok = 0;
          break;
        }
        __nanosleep(20);
      }
      __threadfence();
    }
    ok = __all_sync(0xffffffffu, ok);
    if (threadIdx.x == 0) s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// ----------------------------------------------------------------------
// One point update, FP64, reference arithmetic order (sormcsor.F90:46-71).
// ----------------------------------------------------------------------
__device__ __forceinline__ void relax_f64(double *__restrict__ u, int ij, const GridDev &g, double b, double d,
                                          double lhs, double rhs, double omega, double omega1) {
  const int n1 = g.n8, n2 = 2 * g.n8, n3 = 3 * g.n8, n4 = 4 * g.n8;
  const double m4 = ldcg(u + ij - n4), p4 = ldcg(u + ij + n4);
  const double m3 = ldcg(u + ij - n3), p3 = ldcg(u + ij + n3);
  const double m2 = ldcg(u + ij - n2), p2 = ldcg(u + ij + n2);
  const double m1 = ldcg(u + ij - n1), p1 = ldcg(u + ij + n1);
  const double l4 = ldcg(u + ij - 4), r4 = ldcg(u + ij + 4);
  const double l3 = ldcg(u + ij - 3), r3 = ldcg(u + ij + 3);
  const double l2 = ldcg(u + ij - 2), r2 = ldcg(u + ij + 2);
  const double l1 = ldcg(u + ij - 1), r1 = ldcg(u + ij + 1);
  const double uc = ldcg(u + ij);
  const double ddmi2 =
      A(A(A(M(g.dmu2[0], A(m4, p4)), M(g.dmu2[1], A(m3, p3))), M(g.dmu2[2], A(m2, p2))), M(g.dmu2[3], A(m1, p1)));
  const double ddmi1 =
      A(A(A(M(g.dmu1[0], S(m4, p4)), M(g.dmu1[1], S(m3, p3))), M(g.dmu1[2], S(m2, p2))), M(g.dmu1[3], S(m1, p1)));
  const double ddni2 =
      A(A(A(M(g.dni2[0], A(l4, r4)), M(g.dni2[1], A(l3, r3))), M(g.dni2[2], A(l2, r2))), M(g.dni2[3], A(l1, r1)));
  const double ddni1 =
      A(A(A(M(g.dni1[0], S(l4, r4)), M(g.dni1[1], S(l3, r3))), M(g.dni1[2], S(l2, r2))), M(g.dni1[3], S(l1, r1)));
  const double cc = A(A(A(ddmi2, M(b, ddmi1)), ddni2), M(d, ddni1));
  u[ij] = A(D(M(omega, S(rhs, cc)), lhs), M(omega1, uc));
}

struct CoefF {
  float dmu1[4], dmu2[4], dni1[4], dni2[4];
};

// FP32 correction sweep point update (same operator, FMA allowed) on a band
// of the correction held in shared memory; w is omega / lhs of the point,
// formed once per relaxation call.  Returns the new value.
__device__ __forceinline__ float relax_f32(const float *__restrict__ e, int ij, int n8, const CoefF &c, float b,
                                           float d, float w, float r, float omega1) {
  const int n1 = n8, n2 = 2 * n8, n3 = 3 * n8, n4 = 4 * n8;
  const float m4 = e[ij - n4], p4 = e[ij + n4];
  const float m3 = e[ij - n3], p3 = e[ij + n3];
  const float m2 = e[ij - n2], p2 = e[ij + n2];
  const float m1 = e[ij - n1], p1 = e[ij + n1];
  const float l4 = e[ij - 4], r4 = e[ij + 4];
  const float l3 = e[ij - 3], r3 = e[ij + 3];
  const float l2 = e[ij - 2], r2 = e[ij + 2];
  const float l1 = e[ij - 1], r1 = e[ij + 1];
  const float ec = e[ij];
  float dm2 = c.dmu2[0] * (m4 + p4);
  dm2 = __fmaf_rn(c.dmu2[1], m3 + p3, dm2);
  dm2 = __fmaf_rn(c.dmu2[2], m2 + p2, dm2);
  dm2 = __fmaf_rn(c.dmu2[3], m1 + p1, dm2);
  float dm1 = c.dmu1[0] * (m4 - p4);
  dm1 = __fmaf_rn(c.dmu1[1], m3 - p3, dm1);
  dm1 = __fmaf_rn(c.dmu1[2], m2 - p2, dm1);
  dm1 = __fmaf_rn(c.dmu1[3], m1 - p1, dm1);
  float dn2 = c.dni2[0] * (l4 + r4);
  dn2 = __fmaf_rn(c.dni2[1], l3 + r3, dn2);
  dn2 = __fmaf_rn(c.dni2[2], l2 + r2, dn2);
  dn2 = __fmaf_rn(c.dni2[3], l1 + r1, dn2);
  float dn1 = c.dni1[0] * (l4 - r4);
  dn1 = __fmaf_rn(c.dni1[1], l3 - r3, dn1);
  dn1 = __fmaf_rn(c.dni1[2], l2 - r2, dn1);
  dn1 = __fmaf_rn(c.dni1[3], l1 - r1, dn1);
  const float cc = __fmaf_rn(d, dn1, __fmaf_rn(b, dm1, dm2) + dn2);
  return __fmaf_rn(omega1, ec, w * (r - cc));
}

// ----------------------------------------------------------------------
// Tile-local pieces of one relaxation call.  A tile is a band of ext rows
// [row0,row1) over the full nu width.
// ----------------------------------------------------------------------

// putin ghosts for the tile's rows (src/inout.F90:47-80): ghost columns copy
// nu = 2..5 / nni-1..nni-4, tile 0 also fills the mu ghost rows.
__device__ void tile_ghosts(const GridDev &g, double *u, int t, int isym) {
  const int row0 = g.tile_row0[t], row1 = g.tile_row1[t], n8 = g.n8, nni = g.nni;
  const bool neg = (isym != 1);
  const int nr = row1 - row0;
  for (int k = threadIdx.x; k < nr * 8; k += blockDim.x) {
    const int r = row0 + k / 8, q = k % 8;
    const int base = r * n8;
    if (q < 4) {
      const int j = q + 1;  // ghost col 4-j <- col 4+j
      const double v = ldcg(u + base + 4 + j);
      u[base + 4 - j] = neg ? -v : v;
    } else {
      const int j = q - 3;  // ghost col nni+3+j <- col nni+3-j
      const double v = ldcg(u + base + nni + 3 - j);
      u[base + nni + 3 + j] = neg ? -v : v;
    }
  }
  if (t == 0) {
    for (int k = threadIdx.x; k < 4 * nni; k += blockDim.x) {
      const int i = k / nni + 1, col = 4 + k % nni;  // ghost row 4-i <- row 4+i
      const double v = ldcg(u + (4 + i) * n8 + col);
      u[(4 - i) * n8 + col] = neg ? -v : v;
    }
  }
}

// Axis extrapolation after a micro-sweep (sormcsor.F90:94-129): mu=1 row
// (tile 0), nu=1 and nu=nni columns of the tile's rows; the two corners at
// mu=1 read the freshly extrapolated mu=1 row, so they follow a sync.
template <typename T>
__device__ void tile_boundary(const GridDev &g, T *u, int t, int isym) {
  const int row0 = g.tile_row0[t], row1 = g.tile_row1[t], n8 = g.n8, nni = g.nni;
  const int n1 = n8, n2 = 2 * n8, n3 = 3 * n8, n4 = 4 * n8, n5 = 5 * n8;
  const bool even = (isym == 1);
  const int nrow7 = (t == 0) ? nni - 2 : 0;
  const int r0 = (t == 0) ? 5 : row0;
  const int nside = 2 * (row1 - r0);
  for (int k = threadIdx.x; k < nrow7 + nside; k += blockDim.x) {
    if (k < nrow7) {
      const int ij = 4 * n8 + 5 + k;
      T v = T(0);
      if (even) {
        if constexpr (sizeof(T) == 8) {
          v = A(A(A(A(M(g.exeven[0], ldcg(u + ij + n1)), M(g.exeven[1], ldcg(u + ij + n2))),
                    M(g.exeven[2], ldcg(u + ij + n3))),
                  M(g.exeven[3], ldcg(u + ij + n4))),
                M(g.exeven[4], ldcg(u + ij + n5)));
        } else {
          v = g.exevenf[0] * ldcg(u + ij + n1) + g.exevenf[1] * ldcg(u + ij + n2) +
              g.exevenf[2] * ldcg(u + ij + n3) + g.exevenf[3] * ldcg(u + ij + n4) +
              g.exevenf[4] * ldcg(u + ij + n5);
        }
      }
      u[ij] = v;
    } else {
      const int q = k - nrow7;
      const int r = r0 + q / 2;
      const int side = q % 2;
      const int ij = r * n8 + (side == 0 ? 4 : nni + 3);
      const int s = (side == 0) ? 1 : -1;
      T v = T(0);
      if (even) {
        if constexpr (sizeof(T) == 8) {
          v = A(A(A(A(M(g.exeven[0], ldcg(u + ij + s)), M(g.exeven[1], ldcg(u + ij + 2 * s))),
                    M(g.exeven[2], ldcg(u + ij + 3 * s))),
                  M(g.exeven[3], ldcg(u + ij + 4 * s))),
                M(g.exeven[4], ldcg(u + ij + 5 * s)));
        } else {
          v = g.exevenf[0] * ldcg(u + ij + s) + g.exevenf[1] * ldcg(u + ij + 2 * s) +
              g.exevenf[2] * ldcg(u + ij + 3 * s) + g.exevenf[3] * ldcg(u + ij + 4 * s) +
              g.exevenf[4] * ldcg(u + ij + 5 * s);
        }
      }
      u[ij] = v;
    }
  }
  if (t == 0) {
    __syncthreads();
    if (threadIdx.x < 2) {
      const int ij = 4 * n8 + (threadIdx.x == 0 ? 4 : nni + 3);
      const int s = (threadIdx.x == 0) ? 1 : -1;
      T v = T(0);
      if (even) {
        if constexpr (sizeof(T) == 8) {
          v = A(A(A(A(M(g.exeven[0], ldcg(u + ij + s)), M(g.exeven[1], ldcg(u + ij + 2 * s))),
                    M(g.exeven[2], ldcg(u + ij + 3 * s))),
                  M(g.exeven[3], ldcg(u + ij + 4 * s))),
                M(g.exeven[4], ldcg(u + ij + 5 * s)));
        } else {
          v = g.exevenf[0] * ldcg(u + ij + s) + g.exevenf[1] * ldcg(u + ij + 2 * s) +
              g.exevenf[2] * ldcg(u + ij + 3 * s) + g.exevenf[3] * ldcg(u + ij + 4 * s) +
              g.exevenf[4] * ldcg(u + ij + 5 * s);
        }
      }
      u[ij] = v;
    }
  }
}

// Potential right-hand side for the tile's interior points
// (relaxPots.F90:81-82: rhs = psi_a psi_b g, two successive products).
__device__ void tile_rhs(const GridDev &g, const JobDev &J, int t) {
  const int b0 = g.off[(t * 5) * g.nlev], b1 = g.off[(t * 5 + 5) * g.nlev];
  for (int k = b0 + threadIdx.x; k < b1; k += blockDim.x) {
    const int ij = g.pts[k];
    const int row = ij / g.n8, col = ij - row * g.n8;
    const int ik = (row - 4) * g.nni + (col - 4);
    J.rhs_buf[ik] = M(M(J.psa[ij], J.psb[ij]), g.g[ik]);
  }
}

// ----------------------------------------------------------------------
// Persistent cooperative MCSOR kernel of the relaxation that allocates
// nothing (its fixed scratch has no room for the wavefront's tagged copies):
// all jobs x tiles, 5 colour phases per micro-sweep, grid barrier between
// phases.
// ----------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_mcsor_f64(GridDev g, const __grid_constant__ JobTable jobs, int njobs,
                                                        int nsweeps, BarrierDev bar, unsigned nblocks) {
  const int nitems = njobs * g.ntiles;
  for (int s = 0; s < nsweeps; ++s) {
    for (int c = 0; c < 5; ++c) {
      for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int jb = item / g.ntiles, t = item - jb * g.ntiles;
        const JobDev &J = jobs.j[jb];
        double *u = J.u;
        if (c == 0) {
          if (s == 0) {
            tile_ghosts(g, u, t, J.isym);
            if (J.kind == 1) tile_rhs(g, J, t);  // kind 2: explicit rhs
          } else {
            tile_boundary<double>(g, u, t, J.isym);
          }
          __syncthreads();
        }
        const double omega = J.omega, omega1 = 1.0 - J.omega;  // omega1 = 1 - omega (relaxOrbs.F90:83)
        const double *bt = (J.kind >= 1) ? g.bpot_mu : g.borb_mu;
        const double *rhsv = (J.kind == 1) ? J.rhs_buf : J.rhs;
        for (int l = 0; l < g.nlev; ++l) {
          const int o = (t * 5 + c) * g.nlev + l;
          const int b0 = g.off[o], b1 = g.off[o + 1];
          if (b0 == b1) continue;
          for (int k = b0 + threadIdx.x; k < b1; k += blockDim.x) {
            const int ij = g.pts[k];
            const int row = ij / g.n8, col = ij - row * g.n8;
            const int mu = row - 4, nu = col - 4, ik = mu * g.nni + nu;
            double lhs;
            if (J.kind == 1)
              lhs = (J.idel2 == 0.0) ? g.f3_mu[mu] : A(g.f3_mu[mu], M(J.idel2, g.e[ik]));
            else
              lhs = J.lhs[ik];
            relax_f64(u, ij, g, bt[mu], g.d_nu[nu], lhs, rhsv[ik], omega, omega1);
          }
          __syncthreads();
        }
      }
      if (!(s == nsweeps - 1 && c == 4)) {
        if (!grid_barrier(bar, nblocks)) return;
      }
    }
  }
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int jb = item / g.ntiles, t = item - jb * g.ntiles;
    tile_boundary<double>(g, jobs.j[jb].u, t, jobs.j[jb].isym);
    __syncthreads();
  }
}

// ----------------------------------------------------------------------
// FP64 sweeps as a dataflow wavefront (list-order SOR, sormcsor.F90:20-132,
// over the reference's list): step t holds, for every sweep s still running,
// the interior points of level t - s * delta and the axis points whose
// extrapolation after sweep s belongs to that level (the host schedule,
// build_wave_schedule, proves the updates of a step independent and every
// read value current).  Reference arithmetic order, as relax_f64.
//
// There is no barrier between steps.  The launch keeps every value together
// with its tag, the number of sweeps it has been through, in one 16-byte
// word that is read and written whole; an update waits until the values it
// reads carry the tags its list position asks for (the number of the sweep,
// one more for the points earlier in the list).  Values are not overwritten
// too early: a stencil neighbour reads and is read, so the tags that order
// the new values order the old ones too; the only reads that go one way, the
// fifth point of an axis extrapolation and the mu=1 row's corner, are
// checked in the opposite direction as well (wait_value).  Every warp takes
// its items in step order, so the earliest unfinished update never waits.
//
// What bounds it: the dependent chain of a step.  One FP64 instruction of a
// warp takes ~64 cycles here whatever its active lanes, so kSplit = 4 lanes
// share one point of a narrow step: each forms one of the four derivative
// sums (11 instructions instead of 44 in a row) and the shuffled sums are
// combined in the reference's order; wide steps (kSplit = 1) take a point
// per lane, which issues the fewest FP64 instructions.  SOR, 10 sweeps of one
// 331 x 481 orbital (481 steps): 2.26 ms, 9400 cycles a step of which 2240
// are its FP64 chain, most of the rest the way of a value through L2; 21.8 ms
// with a grid barrier after every step and the sweeps of a step looked up one
// after the other.
// ----------------------------------------------------------------------
constexpr int kWaveThreads = 512;
// level offsets held in shared memory: a usual grid's within the default cap,
// the most that a launch may ask for
constexpr size_t kWaveSmem = 47 * 1024, kWaveSmemMost = 200 * 1024;
constexpr unsigned kTagFixed = 0x7fffffffu;  // values no sweep changes

struct Tagged {
  double v;
  int tag;
};

__device__ __forceinline__ Tagged ld_tagged(const ulonglong2 *p) {
  unsigned long long lo, hi;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return Tagged{__longlong_as_double((long long)lo), int(unsigned(hi))};
}

__device__ __forceinline__ void st_tagged(ulonglong2 *p, double v, int tag) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%0, %1};\n\tst.relaxed.gpu.global.b128 [%2], q;\n\t}" ::"l"(
                   __double_as_longlong(v)),
               "l"((unsigned long long)(unsigned)tag), "l"(p)
               : "memory");
}

// Bounded wait bookkeeping of one warp: false when the launch must stop (its
// own wait ran out, or another block's did).
struct WaveWait {
  unsigned spins = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool again(const BarrierDev &b) {
    if ((++spins & 63u) != 0 && b.limit_ns != 0) return true;
    if (*(volatile int *)b.err) return false;
    const unsigned long long now = globaltimer();
    if (t0 == 0) t0 = now;
    if (now - t0 >= b.limit_ns) {
      atomicCAS(b.err, 0, X2G_ERR_TIMEOUT);
      return false;
    }
    return true;
  }
};

// One warp's next piece of work: kind 0 interior points, 1 axis points, -1
// none left.  Every lane (of a group of kSplit) has its own point; lanes
// past the end of the list have s = -1.
struct WaveItem {
  int kind, jb, s;
  int rc;         // (ext row << 16) | ext col
  unsigned mask;  // interior points: the mask of WaveHost::pts
  __device__ __forceinline__ int row() const { return rc >> 16; }
  __device__ __forceinline__ int col() const { return rc & 0xffff; }
};

// Walks the steps of the schedule, handing this warp groups wid, wid + nw,
// ... of each step: first groups of 32 / kSplit interior points, then groups
// of 32 axis points.  The sweeps that run in a step are looked at by the
// lanes at once, 32 at a time (counts summed and searched with shuffles): a
// loop over the sweeps by every lane took longer than the updates
// themselves (7.3 us a step of 10 sweeps on 331 x 481, all of it here).
template <int kSplit>
struct WaveWalk {
  const int *off, *boff;  // shared memory copies
  int nlev, nblev, most, delta, nsweeps, njobs, T, wid, nw;
  int t, lo, hi, grp, ni, na, gi;  // step, its sweeps, next group, interior and axis points, interior groups
  __device__ __forceinline__ int count(const int *o, int levels, int s) const {
    const int l = t - s * delta;
    return (s <= hi && l < levels) ? o[l + 1] - o[l] : 0;
  }
  __device__ __forceinline__ void open() {
    while (hi < nsweeps - 1 && (hi + 1) * delta <= t) ++hi;
    while (lo * delta + most <= t) ++lo;
    const int lane = threadIdx.x & 31;
    ni = na = 0;
    for (int s = lo; s <= hi; s += 32) {
      ni += __reduce_add_sync(0xffffffffu, count(off, nlev, s + lane));
      na += __reduce_add_sync(0xffffffffu, count(boff, nblev, s + lane));
    }
    ni *= njobs;
    na *= njobs;
    gi = (ni * kSplit + 31) / 32;
    grp = wid;
  }
  __device__ __forceinline__ void start() {
    t = lo = hi = 0;
    open();
  }
  __device__ __forceinline__ WaveItem next(const WaveDev &w) {
    WaveItem it;
    it.kind = -1;
    it.s = -1;
    it.jb = 0;
    it.rc = (4 << 16) | 4;
    it.mask = 0;
    while (t < T && grp >= gi + (na + 31) / 32) {
      if (++t < T) open();
    }
    if (t >= T) return it;
    const int lane = threadIdx.x & 31;
    const bool axis = grp >= gi;
    it.kind = axis ? 1 : 0;
    const int *o = axis ? boff : off;
    const int levels = axis ? nblev : nlev;
    // this lane's point: index q of the step, in sweep s and job jb
    int q = axis ? (grp - gi) * 32 + lane : (grp * 32 + lane) / kSplit;
    grp += nw;
    bool found = false;
    for (int s0 = lo; s0 <= hi; s0 += 32) {
      int sum = count(o, levels, s0 + lane) * njobs;  // points up to and with sweep s0 + lane
#pragma unroll
      for (int d = 1; d < 32; d *= 2) {
        const int x = __shfl_up_sync(0xffffffffu, sum, d);
        if (lane >= d) sum += x;
      }
      // the first sweep whose sum is beyond q
      int f = 0;
#pragma unroll
      for (int d = 16; d > 0; d /= 2)
        if (__shfl_sync(0xffffffffu, sum, (f + d - 1) & 31) <= q) f += d;
      const int before = __shfl_sync(0xffffffffu, sum, (f + 31) & 31), all = __shfl_sync(0xffffffffu, sum, 31);
      if (!found && q < all) {
        found = true;
        const int s = s0 + f, l = t - s * delta, k0 = q - (f > 0 ? before : 0), n = o[l + 1] - o[l];
        const int jb = njobs > 1 ? k0 / n : 0, k = o[l] + k0 - jb * n;
        it.s = s;
        it.jb = jb;
        // the entry is first used when this item's turn comes
        const int2 e = axis ? make_int2(__ldg(w.bpts + k), 0) : __ldg(w.pts + k);
        it.rc = e.x;
        it.mask = unsigned(e.y);
      }
      q -= all;
    }
    return it;
  }
};

// Final value of an update: kept with its tag, and in u after the last sweep.
__device__ __forceinline__ void wave_store(const JobDev &J, int ij, double v, int s, int nsweeps) {
  st_tagged(J.tagged + ij, v, s + 1);
  if (s == nsweeps - 1) J.u[ij] = v;
}

// Axis extrapolation (sormcsor.F90:94-129): the mu=1 row along mu, the nu=1
// and nu=nni columns along nu; five values of this sweep.  The mu=1 row's
// points next to a corner also wait until that corner has read their last
// value.
__device__ __forceinline__ bool wave_axis(const GridDev &g, const JobTable &jobs, const WaveItem &it, int nsweeps,
                                          const BarrierDev &bar) {
  const JobDev &J = jobs.j[it.jb];
  const bool on = it.s >= 0;
  const int row = it.row(), col = it.col(), ij = row * g.n8 + col;
  const int st = (col == 4) ? 1 : (col == g.nni + 3) ? -1 : g.n8;
  int back = 0;  // a corner that reads this point
  if (on && row == 4 && col != 4 && col != g.nni + 3) {
    if (col <= 9) back = 4 * g.n8 + 4;
    else if (col >= g.nni - 2) back = 4 * g.n8 + g.nni + 3;
  }
  double v[5];
  bool got = !on;
  WaveWait ww;
  for (;;) {
    if (!got) {
      bool ok = true;
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const Tagged x = ld_tagged(J.tagged + ij + (k + 1) * st);
        v[k] = x.v;
        ok = ok && x.tag > it.s;
      }
      if (back) ok = ok && ld_tagged(J.tagged + back).tag >= it.s;
      got = ok;
    }
    if (__all_sync(0xffffffffu, got)) break;
    if (!__all_sync(0xffffffffu, ww.again(bar))) return false;
  }
  if (on) {
    double r = 0.0;
    if (J.isym == 1)
      r = A(A(A(A(M(g.exeven[0], v[0]), M(g.exeven[1], v[1])), M(g.exeven[2], v[2])), M(g.exeven[3], v[3])),
            M(g.exeven[4], v[4]));
    wave_store(J, ij, r, it.s, nsweeps);
  }
  return true;
}

// the axis value five points from a point, or 0: an extrapolation's last
// point is the only one that does not read it back (flags of
// WaveHost::pts); which: 0 along mu, 1 along nu
__device__ __forceinline__ int fifth_reader(const GridDev &g, unsigned mask, int ij, int which) {
  if (which == 0) return (mask & 0x10000u) ? ij - 5 * g.n8 : 0;
  return (mask & 0x20000u) ? ij - 5 : (mask & 0x40000u) ? ij + 5 : 0;
}

// a / b, rounded to nearest, from 1 / b = inv.x + inv.y to 106 bits: the
// quotient from both parts is one of the two doubles around a / b, its
// remainder is exact, and one correction by the rounded reciprocal gives the
// rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990, theorem on the final
// step): four operations in place of about ten.  inv.x = 0, and an a near an
// end of the exponent range (or zero): the quotient itself.
__device__ __forceinline__ double quotient(double a, double b, double2 inv) {
  const int ex = (__double2hiint(a) >> 20) & 0x7ff;
  if (unsigned(ex - 500) > 1000u || inv.x == 0.0) return D(a, b);
  const double q = fma(a, inv.x, a * inv.y);
  return fma(fma(-b, q, a), inv.x, q);
}
// 1 / b for quotient; 0 where b is not of moderate size
__device__ __forceinline__ double2 inverse(double b) {
  const int ex = (__double2hiint(b) >> 20) & 0x7ff;
  if (unsigned(ex - 623) > 800u) return make_double2(0.0, 0.0);
  const double r = D(1.0, b);
  return make_double2(r, fma(-b, r, 1.0) * r);
}

// (lhs, rhs), b(mu) and d(nu) of an interior point
template <bool kInverse>
struct WaveCoef {
  double2 lr, inv;
  double b, d;
  __device__ __forceinline__ WaveCoef(const GridDev &g, const JobDev &J, const WaveItem &it) {
    const int mu = it.row() - 4, nu = it.col() - 4;
    const double2 *at = reinterpret_cast<const double2 *>(J.pairs) + (kInverse ? 2 : 1) * (mu * g.nni + nu);
    lr = __ldcg(at);
    inv = kInverse ? __ldcg(at + 1) : make_double2(0.0, 0.0);
    b = __ldg((J.kind >= 1 ? g.bpot_mu : g.borb_mu) + mu);
    d = __ldg(g.d_nu + nu);
  }
};

// interior points, four lanes each: roles 0 / 1 the second / first mu
// derivative, 2 / 3 the nu derivatives
__device__ __forceinline__ bool wave_points4(const GridDev &g, const JobTable &jobs, const WaveItem &it, int nsweeps,
                                             const BarrierDev &bar, const double (&cf)[4]) {
  const JobDev &J = jobs.j[it.jb];
  const bool on = it.s >= 0;
  const int role = threadIdx.x & 3, st = (role < 2) ? g.n8 : 1, bit = (role < 2) ? 2 : 0;
  double m[4], p[4], uc = 0.0;
  unsigned miss = on ? 0x3ffu : 0u;  // values still to come: 8 neighbours, the centre, a fifth reader
  const int ij = it.row() * g.n8 + it.col();
  const WaveCoef<false> co(g, J, it);
  const int fifth = (role == 1) ? 0 : fifth_reader(g, it.mask, ij, role == 0 ? 0 : 1);
  if (!fifth) miss &= ~0x200u;
  WaveWait ww;
  for (;;) {
    Tagged x[4], y[4], c;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (miss & (1u << q)) x[q] = ld_tagged(J.tagged + ij - (4 - q) * st);
      if (miss & (16u << q)) y[q] = ld_tagged(J.tagged + ij + (4 - q) * st);
    }
    if (miss & 256u) c = ld_tagged(J.tagged + ij);
    if (miss & 512u) {
      if (ld_tagged(J.tagged + fifth).tag >= it.s) miss &= ~512u;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = 4 * (3 - q) + bit;
      if ((miss & (1u << q)) && x[q].tag >= it.s + int((it.mask >> e) & 1u)) {
        m[q] = x[q].v;
        miss &= ~(1u << q);
      }
      if ((miss & (16u << q)) && y[q].tag >= it.s + int((it.mask >> (e + 1)) & 1u)) {
        p[q] = y[q].v;
        miss &= ~(16u << q);
      }
    }
    if ((miss & 256u) && c.tag >= it.s) {
      uc = c.v;
      miss &= ~256u;
    }
    if (__all_sync(0xffffffffu, miss == 0)) break;
    if (!__all_sync(0xffffffffu, ww.again(bar))) return false;
    // values at distance 3 or 4 still missing: this warp is steps early and
    // must not take the load units from the warps whose turn it is
    if (__any_sync(0xffffffffu, miss & 0x33u)) __nanosleep(400);
    else if (__any_sync(0xffffffffu, miss & 0x44u)) __nanosleep(100);
  }
  // a - b as a + (-b): the same rounding
  const long long flip = (role & 1) ? (1ll << 63) : 0;
  double a[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) a[q] = A(m[q], __longlong_as_double(__double_as_longlong(p[q]) ^ flip));
  double t = A(A(A(M(cf[0], a[0]), M(cf[1], a[1])), M(cf[2], a[2])), M(cf[3], a[3]));
  t = M(role == 1 ? co.b : role == 3 ? co.d : 1.0, t);
  const int base = threadIdx.x & 28;
  const double ddmi2 = __shfl_sync(0xffffffffu, t, base), bddmi1 = __shfl_sync(0xffffffffu, t, base + 1);
  const double ddni2 = __shfl_sync(0xffffffffu, t, base + 2), dddni1 = __shfl_sync(0xffffffffu, t, base + 3);
  if (on) {
    const double omega = J.omega, omega1 = 1.0 - J.omega;
    const double cc = A(A(A(ddmi2, bddmi1), ddni2), dddni1);
    const double v = A(D(M(omega, S(co.lr.y, cc)), co.lr.x), M(omega1, uc));
    if (role == 0) wave_store(J, ij, v, it.s, nsweeps);
  }
  return true;
}

// kWide: a step holds so many points that the FP64 pipe is the bound.  The
// products of the sums and differences of the neighbours at distance 4 and 3
// then go to the integer pipes (pair_products), 16 of the 53 FP64 operations
// of a point besides its quotient, and the quotient comes from a stored
// reciprocal.  Three or four distances there make the integer side the bound.
// interior points, one lane each
template <bool kWide>
__device__ __forceinline__ bool wave_points1(const GridDev &g, const JobTable &jobs, const WaveItem &it, int nsweeps,
                                             const BarrierDev &bar) {
  const JobDev &J = jobs.j[it.jb];
  const bool on = it.s >= 0;
  double n[16], uc = 0.0;
  const int ij = it.row() * g.n8 + it.col();
  const WaveCoef<kWide> co(g, J, it);
  const int f0 = fifth_reader(g, it.mask, ij, 0), f1 = fifth_reader(g, it.mask, ij, 1);
  bool got = !on;
  WaveWait ww;
  for (;;) {
    if (!got) {
      bool ok = true;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const int k = e / 4 + 1, st = (e & 2) ? k * g.n8 : k;
        const Tagged x = ld_tagged(J.tagged + ((e & 1) ? ij + st : ij - st));
        n[e] = x.v;
        ok = ok && x.tag >= it.s + int((it.mask >> e) & 1u);
      }
      const Tagged c = ld_tagged(J.tagged + ij);
      uc = c.v;
      ok = ok && c.tag >= it.s;
      if (f0) ok = ok && ld_tagged(J.tagged + f0).tag >= it.s;
      if (f1) ok = ok && ld_tagged(J.tagged + f1).tag >= it.s;
      got = ok;
    }
    if (__all_sync(0xffffffffu, got)) break;
    if (!__all_sync(0xffffffffu, ww.again(bar))) return false;
  }
  if (on) {
    double m2[4], m1[4], n2[4], n1[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double xm = n[14 - 4 * q], ym = n[15 - 4 * q], xn = n[12 - 4 * q], yn = n[13 - 4 * q];
      if (!kWide || q >= 2 || !pair_products(xm, ym, g.pmu2[q], g.pmu1[q], m2[q], m1[q])) {
        m2[q] = M(g.dmu2[q], A(xm, ym));
        m1[q] = M(g.dmu1[q], S(xm, ym));
      }
      if (!kWide || q >= 2 || !pair_products(xn, yn, g.pnu2[q], g.pnu1[q], n2[q], n1[q])) {
        n2[q] = M(g.dni2[q], A(xn, yn));
        n1[q] = M(g.dni1[q], S(xn, yn));
      }
    }
    const double ddmi2 = A(A(A(m2[0], m2[1]), m2[2]), m2[3]), ddmi1 = A(A(A(m1[0], m1[1]), m1[2]), m1[3]);
    const double ddni2 = A(A(A(n2[0], n2[1]), n2[2]), n2[3]), ddni1 = A(A(A(n1[0], n1[1]), n1[2]), n1[3]);
    const double omega = J.omega, omega1 = 1.0 - J.omega;
    const double cc = A(A(A(ddmi2, M(co.b, ddmi1)), ddni2), M(co.d, ddni1));
    const double num = M(omega, S(co.lr.y, cc));
    wave_store(J, ij, A(kWide ? quotient(num, co.lr.x, co.inv) : D(num, co.lr.x), M(omega1, uc)), it.s, nsweeps);
  }
  return true;
}

// Threads id of nt: the tagged copy of every function, its ghost cells
// refreshed as putin does (in u too), and the (lhs, rhs) pairs: a potential's
// lhs = f3 + idel^2 e and rhs = psa psb g with the roundings of
// relaxPots.F90:81-95.  kInverse: 1 / lhs after each pair.
template <bool kInverse>
__device__ __forceinline__ void wave_prologue(const GridDev &g, const JobTable &jobs, int njobs, int id, int nt) {
  for (int jb = 0; jb < njobs; ++jb) {
    const JobDev &J = jobs.j[jb];
    for (int k = id; k < g.next; k += nt) {
      const int row = k / g.n8, col = k - row * g.n8;
      int src = k;
      if (row >= 4 && row < g.nmu) {
        if (col < 4) src = row * g.n8 + 8 - col;
        else if (col > g.nni + 3) src = row * g.n8 + 2 * g.nni + 6 - col;
      } else if (row < 4 && col >= 4 && col <= g.nni + 3) {
        src = (8 - row) * g.n8 + col;
      }
      double v = ldcg(J.u + src);
      if (src != k) {
        if (J.isym != 1) v = -v;
        J.u[k] = v;
      }
      const bool swept = row >= 4 && row < g.nmu && col >= 4 && col <= g.nni + 3;  // interior and axis
      st_tagged(J.tagged + k, v, swept ? 0 : int(kTagFixed));
    }
    double2 *pairs = reinterpret_cast<double2 *>(J.pairs);
    for (int k = id; k < g.mxsize; k += nt) {
      double2 lr;
      if (J.kind == 1) {
        const int mu = k / g.nni, ij = (mu + 4) * g.n8 + (k - mu * g.nni) + 4;
        lr.x = (J.idel2 == 0.0) ? g.f3_mu[mu] : A(g.f3_mu[mu], M(J.idel2, g.e[k]));
        lr.y = M(M(J.psa[ij], J.psb[ij]), g.g[k]);
      } else {
        lr = make_double2(J.lhs[k], J.rhs[k]);
      }
      if (kInverse) {
        pairs[2 * k] = lr;
        pairs[2 * k + 1] = inverse(lr.x);
      } else {
        pairs[k] = lr;
      }
    }
  }
}

template <int kSplit, bool kWide>
__global__ void __launch_bounds__(kWaveThreads, 1) k_wave_f64(GridDev g, WaveDev w, const __grid_constant__ JobTable jobs,
                                                             int njobs, int nsweeps, BarrierDev bar, unsigned nblocks) {
  extern __shared__ int s_off[];
  const int nt = int(gridDim.x * blockDim.x), id = int(blockIdx.x * blockDim.x + threadIdx.x);
  for (int k = threadIdx.x; k <= w.nlev; k += blockDim.x) s_off[k] = w.off[k];
  for (int k = threadIdx.x; k <= w.nblev; k += blockDim.x) s_off[w.nlev + 1 + k] = w.boff[k];
  wave_prologue<kWide>(g, jobs, njobs, id, nt);
  if (!grid_barrier(bar, nblocks)) return;
  WaveWalk<kSplit> walk;
  walk.off = s_off;
  walk.boff = s_off + w.nlev + 1;
  walk.nlev = w.nlev;
  walk.nblev = w.nblev;
  walk.delta = w.delta;
  walk.nsweeps = nsweeps;
  walk.njobs = njobs;
  walk.most = w.nlev > w.nblev ? w.nlev : w.nblev;
  walk.T = (nsweeps - 1) * w.delta + walk.most;
  walk.wid = int((threadIdx.x >> 5) * gridDim.x + blockIdx.x);  // neighbouring groups on different SMs
  walk.nw = int(gridDim.x * (blockDim.x >> 5));
  walk.start();
  double cf[4];
  {
    const int role = threadIdx.x & 3;
    const double *c = role == 0 ? g.dmu2 : role == 1 ? g.dmu1 : role == 2 ? g.dni2 : g.dni1;
#pragma unroll
    for (int q = 0; q < 4; ++q) cf[q] = c[q];
  }
  WaveItem it = walk.next(w);
  while (it.kind >= 0) {
    // the next item's list entry and pair travel while this one waits
    const WaveItem nx = walk.next(w);
    bool ok;
    if (it.kind == 1)
      ok = wave_axis(g, jobs, it, nsweeps, bar);
    else if (kSplit == 4)
      ok = wave_points4(g, jobs, it, nsweeps, bar, cf);
    else
      ok = wave_points1<kWide>(g, jobs, it, nsweeps, bar);
    if (!ok) return;
    it = nx;
  }
}

// ----------------------------------------------------------------------
// List-order SOR of a few functions: the same dataflow on values in shared
// memory.  A block owns kRows rows of one job (the mu=1 row included) for the
// whole launch and keeps them, with four rows on each side, as (value, tag)
// words in shared memory.  A runner, kLanes lanes, follows a row's columns in
// one sweep from the middle to one side, in list order, then the axis; it goes
// on as soon as its point's values are there, so the rows of a warp settle one
// column apart.  A warp's runners are both sides of all rows, in march_per
// sweeps, and take every kMarchSweeps-th sweep.  The other warps fetch the
// neighbours' rows, a lane per row, side and sweep, from the tagged copy in
// global memory.  A value of a row outside the block's own is overwritten there
// only after its readers in this block are through (see above), so the copies
// need no further order.
//
// What bounds it: the FP64 chain of a point (2050 cycles with four lanes) and
// one round of loads while a block has few runners at work; more than four
// warps share an SM's FP64 pipe (19 cycles an operation and warp; 23 operations
// for 8 points with four lanes, 33 for 16 with two), hence few rows per block,
// fewer warps on an SM, while there are SMs enough for that, and two lanes where
// the pipe is the bound.  The way of a value through L2, most of a step's 5800
// cycles when every value takes it, is paid once per block of rows.  All nine or
// ten values of a point are loaded at once (one after the other, as each is
// found, took 1550 cycles).  SOR, 10 sweeps of one orbital, wavefront / this:
// 331 x 481 2.26 / 1.14 ms (four rows, two lanes), 151 x 181 0.93 / 0.48, 91 x
// 121 0.62 / 0.36 (two rows, four lanes; four rows 0.63 and 0.40).
// ----------------------------------------------------------------------
constexpr int kMarchSweeps = 10;
constexpr int kMarchFetch = (8 * 2 * kMarchSweeps + 31) / 32;  // warps that fetch
// sweeps that a warp's runners are of, and threads of a block
__host__ __device__ constexpr int march_per(int rows, int lanes) { return 16 / lanes / rows; }
__host__ __device__ constexpr int march_threads(int rows, int lanes) {
  return 32 * (kMarchSweeps / march_per(rows, lanes) + kMarchFetch);
}

// one 128-bit access: a reader must never see a tag without its value (a vector
// of two 64-bit ones may be taken apart)
__device__ __forceinline__ Tagged ld_near(unsigned at) {
  unsigned long long lo, hi;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.cta.shared.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(lo), "=l"(hi)
               : "r"(at)
               : "memory");
  return Tagged{__longlong_as_double((long long)lo), int(unsigned(hi))};
}
__device__ __forceinline__ void st_near(unsigned at, double v, int tag) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%0, %1};\n\tst.relaxed.cta.shared.b128 [%2], q;\n\t}" ::"l"(
                   __double_as_longlong(v)),
               "l"((unsigned long long)(unsigned)tag), "r"(at)
               : "memory");
}

template <int kRows, int kLanes>
__global__ void __launch_bounds__(march_threads(kRows, kLanes), 1)
    k_march_f64(GridDev g, MarchDev w, const __grid_constant__ JobTable jobs, int njobs, int nsweeps, BarrierDev bar,
                unsigned nblocks) {
  extern __shared__ __align__(16) ulonglong2 near[];
  constexpr int kThr = march_threads(kRows, kLanes), kPer = march_per(kRows, kLanes), kWarps = kMarchSweeps / kPer;
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  wave_prologue<true>(g, jobs, njobs, int(blockIdx.x) * kThr + tid, int(gridDim.x) * kThr);
  if (!grid_barrier(bar, nblocks)) return;
  const int bands = int(gridDim.x) / njobs, jb = int(blockIdx.x) / bands;
  const JobDev &J = jobs.j[jb];
  const int n8 = g.n8, nmu = g.nmu;
  const int r0 = 4 + (int(blockIdx.x) - jb * bands) * kRows;
  const unsigned base = unsigned(__cvta_generic_to_shared(near));
  // shared address of ext index ij: rows r0 - 4 .. r0 + kRows + 3
  const int first = (r0 - 4) * n8;
  auto addr = [&](int ij) { return base + unsigned(ij - first) * 16u; };
  for (int k = tid; k < (kRows + 8) * n8; k += kThr) {
    const int ij = min(first + k, g.next - 1);
    const Tagged x = ld_tagged(J.tagged + ij);
    st_near(base + unsigned(k) * 16u, x.v, x.tag);
  }
  __syncthreads();
  WaveWait ww;
  if (warp >= kWarps) {
    // fetch: the four rows on each side
    const int id = tid - 32 * kWarps, h = id & 7, half = id >> 3 & 1, slot = id >> 4;
    const int row = h < 4 ? r0 - 4 + h : r0 + kRows + h - 4;
    bool on = slot < kMarchSweeps && row >= 4 && row < nmu;
    int s = slot, k = 0, n = 0, o = 0;
    if (on) {
      o = w.off[(row - 4) * 2 + half];
      n = w.off[(row - 4) * 2 + half + 1] - o;
    }
    on = on && s < nsweeps && n > 0;
    int ij = on ? __ldg(&w.pts[o].x) : 0;
    while (__any_sync(0xffffffffu, on)) {
      bool got = false;
      if (on) {
        const Tagged x = ld_tagged(J.tagged + ij);
        got = x.tag > s;
        if (got) {
          st_near(addr(ij), x.v, x.tag);
          if (++k == n) {
            k = 0;
            s += kMarchSweeps;
            on = s < nsweeps;
          }
          ij = __ldg(&w.pts[o + k].x);
        }
      }
      if (!__any_sync(0xffffffffu, got) && !__all_sync(0xffffffffu, ww.again(bar))) return;
      if (__any_sync(0xffffffffu, got)) ww = WaveWait();
    }
    return;
  }
  const int role = lane % kLanes, runner = lane / kLanes, half = runner & 1, row = r0 + (runner >> 1) % kRows;
  const bool along_nu = role >= kLanes / 2;
  // four lanes: second and first derivative along mu, then along nu; two: both
  // along mu, along nu (cf2 and cf1)
  double cf2[4], cf1[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    cf2[q] = along_nu ? g.dni2[q] : g.dmu2[q];
    cf1[q] = along_nu ? g.dni1[q] : g.dmu1[q];
    if (kLanes == 4 && (role & 1)) cf2[q] = cf1[q];
  }
  const int st = along_nu ? 1 : n8, bit = along_nu ? 0 : 2;
  const double omega = J.omega, omega1 = 1.0 - J.omega;
  const double bmu = row < nmu ? (J.kind >= 1 ? g.bpot_mu : g.borb_mu)[row - 4] : 0.0;
  int o = 0, n = 0;
  if (row < nmu) {
    o = w.off[(row - 4) * 2 + half];
    n = w.off[(row - 4) * 2 + half + 1] - o;
  }
  const double2 *pairs = reinterpret_cast<const double2 *>(J.pairs) - 2 * (4 * g.nni + 4);  // by ext row * nni + ext col
  for (int s = warp * kPer + (runner >> 1) / kRows; __any_sync(0xffffffffu, s < nsweeps); s += kMarchSweeps) {
    int k = 0;
    bool on = n > 0 && s < nsweeps;
    // (a runner without a row looks at a point of the first one)
    int2 cur = on ? __ldg(w.pts + o) : make_int2(r0 * n8 + 8, 0), nxt = cur, nxt2 = cur;
    if (n > 1) nxt = __ldg(w.pts + o + 1);  // entries three ahead, coefficients one
    if (n > 2) nxt2 = __ldg(w.pts + o + 2);
    auto coef = [&](const int2 &e, double2 &lr, double2 &inv, double &d) {
      if (on && !(unsigned(e.y) & kMarchAxis)) {
        const int col = e.x - row * n8;
        lr = __ldcg(pairs + 2 * (row * g.nni + col));
        inv = __ldcg(pairs + 2 * (row * g.nni + col) + 1);
        d = __ldg(g.d_nu + col - 4);
      }
    };
    double2 lr = make_double2(1.0, 0.0), lr_n = lr, inv = make_double2(1.0, 0.0), inv_n = inv;
    double dnu = 0.0, dnu_n = 0.0;
    coef(cur, lr, inv, dnu);
    bool fresh = true;
    while (__any_sync(0xffffffffu, on)) {
      const int ij = cur.x;
      const unsigned mask = unsigned(cur.y), at = addr(ij);
      const bool axis = (mask & kMarchAxis) != 0;
      if (fresh) {
        coef(nxt, lr_n, inv_n, dnu_n);
        fresh = false;
      }
      // a point's neighbours and its old value, or the five values of an
      // extrapolation; other: a value that is read by this point's and does
      // not read it back
      const int ast = (mask & kMarchAxisMu) ? n8 : (mask & kMarchAxisUp) ? 1 : -1;
      int other = ij;
      if (axis) {
        if ((mask & kMarchAxisMu) && ij - row * n8 <= 9) other = row * n8 + 4;
        else if ((mask & kMarchAxisMu) && ij - row * n8 >= g.nni - 2) other = row * n8 + g.nni + 3;
      } else {
        const int f = fifth_reader(g, mask, ij, along_nu ? 1 : 0);
        other = f ? f : ij;
      }
      Tagged x[4], y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x[q] = ld_near(axis ? at + unsigned((q + 1) * ast * 16) : at - unsigned((4 - q) * st * 16));
        y[q] = ld_near(axis ? at : at + unsigned((4 - q) * st * 16));
      }
      const Tagged c = ld_near(axis ? at + unsigned(5 * ast * 16) : at), z = ld_near(addr(other));
      bool ok = z.tag >= s;
      double m[4], p[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = 4 * (3 - q) + bit;
        m[q] = x[q].v;
        p[q] = y[q].v;
        ok = ok && x[q].tag >= s + (axis ? 1 : int(mask >> e & 1u));
        ok = ok && (axis || y[q].tag >= s + int(mask >> (e + 1) & 1u));
      }
      const double uc = c.v;
      ok = ok && c.tag >= s + (axis ? 1 : 0);
      if (axis && role != 0) ok = true;
      const unsigned waits = __ballot_sync(0xffffffffu, !ok);
      const bool ready = on && (waits >> (lane & ~(kLanes - 1)) & ((1u << kLanes) - 1)) == 0;
      if (!__any_sync(0xffffffffu, ready)) {
        if (!__all_sync(0xffffffffu, ww.again(bar))) return;
        if (ww.spins > 4) __nanosleep(ww.spins > 16 ? 200 : 40);
        continue;
      }
      ww = WaveWait();
      double v = 0.0;
      if (__any_sync(0xffffffffu, ready && !axis)) {
        const int b = lane & ~(kLanes - 1);
        double ddmi2, bddmi1, ddni2, dddni1;
        if (kLanes == 4) {
          // as wave_points4
          const long long flip = (role & 1) ? (1ll << 63) : 0;
          double a[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) a[q] = A(m[q], __longlong_as_double(__double_as_longlong(p[q]) ^ flip));
          double t = A(A(A(M(cf2[0], a[0]), M(cf2[1], a[1])), M(cf2[2], a[2])), M(cf2[3], a[3]));
          t = M(role == 1 ? bmu : role == 3 ? dnu : 1.0, t);
          ddmi2 = __shfl_sync(0xffffffffu, t, b);
          bddmi1 = __shfl_sync(0xffffffffu, t, b + 1);
          ddni2 = __shfl_sync(0xffffffffu, t, b + 2);
          dddni1 = __shfl_sync(0xffffffffu, t, b + 3);
        } else {
          double t2 = M(cf2[0], A(m[0], p[0])), t1 = M(cf1[0], S(m[0], p[0]));
#pragma unroll
          for (int q = 1; q < 4; ++q) {
            t2 = A(t2, M(cf2[q], A(m[q], p[q])));
            t1 = A(t1, M(cf1[q], S(m[q], p[q])));
          }
          t1 = M(along_nu ? dnu : bmu, t1);
          ddmi2 = __shfl_sync(0xffffffffu, t2, b);
          bddmi1 = __shfl_sync(0xffffffffu, t1, b);
          ddni2 = __shfl_sync(0xffffffffu, t2, b + 1);
          dddni1 = __shfl_sync(0xffffffffu, t1, b + 1);
        }
        const double cc = A(A(A(ddmi2, bddmi1), ddni2), dddni1);
        // omega (rhs - cc) and omega1 times the old value, on two lanes at once
        const double o = M(role == 1 ? omega1 : omega, role == 1 ? uc : S(lr.y, cc));
        const double old = __shfl_sync(0xffffffffu, o, b + 1);
        v = A(quotient(o, lr.x, inv), old);  // (of role 0)
      }
      if (ready && axis && role == 0) {
        v = 0.0;
        if (J.isym == 1)
          v = A(A(A(A(M(g.exeven[0], m[0]), M(g.exeven[1], m[1])), M(g.exeven[2], m[2])), M(g.exeven[3], m[3])),
                M(g.exeven[4], uc));
      }
      if (ready) {
        if (role == 0) {
          st_near(at, v, s + 1);
          wave_store(J, ij, v, s, nsweeps);
        }
        cur = nxt;
        lr = lr_n;
        inv = inv_n;
        dnu = dnu_n;
        fresh = true;
        on = ++k < n;
        nxt = nxt2;
        if (k + 2 < n) nxt2 = __ldg(w.pts + o + k + 2);
      }
      __syncwarp();
    }
  }
}

// Axis extrapolation of the correction (tile_boundary<float>) for tiles
// [t0, t1) computed in the band sb held in shared memory (indexed by ext
// index).
__device__ void band_boundary(const GridDev &g, float *sb, int t0, int t1, bool even) {
  const int n8 = g.n8, nni = g.nni;
  const int nrow7 = (t0 == 0) ? nni - 2 : 0;
  const int r0 = (t0 == 0) ? 5 : g.tile_row0[t0];
  const int nside = 2 * (g.tile_row1[t1 - 1] - r0);
  for (int k = threadIdx.x; k < nrow7 + nside; k += blockDim.x) {
    int ij, st;
    if (k < nrow7) {
      ij = 4 * n8 + 5 + k;
      st = n8;
    } else {
      const int q = k - nrow7, r = r0 + q / 2, side = q % 2;
      ij = r * n8 + (side == 0 ? 4 : nni + 3);
      st = (side == 0) ? 1 : -1;
    }
    float v = 0.0f;
    if (even)
      v = g.exevenf[0] * sb[ij + st] + g.exevenf[1] * sb[ij + 2 * st] + g.exevenf[2] * sb[ij + 3 * st] +
          g.exevenf[3] * sb[ij + 4 * st] + g.exevenf[4] * sb[ij + 5 * st];
    sb[ij] = v;
  }
  if (t0 == 0) {
    __syncthreads();
    if (threadIdx.x < 2) {
      const int ij = 4 * n8 + (threadIdx.x == 0 ? 4 : nni + 3);
      const int st = (threadIdx.x == 0) ? 1 : -1;
      float v = 0.0f;
      if (even)
        v = g.exevenf[0] * sb[ij + st] + g.exevenf[1] * sb[ij + 2 * st] + g.exevenf[2] * sb[ij + 3 * st] +
            g.exevenf[3] * sb[ij + 4 * st] + g.exevenf[4] * sb[ij + 5 * st];
      sb[ij] = v;
    }
  }
}

// Shared memory of the band of a run of G tiles with its 4-row halos, as
// whole 16-byte pieces.
__host__ __device__ inline size_t band_smem_bytes(const GridDev &g, int G) {
  return ((size_t(g.st_rows[G]) * g.n8 + 8) * sizeof(float) + 15) / 16 * 16;
}

// Persistent-band FP32 sweep for grids whose bands do not fit one cluster's
// shared memory.  Block b owns, for the whole launch, one run of G
// consecutive tiles of one job (rows [row0, row1)) and keeps the
// correction on those rows, with 4-row halos, in shared memory, as whole
// 16-byte pieces: piece f holds ext indices 4f..4f+3 at sband[4 (f - f0)].
// Every colour phase waits until the blocks within halo reach have
// finished the previous phase (wait_neighbours; this also means they are
// done reading this band's edge rows), refreshes the two halos from the
// correction in global memory (L2), updates the phase's points level by
// level in shared memory, writes to global memory only the new values
// within 4 rows of a band edge shared with another block (that block's
// halo), and publishes its finished phase count.  No grid-wide barrier.
// Same-colour
// stencil neighbours never lie in different tiles, so the values a phase
// changes in a neighbour's rows are never read by this block in that phase,
// and a halo piece that reaches into an own row covers only ghost columns
// (zero throughout).  The kernel ends with u += e and the FP64 axis values
// of u on the band's rows, so the correction never returns to global memory.
template <int kMost>
__global__ void __launch_bounds__(kMost) k_mcsor_f32p(GridDev g, const __grid_constant__ JobTable jobs,
                                                               int nsweeps, int G, BarrierDev bar,
                                                               unsigned *phase) {
  extern __shared__ __align__(16) float sband[];
  const int nrun = (g.ntiles + G - 1) / G;
  const int jb = int(blockIdx.x) / nrun, t0 = (int(blockIdx.x) - jb * nrun) * G;
  const int t1 = (t0 + G < g.ntiles) ? t0 + G : g.ntiles;
  const JobDev &J = jobs.j[jb];
  float *e = J.e32;
  const int n8 = g.n8, nlev = g.nlev;
  const int row0 = g.tile_row0[t0], row1 = g.tile_row1[t1 - 1];
  const int f0 = ((row0 - 4) * n8) >> 2, f1 = ((row1 + 4) * n8 + 3) >> 2;
  const int fa = (row0 * n8 + 3) >> 2, fb = (row1 * n8) >> 2;  // top halo [f0, fa), bottom [fb, f1)
  const int edge_lo = (t0 > 0) ? row0 + 4 : row0, edge_hi = (t1 < g.ntiles) ? row1 - 4 : row1;
  const float4 *src = reinterpret_cast<const float4 *>(e);
  float4 *dst = reinterpret_cast<float4 *>(sband);
  float *sb = sband - 4 * f0;  // indexed by ext index
  // lanes 0..2 watch the runs above, 3..5 the runs below, whose rows reach
  // into this band's halos
  int nbq = -1;
  {
    const int lane = int(threadIdx.x), run = int(blockIdx.x) - jb * nrun;
    if (lane < 6) {
      const int q = (lane < 3) ? run - 1 - lane : run + 1 + (lane - 3);
      if (q >= 0 && q < nrun) {
        const int q0 = q * G, q1 = (q0 + G < g.ntiles) ? q0 + G : g.ntiles;
        const int r0q = g.tile_row0[q0], r1q = g.tile_row1[q1 - 1];
        if ((lane < 3 && r1q > row0 - 4) || (lane >= 3 && r0q < row1 + 4)) nbq = jb * nrun + q;
      }
    }
  }
  const float omega1 = J.omega1f;
  const float *bt = (J.kind >= 1) ? g.bpot_mu32 : g.borb_mu32;
  CoefF cf;
  for (int k = 0; k < 4; ++k) {
    cf.dmu1[k] = g.dmu1f[k];
    cf.dmu2[k] = g.dmu2f[k];
    cf.dni1[k] = g.dni1f[k];
    cf.dni2[k] = g.dni2f[k];
  }
  for (int f = f0 + int(threadIdx.x); f < f1; f += blockDim.x) dst[f - f0] = __ldcg(src + f);
  __syncthreads();
  unsigned done = 0;  // colour phases finished
  for (int s = 0; s < nsweeps; ++s) {
    for (int c = 0; c < 5; ++c) {
      if (s > 0 || c > 0) {
        if (!wait_neighbours(bar, phase, nbq, done)) return;
        for (int f = f0 + int(threadIdx.x); f < fa; f += blockDim.x) dst[f - f0] = __ldcg(src + f);
        for (int f = fb + int(threadIdx.x); f < f1; f += blockDim.x) dst[f - f0] = __ldcg(src + f);
        if (c == 0) {
          __syncthreads();
          band_boundary(g, sb, t0, t1, J.isym == 1);
        }
        __syncthreads();
      }
#pragma unroll 1
      for (int l = 0; l < nlev; ++l) {
        const int *so = g.st_off + (c * nlev + l) * (g.ntiles + 1);
        const int b0 = so[t0], b1 = so[t1];
        if (b0 == b1) continue;
        // four points per thread and pass, their list entries loaded
        // together (points of one colour and level are independent)
        for (int k0 = b0 + int(threadIdx.x); k0 < b1; k0 += 4 * int(blockDim.x)) {
          int rc[4];
          float2 p[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * int(blockDim.x);
            if (k < b1) {
              rc[u] = __ldg(g.st_pts + k);
              p[u] = __ldg(J.rw + k);
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (k0 + u * int(blockDim.x) < b1) {
              const int row = rc[u] >> 16, col = rc[u] & 0xffff, ij = row * n8 + col;
              const float v =
                  relax_f32(sb, ij, n8, cf, bt[row - 4], g.d_nu32[col - 4], p[u].y, p[u].x, omega1);
              sb[ij] = v;
              if (row < edge_lo || row >= edge_hi) e[ij] = v;
            }
          }
        }
        __syncthreads();
      }
      // publish the finished phase (the level loop ended with a block barrier)
      ++done;
      if (threadIdx.x == 0) {
        __threadfence();
        st_release(phase + size_t(blockIdx.x) * kPhaseStride, done);
      }
    }
  }
  // u += e on the band's interior rows, then the FP64 axis values of u on
  // the band's rows (sormcsor.F90:94-129; the axis points read only the
  // band's own rows)
  double *u = J.u;
  const int ra = (row0 > 5) ? row0 : 5, ncol = g.nni - 2, total = (row1 - ra) * ncol;
  for (int k0 = threadIdx.x; k0 < total; k0 += 8 * int(blockDim.x)) {
    // eight loads of u in flight per thread before the adds
    int ij[8];
    double uv[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int k = k0 + q * int(blockDim.x);
      ij[q] = -1;
      if (k < total) {
        ij[q] = (ra + k / ncol) * n8 + 5 + k % ncol;
        uv[q] = __ldcg(u + ij[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (ij[q] >= 0) u[ij[q]] = uv[q] + widen_f32(sb[ij[q]]);
  }
  __syncthreads();
  const bool even = (J.isym == 1);
  const int nrow7 = (t0 == 0) ? g.nni - 2 : 0, nside = 2 * (row1 - ra);
  for (int k = threadIdx.x; k < nrow7 + nside; k += blockDim.x) {
    if (k < nrow7) {
      const int ij = 4 * n8 + 5 + k;
      u[ij] = even ? extrap64(g, u, ij, n8) : 0.0;
    } else {
      const int q = k - nrow7, r = ra + q / 2, side = q % 2;
      const int ij = r * n8 + (side == 0 ? 4 : g.nni + 3);
      u[ij] = even ? extrap64(g, u, ij, side == 0 ? 1 : -1) : 0.0;
    }
  }
  if (t0 == 0) {
    __syncthreads();
    if (threadIdx.x < 2) {
      const int ij = 4 * n8 + (threadIdx.x == 0 ? 4 : g.nni + 3);
      u[ij] = even ? extrap64(g, u, ij, threadIdx.x == 0 ? 1 : -1) : 0.0;
    }
  }
}

// ----------------------------------------------------------------------
// Mixed form: ghost refresh, FP64 residual, FP32 correction, FP64 update.
// ----------------------------------------------------------------------
__device__ __forceinline__ void ghost_point(const GridDev &g, double *u, int k, int isym) {
  // k indexes (rows 4..nmu+3) x 8 ghost columns, then 4 ghost rows x nni
  const int nrows = g.nmu;
  const bool neg = (isym != 1);
  if (k < nrows * 8) {
    const int r = 4 + k / 8, q = k % 8, base = r * g.n8;
    if (q < 4) {
      const int j = q + 1;
      const double v = u[base + 4 + j];
      u[base + 4 - j] = neg ? -v : v;
    } else {
      const int j = q - 3;
      const double v = u[base + g.nni + 3 - j];
      u[base + g.nni + 3 + j] = neg ? -v : v;
    }
  } else {
    k -= nrows * 8;
    const int i = k / g.nni + 1, col = 4 + k % g.nni;
    const double v = u[(4 + i) * g.n8 + col];
    u[(4 - i) * g.n8 + col] = neg ? -v : v;
  }
}

// ----------------------------------------------------------------------
// Elementwise kernels of the SCF path
// ----------------------------------------------------------------------
__global__ void k_ghost(GridDev g, double *u, int isym) {
  const int n = g.nmu * 8 + 4 * g.nni;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) ghost_point(g, u, k, isym);
}

__global__ void k_putin_interior(GridDev g, const double *plain, double *ext) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    ext[(mu + 4) * g.n8 + nu + 4] = plain[k];
  }
}

__global__ void k_putout(GridDev g, const double *ext, double *plain) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    plain[k] = ext[(mu + 4) * g.n8 + nu + 4];
  }
}

// fockHF (src/fock.F90:57-186), per grid point: exact keeps the reference's
// unfused order, otherwise (mixed form) products are fused into FMAs.
template <bool exact>
__device__ __forceinline__ double madd(double a, double b, double c) {  // a*b + c
  if (exact) return A(M(a, b), c);
  return fma(a, b, c);
}

template <bool exact>
__device__ __forceinline__ void fock_point(const GridDev &g, const FockArgs &a, double ee, int k) {
  const int mu = k / g.nni, nu = k - mu * g.nni;
  const int ij = (mu + 4) * g.n8 + nu + 4;
  double fock1 = g.f0[k];
  fock1 = madd<exact>(ee, g.f1[k], fock1);
  if (a.m != 0) fock1 = madd<exact>(double(a.m * a.m), g.e[k], fock1);
  double fock2 = 0.0;
  if (!a.nel1) {
    double wk1 = 0.0;
    for (int q = 0; q < a.nterms; ++q) {
      const FockTerm &T = a.t[q];
      wk1 = madd<exact>(T.coo, T.coul[ij], wk1);
      if (T.mode == 0) {
        double wk2 = M(T.gec, T.ex[ij]);
        if (T.ex2) wk2 = madd<exact>(T.gec2, T.ex2[ij], wk2);
        fock2 = madd<exact>(wk2, T.psi[ij], fock2);
      } else if (T.mode == 1) {
        const double wk2 = M(T.ex[ij], T.psi[ij]);
        fock2 = madd<exact>(T.gec, wk2, fock2);
      }
    }
    a.coulp[k] = wk1;
    a.exchp[k] = fock2;
    fock2 = M(fock2, g.f2[k]);
    fock1 = madd<exact>(wk1, g.f2[k], fock1);
  }
  a.lhs[k] = A(fock1, g.diag);
  a.rhs[k] = fock2;
  if (mu >= g.nmu - 5) {
    const double f1 = g.f1[k];
    a.fa[(mu - (g.nmu - 5)) * g.nni + nu] = (fabs(f1) <= kPrecis) ? 0.0 : D(fock1, f1);
  }
}

template <bool exact>
__global__ void k_fock(GridDev g, FockArgs a) {
  const double ee = *a.ee;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x)
    fock_point<exact>(g, a, ee, k);
}

// the Fock builds of several orbitals from the same state, orbital blockIdx.y
constexpr int kFockBatch = 8;
struct FockBatch {
  FockArgs a[kFockBatch];
};
template <bool exact>
__global__ void k_fock_batch(GridDev g, const __grid_constant__ FockBatch B) {
  const FockArgs &a = B.a[blockIdx.y];
  const double ee = *a.ee;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x)
    fock_point<exact>(g, a, ee, k);
}

// orbAsymptGet (relaxOrbs.F90:415-437): edecay for mu = nmu-4..nmu-1 (0-based)
__global__ void k_asympt_get(GridDev g, const double *fa, double *edecay) {
  const int n = 4 * g.nni;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int jj = k / g.nni, i = k - jj * g.nni;
    const int j = g.nmu - 4 + jj;  // 0-based mu
    (void)j;
    // raiq1 - raiq from the grid's table; x**0.25 as sqrt(sqrt(x))
    const double dr = g.asy[size_t(50) * n + k];
    const double fj = fa[(jj + 1) * g.nni + i], fjm = fa[jj * g.nni + i];
    edecay[k] = sqrt(sqrt(fabs(fj / fjm))) * exp(sqrt(fabs(fjm)) * dr);
  }
}

// orbAsymptSet (relaxOrbs.F90:444-462), rows in order
__global__ void k_asympt_set(GridDev g, double *psi, const double *edecay) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.nni; i += gridDim.x * blockDim.x) {
    for (int jj = 0; jj < 4; ++jj) {
      const int j = g.nmu - 4 + jj;
      const int ij = (j + 4) * g.n8 + i + 4;
      psi[ij] = M(psi[ij - g.n8], edecay[jj * g.nni + i]);
    }
  }
}

// orbAsymptGet / orbAsymptSet of several orbitals, orbital blockIdx.y
__global__ void k_asympt_get_batch(GridDev g, const __grid_constant__ OrbDecayList L) {
  const int n = 4 * g.nni, o = blockIdx.y;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int jj = k / g.nni, i = k - jj * g.nni;
    const double dr = g.asy[size_t(50) * n + k];
    const double fj = L.fa[o][(jj + 1) * g.nni + i], fjm = L.fa[o][jj * g.nni + i];
    L.edecay[o][k] = sqrt(sqrt(fabs(fj / fjm))) * exp(sqrt(fabs(fjm)) * dr);
  }
}
__global__ void k_asympt_set_batch(GridDev g, const __grid_constant__ OrbDecayList L) {
  const int o = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.nni; i += gridDim.x * blockDim.x)
    for (int jj = 0; jj < 4; ++jj) {
      const int j = g.nmu - 4 + jj;
      const int ij = (j + 4) * g.n8 + i + 4;
      L.psi[o][ij] = M(L.psi[o][ij - g.n8], L.edecay[o][jj * g.nni + i]);
    }
}

// setCiOrb (scfUtils.F90:380-434)
__global__ void k_setci(GridDev g, double *psi, int ihomo) {
  const int n2 = g.nni / 2 + 1;
  const int n = (n2 - 1) * g.nmu;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int mu = k / (n2 - 1), ni = k - mu * (n2 - 1);  // ni 0-based = reference ni-1
    const int row = (mu + 4) * g.n8 + 4;
    const double v = psi[row + ni];
    psi[row + (g.nni - 1 - ni)] = (ihomo == 1) ? v : -v;
  }
  if (ihomo != 1) {
    for (int mu = blockIdx.x * blockDim.x + threadIdx.x; mu < g.nmu; mu += gridDim.x * blockDim.x)
      psi[(mu + 4) * g.n8 + 4 + (n2 - 1)] = 0.0;
  }
}

// norm scaling: psi = (1/sqrt(xnorm)) psi over the plain region (normOrtho.F90:50-52)
__global__ void k_scale(GridDev g, double *psi, const double *xnorm) {
  const double zarea = D(1.0, sqrt(*xnorm));
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * g.n8 + nu + 4;
    psi[ij] = M(zarea, psi[ij]);
  }
}

// norm scaling followed by setCiOrb (normOrtho.F90:50-52, scfUtils.F90:380-
// 434) in one pass: the left half of each row is scaled and mirrored, the
// middle column scaled (gerade) or zeroed (ungerade)
__global__ void k_scale_setci(GridDev g, double *psi, const double *xnorm, int ihomo) {
  const double zarea = D(1.0, sqrt(*xnorm));
  const int n2 = g.nni / 2 + 1;
  const int n = n2 * g.nmu;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int mu = k / n2, ni = k - mu * n2;
    const int row = (mu + 4) * g.n8 + 4;
    if (ni < n2 - 1) {
      const double v = M(zarea, psi[row + ni]);
      psi[row + ni] = v;
      psi[row + (g.nni - 1 - ni)] = (ihomo == 1) ? v : -v;
    } else {
      psi[row + ni] = (ihomo == 1) ? M(zarea, psi[row + ni]) : 0.0;
    }
  }
}

struct PtrList {
  const double *p[kMaxTerms];
};

// Gram-Schmidt step of ortho (normOrtho.F90:175-188)
__global__ void k_ortho_apply(GridDev g, double *psi, PtrList others, int n, const double *ovl) {
  double ano = 0.0;
  for (int q = 0; q < n; ++q) ano = A(ano, M(ovl[q], ovl[q]));
  ano = D(sqrt(A(1.0, ano)), S(1.0, M(ano, ano)));
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * g.n8 + nu + 4;
    double v = psi[ij];
    for (int q = 0; q < n; ++q) v = A(M(-ovl[q], others.p[q][ij]), v);
    psi[ij] = M(ano, v);
  }
}

// vexch/mulex normalised associated Legendre functions P_k^q(cos th) for
// k = 1..mpole (scfUtils.F90:856-1270).  legacy_m3 reproduces vexch's m=3
// branch, which uses sin^2 in place of sin.
__device__ void assoc_legendre(int mt, int mpole, double costh, double *dome, bool legacy_m3) {
  for (int k = 0; k < 10; ++k) dome[k] = 0.0;
  if (mt > 4) return;
  double c2, c4, c6, c8, si, si2, si3;
  if (mt == 0) {
    dome[1] = costh;
    dome[2] = (3.0 * costh * costh - 1.0) * 0.50;
    for (int n = 2; n <= mpole - 1; n++)
      dome[n + 1] = (double(2 * n + 1) * costh * dome[n] - double(n) * dome[n - 1]) / double(n + 1);
  } else if (mt == 1) {
    c2 = costh * costh;
    si2 = fabs(1.0 - c2);
    si = sqrt(si2);
    c4 = c2 * c2;
    c6 = c4 * c2;
    dome[1] = -si / sqrt(2.0);
    dome[2] = -3.0 * si * costh / sqrt(6.0);
    dome[3] = (3.0 / 2.0) * si * (1.0 - 5.0 * c2) / sqrt(12.0);
    dome[4] = (5.0 / 2.0) * si * costh * (3.0 - 7.0 * c2) / sqrt(20.0);
    dome[5] = (15.0 / 8.0) * si * (-1.0 + 14.0 * c2 - 21.0 * c4) / sqrt(30.0);
    dome[6] = (21.0 / 8.0) * si * costh * (-5.0 + 30.0 * c2 - 33.0 * c4) / sqrt(42.0);
    dome[7] = (7.0 / 16.0) * si * (5.0 - 135.0 * c2 + 495.0 * c4 - 429.0 * c6) / sqrt(56.0);
    dome[8] = (9.0 / 16.0) * si * costh * (35.0 - 385.0 * c2 + 1001.0 * c4 - 715.0 * c6) / sqrt(72.0);
  } else if (mt == 2) {
    c2 = costh * costh;
    si2 = fabs(1.0 - c2);
    c4 = c2 * c2;
    c6 = c4 * c2;
    c8 = c6 * c2;
    dome[2] = 3.0 * si2 / sqrt(24.0);
    dome[3] = 15.0 * costh * si2 / sqrt(120.0);
    dome[4] = (15.0 / 2.0) * (-1.0 + 8.0 * c2 - 7.0 * c4) / sqrt(360.0);
    dome[5] = (105.0 / 2.0) * costh * (-1.0 + 4.0 * c2 - 3.0 * c4) / sqrt(840.0);
    dome[6] = (105.0 / 8.0) * (1.0 - 19.0 * c2 + 51.0 * c4 - 33.0 * c6) / sqrt(1680.0);
    dome[7] = (63.0 / 8.0) * costh * (15.0 - 125.0 * c2 + 253.0 * c4 - 143.0 * c6) / sqrt(3024.0);
    dome[8] = (315.0 / 8.0) * (-1.0 + 34.0 * c2 - 176.0 * c4 + 286.0 * c6 - 143.0 * c8) / sqrt(5040.0);
  } else if (mt == 3) {
    c2 = costh * costh;
    si2 = fabs(1.0 - c2);
    si = legacy_m3 ? si2 : sqrt(si2);
    si3 = si2 * si;
    c4 = c2 * c2;
    dome[3] = -15.0 * si3 / sqrt(720.0);
    dome[4] = -105.0 * si3 * costh / sqrt(5040.0);
    dome[5] = -(105.0 / 2.0) * si3 * (-1.0 + 9.0 * c2) / sqrt(20160.0);
    dome[6] = -(315.0 / 2.0) * si3 * costh * (-3.0 + 11.0 * c2) / sqrt(60480.0);
    dome[7] = -(315.0 / 8.0) * si3 * (3.0 - 66.0 * c2 + 143.0 * c4) / sqrt(151200.0);
    dome[8] = -(3465.0 / 8.0) * si3 * costh * (3.0 - 26.0 * c2 + 39.0 * c4) / sqrt(332640.0);
  } else if (mt == 4) {
    c2 = costh * costh;
    c4 = c2 * c2;
    c6 = c4 * c2;
    c8 = c6 * c2;
    dome[4] = 105.0 * (1.0 - 2.0 * c2 + c4) / sqrt(40320.0);
    dome[5] = 945.0 * costh * (1.0 - 2.0 * c2 + c4) / sqrt(362880.0);
    dome[6] = (945.0 / 2.0) * (-1.0 + 13 * c2 - 23.0 * c4 + 11.0 * c6) / sqrt(1814400.0);
    dome[7] = (3465.0 / 2.0) * costh * (-3.0 + 19 * c2 - 29.0 * c4 + 13.0 * c6) / sqrt(6652800.0);
    dome[8] = (10395.0 / 8.0) * (1.0 - 28.0 * c2 + 118.0 * c4 - 156.0 * c6 + 65.0 * c8) / sqrt(19958400.0);
  }
  for (int k = mpole + 1; k <= 8; ++k) dome[k] = 0.0;
}

// Moment tables of a grid: exchange moment weights over the plain grid and
// the boundary functions of potAsympt on mu = nmu-4..nmu-1 (0-based),
// evaluated once per grid with the formulas of coulAsympt/vcoul,
// exchAsympt/vexch and exchMom (scfUtils.F90:615-1270).
__global__ void k_moment_tables(GridDev g, double *exm, double *asy) {
  const int stride = gridDim.x * blockDim.x;
  double dome[10];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += stride) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const double rr = sqrt(g.vxisq[mu] + g.vetasq[nu] - 1.0);
    const double xrr = g.r2 * rr;
    const double costh = (fabs(rr) > kPrecis) ? g.veta[nu] * g.vxi[mu] / rr : 0.0;
    const double wk = g.wgt2[k] * g.f4[k];
    for (int idel = 0; idel <= 4; ++idel) {
      assoc_legendre(idel, g.mpole, costh, dome, false);
      double xw = xrr;
      for (int q = 0; q < g.mpole; ++q) {
        if (q > 0) xw = xw * xrr;
        exm[(size_t(idel) * 8 + q) * g.mxsize + k] = wk * (dome[q + 1] * xw);
      }
    }
  }
  const int P = 4 * g.nni;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += stride) {
    const int jj = p / g.nni, i = p - jj * g.nni, j = g.nmu - 4 + jj;
    const double rr = sqrt(g.vxisq[j] + g.vetasq[i] - 1.0);
    asy[p] = g.r2 * g.vxi[j];
    asy[size_t(50) * P + p] = sqrt(g.vxisq[j - 1] + g.vetasq[i] - 1.0) - rr;  // orbAsymptGet's raiq1 - raiq
    const double rr1 = 1.0 / (rr * g.r2);
    asy[P + p] = rr1;
    const double costh = g.veta[i] * g.vxi[j] / rr;
    dome[1] = costh;
    dome[2] = (3.0 * costh * costh - 1.0) * 0.5;
    for (int m = 2; m <= g.mpole - 1; m++)
      dome[m + 1] = (double(2 * m + 1) * costh * dome[m] - double(m) * dome[m - 1]) / double(m + 1);
    double rp = rr1;
    for (int m = 1; m <= 8; m++) {
      rp = rp * rr1;
      asy[size_t(2 + m - 1) * P + p] = (m <= g.mpole) ? dome[m] * rp : 0.0;
    }
    const double costx = (fabs(rr) > kPrecis) ? costh : 0.0;
    const double rs = rr * g.r2;
    for (int idel = 0; idel <= 4; ++idel) {
      assoc_legendre(idel, g.mpole, costx, dome, true);  // vexch's m=3 branch
      double xrn = rs;
      for (int m = 1; m <= 8; m++) {
        xrn = xrn * rs;
        asy[size_t(10 + idel * 8 + m - 1) * P + p] = (m <= g.mpole) ? dome[m] / xrn : 0.0;
      }
    }
  }
}

// potAsympt: Coulomb (coulAsympt/vcoul) and exchange (exchAsympt/vexch)
// boundary values on mu = nmu-4..nmu-1 (0-based) from the grid's tables.
__global__ void k_asympt(GridDev g, AsymptArgs a) {
  const AsymptItem &it = a.it[blockIdx.y];
  const int P = 4 * g.nni;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x) {
    const int jj = p / g.nni, i = p - jj * g.nni;
    const int ij = (g.nmu + jj) * g.n8 + i + 4;
    double pe = 0.0;
    if (it.type == 0) {
      const double *cm = a.cmulti + it.idx * 8;
      for (int m = 1; m <= g.mpole; m++) pe = fma(cm[m - 1], g.asy[size_t(1 + m) * P + p], pe);
      pe = g.asy[P + p] + pe;
    } else if (it.idel <= 4) {
      const double *xm = a.excm + it.idx * 8;
      const double *X = g.asy + size_t(10 + it.idel * 8) * P + p;
      for (int m = 1; m <= g.mpole; m++) pe = fma(X[size_t(m - 1) * P], xm[m - 1], pe);
    }
    it.pot[ij] = g.asy[p] * pe;
  }
}

__global__ void k_zero(double *p, size_t n) {
  for (size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x; k < n; k += size_t(gridDim.x) * blockDim.x) p[k] = 0.0;
}

// ----------------------------------------------------------------------
// Deterministic reductions: fixed grid -> per-block partials -> the last
// block to finish sums the partials in block order.
// ----------------------------------------------------------------------
constexpr int kRedBlocks = 160, kRedBlocksMax = 608;
// blocks of a single-launch reduction over the grid: 160 up to ~160k
// points, one per 1024 points above that (more loads in flight on large
// grids), at most 608; fixed per grid, so every sum runs in the same order
// on every call
inline int red_blocks(const GridDev &g) {
  const int b = g.mxsize / 1024;
  return b < kRedBlocks ? kRedBlocks : (b > kRedBlocksMax ? kRedBlocksMax : b);
}
constexpr int kMaxK = 16;

// The sums over a warp of P values each (a power of two up to 16): lane q 32 /
// P returns that of v[q].  At every halving of the tree the two lanes of a pair
// also share the values left, so P values take P - 1 + log2(32 / P) additions
// and not 5 P; each value's tree and its roundings are those of a shuffle tree
// by itself (additions only swap their operands).
template <int P>
__device__ __forceinline__ double warp_sums(double (&x)[P]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int n = P; n > 1; n /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < n / 2; ++j) {
      const double keep = up ? x[j + n / 2] : x[j], send = up ? x[j] : x[j + n / 2];
      x[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = x[0];
#pragma unroll
  for (; o > 0; o /= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The block's sums of K values, value q < n of block b to base[b bstride + q
// qstride].  FP64 additions bound the reductions (the trees of 16 values took
// 80 a warp, 19 cycles each of the SM's pipe).
template <int K>
__device__ void block_sum_store(double (&v)[K], double *base, int bstride, int qstride, int n = K) {
  constexpr int P = K == 1 ? 1 : K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : 16;
  __shared__ double sh[kThreads / 32][P];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double x[P];
#pragma unroll
  for (int q = 0; q < P; ++q) x[q] = q < K ? v[q] : 0.0;
  const double sum = warp_sums<P>(x);
  if (lane % (32 / P) == 0) sh[w][lane / (32 / P)] = sum;
  __syncthreads();
  if (threadIdx.x < n) {
    double s = 0.0;
    for (int i = 0; i < kThreads / 32; ++i) s += sh[i][threadIdx.x];
    base[size_t(blockIdx.x) * bstride + size_t(threadIdx.x) * qstride] = s;
  }
}
template <int K>
__device__ void block_sum_store(double (&v)[K], double *partials) {
  block_sum_store<K>(v, partials, K, 1);
}

// Every block stores its K partial sums; the block that finishes last (an
// atomic ticket, reset by that block) sums the partials of all blocks in
// block order -- the same order on every run -- and
// writes out[0..nout).  Returns true in that block.  No block waits for
// another.
// The sums over the blocks of nq <= kMaxK slots, slot q of block b at base[b *
// bstride + q * qstride]: thread t adds blocks t, t + blockDim, ..., then a
// warp tree, then the warp totals in warp order.  out[] in shared memory, valid
// in every thread on return
__device__ void sum_partials_multi(const double *base, int bstride, int qstride, int nq, int nblocks, double *out) {
  __shared__ double sh[kThreads / 32][kMaxK];
  double s[kMaxK];
#pragma unroll
  for (int q = 0; q < kMaxK; ++q) s[q] = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
#pragma unroll
    for (int q = 0; q < kMaxK; ++q)
      if (q < nq) s[q] += __ldcg(base + size_t(b) * bstride + size_t(q) * qstride);
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (nq <= 3) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double x[1] = {s[q]};
      if (q < nq) x[0] = warp_sums<1>(x);
      if (q < nq && lane == 0) sh[w][q] = x[0];
    }
  } else {
    const double sum = warp_sums<kMaxK>(s);
    if (lane % (32 / kMaxK) == 0) sh[w][lane / (32 / kMaxK)] = sum;
  }
  __syncthreads();
  if (threadIdx.x < nq) {
    double t = 0.0;
    for (int i = 0; i < kThreads / 32; ++i) t += sh[i][threadIdx.x];
    out[threadIdx.x] = t;
  }
  __syncthreads();
}

template <int K>
__device__ bool block_sum_finish(double (&v)[K], double *partials, double *out, int nout, unsigned *ticket) {
  __shared__ bool s_last;
  block_sum_store<K>(v, partials);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!s_last) return false;
  __threadfence();
  __shared__ double s_out[kMaxK];
  sum_partials_multi(partials, K, 1, nout, int(gridDim.x), s_out);
  if (threadIdx.x == 0) {
    for (int q = 0; q < nout; ++q) out[q] = s_out[q];
    *ticket = 0u;
  }
  return true;
}

__global__ void k_norm(GridDev g, const double *psi, double *partials, double *out, unsigned *ticket) {
  double v[1] = {0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const double p = psi[(mu + 4) * g.n8 + nu + 4];
    v[0] += g.wgt2[k] * M(M(p, p), g.f4[k]);
  }
  block_sum_finish<1>(v, partials, out, 1, ticket);
}

__global__ void k_overlaps(GridDev g, const double *psi, PtrList o, int n, double *partials, double *out,
                           unsigned *ticket) {
  double v[kMaxK];
  for (int q = 0; q < kMaxK; ++q) v[q] = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * g.n8 + nu + 4;
    const double p = psi[ij], w = g.wgt2[k], f4 = g.f4[k];
    for (int q = 0; q < n; ++q) v[q] += w * M(M(p, o.p[q][ij]), f4);
  }
  block_sum_finish<kMaxK>(v, partials, out, n, ticket);
}

// One round of the orthonormalisation of several orbitals (normOrtho.F90:
// 14-59, 103-207, scfUtils.F90:380-434): orbital blockIdx.y of the round's
// list.  Each orbital's sums run over the same blocks in the same order as
// k_norm / k_overlaps, so the results equal the one-orbital launches.
constexpr int kRoundItems = 12;
struct OrthoItem {
  double *psi;
  const double *o[kMaxK];  // orthogonalisation partners (normalised earlier)
  int n;                   // number of partners
  int ihomo;               // 0: scale only; +-1: scale and setCiOrb
  double *norm_out;        // sum wgt2 psi psi f4
  double *ovl_out;         // overlaps with the partners
};
struct OrthoRound {
  OrthoItem it[kRoundItems];
};

__global__ void k_norm_round(GridDev g, const __grid_constant__ OrthoRound R, double *partials, unsigned *tickets) {
  const OrthoItem &I = R.it[blockIdx.y];
  double v[1] = {0.0};
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const double p = I.psi[(mu + 4) * g.n8 + nu + 4];
    v[0] += g.wgt2[k] * M(M(p, p), g.f4[k]);
  }
  block_sum_finish<1>(v, partials + size_t(blockIdx.y) * gridDim.x, I.norm_out, 1, tickets + blockIdx.y);
}

__global__ void k_scale_round(GridDev g, const __grid_constant__ OrthoRound R) {
  const OrthoItem &I = R.it[blockIdx.y];
  const double zarea = D(1.0, sqrt(*I.norm_out));
  if (I.ihomo == 0) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
      const int mu = k / g.nni, nu = k - mu * g.nni;
      const int ij = (mu + 4) * g.n8 + nu + 4;
      I.psi[ij] = M(zarea, I.psi[ij]);
    }
    return;
  }
  const int n2 = g.nni / 2 + 1;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n2 * g.nmu; k += gridDim.x * blockDim.x) {
    const int mu = k / n2, ni = k - mu * n2;
    const int row = (mu + 4) * g.n8 + 4;
    if (ni < n2 - 1) {
      const double v = M(zarea, I.psi[row + ni]);
      I.psi[row + ni] = v;
      I.psi[row + (g.nni - 1 - ni)] = (I.ihomo == 1) ? v : -v;
    } else {
      I.psi[row + ni] = (I.ihomo == 1) ? M(zarea, I.psi[row + ni]) : 0.0;
    }
  }
}

__global__ void k_overlaps_round(GridDev g, const __grid_constant__ OrthoRound R, double *partials,
                                 unsigned *tickets) {
  const OrthoItem &I = R.it[blockIdx.y];
  double v[kMaxK];
  for (int q = 0; q < kMaxK; ++q) v[q] = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * g.n8 + nu + 4;
    const double p = I.psi[ij], w = g.wgt2[k], f4 = g.f4[k];
    for (int q = 0; q < I.n; ++q) v[q] += w * M(M(p, I.o[q][ij]), f4);
  }
  block_sum_finish<kMaxK>(v, partials + size_t(blockIdx.y) * gridDim.x * kMaxK, I.ovl_out, I.n,
                          tickets + blockIdx.y);
}

__global__ void k_ortho_round(GridDev g, const __grid_constant__ OrthoRound R) {
  const OrthoItem &I = R.it[blockIdx.y];
  const double *ovl = I.ovl_out;
  double ano = 0.0;
  for (int q = 0; q < I.n; ++q) ano = A(ano, M(ovl[q], ovl[q]));
  ano = D(sqrt(A(1.0, ano)), S(1.0, M(ano, ano)));
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * g.n8 + nu + 4;
    double v = I.psi[ij];
    for (int q = 0; q < I.n; ++q) v = A(M(-ovl[q], I.o[q][ij]), v);
    I.psi[ij] = M(ano, v);
  }
}

// Every round of an iteration's orthonormalisation in one cooperative
// launch: the norms and scalings (and setCiOrb) of every orbital, then per
// round the overlaps with the partners and the Gram-Schmidt step of each of
// its orbitals, separated by grid barriers.  Each block stores the same per-block partial
// sums as k_norm_round / k_overlaps_round (same blocks, same points, same
// order) and every block adds them up in the order of block_sum_finish, so
// the results equal the per-round launches bit for bit.
constexpr int kOrthoItems = 32, kOrthoRounds = 16;
struct OrthoPlan {
  OrthoItem it[kOrthoItems];
  int round_off[kOrthoRounds + 1];
  int nrounds;
};

// The phases below take up to kGroup orbitals (or orbital-partner pairs) of
// a round in one pass over the points, so that their loads are in flight
// together; each orbital's (pair's) per-thread sum still runs over the same
// points in the same order, and block_sum_store reduces every slot the same
// way whatever the number of slots stored, so the sums are those of the
// one-orbital kernels.
constexpr int kGroup = 8;

// scaling (and setCiOrb) of items [a, b) of the plan with zarea[j]
__device__ void scale_items(const GridDev &g, const OrthoPlan &P, int a, int b, const double *zarea) {
  const int stride = gridDim.x * blockDim.x, n2 = g.nni / 2 + 1;
  const int homo = P.it[a].ihomo != 0;  // one kind per call (the caller groups them)
  const int n = homo ? n2 * g.nmu : g.mxsize;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
      if (a + j >= b) break;
      const OrthoItem &I = P.it[a + j];
      if (!homo) {
        const int mu = k / g.nni, nu = k - mu * g.nni;
        const int ij = (mu + 4) * g.n8 + nu + 4;
        I.psi[ij] = M(zarea[j], I.psi[ij]);
      } else {
        const int mu = k / n2, ni = k - mu * n2;
        const int row = (mu + 4) * g.n8 + 4;
        if (ni < n2 - 1) {
          const double v = M(zarea[j], I.psi[row + ni]);
          I.psi[row + ni] = v;
          I.psi[row + (g.nni - 1 - ni)] = (I.ihomo == 1) ? v : -v;
        } else {
          I.psi[row + ni] = (I.ihomo == 1) ? M(zarea[j], I.psi[row + ni]) : 0.0;
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_orthonormalise(GridDev g, const __grid_constant__ OrthoPlan P,
                                                             double *partials, BarrierDev bar) {
  __shared__ double s_val[kGroup * kMaxK];
  __shared__ int s_item[kMaxK], s_q[kMaxK];
  const int nb = int(gridDim.x);
  // An orbital is changed only in its own round, after its partners'
  // rounds: its norm and scaling read nothing another round writes, so the
  // norms and scalings of every round run first, in one pass, and the rounds
  // keep only their overlaps and Gram-Schmidt steps.
  const int n = P.round_off[P.nrounds];
  for (int a = 0; a < n; a += kGroup) {
    double v[kGroup];
#pragma unroll
    for (int j = 0; j < kGroup; ++j) v[j] = 0.0;
#pragma unroll 4
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
      const int mu = k / g.nni, nu = k - mu * g.nni;
      const int ij = (mu + 4) * g.n8 + nu + 4;
      const double w2 = g.wgt2[k], f4 = g.f4[k];
#pragma unroll
      for (int j = 0; j < kGroup; ++j) {
        if (a + j >= n) break;
        const double p = P.it[a + j].psi[ij];
        v[j] += w2 * M(M(p, p), f4);
      }
    }
    block_sum_store<kGroup>(v, partials + size_t(a) * nb, 1, nb, min(kGroup, n - a));
    __syncthreads();
  }
  __threadfence();
  if (!grid_barrier(bar, unsigned(nb))) return;
  // totals (every block, in block order), then the scaling, grouped by kind
  for (int a = 0; a < n;) {
    int b = a;
    while (b < n && b - a < kGroup && (P.it[b].ihomo != 0) == (P.it[a].ihomo != 0)) ++b;
    double zarea[kGroup];
    sum_partials_multi(partials + size_t(a) * nb, 1, nb, b - a, nb, s_val);
    for (int j = 0; j < b - a; ++j) {
      const double norm = s_val[j];
      if (blockIdx.x == 0 && threadIdx.x == 0) *P.it[a + j].norm_out = norm;
      zarea[j] = D(1.0, sqrt(norm));
    }
    __syncthreads();  // s_val is reused below
    scale_items(g, P, a, b, zarea);
    a = b;
  }
  for (int r = 0; r < P.nrounds; ++r) {
    const int i0 = P.round_off[r], i1 = P.round_off[r + 1];
    bool partners = false;
    for (int i = i0; i < i1; ++i) partners = partners || P.it[i].n > 0;
    if (!partners) continue;
    // the scalings and the earlier rounds' Gram-Schmidt steps done
    // everywhere before this round's overlaps
    __threadfence();
    if (!grid_barrier(bar, unsigned(nb))) return;
    // overlaps: (item, partner) slots of the round, kMaxK at a time; values
    // other blocks wrote in this launch are read through L2
    int slot0 = 0;
    for (int i = i0; i < i1;) {
      // a slot group: at most kGroup items and kMaxK (item, partner) slots
      int nslot = 0, iend = i;
      while (iend < i1 && iend - i < kGroup && nslot + P.it[iend].n <= kMaxK) nslot += P.it[iend++].n;
      if (iend == i) break;  // an item alone has at most kMaxK partners
      if (threadIdx.x == 0) {
        int t = 0;
        for (int x = i; x < iend; ++x)
          for (int q = 0; q < P.it[x].n; ++q, ++t) {
            s_item[t] = x;
            s_q[t] = q;
          }
      }
      __syncthreads();
      double v[kMaxK];
#pragma unroll
      for (int t = 0; t < kMaxK; ++t) v[t] = 0.0;
      for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
        const int mu = k / g.nni, nu = k - mu * g.nni;
        const int ij = (mu + 4) * g.n8 + nu + 4;
        const double w = g.wgt2[k], f4 = g.f4[k];
#pragma unroll
        for (int t = 0; t < kMaxK; ++t) {
          if (t >= nslot) break;
          const OrthoItem &I = P.it[s_item[t]];
          const double p = __ldcg(I.psi + ij);
          v[t] += w * M(M(p, __ldcg(I.o[s_q[t]] + ij)), f4);
        }
      }
      block_sum_store<kMaxK>(v, partials + size_t(slot0) * nb);
      __syncthreads();
      slot0 += kMaxK;
      i = iend;
    }
    __threadfence();
    if (!grid_barrier(bar, unsigned(nb))) return;
    // totals, then the Gram-Schmidt step of up to kGroup items at a time
    slot0 = 0;
    for (int i = i0; i < i1;) {
      int nslot = 0, iend = i;
      while (iend < i1 && iend - i < kGroup && nslot + P.it[iend].n <= kMaxK) nslot += P.it[iend++].n;
      if (iend == i) break;
      {
        __shared__ double tot[kMaxK];
        sum_partials_multi(partials + size_t(slot0) * nb, kMaxK, 1, nslot, nb, tot);
        if (threadIdx.x == 0)
          for (int x = i, t = 0; x < iend; ++x)
            for (int q = 0; q < P.it[x].n; ++q, ++t) {
              s_val[(x - i) * kMaxK + q] = tot[t];
              if (blockIdx.x == 0) P.it[x].ovl_out[q] = tot[t];
            }
      }
      __syncthreads();
      {
        const int a = i, b = iend;
        double ano[kGroup];
        for (int j = 0; j < b - a; ++j) {
          const OrthoItem &I = P.it[a + j];
          const double *ovl = s_val + j * kMaxK;
          double x = 0.0;
          for (int q = 0; q < I.n; ++q) x = A(x, M(ovl[q], ovl[q]));
          ano[j] = D(sqrt(A(1.0, x)), S(1.0, M(x, x)));
        }
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
          const int mu = k / g.nni, nu = k - mu * g.nni;
          const int ij = (mu + 4) * g.n8 + nu + 4;
#pragma unroll
          for (int j = 0; j < kGroup; ++j) {
            if (a + j >= b) break;
            const OrthoItem &I = P.it[a + j];
            if (I.n == 0) continue;
            const double *ovl = s_val + j * kMaxK;
            double v = __ldcg(I.psi + ij);
            for (int q = 0; q < I.n; ++q) v = A(M(-ovl[q], __ldcg(I.o[q] + ij)), v);
            I.psi[ij] = M(ano[j], v);
          }
        }
      }
      __syncthreads();
      slot0 += kMaxK;
      i = iend;
    }
  }
}

// The same orthonormalisation through the inner products of the orbitals
// (one pass over the points, one grid barrier, one pass applying the
// result).  With Z_j the orbital after setCiOrb (homonuclear: the first half
// of each row mirrored onto the second, the sign by g/u) and <a,b> = sum
// wgt2 f4 a b, the loop "scale orbital j by 1/sqrt(<X_j,X_j>) (then setCiOrb),
// then Gram-Schmidt against its partners Y_q" (normOrtho.F90:14-59,
// 103-207) makes every final orbital a combination Y_j = sum_m C_jm Z_m of
// the orbitals of its symmetry block, and the loop's overlaps are
//   ovl_q = zarea_j sum_m C_qm <Z_j, Z_m>,
// so C, the norms and the overlaps follow exactly from the Gram matrix, in
// the reference's orbital order.  Equal to the loop in exact arithmetic; the
// rounding differs (the loop's sums of the scaled, partly orthogonalised
// orbitals become sums of products of inner products).
constexpr int kGramOrbs = 16, kGramSlots = 64;
struct GramPlan {
  double *psi[kGramOrbs];
  double *norm_out[kGramOrbs], *ovl_out[kGramOrbs];
  int ihomo[kGramOrbs];               // 0 heteronuclear; +-1 setCiOrb parity
  int npart[kGramOrbs];
  signed char part[kGramOrbs][kGramOrbs];  // partners (plan indices, earlier in the order)
  signed char slot_of[kGramOrbs][kGramOrbs];  // slot of <Z_a, Z_b> (a != b), of <X_a, X_a> (a == b)
  signed char sa[kGramSlots], sb[kGramSlots];
  int n, nslots, homo;
};

__global__ void __launch_bounds__(kThreads) k_orthonormalise_gram(GridDev g, const __grid_constant__ GramPlan P,
                                                                  double *partials, BarrierDev bar) {
  __shared__ double s_h[kGramSlots];
  __shared__ double s_z[kGramOrbs];
  __shared__ double s_c[kGramOrbs][kGramOrbs];
  const int nb = int(gridDim.x), n = P.n, n2 = g.nni / 2 + 1;
  // inner products, kMaxK slots per pass; the values are read where the
  // slot needs them (L1 serves the repeats), so nothing is indexed at run
  // time in registers
  for (int s0 = 0; s0 < P.nslots; s0 += kMaxK) {
    double v[kMaxK];
#pragma unroll
    for (int t = 0; t < kMaxK; ++t) v[t] = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
      const int mu = k / g.nni, nu = k - mu * g.nni;
      const int row = (mu + 4) * g.n8 + 4;
      // Z at this point: the orbital itself, or its mirrored first-half value
      int src = nu, middle = 0, second = 0;
      if (P.homo) {
        if (nu > n2 - 1) {
          src = g.nni - 1 - nu;
          second = 1;
        } else if (nu == n2 - 1) {
          middle = 1;
        }
      }
      const double w = g.wf[k];
#pragma unroll
      for (int t = 0; t < kMaxK; ++t) {
        if (s0 + t >= P.nslots) break;
        const int a = P.sa[s0 + t], b = P.sb[s0 + t];
        double pr;
        if (a == b) {
          const double x = P.psi[a][row + nu];
          pr = M(x, x);
        } else {
          double za = P.psi[a][row + src], zb = P.psi[b][row + src];
          if (middle) {
            za = (P.ihomo[a] == 1) ? za : 0.0;
            zb = (P.ihomo[b] == 1) ? zb : 0.0;
          } else if (second) {
            za = (P.ihomo[a] == -1) ? -za : za;
            zb = (P.ihomo[b] == -1) ? -zb : zb;
          }
          pr = M(za, zb);
        }
        v[t] = fma(w, pr, v[t]);
      }
    }
    block_sum_store<kMaxK>(v, partials + size_t(s0) * nb);
    __syncthreads();
  }
  __threadfence();
  if (!grid_barrier(bar, unsigned(nb))) return;
  // totals, one slot per warp at a time, in block order
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = warp; t < P.nslots; t += kThreads / 32) {
      const double *base = partials + size_t(t / kMaxK * kMaxK) * nb + (t % kMaxK);
      double x = 0.0;
      for (int b = lane; b < nb; b += 32) x += __ldcg(base + size_t(b) * kMaxK);
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) s_h[t] = x;
    }
  }
  __syncthreads();
  if (threadIdx.x < n) s_z[threadIdx.x] = D(1.0, sqrt(s_h[P.slot_of[threadIdx.x][threadIdx.x]]));
  __syncthreads();
  // the coefficients, in the reference's orbital order (every block alike)
  if (threadIdx.x == 0) {
    for (int j = 0; j < n; ++j)
      for (int m = 0; m < n; ++m) s_c[j][m] = 0.0;
    for (int j = 0; j < n; ++j) {
      const double zarea = s_z[j];
      double ovl[kGramOrbs];
      double x = 0.0;
      for (int p = 0; p < P.npart[j]; ++p) {
        const int q = P.part[j][p];
        double sum = 0.0;
        for (int m = 0; m < n; ++m) {
          const int sl = P.slot_of[j][m];
          if (s_c[q][m] != 0.0 && sl >= 0) sum = A(sum, M(s_c[q][m], s_h[sl]));
        }
        ovl[p] = M(zarea, sum);
        x = A(x, M(ovl[p], ovl[p]));
      }
      if (P.npart[j] == 0) {
        s_c[j][j] = zarea;
      } else {
        const double ano = D(sqrt(A(1.0, x)), S(1.0, M(x, x)));
        double row[kGramOrbs];
        for (int m = 0; m < n; ++m) row[m] = (m == j) ? zarea : 0.0;
        for (int p = 0; p < P.npart[j]; ++p) {
          const int q = P.part[j][p];
          for (int m = 0; m < n; ++m) row[m] = A(row[m], M(-ovl[p], s_c[q][m]));
        }
        for (int m = 0; m < n; ++m) s_c[j][m] = M(ano, row[m]);
      }
      if (blockIdx.x == 0) {
        *P.norm_out[j] = s_h[P.slot_of[j][j]];
        for (int p = 0; p < P.npart[j]; ++p) P.ovl_out[j][p] = ovl[p];
      }
    }
  }
  __syncthreads();
  // Y = C Z, each thread owning its points (homonuclear: a first-half point
  // and its mirror, read once, written both)
  const int npts = P.homo ? n2 * g.nmu : g.mxsize;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < npts; k += gridDim.x * blockDim.x) {
    int mu, nu;
    if (P.homo) {
      mu = k / n2;
      nu = k - mu * n2;
    } else {
      mu = k / g.nni;
      nu = k - mu * g.nni;
    }
    const int row = (mu + 4) * g.n8 + 4;
    const bool middle = P.homo && nu == n2 - 1;
    double z[kGramOrbs];
#pragma unroll
    for (int j = 0; j < kGramOrbs; ++j) {
      if (j >= n) break;
      const double x = __ldcg(P.psi[j] + row + nu);
      z[j] = (middle && P.ihomo[j] != 1) ? 0.0 : x;
    }
#pragma unroll
    for (int j = 0; j < kGramOrbs; ++j) {
      if (j >= n) break;
      double y = 0.0;
#pragma unroll
      for (int m = 0; m < kGramOrbs; ++m) {
        if (m > j) break;
        if (s_c[j][m] != 0.0) y = A(y, M(s_c[j][m], z[m]));
      }
      P.psi[j][row + nu] = y;
      if (P.homo && !middle) P.psi[j][row + (g.nni - 1 - nu)] = (P.ihomo[j] == 1) ? y : -y;
    }
  }
}

// EaHF = oneelij(i,i) + (J + K): per point terms of integrals.F90:406-480
// and lagrangeMultipliers.F90:67-72.  psi's ghost cells are read as the
// mirrored interior values (identical to a putin ghost refresh); exact keeps
// the reference's unfused order, otherwise products are fused (mixed form).
// EaHF of one orbital (lagrangeMultipliers.F90:21-107 with the kinetic
// term of integrals.F90:406-480): the per-thread partial sums of one block
template <bool exact>
__device__ __forceinline__ void eahf_partials(const GridDev &g, const double *psi, int isym, int m,
                                              const double *coulp, const double *exchp, double (&v)[5]) {
  const int n8 = g.n8;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * n8 + nu + 4;
    // diffnu: sum_k f(nu+k-4) dni(k,nu); diffmu: sum_k f(mu+k-4) dmu(k,mu) (dgemv order)
    double sn = 0.0, sm = 0.0;
    const double *dn = g.dni9 + 9 * nu, *dm = g.dmu9 + 9 * mu;
    if (mu >= 4 && nu >= 4 && nu <= g.nni - 5) {
#pragma unroll
      for (int q = 0; q < 9; ++q) sn = madd<exact>(psi[ij + q - 4], dn[q], sn);
#pragma unroll
      for (int q = 0; q < 9; ++q) sm = madd<exact>(psi[ij + (q - 4) * n8], dm[q], sm);
    } else {
#pragma unroll
      for (int q = 0; q < 9; ++q) sn = madd<exact>(ghost_read(g, psi, mu + 4, nu + q, isym), dn[q], sn);
#pragma unroll
      for (int q = 0; q < 9; ++q) sm = madd<exact>(ghost_read(g, psi, mu + q, nu + 4, isym), dm[q], sm);
    }
    double kin = A(sn, sm);
    const double p = psi[ij];
    if (m != 0) kin = madd<exact>(M(double(m * m), g.e[k]), p, kin);
    const double pf0 = M(p, g.f0[k]);
    const double w1 = g.wgt1[k], w2 = g.wgt2[k];
    if (exact) {
      const double t = M(A(pf0, kin), p);
      v[0] += w1 * t;                   // oneel
      v[1] += w1 * M(kin, p);           // kinetic (+ m^2 e term)
      v[2] += w1 * M(pf0, p);           // nuclear
      v[3] += w2 * M(M(p, coulp[k]), p);
      v[4] += w2 * M(p, exchp[k]);
    } else {
      const double kp = kin * p, np = pf0 * p;
      v[1] = fma(w1, kp, v[1]);
      v[2] = fma(w1, np, v[2]);
      v[3] = fma(w2, (p * coulp[k]) * p, v[3]);
      v[4] = fma(w2, p * exchp[k], v[4]);
    }
  }
  if (!exact) v[0] = v[1] + v[2];  // oneel = kinetic + nuclear, summed per block
}

// EaHF and its parts from the summed quadratures (lagrangeMultipliers.F90:67-72)
__device__ __forceinline__ void eahf_store(const double *sums, double *ee_out, double *parts) {
  const double woneel = sums[0], wc = sums[3], wx = -sums[4];
  *ee_out = woneel + (wc + wx);
  if (parts) {
    parts[0] = sums[1];
    parts[1] = sums[2];
    parts[2] = woneel;
    parts[3] = wc;
    parts[4] = wx;
  }
}

template <bool exact>
__global__ void k_eahf(GridDev g, const double *psi, int isym, int m, const double *coulp, const double *exchp,
                       double *partials, double *sums, double *ee_out, double *parts, unsigned *ticket) {
  double v[5] = {0, 0, 0, 0, 0};
  eahf_partials<exact>(g, psi, isym, m, coulp, exchp, v);
  if (block_sum_finish<5>(v, partials, sums, 5, ticket) && threadIdx.x == 0) eahf_store(sums, ee_out, parts);
}

// EaHF of several orbitals in one launch: orbital blockIdx.y with its own
// partials, sums and ticket, reduced in the same block order as k_eahf
constexpr int kEahfItems = 36;
struct EahfList {
  EahfItem it[kEahfItems];
};
template <bool exact>
__global__ void k_eahf_batch(GridDev g, const __grid_constant__ EahfList L, double *partials, unsigned *tickets) {
  const EahfItem &I = L.it[blockIdx.y];
  double v[5] = {0, 0, 0, 0, 0};
  eahf_partials<exact>(g, I.psi, I.isym, I.m, I.coulp, I.exchp, v);
  double *part = partials + size_t(blockIdx.y) * (gridDim.x * 5 + 5);
  if (block_sum_finish<5>(v, part, part + size_t(gridDim.x) * 5, 5, tickets + blockIdx.y) && threadIdx.x == 0)
    eahf_store(part + size_t(gridDim.x) * 5, I.ee_out, I.parts);
}

struct TripleList {
  TripleItem it[kMaxK];
};

__global__ void k_triples(GridDev g, TripleList L, int n, double *partials, double *out, unsigned *ticket) {
  double v[kMaxK];
  for (int q = 0; q < kMaxK; ++q) v[q] = 0.0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
    const int mu = k / g.nni, nu = k - mu * g.nni;
    const int ij = (mu + 4) * g.n8 + nu + 4;
    const double w = g.wgt2[k];
    for (int q = 0; q < n; ++q) {
      double t = M(L.it[q].a[ij], L.it[q].b[ij]);
      if (L.it[q].c) t = M(t, L.it[q].c[ij]);
      v[q] += w * t;
    }
  }
  block_sum_finish<kMaxK>(v, partials, out, n, ticket);
}

// coulMom (scfUtils.F90:490-603) and exchMom (scfUtils.F90:615-844, with
// the grid's weighted P_k^q r^k tables) of a batch of items (blockIdx.y =
// item), each with its own gridDim.x partial sums and ticket, so every
// item's sum runs in a fixed order
constexpr int kMomentItems = 64;
struct MomentList {
  MomentItem it[kMomentItems];
};
__global__ void k_moments(GridDev g, const __grid_constant__ MomentList L, int homo, double *partials,
                          unsigned *tickets) {
  const MomentItem &m = L.it[blockIdx.y];
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (m.coul) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
      const int mu = k / g.nni, nu = k - mu * g.nni;
      const double p = m.psa[(mu + 4) * g.n8 + nu + 4];
      const double wk1 = M(M(p, p), g.f4[k]);
      for (int q = 0; q < g.mpole; ++q) {
        if (homo && (q % 2 == 0)) continue;
        v[q] += g.wgt2[k] * M(g.leg[size_t(q) * g.mxsize + k], wk1);
      }
    }
  } else if (m.idel <= 4) {
    const double *T = g.exm + size_t(m.idel) * 8 * g.mxsize;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < g.mxsize; k += gridDim.x * blockDim.x) {
      const int mu = k / g.nni, nu = k - mu * g.nni;
      const int ij = (mu + 4) * g.n8 + nu + 4;
      const double wk1 = m.psa[ij] * m.psb[ij];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < g.mpole) v[q] = fma(T[size_t(q) * g.mxsize + k], wk1, v[q]);
    }
  }
  block_sum_finish<8>(v, partials + size_t(blockIdx.y) * gridDim.x * 8, m.out, g.mpole, tickets + blockIdx.y);
}

// Checks narrow_f64 / widen_f32 against the hardware conversions on n
// values: edge cases, then bit patterns from a counter hash.  Counts
// mismatches outside the documented flush ranges (float subnormals); NaNs
// must map to NaNs.
__global__ void k_convert_selftest(long n, unsigned long long seed, unsigned long long *bad) {
  unsigned long long nb = 0;
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) {
    unsigned long long h = (unsigned long long)i * 0x9E3779B97F4A7C15ull + seed;
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 29;
    double x = __longlong_as_double((long long)h);
    if (i < 16) {
      const double edge[16] = {0.0, -0.0, 1.0, -1.0, 3.4028234663852886e38, 3.4028235677973366e38, 1e39, -1e39,
                               1.1754943508222875e-38, 1.1754942e-38, 1e-300, 0.1, 1.0 + 0x1p-24, 1.0 + 0x1p-23 + 0x1p-24,
                               __longlong_as_double(0x7ff0000000000000ll), __longlong_as_double(0x7ff8000000000001ll)};
      x = edge[i];
    }
    // narrowing
    const float a = narrow_f64(x), b = __double2float_rn(x);
    const bool sub = fabs(x) < 1.1754943508222875e-38 && x != 0.0;
    if (!sub) {
      if (isnan(b)) nb += isnan(a) ? 0 : 1;
      else nb += (__float_as_uint(a) == __float_as_uint(b)) ? 0 : 1;
    }
    // widening of a float pattern
    const float f = __uint_as_float(unsigned(h >> 32));
    const double wa = widen_f32(f), wb = double(f);
    const bool fsub = (__float_as_uint(f) & 0x7f800000u) == 0 && (__float_as_uint(f) & 0x7fffffu) != 0;
    if (!fsub) {
      if (isnan(wb)) nb += isnan(wa) ? 0 : 1;
      else nb += (__double_as_longlong(wa) == __double_as_longlong(wb)) ? 0 : 1;
    }
  }
  if (nb) atomicAdd(bad, nb);
}

inline int grid_blocks(int n) {
  int b = (n + kThreads - 1) / kThreads;
  return b < 1 ? 1 : (b > 1184 ? 1184 : b);
}

}  // namespace

// ======================================================================
// launchers
// ======================================================================

static double *reduction_partials(x2g_ctx *ctx, int K) {
  size_t need = size_t(kRedBlocksMax) * K * sizeof(double) + 64 * sizeof(double);
  if (ctx->red_bytes < need) {
    if (ctx->red) cudaFree(ctx->red);
    ctx->red = nullptr;
    ctx->red_bytes = 0;
    if (cudaMalloc(&ctx->red, need) != cudaSuccess) return nullptr;
    ctx->red_bytes = need;
  }
  return static_cast<double *>(ctx->red);
}

// Job-table entry of one x2g_job (kind 0 orbital with borb; 1 potential
// built from psa/psb; 2 potential given explicit lhs/rhs arrays, bpot).
static bool make_job(const x2g_job &x, JobDev &d) {
  const bool explicit_lr = (x.lhs && x.rhs);
  if (!x.u || (x.kind != 0 && x.kind != 1) || (x.kind == 0 && !explicit_lr) ||
      (x.kind == 1 && !explicit_lr && (!x.psa || !x.psb)) || (x.isym != 1 && x.isym != -1))
    return false;
  d = JobDev{};
  d.u = x.u;
  d.lhs = x.lhs;
  d.rhs = x.rhs;
  d.psa = x.psa;
  d.psb = x.psb;
  d.omega = x.omega;
  d.omegaf = float(x.omega);
  d.omega1f = float(1.0 - x.omega);
  d.idel2 = double(x.idel * x.idel);
  d.isym = x.isym;
  d.kind = (x.kind == 1 && explicit_lr) ? 2 : x.kind;
  return true;
}

static int take_event(x2g_ctx *ctx, cudaEvent_t *ev) {
  if (!ctx->event_pool.empty()) {
    *ev = ctx->event_pool.back();
    ctx->event_pool.pop_back();
    return X2G_OK;
  }
  cudaError_t err = cudaEventCreate(ev);
  return (err == cudaSuccess) ? X2G_OK : cuda_status(err, "profiling event");
}

// Co-resident clusters of `size` CTAs of a cluster sweep kernel on the
// context's device (0: it cannot run).  The function's attributes are shared
// by every context and thread of the process: its dynamic shared memory cap is
// set to the device's opt-in maximum (never lowered, so concurrent contexts
// cannot undercut each other) and clusters above 8 CTAs are allowed.
static int cluster_active(x2g_ctx *ctx, const void *fn, int size, int threads, size_t smem) {
  if (ctx->cluster_smem < 0) {
    int optin = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess) {
      (void)cudaGetLastError();
      optin = 0;
    }
    ctx->cluster_smem = optin;
  }
  if (!fn || smem > size_t(ctx->cluster_smem)) return 0;
  int n = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->cluster_smem) == cudaSuccess &&
      cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t q = {};
    q.gridDim = dim3(unsigned(size));
    q.blockDim = dim3(unsigned(threads));
    q.dynamicSmemBytes = smem;
    cudaLaunchAttribute qa[1];
    qa[0].id = cudaLaunchAttributeClusterDimension;
    qa[0].val.clusterDim.x = unsigned(size);
    qa[0].val.clusterDim.y = 1;
    qa[0].val.clusterDim.z = 1;
    q.attrs = qa;
    q.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &q) != cudaSuccess) n = 0;
  }
  (void)cudaGetLastError();
  return n;
}

// A kernel and band plan of the on-chip sweep.
struct ColChoice {
  const ColPlan *plan = nullptr;
  const void *fn = nullptr;
  bool sep = false;
  int rows = 0;
  size_t smem = 0;
  int active = 0;  // co-resident clusters
  int wave = 0;    // jobs of a launch
};

// The kernels of the on-chip sweep that can run this grid's band plans here,
// asked once per grid size: plain, sep, sep with two CTAs per SM.
static const std::vector<x2g_ctx::ColumnShape> &column_shapes(x2g_ctx *ctx, const HostGrid &h) {
  for (const auto &s : ctx->columns)
    if (s.nni == h.nni && s.nmu == h.nmu) return s.shapes;
  x2g_ctx::ColumnShapes out{h.nni, h.nmu, {}};
  for (size_t i = 0; i < h.s->columns.size(); ++i)
    for (int kind = 0; kind < 3; ++kind) {
      const ColPlan &p = h.s->columns[i];
      int pitch = 0;
      const ColKernel k = column_kernel(p, kind > 0, kind == 2, std::max(p.pitch, p.warps * 32), pitch);
      if (!k.fn) continue;
      x2g_ctx::ColumnShape c{int(i), k.fn, kind > 0, column_rows(p, k.slots), 0, 0};
      c.smem = column_smem(c.rows, pitch, c.sep, p.warps * p.groups * 32);
      c.active = cluster_active(ctx, c.fn, p.size, p.warps * p.groups * 32, c.smem);
      if (c.active > 0) out.shapes.push_back(c);
    }
  ctx->columns.push_back(std::move(out));
  return ctx->columns.back().shapes;
}

// Expected time of one launch of the on-chip sweep over `jobs` jobs, in us for
// 10 sweeps: a start-up and, per slot (point of a colour in a thread's rows),
// the latency of a few warps or the issue slots of the warps that share an SM.
// Clusters rarely fill more than nine tenths of the SMs (whole clusters lie in
// one group of SMs).  Measured, us: 151x241, two threads per column: 3 slots
// 57, 4 66, 5 74; 331x481 likewise: 4 slots 96, 5 114; one thread per column,
// one CTA on an SM: 7 slots 117, 9 139, two: 7 160, 9 207.  So 22 potentials
// of 331x481 run as one wave of 11-CTA clusters (209) and not as two of 16-CTA
// ones (320), 64 of 151x241 as two launches of 32 (214; 287 on the kernel with
// fixed clusters of 8).
static double column_time(const ColPlan &p, int jobs, int num_sms) {
  const int share = (jobs * p.size + num_sms * 9 / 10 - 1) / (num_sms * 9 / 10);
  return 30.0 + p.slots * std::max(12.0, 0.8 * p.warps * p.groups * share);
}

// The on-chip sweep for njobs jobs (sep: all of them potentials with a
// separable lhs), or none: the kernel and cluster size with the least expected
// time for the waves of co-resident clusters they take.
static ColChoice choose_columns(x2g_ctx *ctx, const HostGrid &h, int njobs, bool sep) {
  ColChoice best;
  double best_time = 0;
  if (ctx->no_cluster) return best;
  for (const x2g_ctx::ColumnShape &c : column_shapes(ctx, h)) {
    if (c.sep != sep) continue;
    const ColPlan &p = h.s->columns[size_t(c.plan)];
    const int wave = std::min(c.active, kParamJobs);
    const double time = njobs / wave * column_time(p, wave, ctx->num_sms) +
                        (njobs % wave ? column_time(p, njobs % wave, ctx->num_sms) : 0.0);
    if (!best.plan || time < best_time) {
      best = {&p, c.fn, sep, c.rows, c.smem, c.active, wave};
      best_time = time;
    }
  }
  return best;
}

static const void *band_kernel(int threads) {
  return threads == kBandThreads ? (const void *)k_mcsor_f32p<kBandThreads> : (const void *)k_mcsor_f32p<2 * kBandThreads>;
}

// Launch shape of the persistent-band sweep: the most jobs per launch (at
// most `most`) and the shortest tile runs G for which every (job, run) gets
// its own co-resident block, at two 512-thread blocks per SM (the band's
// shared memory must fit twice) or, where that holds more jobs, one block of
// 1024: its band is twice as high with the same halos.  A launch takes 285 us
// and 30 per job of 781 x 1201 (10 sweeps), so fewer launches are faster: seven
// jobs 544 us in one launch of the large blocks, 758 in two of the small ones;
// six 468 (480 in large ones).  The functions' shared memory cap is raised once
// to the device's opt-in maximum, as for the cluster kernel.
static int persistent_shape(x2g_ctx *ctx, const GridDev &g, int most, int *nj, int *G, size_t *smem,
                            int *threads = nullptr) {
  if (!ctx->band_attr) {
    // the cap counts dynamic bytes only: the opt-in maximum less the
    // kernel's static shared memory (the neighbour wait's flag)
    int optin = 0;
    cudaFuncAttributes fa{};
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, band_kernel(kBandThreads)) != cudaSuccess ||
        cudaFuncSetAttribute(band_kernel(kBandThreads), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - int(fa.sharedSizeBytes)) != cudaSuccess ||
        cudaFuncSetAttribute(band_kernel(2 * kBandThreads), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             optin - int(fa.sharedSizeBytes)) != cudaSuccess) {
      (void)cudaGetLastError();
      return set_status(X2G_ERR_CUDA, "persistent sweep attributes could not be set");
    }
    ctx->band_attr = optin - int(fa.sharedSizeBytes);
    int per_sm = 0;
    if (cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx->device) != cudaSuccess)
      return set_status(X2G_ERR_CUDA, "device attribute query failed");
    ctx->band_sm_smem = per_sm;
  }
  for (int n = most; n >= 1; --n)
    for (int bpsm = 2; bpsm >= 1; --bpsm)
      for (int r = 1; r <= Schedule::kBandRuns; ++r) {
        const size_t sm = band_smem_bytes(g, r);
        if (sm > size_t(ctx->band_attr) || int(size_t(ctx->band_sm_smem) / (sm + 1024)) < bpsm) break;
        const int items = n * ((g.ntiles + r - 1) / r), nt = kBandThreads * (bpsm == 1 ? 2 : 1);
        if (items > bpsm * ctx->num_sms) continue;
        // confirm with the occupancy calculator (once per shared size)
        const long key = long(sm) * 2 + bpsm - 1;
        if (ctx->band_key != key) {
          int per = 0;
          cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, band_kernel(nt), nt, sm);
          if (err != cudaSuccess) return cuda_status(err, "occupancy query");
          ctx->band_key = key;
          ctx->band_blocks = per * ctx->num_sms;
        }
        if (items > ctx->band_blocks) continue;
        *nj = n;
        *G = r;
        *smem = sm;
        if (threads) *threads = nt;
        return X2G_OK;
      }
  return set_status(X2G_ERR_ARG, "grid too large for the persistent FP32 sweep");
}

// Co-resident blocks of the cooperative FP64 sweep on the context's device
// (asked once per context).
static int f64_block_limit(x2g_ctx *ctx) {
  if (ctx->f64_blocks > 0) return X2G_OK;
  int per_sm = 0;
  cudaError_t err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_mcsor_f64, kThreads, 0);
  if (err != cudaSuccess) return cuda_status(err, "occupancy query");
  if (per_sm < 1) return set_status(X2G_ERR_CUDA, "cooperative FP64 sweep cannot be resident");
  ctx->f64_blocks = per_sm * ctx->num_sms;
  return X2G_OK;
}

// One launch of the on-chip cluster sweep over the jobs of jt, timed with the
// context's events when profiling.
static int cluster_sweep(x2g_ctx *ctx, const GridDev &g, const ColChoice &c, JobTable &jt, int njobs, int nsweeps) {
  x2g_ctx::Pending pe{};
  if (ctx->profiling) {
    int rc;
    if ((rc = take_event(ctx, &pe.a)) || (rc = take_event(ctx, &pe.b))) return rc;
    pe.precision = 1;
    pe.points = double(njobs) * double(g.nni - 2) * double(g.nmu - 5) * double(nsweeps);
    cudaEventRecord(pe.a, ctx->stream);
  }
  int free = ctx->mixed_free;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(njobs * c.plan->size));
  cfg.blockDim = dim3(unsigned(32 * c.plan->warps * c.plan->groups));
  cfg.dynamicSmemBytes = c.smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = unsigned(c.plan->size);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  GridDev gd = g;
  ColPlan plan = *c.plan;
  plan.rows = c.rows;
  for (int k = 0; k < 4; ++k) {
    plan.c2[k] = make_float2(g.dmu2f[k], g.dni2f[k]);
    plan.c1[k] = make_float2(g.dmu1f[k], g.dni1f[k]);
    plan.m1[k] = make_float2(g.dmu1f[k], -g.dmu1f[k]);
    plan.m2[k] = make_float2(g.dmu2f[k], g.dmu2f[k]);
  }
  plan.neg = make_float2(-1.0f, -1.0f);
  BarrierDev limit{ctx->bar, ctx->bar + 1, reinterpret_cast<int *>(ctx->bar + 2), ctx->wait_limit_ns};
  void *args[] = {&gd, &plan, &jt, &nsweeps, &free, &limit};
  cudaError_t err = cudaLaunchKernelExC(&cfg, c.fn, args);
  if (err != cudaSuccess) return cuda_status(err, "cluster MCSOR launch");
  ctx->launches += 1;
  if (ctx->profiling) {
    cudaEventRecord(pe.b, ctx->stream);
    ctx->pending.push_back(pe);
  }
  return X2G_OK;
}

// Mixed form on chip: the jobs in waves of the co-resident clusters.  The
// first wave's FP64 residual, then each later wave's on the low-priority
// auxiliary stream, beside the sweep before it (on the SMs and the FP64 pipes
// that leaves free); each sweep waits for its own wave's residual.  The short
// wave (the remainder) goes first: its residual is the only one on the
// critical path.  job(i): the table entry of job i.
template <class JobOf>
static int relax_on_chip(x2g_ctx *ctx, const GridDev &g, const ColChoice &col, int njobs, int nsweeps, bool fixed,
                         JobOf job) {
  const bool overlap = ctx->residual_overlap != 0;
  const int first = njobs % col.wave ? njobs % col.wave : col.wave;
  cudaError_t err;
  JobTable cur{}, next{};
  auto table = [&](int i0, int n, JobTable &t) {
    for (int i = 0; i < n; ++i) t.j[i] = job(i0 + i);
  };
  auto residual = [&](const JobTable &t, int n, cudaStream_t s) {
    launch_residual(g, t, n, fixed, false, !col.sep, s);
    ctx->launches += 1;
  };
  table(0, first, cur);
  residual(cur, first, ctx->stream);
  if (overlap && first < njobs &&
      ((err = cudaEventRecord(ctx->ev_split[0], ctx->stream)) != cudaSuccess ||
       (err = cudaStreamWaitEvent(ctx->aux, ctx->ev_split[0], 0)) != cudaSuccess))
    return cuda_status(err, "residual overlap");
  for (int i0 = 0, n = first, c = 0; i0 < njobs; i0 += n, n = col.wave, ++c) {
    const bool more = i0 + n < njobs;
    cudaEvent_t ev = ctx->ev_split[(c + 1) & 1];
    if (more) {
      table(i0 + n, col.wave, next);
      residual(next, col.wave, overlap ? ctx->aux : ctx->stream);
      if (overlap && (err = cudaEventRecord(ev, ctx->aux)) != cudaSuccess) return cuda_status(err, "residual overlap");
    }
    int rc = cluster_sweep(ctx, g, col, cur, n, nsweeps);
    if (rc) return rc;
    if (more && overlap && (err = cudaStreamWaitEvent(ctx->stream, ev, 0)) != cudaSuccess)
      return cuda_status(err, "residual overlap");
    cur = next;
  }
  return X2G_OK;
}

// Mixed form in persistent bands: one launch batch (at most kParamJobs jobs).
static int relax_bands(x2g_ctx *ctx, const GridDev &g, JobTable &jt, int njobs, int nsweeps, bool fixed, int G,
                       size_t smem, int threads) {
  cudaError_t err;
  x2g_ctx::Pending pe{};
  launch_residual(g, jt, njobs, fixed, true, true, ctx->stream);
  ctx->launches += 1;
  if (ctx->profiling) {
    int rc;
    if ((rc = take_event(ctx, &pe.a)) || (rc = take_event(ctx, &pe.b))) return rc;
    pe.precision = 1;
    pe.points = double(njobs) * double(g.nni - 2) * double(g.nmu - 5) * double(nsweeps);
    cudaEventRecord(pe.a, ctx->stream);
  }
  // persistent-band sweep, one block per (job, run of G tiles), phase counts
  // zeroed.  The error word keeps an earlier launch's timeout until
  // x2g_synchronize reports it
  const unsigned nb = unsigned(njobs * ((g.ntiles + G - 1) / G));
  if (nb > unsigned(kPhaseBlocks)) return set_status(X2G_ERR_ARG, "too many blocks for the phase counts");
  err = cudaMemsetAsync(ctx->bar + kPhaseWords, 0, size_t(kPhaseBlocks) * kPhaseStride * sizeof(unsigned), ctx->stream);
  if (err != cudaSuccess) return cuda_status(err, "barrier reset");
  BarrierDev bar{ctx->bar, ctx->bar + 1, reinterpret_cast<int *>(ctx->bar + 2), ctx->wait_limit_ns};
  unsigned *phase = ctx->bar + kPhaseWords;
  int ns = nsweeps;
  GridDev gd = g;
  void *args[] = {&gd, &jt, &ns, &G, &bar, &phase};
  err = cudaLaunchCooperativeKernel(band_kernel(threads), dim3(nb), dim3(unsigned(threads)), args, smem, ctx->stream);
  if (err != cudaSuccess) return cuda_status(err, "cooperative MCSOR launch");
  ctx->launches += 1;
  if (ctx->profiling) {
    cudaEventRecord(pe.b, ctx->stream);
    ctx->pending.push_back(pe);
  }
  // the update u += e and the axis of u are that kernel's epilogue
  return X2G_OK;
}

struct MarchKernel {
  const void *fn;
  int threads;
};
// two lanes a point where all of a block's sweeps are at work on a row at once
// (they follow each other 8 columns apart): 331 x 481, four rows, 1.14 ms (four
// lanes 1.28); 151 x 181, two functions 585 us (558); 91 x 121, four 427 (365)
static MarchKernel march_kernel(int rows, int nsweeps, int nni) {
  if (rows == 2) return {(const void *)k_march_f64<2, 4>, march_threads(2, 4)};
  if (rows == 8) return {(const void *)k_march_f64<8, 2>, march_threads(8, 2)};
  if (std::min(nsweeps, nni / 16) < kMarchSweeps) return {(const void *)k_march_f64<4, 4>, march_threads(4, 4)};
  return {(const void *)k_march_f64<4, 2>, march_threads(4, 2)};
}

// whether blocks of the marching SOR sweep can be resident with this much
// shared memory (its cap is set to the device's opt-in maximum, once)
static bool march_fits(x2g_ctx *ctx, size_t smem) {
  if (ctx->march_smem < 0) {
    int optin = 0;
    bool ok = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device) == cudaSuccess &&
              (optin -= 1024) > 0;  // the barrier's flag
    auto fits = [&](const void *fn, int threads) {
      int a = 0;
      return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) == cudaSuccess &&
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, fn, threads, size_t(optin)) == cudaSuccess && a >= 1;
    };
    for (int rows = 2; rows <= 8; rows *= 2)
      for (int sweeps : {1, kMarchSweeps}) {
        const MarchKernel k = march_kernel(rows, sweeps, 16 * kMarchSweeps);
        ok = ok && fits(k.fn, k.threads);
      }
    (void)cudaGetLastError();
    ctx->march_smem = ok ? optin : 0;
  }
  return smem <= size_t(ctx->march_smem);
}

// FP64 relaxation over the wavefront schedule w, in cooperative launches of
// at most kParamJobs jobs and kWaveScratch bytes of scratch (the tagged copy
// and the (lhs, rhs) pairs of a launch's jobs, used by the launches in turn;
// 32 jobs of 331 x 481 are 248 MB, and a launch of one 781 x 1201 job already has
// points enough in a step to fill the GPU).
constexpr size_t kWaveScratch = size_t(256) << 20;
static int relax_wave(x2g_ctx *ctx, const GridDev &g, const WaveDev &w, const x2g_job *jobs, int njobs, int nsweeps,
                      bool profile, const MarchDev *march = nullptr) {
  // SOR: the marching sweep with the fewest rows a block (2, 4, 8) that give
  // every block its own SM, else the wavefront.  10 sweeps, us, this /
  // wavefront: two functions of 331 x 481 (eight rows) 1704 / 2462, four and
  // six of 151 x 181 (eight) 765 / 952 and 769 / 1032, four and eight of 91 x
  // 121 (four, eight) 365 / 641 and 483 / 681; beyond that the wavefront is
  // bound by the FP64 pipe, which this uses worse
  int rows = 0;
  for (int r = 8; r >= 2 && march; r /= 2)
    if (njobs * ((g.nmu - 4 + r - 1) / r) <= ctx->num_sms && march_fits(ctx, size_t(r + 8) * g.n8 * 16)) rows = r;
  if (!rows) march = nullptr;
  const size_t tagged = (size_t(g.next) * 16 + 255) / 256 * 256, pairs = (size_t(g.mxsize) * 32 + 255) / 256 * 256;
  const int most =
      std::max(1, std::min(std::min(njobs, kParamJobs), int(std::min(kWaveScratch / (tagged + pairs), size_t(kParamJobs)))));
  char *scratch = static_cast<char *>(ctx_workspace(ctx, (tagged + pairs) * size_t(most)));
  if (!scratch) return set_status(X2G_ERR_ALLOC, "workspace allocation failed");
  const size_t smem = size_t(w.nlev + w.nblev + 2) * sizeof(int);
  if (smem > kWaveSmemMost) return set_status(X2G_ERR_ARG, "grid too large for the wavefront's level table");
  if (ctx->wave_ok < 0) {
    int a = 0, b = 0;
    int w = 0;
    cudaError_t e = cudaSuccess;
    for (const void *fn : {(const void *)k_wave_f64<4, false>, (const void *)k_wave_f64<1, false>,
                           (const void *)k_wave_f64<1, true>})
      if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kWaveSmemMost));
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, (const void *)k_wave_f64<4, false>, kWaveThreads, kWaveSmem);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)k_wave_f64<1, false>, kWaveThreads, kWaveSmem);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&w, (const void *)k_wave_f64<1, true>, kWaveThreads, kWaveSmem);
    if (e != cudaSuccess) return cuda_status(e, "occupancy query");
    ctx->wave_ok = (a >= 1 && b >= 1 && w >= 1) ? 1 : 0;
  }
  if (!ctx->wave_ok) return set_status(X2G_ERR_CUDA, "cooperative FP64 sweep cannot be resident");
  for (int b0 = 0; b0 < njobs; b0 += most) {
    const int nb = std::min(njobs - b0, most);
    JobTable jt{};
    for (int i = 0; i < nb; ++i) {
      if (!make_job(jobs[b0 + i], jt.j[i])) return set_status(X2G_ERR_ARG, "bad relaxation job");
      char *p = scratch + (tagged + pairs) * size_t(i);
      jt.j[i].tagged = reinterpret_cast<ulonglong2 *>(p);
      jt.j[i].pairs = reinterpret_cast<double *>(p + tagged);
    }
    cudaError_t err = cudaMemsetAsync(ctx->bar, 0, 2 * sizeof(unsigned), ctx->stream);
    if (err != cudaSuccess) return cuda_status(err, "barrier reset");
    BarrierDev bar{ctx->bar, ctx->bar + 1, reinterpret_cast<int *>(ctx->bar + 2), ctx->wait_limit_ns};
    // four lanes per point while the average step is narrow: MCSOR, 10
    // sweeps, four lanes / one lane: 289 / 329 us at 58 points a step and SM
    // (151 x 241, 2 jobs), 369 / 368 us at 85 (91 x 121, 10 jobs), 507 / 389
    // us at 145 (151 x 241, 5 jobs).  One lane, FP64 pipe
    // alone / its wide form: 785 / 842 us at 386 (331 x 481, 3 jobs), 896 / 901
    // at 515 (4), 1256 / 1250 at 694 (151 x 241, 24), 1034 / 982 at 644 (331 x
    // 481, 5), 4290 / 3850 at 2833 (22)
    const double steps = double(nsweeps - 1) * w.delta + std::max(w.nlev, w.nblev);
    const double per_sm = double(nb) * nsweeps * double(g.nni - 2) * double(g.nmu - 5) / steps / ctx->num_sms;
    x2g_ctx::Pending pe{};
    if (profile && ctx->profiling) {
      int rc;
      if ((rc = take_event(ctx, &pe.a)) || (rc = take_event(ctx, &pe.b))) return rc;
      pe.precision = 0;
      pe.points = double(nb) * double(g.nni - 2) * double(g.nmu - 5) * double(nsweeps);
      cudaEventRecord(pe.a, ctx->stream);
    }
    unsigned nblocks = unsigned(ctx->num_sms);
    int nj = nb, ns = nsweeps;
    GridDev gd = g;
    WaveDev wd = w;
    if (march) {
      MarchDev md = *march;
      nblocks = unsigned(nb * ((g.nmu - 4 + rows - 1) / rows));
      void *args[] = {&gd, &md, &jt, &nj, &ns, &bar, &nblocks};
      const MarchKernel k = march_kernel(rows, ns, g.nni);
      err = cudaLaunchCooperativeKernel(k.fn, dim3(nblocks), dim3(unsigned(k.threads)), args,
                                        size_t(rows + 8) * g.n8 * 16, ctx->stream);
      if (err != cudaSuccess) return cuda_status(err, "cooperative SOR launch");
      ctx->launches += 1;
      continue;
    }
    void *args[] = {&gd, &wd, &jt, &nj, &ns, &bar, &nblocks};
    err = cudaLaunchCooperativeKernel(per_sm < 85.0               ? (const void *)k_wave_f64<4, false>
                                      : per_sm < 600.0 || !g.pairs ? (const void *)k_wave_f64<1, false>
                                                                   : (const void *)k_wave_f64<1, true>,
                                      dim3(nblocks), dim3(kWaveThreads), args, smem, ctx->stream);
    if (err != cudaSuccess) return cuda_status(err, "cooperative FP64 sweep launch");
    ctx->launches += 1;
    if (profile && ctx->profiling) {
      cudaEventRecord(pe.b, ctx->stream);
      ctx->pending.push_back(pe);
    }
  }
  return X2G_OK;
}

constexpr long kFixedPoints = 1 << 16;  // fewest points of a function whose residual alone is taken in fixed point

// co-resident clusters of the cluster sweep and of its potentials' variant
// for large batches on this grid on the context's device (0: that kernel
// cannot run it)
int cluster_occupancy(x2g_ctx *ctx, x2g_grid *grid, int *plain, int *pot) {
  if (plain) *plain = choose_columns(ctx, grid->h, kParamJobs, false).active;
  if (pot) *pot = choose_columns(ctx, grid->h, kParamJobs, true).active;
  return set_status(X2G_OK, "");
}

int launch_relax(x2g_ctx *ctx, x2g_grid *grid, const x2g_job *jobs, int njobs, int nsweeps, int precision) {
  if (njobs <= 0) return X2G_OK;
  if (nsweeps <= 0) return set_status(X2G_ERR_ARG, "nsweeps must be positive");
  if (precision == X2G_SOR) return relax_wave(ctx, grid->d, grid->d.sor, jobs, njobs, nsweeps, false, &grid->d.march);
  // FP64 MCSOR: the same sweep over the colour-ordered list.  The barrier
  // sweep (k_mcsor_f64, 50 phases of three dependent levels) took 7.03 ms for
  // 22 potentials of 331 x 481, 1.80 ms for 5 and 0.52 ms for one 91 x 121
  // orbital; the wavefront 4.29, 1.04 and 0.25 ms
  if (precision == X2G_FP64) return relax_wave(ctx, grid->d, grid->d.mcsor, jobs, njobs, nsweeps, true);
  if (precision != X2G_MIXED) return set_status(X2G_ERR_ARG, "unknown relaxation form");
  const GridDev &g = grid->d;
  // potentials built from orbitals have a separable lhs: batches of them
  // beyond the plain kernel's clusters take the kernel that forms omega / lhs
  // itself (22 of 331x481: 173 us, the plain kernel's two waves of 13 and 9
  // 233; 64 of 151x241 191 and 284); below that the plain kernel's results are
  // the persistent-band sweep's bit for bit
  bool separable = true;
  for (int i = 0; i < njobs && separable; ++i) separable = (jobs[i].kind == 1 && !(jobs[i].lhs && jobs[i].rhs));
  ColChoice col = choose_columns(ctx, grid->h, njobs, false);
  if (separable && (ctx->pot_clusters == 1 || (ctx->pot_clusters == 2 && njobs > col.active))) {
    const ColChoice c = choose_columns(ctx, grid->h, njobs, true);
    if (c.plan) col = c;
  }
  if (col.plan && !col.sep && ctx->auto_band && njobs > col.active) {
    // more jobs than co-resident clusters: the cluster kernel would run in
    // waves, while the persistent-band kernel may hold the whole batch
    int nj = 0, G1 = 0;
    size_t sm1 = 0;
    const int want = njobs < kParamJobs ? njobs : kParamJobs;
    if (persistent_shape(ctx, g, want, &nj, &G1, &sm1) == X2G_OK && nj >= want) col = ColChoice();
    set_status(X2G_OK, "");
  }
  // their stencil sums in fixed point with the potentials' kernel, and on grids
  // that no on-chip kernel holds, where a function alone has tiles enough (smooth
  // functions, us, and by FMAs: 22 of 331x481 61 and 149, one of 811x121 9.0 and
  // 10.1, seven of 781x1201 116 and 345; one of 151x241 8.8 and 6.5.  Points left
  // to FMAs make a tail of some us: with the plain kernel, four of 301x481 with
  // azimuthal numbers 0 to 2 take 4 us longer so than by FMAs alone).
  // The kernel and the grid decide, not the number of jobs, so that a function's
  // result does not depend on its batch, and the plain kernel's results (mode 0,
  // SCFs in the reference's order) stay the persistent-band sweep's
  const bool fixed = separable && ctx->pot_clusters != 0 &&
                     (col.sep || (column_shapes(ctx, grid->h).empty() && long(g.nni - 2) * (g.nmu - 5) >= kFixedPoints));
  // per-job scratch: FP32 correction, residual and omega/lhs
  const size_t per_job =
      (size_t(g.next) * sizeof(float) + 2 * size_t(g.mxsize) * sizeof(float) + 256) / 256 * 256 + 256;
  char *scratch = static_cast<char *>(ctx_workspace(ctx, per_job * njobs + 256));
  if (!scratch) return set_status(X2G_ERR_ALLOC, "workspace allocation failed");
  {
    JobDev d;
    for (int i = 0; i < njobs; ++i)
      if (!make_job(jobs[i], d)) return set_status(X2G_ERR_ARG, "bad relaxation job");
  }
  auto job = [&](int i) {
    JobDev d;
    make_job(jobs[i], d);
    char *p = scratch + per_job * size_t(i);
    d.e32 = reinterpret_cast<float *>(p);
    d.r32 = reinterpret_cast<float *>(p + (size_t(g.next) * sizeof(float) + 127) / 128 * 128);
    d.w32 = d.r32 + g.mxsize;
    d.rw = reinterpret_cast<float2 *>(d.r32);  // persistent-band sweep: pairs over r32 and w32
    return d;
  };
  if (col.plan) return relax_on_chip(ctx, g, col, njobs, nsweeps, fixed, job);
  // the persistent-band sweep takes as many jobs per launch as give every
  // (job, run of tiles) its own co-resident block
  int per_launch = kParamJobs, G = 0, threads = kBandThreads;
  size_t smem = 0;
  int rc = persistent_shape(ctx, g, njobs < kParamJobs ? njobs : kParamJobs, &per_launch, &G, &smem, &threads);
  if (rc) return rc;
  for (int b0 = 0; b0 < njobs; b0 += per_launch) {
    int nb = (njobs - b0 < per_launch) ? njobs - b0 : per_launch;
    // a short last launch in shorter bands, so that it fills the SMs too (33 jobs
    // of 781 x 1201 in launches of six: 2728 us, 2745 with the last three in runs
    // of six tiles)
    if (nb < per_launch && (rc = persistent_shape(ctx, g, nb, &nb, &G, &smem, &threads))) return rc;
    JobTable jt{};
    for (int i = 0; i < nb; ++i) jt.j[i] = job(b0 + i);
    if ((rc = relax_bands(ctx, g, jt, nb, nsweeps, fixed, G, smem, threads))) return rc;
  }
  // barrier error word: checked by the caller at its next synchronisation
  return X2G_OK;
}

// Scratch layout of launch_relax_in_scratch: 4 barrier words, a reserved
// region the size of a job table, then one plain right-hand-side buffer per
// job (256-byte aligned).  The job-table size is part of the documented
// limit of x2g_relax_noalloc.
static_assert(sizeof(JobDev) == 112, "x2g_relax_noalloc documents 112-byte job-table entries");
size_t relax_scratch_bytes(const GridDev &g, int njobs) {
  const size_t head = 256;
  const size_t table = (sizeof(JobDev) * size_t(njobs) + 255) / 256 * 256;
  const size_t plain = (size_t(g.mxsize) * sizeof(double) + 255) / 256 * 256;
  return head + table + plain * size_t(njobs);
}

int launch_relax_in_scratch(x2g_ctx *ctx, x2g_grid *grid, const x2g_job *jobs, int njobs, int nsweeps,
                            void *scratch, size_t scratch_bytes) {
  const GridDev &g = grid->d;
  if (njobs <= 0 || nsweeps <= 0) return set_status(X2G_ERR_ARG, "njobs and nsweeps must be positive");
  const size_t need = relax_scratch_bytes(g, njobs);
  if (need > scratch_bytes) return set_status(X2G_ERR_ARG, "batch does not fit the scratch");
  char *base = static_cast<char *>(scratch);
  unsigned *barw = reinterpret_cast<unsigned *>(base);
  char *rhs0 = base + 256 + (sizeof(JobDev) * size_t(njobs) + 255) / 256 * 256;
  const size_t plain = (size_t(g.mxsize) * sizeof(double) + 255) / 256 * 256;
  for (int b0 = 0; b0 < njobs; b0 += kParamJobs) {
    const int nb = (njobs - b0 < kParamJobs) ? njobs - b0 : kParamJobs;
    JobTable jt{};
    for (int i = 0; i < nb; ++i)
      if (!make_job(jobs[b0 + i], jt.j[i])) return set_status(X2G_ERR_ARG, "bad relaxation job");
  }
  int rc = f64_block_limit(ctx);
  if (rc) return rc;
  // the error word is cleared once per call; between launches only the
  // arrival count and generation, so that a timeout of one launch is still
  // there when the caller reads it after the last
  cudaError_t err = cudaMemsetAsync(barw, 0, 4 * sizeof(unsigned), ctx->stream);
  if (err != cudaSuccess) return cuda_status(err, "scratch barrier reset");
  for (int b0 = 0; b0 < njobs; b0 += kParamJobs) {
    const int nb = (njobs - b0 < kParamJobs) ? njobs - b0 : kParamJobs;
    JobTable jt{};
    for (int i = 0; i < nb; ++i) {
      make_job(jobs[b0 + i], jt.j[i]);
      jt.j[i].rhs_buf = reinterpret_cast<double *>(rhs0 + plain * size_t(b0 + i));
    }
    if (b0 > 0) {
      err = cudaMemsetAsync(barw, 0, 2 * sizeof(unsigned), ctx->stream);
      if (err != cudaSuccess) return cuda_status(err, "scratch barrier reset");
    }
    BarrierDev bar{barw, barw + 1, reinterpret_cast<int *>(barw + 2), ctx->wait_limit_ns};
    const int nitems = nb * g.ntiles, cap = ctx->f64_blocks;
    unsigned nblocks = unsigned(nitems < cap ? nitems : cap);
    if (nblocks < 1) nblocks = 1;
    int nj = nb, ns = nsweeps;
    GridDev gd = g;
    void *args[] = {&gd, &jt, &nj, &ns, &bar, &nblocks};
    err = cudaLaunchCooperativeKernel((const void *)k_mcsor_f64, dim3(nblocks), dim3(kThreads), args, 0, ctx->stream);
    if (err != cudaSuccess) return cuda_status(err, "cooperative MCSOR launch");
    ctx->launches += 1;
  }
  return X2G_OK;
}

void launch_ghost_fill(x2g_ctx *ctx, const GridDev &g, double *u, int isym) {
  k_ghost<<<grid_blocks(g.nmu * 8 + 4 * g.nni), kThreads, 0, ctx->stream>>>(g, u, isym);
  ctx->launches++;
}

void launch_putin(x2g_ctx *ctx, const GridDev &g, int isym, const double *plain, double *ext) {
  k_putin_interior<<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, plain, ext);
  k_ghost<<<grid_blocks(g.nmu * 8 + 4 * g.nni), kThreads, 0, ctx->stream>>>(g, ext, isym);
  ctx->launches += 2;
}

void launch_putout(x2g_ctx *ctx, const GridDev &g, const double *ext, double *plain) {
  k_putout<<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, ext, plain);
  ctx->launches++;
}

void launch_fock(x2g_ctx *ctx, const GridDev &g, const FockArgs &a) {
  if (a.exact)
    k_fock<true><<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, a);
  else
    k_fock<false><<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, a);
  ctx->launches++;
}

void launch_fock_batch(x2g_ctx *ctx, const GridDev &g, const FockArgs *a, int n) {
  for (int b = 0; b < n; b += kFockBatch) {
    const int m = (n - b < kFockBatch) ? n - b : kFockBatch;
    FockBatch B{};
    for (int q = 0; q < m; ++q) B.a[q] = a[b + q];
    const dim3 gg(grid_blocks(g.mxsize), m);
    if (a[0].exact)
      k_fock_batch<true><<<gg, kThreads, 0, ctx->stream>>>(g, B);
    else
      k_fock_batch<false><<<gg, kThreads, 0, ctx->stream>>>(g, B);
    ctx->launches++;
  }
}

void launch_asympt_get_batch(x2g_ctx *ctx, const GridDev &g, const OrbDecayList &L, int n) {
  if (n <= 0) return;
  k_asympt_get_batch<<<dim3(grid_blocks(4 * g.nni), n), kThreads, 0, ctx->stream>>>(g, L);
  ctx->launches++;
}

void launch_asympt_set_batch(x2g_ctx *ctx, const GridDev &g, const OrbDecayList &L, int n) {
  if (n <= 0) return;
  k_asympt_set_batch<<<dim3(grid_blocks(g.nni), n), kThreads, 0, ctx->stream>>>(g, L);
  ctx->launches++;
}

void launch_asympt_get(x2g_ctx *ctx, const GridDev &g, const double *fa, double *edecay) {
  k_asympt_get<<<grid_blocks(4 * g.nni), kThreads, 0, ctx->stream>>>(g, fa, edecay);
  ctx->launches++;
}

void launch_asympt_set(x2g_ctx *ctx, const GridDev &g, double *psi, const double *edecay) {
  k_asympt_set<<<grid_blocks(g.nni), kThreads, 0, ctx->stream>>>(g, psi, edecay);
  ctx->launches++;
}

void launch_setci(x2g_ctx *ctx, const GridDev &g, double *psi, int ihomo) {
  k_setci<<<grid_blocks((g.nni / 2) * g.nmu), kThreads, 0, ctx->stream>>>(g, psi, ihomo);
  ctx->launches++;
}

void launch_scale(x2g_ctx *ctx, const GridDev &g, double *psi, const double *norm_dev) {
  k_scale<<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, psi, norm_dev);
  ctx->launches++;
}

void launch_scale_setci(x2g_ctx *ctx, const GridDev &g, double *psi, const double *norm_dev, int ihomo) {
  k_scale_setci<<<grid_blocks((g.nni / 2 + 1) * g.nmu), kThreads, 0, ctx->stream>>>(g, psi, norm_dev, ihomo);
  ctx->launches++;
}

void launch_ortho_apply(x2g_ctx *ctx, const GridDev &g, double *psi, const double *const *others, int n,
                        const double *ovl_dev) {
  PtrList L{};
  for (int q = 0; q < n && q < kMaxTerms; ++q) L.p[q] = others[q];
  k_ortho_apply<<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, psi, L, n, ovl_dev);
  ctx->launches++;
}

int convert_selftest(x2g_ctx *ctx, long n, unsigned long long seed, unsigned long long *mismatches) {
  unsigned long long *d = nullptr;
  cudaError_t e = cudaMallocAsync(&d, sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(d, 0, sizeof(unsigned long long), ctx->stream);
  if (e == cudaSuccess) {
    k_convert_selftest<<<4 * ctx->num_sms, kThreads, 0, ctx->stream>>>(n, seed, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(mismatches, d, sizeof(unsigned long long), cudaMemcpyDeviceToHost, ctx->stream);
  if (d) cudaFreeAsync(d, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  return (e == cudaSuccess) ? X2G_OK : cuda_status(e, "conversion self-test");
}

int build_moment_tables(x2g_ctx *ctx, const GridDev &g, double *exm, double *asy) {
  k_moment_tables<<<grid_blocks(g.mxsize), kThreads, 0, ctx->stream>>>(g, exm, asy);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  return (e == cudaSuccess) ? X2G_OK : cuda_status(e, "moment tables");
}

void launch_asympt(x2g_ctx *ctx, const GridDev &g, const AsymptArgs &a) {
  if (a.n <= 0) return;
  dim3 gg(grid_blocks(4 * g.nni), a.n);
  k_asympt<<<gg, kThreads, 0, ctx->stream>>>(g, a);
  ctx->launches++;
}

void launch_zero(x2g_ctx *ctx, double *p, size_t n) {
  k_zero<<<grid_blocks(int(n < (1u << 30) ? n : (1u << 30))), kThreads, 0, ctx->stream>>>(p, n);
  ctx->launches++;
}

void launch_norm(x2g_ctx *ctx, const GridDev &g, const double *psi, double *out) {
  double *part = reduction_partials(ctx, 1);
  k_norm<<<red_blocks(g), kThreads, 0, ctx->stream>>>(g, psi, part, out, ctx->bar + 3);
  ctx->launches += 1;
}

void launch_overlaps(x2g_ctx *ctx, const GridDev &g, const double *psi, const double *const *others, int n,
                     double *out) {
  double *part = reduction_partials(ctx, kMaxK);
  for (int b = 0; b < n; b += kMaxK) {
    const int m = (n - b < kMaxK) ? n - b : kMaxK;
    PtrList L{};
    for (int q = 0; q < m; ++q) L.p[q] = others[b + q];
    k_overlaps<<<red_blocks(g), kThreads, 0, ctx->stream>>>(g, psi, L, m, part, out + b, ctx->bar + 3);
    ctx->launches += 1;
  }
}

// one orthonormalisation round: norms, scaling (and setCiOrb), overlaps
// with the partners, Gram-Schmidt, each over all orbitals of the round
void launch_ortho_round(x2g_ctx *ctx, const GridDev &g, const OrthoOrbital *orbs, int n) {
  const int nb = red_blocks(g);
  for (int b = 0; b < n; b += kRoundItems) {
    const int m = (n - b < kRoundItems) ? n - b : kRoundItems;
    OrthoRound R{};
    bool any_partner = false;
    for (int q = 0; q < m; ++q) {
      const OrthoOrbital &x = orbs[b + q];
      OrthoItem &I = R.it[q];
      I.psi = x.psi;
      I.n = x.n;
      for (int k = 0; k < x.n; ++k) I.o[k] = x.partners[k];
      I.ihomo = x.ihomo;
      I.norm_out = x.norm_out;
      I.ovl_out = x.ovl_out;
      any_partner = any_partner || x.n > 0;
    }
    double *part = reduction_partials(ctx, kMaxK * kRoundItems);
    k_norm_round<<<dim3(nb, m), kThreads, 0, ctx->stream>>>(g, R, part, ctx->bar + kMomentTickets);
    k_scale_round<<<dim3(grid_blocks(g.mxsize), m), kThreads, 0, ctx->stream>>>(g, R);
    ctx->launches += 2;
    if (any_partner) {
      k_overlaps_round<<<dim3(nb, m), kThreads, 0, ctx->stream>>>(g, R, part, ctx->bar + kMomentTickets);
      k_ortho_round<<<dim3(grid_blocks(g.mxsize), m), kThreads, 0, ctx->stream>>>(g, R);
      ctx->launches += 2;
    }
  }
}

// the Gram-matrix form of one iteration's orthonormalisation; false: the
// plan does not fit it (more orbitals or inner products than it holds, too
// few co-resident blocks), the caller takes the round-by-round form
bool launch_orthonormalise_gram(x2g_ctx *ctx, const GridDev &g, const OrthoOrbital *orbs, int n,
                                const int *partner_index) {
  if (n < 1 || n > kGramOrbs) return false;
  GramPlan P{};
  P.n = n;
  P.homo = orbs[0].ihomo != 0;
  for (int j = 0; j < n; ++j) {
    P.psi[j] = orbs[j].psi;
    P.norm_out[j] = orbs[j].norm_out;
    P.ovl_out[j] = orbs[j].ovl_out;
    P.ihomo[j] = orbs[j].ihomo;
    if ((orbs[j].ihomo != 0) != (P.homo != 0)) return false;
    P.npart[j] = orbs[j].n;
    for (int p = 0; p < orbs[j].n; ++p) P.part[j][p] = (signed char)partner_index[j * kGramOrbs + p];
    for (int m = 0; m < kGramOrbs; ++m) P.slot_of[j][m] = -1;
  }
  // slots: every norm, then <Z_a, Z_b> of every pair of a symmetry block
  // (the orbitals a partner chain connects)
  std::vector<int> blk(size_t(n), -1);
  int nblk = 0;
  for (int j = 0; j < n; ++j) {
    if (blk[size_t(j)] < 0) blk[size_t(j)] = nblk++;
    for (int p = 0; p < orbs[j].n; ++p) {
      const int q = partner_index[j * kGramOrbs + p];
      if (q < 0 || q >= j) return false;
      if (blk[size_t(q)] != blk[size_t(j)]) {
        const int from = blk[size_t(q)], to = blk[size_t(j)];
        for (auto &b : blk)
          if (b == from) b = to;
      }
    }
  }
  int ns = 0;
  for (int j = 0; j < n; ++j) {
    P.slot_of[j][j] = (signed char)ns;
    P.sa[ns] = P.sb[ns] = (signed char)j;
    ++ns;
  }
  for (int a = 0; a < n; ++a)
    for (int b = a + 1; b < n; ++b)
      if (blk[size_t(a)] == blk[size_t(b)]) {
        if (ns >= kGramSlots) return false;
        P.slot_of[a][b] = P.slot_of[b][a] = (signed char)ns;
        P.sa[ns] = (signed char)a;
        P.sb[ns] = (signed char)b;
        ++ns;
      }
  P.nslots = ns;
  if (ctx->gram_blocks < 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_orthonormalise_gram, kThreads, 0) !=
        cudaSuccess)
      per_sm = 0;
    (void)cudaGetLastError();
    ctx->gram_blocks = per_sm * ctx->num_sms;
  }
  // two blocks per SM (the passes are latency bound), at most the partials' room
  const int nb = std::min(std::min(2 * ctx->num_sms, ctx->gram_blocks), kRedBlocksMax);
  if (nb < 1) return false;
  double *part = reduction_partials(ctx, ((ns + kMaxK - 1) / kMaxK) * kMaxK);
  if (!part) return false;
  if (cudaMemsetAsync(ctx->bar, 0, 2 * sizeof(unsigned), ctx->stream) != cudaSuccess) return false;
  BarrierDev bar{ctx->bar, ctx->bar + 1, reinterpret_cast<int *>(ctx->bar + 2), ctx->wait_limit_ns};
  GridDev gd = g;
  void *args[] = {&gd, &P, &part, &bar};
  if (cudaLaunchCooperativeKernel((const void *)k_orthonormalise_gram, dim3(nb), dim3(kThreads), args, 0,
                                  ctx->stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  ctx->launches += 1;
  return true;
}

// every round in one cooperative launch; false: the plan does not fit it
// (more orbitals or rounds than its table holds, or too few co-resident
// blocks), the caller then launches round by round
bool launch_orthonormalise(x2g_ctx *ctx, const GridDev &g, const OrthoOrbital *orbs, const int *round_off,
                           int nrounds) {
  const int n = round_off[nrounds];
  if (n > kOrthoItems || nrounds > kOrthoRounds || nrounds < 1) return false;
  const int nb = red_blocks(g);
  if (ctx->ortho_blocks < 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void *)k_orthonormalise, kThreads, 0) !=
        cudaSuccess)
      per_sm = 0;
    (void)cudaGetLastError();
    ctx->ortho_blocks = per_sm * ctx->num_sms;
  }
  if (nb > ctx->ortho_blocks) return false;
  OrthoPlan P{};
  for (int q = 0; q < n; ++q) {
    const OrthoOrbital &x = orbs[q];
    OrthoItem &I = P.it[q];
    I.psi = x.psi;
    I.n = x.n;
    for (int k = 0; k < x.n; ++k) I.o[k] = x.partners[k];
    I.ihomo = x.ihomo;
    I.norm_out = x.norm_out;
    I.ovl_out = x.ovl_out;
  }
  int most = n;  // the norms of every item, or a round's overlap slot groups (kMaxK slots each)
  for (int r = 0; r <= nrounds; ++r) P.round_off[r] = round_off[r];
  for (int r = 0; r < nrounds; ++r) most = std::max(most, kMaxK * (round_off[r + 1] - round_off[r]));
  P.nrounds = nrounds;
  double *part = reduction_partials(ctx, most);
  if (!part) return false;
  if (cudaMemsetAsync(ctx->bar, 0, 2 * sizeof(unsigned), ctx->stream) != cudaSuccess) return false;
  BarrierDev bar{ctx->bar, ctx->bar + 1, reinterpret_cast<int *>(ctx->bar + 2), ctx->wait_limit_ns};
  GridDev gd = g;
  void *args[] = {&gd, &P, &part, &bar};
  if (cudaLaunchCooperativeKernel((const void *)k_orthonormalise, dim3(nb), dim3(kThreads), args, 0, ctx->stream) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  ctx->launches += 1;
  return true;
}

void launch_eahf(x2g_ctx *ctx, const GridDev &g, const double *psi, int isym, int m, const double *coulp,
                 const double *exchp, double *ee_out, double *parts, bool exact) {
  double *part = reduction_partials(ctx, 5);
  const int nb = red_blocks(g);
  double *sums = part + size_t(nb) * 5;
  if (exact)
    k_eahf<true><<<nb, kThreads, 0, ctx->stream>>>(g, psi, isym, m, coulp, exchp, part, sums, ee_out, parts,
                                                   ctx->bar + 3);
  else
    k_eahf<false><<<nb, kThreads, 0, ctx->stream>>>(g, psi, isym, m, coulp, exchp, part, sums, ee_out, parts,
                                                    ctx->bar + 3);
  ctx->launches += 1;
}

void launch_eahf_batch(x2g_ctx *ctx, const GridDev &g, const EahfItem *items, int n, bool exact) {
  const int nb = red_blocks(g);
  for (int b = 0; b < n; b += kEahfItems) {
    const int m = (n - b < kEahfItems) ? n - b : kEahfItems;
    EahfList L{};
    for (int q = 0; q < m; ++q) L.it[q] = items[b + q];
    double *part = reduction_partials(ctx, 5 * kEahfItems + 5 * kEahfItems / 4);
    if (exact)
      k_eahf_batch<true><<<dim3(nb, m), kThreads, 0, ctx->stream>>>(g, L, part, ctx->bar + kMomentTickets);
    else
      k_eahf_batch<false><<<dim3(nb, m), kThreads, 0, ctx->stream>>>(g, L, part, ctx->bar + kMomentTickets);
    ctx->launches += 1;
  }
}

void launch_triples(x2g_ctx *ctx, const GridDev &g, const TripleItem *items, int n, double *out) {
  double *part = reduction_partials(ctx, kMaxK);
  for (int b = 0; b < n; b += kMaxK) {
    const int m = (n - b < kMaxK) ? n - b : kMaxK;
    TripleList L{};
    for (int q = 0; q < m; ++q) L.it[q] = items[b + q];
    k_triples<<<red_blocks(g), kThreads, 0, ctx->stream>>>(g, L, m, part, out + b, ctx->bar + 3);
    ctx->launches += 1;
  }
}

void launch_moments(x2g_ctx *ctx, const GridDev &g, const MomentItem *items, int n, int homo) {
  for (int b = 0; b < n; b += kMomentItems) {
    const int m = (n - b < kMomentItems) ? n - b : kMomentItems;
    double *part = reduction_partials(ctx, 8 * m);
    MomentList L{};
    for (int q = 0; q < m; ++q) L.it[q] = items[b + q];
    k_moments<<<dim3(red_blocks(g), m), kThreads, 0, ctx->stream>>>(g, L, homo, part, ctx->bar + kMomentTickets);
    ctx->launches += 1;
  }
}


}  // namespace x2g

extern "C" int x2g_host_column_plan(int nnu, int nmu, int csize, int groups, int potentials, int *slots, int *maxrows,
                                    int *row0, int *cut, int *kernel_slots, int *kernel_rows, long *smem) {
  using namespace x2g;
  ColPlan p;
  if (potentials < 0 || potentials > 2 || (groups != 1 && groups != 2) || nnu < 31 || nmu < 31 ||
      !column_plan(nnu, nmu, csize, groups, p))
    return set_status(X2G_ERR_SCHEDULE, "no such band plan");
  int pitch = 0;
  const ColKernel k = column_kernel(p, potentials > 0, potentials == 2, std::max(p.pitch, p.warps * 32), pitch);
  if (slots) *slots = p.slots;
  if (maxrows) *maxrows = p.maxrows;
  if (row0) std::copy(p.row0, p.row0 + csize + 1, row0);
  if (cut) std::copy(p.cut, p.cut + csize, cut);
  const int rows = k.fn ? column_rows(p, k.slots) : 0;
  if (kernel_slots) *kernel_slots = k.fn ? k.slots : 0;
  if (kernel_rows) *kernel_rows = rows;
  if (smem) *smem = k.fn ? long(column_smem(rows, pitch, potentials > 0, p.warps * p.groups * 32)) : 0;
  return set_status(X2G_OK, "");
}
