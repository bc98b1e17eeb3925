// Device helpers shared by the kernels of the mixed form.
#pragma once

#include "x2g_internal.h"

namespace x2g {

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// double -> float with round to nearest even, on the integer pipes (GB300
// issues conversion instructions on its narrow FP64 pipe); values beyond the
// float range become infinities, values below its normal range signed zero
__device__ __forceinline__ float narrow_f64(double x) {
  const unsigned hi = unsigned(__double2hiint(x)), lo = unsigned(__double2loint(x)), mag = hi & 0x7fffffffu;
  // 24 bits: 21 from hi, 3 from lo; the remaining 29 round (a carry may go
  // into the exponent)
  const unsigned long long t = ((unsigned long long)mag << 32 | lo) + (0x0fffffffu + (lo >> 29 & 1u));
  unsigned f = unsigned(t >> 29) - (896u << 23);
  f = mag >= (1151u << 20) ? 0x7f800000u : f;
  f = mag > 0x7ff00000u || (mag == 0x7ff00000u && lo != 0) ? 0x7fc00000u : f;
  f = mag < (897u << 20) ? 0u : f;
  return __uint_as_float(hi & 0x80000000u | f);
}

// float -> double by bit manipulation on the integer pipes (GB300 issues
// conversion instructions on its narrow FP64 pipe); exact for normal floats,
// infinities and NaNs; float subnormals (|e| < 1.2e-38, far below any
// correction that matters) become signed zero
__device__ __forceinline__ double widen_f32(float f) {
  const unsigned b = __float_as_uint(f), ex = (b >> 23) & 0xffu, m = b & 0x7fffffu;
  const unsigned sign = b & 0x80000000u;
  if (ex == 0) return __hiloint2double(int(sign), 0);
  const unsigned dex = (ex == 0xffu) ? 0x7ffu : ex + 896u;
  return __hiloint2double(int(sign | (dex << 20) | (m >> 3)), int(m << 29));
}

// u at ext (row, col) with the putin ghost cells (inout.F90:47-80) read as
// the mirrored interior value, negated for odd functions (a sign-bit flip);
// the corner ghosts, never filled by putin, are not reachable by the cross
// stencil
__device__ __forceinline__ double ghost_read(const GridDev &g, const double *u, int row, int col, int isym) {
  bool m = false;
  if (col < 4) {
    col = 8 - col;
    m = true;
  } else if (col > g.nni + 3) {
    col = 2 * g.nni + 6 - col;
    m = true;
  }
  if (row < 4) {
    row = 8 - row;
    m = true;
  }
  const double v = u[row * g.n8 + col];
  return (m && isym != 1) ? __longlong_as_double(__double_as_longlong(v) ^ (1ll << 63)) : v;
}

// FP64 axis extrapolation of one point from its 5 neighbours at stride st
// (sormcsor.F90:94-129 order)
__device__ __forceinline__ double extrap64(const GridDev &g, const double *u, int ij, int st) {
  double v = __dadd_rn(__dmul_rn(g.exeven[0], u[ij + st]), __dmul_rn(g.exeven[1], u[ij + 2 * st]));
  v = __dadd_rn(v, __dmul_rn(g.exeven[2], u[ij + 3 * st]));
  v = __dadd_rn(v, __dmul_rn(g.exeven[3], u[ij + 4 * st]));
  return __dadd_rn(v, __dmul_rn(g.exeven[4], u[ij + 5 * st]));
}

// axis extrapolation of the correction from the five values at stride s
__device__ __forceinline__ float ex5f(const float *ex, const float *p, int s) {
  return ex[0] * p[s] + ex[1] * p[2 * s] + ex[2] * p[3 * s] + ex[3] * p[4 * s] + ex[4] * p[5 * s];
}

// split cluster barrier: arrive releases this thread's earlier shared and
// distributed-shared writes, wait acquires every CTA's released writes
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

}  // namespace x2g
