// On-chip FP32 correction sweep of the mixed form, one column per thread.
//
// One relaxation job per thread-block cluster.  CTA k owns ext rows [row0[k],
// row0[k+1]) and keeps the correction e on them, with 4-row halos, in shared
// memory for all micro-sweeps; a thread owns one ext column of the band, or of
// half of it (kGroups = 2).  In a colour phase a thread updates the points of
// that colour in its column: every fifth row, since the list position p = a
// (N_nu - 2) + b of a point (a, b the places of its row and column in the
// "middle" order, initCBAllocArrays.F90:2503-2544; N_nu - 2 = -1 mod 5) has
// colour p mod 5 = (b - a) mod 5.  Lanes take neighbouring columns and the row
// pitch is a multiple of 32 words, so no load or store has a bank conflict
// whatever rows the lanes are at, and a column's successive points share four
// of the rows they read.  The residual of a thread's points stays in its
// registers.
//
// The middle order runs outwards from the middle row and column, so four
// points next to each middle line have a neighbour of their own colour (the
// seams): columns m, m-1 come before m+2, m+3 (m the last column of the first
// half), rows likewise.  The row seam lies inside one thread's rows, which go
// up the column in list order.  The column seam lies inside one warp, where
// the dependent lanes form their value again from their partner's new one.
//
// A phase: wait for the neighbours' halo values of the last phase, the points
// up the column, the band's first and last rows pushed into the neighbours'
// halos, the CTA's barrier.  A phase never reads a value of its own colour
// outside the band, so pushes and reads of one phase do not meet; the halo
// barriers alternate by the phase's parity.  The pushes are asynchronous stores
// counted on the receiver's barrier: a cluster barrier per phase took 440
// cycles, 665 with plain stores into the neighbours' memory to drain.
//
// Every wait is bounded by the context's limit and looks at its error word.
// After one that runs out (or where the word is set before the launch) a block
// leaves the sweeps at the next sweep's start, tells its cluster, and no block of
// it writes u.
//
// What bounds it: waiting.  An instruction issues in two cycles of five (70 of a
// warp per slot of 32 points: 17 loads and stores, 20 packed operations of two
// roundings each, 12 for potentials, addresses and moves), no pipe is above 52 %:
// the warps wait for their loads, for the instruction before and, 1.5 stalls per
// issue, at the phase's barrier; where a launch is small, for the latency of a
// phase (0.9 us at three slots).  Against the sweep with a list of points per warp
// and a cluster barrier per colour and level (10 sweeps, us): one orbital of 151 x
// 241 58 (106), of 331 x 481 98 (132), six 101 (132), 22 potentials of 331 x 481 174
// (two waves, 382; 210 with relax_f32's order of operations).
#pragma once

#include <cooperative_groups.h>

#include "x2g_device.cuh"
#include "x2g_kernels.cuh"

namespace x2g {

constexpr int kColGuard = 32;  // words before and after the band that idle lanes may read

// Rows the arrays of a CTA hold after the band's first: every thread goes
// through all kM slots of the instantiation, lanes without a point in a slot
// (and bands with fewer) reading on past their rows.
inline int column_rows(const ColPlan &p, int slots) {
  int cut = 0;
  for (int k = 0; k < p.size && p.groups == 2; ++k) cut = p.cut[k] > cut ? p.cut[k] : cut;
  const int over = cut + 5 * slots;
  return (over > p.maxrows ? over : p.maxrows) + 4;
}

// dynamic shared memory of one CTA: the band with halos and guards, omega /
// lhs of the band's points (not for kSep), (b, lhs row term) of its rows, the
// halo barriers and the bytes they count, and every thread's rows by colour
inline size_t column_smem(int rows, int pitch, bool sep, int threads) {
  return (size_t(rows + 4 + (sep ? 0 : rows)) * pitch + 2 * kColGuard + 64) * sizeof(float) +
         size_t(rows) * sizeof(float2) + 80 + size_t(5) * threads * sizeof(unsigned);
}

// The instantiations, by the most points of a colour in a column (null: none
// holds that many).  kPitch...: their row pitch and most threads of a group;
// pair: two CTAs per SM.
constexpr int kPitchThin = 160, kPitchSlim = 256, kPitchNarrow = 352, kPitchWide = 512, kPitchBroad = 544, kPitchFlat = 800;
struct ColKernel {
  const void *fn;
  int slots;
};
ColKernel column_kernel_split(int slots, bool sep);  // narrow, two threads per column
ColKernel column_kernel_pair(int slots, bool sep);   // narrow, two CTAs per SM (sep only)
ColKernel column_kernel_wide(int slots, bool sep);   // wide
ColKernel column_kernel_broad(int slots, bool sep);  // broad
ColKernel column_kernel_slim(int slots, bool sep);   // tall grids of few columns, two threads per column
ColKernel column_kernel_thin(int slots, bool sep);   // the same, of fewer still
ColKernel column_kernel_flat(int slots, bool sep);   // many columns, few rows
// The instantiation for a plan whose columns need a pitch of `need` (pair: two
// CTAs per SM), and its pitch.
inline ColKernel column_kernel(const ColPlan &p, bool sep, bool pair, int need, int &pitch) {
  pitch = kPitchNarrow;
  if (pair) return p.groups == 1 && need <= pitch ? column_kernel_pair(p.slots, sep) : ColKernel{nullptr, 0};
  if (need <= kPitchNarrow) {
    if (p.groups != 2) return {nullptr, 0};
    // five slots reach 800 rows; beyond, the largest cluster takes more of them
    // (one orbital of 151 x 811 89 us, in the persistent bands 238; 241 x 901 114
    // and 253, 271 x 811 126 and 251)
    if (p.slots <= 5) return column_kernel_split(p.slots, sep);
    if (p.size != kMaxCluster) return {nullptr, 0};
    if (need <= kPitchThin && p.slots > 10) {
      pitch = kPitchThin;
      return column_kernel_thin(p.slots, sep);
    }
    if (need <= kPitchSlim) {
      pitch = kPitchSlim;
      return column_kernel_slim(p.slots, sep);
    }
    return column_kernel_split(p.slots, sep);
  }
  if (p.groups != 1) return {nullptr, 0};
  // 541 x 31: 93 us, in the persistent bands 252
  pitch = need <= kPitchWide ? kPitchWide : need <= kPitchBroad ? kPitchBroad : kPitchFlat;
  if (need > pitch) return {nullptr, 0};
  return pitch == kPitchWide    ? column_kernel_wide(p.slots, sep)
         : pitch == kPitchBroad ? column_kernel_broad(p.slots, sep)
                                : column_kernel_flat(p.slots, sep);
}

namespace {

__device__ __forceinline__ unsigned smem_addr(const void *p) { return unsigned(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void st_cta(unsigned addr, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned in_cta(unsigned addr, int rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
  return a;
}
// store into another CTA's shared memory, counted on that CTA's barrier
__device__ __forceinline__ void push_halo(unsigned addr, float v, unsigned bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v), "r"(bar)
               : "memory");
}
// (negative: nothing)
__device__ __forceinline__ void expect_bytes(unsigned bar, int bytes) {
  if (bytes >= 0)
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool poll_bar(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
// the same without suspending
__device__ __forceinline__ bool test_bar(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
// a wait for a neighbour's halo values, a few polls as a rule; false: it ran
// out (now recorded), or another one did
__device__ __forceinline__ bool wait_halo(unsigned bar, unsigned parity, const BarrierDev &b) {
  if (b.limit_ns != 0 ? poll_bar(bar, parity) : test_bar(bar, parity)) return true;
  unsigned long long t0 = 0;
  for (unsigned k = 1; b.limit_ns != 0; ++k) {
    if (poll_bar(bar, parity)) return true;
    if ((k & 15u) != 0) continue;
    if (*(volatile int *)b.err) return false;
    const unsigned long long now = globaltimer();
    if (t0 == 0) t0 = now;
    if (now - t0 >= b.limit_ns) break;
  }
  atomicCAS(b.err, 0, X2G_ERR_TIMEOUT);
  return false;
}

struct ColThread {
  float wl[4], wr[4];  // kSep: nu weights of the neighbours at distance 4, 3, 2, 1
  float cs;            // kSep: the seam partner's weight
  float d, lq, omega, omega1;
  int lane, src;        // this lane and the column seam's partner lane (itself: no partner)
  int warp, seam_warp;  // equal: this warp holds the column seam
};

// two products and sums, sums or products at once, each rounded as alone
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(a));
  return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

__device__ __forceinline__ float rcp_fast(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// the new value of a point with residual r from its column's rows v[0..8]
// (-4..4), its row's columns h[0..3] (-4..-1) and h[4..7] (1..4), b of its row
// and t: omega / lhs, or the lhs row term (kSep); the operations and roundings
// of relax_f32, those along mu and nu in one instruction
template <bool kSep>
__device__ __forceinline__ float col_value(const ColPlan &p, const ColThread &T, const float *v, const float *h, float b,
                                           float t, float r) {
  if (kSep) {
    // a neighbour and its mirror image, weighted by dmu2 +- b dmu1 along mu
    // and by dni2 +- d dni1 (fixed for the column) along nu, in one instruction
    const unsigned long long *m1 = reinterpret_cast<const unsigned long long *>(p.m1);
    const unsigned long long *m2 = reinterpret_cast<const unsigned long long *>(p.m2);
    unsigned long long cc = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned long long wm = fma2(pack2(b, b), m1[q], m2[q]);
      cc = q == 0 ? mul2(wm, pack2(v[q], v[8 - q])) : fma2(wm, pack2(v[q], v[8 - q]), cc);
      cc = fma2(pack2(T.wl[q], T.wr[q]), pack2(h[q], h[7 - q]), cc);
    }
    const float2 sum = unpack2(cc);
    const float w = T.omega * rcp_fast(t - T.lq);
    float out = __fmaf_rn(T.omega1, v[4], w * (r - (sum.x + sum.y)));
    if (T.warp == T.seam_warp) {
      // the partner column's change since the old value used above, weighted
      // (0 without a partner)
      out = __fmaf_rn(-w * T.cs, __shfl_sync(0xffffffffu, out - v[4], T.src), out);
    }
    return out;
  }
  const unsigned long long *c2 = reinterpret_cast<const unsigned long long *>(p.c2);
  const unsigned long long *c1 = reinterpret_cast<const unsigned long long *>(p.c1);
  unsigned long long s2 = 0, s1 = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const unsigned long long lo = pack2(v[q], h[q]), hi = pack2(v[8 - q], h[7 - q]);
    const unsigned long long sum = add2(lo, hi), dif = fma2(hi, *reinterpret_cast<const unsigned long long *>(&p.neg), lo);
    s2 = q == 0 ? mul2(c2[q], sum) : fma2(c2[q], sum, s2);
    s1 = q == 0 ? mul2(c1[q], dif) : fma2(c1[q], dif, s1);
  }
  const float2 d2 = unpack2(s2), d1 = unpack2(s1);
  const float w = t;
  const float mu = __fmaf_rn(b, d1.x, d2.x);
  float out = __fmaf_rn(T.omega1, v[4], w * (r - __fmaf_rn(T.d, d1.y, mu + d2.y)));
  if (T.warp == T.seam_warp) {
    // the partner column's new value in place of its old one (a lane and its
    // partner have the same rows, so both have a point here or neither)
    const float other = __shfl_sync(0xffffffffu, out, T.src);
    if (T.src != T.lane) {
      const float l4 = T.src + 4 == T.lane ? other : h[0], l2 = T.src + 2 == T.lane ? other : h[2];
      float dn2 = p.c2[0].y * (l4 + h[7]), dn1 = p.c1[0].y * (l4 - h[7]);
      dn2 = __fmaf_rn(p.c2[1].y, h[1] + h[6], dn2);
      dn1 = __fmaf_rn(p.c1[1].y, h[1] - h[6], dn1);
      dn2 = __fmaf_rn(p.c2[2].y, l2 + h[5], dn2);
      dn1 = __fmaf_rn(p.c1[2].y, l2 - h[5], dn1);
      dn2 = __fmaf_rn(p.c2[3].y, h[3] + h[4], dn2);
      dn1 = __fmaf_rn(p.c1[3].y, h[3] - h[4], dn1);
      out = __fmaf_rn(T.omega1, v[4], w * (r - __fmaf_rn(T.d, dn1, mu + dn2)));
    }
  }
  return out;
}

// kM: most points of one colour in a thread's rows; kSep: potentials, omega /
// lhs from a row and a column term (fast reciprocal: the correction sweep is
// the inner solver of the FP64 defect correction, whose fixed point does not
// depend on it); kPitch: the row pitch and most threads of a group
template <int kM, bool kSep, int kPitch, int kGroups, int kMinBlocks>
__global__ void __launch_bounds__(kPitch * kGroups, kMinBlocks)
    k_columns(GridDev g, const __grid_constant__ ColPlan p, const __grid_constant__ JobTable jobs, int nsweeps,
              int free, BarrierDev limit) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int C = p.size, rank = int(cl.block_rank());
  const JobDev &J = jobs.j[blockIdx.x / C];
  const bool even = (J.isym == 1);
  const int n8 = g.n8, nni = g.nni;
  const int R0 = p.row0[rank], n = p.row0[rank + 1] - R0;
  extern __shared__ __align__(16) float smem[];
  const int tid = int(threadIdx.x), nt = int(blockDim.x), lane = tid & 31;
  // through a shuffle, so that the branches on it are known to be uniform in
  // the warp (as divergent ones they took 85 of 140 instructions per update)
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int group = (kGroups == 2 && warp >= p.warps) ? 1 : 0;
  const int col = 5 + tid - group * p.warps * 32 - p.shift;
  const int ne = (p.rows + 4) * kPitch + 2 * kColGuard + 64;
  float *const E = smem + kColGuard + 4 * kPitch;  // band row 0, ext column 0
  float *const W = smem + ne;
  float2 *const BL = reinterpret_cast<float2 *>(W + (kSep ? 0 : p.rows * kPitch));
  const int w_off = int(W - E);
  const bool in = col >= 5 && col <= nni + 2;  // the thread has a column
  const int err0 = tid == 0 ? *(volatile int *)limit.err : 0;
  const int nu = in ? col - 4 : 1;
  for (int k = tid; k < ne; k += nt) smem[k] = 0.0f;
  for (int k = tid; k < p.rows; k += nt) {
    const int mu = (k < n ? R0 + k : R0) - 4;
    // potentials: lhs = f3 + idel^2 e with e = e_mu - e_nu, the row term in
    // FP64, then both terms in FP32
    BL[k] = make_float2((J.kind >= 1 ? g.bpot_mu32 : g.borb_mu32)[mu],
                        kSep ? narrow_f64(fma(J.idel2, g.e_mu[mu], g.f3_mu[mu])) : 0.0f);
  }
  // this thread's rows [g0, g1) of the band
  const int g0 = group ? p.cut[rank] : 0, g1 = (kGroups == 2 && !group) ? p.cut[rank] : n;
  if (!kSep && in) {
#pragma unroll 4
    for (int lr = g0; lr < g1; ++lr) W[lr * kPitch + col] = J.w32[(R0 + lr - 4) * nni + nu];
  }
  // A row below the seam (the first half of the middle order) has a = nmux -
  // 1 - row, one above it a = row - 5; so lower rows of a column have colour b
  // - a = b - nmux + 1 + row, upper ones b + 5 - row; the seam-free colouring
  // is col - row.  Part A of the thread's rows ends at the seam, if that lies
  // in them; part B starts there.
  const int nmux = (g.nmu + 7) / 2, nnix = (nni + 7) / 2;  // first row of the upper half; 1-based last column of the first
  const int A0 = R0 + g0, A1 = R0 + g1;
  const bool two = !free && A0 < nmux && A1 > nmux;
  const bool lower = !free && A0 < nmux;
  const int na = two ? nmux - A0 : g1 - g0;
  const int ma = (na + 4) / 5, mm = ma + (g1 - g0 - na + 4) / 5;  // slots of part A, of all rows
  const int b = (col < nnix) ? nnix - 1 - col : col - 5;
  // Fixed for the launch, packed and partly in shared memory to keep the
  // registers for the residuals.  info, per colour: the points of part A (bits 0..7), whether the column's
  // first / last point is within four rows of the band's start / end (8, 9),
  // the first row (10..19) and the last row of both parts (20..31).  parts:
  // slots of part A (0..7), of both (8..15); part B: rows (16..23), its first
  // row for colour 0 as an offset mod 5 (24..26).
  unsigned *const info = reinterpret_cast<unsigned *>(BL + p.rows) + 20 + tid;  // [colour * threads]
  unsigned parts = unsigned(two ? ma : 255) | unsigned(g1 - g0 - na) << 16 | unsigned(((b - nmux) % 5 + 5) % 5) << 24;
  const int row_b = g0 + na - 5 * ma;  // part B's first row as if it had part A's slots before it
  float r[5][kM];
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    const int k = lower ? nmux - 1 - b - A0 + c : (free ? col : b) - A0 - c;
    const int fa = (k % 5 + 5) % 5, fb = ((b - nmux - c) % 5 + 5) % 5;
    const int ca = in ? (na - fa + 4) / 5 : 0, cb = in ? (g1 - g0 - na - fb + 4) / 5 : 0;
    const int last = two ? g0 + na + fb + 5 * (cb - 1) : g0 + fa + 5 * (ca - 1);
    info[c * nt] = unsigned(ca) | (in && ca > 0 && g0 + fa < 4 ? 0x100u : 0u) | (in && ca > 0 && last >= n - 4 ? 0x200u : 0u) |
              unsigned(g0 + fa) << 10 | unsigned(max(last, 0)) << 20;
    const float *s = J.r32 + (R0 + g0 - 4) * nni + nu;
#pragma unroll
    for (int m = 0; m < kM; ++m) {
      const bool has = (m < ma) ? m < ca : m < mm && m - ma < cb;
      r[c][m] = has ? s[((m < ma) ? fa + 5 * m : na + fb + 5 * (m - ma)) * nni] : 0.0f;
    }
  }
  // halo barriers: [side][phase parity], side 0 the values from the CTA before
  // and the bytes that each colour's phase receives, [side][colour]; failed: a
  // wait has run out, of this block (or, before it began, elsewhere); skip: one
  // of the cluster's blocks, which write it once they are through
  const unsigned bar0 = smem_addr(BL + p.rows);
  int *const s_bytes = reinterpret_cast<int *>(BL + p.rows) + 8;
  volatile int *const failed = s_bytes + 10, *const skip = s_bytes + 11;
  const bool has_up = rank > 0, has_dn = rank < C - 1;
  // this thread's column at band row 0 in the neighbours' arrays
  const unsigned own = smem_addr(E + col);
  const unsigned up = has_up ? in_cta(own, rank - 1) + unsigned((R0 - p.row0[rank - 1]) * kPitch * 4) : 0u;
  const unsigned dn = has_dn ? in_cta(own, rank + 1) - unsigned(n * kPitch * 4) : 0u;
  const unsigned up_bar = has_up ? in_cta(bar0, rank - 1) + 16u : 0u;  // its side 1
  const unsigned dn_bar = has_dn ? in_cta(bar0, rank + 1) : 0u;
  if (tid == 0) {
    *failed = err0;
    *skip = 0;
  }
  if (tid < 4)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + 8u * tid) : "memory");
#pragma unroll 1
  for (int c = 0; c < 5; ++c) {
    // rows R0-4..R0-1 and R0+n..R0+n+3 of this column: one of them has the
    // colour unless the row that would is the fifth
    auto place = [&](int row) {  // (row's colour - c) mod 5
      const int k = free ? col - row : row < nmux ? b - nmux + 1 + row : b - row;
      return ((k - c) % 5 + 5) % 5;
    };
    int above = 0, below = 0;
#pragma unroll
    for (int k = 1; k <= 4; ++k) {
      above += place(R0 - k) == 0;
      below += place(R0 + n - 1 + k) == 0;
    }
    const int na_ = __syncthreads_count(in && group == 0 && has_up && above > 0);
    const int nb_ = __syncthreads_count(in && group == 0 && has_dn && below > 0);
    if (tid == 0) {
      s_bytes[c] = has_up ? 4 * na_ : -1;
      s_bytes[5 + c] = has_dn ? 4 * nb_ : -1;
    }
  }
  ColThread T;
  T.omega = J.omegaf;
  T.omega1 = J.omega1f;
  T.d = in ? g.d_nu32[nu] : 0.0f;
  T.lq = (kSep && in) ? narrow_f64(J.idel2 * g.e_nu[nu]) : 0.0f;
  if (kSep) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      T.wl[q] = __fmaf_rn(T.d, g.dni1f[q], g.dni2f[q]);
      T.wr[q] = __fmaf_rn(-T.d, g.dni1f[q], g.dni2f[q]);
    }
  }
  // column seam: 1-based columns nnix + 2 and nnix + 3 read the new values of
  // nnix and nnix - 1, two and four columns to their left
  T.lane = lane;
  T.src = lane - (free ? 0 : (col == nnix + 1) ? 2 : (col == nnix + 2) ? 4 : 0);
  if (kSep) T.cs = T.src == lane ? 0.0f : T.src + 2 == lane ? T.wl[2] : T.wl[0];
  T.warp = warp;
  T.seam_warp = free ? -1 : (nnix - 7 + p.shift) / 32 + group * p.warps;
  // arm both parities of a side for the values of the first two phases.  After
  // a failed wait (-1) the barrier's last turn may still be open, and one more
  // arrival than it has room for faults; nothing waits for it any more
  auto arm = [&](int side, int c, int parity) {
    expect_bytes(bar0 + unsigned(16 * side + 8 * parity), *(volatile int *)(s_bytes + 5 * side + c));
  };
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncthreads();
  if (tid < 4) arm(tid >> 1, tid & 1, tid & 1);
  cluster_arrive();  // this band is zeroed and its barriers armed: neighbours may push into its halos
  cluster_wait();
  int phase = 0;
  const bool push_up = has_up && group == 0, push_dn = has_dn && g1 == n;
  bool wait_up = push_up, wait_dn = push_dn;
  for (int s = 0; s < nsweeps; ++s) {
    // only this block's waits write the flag, and none comes between the barrier
    // before this and the next one, so its threads agree; it stays until the
    // whole cluster is through
    if (*failed) break;
    if (s > 0) {
      // axis of e for the band's rows; the mu=1 row is band row -1 of the
      // first CTA
      if (rank == 0 && in && group == 0) {
        E[-kPitch + col] = even ? ex5f(g.exevenf, E - kPitch + col, kPitch) : 0.0f;
      }
      for (int k = tid; k < 2 * n; k += nt) {
        float *const q = E + (k / 2) * kPitch + (k % 2 == 0 ? 4 : nni + 3);
        *q = even ? ex5f(g.exevenf, q, k % 2 == 0 ? 1 : -1) : 0.0f;
      }
      __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < 5; ++c, ++phase) {
      if (phase > 0) {
        // the neighbours' values of phase - 1
        const int use = (phase - 1) >> 1, parity = (phase - 1) & 1;
        bool ok = true;
        if (wait_up) ok = wait_halo(bar0 + 8u * parity, use & 1, limit);
        if (ok && wait_dn) ok = wait_halo(bar0 + 16u + 8u * parity, use & 1, limit);
        if (!ok) {  // to the end of this sweep with the values that are there
          *failed = 1;
#pragma unroll 1
          for (int k = 0; k < 10; ++k) *(volatile int *)(s_bytes + k) = -1;
          wait_up = wait_dn = false;
        }
      }
      // formed anew in every phase: hoisted out of the sweeps, the addresses of
      // all phases would not fit the registers
      const unsigned q = info[c * nt];
      unsigned pt = parts;
      asm volatile("" : "+r"(pt));
      pt = __shfl_sync(0xffffffffu, pt, 0) & 0xffffffu;  // uniform but for the column's offset
      const int ma = int(pt & 0xffu);
      const int row = int((q >> 10) & 0x3ffu);
      float *e = E + row * kPitch + col;
      const float2 *bl = BL + row;
      int cnt = int(q & 0xffu);
      float v[9];  // rows -4..4 of the column around the point
#pragma unroll
      for (int m = 0; m < kM; ++m) {
        if (m == 0) {
#pragma unroll
          for (int i = 5; i < 9; ++i) v[i] = e[(i - 9) * kPitch];
        } else if (m == ma) {  // on the other side of the row seam
          int fb = int(parts >> 24) - c;
          fb = fb < 0 ? fb + 5 : fb;
          e = E + (row_b + fb) * kPitch + col;
          bl = BL + row_b + fb;
          cnt = cnt > 0 ? ma + (int(pt >> 16) - fb + 4) / 5 : 0;
#pragma unroll
          for (int i = 5; i < 9; ++i) v[i] = e[(5 * m + i - 9) * kPitch];
        }
        // rows -4..-1 are rows 1..4 of the point before
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = v[i + 5];
#pragma unroll
        for (int i = 4; i < 9; ++i) v[i] = e[(5 * m + i - 4) * kPitch];
        float h[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          h[i] = e[5 * m * kPitch + i - 4];
          h[4 + i] = e[5 * m * kPitch + i + 1];
        }
        const float2 x = bl[5 * m];
        const float out = col_value<kSep>(p, T, v, h, x.x, kSep ? x.y : e[5 * m * kPitch + w_off], r[c][m]);
        if (m < cnt) e[5 * m * kPitch] = out;
      }
      // the band's first and last four rows, into the neighbours' halos
      if (s < nsweeps - 1 || c < 4) {
        const unsigned at = 8u * (phase & 1);
        if (push_up && (q & 0x100u)) push_halo(up + unsigned(row * kPitch * 4), E[row * kPitch + col], up_bar + at);
        if (push_dn && (q & 0x200u)) {
          const int last = int(q >> 20);
          push_halo(dn + unsigned(last * kPitch * 4), E[last * kPitch + col], dn_bar + at);
        }
      }
      __syncthreads();
      // every thread has waited for phase - 1: its barriers' next turn
      if (phase > 0 && tid < 2) arm(tid, (c + 1) % 5, (phase - 1) & 1);
    }
  }
  if (tid < C && *failed) st_cta(in_cta(smem_addr(s_bytes + 11), tid), 1);
  cluster_arrive();
  cluster_wait();  // no CTA leaves while a neighbour may still write its halo
  if (*skip) {
    // u stays as it was.  Values pushed before the cluster's barrier and not
    // waited for may be on their way into this CTA's memory for a microsecond:
    // it is kept for a hundred
    const unsigned long long t0 = globaltimer();
    for (int k = 0; k < 1024 && globaltimer() - t0 < 100000; ++k) __nanosleep(1000);
    return;
  }
  // u += e on the band, then the FP64 axis of u for its rows (the mu=1 row
  // and the corners by the first CTA)
  double *const u = J.u;
  if (in) {
    const int ij = R0 * n8 + col;
#pragma unroll 1
    for (int lr = g0; lr < g1; lr += 8) {
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (lr + q < g1) v[q] = u[ij + (lr + q) * n8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (lr + q < g1) u[ij + (lr + q) * n8] = v[q] + widen_f32(E[(lr + q) * kPitch + col]);
    }
  }
  __syncthreads();
  const int nrow4 = (rank == 0) ? nni - 2 : 0;
  for (int k = tid; k < nrow4 + 2 * n; k += nt) {
    if (k < nrow4) {
      const int ij = 4 * n8 + 5 + k;
      u[ij] = even ? extrap64(g, u, ij, n8) : 0.0;
    } else {
      const int q = k - nrow4, row = R0 + q / 2, side = q % 2;
      const int ij = row * n8 + (side == 0 ? 4 : nni + 3);
      u[ij] = even ? extrap64(g, u, ij, side == 0 ? 1 : -1) : 0.0;
    }
  }
  __syncthreads();
  if (rank == 0 && tid < 2) {
    const int ij = 4 * n8 + (tid == 0 ? 4 : nni + 3);
    u[ij] = even ? extrap64(g, u, ij, tid == 0 ? 1 : -1) : 0.0;
  }
}

}  // namespace
}  // namespace x2g
