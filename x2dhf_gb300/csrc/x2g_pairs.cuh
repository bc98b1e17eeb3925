// FP64 arithmetic on the integer pipes, bit for bit the FP64 unit's.  A warp's
// FP64 instruction takes the SM 19 cycles (76 of each quarter's when all four
// want it); the four that pair_products replaces, 304, are about 150 integer
// instructions that issue beside it.
#pragma once

#include <cuda_runtime.h>

namespace x2g {

// A constant factor: its mantissa with the leading bit at bit 63, its exponent
// field and its sign bit (a normal number).
struct PairCoef {
  unsigned hi, lo;
  int ex;
  unsigned sign;
};

namespace pairs {

__host__ __device__ __forceinline__ int top_zeros(unsigned long long x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}
__host__ __device__ __forceinline__ unsigned long long bits_of(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long b;
  __builtin_memcpy(&b, &x, 8);
  return b;
#endif
}
__host__ __device__ __forceinline__ double of_bits(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  __builtin_memcpy(&x, &b, 8);
  return x;
#endif
}

// 1 if 64 bits with the leading one at bit 63 round up to 53 (ties to even);
// bit 0 also stands for everything below it
__host__ __device__ __forceinline__ unsigned rounds_up(unsigned lo) {
  return (lo & 0x7ffu) + (lo >> 11 & 1u) > 0x400u ? 1u : 0u;
}

// m (leading one at bit 63, bit 0 sticky) rounded to 53 bits, times c, rounded:
// the double's bits; ex: the exponent field of m as 1.x
__host__ __device__ __forceinline__ unsigned long long round_times(unsigned long long m, int ex, const PairCoef &c) {
  unsigned lo = unsigned(m), hi = unsigned(m >> 32);
  const unsigned long long r =
      ((unsigned long long)hi << 32 | (lo & ~0x7ffu)) + ((unsigned long long)rounds_up(lo) << 11);
  lo = unsigned(r);
  hi = unsigned(r >> 32);
  if (!(hi & 0x80000000u)) {  // up to the next power of two
    hi = 0x80000000u;
    ++ex;
  }
  // the product's upper 64 bits; the lower ones only as zero or not
  const unsigned long long p0 = (unsigned long long)lo * c.lo;
  const unsigned long long p1 = (unsigned long long)lo * c.hi + (p0 >> 32);
  const unsigned long long p2 = (unsigned long long)hi * c.lo + unsigned(p1);
  const unsigned long long p = (unsigned long long)hi * c.hi + (p1 >> 32) + (p2 >> 32);
  const unsigned low = unsigned(p2) | unsigned(p0);
  unsigned ph = unsigned(p >> 32), pl = unsigned(p);
  const int n = ph & 0x80000000u ? 0 : 1;
  ph = n ? ph << 1 | pl >> 31 : ph;
  pl = n ? pl << 1 | unsigned(p2) >> 31 : pl;
  // (p2's top bit moved up: counted in low all the same, which can only turn
  // a tie away from a tie when it is set, and then pl's bit 0 is set too)
  pl |= low != 0 ? 1u : 0u;
  const int e = ex + c.ex - 1023 - n;  // the result's exponent field less one
  return (((unsigned long long)ph << 32 | pl) >> 11) + rounds_up(pl) + ((unsigned long long)unsigned(e) << 52);
}

}  // namespace pairs

// t2 = c2 (x + y) and t1 = c1 (x - y), every operation rounded to nearest as
// the FP64 unit does; false (nothing written) where the larger of |x| and |y|
// is zero or so near an end of the exponent range that a result could leave it
__host__ __device__ __forceinline__ bool pair_products(double x, double y, const PairCoef &c2, const PairCoef &c1,
                                                       double &t2, double &t1) {
  using namespace pairs;
  const unsigned long long kMag = ~(1ull << 63);
  const unsigned long long xb = bits_of(x), yb = bits_of(y), xm = xb & kMag, ym = yb & kMag;
  const bool swap = ym > xm;
  const unsigned long long bm = swap ? ym : xm, sm = swap ? xm : ym;
  const int ex = int(unsigned(bm >> 52)), d = ex - int(unsigned(sm >> 52));
  if (unsigned(ex - 300) > 1400u) return false;
  const unsigned xs = unsigned(xb >> 32) & 0x80000000u, ys = unsigned(yb >> 32) & 0x80000000u;
  const bool same = xs == ys;
  const unsigned long long kOne = 1ull << 52, kFrac = kOne - 1;
  const unsigned long long a = (kOne | (bm & kFrac)) << 10, b = (kOne | (sm & kFrac)) << 10;
  // b on a's scale, bit 0 standing for what is shifted out (a subnormal b is
  // shifted out as a whole)
  const int s = d < 63 ? d : 63;
  unsigned long long t = b >> s;
  t |= (t << s) != b ? 1ull : 0ull;
  t = sm == 0 ? 0ull : t;
  // |x| + |y| and |x| - |y| with the leading one at bit 63
  unsigned long long p = a + t, q = a - t;
  const int n = int(p >> 63) ^ 1;
  p <<= n;
  const int z = top_zeros(q) & 63;
  q <<= z;
  const PairCoef &cp = same ? c2 : c1, &cq = same ? c1 : c2;
  const unsigned bs = swap ? ys : xs;
  unsigned long long rp = round_times(p, ex + 1 - n, cp);
  unsigned long long rq = q == 0 ? 0ull : round_times(q, ex + 1 - z, cq);
  // the sum has the larger one's sign, the difference that of x or -y; equal
  // values leave +0
  const unsigned ds = swap ? bs ^ 0x80000000u : bs;
  const unsigned sp = (same ? bs : ds) ^ cp.sign, sq = (q == 0 ? 0u : same ? ds : bs) ^ cq.sign;
  rp |= (unsigned long long)sp << 32;
  rq |= (unsigned long long)sq << 32;
  t2 = of_bits(same ? rp : rq);
  t1 = of_bits(same ? rq : rp);
  return true;
}

// c as a PairCoef; false if it is not a normal number of moderate size
inline bool pair_coef(double c, PairCoef &out) {
  const unsigned long long b = pairs::bits_of(c);
  out.ex = int(unsigned(b >> 52) & 0x7ffu);
  out.sign = unsigned(b >> 32) & 0x80000000u;
  const unsigned long long m = ((1ull << 52) | (b & ((1ull << 52) - 1))) << 11;
  out.hi = unsigned(m >> 32);
  out.lo = unsigned(m);
  return out.ex > 923 && out.ex < 1123;
}

}  // namespace x2g
