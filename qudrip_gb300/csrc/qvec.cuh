// qvec.cuh -- inner products of FP64 vectors in integer arithmetic.
//
// GB300 issues one warp-wide FP64 instruction per 76 cycles and SM quarter
// (measured; the same for one active lane as for 32), but a 32 x 32 -> 64-bit
// multiply-add per 4.  A vector is therefore also kept as 55-bit integers on a
// scale of its tile's largest element, u 2^-28 (h 2^28 + l) with |h|, |l| <=
// 2^27, two 32-bit words per real (the 8 bytes a double takes).  A product of
// two of them is three multiply-adds into 64-bit accumulators that cannot
// overflow over 128 complex terms (h h' and h l' + l h'; the dropped l l' is
// below 2^-56 of the scale), so a real multiply-add costs 12 cycles instead of
// 76, and sums across threads are integer adds.  Each element is within 2^-56
// of the tile's largest, so a sum is within some 2^-56 of the product of its
// vectors' norms: what an inner product of FP64 vectors is accurate to.  (An
// element far below its tile's largest keeps fewer bits than FP64 gives it.
// Sums do not need them; stored vectors do, and are not formed from these.)
#pragma once

#include "vec.cuh"

namespace qd {

template <typename VV>
struct QVec;
template <>
struct QVec<double> {
  using T = int2;
};
template <>
struct QVec<cplx> {
  using T = int4;
};

// The scale of a tile from the largest high word among its elements' magnitudes: elements are below
// 2^E.  A tile of zeros (or denormals) quantises to zeros; one with a NaN or infinity gets u = NaN.
struct QScale {
  int E;
  double u;  // 2^(E - 27)
};
__device__ __forceinline__ unsigned q_mag(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned q_mag(cplx v) { return max(q_mag(v.re), q_mag(v.im)); }
__device__ __forceinline__ QScale q_scale(unsigned mag) {
  const int e = (int)(mag >> 20);
  QScale s;
  s.E = e - 1022;
  const int ue = s.E - 27 + 1023;
  if (e == 0x7ff) s.u = __longlong_as_double(0x7ff8000000000000ll);
  else s.u = (ue > 0) ? __hiloint2double(ue << 20, 0) : 0.0;
  return s;
}

// v on the scale 2^E: round(v 2^(55 - E)) as h 2^28 + l.
__device__ __forceinline__ int2 q_fix(double v, int E) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((b >> 52) & 0x7ff);
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | 0x10000000000000ull;
  const int sh = e - 1020 - E;  // at most 2
  long long q;
  if (sh >= 0) q = (long long)(m << min(sh, 2));
  else q = (sh < -54) ? 0ll : (long long)((m + (1ull << (-sh - 1))) >> (-sh));
  if (e == 0) q = 0;
  if (b < 0) q = -q;
  const int h = (int)((q + (1ll << 27)) >> 28);
  return make_int2(h, (int)(q - ((long long)h << 28)));
}
__device__ __forceinline__ int2 q_of(double v, int E) { return q_fix(v, E); }
__device__ __forceinline__ int4 q_of(cplx v, int E) {
  const int2 a = q_fix(v.re, E), b = q_fix(v.im, E);
  return make_int4(a.x, a.y, b.x, b.y);
}

// sum of a b: hh + x 2^-28 in units of the two scales' product
struct QAcc {
  long long hh = 0, x = 0;
  // a + b c in one instruction (from C++ the compiler made 64 x 64-bit products of factors that it had
  // seen computed in 64 bits: 44 instead of 21 multiplier instructions for a complex term)
  static __device__ __forceinline__ void madw(long long& a, int b, int c) {
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(b), "r"(c));
  }
  __device__ __forceinline__ void mac(int ah, int al, int bh, int bl) {
    madw(hh, ah, bh);
    madw(x, ah, bl);
    madw(x, al, bh);
  }
  __device__ __forceinline__ long long value() const { return hh + ((x + (1ll << 27)) >> 28); }
};

// Integer totals of a complex (or real) sum, split so that sums over threads cannot overflow.
struct QSum {
  long long hi;  // units of 2^24
  unsigned lo;   // below 2^24 as set; at most 256 such are added
  __device__ __forceinline__ void set(long long v) {
    hi = v >> 24;
    lo = (unsigned)v & 0xffffffu;
  }
  __device__ __forceinline__ void add(long long h, unsigned l) {
    hi += h;
    lo += l;
  }
  __device__ __forceinline__ double value() const {  // one rounding: hi 2^24 + lo
    return fma((double)hi, 16777216.0, (double)lo);
  }
};
__device__ __forceinline__ QSum q_warp_sum(QSum s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    s.add(__shfl_xor_sync(0xffffffffu, s.hi, o), __shfl_xor_sync(0xffffffffu, s.lo, o));
  s.hi += s.lo >> 24;
  s.lo &= 0xffffffu;
  return s;
}

// <v, w> of quantised elements
template <typename VV>
struct QDot;
template <>
struct QDot<double> {
  QAcc r;
  __device__ __forceinline__ void add(int2 v, int2 w) { r.mac(v.x, v.y, w.x, w.y); }
  __device__ __forceinline__ long long re() const { return r.value(); }
  __device__ __forceinline__ long long im() const { return 0; }
};
template <>
struct QDot<cplx> {
  QAcc r, a, b;
  __device__ __forceinline__ void add(int4 v, int4 w) {  // conj(v) w
    r.mac(v.x, v.y, w.x, w.y);
    r.mac(v.z, v.w, w.z, w.w);
    a.mac(v.x, v.y, w.z, w.w);
    b.mac(v.z, v.w, w.x, w.y);
  }
  __device__ __forceinline__ long long re() const { return r.value(); }
  __device__ __forceinline__ long long im() const { return a.value() - b.value(); }
};

}  // namespace qd
