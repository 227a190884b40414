// lanres.cu -- the Lanczos recurrence as one persistent launch.
//
// A step (krylov.cu) is a product, three inner products, an update and a norm.
// Launched step by step it cannot take less than its launches and their
// reductions: at dim 12,870 the one-launch step of the uniform-coupling form
// took 18 us, at dim 184,756 the three kernels of a complex step 66 us, where
// the arithmetic is 0.3 and 15.  Here the grid (clusters of eight blocks, one
// block per SM) stays for all steps, a block keeps its rows of the last two
// vectors and of w in shared memory, and the blocks exchange one small sum a
// step (gridx.cuh): the inner products of the product with the two last
// vectors, and, from the update before, the norm of the newest vector and its
// overlap with the one before, which scale everything.  The product gathers
// the newest vector as its rows arrive from the other blocks.
//
// The block's sums of its threads' partial sums are integer adds: a warp-wide
// FP64 add takes 76 cycles on GB300 and a butterfly of seven values over
// sixteen warps 10,600; as 57-bit integers on the scale of the largest partial
// sum (53 bits across warps) it is 2,200: one rounding at 2^-54 of the largest a
// warp and at 2^-58 a thread, where the tree of FP64 adds has nine.
//
// Hermitian::LanczosSolver runs here with its basis kept, where the reference
// forms every vector a second time for the Ritz vector.
//
// Measured (GB300): a step at dim 12,870 (uniform couplings) 18 -> 9 us, complex
// at dim 184,756 61 -> 24 us (the FP64 product is 12 of them, the exchange most
// of the rest; 28 us before a block took its rows in order of their length),
// real couplings per bond there 41 -> 19 us; Hermitian solver at dim 4,900 2.3
// -> 0.42 ms a solve.
//
// A matrix-free solve forms its rows from the compiled transitions (couplings that differ: a test per
// transition and a rank per entry, 33 us a step at dim 184,756 against 19 on the stored matrix) or from the
// block tables of the sector (uniform couplings: 917 us a solve at 18 sites against 830 on the stored columns,
// the same bits); it reads no stored matrix.
// Mean error against 64-bit references over 24 random cases each: ground-state
// eigenvalues 7.2e-16 (launched step by step: 8.1e-16), evolved states 2.19e-15
// (2.24e-15), the Hermitian solver's eigenvalues 4.7e-16 (5.2e-16).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fxblock.cuh"
#include "gridx.cuh"
#include "lanres.cuh"
#include "mfrow.cuh"
#include "qvec.cuh"
#include "scan.cuh"

namespace qd {

constexpr int kLanThreads = 512;
constexpr int kLanMinRows = 96;  // rows of a block before the grid covers every SM
// Clusters of eight keep the exchange short; of four cover more SMs (144 of 152 against 120, which is
// what one block per SM and whole clusters per GPC leave), which pays once a block's rows outweigh it.
// Complex vectors, four steps of m = 32, on eight and four: 48,620 rows 1,881 and 1,791 us, 184,756 4,510
// and 3,941; real, whole solves: 48,620 rows 793 and 836 us, 92,378 1,032 and 1,046, 184,756 1,478 and
// 1,402, 705,432 5,365 and 4,220.  Clusters of two (152 SMs) were at most 2% faster and up to 10% slower.
template <typename VV>
constexpr int64_t lan_wide_rows() {
  return sizeof(VV) == sizeof(double) ? 1 << 17 : 1 << 15;
}
constexpr int kLanMaxExp = 32;
// Fixed-point copies of the basis during a run on uniform couplings (given back at its end): 122 steps a launch
// at 65,536 rows.
constexpr int64_t kLanCopyBytes = 128ll << 20;
// A block's rows of three vectors and their order by length; the transitions' 16-byte words follow.
template <typename VV>
__host__ __device__ constexpr size_t lan_rows_smem(int rows) {
  return ((size_t)rows * (3 * sizeof(VV) + sizeof(short)) + 15) / 16 * 16;
}
static_assert(sizeof(MfEntry) % 16 == 0 && alignof(MfEntry) <= 16 &&
                  2 * sizeof(uint2) + sizeof(cplx) <= sizeof(MfEntry),
              "staged behind the rows in either form, aligned");

template <typename MV, typename VV>
struct LanArgs {
  int64_t n, ld;
  int rows;               // most rows of a block
  const int* row_first;   // first row of each block, then n
  const int64_t* rowptr;
  const int32_t* colidx;
  const MV* vals;
  const double* fxdiag;  // uniform couplings: the diagonal (null: zero), c 2^-F and F
  double cF;
  int F;
  const int32_t *fxptr, *fxcol;  // its off-diagonal columns
  XInt* XV;              // fixed-point copy of V[k] at XV + (k - first + 1) ld
  VV* V;
  int first, last;
  double stop_below;
  VV *alpha, *beta;
  double *nrm, *scl;
  int* stop;
  int* ovf;
  // the Krylov exponential
  const cplx* psi;  // the state, read in the first step only
  cplx* out;        // the new one; may be psi
  double h;
  int* act;
  long long* matvecs;
  double* slots;
  int xstride;
  GridX X;
};

// Columns from the compiled transitions: no stored matrix is read.
template <typename MV, typename VV>
struct LanMfArgs : LanArgs<MV, VV> {
  MfRows mf;
  Mf32 mf32;        // the ranking in 32 bits where that holds (nf > 0)
  BlockTables blk;  // uniform couplings: the sector's block tables instead (state not null)
  const MV* diag;   // the diagonal beside them (FP64 product)
};
template <typename MV, typename VV, bool kMf>
using LanArgsOf = std::conditional_t<kMf, LanMfArgs<MV, VV>, LanArgs<MV, VV>>;

__device__ __forceinline__ __int128 lan_shfl(__int128 v, int o) {
  const unsigned long long lo = __shfl_xor_sync(0xffffffffu, (unsigned long long)v, o);
  const long long hi = __shfl_xor_sync(0xffffffffu, (long long)(v >> 64), o);
  return ((__int128)hi << 64) | lo;
}

// One row of H x (FP64), shared by `lanes` threads, four loads in flight.  wait: x is being written in
// this launch, an element is taken once it is there.
template <typename MV, typename VV>
__device__ __forceinline__ VV lan_row(const LanArgs<MV, VV>& A, const VV* x, int64_t r, bool live, int sub, int lanes,
                                      bool wait) {
  VV acc = vzero(VV{});
  if (live) {
    const int64_t e = __ldg(A.rowptr + r + 1);
    for (int64_t k = __ldg(A.rowptr + r) + sub; k < e; k += 4 * lanes) {
      int32_t c[4];
      MV v[4];
      VV xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u * lanes < e) {
          c[u] = __ldg(A.colidx + k + u * lanes);
          v[u] = ld_ro(A.vals + k + u * lanes);
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u * lanes < e) xv[u] = x_peek(x + c[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u * lanes < e) {
          if (wait) x_await(A.X, x + c[u], xv[u]);
          acc = vfma(v[u], xv[u], acc);
        }
    }
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) acc = vadd(acc, shfl_xor(acc, o));
  return acc;
}

// The transitions in shared memory, and which of the two ranks holds.
template <typename MV>
struct LanEnt {
  const MfEntry* ent;          // 64-bit form
  const uint2 *test, *move;    // 32-bit form: (support, output pattern), (flip, sign mask)
  const MV* amp;
};

// The columns of row r from the transitions: take(c, a, on) with up to four at a time, in entry order,
// every lanes-th transition from sub.  kUni: transitions of amplitude zero are no columns.
template <bool kUni, typename MV, typename VV, typename F>
__device__ __forceinline__ void lan_mf_columns(const LanMfArgs<MV, VV>& A, const LanEnt<MV>& E, int64_t r, int sub, int lanes,
                                               F&& take) {
  const uint64_t s = __ldg(A.mf.basis + r);
  const int nent = A.mf.nent;
  const bool narrow = A.mf32.nf > 0;
  for (int e0 = 0; e0 < nent; e0 += 32) {
    unsigned mask = 0;
    if (narrow) {
      for (int q = sub; q < 32 && e0 + q < nent; q += lanes) {
        const uint2 t = E.test[e0 + q];
        mask |= (unsigned)(((uint32_t)s & t.x) == t.y) << q;
      }
    } else {
      for (int q = sub; q < 32 && e0 + q < nent; q += lanes)
        mask |= (unsigned)((s & E.ent[e0 + q].sup) == E.ent[e0 + q].outb) << q;
    }
    while (mask) {
      int32_t c[4];
      MV a[4];
      bool on[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        on[u] = mask != 0;
        if (on[u]) {
          const int e = e0 + __ffs(mask) - 1;
          mask &= mask - 1;
          bool odd;
          if (narrow) {
            const uint2 m = E.move[e];
            const uint32_t t = (uint32_t)s ^ m.x;
            uint32_t col;
            on[u] = mf_rank32(A.mf32, t, col);
            c[u] = (int32_t)col;
            a[u] = E.amp[e];
            odd = __popc(t & m.y) & 1;
          } else {
            const uint64_t t = s ^ E.ent[e].flip;
            const int64_t col = mf_rank(A.mf, t);
            on[u] = col < A.mf.dim;
            c[u] = (int32_t)col;
            a[u] = amp_of((MV*)nullptr, E.ent[e].amp);
            odd = __popcll(t & E.ent[e].jw) & 1;
          }
          if constexpr (kUni) on[u] = on[u] && a[u] != 0.0;
          else if (odd) a[u] = vneg(a[u]);
        }
      }
      take(c, a, on);
    }
  }
}

// The same from the block tables.
template <typename F>
__device__ __forceinline__ void lan_block_columns(const BlockTables& B, int64_t r, int sub, int lanes, F&& take) {
  const uint32_t s = __ldg(B.state + r), lmask = (1u << B.lowbits) - 1u;
  const uint32_t h = s >> B.lowbits, l = s & lmask;
  const int base = __ldg(B.off + h), i = (int)r - base, dl = __ldg(B.ldeg + l), d = dl + __ldg(B.hdeg + h);
  const uint16_t* la = B.ladj + (size_t)l * B.lstride;
  const int32_t* ha = B.hadj + (size_t)h * B.hstride - dl;
  const double none[4] = {};
  for (int j = sub; j < d; j += 4 * lanes) {
    int32_t c[4];
    bool on[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int q = j + u * lanes;
      on[u] = q < d;
      if (on[u]) c[u] = q < dl ? base + (int)__ldg(la + q) : __ldg(ha + q) + i;
    }
    take(c, none, on);
  }
  for (int t = sub; t < B.ncross; t += lanes) {
    if ((s & B.cross[3 * t]) != B.cross[3 * t + 1]) continue;
    const uint32_t c = s ^ B.cross[3 * t + 2];
    const int32_t col[4] = {__ldg(B.off + (c >> B.lowbits)) + (int)__ldg(B.rank_low + (c & lmask)), 0, 0, 0};
    const bool on[4] = {true, false, false, false};
    take(col, none, on);
  }
}

// One row of H x from the transitions; own = x of the row.
template <typename MV, typename VV>
__device__ __forceinline__ VV lan_row_mf(const LanMfArgs<MV, VV>& A, const LanEnt<MV>& ent, const VV* x, int64_t r,
                                         bool live, int sub, int lanes, bool wait, VV own) {
  VV acc = vzero(VV{});
  if (live) {
    if (sub == 0) acc = vfma(ld_ro(A.diag + r), own, acc);
    lan_mf_columns<false>(A, ent, r, sub, lanes, [&](const int32_t (&c)[4], const MV (&a)[4], const bool (&on)[4]) {
      VV xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (on[u]) xv[u] = x_peek(x + c[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (on[u]) {
          if (wait) x_await(A.X, x + c[u], xv[u]);
          acc = vfma(a[u], xv[u], acc);
        }
    });
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) acc = vadd(acc, shfl_xor(acc, o));
  return acc;
}

// The same for uniform couplings: the 128-bit fixed-point copies (fxsum.cuh) that the blocks keep beside
// their rows, summed exactly and rounded once, so that the bits do not depend on where the columns come from
// (the form's list, block tables or the transitions); the diagonal apart.  Every off-diagonal value is one c.  (Converting
// each gathered double instead took twice the FP64 product's time.)
template <bool kMf>
__device__ __forceinline__ double lan_row_uniform(const LanArgsOf<double, double, kMf>& A, const LanEnt<double>& ent,
                                                  const XInt* x, int64_t r, bool live, int sub, int lanes, double own) {
  __int128 acc = 0;
  if (live) {
    if constexpr (kMf) {
      auto add = [&](const int32_t (&c)[4], const double (&)[4], const bool (&on)[4]) {
        XInt xv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (on[u]) xv[u] = x_peek(x + c[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (on[u]) {
            x_await(A.X, x + c[u], xv[u]);
            acc += x_value(xv[u]);
          }
      };
      if (A.blk.state) lan_block_columns(A.blk, r, sub, lanes, add);
      else lan_mf_columns<true>(A, ent, r, sub, lanes, add);
    } else {
      // the form's own list of off-diagonal columns, or the stored rows, explicit zeros skipped (with the list
      // alone the compiler's schedule takes 9.1 us a step at dim 12,870, with both 8.8)
      const bool listed = A.fxptr != nullptr;
      const int32_t* col = listed ? A.fxcol : A.colidx;
      const int64_t e = listed ? (int64_t)__ldg(A.fxptr + r + 1) : __ldg(A.rowptr + r + 1);
      for (int64_t k = (listed ? (int64_t)__ldg(A.fxptr + r) : __ldg(A.rowptr + r)) + sub; k < e; k += 4 * lanes) {
        int32_t c[4];
        XInt xv[4];
        bool on[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          on[u] = k + u * lanes < e;
          if (on[u]) c[u] = __ldg(col + k + u * lanes);
          if (!listed && on[u]) on[u] = c[u] != (int32_t)r && __ldg(A.vals + k + u * lanes) != 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (on[u]) xv[u] = x_peek(x + c[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (on[u]) {
            x_await(A.X, x + c[u], xv[u]);
            acc += x_value(xv[u]);
          }
      }
    }
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) acc += lan_shfl(acc, o);
  const double dx = (live && A.fxdiag) ? __ldg(A.fxdiag + r) * own : 0.0;
  return fma(A.cF, (double)acc, dx);
}

// v on the scale 2^E (|v| < 2^E) in units of 2^(E - 57): a warp's sum fits 64 bits
__device__ __forceinline__ long long lan_fix(double v, int E) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((b >> 52) & 0x7ff);
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | 0x10000000000000ull;
  const int sh = E + 1018 - e;  // >= -4
  long long q = (e == 0 || sh > 53) ? 0ll : (long long)(sh > 0 ? (m + (1ull << (sh - 1))) >> sh : m << -sh);
  return b < 0 ? -q : q;
}

template <int T>
struct LanShared {
  unsigned mx[8][T / 32];
  long long q[8][T / 32];
  double v[8], red[8];
  double sw, c1[2], c2[2];  // the update's scale and coefficients (re, im)
  double s1, s2;            // scales of V[k-1] and V[k-2]
  int stop;
};

// The block's sums of NV values per thread into S.v (complete after the next block barrier).
// Only the first nact warps hold any (the others' slots are zero from the start).
template <int NV, int T>
__device__ __forceinline__ void lan_block_sums(LanShared<T>& S, const double (&v)[NV], int nact) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int nw = T / 32;
  if (warp < nact) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const unsigned m = __reduce_max_sync(0xffffffffu, q_mag(v[i]));
      if (lane == 0) S.mx[i][warp] = m;
    }
  }
  __syncthreads();
  unsigned mag[NV];
  if (warp < nact) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      mag[i] = __reduce_max_sync(0xffffffffu, lane < nw ? S.mx[i][lane] : 0u);
      long long q = lan_fix(v[i], (int)(mag[i] >> 20) - 1022);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (lane == 0) S.q[i][warp] = (q + 8) >> 4;  // units of 2^(E - 53): the block's sum fits as well
    }
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      long long q = lane < nw ? S.q[i][lane] : 0ll;
#pragma unroll
      for (int o = nw / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      if (lane == i) {
        const int e = (int)(mag[i] >> 20), ue = e - 1022 - 53 + 1023;
        S.v[i] = (e == 0x7ff) ? __longlong_as_double(0x7ff8000000000000ll)
                              : (ue > 0 ? (double)q * __hiloint2double(ue << 20, 0) : 0.0);
      }
    }
  }
}

__device__ __forceinline__ double lan_re(double v) { return v; }
__device__ __forceinline__ double lan_re(cplx v) { return v.re; }
__device__ __forceinline__ double lan_im(double) { return 0.0; }
__device__ __forceinline__ double lan_im(cplx v) { return v.im; }
__device__ __forceinline__ void lan_make(double& d, double re, double) { d = re; }
__device__ __forceinline__ void lan_make(cplx& d, double re, double im) { d = mkc(re, im); }
__device__ __forceinline__ double lan_redot(double a, double b, double acc) { return fma(a, b, acc); }
__device__ __forceinline__ double lan_redot(cplx a, cplx b, double acc) {
  return fma(a.im, b.im, fma(a.re, b.re, acc));
}

// y = exp(-i h T) e_0, T = tridiag(al[0 .. act), be[1 .. act)), by one warp: Taylor terms on sub-steps of
// infinity-norm at most 1 (as texp_kernel, krylov.cu, with its terms counted from the remainder bound).  The
// caller bounds ||h T|| (kLanMaxTheta, krylov.cu).
__device__ __forceinline__ void lan_texp(int act, double h, double d, double e, double& yr, double& yi) {
  const int lane = threadIdx.x & 31;
  double em = __shfl_up_sync(0xffffffffu, e, 1);
  if (lane == 0) em = 0.0;
  const double rs = fabs(d) + fabs(e) + fabs(em);
  const unsigned mx = __reduce_max_sync(0xffffffffu, q_mag(rs));
  const double theta = __hiloint2double((int)mx, -1) * fabs(h);
  // one for a NaN and for what a run leaves whose wait has run out (its result is discarded)
  const int steps = (theta <= 2.0 * kLanMaxTheta) ? max(1, (int)ceil(theta)) : 1;
  const double hs = h / steps, th = theta / steps;
  // lane p holds hs / p; terms to th^p / p! <= 1e-18
  const double f = lane > 0 ? hs / lane : 0.0;
  int terms = 1;
  double b = th;
  while (b > 1e-18 && terms < 30) {
    ++terms;
    b *= th / terms;
  }
  yr = (lane == 0) ? 1.0 : 0.0;
  yi = 0.0;
  for (int s = 0; s < steps; ++s) {
    double tr = yr, ti = yi;
    for (int p = 1; p <= terms; ++p) {
      const double fp = __shfl_sync(0xffffffffu, f, p);
      const double rdn = __shfl_down_sync(0xffffffffu, tr, 1), idn = __shfl_down_sync(0xffffffffu, ti, 1);
      const double rup = __shfl_up_sync(0xffffffffu, tr, 1), iup = __shfl_up_sync(0xffffffffu, ti, 1);
      // e and em are 0 beyond the matrix, so the shuffles' ends drop out
      const double kr = fma(d, tr, fma(e, rdn, em * rup)), ki = fma(d, ti, fma(e, idn, em * iup));
      tr = fp * ki;
      ti = -fp * kr;
      yr += tr;
      yi += ti;
    }
  }
}

// The block's rows in order of their length, longest first (lengths from kLanBins - 1 on alike; equal ones in
// their own order), so that a warp issues as many FP64 multiply-adds as its rows have entries and not as the
// longest of 32 neighbours has.  scratch: (R / 32 + 2) kLanBins shorts.
constexpr int kLanBins = 64;
template <int T, typename F>
__device__ void lan_sort_rows(F&& length, int R, short* order, short* scratch) {
  const int tid = threadIdx.x, lane = tid & 31, chunks = (R + 31) / 32;
  short* base = scratch + chunks * kLanBins;
  for (int i = tid; i < chunks * kLanBins; i += T) scratch[i] = 0;
  __syncthreads();
  for (int pass = 0; pass < 2; ++pass) {
    for (int r = tid; r - lane < R; r += T) {
      const unsigned live = __ballot_sync(0xffffffffu, r < R);
      if (r < R) {
        const int len = (int)min(length(r), (int64_t)kLanBins - 1);
        const unsigned same = __match_any_sync(live, len), before = same & ((1u << lane) - 1u);
        short* h = scratch + (r >> 5) * kLanBins + len;
        if (pass == 0) {
          if (!before) *h = (short)__popc(same);
        } else {
          order[base[len] + *h + __popc(before)] = (short)r;
        }
      }
    }
    __syncthreads();
    if (pass == 0) {
      if (tid < kLanBins) {
        int run = 0;
        for (int c = 0; c < chunks; ++c) {
          const int t = scratch[c * kLanBins + tid];
          scratch[c * kLanBins + tid] = (short)run;
          run += t;
        }
        base[kLanBins + tid] = (short)run;
      }
      __syncthreads();
      if (tid < kLanBins) {
        int b = 0;
        for (int i = tid + 1; i < kLanBins; ++i) b += base[kLanBins + i];
        base[tid] = (short)b;
      }
      __syncthreads();
    }
  }
}

// Transitions of a row (its length but for the diagonal's entry and what leaves the sector).
template <typename MV, typename VV>
__device__ __forceinline__ int64_t lan_mf_length(const LanMfArgs<MV, VV>& A, const LanEnt<MV>& E, int64_t r) {
  const uint64_t s = __ldg(A.mf.basis + r);
  int n = 0;
  if (A.mf32.nf > 0)
    for (int e = 0; e < A.mf.nent; ++e) n += ((uint32_t)s & E.test[e].x) == E.test[e].y;
  else
    for (int e = 0; e < A.mf.nent; ++e) n += (s & E.ent[e].sup) == E.ent[e].outb;
  return n;
}

template <typename MV, typename VV, bool kOne, bool kUni, bool kPaige, bool kExp, bool kMf>
__global__ void __launch_bounds__(kLanThreads, 1) lan_kernel(LanArgsOf<MV, VV, kMf> A) {
  constexpr int T = kLanThreads, kPer = sizeof(VV) / sizeof(double);
  constexpr int NV = kPaige ? 2 : 1 + 3 * kPer;
  extern __shared__ __align__(16) unsigned char lan_smem[];
  __shared__ LanShared<T> S;
  __shared__ double talpha[kExp ? kLanMaxExp + 1 : 1], tnrm[kExp ? kLanMaxExp + 1 : 1], tscl[kExp ? kLanMaxExp + 1 : 1];
  __shared__ cplx y[kExp ? kLanMaxExp : 1];
  const int tid = threadIdx.x;
  const int64_t r0 = A.row_first[blockIdx.x];
  const int R = A.row_first[blockIdx.x + 1] - (int)r0;
  VV* ring = reinterpret_cast<VV*>(lan_smem);  // V[k] of the block's rows at ring + (k % 3) rows
  VV* Vg = A.V + r0;
  const GridX& X = A.X;
  if (kUni && A.first > 1 && *A.stop != 0) return;  // an earlier launch of the run broke down
  const bool mute = X.hold && blockIdx.x == 0;
  int lanes = 1;
  while (lanes < 4 && 2 * lanes * A.rows <= (kUni ? 512 : 256)) lanes *= 2;
  short* order = reinterpret_cast<short*>(ring + 3 * (size_t)A.rows);
  LanEnt<MV> ent{};
  if constexpr (kMf) {
    unsigned char* p = lan_smem + lan_rows_smem<VV>(A.rows);
    const int nent = A.mf.nent;
    if (A.mf32.nf > 0) {
      uint2 *test = reinterpret_cast<uint2*>(p), *move = test + nent;
      MV* amp = reinterpret_cast<MV*>(move + nent);
      for (int i = tid; i < nent; i += T) {
        const MfEntry E = A.mf.ent[i];
        test[i] = make_uint2((uint32_t)E.sup, (uint32_t)E.outb);
        move[i] = make_uint2((uint32_t)E.flip, (uint32_t)E.jw);
        amp[i] = amp_of((MV*)nullptr, E.amp);
      }
      ent.test = test;
      ent.move = move;
      ent.amp = amp;
    } else {
      MfEntry* e = reinterpret_cast<MfEntry*>(p);
      for (int i = tid; i < nent; i += T) e[i] = A.mf.ent[i];
      ent.ent = e;
    }
    __syncthreads();
  }
  if constexpr (!kUni)
    if (lanes == 1)
      lan_sort_rows<T>(
          [&](int r) -> int64_t {
            if constexpr (kMf) return lan_mf_length(A, ent, r0 + r);
            else return __ldg(A.rowptr + r0 + r + 1) - __ldg(A.rowptr + r0 + r);
          },
          R, order, reinterpret_cast<short*>(ring));
  double vals[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) vals[i] = 0.0;
  const int nact = max(1, min(T / 32, (R * lanes + 31) / 32));  // warps with rows
  for (int i = tid; i < 8 * (T / 32); i += T) {
    S.mx[i / (T / 32)][i % (T / 32)] = 0;
    S.q[i / (T / 32)][i % (T / 32)] = 0;
  }
  if (kExp && tid == 0) S.s1 = S.s2 = 0.0;
  // the rows of the vectors the first step reads; kExp: V[0] = psi, its norm still to come
  if (kExp) {
    for (int r = tid; r < R; r += T) {
      VV v;
      lan_make(v, A.psi[r0 + r].re, A.psi[r0 + r].im);
      ring[r] = v;
      Vg[r] = v;
      vals[NV - 1] = lan_redot(v, v, vals[NV - 1]);
    }
  } else {
    for (int b = 1; b <= 2; ++b) {
      const int j = A.first - b;
      if (j >= 0)
        for (int r = tid; r < R; r += T) ring[(size_t)(j % 3) * A.rows + r] = Vg[(int64_t)j * A.ld + r];
    }
    if (!kPaige && A.first > 1) {  // <V1, V2>
      __syncthreads();
      VV d3 = vzero(VV{});
      const VV *u1 = ring + (size_t)((A.first - 1) % 3) * A.rows, *u2 = ring + (size_t)((A.first - 2) % 3) * A.rows;
      for (int r = tid; r < R; r += T) d3 = vdotfma(u1[r], u2[r], d3);
      vals[2 * kPer] = lan_re(d3);
      if (kPer == 2) vals[2 * kPer + 1] = lan_im(d3);
    }
    if (tid == 0) {
      S.s1 = A.scl[A.first - 1];
      S.s2 = A.first > 1 ? A.scl[A.first - 2] : 0.0;
    }
  }
  __syncthreads();
  int ov = 0, stop = 0;
  if constexpr (kUni)
    for (int r = tid; r < R; r += T)
      if (!mute) x_put(A.XV + r0 + r, fx_from_double(ring[(size_t)((A.first - 1) % 3) * A.rows + r], A.F, &ov));
  for (int k = A.first; k <= A.last; ++k) {
    const VV* u1 = ring + (size_t)((k - 1) % 3) * A.rows;
    const VV* u2 = ring + (size_t)((k + 1) % 3) * A.rows;  // V[k-2]
    VV* w = ring + (size_t)(k % 3) * A.rows;
    const bool has2 = k >= 2, known = !kExp && k == A.first;  // known: V[k-1]'s scale is from before
    const VV* x = A.V + (int64_t)(k - 1) * A.ld;
    if constexpr (kExp && sizeof(VV) == sizeof(cplx))
      if (k == 1) x = reinterpret_cast<const VV*>(A.psi);
    // w = H V1 (not scaled) and its inner products
    {
      VV d1 = vzero(VV{}), d2 = vzero(VV{});
      double d2re = 0.0;
      const int g = tid / lanes, sub = tid & (lanes - 1), per = T / lanes;
      for (int i = g; (i & ~(32 / lanes - 1)) < R; i += per) {  // whole warps
        const bool live = i < R;
        const int r = (!kUni && lanes == 1 && live) ? order[i] : i;
        VV a;
        if constexpr (kUni)
          a = lan_row_uniform<kMf>(A, ent, A.XV + (int64_t)(k - A.first) * A.ld, r0 + r, live, sub, lanes,
                                   live ? u1[r] : 0.0);
        else if constexpr (kMf)
          a = lan_row_mf(A, ent, x, r0 + r, live, sub, lanes, k > A.first, live ? u1[r] : vzero(VV{}));
        else a = lan_row(A, x, r0 + r, live, sub, lanes, k > A.first);
        if (live && sub == 0) {
          w[r] = a;
          if (kPaige) {
            d2re = lan_redot(u1[r], a, d2re);
          } else {
            d2 = vdotfma(u1[r], a, d2);
            if (has2) d1 = vdotfma(u2[r], a, d1);
          }
        }
      }
      if (kPaige) {
        vals[0] = d2re;
      } else {
        vals[0] = lan_re(d1);
        vals[kPer] = lan_re(d2);
        if (kPer == 2) {
          vals[1] = lan_im(d1);
          vals[kPer + 1] = lan_im(d2);
        }
      }
    }
    lan_block_sums<NV, T>(S, vals, nact);
    __syncthreads();
    x_sum<kOne>(X, A.slots + (size_t)(k - A.first) * A.xstride, S.v, NV, S.red);
    // the scale of V1 from its norm, alpha and beta, and the update's coefficients: one chain of scalar
    // FP64 operations (64 cycles each), what the update does not wait for on a second warp
    if (tid == 0) {
      const double s1 = known ? S.s1 : rsqrt(S.red[NV - 1]), s2 = S.s2;
      double ar, ai = 0.0, br = 0.0, bi = 0.0;
      if (kPaige) {
        ar = (s1 * s1) * S.red[0];
        br = !has2 ? 0.0 : (known ? 1.0 / s1 : S.red[NV - 1] * s1);  // ||V1||
      } else {
        const double* d = S.red;
        const double s12 = s1 * s2;
        br = has2 ? s12 * d[0] : 0.0;
        ar = s1 * d[kPer];
        if (kPer == 2) {
          bi = has2 ? s12 * d[1] : 0.0;
          ai = s1 * d[kPer + 1];
        }
        if (has2) {  // - (beta s2) <V1, V2>
          const double pr = br * s2, pi = bi * s2, qr = d[2 * kPer], qi = kPer == 2 ? d[2 * kPer + 1] : 0.0;
          ar = fma(-pr, qr, ar);
          if (kPer == 2) {
            ar = fma(pi, qi, ar);
            ai = fma(-pr, qi, fma(-pi, qr, ai));
          }
        }
        ar *= s1;
        ai *= s1;
      }
      S.sw = s1;
      S.c1[0] = ar * s1;
      S.c1[1] = ai * s1;
      S.c2[0] = br * s2;
      S.c2[1] = bi * s2;
      if (kExp) {
        talpha[k] = ar;
      } else if (blockIdx.x == 0) {
        VV v;
        lan_make(v, ar, ai);
        A.alpha[k] = v;
        lan_make(v, br, bi);
        if (A.beta) A.beta[k] = v;
      }
    } else if (tid == T - 32) {
      S.stop = 0;
      if (!known) {
        const double n2 = S.red[NV - 1], s1 = rsqrt(n2), nr = n2 > 0.0 ? n2 * s1 : n2;
        S.stop = (k > 1 || !kExp) && nr < A.stop_below;
        if (kExp) {
          tnrm[k - 1] = nr;
          tscl[k - 1] = s1;
        } else if (blockIdx.x == 0) {
          A.nrm[k - 1] = nr;
          A.scl[k - 1] = s1;
        }
      }
    }
    __syncthreads();
    if (S.stop) {
      stop = k - 1;
      break;
    }
    // V[k] = (s1 w - (beta s2) V2) - (alpha s1) V1, its norm and its overlap with V1
    {
      const double sw = S.sw;
      if (tid == 0) S.s2 = S.s1 = sw;
      VV a, b, d3 = vzero(VV{});
      lan_make(a, S.c1[0], S.c1[1]);
      lan_make(b, S.c2[0], S.c2[1]);
      double n2 = 0.0;
      VV* vk = Vg + (int64_t)k * A.ld;
      for (int r = tid; r < R; r += T) {
        VV o = vscale(sw, w[r]);
        if constexpr (kPaige) {  // real coefficients
          if (has2) o = vfma(-S.c2[0], u2[r], o);
          o = vfma(-S.c1[0], u1[r], o);
        } else {
          if (has2) o = vsubmul(o, b, u2[r]);
          o = vsubmul(o, a, u1[r]);
        }
        w[r] = o;
        if constexpr (kUni) {
          vk[r] = o;
          if (!mute) x_put(A.XV + (int64_t)(k - A.first + 1) * A.ld + r0 + r, fx_from_double(o, A.F, &ov));
        } else {
          if (!mute) x_put(vk + r, o);
        }
        n2 = lan_redot(o, o, n2);
        if (!kPaige) d3 = vdotfma(o, u1[r], d3);
      }
      vals[NV - 1] = n2;
      if (!kPaige) {
        vals[2 * kPer] = lan_re(d3);
        if (kPer == 2) vals[2 * kPer + 1] = lan_im(d3);
      }
    }
    __syncthreads();
  }
  if (kUni && ov) *A.ovf = 1;
  if (!kExp || !stop) {
    if (!stop) {  // the last vector's norm
      lan_block_sums<NV, T>(S, vals, nact);
      __syncthreads();
      x_sum<kOne>(X, A.slots + (size_t)(A.last + 1 - A.first) * A.xstride, S.v, NV, S.red);
      if (tid == 0) {
        const double n2 = S.red[NV - 1], nr = n2 > 0.0 ? n2 * rsqrt(n2) : n2;
        S.stop = nr < A.stop_below;
        if (!kExp && blockIdx.x == 0) {
          A.nrm[A.last] = nr;
          A.scl[A.last] = rsqrt(n2);
        }
      }
      __syncthreads();
      if (S.stop) stop = A.last;
    }
    if (!kExp) {
      if (blockIdx.x == 0 && tid == 0 && stop) *A.stop = stop;
      return;
    }
  }
  if constexpr (kExp) {
    // expandBasis<0>'s count: the breaking step is kept
    const int act = stop ? stop : A.last;
    if (tid < 32) {
      const double d = tid < act ? talpha[tid + 1] : 0.0, e = tid + 1 < act ? tnrm[tid + 1] : 0.0;
      double yr, yi;
      lan_texp(act, A.h, d, e, yr, yi);
      if (tid < act) y[tid] = mkc(yr * tscl[tid], yi * tscl[tid]);
    }
    __syncthreads();
    if (blockIdx.x == 0 && tid == 0) {
      *A.act = act;
      *A.matvecs += act;
    }
    if constexpr (sizeof(VV) == sizeof(cplx)) {
      cplx* out = A.out + r0;
      for (int r = tid; r < R; r += T) {
        const cplx* v = reinterpret_cast<const cplx*>(Vg) + r;
        cplx a = mkc(0.0, 0.0);
        int j = 0;
        for (; j + 4 <= act; j += 4, v += 4 * A.ld) {
          const cplx v0 = v[0], v1 = v[A.ld], v2 = v[2 * A.ld], v3 = v[3 * A.ld];
          a = vfma(y[j], v0, a);
          a = vfma(y[j + 1], v1, a);
          a = vfma(y[j + 2], v2, a);
          a = vfma(y[j + 3], v3, a);
        }
        for (; j < act; ++j, v += A.ld) a = vfma(y[j], v[0], a);
        out[r] = a;
      }
    }
  }
}

// ---------------------------------------------------------------- host
// First rows of `grid` blocks of nearly equal work: a row costs about what six entries do (its share of
// the inner products, the update and the norm).  Equal row counts left the blocks of a spin chain, whose
// rows' lengths follow their states, waiting for the longest: 24,000 of 65,000 cycles a step at L = 20.
__global__ void lan_rows_kernel(int64_t n, const int64_t* rowptr, int grid, int* first) {
  const double total = (double)rowptr[n] + 6.0 * (double)n;
  for (int b = threadIdx.x; b <= grid; b += blockDim.x) {
    const double want = total * b / grid;
    int64_t lo = 0, hi = n;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if ((double)rowptr[mid] + 6.0 * (double)mid < want) lo = mid + 1;
      else hi = mid;
    }
    first[b] = b == grid ? (int)n : (int)lo;
  }
}

// The rows' lengths as the stored matrix has them (an entry of the diagonal where one of its nd transitions
// dia applies), so that solves on either split the rows alike.
__global__ void lan_mf_lengths_kernel(const __grid_constant__ MfRows M, const MfEntry* dia, int nd, int64_t* len) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= M.dim; r += (int64_t)gridDim.x * blockDim.x) {
    int64_t n = 0;
    if (r < M.dim) {
      const uint64_t s = __ldg(M.basis + r);
      for (int e = 0; e < M.nent; ++e)
        if ((s & M.ent[e].sup) == M.ent[e].outb) n += mf_rank(M, s ^ M.ent[e].flip) < M.dim;
      bool diag = false;
      for (int e = 0; e < nd; ++e) diag |= (s & dia[e].sup) == dia[e].outb;
      n += diag;
    }
    len[r] = n;
  }
}

// The kernel for one block or many; cfg for the grid the sector takes.  False when the device does not hold
// the grid at once, or a block its rows.
template <typename VV, typename K>
static bool lan_plan(qd_ham* H, bool mf, K kern1, K kern_many, LanPlan& P, cudaLaunchConfig_t& cfg,
                     cudaLaunchAttribute (&at)[2], K& kern) {
  Ctx* ctx = H->ctx;
  const int64_t n = H->dim;
  const int csize = n <= kLanOneBlock ? 1 : (n <= lan_wide_rows<VV>() ? 8 : 4);  // one block: an exchange would cost more than it saves
  kern = csize == 1 ? kern1 : kern_many;
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)csize;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kLanThreads);
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = csize == 1 ? 1 : 2;
  const auto smem_of = [&](int rows) { return lan_rows_smem<VV>(rows) + (mf ? H->mf_nent * sizeof(MfEntry) : 0); };
  if (P.none) return false;
  if (!P.ok) {
    int maxsm = 0;
    QD_CUDA(cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
    int ncl = csize == 1 ? 1 : (int)std::min<int64_t>(ctx->num_sms / csize, ceil_div(n, csize * kLanMinRows));
    int rows = (int)n;
    std::vector<int> first;
    const int64_t* rowptr = H->rowptr.p;
    DBuf<int64_t> len;
    if (mf) {  // the lengths that the transitions give, summed
      std::vector<MfEntry> off, dia;
      compile_terms(H, off, dia);
      DBuf<MfEntry> ddia(dia.size());
      if (!dia.empty())
        QD_CUDA(cudaMemcpyAsync(ddia.p, dia.data(), dia.size() * sizeof(MfEntry), cudaMemcpyHostToDevice, ctx->stream));
      len.alloc(n + 1);
      lan_mf_lengths_kernel<<<(unsigned)ceil_div(n + 1, 256), 256, 0, ctx->stream>>>(mf_rows(H), ddia.p, (int)dia.size(),
                                                                                    len.p);
      QD_CHECK_LAUNCH();
      QD_LAUNCHED(ctx);
      exclusive_scan_i64(ctx, len.p, len.p, n + 1);
      rowptr = len.p;
    }
    for (;;) {
      const int grid = ncl * csize;
      if (P.first.n < (size_t)grid + 1) P.first.alloc(grid + 1);
      lan_rows_kernel<<<1, 256, 0, ctx->stream>>>(n, rowptr, grid, P.first.p);
      QD_CHECK_LAUNCH();
      QD_LAUNCHED(ctx);
      if (csize > 1) {
        first.resize(grid + 1);
        QD_CUDA(cudaMemcpyAsync(first.data(), P.first.p, (grid + 1) * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
        QD_CUDA(cudaStreamSynchronize(ctx->stream));
        rows = 1;
        for (int b = 0; b < grid; ++b) rows = std::max(rows, first[b + 1] - first[b]);
      }
      P.none = smem_of(rows) + 8192 > (size_t)maxsm;
      if (P.none) return false;
      if (csize == 1) break;
      allow_dynamic_smem(kern, ctx->device);
      cfg.gridDim = dim3((unsigned)grid);
      cfg.dynamicSmemBytes = smem_of(rows);
      cudaLaunchConfig_t q = cfg;
      q.attrs = at + 1;
      q.numAttrs = 1;
      int fit = 0;
      QD_CUDA(cudaOccupancyMaxActiveClusters(&fit, kern, &q));
      if (fit >= ncl) break;
      P.none = fit < 1;
      if (P.none) return false;
      ncl = fit;
    }
    P.ok = true;
    P.csize = csize;
    P.ncl = ncl;
    P.rows = rows;
  }
  cfg.gridDim = dim3((unsigned)(P.ncl * csize));
  cfg.dynamicSmemBytes = smem_of(P.rows);
  allow_dynamic_smem(kern, ctx->device);
  return true;
}

template <typename MV, typename VV>
static LanArgs<MV, VV> lan_args(qd_ham* H, const MV* vals, bool mf, const LanPlan& P, VV* V, int64_t ld, int first, int last,
                                int nv, int* flags, DBuf<double>* slots, XInt* xv) {
  Ctx* ctx = H->ctx;
  LanArgs<MV, VV> A;
  std::memset(&A, 0, sizeof(A));
  A.n = H->dim;
  A.ld = ld;
  A.rows = P.rows;
  A.row_first = P.first.p;
  if (!mf) {
    A.rowptr = H->rowptr.p;
    A.colidx = H->colidx.p;
    A.vals = vals;
  }
  A.V = V;
  A.first = first;
  A.last = last;
  A.xstride = P.ncl * P.csize * nv;
  const size_t want = (size_t)(last + 2 - first) * A.xstride;
  if (slots->n < want) slots->alloc(want);
  A.slots = slots->p;
  A.X.abort = flags + 1;
  const unsigned wait_out = step_wait_out_polls();
  A.X.polls = wait_out ? wait_out : kXPolls;
  A.X.hold = wait_out != 0;
  // everything this launch writes for the other blocks starts empty
  QD_CUDA(cudaMemsetAsync(A.slots, kXEmptyByte, want * sizeof(double), ctx->stream));
  if (xv)
    QD_CUDA(cudaMemsetAsync(xv, kXEmptyByte, (size_t)(last + 2 - first) * ld * sizeof(XInt), ctx->stream));
  else
    QD_CUDA(cudaMemsetAsync(V + (int64_t)first * ld, kXEmptyByte, (size_t)(last + 1 - first) * ld * sizeof(VV), ctx->stream));
  A.XV = xv;
  return A;
}

// Steps first .. last of r in one launch.
template <typename MV, typename VV, bool kUni, bool kPaige, bool kMf, typename K>
static void lan_launch_steps(qd_ham* H, const LanRun<MV, VV>& r, const LanPlan& P, const cudaLaunchConfig_t& cfg, K kern,
                             XInt* xv, int first, int last) {
  Ctx* ctx = H->ctx;
  constexpr int kPer = sizeof(VV) / sizeof(double);
  LanArgs<MV, VV> A =
      lan_args(H, r.vals, kMf, P, r.V, r.ld, first, last, kPaige ? 2 : 1 + 3 * kPer, r.flags, r.slots, xv);
  if (kUni) {
    A.fxdiag = r.form->diag_zero ? nullptr : r.form->diag.p;
    A.cF = std::ldexp(r.form->c, -r.form->F);
    if (!kMf) {
      A.fxptr = r.form->rowptr.p;
      A.fxcol = r.form->colidx.p;
    }
    A.F = r.form->F;
    A.ovf = r.flags;
  }
  A.stop_below = r.stop_below;
  A.alpha = r.alpha;
  A.beta = r.beta;
  A.nrm = r.nrm;
  A.scl = r.scl;
  A.stop = r.stop;
  if constexpr (kMf) {
    LanMfArgs<MV, VV> M;
    std::memset(&M, 0, sizeof(M));
    static_cast<LanArgs<MV, VV>&>(M) = A;
    M.mf = mf_rows(H);
    if (!mf32_prepare(H, M.mf32)) M.mf32.nf = 0;
    if constexpr (std::is_same<MV, double>::value) M.diag = H->diag_r.p;
    else M.diag = H->diag_c.p;
    if (kUni && r.form->use_blk && r.form->blk_state > 0) M.blk = block_tables(*r.form);
    QD_CUDA(cudaLaunchKernelEx(&cfg, kern, M));
  } else {
    QD_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
  }
  QD_LAUNCHED(ctx);
}

template <typename MV, typename VV, bool kUni, bool kPaige, bool kMf>
static bool lan_launch(qd_ham* H, const LanRun<MV, VV>& r) {
  constexpr int kC = sizeof(VV) == sizeof(cplx);
  LanPlan& P = ham_workspace(H).lan_plan[kMf ? 5 + kC : 2 * kC + kPaige];
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  auto kern = lan_kernel<MV, VV, true, kUni, kPaige, false, kMf>;
  if (!lan_plan<VV>(H, kMf, kern, lan_kernel<MV, VV, false, kUni, kPaige, false, kMf>, P, cfg, at, kern)) return false;
  // as many steps a launch as the copies' memory holds; a later launch makes the first copy again, and its
  // bits are those of one launch
  int most = r.last + 1 - r.first;
  DBuf<XInt> xv;
  if (kUni) {
    most = (int)std::min<int64_t>(most, std::max<int64_t>(kLanCopyBytes / (r.ld * (int64_t)sizeof(XInt)) - 1, 1));
    try {
      xv.alloc((size_t)(most + 1) * r.ld);
    } catch (const Error&) {  // the steps launched one by one need two copies
      clear_error();
      return false;
    }
  }
  for (int first = r.first; first <= r.last; first += most)
    lan_launch_steps<MV, VV, kUni, kPaige, kMf>(H, r, P, cfg, kern, xv.p, first, std::min(r.last, first + most - 1));
  return true;
}

template <typename MV, typename VV>
bool lan_res_run(qd_ham* H, const LanRun<MV, VV>& r) {
  if constexpr (std::is_same<VV, double>::value)
    if (r.form) return r.mf ? lan_launch<MV, VV, true, false, true>(H, r) : lan_launch<MV, VV, true, false, false>(H, r);
  if (r.rule == kLanPaige) return lan_launch<MV, VV, false, true, false>(H, r);
  return r.mf ? lan_launch<MV, VV, false, false, true>(H, r) : lan_launch<MV, VV, false, false, false>(H, r);
}
template bool lan_res_run<double, double>(qd_ham*, const LanRun<double, double>&);
template bool lan_res_run<double, cplx>(qd_ham*, const LanRun<double, cplx>&);
template bool lan_res_run<cplx, cplx>(qd_ham*, const LanRun<cplx, cplx>&);

template <typename MV>
bool lan_res_evolve(qd_ham* H, const MV* vals, const cplx* psi, cplx* out, cplx* V, int64_t ld, int kdim, double h,
                    int* act, long long* matvecs, int* flags, DBuf<double>* slots) {
  Ctx* ctx = H->ctx;
  LanPlan& P = ham_workspace(H).lan_plan[4];
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  auto kern = lan_kernel<MV, cplx, true, false, true, true, false>;
  if (kdim > kLanMaxExp ||
      !lan_plan<cplx>(H, false, kern, lan_kernel<MV, cplx, false, false, true, true, false>, P, cfg, at, kern))
    return false;
  LanArgs<MV, cplx> A = lan_args<MV, cplx>(H, vals, false, P, V, ld, 1, kdim, 2, flags, slots, nullptr);
  A.stop_below = 1e-10;
  A.psi = psi;
  A.out = out;
  A.h = h;
  A.act = act;
  A.matvecs = matvecs;
  QD_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
  QD_LAUNCHED(ctx);
  return true;
}
template bool lan_res_evolve<double>(qd_ham*, const double*, const cplx*, cplx*, cplx*, int64_t, int, double, int*, long long*, int*, DBuf<double>*);
template bool lan_res_evolve<cplx>(qd_ham*, const cplx*, const cplx*, cplx*, cplx*, int64_t, int, double, int*, long long*, int*, DBuf<double>*);

}  // namespace qd
