// arnres.cu -- the Arnoldi recurrence of evolve and getGroundState (herm = 0)
// as one persistent launch.
//
// expandBasis<0> (sparse_algorithm.hpp:372-393) per step: w = H v_{idx-1},
// orthogonalised against v_0 .. v_{idx-1} by classical Gram-Schmidt applied
// twice, its norm.  As separate kernels a step is seven launches whose work at a
// few thousand rows is a microsecond each: at dim 4,900 and m = 30 a step of
// the recurrence took 115 us, 99 of them in the projections, which ran on three
// blocks.  Here every block of one co-resident grid owns a slice of the rows
// for the whole recurrence and the blocks exchange two small sums a step
// (gridx.cuh) and the rows of the newest vector, which the product gathers as
// they arrive:
//   1. w = H V[k-1]; its projections and ||V[k-1]||^2, which scales them;
//   2. w -= V c, projections of what is left;   3. V[k] = w - V c'.
// For a Hermitian H the exact projections of pass 1 vanish but for the last
// two vectors, so pass 1 projects on those alone and pass 2 removes what
// rounding left on all of them: the same two-fold orthogonality for half the
// work.  The basis is stored unnormalised with its scales.
//
// The projections and norms run in integer arithmetic on 55-bit copies of the
// block's rows in shared memory (qvec.cuh): a sum rounds relative to its largest
// terms in FP64 as well.  The product, the removal of the projections (on the
// vectors themselves, from L1 and L2) and the combination are FP64, so that what
// is stored keeps the relative accuracy of each row; with the removal on the
// copies, amplitudes of a localised state some 1e-14 below its largest were lost.
// Over 41 evolutions, 137 damped or unitary quench states and 16 ground states of
// random sizes the mean error against 64-bit references is 3.9e-16, 6.7e-16 and
// 6.0e-16 (passes over a basis in memory: 4.3e-16, 7.6e-16 and 6.3e-16).
//
// The exponential of the small Hessenberg matrix (act <= 32) is a Taylor series
// of exp(-i h K) e_0 on sub-steps of norm <= 1, formed redundantly by every
// block, and the combination uses the block's own rows: evolve is one launch.
//
// Measured (GB300, SM clock 1.9 GHz): dim 4,900, m = 30, not Hermitian: 3.3 ms
// -> 0.60 ms a step; dim 36, m = 20: 0.56 -> 0.18 ms; ground state of the 4 x 4
// cluster (dim 12,870, 40 columns, real vectors): 6.5 -> 1.1 ms.  A column at dim
// 4,900 is 38,000 cycles: the two exchanges 14,600, the projections and their
// removal 17,000 (14,000 with the removal in integers), the product 2,800, the
// rest scalar FP64 operations between block barriers (16,000 cycles a column in
// all on one block of 36 rows).
// Operators whose rows do not fit (about 60,000 rows at m = 30) take passes over
// a basis in memory (gspass.cu), as served requests do.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "arnres.cuh"
#include "dense.h"
#include "evolve.cuh"
#include "gridx.cuh"
#include "krylov.cuh"
#include "qvec.cuh"

namespace qd {

constexpr int kArnThreads = 512;
constexpr int kArnCluster = 8;  // blocks per cluster
constexpr int kArnLdh = kArnMaxVecs + 1;
constexpr int kArnHs = kArnMaxExp + 1;
constexpr int kArnMaxSubsteps = 64;
constexpr double kArnTerms = 1e-24;  // the last Taylor term's bound: small components keep their own accuracy
constexpr int kArnMinRows = 64;     // rows of a block before the grid covers every SM
constexpr int kArnMaxResRows = 3800;  // rows of a resident block: its sums stay within 128 terms a thread

// 1 / p
__constant__ double kArnInv[32] = {0.0,      1.0,      1.0 / 2,  1.0 / 3,  1.0 / 4,  1.0 / 5,  1.0 / 6,  1.0 / 7,
                                   1.0 / 8,  1.0 / 9,  1.0 / 10, 1.0 / 11, 1.0 / 12, 1.0 / 13, 1.0 / 14, 1.0 / 15,
                                   1.0 / 16, 1.0 / 17, 1.0 / 18, 1.0 / 19, 1.0 / 20, 1.0 / 21, 1.0 / 22, 1.0 / 23,
                                   1.0 / 24, 1.0 / 25, 1.0 / 26, 1.0 / 27, 1.0 / 28, 1.0 / 29, 1.0 / 30, 1.0 / 31};

template <typename MV, typename VV>
struct ArnArgs {
  int64_t n, ld;
  int rows;  // rows per block
  int ldr;   // shared-memory stride of a basis vector (odd)
  const int64_t* rowptr;
  const int32_t* colidx;
  const MV* vals;
  const cplx* psi_in;
  VV* V;
  cplx* hcol;
  ArnStatus* st;
  int kdim, first, last, herm;
  // evolve only
  cplx* psi_out;
  double h;
  double* slots;   // two exchanges a step and a last one, xstride slots each
  size_t xstride;
  GridX X;
};

__device__ __forceinline__ void arn_from(cplx& d, cplx v) { d = v; }
__device__ __forceinline__ void arn_from(double& d, cplx v) { d = v.re; }
__device__ __forceinline__ cplx arn_c(double v) { return mkc(v, 0.0); }
__device__ __forceinline__ cplx arn_c(cplx v) { return v; }
__device__ __forceinline__ double arn_re(double v) { return v; }
__device__ __forceinline__ double arn_re(cplx v) { return v.re; }

// One row of H x, `lanes` threads (a power of two, one of them this one) sharing it; four loads in
// flight; the sum in every one of them.  x is written by all blocks in this launch: an element is taken
// once it is there.
template <typename MV, typename VV>
__device__ __forceinline__ VV arn_row(const ArnArgs<MV, VV>& A, const VV* x, int64_t r, bool live, int sub, int lanes) {
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
          x_await(A.X, x + c[u], xv[u]);
          acc = vfma(v[u], xv[u], acc);
        }
    }
  }
  for (int o = lanes >> 1; o > 0; o >>= 1) acc = vadd(acc, shfl_xor(acc, o));
  return acc;
}

template <typename VV, int T>
struct ArnShared {
  QSum part[2 * T];             // partial projections (re, im), or partial updates
  double xv[2 * kArnMaxVecs + 2];   // this block's sums
  double red[2 * kArnMaxVecs + 2];  // the grid's
  VV c1[kArnMaxVecs];           // projections of the first pass
  VV cf[kArnMaxVecs];           // coefficients on the stored vectors
  double scl[kArnMaxVecs + 2];
  double u[kArnMaxVecs + 2];    // scales of the block's quantised vectors
  double us[kArnMaxVecs + 2];   // u[j] scl[j]
  double nrm2;
  unsigned mx[32];
  int stop;
};

// The largest magnitude word over the block (every thread gets it).
template <typename VV, int T>
__device__ __forceinline__ unsigned arn_block_max(ArnShared<VV, T>& S, unsigned m) {
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) S.mx[threadIdx.x >> 5] = m;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  m = __reduce_max_sync(0xffffffffu, lane < T / 32 ? S.mx[lane] : 0u);
  __syncthreads();
  return m;
}

// The block's share of the projections <v_{j0+j}, w>, j < J, into S.xv: resident vectors.
// Thread (j, c) takes rows c, c + C, ... (a warp's lanes hold different vectors).
template <typename VV, int T>
__device__ void arn_dots_res(ArnShared<VV, T>& S, const typename QVec<VV>::T* Vs, int ldr, int j0, int J,
                             const typename QVec<VV>::T* w, double uw, int R) {
  const int tid = threadIdx.x;
  const int C = max(1, min(min(T / J, 32), R));
  if (tid < J * C) {
    const int c = tid / J, j = tid - c * J;
    const typename QVec<VV>::T* v = Vs + (size_t)(j0 + j) * ldr;
    QDot<VV> a;
    for (int r = c; r < R; r += C) a.add(v[r], w[r]);
    S.part[2 * tid].set(a.re());
    S.part[2 * tid + 1].set(a.im());
  }
  __syncthreads();
  // four lanes a value: every fourth chunk each
  constexpr int kPer = sizeof(VV) / sizeof(double);
  const int nv = kPer * J;
  for (int b = 0; b < nv; b += T / 4) {
    const int v4 = b + (tid >> 2);
    if (b + ((tid & ~31) >> 2) < nv) {  // whole warps
      const int j = min(v4, nv - 1) / kPer, q = min(v4, nv - 1) - kPer * j;
      QSum t{0, 0u};
      for (int c = tid & 3; c < C; c += 4) {
        const QSum x = S.part[2 * (c * J + j) + q];
        t.add(x.hi, x.lo);
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1)
        t.add(__shfl_xor_sync(0xffffffffu, t.hi, o), __shfl_xor_sync(0xffffffffu, t.lo, o));
      if ((tid & 3) == 0 && v4 < nv) S.xv[v4] = (uw * S.us[j0 + j]) * t.value();
    }
  }
  __syncthreads();
}

// put(r, sum_j cf[j] V_j[r]) on the block's rows, J vectors of stride ld from V, in FP64 from the vectors in memory
// (L1 and L2); thread (r, c) takes every JC-th vector when the rows alone leave threads idle (an evolution of m =
// 30 at dim 4,900: 647 us with one thread a row, 601 with two to four, 613 with eight).
template <typename VV, int T, typename F>
__device__ void arn_comb(ArnShared<VV, T>& S, const VV* V, int64_t ld, int J, int R, F&& put) {
  const int tid = threadIdx.x;
  const int JC = R > 0 ? max(1, min(min(T / R, J), 4)) : 1;
  auto row = [&](int r, int c) {
    const VV* v = V + r + (int64_t)c * ld;
    const int64_t hop = (int64_t)JC * ld;
    VV a = vzero(VV{});
    int j = c;
    for (; j + 3 * JC < J; j += 4 * JC, v += 4 * hop) {
      const VV v0 = v[0], v1 = v[hop], v2 = v[2 * hop], v3 = v[3 * hop];
      a = vfma(S.cf[j], v0, a);
      a = vfma(S.cf[j + JC], v1, a);
      a = vfma(S.cf[j + 2 * JC], v2, a);
      a = vfma(S.cf[j + 3 * JC], v3, a);
    }
    // the last three at most: their loads in flight together, as many multiply-adds as the warp has (predicated
    // ones issue as well)
    if (j < J) {
      const VV v0 = v[0];
      VV v1 = v0, v2 = v0;
      if (j + JC < J) v1 = v[hop];
      if (j + 2 * JC < J) v2 = v[2 * hop];
      a = vfma(S.cf[j], v0, a);
#pragma unroll 1
      for (int u = 1; j + u * JC < J; ++u) a = vfma(S.cf[j + u * JC], u == 1 ? v1 : v2, a);
    }
    return a;
  };
  if (JC < 2) {
    for (int r = tid; r < R; r += T) put(r, row(r, 0));
  } else {
    VV* part = reinterpret_cast<VV*>(S.part);
    if (tid < R * JC) part[tid] = row(tid % R, tid / R);
    __syncthreads();
    if (tid < R) {
      VV a = part[tid];
      for (int c = 1; c < JC; ++c) a = vadd(a, part[c * R + tid]);
      put(tid, a);
    }
  }
}

// y = exp(-i h K) e_0 for the act x act Hessenberg matrix in hs (column i at i * kArnHs): Taylor
// terms on sub-steps of infinity-norm at most 1, each to its remainder bound.  Four lanes a row; the
// plan (a few FP64 divisions and roots) on one warp, since an FP64 instruction costs 76 cycles in
// every warp that runs it.  A Hermitian H's matrix is tridiagonal up to rounding (band): only that is
// used.  False when the norm asks for more sub-steps than kArnMaxSubsteps (or is not finite).
__device__ bool arn_expm(const cplx* hs, int act, double h, bool band, cplx (*t)[kArnMaxExp], cplx* y, double* work) {
  __shared__ int steps, terms;
  __shared__ double fac[32];  // (h / steps) / p
  const int tid = threadIdx.x, row = tid >> 2, c4 = tid & 3;
  static_assert(kArnThreads >= 4 * kArnMaxExp && kArnMaxExp <= 32, "four lanes a row");
  const int c0 = max(row - 1, 0) + c4, c1 = band ? min(act, row + 2) : act;
  if (row / 8 * 8 < act) {  // warps with a row
    double rs = 0.0;
    if (row < act)
      for (int c = c0; c < c1; c += 4) {
        const cplx v = hs[c * kArnHs + row];
        rs += fabs(v.re) + fabs(v.im);
      }
    for (int o = 2; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
    if (c4 == 0 && row < act) work[row] = rs;
  }
  if (tid < act) y[tid] = mkc(tid == 0 ? 1.0 : 0.0, 0.0);
  __syncthreads();
  if (tid < 32) {
    double nrm = (tid < act) ? work[tid] : 0.0;
    const unsigned fine = __all_sync(0xffffffffu, nrm < 1e300);  // not for a NaN
    const unsigned mx = __reduce_max_sync(0xffffffffu, q_mag(nrm));
    nrm = __hiloint2double((int)mx, -1);  // at most 2^-20 above the largest
    const double theta = nrm * fabs(h);
    int st = -1, tm = 1;
    if (fine && theta <= (double)kArnMaxSubsteps) {
      st = max(1, (int)ceil(theta));
      const double hst = h / st, th = theta / st;
      double b = 1.0;  // th^i / i!
      for (int i = 1; i <= 30; ++i) {
        b *= th * kArnInv[i];
        if (b <= kArnTerms) break;
        tm = i;
      }
      fac[tid] = (tid >= 1) ? hst * kArnInv[tid] : 0.0;
    }
    if (tid == 0) {
      steps = st;
      terms = tm;
    }
  }
  __syncthreads();
  if (steps < 0) return false;
  for (int s = 0; s < steps; ++s) {
    if (tid < act) t[0][tid] = y[tid];
    __syncthreads();
    for (int p = 1; p <= terms; ++p) {
      const cplx* src = t[(p - 1) & 1];
      if (row / 8 * 8 < act) {
        cplx a = mkc(0.0, 0.0);
        if (row < act)
          for (int c = c0; c < c1; c += 4) a = vfma(hs[c * kArnHs + row], src[c], a);
        for (int o = 2; o > 0; o >>= 1) a = vadd(a, shfl_xor(a, o));
        if (c4 == 0 && row < act) {
          const cplx tn = mkc(fac[p] * a.im, -fac[p] * a.re);  // (-i f) a
          t[p & 1][row] = tn;
          y[row] = vadd(y[row], tn);
        }
      }
      __syncthreads();
    }
  }
  return true;
}

template <typename MV, typename VV, bool kExp, bool kOne>
__global__ void __launch_bounds__(kArnThreads, 1) arn_kernel(ArnArgs<MV, VV> A) {
  using QT = typename QVec<VV>::T;
  constexpr int T = kArnThreads;
  extern __shared__ __align__(16) unsigned char arn_smem[];
  __shared__ ArnShared<VV, T> S;
  const int tid = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * A.rows;
  const int R = (int)max((int64_t)0, min((int64_t)A.rows, A.n - r0));
  cplx* hs = reinterpret_cast<cplx*>(arn_smem);  // kExp: the Hessenberg matrix
  VV* wd = reinterpret_cast<VV*>(arn_smem + (kExp ? sizeof(cplx) * kArnHs * kArnMaxExp : 0));  // w of the rows
  QT* wq = reinterpret_cast<QT*>(wd + A.ldr);  // the same quantised
  QT* Vs = wq + A.ldr;                         // vector j quantised at Vs + j ldr
  VV* Vg = A.V + r0;                           // the block's rows in memory: vector j at Vg + j ld
  constexpr int kPer = sizeof(VV) / sizeof(double);
  const GridX& X = A.X;
  if (kExp)
    for (int i = tid; i < kArnHs * kArnMaxExp; i += T) hs[i] = mkc(0.0, 0.0);
  // lanes per row of the product: more loads in flight for a short slice, on few enough warps
  // that the lanes' FP64 sums do not cost more than the waits they save
  int lanes = 1;
  while (lanes < 4 && 2 * lanes * R <= 160) lanes *= 2;

  // wd quantised into dst; the scale returned to every thread
  auto quantise = [&](unsigned mag, QT* dst) {
    const QScale q = q_scale(arn_block_max<VV, T>(S, mag));
    for (int i = tid; i < R; i += T) dst[i] = q_of(wd[i], q.E);
    return q.u;
  };

  // The block's ||v||^2 of the rows just quantised on the scale u (each thread its own), in thread 0: integers
  // again, where the sum of FP64 values over sixteen warps takes 2,000 cycles.
  const int nact = (min(R, T) + 31) / 32;  // warps with rows
  auto norm2 = [&](const QT* v, double u) {
    QSum t{0, 0u};
    if ((tid >> 5) < nact) {
      QDot<VV> a;
      for (int i = tid; i < R; i += T) a.add(v[i], v[i]);
      t.set(a.re());
      t = q_warp_sum(t);
      if ((tid & 31) == 0) S.part[tid >> 5] = t;
    }
    __syncthreads();
    if (tid < 32) {
      t = tid < nact ? S.part[tid] : QSum{0, 0u};
      t = q_warp_sum(t);
    }
    return tid == 0 ? t.value() * u * u : 0.0;
  };
  const bool mute = X.hold && blockIdx.x == 0;
  // The norm of vector j from its square: one thread (a square root in every warp would take longer than
  // the exchange).
  auto set_norm = [&](int j, double n2) {
    const double s = rsqrt(n2), nr = n2 > 0.0 ? n2 * s : n2;
    S.scl[j] = s;
    S.us[j] = S.u[j] * s;
    S.stop = (j == 0) ? !(n2 > 0.0) : nr < 1e-10;
    if (kExp && j > 0) hs[(j - 1) * kArnHs + j] = mkc(nr, 0.0);
    if (blockIdx.x == 0) {
      if (j == 0) A.st->zero = (n2 > 0.0) ? 0 : 1;
      A.st->nrm[j] = nr;
      A.st->scl[j] = s;
    }
  };
  // this block's share of ||V[j]||^2, in thread 0 until the next exchange takes it along
  double nshare = 0.0;

  if (A.first == 1) {
    unsigned mag = 0;
    for (int r = tid; r < R; r += T) {
      VV v;
      arn_from(v, A.psi_in[r0 + r]);
      if (!mute) x_put(Vg + r, v);
      wd[r] = v;
      mag = max(mag, q_mag(v));
    }
    const double u = quantise(mag, Vs);
    if (tid == 0) S.u[0] = S.us[0] = u;
    nshare = norm2(Vs, u);
  } else {
    for (int j = tid; j < A.first; j += T) S.scl[j] = A.st->scl[j];
    __syncthreads();
    for (int j = 0; j < A.first; ++j) {
      unsigned mag = 0;
      for (int r = tid; r < R; r += T) {
        const VV v = Vg[(int64_t)j * A.ld + r];
        wd[r] = v;
        mag = max(mag, q_mag(v));
      }
      const double u = quantise(mag, Vs + (size_t)j * A.ldr);
      if (tid == 0) {
        S.u[j] = u;
        S.us[j] = u * S.scl[j];
      }
    }
    __syncthreads();
  }

  int stop = 0;
  for (int J = A.first; J <= A.last; ++J) {
    const VV* x = A.V + (int64_t)(J - 1) * A.ld;
    VV* wg = Vg + (int64_t)J * A.ld;
    const int J1 = A.herm ? min(J, 2) : J, j1 = J - J1;  // vectors of the first pass
    double* slot1 = A.slots + (size_t)(2 * (J - A.first)) * A.xstride;
    double* slot2 = slot1 + A.xstride;
    const bool scaled = J == A.first && A.first > 1;  // V[J-1]'s scale is known from an earlier launch
    // 1: w = H V[J-1], not yet scaled, its projections, and the norm of V[J-1], which scales both
    {
      const int g = tid / lanes, sub = tid & (lanes - 1), per = T / lanes;
      unsigned mag = 0;
      for (int r = g; (r & ~(32 / lanes - 1)) < R; r += per) {  // whole warps
        const VV a = arn_row(A, x, r0 + r, r < R, sub, lanes);
        if (r < R && sub == 0) {
          wd[r] = a;
          mag = max(mag, q_mag(a));
        }
      }
      const double uw = quantise(mag, wq);
      __syncthreads();
      arn_dots_res<VV, T>(S, Vs, A.ldr, j1, J1, wq, uw, R);
      if (tid == 0) S.xv[J1 * kPer] = nshare;
    }
    __syncthreads();
    x_sum<kOne>(X, slot1, S.xv, J1 * kPer + 1, S.red);
    if (tid == 0 && !scaled) set_norm(J - 1, S.red[J1 * kPer]);
    __syncthreads();
    if (S.stop && J > 1 && !scaled) {  // sparse_algorithm.hpp:387: the breaking step counts
      stop = J - 1;
      break;
    }
    if (!kExp && S.stop && !scaled) return;  // a zero start vector: the host reports it (evolve goes on, as NaNs)
    const double sx = S.scl[J - 1];
    if (tid < J1) {
      // <v_j, w> = sx <v_j, H V[J-1]>, and v_{J-1}'s own scale, which its share above did not have
      VV c = vscale(sx, reinterpret_cast<const VV*>(S.red)[tid]);
      if (tid == J1 - 1 && !scaled) c = vscale(sx, c);
      S.c1[tid] = c;
      S.cf[tid] = vscale(S.scl[j1 + tid], c);
    }
    __syncthreads();
    // 2: the first pass taken out, projections of what is left
    {
      unsigned mag = 0;
      arn_comb<VV, T>(S, Vg + (int64_t)j1 * A.ld, A.ld, J1, R, [&](int r, VV sum) {
        const VV o = vfma(sx, wd[r], vscale(-1.0, sum));
        wd[r] = o;
        mag = max(mag, q_mag(o));
      });
      const double uw = quantise(mag, wq);
      __syncthreads();
      arn_dots_res<VV, T>(S, Vs, A.ldr, 0, J, wq, uw, R);
    }
    x_sum<kOne>(X, slot2, S.xv, J * kPer, S.red);
    if (tid < J) {
      const VV c = reinterpret_cast<const VV*>(S.red)[tid];
      S.cf[tid] = vscale(S.scl[tid], c);
      const VV hij = (tid >= j1) ? vadd(S.c1[tid - j1], c) : c;
      if (kExp) hs[(J - 1) * kArnHs + tid] = arn_c(hij);
      if (blockIdx.x == 0) {
        if (kExp) A.hcol[(size_t)(J - 1) * kArnLdh + tid] = arn_c(hij);
        if (tid == J - 1) A.st->alpha[J] = arn_re(hij);
      }
    }
    // 3: the second pass taken out, the norm, and the rows for everybody's gathers
    __syncthreads();
    unsigned mag = 0;
    arn_comb<VV, T>(S, Vg, A.ld, J, R, [&](int r, VV sum) {
      const VV o = vadd(wd[r], vscale(-1.0, sum));
      wd[r] = o;
      if (!mute) x_put(wg + r, o);
      mag = max(mag, q_mag(o));
    });
    // the last column's vector is projected on no more: only its norm is needed
    QT* dst = J < A.kdim ? Vs + (size_t)J * A.ldr : wq;
    const double u = quantise(mag, dst);
    if (J < A.kdim && tid == 0) S.u[J] = S.us[J] = u;
    nshare = norm2(dst, u);
  }
  if (!stop) {  // the last vector's norm
    if (tid == 0) S.xv[0] = nshare;
    __syncthreads();
    x_sum<kOne>(X, A.slots + (size_t)(2 * (A.last + 1 - A.first)) * A.xstride, S.xv, 1, S.red);
    if (tid == 0) set_norm(A.last, S.red[0]);
    __syncthreads();
    if (S.stop) stop = A.last;
  }
  if (blockIdx.x == 0 && tid == 0) A.st->stop = stop;
  if (!kExp) return;
  const int act = stop ? stop : A.last;
  __shared__ cplx tt[2][kArnMaxExp];
  __shared__ cplx y[kArnMaxExp];
  if (tid == 0) hs[(act - 1) * kArnHs + act] = mkc(0.0, 0.0);
  __syncthreads();
  const bool ok = arn_expm(hs, act, A.h, A.herm != 0, tt, y, S.red);
  if (blockIdx.x == 0 && tid == 0) A.st->need_host = ok ? 0 : 1;
  if (!ok) return;
  if (tid < act) y[tid] = vscale(S.scl[tid], y[tid]);
  __syncthreads();
  // psi_out = sum_j y_j v_j on the block's rows
  if constexpr (kPer == 2) {
    if (tid < act) S.cf[tid] = y[tid];
    __syncthreads();
    cplx* out = A.psi_out + r0;
    arn_comb<VV, T>(S, Vg, A.ld, act, R, [&](int r, VV sum) { out[r] = sum; });
  }
}

// ---------------------------------------------------------------- host
static bool arn_coop(Ctx* ctx) {
  static const int coop = [&] {  // once per process (thread-safe initialisation)
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrCooperativeLaunch, ctx->device) != cudaSuccess) v = 0;
    return v;
  }();
  return coop != 0;
}

// Served requests keep the kernels launched one by one: a co-resident grid waits for room beside
// the other lanes' kernels, and an operator with a product kernel of the caller's choice launches that.
// QD_KRYLOV_STEP=split keeps them for every call.
bool arn_res_fits(qd_ham* H, int kdim) {
  const char* e = std::getenv("QD_KRYLOV_STEP");
  if (e && std::strcmp(e, "split") == 0) return false;
  return !H->one_shot && !H->spmv_chosen && kdim >= 1 && kdim < kArnMaxVecs && H->dim >= 1 && H->dim < (int64_t)1 << 30 &&
         arn_coop(H->ctx);
}

// True if buffers moved: what an earlier launch left in them is gone.
static bool arn_ensure(ArnRes& B, int64_t n, int kdim, bool real_v, size_t slots) {
  bool moved = false;
  if (B.n != n || B.kdim != kdim || B.real_v != real_v) {
    B.n = 0;  // until the memory is there
    B.kdim = kdim;
    B.real_v = real_v;
    B.ld = (n + 31) / 32 * 32;
    B.ncl = 0;
    B.V.alloc((size_t)(kdim + 1) * B.ld * (real_v ? sizeof(double) : sizeof(cplx)));
    B.n = n;
    moved = true;
  }
  if (!B.hcol.p) B.hcol.alloc((size_t)kArnLdh * (kArnMaxExp + 1));
  const size_t want = sizeof(ArnStatus) + slots * sizeof(double);
  if (B.slots.n < want) {
    B.slots.alloc(want);
    moved = true;  // the status holds the stored vectors' scales
  }
  return moved;
}

template <typename MV, typename VV, bool kExp>
static bool arn_launch(qd_ham* H, const MV* vals, ArnRes& B, const cplx* psi_in, cplx* psi_out, double h, int kdim,
                       int first, int last) {
  Ctx* ctx = H->ctx;
  const int64_t n = H->dim;
  constexpr int kPer = sizeof(VV) / sizeof(double);
  const size_t fixed = kExp ? sizeof(cplx) * kArnHs * kArnMaxExp : 0;
  const auto smem_of = [&](int rows) { return fixed + (size_t)(kdim + 2) * (rows | 1) * sizeof(VV); };
  int maxsm = 0;
  QD_CUDA(cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  // one block up to 64 rows (an exchange would cost more than it saves), then clusters of eight blocks
  // of at least kArnMinRows rows, as many as fit the device at once
  const bool one = n <= 64;
  auto kern = one ? arn_kernel<MV, VV, kExp, true> : arn_kernel<MV, VV, kExp, false>;
  int ncl = one ? 1 : (int)std::min<int64_t>(ctx->num_sms / kArnCluster, ceil_div(n, kArnCluster * kArnMinRows));
  int rows = 0;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = kArnCluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kArnThreads);
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = one ? 1 : 2;
  if (B.n == n && B.kdim == kdim && B.real_v == (kPer == 1) && B.ncl > 0) {
    ncl = B.ncl;
    rows = B.rows;
  } else {
    for (;;) {
      rows = (int)ceil_div(n, one ? 1 : ncl * kArnCluster);
      if (smem_of(rows) + sizeof(ArnShared<VV, kArnThreads>) + 4096 > (size_t)maxsm || rows > kArnMaxResRows) return false;
      if (one) break;
      allow_dynamic_smem(kern, ctx->device);
      cfg.gridDim = dim3((unsigned)(ncl * kArnCluster));
      cfg.dynamicSmemBytes = smem_of(rows);
      cfg.attrs = at + 1;
      cfg.numAttrs = 1;
      int fit = 0;
      QD_CUDA(cudaOccupancyMaxActiveClusters(&fit, kern, &cfg));
      cfg.attrs = at;
      cfg.numAttrs = 2;
      if (fit >= ncl) break;
      if (fit < 1) return false;
      ncl = fit;
    }
  }
  const int grid = one ? 1 : ncl * kArnCluster;
  const size_t smem = smem_of(rows), xstride = (size_t)grid * (kPer * kdim + 1);
  cfg.gridDim = dim3((unsigned)grid);
  cfg.dynamicSmemBytes = smem;
  const bool moved = arn_ensure(B, n, kdim, kPer == 1, (2 * (size_t)kdim + 1) * xstride);
  QD_REQUIRE(!moved || first == 1, QD_ERR_INVALID, "the open solve's basis is gone: start it again");
  B.ncl = ncl;
  B.rows = rows;
  ArnArgs<MV, VV> A;
  std::memset(&A, 0, sizeof(A));
  A.n = n;
  A.ld = B.ld;
  A.rows = rows;
  A.ldr = rows | 1;
  A.rowptr = H->rowptr.p;
  A.colidx = H->colidx.p;
  A.vals = vals;
  A.psi_in = psi_in;
  A.V = reinterpret_cast<VV*>(B.V.p);
  A.kdim = kdim;
  A.hcol = B.hcol.p;
  A.st = reinterpret_cast<ArnStatus*>(B.slots.p);
  A.first = first;
  A.last = last;
  A.herm = (H->flags & QD_HAM_HERMITIAN) ? 1 : 0;
  // the blocks write their rows one by one: apart from the caller's state until none of them has given up a wait
  const bool apart = kExp && !one;
  if (apart && B.out.n < (size_t)n) B.out.alloc(n);
  A.psi_out = apart ? B.out.p : psi_out;
  A.h = h;
  A.slots = reinterpret_cast<double*>(B.slots.p + sizeof(ArnStatus));
  A.xstride = xstride;
  A.X.abort = &A.st->abort;
  const unsigned wait_out = step_wait_out_polls();
  A.X.polls = wait_out ? wait_out : kXPolls;
  A.X.hold = wait_out != 0;
  // every slot this launch writes, empty: the vectors (gathered as they are written), the exchanges
  // and, on a fresh start, the status (a continued one keeps the stored vectors' scales)
  const int v0 = (first == 1) ? 0 : first;
  QD_CUDA(cudaMemsetAsync(A.V + (int64_t)v0 * B.ld, kXEmptyByte, (size_t)(last + 1 - v0) * B.ld * sizeof(VV),
                          ctx->stream));
  const size_t slot_bytes = (2 * (size_t)(last + 1 - first) + 1) * xstride * sizeof(double);
  if (first == 1) {
    QD_CUDA(cudaMemsetAsync(B.slots.p, kXEmptyByte, sizeof(ArnStatus) + slot_bytes, ctx->stream));
  } else {
    QD_CUDA(cudaMemsetAsync(&A.st->abort, kXEmptyByte, sizeof(int), ctx->stream));
    QD_CUDA(cudaMemsetAsync(A.slots, kXEmptyByte, slot_bytes, ctx->stream));
  }
  allow_dynamic_smem(kern, ctx->device);
  QD_CUDA(cudaLaunchKernelEx(&cfg, kern, A));
  QD_LAUNCHED(ctx);
  if (apart) launch_commit(ctx, n, B.out.p, psi_out, &A.st->abort, &A.st->need_host);
  QD_CUDA(cudaMemcpyAsync(&B.host, A.st, sizeof(ArnStatus), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  QD_REQUIRE(B.host.abort != kXAborted, QD_ERR_TIMEOUT, "an Arnoldi step's blocks did not meet within the wait limit");
  return true;
}

bool arn_res_evolve(qd_ham* H, ArnRes& B, const cplx* psi_in, cplx* psi_out, double h, int steps, int* act_out) {
  const bool real = (H->flags & QD_HAM_REAL) != 0;
  const bool ran =
      real ? arn_launch<double, cplx, true>(H, H->vals_r.p, B, psi_in, psi_out, h, steps, 1, steps)
           : arn_launch<cplx, cplx, true>(H, H->vals_c.p, B, psi_in, psi_out, h, steps, 1, steps);
  if (!ran) return false;
  const int act = B.host.stop ? B.host.stop : steps;
  if (act_out) *act_out = act;
  if (!B.host.need_host) return true;
  // a large ||h K||: scaling and squaring on the host, as the kernels launched one by one do
  Ctx* ctx = H->ctx;
  std::vector<cplx> hc((size_t)kArnLdh * act);
  QD_CUDA(cudaMemcpyAsync(hc.data(), B.hcol.p, hc.size() * sizeof(cplx), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  dense::Mat K((size_t)act * act, dense::cd(0.0, 0.0)), E;
  for (int i = 0; i < act; ++i) {
    for (int j = 0; j <= i; ++j) K[(size_t)i * act + j] = dense::cd(hc[(size_t)i * kArnLdh + j].re, hc[(size_t)i * kArnLdh + j].im);
    if (i + 1 < act) K[(size_t)i * act + i + 1] = B.host.nrm[i + 1];
  }
  for (auto& a : K) a *= dense::cd(0.0, -h);
  QD_REQUIRE(dense::expm(K, act, E), QD_ERR_INVALID, "matrix exponential failed");
  std::vector<cplx> e(act);
  for (int j = 0; j < act; ++j) e[j] = mkc(E[j].real() * B.host.scl[j], E[j].imag() * B.host.scl[j]);
  QD_CUDA(cudaMemcpyAsync(B.hcol.p, e.data(), act * sizeof(cplx), cudaMemcpyHostToDevice, ctx->stream));
  launch_ev_combine(ctx, H->dim, reinterpret_cast<const cplx*>(B.V.p), B.ld, act, B.hcol.p, psi_out);
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  return true;
}

bool arn_res_steps(qd_ham* H, ArnRes& B, const cplx* psi, int kdim, bool real_v, int first, int last) {
  if (H->flags & QD_HAM_REAL) {
    if (real_v) return arn_launch<double, double, false>(H, H->vals_r.p, B, psi, nullptr, 0.0, kdim, first, last);
    return arn_launch<double, cplx, false>(H, H->vals_r.p, B, psi, nullptr, 0.0, kdim, first, last);
  }
  return arn_launch<cplx, cplx, false>(H, H->vals_c.p, B, psi, nullptr, 0.0, kdim, first, last);
}

}  // namespace qd
