// batch.cu -- many Lanczos ground states in one persistent launch.
//
// The mixed-precision form of the reference's Lanczos (sparse_algorithm.hpp:
// 395-425, 564-585) for a packed work list of independent, uneven instances:
//   * an instance is owned by one CTA or by a thread-block cluster of 2 to 8,
//     by its dimension and the work of the call (batch_widths; an instance's
//     bits depend on this size); CTAs and clusters take the next instance of
//     their size from an atomic counter;
//   * each CTA of a cluster keeps a slice of the rows of every vector, and the
//     inner products are combined through distributed shared memory (each CTA
//     adds the CTAs' partials in rank order, so every CTA holds the same bits)
//     between hardware cluster barriers -- one SM's memory parallelism is far
//     too little for an instance of 10^5 rows;
//   * the lists are sorted by decreasing nnz (longest first);
//   * matrix values and Krylov vectors are FP32 and so is the product;
//   * every inner product keeps FP32 partial sums over at most 64 elements per
//     thread (16 in the Gram-Schmidt coefficients); a warp adds them exactly, in
//     integers (f_fix), and warps, CTAs and tiles are added in FP64;
//   * after the three-term step (the reference's local orthogonalisation
//     against the two previous vectors) the new vector is orthogonalised
//     once more against the whole stored basis (classical Gram-Schmidt);
//   * the tridiagonal matrix (FP64) is solved on the device by the block: the
//     lowest eigenvalue by bisection, its vector by inverse iteration;
//   * the Ritz vector gets one FP64 refinement: E = psi^T H psi / psi^T psi with
//     the FP64 matrix values and FP64 accumulation.
// No CTA spins on another: the only shared state is the work counter, and the
// CTAs of a cluster meet only at hardware cluster barriers, which the
// hardware schedules together and every CTA of a cluster reaches the same
// number of times (the instance index and every stopping decision are the
// same in all of them).
//
// Measured (GB300), 80 steps.  With the threads' partials added in FP64, the
// step's scalars formed in every warp, a conversion of each coefficient in the
// update's inner loop and QL on one thread, FP64 issue (72 cycles a warp
// instruction, conversions included) set the time: 32 chains of 12, 14, 16 and
// 18 sites 15.2, 16.3, 23.8 and 25.7 ms; now 1.3, 2.9, 3.9 and 11.8 ms, and 96
// mixed chains of 14 to 18 sites 37.5 -> 15.8 ms.  At 18 sites on 8 CTAs a step
// is 300,000 cycles: the product 100,000 (its gathers and the strided reads of
// the columns), the coefficients 70,000 and the update 65,000 (HBM), the rest
// the barriers' waits.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <numeric>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "batch.cuh"
#include "krylov.cuh"
#include "tridiag.cuh"

namespace cg = cooperative_groups;

namespace qd {

constexpr int kBatchThreads = 512;  // two CTAs per SM
constexpr int kBatchMaxSteps = 256;
constexpr int kChunk = 64;  // FP32 partial sums cover at most this many elements
constexpr int64_t kClusterMinDim = 32768;
constexpr int64_t kBatchSplitMinDim = 8192;  // below it an instance stays on one CTA
constexpr int64_t kBatchMinRows = 1024;      // slices are not made shorter

constexpr int kWTile = 4096;  // elements of w staged in shared memory for the Gram-Schmidt coefficients

struct BlockScratch {
  float wt[kWTile];
  double red[kBatchThreads / 32];
  double red3[kBatchThreads / 32][3];
  long long fq[3][kBatchThreads / 32];    // warps' integer sums and their exponents
  unsigned fe[3][kBatchThreads / 32];
  float fu[kBatchThreads / 32];
  double bcast;
  double bcast3[3];
  double xp[2], bc[2];                    // this CTA's partial of a cluster sum, and the sum
  double xp3[2][3];
  double al, bp;                          // the step's alpha and beta before the Gram-Schmidt pass
  float c1, c2;                           // the same on the stored vectors
  double ga, gb;                          // bracket of the lowest eigenvalue
  unsigned gm[4];
  double hp[2][kBatchMaxSteps + 2];       // this CTA's partials of the Gram-Schmidt coefficients
  double alpha[kBatchMaxSteps + 2];
  double beta[kBatchMaxSteps + 2];
  double y[kBatchMaxSteps + 2];
  double h[kBatchMaxSteps + 2];
  float cf[kBatchMaxSteps + 2];           // update coefficients of the stored vectors, negated; Ritz coefficients
  double scl[kBatchMaxSteps + 2];         // basis vector j is scl[j] * V[j] (V stored unnormalised)
  int stop;
  int idx;
};

// The device's nanosecond clock (the instance schedule in out[5], out[6]).
__device__ __forceinline__ unsigned long long batch_clock_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---- sums of FP32 partials in integers
// An FP64 instruction takes an SM quarter 64 to 76 cycles whatever its active lanes, conversions included: the
// FP64 sums of the threads' FP32 partials took several times the products that they summed.  A warp adds them as
// integers instead, exact down to 2^-30 of the last place of the largest (2^-54 of it: FP64 rounds its sums at
// 2^-53), and one conversion serves a warp's sum, or a lane each the sums of many vectors.
__device__ __forceinline__ unsigned f_mag(float v) { return __float_as_uint(v) & 0x7fffffffu; }
// The exponent field of the largest magnitude word of a warp.
__device__ __forceinline__ unsigned f_top(unsigned mag) { return max(__reduce_max_sync(0xffffffffu, mag) >> 23, 1u); }
// v as an integer in units of 2^(e - 180), e at least its exponent field: below 2^54.
__device__ __forceinline__ long long f_fix(float v, unsigned e) {
  const unsigned b = __float_as_uint(v);
  const unsigned ev = (b >> 23) & 0xffu;
  const unsigned m = (b & 0x7fffffu) | (ev ? 0x800000u : 0u);
  const int sh = 30 - (int)(e - max(ev, 1u));
  const long long q = sh >= 0 ? (long long)m << sh : (long long)(m >> min(-sh, 31));
  return (int)b < 0 ? -q : q;
}
__device__ __forceinline__ double f_unit(unsigned e) {  // NaN when a value was not finite
  return e == 0xffu ? __longlong_as_double(0x7ff8000000000000ll) : __hiloint2double((int)(e + 843) << 20, 0);
}
__device__ __forceinline__ long long f_warp_sum(long long q) {  // at most 256 values
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
  return q;
}
// Block sums of NV values per thread into out (shared memory), complete after the caller's next barrier.
template <int NV>
__device__ __forceinline__ void block_sum_f(const float (&v)[NV], BlockScratch& S, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const unsigned e = f_top(f_mag(v[q]));
    const long long t = f_warp_sum(f_fix(v[q], e));
    if (lane == 0) {
      S.fq[q][warp] = t;
      S.fe[q][warp] = e;
    }
  }
  __syncthreads();
  if (warp < NV) {  // warps 0 .. NV - 1, each on its own SM quarter
    constexpr int nw = kBatchThreads / 32;
    double t = lane < nw ? (double)S.fq[warp][lane] * f_unit(S.fe[warp][lane]) : 0.0;
#pragma unroll
    for (int o = nw / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) out[warp] = t;
  }
}

// FP64 sum over the block of per-thread values; every thread gets the result.
__device__ double block_sum_all(double v, BlockScratch& S) {
  v = warp_sum0(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) S.red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double t = (lane < (int)(blockDim.x >> 5)) ? S.red[lane] : 0.0;
    t = warp_sum0(t);
    if (lane == 0) S.bcast = t;
  }
  __syncthreads();
  return S.bcast;
}

// The same for three values at once.
__device__ void block_sum_all3(double (&v)[3], BlockScratch& S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = warp_sum0(v[q]);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q) S.red3[warp][q] = v[q];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double t = (lane < (int)(blockDim.x >> 5)) ? S.red3[lane][q] : 0.0;
      t = warp_sum0(t);
      if (lane == 0) S.bcast3[q] = t;
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 3; ++q) v[q] = S.bcast3[q];
}

// <a, b> over [lo, hi) with FP32 products and partials over <= kChunk
// elements, FP64 beyond; the block's total in every thread.  lo is a
// multiple of 32 and the vectors start on a 32-element boundary.
__device__ double block_dot(const float* __restrict__ a, const float* __restrict__ b, int64_t lo, int64_t hi,
                            BlockScratch& S) {
  double dacc = 0.0;
  float acc = 0.f;
  int cnt = 0;
  const int64_t q0 = lo >> 2, q1 = hi >> 2;
  const float4* a4 = reinterpret_cast<const float4*>(a);
  const float4* b4 = reinterpret_cast<const float4*>(b);
#pragma unroll 4
  for (int64_t i = q0 + threadIdx.x; i < q1; i += blockDim.x) {
    const float4 x = a4[i], y = b4[i];
    acc = fmaf(x.x, y.x, acc);
    acc = fmaf(x.y, y.y, acc);
    acc = fmaf(x.z, y.z, acc);
    acc = fmaf(x.w, y.w, acc);
    if (++cnt == kChunk / 4) {
      dacc += (double)acc;
      acc = 0.f;
      cnt = 0;
    }
  }
  for (int64_t i = (q1 << 2) + threadIdx.x; i < hi; i += blockDim.x) acc = fmaf(a[i], b[i], acc);
  dacc += (double)acc;
  return block_sum_all(dacc, S);
}

// y = H x on rows [lo, hi) (FP32 values, FP32 accumulation), one thread per
// row, two rows per thread at a time (r and r + blockDim.x: two independent
// chains of four gathers), each summed in its entry order.  x is a basis
// vector written earlier in the same launch (by this CTA or, for a cluster, by
// all of its CTAs), so it is read with ordinary loads, not the read-only path.
template <bool kUniform>
__device__ __forceinline__ void rows_f32(const BatchInst& I, const float* x, int64_t b0, int m0, int64_t b1, int m1,
                                         float& a0, float& a1) {
  const int32_t* c0 = I.colidx + b0;
  const int32_t* c1 = I.colidx + b1;
  const float* v0 = I.vals_f + b0;
  const float* v1 = I.vals_f + b1;
  const int m = max(m0, m1);
  for (int k = 0; k < m; k += 4) {  // eight gathers in flight, also over the ends of the rows
    int32_t c[8];
    float v[8], xv[8];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool p0 = k + u < m0, p1 = k + u < m1;
      c[u] = p0 ? c0[k + u] : -1;
      c[4 + u] = p1 ? c1[k + u] : -1;
      if (!kUniform) {
        v[u] = p0 ? v0[k + u] : 0.f;
        v[4 + u] = p1 ? v1[k + u] : 0.f;
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) xv[u] = c[u] >= 0 ? x[c[u]] : 0.f;
    if (kUniform) {
      a0 += (xv[0] + xv[1]) + (xv[2] + xv[3]);
      a1 += (xv[4] + xv[5]) + (xv[6] + xv[7]);
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        a0 = fmaf(v[u], xv[u], a0);
        a1 = fmaf(v[4 + u], xv[4 + u], a1);
      }
    }
  }
}

// The product of the step and, row by row as it is formed, this thread's
// shares of <V2, y>, <V1, y> and <V1, V2> (FP32 over at most kChunk rows, FP64
// beyond; V2 null on the first step).
struct ProdDots {
  float fa = 0.f, fb = 0.f, fc = 0.f;
  double da = 0.0, db = 0.0, dc = 0.0;
  int cnt = 0;
  __device__ __forceinline__ void add(const float* x, const float* v2, int64_t r, float yr) {
    const float x1 = x[r];
    fb = fmaf(x1, yr, fb);
    if (v2) {
      const float x2 = v2[r];
      fa = fmaf(x2, yr, fa);
      fc = fmaf(x1, x2, fc);
    }
    if (++cnt == kChunk) flush();
  }
  __device__ __forceinline__ void flush() {
    da += (double)fa;
    db += (double)fb;
    dc += (double)fc;
    fa = fb = fc = 0.f;
    cnt = 0;
  }
};

// kUniform: every off-diagonal value is one c (uniform hopping, any diagonal): y_r = c (sum of x over the
// row's stored columns) + e_r x_r with e_r = d_r - c where the row stores its diagonal (else 0), the column
// indices the only per-entry reads (no values).
template <bool kUniform>
__device__ void block_spmv_f32(const BatchInst& I, const float* x, const float* v2, float* __restrict__ y, int64_t lo,
                               int64_t hi, ProdDots& pd) {
  const float c = kUniform ? __ldg(I.coff) : 0.f;
  const int64_t bs = blockDim.x;
  auto finish = [&](int64_t row, float sum) {
    const float yr = kUniform ? fmaf(c, sum, __ldg(I.diag_f + row) * x[row]) : sum;
    y[row] = yr;
    pd.add(x, v2, row, yr);
  };
  for (int64_t r = lo + threadIdx.x; r < hi; r += 2 * bs) {
    const bool two = r + bs < hi;
    const int64_t b0 = I.rowptr[r], b1 = two ? I.rowptr[r + bs] : b0;
    const int m0 = (int)(I.rowptr[r + 1] - b0), m1 = two ? (int)(I.rowptr[r + bs + 1] - b1) : 0;
    float a0 = 0.f, a1 = 0.f;
    rows_f32<kUniform>(I, x, b0, m0, b1, m1, a0, a1);
    finish(r, a0);
    if (two) finish(r + bs, a1);
  }
}

// ---------------------------------------------------------------- uniform check
struct BunJob {
  int64_t n;
  const int64_t* rowptr;
  const int32_t* colidx;
  const float* vals;
  int* flag;
  float* c;
  float* d;
};

// One CTA per Hamiltonian: c = the first off-diagonal value (rows in order), then flag = 1
// if every off-diagonal value equals c and c is not 0 (an explicit zero off the diagonal
// fails: the uniform form would add it as c), and d_r = diagonal - c where the row stores
// its diagonal, else 0.
__global__ void __launch_bounds__(512) bun_check_kernel(const BunJob* jobs) {
  const BunJob J = jobs[blockIdx.x];
  __shared__ float sc;
  __shared__ int found, bad;
  __shared__ unsigned long long first;  // the first row with an off-diagonal entry
  if (threadIdx.x == 0) {
    found = 0;
    bad = 0;
    first = ~0ull;
  }
  __syncthreads();
  for (int64_t r = threadIdx.x; r < J.n; r += blockDim.x) {
    bool off = false;
    for (int64_t k = J.rowptr[r]; k < J.rowptr[r + 1] && !off; ++k) off = J.colidx[k] != (int32_t)r;
    if (off) {
      atomicMin(&first, (unsigned long long)r);
      break;  // this thread's later rows are larger
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && first != ~0ull) {
    const int64_t r = (int64_t)first;
    for (int64_t k = J.rowptr[r]; k < J.rowptr[r + 1]; ++k)
      if (J.colidx[k] != (int32_t)r) {
        sc = J.vals[k];
        found = 1;
        break;
      }
  }
  __syncthreads();
  const float c = found ? sc : 0.f;
  for (int64_t r = threadIdx.x; r < J.n; r += blockDim.x) {
    float d = 0.f;  // d_r - c where the row stores its diagonal (its x_r is in the column sum), else 0
    for (int64_t k = J.rowptr[r]; k < J.rowptr[r + 1]; ++k) {
      if (J.colidx[k] == (int32_t)r) d = J.vals[k] - c;
      else if (J.vals[k] != c || c == 0.f) bad = 1;
    }
    J.d[r] = d;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    *J.flag = (found && !bad) ? 1 : 0;
    *J.c = c;
  }
}

// The check for the Hamiltonians of a call that have not had it, in one launch.
static void check_uniform(Ctx* ctx, qd_ham* const* hams, int ninst) {
  std::vector<BunJob> jobs;
  std::vector<qd_ham*> done;
  for (int i = 0; i < ninst; ++i) {
    qd_ham* H = hams[i];
    if (H->bun_checked || std::find(done.begin(), done.end(), H) != done.end()) continue;
    H->bun_d.alloc(H->dim + 4);  // e_r, then c at [dim], the flag's bits at [dim + 1]
    float* c = H->bun_d.p + H->dim;
    jobs.push_back(BunJob{H->dim, H->rowptr.p, H->colidx.p, H->vals_f.p, reinterpret_cast<int*>(c + 1), c,
                          H->bun_d.p});
    done.push_back(H);
  }
  if (jobs.empty()) return;
  DBuf<BunJob> dj(jobs.size());
  QD_CUDA(cudaMemcpyAsync(dj.p, jobs.data(), jobs.size() * sizeof(BunJob), cudaMemcpyHostToDevice, ctx->stream));
  for (size_t j0 = 0; j0 < jobs.size(); j0 += 65535) {
    const unsigned cnt = (unsigned)std::min<size_t>(65535, jobs.size() - j0);
    bun_check_kernel<<<cnt, 512, 0, ctx->stream>>>(dj.p + j0);
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
  }
  QD_CUDA(cudaStreamSynchronize(ctx->stream));  // dj is freed on return
  for (qd_ham* H : done) H->bun_checked = true;
}

// ---------------------------------------------------------------- cluster sums
// A barrier over the instance's CTAs (the block for C == 1).
template <int C>
__device__ __forceinline__ void inst_sync() {
  if constexpr (C > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// The instance total of a block total: every CTA adds the C partials in rank
// order from distributed shared memory.  Double-buffered: a buffer is written
// again only two sums later, after every CTA has passed the barrier between.
template <int C>
__device__ double inst_sum(double block_total, BlockScratch& S, int& buf) {
  if constexpr (C == 1) {
    return block_total;
  } else {
    cg::cluster_group cl = cg::this_cluster();
    if (threadIdx.x == 0) S.xp[buf] = block_total;
    cl.sync();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int r = 0; r < C; ++r) t += *cl.map_shared_rank(&S.xp[buf], r);
      S.bc[buf] = t;
    }
    __syncthreads();
    const double t = S.bc[buf];
    buf ^= 1;
    return t;
  }
}

// Lowest eigenpair of tridiag(d, e) (n <= kBatchMaxSteps), by the whole block: the eigenvalue by bisection
// (128 points a round, a warp on each SM quarter: is any leading minor of T - x not positive?), the vector by
// three steps of inverse iteration with partial pivoting (the reorthogonalised Lanczos matrix has no spurious
// copies).  Eigenvalues by QL and the same iteration on one thread took 5 ms at n = 80, FP64 instructions
// taking 72 cycles each.  A matrix that is not finite has NaN for its eigenvalue.
constexpr int kTriWork = kBatchMaxSteps + 2;
__device__ double block_tridiag_lowest(int n, const double* d, const double* e, double* y, BlockScratch& S) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  double* work = reinterpret_cast<double*>(S.wt);  // the tile of w is free
  static_assert(sizeof(float) * kWTile >= 7 * sizeof(double) * kTriWork, "scratch");
  double *dl = work, *dd = dl + kTriWork, *du = dd + kTriWork, *du2 = du + kTriWork, *rd = du2 + kTriWork,
         *e2 = rd + kTriWork;
  int* piv = reinterpret_cast<int*>(e2 + kTriWork);
  if (warp == 0) {
    double glo = 1e300, dmin = 1e300;
    bool bad = false;  // fmin drops a NaN
    for (int i = lane; i < n; i += 32) {
      const double el = i > 0 ? fabs(e[i - 1]) : 0.0, er = i + 1 < n ? fabs(e[i]) : 0.0;
      bad |= !isfinite(d[i]) || !isfinite(er);
      glo = fmin(glo, d[i] - (el + er));
      dmin = fmin(dmin, d[i]);
      e2[i] = er * er;
    }
    for (int o = 16; o > 0; o >>= 1) {
      glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
      dmin = fmin(dmin, __shfl_xor_sync(0xffffffffu, dmin, o));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {  // the lowest eigenvalue is at most the least diagonal element
      const double nan = __longlong_as_double(0x7ff8000000000000ll);
      S.ga = bad ? nan : glo - 1e-15 * fabs(glo);
      S.gb = bad ? nan : dmin;
    }
  }
  __syncthreads();
  for (int round = 0; round < 9; ++round) {  // 128^9 = 2^63
    const double a = S.ga, b = S.gb;
    bool has = true;
    if (threadIdx.x < 127) {
      const double x = fma(b - a, (double)(threadIdx.x + 1) * 0.0078125, a);
      double p0 = 1.0, p1 = d[0] - x;
      has = !(p1 > 0.0);
      for (int i = 1; i < n; ++i) {
        const double p2 = fma(d[i] - x, p1, -e2[i - 1] * p0);
        has |= !(p2 > 0.0);
        p0 = p1;
        p1 = p2;
        if ((i & 3) == 0) {  // p1 back to [1, 2), p0 with it
          const int sh = ((__double2hiint(p1) >> 20) & 0x7ff) - 1023, e0 = (__double2hiint(p0) >> 20) & 0x7ff;
          p0 = e0 - sh > 0 && e0 - sh < 2047 ? __hiloint2double(__double2hiint(p0) - sh * (1 << 20), __double2loint(p0))
                                             : 0.0;
          p1 = __hiloint2double(__double2hiint(p1) - sh * (1 << 20), __double2loint(p1));
        }
      }
    }
    if (warp < 4) {
      const unsigned m = __ballot_sync(0xffffffffu, has);
      if (lane == 0) S.gm[warp] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;  // the first point with an eigenvalue below it (the last, b, at least)
      for (; t < 127 && !((S.gm[t >> 5] >> (t & 31)) & 1u); t = (S.gm[t >> 5] >> (t & 31)) ? t + 1 : (t | 31) + 1) {
      }
      if (t < 127) S.gb = fma(b - a, (double)(t + 1) * 0.0078125, a);
      if (t > 0) S.ga = fma(b - a, (double)t * 0.0078125, a);
    }
    __syncthreads();
  }
  const double lam = S.gb;
  // (T - sigma I) y = b, sigma just below lam; Gaussian elimination with partial pivoting on the
  // tridiagonal band (three diagonals + fill-in), factored once
  if (warp == 0) {
    const double sigma = lam - 1e-10 * fmax(fabs(lam), 1.0);
    for (int i = lane; i < n; i += 32) {
      dd[i] = d[i] - sigma;
      du[i] = dl[i] = (i + 1 < n) ? e[i] : 0.0;
      du2[i] = 0.0;
      y[i] = 1.0;
    }
    __syncwarp();
    if (lane == 0) {
      for (int i = 0; i < n - 1; ++i) {
        if (fabs(dd[i]) >= fabs(dl[i])) {
          piv[i] = i;
          const double f = (dd[i] != 0.0) ? dl[i] / dd[i] : 0.0;
          dl[i] = f;
          dd[i + 1] -= f * du[i];
        } else {
          piv[i] = i + 1;
          const double f = dd[i] / dl[i];
          dd[i] = dl[i];
          dl[i] = f;
          const double t = du[i];
          du[i] = dd[i + 1];
          dd[i + 1] = t - f * dd[i + 1];
          if (i < n - 2) {
            du2[i] = du[i + 1];
            du[i + 1] = -f * du[i + 1];
          }
        }
      }
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) rd[i] = 1.0 / ((dd[i] != 0.0) ? dd[i] : 1e-300);
    __syncwarp();
    for (int it = 0; it < 3; ++it) {
      if (lane == 0) {  // solve L U x = P b
        double yi = y[0];
        for (int i = 0; i < n - 1; ++i) {
          const double yn = y[i + 1];
          if (piv[i] == i) {
            y[i] = yi;
            yi = yn - dl[i] * yi;
          } else {
            y[i] = yn;
            yi = yi - dl[i] * yn;
          }
        }
        double y1 = 0.0, y2 = 0.0;  // y[i + 1], y[i + 2]
        for (int i = n - 1; i >= 0; --i) {
          double v = (i == n - 1) ? yi : y[i];
          v = (v - du[i] * y1 - du2[i] * y2) * rd[i];
          y[i] = v;
          y2 = y1;
          y1 = v;
        }
      }
      __syncwarp();
      double nr = 0.0;
      for (int i = lane; i < n; i += 32) nr += y[i] * y[i];
      for (int o = 16; o > 0; o >>= 1) nr += __shfl_xor_sync(0xffffffffu, nr, o);
      nr = 1.0 / sqrt(nr);
      for (int i = lane; i < n; i += 32) y[i] *= nr;
      __syncwarp();
    }
  }
  __syncthreads();
  return lam;
}

// float4s on their way to a thread's own slots of a ring, kBatchRing deep: rows of `per` blocks of 32 float4s,
// `left` of them, `stride` floats apart; lane l takes float4 l of each block, zeros from float4 `len` of a row on.
constexpr int kBatchRing = 8;
constexpr size_t kBatchRingBytes = (size_t)kBatchThreads * kBatchRing * sizeof(float4);
struct BatchStream {
  const float* p;  // the row
  int64_t stride;
  unsigned base, in, out;
  int per, b, left, len;
  __device__ __forceinline__ void fetch() {
    if (left > 0) {
      const int i = 32 * b + (int)(threadIdx.x & 31);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(base + in), "l"(p + 4 * (i < len ? i : 0)),
                   "r"(i < len ? 16 : 0)
                   : "memory");
      if (++b == per) {
        b = 0;
        p += stride;
        --left;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    in = (in + 16 * kBatchThreads) & (unsigned)(kBatchRingBytes - 1);
  }
  __device__ __forceinline__ void begin(const float* rows, int64_t st, int count, int blocks, int length, float4* slot) {
    p = rows;
    stride = st;
    left = count;
    per = blocks;
    len = length;
    b = 0;
    base = (unsigned)__cvta_generic_to_shared(slot);
    in = out = 0;
#pragma unroll
    for (int i = 0; i < kBatchRing - 1; ++i) fetch();
  }
  __device__ __forceinline__ float4 next() {
    fetch();  // into the slot that the float4 before left
    asm volatile("cp.async.wait_group %0;" ::"n"(kBatchRing - 1) : "memory");
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(base + out));
    out = (out + 16 * kBatchThreads) & (unsigned)(kBatchRingBytes - 1);
    return v;
  }
};

template <int C>
__global__ void __launch_bounds__(kBatchThreads, 2) batch_lanczos_kernel(const BatchInst* __restrict__ list, int ninst,
                                                                     unsigned* counter) {
  __shared__ BlockScratch S;
  extern __shared__ __align__(16) float4 batch_ring[];  // C > 1
  int rank = 0;
  if constexpr (C > 1) rank = (int)cg::this_cluster().block_rank();
  int buf = 0, hbuf = 0;
  for (;;) {
    if (rank == 0 && threadIdx.x == 0) S.idx = (int)atomicAdd(counter, 1u);
    inst_sync<C>();
    int idx;
    if constexpr (C > 1) idx = *cg::this_cluster().map_shared_rank(&S.idx, 0);
    else idx = S.idx;
    inst_sync<C>();
    if (idx >= ninst) return;  // the same index in every CTA of the cluster
    const BatchInst I = list[idx];
    const unsigned long long t_start = batch_clock_ns();
    const int64_t n = I.dim;
    // this CTA's rows: a slice of 32-element multiples (the whole vector for C == 1)
    const int64_t per = ((n + C - 1) / C + 31) / 32 * 32;
    const int64_t lo = std::min<int64_t>(n, (int64_t)rank * per), hi = std::min<int64_t>(n, lo + per);
    float* V = I.V;
    float* w = I.w;
    const bool uni = I.uniform && __ldg(I.uniform) == 1;
    // v_0 = v0 / ||v0||
    const double nrm0 = sqrt(inst_sum<C>(block_dot(I.v0, I.v0, lo, hi, S), S, buf));
    const float inv0 = (float)(1.0 / nrm0);
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) V[i] = I.v0[i] * inv0;
    // the last float4s of the vectors are read whole: zeros past the end
    const int64_t pad = (hi == n && lo < n) ? I.ld : hi;
    for (int64_t i = hi + threadIdx.x; i < pad; i += blockDim.x) V[i] = 0.f;
    // so few rows a thread that none of its FP32 partials spans more than kChunk elements
    const bool few = per <= (int64_t)(kChunk - 4) * kBatchThreads;
    if (threadIdx.x == 0) {
      S.stop = 0;
      S.scl[0] = 1.0;
    }
    inst_sync<C>();
    int act = I.steps;
    // The basis is stored unnormalised: vector j is scl[j] V[j].  A step forms y = H V[k-1]
    // with the three inner products of the reference's local orthogonalisation, folds
    // u = y - c2 V[k-2] - c1 V[k-1] into the first read of the Gram-Schmidt pass, and
    // writes the orthogonalised u, times a power of two near 1 / ||u||, to V[k] itself.
    for (int k = 1; k <= I.steps; ++k) {
      const float* v1 = V + (int64_t)(k - 1) * I.ld;
      const float* v2 = (k >= 2) ? V + (int64_t)(k - 2) * I.ld : nullptr;
      ProdDots pd;
      if (uni) block_spmv_f32<true>(I, v1, v2, w, lo, hi, pd);
      else block_spmv_f32<false>(I, v1, v2, w, lo, hi, pd);
      // <V2, y>, <V1, y>, <V1, V2> of the instance; the scalars of the step on one thread
      double* d3 = S.xp3[buf];
      if (few) {
        const float f3[3] = {pd.fa, pd.fb, pd.fc};
        block_sum_f<3>(f3, S, d3);
      } else {
        pd.flush();
        double t3[3] = {pd.da, pd.db, pd.dc};
        block_sum_all3(t3, S);
        if (threadIdx.x < 3) d3[threadIdx.x] = threadIdx.x == 0 ? t3[0] : threadIdx.x == 1 ? t3[1] : t3[2];
      }
      inst_sync<C>();
      if (threadIdx.x < 32) {
        double t = 0.0;
        if constexpr (C > 1) {
          if (threadIdx.x < 3)
#pragma unroll 1
            for (int r = 0; r < C; ++r) t += cg::this_cluster().map_shared_rank(&S.xp3[buf][0], r)[threadIdx.x];
        } else {
          if (threadIdx.x < 3) t = d3[threadIdx.x];
        }
        const double ta = __shfl_sync(0xffffffffu, t, 0), tb = __shfl_sync(0xffffffffu, t, 1),
                     tc = __shfl_sync(0xffffffffu, t, 2);
        // bp = <v2, w>, al = <v1, w - bp v2> in the true (normalised) vectors
        const double s1 = S.scl[k - 1], s2 = (k >= 2) ? S.scl[k - 2] : 0.0;
        const double bp = v2 ? s2 * s1 * ta : 0.0;
        const double al = s1 * (s1 * tb - bp * s2 * tc);
        if (threadIdx.x == 0) {
          S.bp = bp;
          S.al = al;
          S.c1 = (float)al;
          S.c2 = (float)(s2 * s2 * ta);
        }
      }
      buf ^= 1;
      __syncthreads();
      const float c2 = v2 ? S.c2 : 0.f, c1 = S.c1;
      // one full Gram-Schmidt pass against v_0 .. v_{k-1}
      double nacc = 0.0;  // this thread's share of the stored V[k]'s squared norm, but for its last FP32 partial
      float nshare = 0.f;
      float tk = 1.f;     // the power of two V[k] is stored with
      {
        const int64_t q0 = lo >> 2, q1 = hi >> 2;
        double* part = (C > 1) ? S.hp[hbuf] : S.h;
        // g_j = <V_j, u>, j < k, and ||u||^2 in part[k]: u formed tile by tile into shared
        // memory (and written back for the update), a warp per basis vector within a
        // tile, eight float4 of V_j in flight per lane
        {
          const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
          float uf = 0.f;     // ||u||^2, for its exponent alone
          double gacc = 0.0;  // lane i: vector warp + nw i
          for (int64_t t0 = lo; t0 < hi; t0 += kWTile) {
            const int tn = (int)std::min<int64_t>(hi - t0, kWTile);
            const int nq = tn >> 2, nq4 = (tn + 3) >> 2;  // t0 is a multiple of 32: float4-aligned
            __syncthreads();  // the previous tile's readers are done
            for (int i = threadIdx.x; i < nq; i += blockDim.x) {
              float4 u = reinterpret_cast<const float4*>(w + t0)[i];
              const float4 p1 = reinterpret_cast<const float4*>(v1 + t0)[i];
              if (v2) {
                const float4 p2 = reinterpret_cast<const float4*>(v2 + t0)[i];
                u.x = fmaf(-c2, p2.x, u.x);
                u.y = fmaf(-c2, p2.y, u.y);
                u.z = fmaf(-c2, p2.z, u.z);
                u.w = fmaf(-c2, p2.w, u.w);
              }
              u.x = fmaf(-c1, p1.x, u.x);
              u.y = fmaf(-c1, p1.y, u.y);
              u.z = fmaf(-c1, p1.z, u.z);
              u.w = fmaf(-c1, p1.w, u.w);
              reinterpret_cast<float4*>(S.wt)[i] = u;
              reinterpret_cast<float4*>(w + t0)[i] = u;
              uf = fmaf(u.x, u.x, uf);
              uf = fmaf(u.y, u.y, uf);
              uf = fmaf(u.z, u.z, uf);
              uf = fmaf(u.w, u.w, uf);
            }
            for (int i = (nq << 2) + threadIdx.x; i < kWTile; i += blockDim.x) {  // the end of the rows, then zeros
              float u = 0.f;
              if (i < tn) {
                u = w[t0 + i];
                if (v2) u = fmaf(-c2, v2[t0 + i], u);
                u = fmaf(-c1, v1[t0 + i], u);
                w[t0 + i] = u;
                uf = fmaf(u, u, uf);
              }
              S.wt[i] = u;
            }
            __syncthreads();
            const float4* ws4 = reinterpret_cast<const float4*>(S.wt);
            long long qs = 0;
            unsigned es = 1;
            int mine = 0;
            // clusters: the vectors' float4s of the tile come through a ring of asynchronous copies that each thread
            // reads back itself, vector after vector, kBatchRing of them in flight
            const int nc = (nq4 + 127) >> 7;
            BatchStream ring;
            if constexpr (C > 1)
              ring.begin(V + (int64_t)warp * I.ld + t0, (int64_t)nw * I.ld, warp < k ? (k - warp + nw - 1) / nw : 0, 4 * nc,
                         nq4, batch_ring + threadIdx.x);
            for (int j = warp; j < k; j += nw, ++mine) {
              float c[kWTile / 512];  // FP32 over 16 elements
              unsigned mag = 0;
              if constexpr (C > 1) {
#pragma unroll
                for (int h = 0; h < kWTile / 512; ++h) {
                  c[h] = 0.f;
                  if (h < nc) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                      const float4 x = ring.next();
                      const float4 y = ws4[128 * h + 32 * q + lane];
                      c[h] = fmaf(x.x, y.x, c[h]);
                      c[h] = fmaf(x.y, y.y, c[h]);
                      c[h] = fmaf(x.z, y.z, c[h]);
                      c[h] = fmaf(x.w, y.w, c[h]);
                    }
                    mag = max(mag, f_mag(c[h]));
                  }
                }
              } else {
                const float4* vj4 = reinterpret_cast<const float4*>(V + (int64_t)j * I.ld + t0);
#pragma unroll
                for (int h = 0; h < kWTile / 1024; ++h) {
                  c[2 * h] = c[2 * h + 1] = 0.f;
                  if (256 * h < nq4) {
                    float4 x[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                      const int i = 256 * h + 32 * q + lane;
                      x[q] = i < nq4 ? vj4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                      const float4 y = ws4[256 * h + 32 * q + lane];
                      float acc = c[2 * h + (q >> 2)];
                      acc = fmaf(x[q].x, y.x, acc);
                      acc = fmaf(x[q].y, y.y, acc);
                      acc = fmaf(x[q].z, y.z, acc);
                      acc = fmaf(x[q].w, y.w, acc);
                      c[2 * h + (q >> 2)] = acc;
                    }
                    mag = max(mag, max(f_mag(c[2 * h]), f_mag(c[2 * h + 1])));
                  }
                }
              }
              const unsigned e = f_top(mag);
              long long t = 0;
#pragma unroll
              for (int h = 0; h < kWTile / 512; ++h)
                if (h < nc) t += f_fix(c[h], e);
              t = f_warp_sum(t);
              if (lane == mine) {
                qs = t;
                es = e;
              }
            }
            gacc = fma((double)qs, f_unit(es), gacc);  // tile by tile, in order: the same bits in every run
          }
          if (warp + nw * lane < k) part[warp + nw * lane] = gacc;
          // ||u||^2 of this CTA's rows into part[k]
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) uf += __shfl_xor_sync(0xffffffffu, uf, o);
          if (lane == 0) S.fu[warp] = uf;
          __syncthreads();
          if (threadIdx.x == 0) {
            float t = 0.f;
            for (int q = 0; q < nw; ++q) t += S.fu[q];
            part[k] = (double)t;
          }
        }
        if constexpr (C > 1) {  // the coefficients of the whole vector, the same bits in every CTA
          cg::cluster_group cl = cg::this_cluster();
          cl.sync();
          for (int j = threadIdx.x; j <= k; j += blockDim.x) {
            double t = 0.0;
#pragma unroll 1
            for (int r = 0; r < C; ++r) t += *cl.map_shared_rank(&S.hp[hbuf][j], r);
            S.h[j] = t;
          }
          hbuf ^= 1;
        }
        __syncthreads();
        // update coefficients of the stored vectors: u' = u - sum_j scl[j]^2 g_j V[j]
        for (int j = threadIdx.x; j < k; j += blockDim.x) S.cf[j] = -(float)(S.scl[j] * S.scl[j] * S.h[j]);
        {
          // tk ||u|| in [0.5, 1), from the exponent of ||u||^2
          const unsigned hw = (unsigned)__double2hiint(S.h[k]);
          const int e2 = (int)(hw >> 20) - 1022;
          if (hw >= 0x00100000u && hw < 0x7ff00000u) tk = ldexpf(1.f, -((e2 + 1) >> 1));
        }
        __syncthreads();
        // V[k] = tk (u - sum_j c_j V[j]), and its squared norm (FP32 over at most kChunk elements)
        const float4* wm4 = reinterpret_cast<const float4*>(w);
        float4* vk4 = reinterpret_cast<float4*>(V + (int64_t)k * I.ld);
        const int64_t bs = blockDim.x;
        float nf = 0.f;
        int ncnt = 0;
        int64_t i = q0 + threadIdx.x;
        for (; i + bs < q1; i += 2 * bs) {  // two float4 of u per thread: two independent chains
          float4 x = wm4[i], u = wm4[i + bs];
#pragma unroll 4
          for (int j = 0; j < k; ++j) {
            const float c = S.cf[j];
            const float4* vj4 = reinterpret_cast<const float4*>(V + (int64_t)j * I.ld);
            const float4 y = vj4[i], z = vj4[i + bs];
            x.x = fmaf(c, y.x, x.x);
            x.y = fmaf(c, y.y, x.y);
            x.z = fmaf(c, y.z, x.z);
            x.w = fmaf(c, y.w, x.w);
            u.x = fmaf(c, z.x, u.x);
            u.y = fmaf(c, z.y, u.y);
            u.z = fmaf(c, z.z, u.z);
            u.w = fmaf(c, z.w, u.w);
          }
          x = make_float4(x.x * tk, x.y * tk, x.z * tk, x.w * tk);
          u = make_float4(u.x * tk, u.y * tk, u.z * tk, u.w * tk);
          vk4[i] = x;
          vk4[i + bs] = u;
          nf = fmaf(x.x, x.x, nf);
          nf = fmaf(x.y, x.y, nf);
          nf = fmaf(x.z, x.z, nf);
          nf = fmaf(x.w, x.w, nf);
          nf = fmaf(u.x, u.x, nf);
          nf = fmaf(u.y, u.y, nf);
          nf = fmaf(u.z, u.z, nf);
          nf = fmaf(u.w, u.w, nf);
          if (!few && ++ncnt == kChunk / 8) {
            nacc += (double)nf;
            nf = 0.f;
            ncnt = 0;
          }
        }
        if (!few) {
          nacc += (double)nf;
          nf = 0.f;
          ncnt = 0;
        }
        for (; i < q1; i += bs) {
          float4 x = wm4[i];
#pragma unroll 4
          for (int j = 0; j < k; ++j) {
            const float c = S.cf[j];
            const float4 y = reinterpret_cast<const float4*>(V + (int64_t)j * I.ld)[i];
            x.x = fmaf(c, y.x, x.x);
            x.y = fmaf(c, y.y, x.y);
            x.z = fmaf(c, y.z, x.z);
            x.w = fmaf(c, y.w, x.w);
          }
          x = make_float4(x.x * tk, x.y * tk, x.z * tk, x.w * tk);
          vk4[i] = x;
          nf = fmaf(x.x, x.x, nf);
          nf = fmaf(x.y, x.y, nf);
          nf = fmaf(x.z, x.z, nf);
          nf = fmaf(x.w, x.w, nf);
          if (!few && ++ncnt == kChunk / 4) {
            nacc += (double)nf;
            nf = 0.f;
            ncnt = 0;
          }
        }
        float* vk = V + (int64_t)k * I.ld;
        for (int64_t i = (q1 << 2) + threadIdx.x; i < hi; i += blockDim.x) {
          float wi = w[i];
          for (int j = 0; j < k; ++j) wi = fmaf(S.cf[j], V[(int64_t)j * I.ld + i], wi);
          wi *= tk;
          vk[i] = wi;
          nf = fmaf(wi, wi, nf);
        }
        for (int64_t i = hi + threadIdx.x; i < pad; i += blockDim.x) vk[i] = 0.f;
        nshare = nf;
      }
      // ||V[k]||^2 as stored; the barrier also completes V[k] for the next product
      if (few) {
        const float f1[1] = {nshare};
        block_sum_f<1>(f1, S, &S.xp[buf]);
      } else {
        const double t = block_sum_all(nacc + (double)nshare, S);
        if (threadIdx.x == 0) S.xp[buf] = t;
      }
      inst_sync<C>();
      if (threadIdx.x == 0) {
        double n2 = 0.0;
        if constexpr (C > 1) {
#pragma unroll 1
          for (int r = 0; r < C; ++r) n2 += *cg::this_cluster().map_shared_rank(&S.xp[buf], r);
        } else {
          n2 = S.xp[buf];
        }
        const double rs = rsqrt(n2), nst = n2 > 0.0 ? n2 * rs : n2;
        const double nr = S.scl[k - 1] * nst * (double)(1.f / tk);  // beta_k
        S.alpha[k] = S.al + S.scl[k - 1] * S.scl[k - 1] * S.h[k - 1];  // al + <v_{k-1}, u> in the true vectors
        S.beta[k] = nr;
        S.scl[k] = (nst > 0.0) ? rs : 0.0;
        // breakdown (sparse_algorithm.hpp:421): the reference's 1e-10, or the
        // FP32 resolution of the recurrence, or an exhausted space
        const double scale = fabs(S.al) + fabs(S.bp) + (k >= 2 ? S.beta[k - 1] : 0.0);
        if (nr < 1e-10 || nr < 1e-5 * scale || k >= n) S.stop = k;
      }
      buf ^= 1;
      __syncthreads();
      if (S.stop) {  // the same decision in every CTA of the cluster
        act = k;     // v_0 .. v_{k-1} span an invariant subspace: T_k is exact
        break;
      }
    }
    if (act < 1) act = 1;
    // lowest Ritz pair of tridiag(alpha_1..act, beta_1..act-1), the same in every CTA
    const double lam = block_tridiag_lowest(act, S.alpha + 1, S.beta + 1, S.y, S);
    if (rank == 0 && threadIdx.x == 0) {
      I.out[0] = lam;
      I.out[3] = act;
      I.out[4] = S.stop ? 1 : 0;
    }
    for (int k = threadIdx.x; k < act; k += blockDim.x) S.cf[k] = (float)(S.y[k] * S.scl[k]);
    __syncthreads();
    // Ritz vector psi = sum_k y_k v_k (FP32 storage)
    for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      float acc = 0.f;
#pragma unroll 8
      for (int k = 0; k < act; ++k) acc = fmaf(S.cf[k], V[(int64_t)k * I.ld + i], acc);
      I.psi[i] = acc;
    }
    inst_sync<C>();  // the refinement reads all of psi
    // FP64 refinement: Rayleigh quotient with the FP64 values
    double num = 0.0, den = 0.0;
    for (int64_t r = lo + threadIdx.x; r < hi; r += blockDim.x) {
      double hr = 0.0;
      for (int64_t e = I.rowptr[r]; e < I.rowptr[r + 1]; ++e) hr = fma(I.vals_d[e], (double)I.psi[I.colidx[e]], hr);
      const double pr = (double)I.psi[r];
      num = fma(pr, hr, num);
      den = fma(pr, pr, den);
    }
    num = inst_sum<C>(block_sum_all(num, S), S, buf);
    den = inst_sum<C>(block_sum_all(den, S), S, buf);
    if (rank == 0 && threadIdx.x == 0) {
      I.out[1] = num / den;
      I.out[2] = den;
      I.out[5] = (double)t_start;
      I.out[6] = (double)batch_clock_ns();
      I.out[7] = (double)C;
    }
    inst_sync<C>();
  }
}

// Launches kernel C over `count` instances of `list` with `grid` CTAs
// (clusters of C CTAs for C > 1).
template <int C>
static void launch_batch(Ctx* ctx, cudaStream_t stream, const BatchInst* list, int count, unsigned* counter,
                         int grid) {
  if (count <= 0) return;
  if constexpr (C > 1) allow_dynamic_smem(batch_lanczos_kernel<C>, ctx->device);
  if constexpr (C == 1) {
    batch_lanczos_kernel<1><<<grid, kBatchThreads, 0, stream>>>(list, count, counter);
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kBatchThreads);
    cfg.dynamicSmemBytes = kBatchRingBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    QD_CUDA(cudaLaunchKernelEx(&cfg, batch_lanczos_kernel<C>, list, count, counter));
  }
  QD_CHECK_LAUNCH();
  QD_LAUNCHED(ctx);
}

// Clusters of C CTAs the device keeps resident at once (0 if none).
template <int C>
static int resident_clusters(Ctx* ctx) {
  if (C == 1) return 2 * ctx->num_sms;
  static thread_local int cached = -1;
  if (cached >= 0) return cached;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(C * 2 * ctx->num_sms));
  cfg.blockDim = dim3(kBatchThreads);
  cfg.dynamicSmemBytes = kBatchRingBytes;
  allow_dynamic_smem(batch_lanczos_kernel<C>, ctx->device);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, batch_lanczos_kernel<C>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  cached = n;
  return n;
}

constexpr int kBatchSizes = 6;
static const int kBatchSize[kBatchSizes] = {1, 2, 3, 4, 6, 8};

template <typename F>
static void batch_size(int c, F&& f) {
  switch (c) {
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 8: f(std::integral_constant<int, 8>()); break;
    default: f(std::integral_constant<int, 1>()); break;
  }
}

// CTAs per instance.  While slots are free a call takes as long as its longest slice of rows, so the slices are
// as short as the device has CTA slots for, down to kBatchMinRows.  32 chains each of 14, 16 and 18 sites, 80
// steps: 19.4 ms on 1, 1 and 8 CTAs, 22.0 on 1, 4 and 4, 17.1 on 1, 2 and 6, which this takes; 32 of 16 sites
// 11.3, 8.5, 5.6 and 4.5 ms on 1, 2, 4 and 8.  A call with more instances than slots keeps 2 CTAs for dimensions
// from kClusterMinDim and one below: more instances side by side beat wider clusters there.
static std::vector<int> batch_widths(Ctx* ctx, qd_ham* const* hams, int ninst) {
  int most[kBatchSizes];
  for (int k = 0; k < kBatchSizes; ++k)
    batch_size(kBatchSize[k], [&](auto c) { most[k] = resident_clusters<decltype(c)::value>(ctx); });
  const int64_t slots = most[0];
  auto size_of = [&](int64_t dim, int64_t rows) {  // index of the least size with slices of at most `rows`
    if (dim < kBatchSplitMinDim) return 0;
    int k = (dim >= kClusterMinDim && most[1] > 0) ? 1 : 0;
    while (k + 1 < kBatchSizes && dim > rows * kBatchSize[k]) ++k;
    while (k > 0 && most[k] < 1) --k;
    return k;
  };
  auto fits = [&](int64_t rows) {
    int64_t used = 0, n[kBatchSizes] = {};
    for (int i = 0; i < ninst; ++i) {
      const int k = size_of(hams[i]->dim, rows);
      used += kBatchSize[k];
      ++n[k];
    }
    for (int k = 0; k < kBatchSizes; ++k)
      if (n[k] > most[k]) return false;
    return used <= slots;
  };
  std::vector<int64_t> cand;
  for (int i = 0; i < ninst; ++i)
    for (int k = 0; k < kBatchSizes; ++k)
      cand.push_back(std::max<int64_t>(ceil_div(hams[i]->dim, kBatchSize[k]), kBatchMinRows));
  std::sort(cand.begin(), cand.end());
  cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
  size_t lo = 0, hi = cand.size() - 1;  // the least slice that fits, else the longest
  while (lo < hi) {
    const size_t mid = (lo + hi) / 2;
    if (fits(cand[mid])) hi = mid;
    else lo = mid + 1;
  }
  std::vector<int> width(ninst);
  for (int i = 0; i < ninst; ++i) width[i] = kBatchSize[size_of(hams[i]->dim, cand[lo])];
  return width;
}

void batch_lanczos(Ctx* ctx, qd_ham* const* hams, const double* const* v0s, int ninst, int steps, double* out) {
  QD_REQUIRE(ninst >= 1, QD_ERR_INVALID, "empty batch");
  QD_REQUIRE(steps >= 1 && steps <= kBatchMaxSteps, QD_ERR_INVALID, "steps must be in 1..%d", kBatchMaxSteps);
  std::vector<int> order(ninst);
  std::iota(order.begin(), order.end(), 0);
  for (int i = 0; i < ninst; ++i) {
    QD_REQUIRE(hams[i] && v0s[i], QD_ERR_INVALID, "instance %d: null argument", i);
    QD_REQUIRE(hams[i]->flags & QD_HAM_REAL, QD_ERR_UNSUPPORTED,
               "instance %d: the batched mixed-precision solver needs a real Hamiltonian", i);
    QD_REQUIRE(hams[i]->ctx == ctx, QD_ERR_INVALID, "instance %d: Hamiltonian of another context", i);
    QD_REQUIRE(hams[i]->dim >= 1, QD_ERR_INVALID, "instance %d: the sector has no state", i);
  }
  // QD_BATCH_UNIFORM=0 keeps the valued product for every instance
  const char* uenv = std::getenv("QD_BATCH_UNIFORM");
  const bool uniform_ok = !(uenv && std::strcmp(uenv, "0") == 0);
  if (uniform_ok) check_uniform(ctx, hams, ninst);
  // wider clusters first, each size longest first
  const std::vector<int> width = batch_widths(ctx, hams, ninst);
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return width[a] != width[b] ? width[a] > width[b] : hams[a]->nnz > hams[b]->nnz;
  });
  // one arena for every instance's basis, work vector and Ritz vector
  std::vector<int64_t> off_V(ninst), off_w(ninst), off_psi(ninst);
  int64_t total = 0;
  for (int i = 0; i < ninst; ++i) {
    const int64_t ld = (hams[i]->dim + 31) / 32 * 32;
    off_V[i] = total;
    total += (int64_t)(steps + 1) * ld;
    off_w[i] = total;
    total += ld;
    off_psi[i] = total;
    total += ld;
  }
  DBuf<float> arena(total);
  DBuf<double> dout((size_t)ninst * 8);
  QD_CUDA(cudaMemsetAsync(dout.p, 0, dout.bytes(), ctx->stream));
  // the start vectors, in FP32, in one copy
  int64_t v0_total = 0;
  for (int i = 0; i < ninst; ++i) v0_total += (hams[i]->dim + 31) / 32 * 32;
  std::unique_ptr<float[]> h32(new float[(size_t)std::max<int64_t>(v0_total, 1)]);
  DBuf<float> v0buf(v0_total);
  std::vector<int64_t> off_h(ninst);
  for (int i = 0; i < ninst; ++i) off_h[i] = (i == 0) ? 0 : off_h[i - 1] + (hams[i - 1]->dim + 31) / 32 * 32;
  {
    // FP64 -> FP32 on up to eight host threads, instances dealt round-robin (padding zeroed)
    const int nt = (int)std::max<int64_t>(1, std::min<int64_t>(8, v0_total >> 20));
    auto convert = [&](int t) {
      for (int i = t; i < ninst; i += nt) {
        const int64_t d = hams[i]->dim, ld = (d + 31) / 32 * 32;
        float* o = h32.get() + off_h[i];
        const double* v = v0s[i];
        for (int64_t q = 0; q < d; ++q) o[q] = (float)v[q];
        for (int64_t q = d; q < ld; ++q) o[q] = 0.f;
      }
    };
    std::vector<std::thread> pool;
    for (int t = 1; t < nt; ++t) pool.emplace_back(convert, t);
    convert(0);
    for (auto& th : pool) th.join();
  }
  QD_CUDA(cudaMemcpyAsync(v0buf.p, h32.get(), (size_t)v0_total * sizeof(float), cudaMemcpyHostToDevice,
                          ctx->stream));
  // the work list, one launch per cluster size
  std::vector<BatchInst> list(ninst);
  for (int q = 0; q < ninst; ++q) {
    const int i = order[q];
    const qd_ham* H = hams[i];
    BatchInst& I = list[q];
    std::memset(&I, 0, sizeof(I));
    I.dim = H->dim;
    I.steps = steps;
    I.ld = (H->dim + 31) / 32 * 32;
    I.rowptr = H->rowptr.p;
    I.colidx = H->colidx.p;
    I.vals_f = H->vals_f.p;
    I.uniform = uniform_ok ? reinterpret_cast<const int*>(H->bun_d.p + H->dim + 1) : nullptr;
    I.coff = H->bun_d.p + H->dim;
    I.diag_f = H->bun_d.p;
    I.vals_d = H->vals_r.p;
    I.v0 = v0buf.p + off_h[i];
    I.V = arena.p + off_V[i];
    I.w = arena.p + off_w[i];
    I.psi = arena.p + off_psi[i];
    I.out = dout.p + (size_t)i * 8;
  }
  DBuf<BatchInst> dlist(ninst);
  QD_CUDA(cudaMemcpyAsync(dlist.p, list.data(), ninst * sizeof(BatchInst), cudaMemcpyHostToDevice, ctx->stream));
  DBuf<unsigned> counter(kBatchSizes);
  QD_CUDA(cudaMemsetAsync(counter.p, 0, counter.bytes(), ctx->stream));
  // The widest clusters go first, each size but the last on a high-priority side stream: the clusters are
  // placed before the narrower ones and the single CTAs, which take the SM slots they leave (and free at the
  // end).  Every instance is computed by its own CTAs in a fixed order, so the results do not depend on the
  // overlap.
  struct Side {
    cudaStream_t s = nullptr;
    cudaEvent_t done = nullptr;
    ~Side() {
      if (done) cudaEventDestroy(done);
      if (s) {
        cudaStreamSynchronize(s);  // after an error its kernel may still run, and the buffers are given back next
        cudaStreamDestroy(s);
      }
    }
  } side[kBatchSizes];
  struct InEvent {
    cudaEvent_t e = nullptr;
    ~InEvent() {
      if (e) cudaEventDestroy(e);
    }
  } in;
  const bool timing = std::getenv("QD_TIMING") != nullptr;
  if (timing) QD_CUDA(cudaEventRecord(ctx->events[12], ctx->stream));
  std::string plan;
  for (int q0 = 0, li = 0; q0 < ninst; ++li) {
    const int c = width[order[q0]];
    int q1 = q0;
    while (q1 < ninst && width[order[q1]] == c) ++q1;
    cudaStream_t st = ctx->stream;
    if (q1 < ninst) {  // not the last size
      int least = 0, greatest = 0;
      if (!in.e) {
        QD_CUDA(cudaEventCreateWithFlags(&in.e, cudaEventDisableTiming));
        QD_CUDA(cudaEventRecord(in.e, ctx->stream));  // the list, the start vectors and the counters are in place
      }
      QD_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
      QD_CUDA(cudaStreamCreateWithPriority(&side[li].s, cudaStreamNonBlocking, greatest));
      QD_CUDA(cudaEventCreateWithFlags(&side[li].done, cudaEventDisableTiming));
      QD_CUDA(cudaStreamWaitEvent(side[li].s, in.e, 0));
      st = side[li].s;
    }
    batch_size(c, [&](auto k) {
      constexpr int C = decltype(k)::value;
      launch_batch<C>(ctx, st, dlist.p + q0, q1 - q0, counter.p + li, C * std::min(q1 - q0, resident_clusters<C>(ctx)));
    });
    if (side[li].s) QD_CUDA(cudaEventRecord(side[li].done, side[li].s));
    if (timing) plan += " " + std::to_string(q1 - q0) + " x " + std::to_string(c);
    q0 = q1;
  }
  for (Side& sd : side)
    if (sd.s) QD_CUDA(cudaStreamWaitEvent(ctx->stream, sd.done, 0));
  if (timing) QD_CUDA(cudaEventRecord(ctx->events[13], ctx->stream));
  QD_CUDA(cudaMemcpyAsync(out, dout.p, (size_t)ninst * 8 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  if (timing) {
    float a = 0.f;
    QD_CUDA(cudaEventElapsedTime(&a, ctx->events[12], ctx->events[13]));
    std::fprintf(stderr, "[qd timing] batch: instances x CTAs:%s: %.3f ms\n", plan.c_str(), a);
  }
}

}  // namespace qd
