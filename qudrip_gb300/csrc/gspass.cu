// gspass.cu -- classical Gram-Schmidt, twice, over a Krylov basis in memory: the
// step of expandBasis<0> (sparse_algorithm.hpp:372-393) for sectors whose rows do
// not fit the persistent recurrence (arnres.cu) and for served requests.
//
// In FP64 the projections and their removal are bound by FP64 issue (76 cycles
// a warp instruction and SM quarter): at 705,432 rows and 16 columns they took
// 94 and 44 us a launch where the vectors' bytes take 14.  The projections run
// on 55-bit integers here (qvec.cuh), with one scale per vector and tile of rows:
//   dots    c_j = <V_j, w>: a warp owns a tile, holds its rows of w quantised in
//           registers and passes over the vectors, four vectors' totals to one
//           warp sum; lane j then keeps vector j's total in FP64, one
//           conversion per tile.
//   update  w -= sum_j c_j V_j in FP64, on the vectors themselves: what is stored
//           keeps the relative accuracy of each row, also where a tile's largest
//           is orders of magnitude above it (a localised state).
// A vector's rows come through a ring of asynchronous copies that each thread
// reads back itself, no barrier.
// Pass 1 is dots; its update runs in the same launch as pass 2's dots, and pass
// 2's update also forms the norm (of the quantised rows, so in integers as
// well).  A step is four launches with the product instead of seven, and reads
// the basis three times instead of four.  For a Hermitian H the exact
// projections of pass 1 vanish but for the last two vectors, <v_{k-1}, H
// v_{k-1}>, whose sum the product's launch begins, and the last norm: three
// launches, twice through the basis.  The vectors stay unnormalised with their
// scales, which saves a pass; the product's own scale applies them.
//
// Measured (GB300), two steps of the recurrence and exponential, Hermitian:
// 705,432 rows, m = 16: 10.4 -> 4.87 ms; 184,756 rows, m = 30: 10.2 -> 4.6 ms;
// 2,704,156 rows, m = 30: 94.8 -> 37.8 ms (4.25, 3.7 and 29.5 with the removal on
// the integer copies).  At 705,432 rows a step's product is 62 us (bound by FP64
// issue and its gathers), the dots 52 us at 12 vectors, bound by the latencies
// between a warp's integer instructions (a third of the issue slots) with HBM at
// half its rate (more warps, deeper rings and smaller tiles measured the same),
// the update 70, bound by FP64 issue.
#include <algorithm>

#include "gspass.cuh"
#include "krylov.cuh"
#include "qvec.cuh"
#include "spmv.cuh"

namespace qd {

constexpr int kGsThreads = 512;
constexpr int kGsWarps = kGsThreads / 32;
constexpr int kGsChunk = 32;  // vectors per launch of the dots: one per lane
constexpr int kGsRing = 8;   // rows a thread holds in its ring
constexpr size_t kGsSmem = (size_t)kGsThreads * kGsRing * sizeof(int4);

struct GsArgs {
  int64_t n, ld, ntiles;
  const cplx* V;
  const int4* Vq;
  double* u;
  const cplx* src;
  cplx* dst;
  // update: coefficients cu[j] on vectors j0 <= j < j1
  const cplx* cu;
  int j0, j1;
  // dots with vectors d0 .. d0 + J - 1
  int d0, J;
  cplx* cd;
  cplx* hcol;
  bool hadd;  // hcol[j] holds the first pass's value
  // first pass of a Hermitian step: ndots shares of <V_{step-1}, w> (none: cu and hcol hold the first pass)
  double* dots;
  int64_t ndots;
  // norm: the result is vector k
  int k;
  cplx* Vk;
  int4* Vqk;
  double* scl;
  double* nrm;
  double* partials;
  unsigned* ticket;
  int* stop;
  int step;
};

__device__ __forceinline__ bool gs_stopped(const GsArgs& A) {
  const int st = *A.stop;
  return st != 0 && st < A.step;
}

// The thread's rows r0 + 32 i + lane of one vector, from p, on their way to its slots of one stage.  The
// vectors' strides are whole tiles and the rows past the end are zeros: no bounds.
template <int RPL>
__device__ __forceinline__ void gs_fetch(const int4* p, unsigned slot) {
#pragma unroll
  for (int i = 0; i < RPL; ++i)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot + 512 * i), "l"(p + 32 * i) : "memory");
}
__device__ __forceinline__ void gs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void gs_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The exponent E of a tile's scale u = 2^(E - 27); a tile that quantised to zeros (u = 0) does so again.
__device__ __forceinline__ int gs_exp(double u) {
  const int e = (int)(((unsigned)__double2hiint(u) >> 20) & 0x7ff);
  return e ? e - 1023 + 27 : 1 << 20;
}
__device__ __forceinline__ cplx gs_read_fp(unsigned slot) {
  double re, im;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(re), "=d"(im) : "r"(slot));
  return mkc(re, im);
}
template <bool kQ>
__device__ __forceinline__ int4 gs_read(unsigned slot, int E) {
  if (!kQ) return q_of(gs_read_fp(slot), E);
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(slot));
  return v;
}

// A tile's rows of J vectors in turn, their copies ahead: begin() starts them (what is computed up to the
// first next() hides their latency), next() waits for the next vector's and returns its slots.
template <int RPL, bool kQ>
struct GsStream {
  static constexpr int D = kGsRing / RPL;
  static constexpr unsigned kStage = 512 * RPL;
  unsigned ring;  // this thread's first slot
  const int4* p = nullptr;
  int64_t ld = 0;
  int left = 0;
  unsigned in = 0, out = 0;  // byte offsets of the next stages to fill and to read
  __device__ __forceinline__ void fetch() {
    if (left > 0) gs_fetch<RPL>(p, ring + in);
    gs_commit();
    --left;
    p += ld;
    in = (in + kStage) & (D * kStage - 1);
  }
  __device__ __forceinline__ void begin(const GsArgs& A, int j0, int J, int64_t r0) {
    ld = A.ld;
    p = (kQ ? A.Vq : reinterpret_cast<const int4*>(A.V)) + (int64_t)j0 * ld + r0 + (threadIdx.x & 31);
    left = J;
    in = out = 0;
#pragma unroll
    for (int j = 0; j < D - 1; ++j) fetch();
  }
  __device__ __forceinline__ unsigned next() {
    fetch();  // into the slots that the vector before left
    gs_wait<D - 1>();
    const unsigned v = ring + out;
    out = (out + kStage) & (D * kStage - 1);
    return v;
  }
};

// w -= sum over j0 <= j < j1 of cu[j] V_j on tile t, in FP64 from the vectors themselves: the copies' scales
// are their tiles', and what is stored keeps the accuracy of each row.
template <int RPL>
__device__ __forceinline__ void gs_remove(const GsArgs& A, unsigned ring, int64_t t, cplx* w, cplx* cf,
                                          double alpha = 0.0) {
  const int lane = threadIdx.x & 31;
  const int64_t r0 = t * (32 * RPL);
  GsStream<RPL, false> S;
  S.ring = ring;
  for (int c0 = A.j0; c0 < A.j1; c0 += kGsChunk) {
    const int J = min(kGsChunk, A.j1 - c0);
    S.begin(A, c0, J, r0);
    __syncwarp();
    if (lane < J) {
      const int j = c0 + lane;
      if (A.ndots) cf[lane] = mkc(A.scl[j] * (j == A.step - 1 ? alpha : A.nrm[A.step - 1]), 0.0);
      else cf[lane] = A.cu[j];
    }
    __syncwarp();
    for (int j = 0; j < J; ++j) {
      const unsigned v = S.next();
      const cplx c = cf[j];
#pragma unroll
      for (int i = 0; i < RPL; ++i) w[i] = vsubmul(w[i], c, gs_read_fp(v + 512 * i));
    }
  }
}

// The blocks' values, block b's v-th at partials[v grid + b], summed in block order by the last block to
// arrive: a warp a value.  True in every thread of that block, the sums in out.
__device__ __forceinline__ bool gs_grid_sum(const GsArgs& A, const double* mine, int nv, double* out) {
  __shared__ bool last;
  const int G = (int)gridDim.x;
  if (threadIdx.x < nv) A.partials[(int64_t)threadIdx.x * G + blockIdx.x] = mine[threadIdx.x];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(A.ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int lane = threadIdx.x & 31;
#pragma unroll 2
  for (int v = threadIdx.x >> 5; v < nv; v += kGsWarps) {
    double a = 0.0;
#pragma unroll 5
    for (int b = lane; b < G; b += 32) a += ld_cg(A.partials + (int64_t)v * G + b);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) out[v] = a;
  }
  if (threadIdx.x == 0) *A.ticket = 0u;
  __syncthreads();
  return true;
}

// The warp's first tile, gridDim.x kGsWarps on to the next.
__device__ __forceinline__ int64_t gs_first_tile() {
  return (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
}

template <int RPL, bool kUpd, bool kQ>
__global__ void __launch_bounds__(kGsThreads, 1) gs_dots_kernel(GsArgs A) {
  if (gs_stopped(A)) return;
  extern __shared__ __align__(16) int4 gs_ring[];
  __shared__ cplx cf[kGsWarps][kGsChunk];
  __shared__ long long tot[kGsWarps][2 * kGsChunk];
  __shared__ double bs[kGsWarps][2 * kGsChunk];
  __shared__ double sum[2 * kGsChunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  GsStream<RPL, kQ> S;
  S.ring = (unsigned)__cvta_generic_to_shared(gs_ring + warp * (32 * kGsRing) + lane);
  // <v_{step-1}, w>, the same in every block
  double alpha = 0.0;
  if (A.ndots) {
    alpha = block_sum(strided_sum<8>(A.dots, (int)A.ndots, 0.0), sum);
    if (threadIdx.x == 0) sum[0] = A.scl[A.step - 1] * alpha;
    __syncthreads();
    alpha = sum[0];
    __syncthreads();
  }
  double are = 0.0, aim = 0.0;  // vector d0 + lane
  for (int64_t t = gs_first_tile(); t < A.ntiles; t += (int64_t)gridDim.x * kGsWarps) {
    const int64_t r0 = t * (32 * RPL);
    cplx w[RPL];
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int64_t r = r0 + 32 * i + lane;
      w[i] = (r < A.n) ? A.src[r] : mkc(0.0, 0.0);
    }
    const double uj = (lane < A.J) ? A.u[(int64_t)(A.d0 + lane) * A.ntiles + t] : 0.0;
    if (kUpd) gs_remove<RPL>(A, S.ring, t, w, cf[warp], alpha);
    S.begin(A, A.d0, A.J, r0);
    unsigned mag = 0;
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int64_t r = r0 + 32 * i + lane;
      if (kUpd && r < A.n) A.dst[r] = w[i];
      mag = max(mag, q_mag(w[i]));
    }
    const QScale q = q_scale(__reduce_max_sync(0xffffffffu, mag));
    int4 wq[RPL];
#pragma unroll
    for (int i = 0; i < RPL; ++i) wq[i] = q_of(w[i], q.E);
    for (int jb = 0; jb < A.J; jb += 4) {
      long long val[8];  // (re, im) of four vectors, in units of 2^-53 so that a warp's sum fits
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        QDot<cplx> a;
        if (jb + jj < A.J) {
          const unsigned v = S.next();
          const int E = kQ ? 0 : gs_exp(__shfl_sync(0xffffffffu, uj, jb + jj));
#pragma unroll
          for (int i = 0; i < RPL; ++i) a.add(gs_read<kQ>(v + 512 * i, E), wq[i]);
        }
        val[2 * jj] = (a.re() + 1) >> 1;
        val[2 * jj + 1] = (a.im() + 1) >> 1;
      }
      // eight warp sums: each step halves the values a lane keeps
#pragma unroll
      for (int h = 4; h >= 1; h >>= 1) {
        const bool up = (lane & (4 * h)) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
          const long long send = up ? val[i] : val[i + h], keep = up ? val[i + h] : val[i];
          val[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * h);
        }
      }
      val[0] += __shfl_xor_sync(0xffffffffu, val[0], 2);
      val[0] += __shfl_xor_sync(0xffffffffu, val[0], 1);
      if ((lane & 3) == 0) tot[warp][2 * jb + (lane >> 2)] = val[0];
    }
    __syncwarp();
    if (lane < A.J) {
      const double s = (q.u * uj) * 2.0;
      are = fma(s, (double)tot[warp][2 * lane], are);
      aim = fma(s, (double)tot[warp][2 * lane + 1], aim);
    }
    __syncwarp();
  }
  bs[warp][2 * lane] = are;
  bs[warp][2 * lane + 1] = aim;
  __syncthreads();
  if (threadIdx.x < 2 * kGsChunk) {
    double a = 0.0;
#pragma unroll
    for (int i = 0; i < kGsWarps; ++i) a += bs[i][threadIdx.x];
    sum[threadIdx.x] = a;
  }
  __syncthreads();
  if (!gs_grid_sum(A, sum, 2 * A.J, bs[0])) return;
  if (threadIdx.x < A.J) {
    const int j = A.d0 + threadIdx.x;
    const double s = A.scl[j];
    const cplx h = mkc(s * bs[0][2 * threadIdx.x], s * bs[0][2 * threadIdx.x + 1]);
    A.cd[j] = vscale(s, h);
    cplx h0 = mkc(0.0, 0.0);
    if (A.ndots) {
      if (j == A.step - 1) h0 = mkc(alpha, 0.0);
      else if (j == A.step - 2) h0 = mkc(A.nrm[A.step - 1], 0.0);
    } else if (A.hadd) {
      h0 = A.hcol[j];
    }
    A.hcol[j] = vadd(h0, h);
  }
}

// dst = src without its components on vectors j0 .. j1 - 1, as vector k of the basis with its scale.
template <int RPL, bool kQ>
__global__ void __launch_bounds__(kGsThreads, 1) gs_update_kernel(GsArgs A) {
  if (gs_stopped(A)) return;
  extern __shared__ __align__(16) int4 gs_ring[];
  __shared__ cplx cf[kGsWarps][kGsChunk];
  __shared__ double bs[kGsWarps];
  __shared__ double sum[1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(gs_ring + warp * (32 * kGsRing) + lane);
  double acc = 0.0;
  // from the last tile down: the dots that ran before left the last tiles in L2
  for (int64_t t = A.ntiles - 1 - gs_first_tile(); t >= 0; t -= (int64_t)gridDim.x * kGsWarps) {
    const int64_t r0 = t * (32 * RPL);
    cplx w[RPL];
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int64_t r = r0 + 32 * i + lane;
      w[i] = (r < A.n) ? A.src[r] : mkc(0.0, 0.0);
    }
    gs_remove<RPL>(A, ring, t, w, cf[warp]);
    unsigned mag = 0;
#pragma unroll
    for (int i = 0; i < RPL; ++i) mag = max(mag, q_mag(w[i]));
    const QScale q = q_scale(__reduce_max_sync(0xffffffffu, mag));
    QAcc n2;
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
      const int64_t r = r0 + 32 * i + lane;
      const int4 x = q_of(w[i], q.E);
      if (r < A.n) {
        A.Vk[r] = w[i];
        if (kQ) A.Vqk[r] = x;
      }
      n2.mac(x.x, x.y, x.x, x.y);
      n2.mac(x.z, x.w, x.z, x.w);
    }
    long long s = (n2.value() + 1) >> 1;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    acc = fma((double)s, (q.u * q.u) * 2.0, acc);
    if (lane == 0) A.u[(int64_t)A.k * A.ntiles + t] = q.u;
  }
  if (lane == 0) bs[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
#pragma unroll
    for (int i = 0; i < kGsWarps; ++i) a += bs[i];
    sum[0] = a;
  }
  __syncthreads();
  if (!gs_grid_sum(A, sum, 1, bs)) return;
  if (threadIdx.x == 0) {
    const double nr = sqrt(bs[0]);
    A.scl[A.k] = 1.0 / nr;
    A.nrm[A.k] = nr;
    if (A.k > 0 && nr < 1e-10 && *A.stop == 0) *A.stop = A.k;  // sparse_algorithm.hpp:387
  }
}

// w = scl H v, a thread per row, and each warp's share of <v, w> (real: H is Hermitian) for the next launch
// to add.  The product is bound by FP64 issue and its gathers; the common kernel's sum of the dot, a tree of
// complex sums per row and a block barrier, made its launch 78 us of 56 at 705,432 rows.  Here a warp takes
// several rows per lane, sums its lanes in integers and ends without a barrier.
constexpr int kGsProductThreads = 128;
static int gs_sets(int64_t n) { return n >= (1 << 18) ? 4 : 1; }

template <typename MV>
__global__ void __launch_bounds__(kGsProductThreads) gs_product_kernel(GsArgs A, const int64_t* __restrict__ rowptr,
                                                                       const int32_t* __restrict__ colidx,
                                                                       const MV* __restrict__ vals,
                                                                       const cplx* __restrict__ x, const double* scale,
                                                                       cplx* __restrict__ y, int sets) {
  if (gs_stopped(A)) return;
  const int64_t gw = ((int64_t)blockIdx.x * kGsProductThreads + threadIdx.x) >> 5;
  const double scl = *scale;
  double d = 0.0;
#pragma unroll 1
  for (int i = 0; i < sets; ++i) {
    const int64_t r = (gw * sets + i) * 32 + (threadIdx.x & 31);
    if (r >= A.n) break;
    const int64_t e = rowptr[r + 1];
    int64_t k = rowptr[r];
    cplx acc = mkc(0.0, 0.0);
    for (; k + 4 <= e; k += 4) {
      int32_t c[4];
      MV v[4];
      cplx xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        c[u] = ld_plain(colidx + k + u);
        v[u] = ld_plain(vals + k + u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = ld_ro(x + c[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) acc = vfma(v[u], xv[u], acc);
    }
    for (; k < e; ++k) acc = vfma(ld_plain(vals + k), ld_ro(x + ld_plain(colidx + k)), acc);
    acc = vscale(scl, acc);
    y[r] = acc;
    const cplx xr = ld_ro(x + r);
    d = fma(xr.im, acc.im, fma(xr.re, acc.re, d));
  }
  const QScale q = q_scale(__reduce_max_sync(0xffffffffu, q_mag(d)));
  const int2 h = q_of(d, q.E);
  long long s = ((long long)h.x << 28) + h.y;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0 && gw * sets * 32 < A.n) A.dots[gw] = (double)s * (q.u * 3.7252902984619140625e-09);  // 2^-28
}

// Warps of the product; their shares of the dot.
static int64_t gs_product_warps(int64_t n) { return ceil_div(n, 32 * gs_sets(n)); }

// The rows past the end of each vector.
template <typename T>
static void gs_zero_tails(T* p, int64_t n, int64_t ld, int vecs, cudaStream_t s) {
  if (ld > n) QD_CUDA(cudaMemset2DAsync(p + n, ld * sizeof(T), 0, (ld - n) * sizeof(T), vecs, s));
}

bool GsBasis::ensure(Ctx* ctx, int64_t n_, int vecs_, bool herm, bool copies) {
  if (n_ == n && vecs_ == vecs && herm == (dots.p != nullptr)) return false;
  n = 0;  // until every buffer is there
  // Tiles of 128 rows amortise their conversions better, tiles of 64 fill the SMs' warps sooner: two steps
  // of m = 16 (m = 30) at 12,870 rows 1.11 against 1.02 ms, 48,620 rows (2.81) against (2.50), 92,378 rows 1.37
  // against 1.32, 184,756 rows 1.89 (4.56) against 1.96 ms (4.77).
  rpl = (n_ >= 64 * (int64_t)ctx->num_sms * kGsWarps) ? 4 : 2;
  ntiles = ceil_div(n_, 32 * rpl);
  grid = (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)ctx->num_sms));
  ld = ntiles * 32 * rpl;
  V.alloc((size_t)vecs_ * ld);
  u.alloc((size_t)vecs_ * ntiles);
  w.alloc(ld);
  coef.alloc(2 * (size_t)vecs_);
  if (herm) dots.alloc(gs_product_warps(n_));
  else dots.release();
  scl.alloc(vecs_);
  nrm.alloc(vecs_);
  partials.alloc((size_t)grid * 2 * kGsChunk);
  ticket.alloc(1);
  stop.alloc(1);
  QD_CUDA(cudaMemsetAsync(ticket.p, 0, sizeof(unsigned), ctx->stream));
  gs_zero_tails(V.p, n_, ld, vecs_, ctx->stream);
  Vq.release();
  size_t fr = 0, total = 0;
  if (copies && cudaMemGetInfo(&fr, &total) == cudaSuccess && (size_t)vecs_ * ld * sizeof(int4) <= fr / 4) {
    try {
      Vq.alloc((size_t)vecs_ * ld);
      gs_zero_tails(Vq.p, n_, ld, vecs_, ctx->stream);
    } catch (const Error&) {  // another thread took the memory meanwhile
      clear_error();
      Vq.release();
    }
  }
  vecs = vecs_;
  n = n_;
  return true;
}

static GsArgs gs_args(GsBasis& B, int step) {
  GsArgs A{};
  A.n = B.n;
  A.ld = B.ld;
  A.ntiles = B.ntiles;
  A.V = B.V.p;
  A.Vq = B.Vq.p;
  A.u = B.u.p;
  A.scl = B.scl.p;
  A.nrm = B.nrm.p;
  A.partials = B.partials.p;
  A.dots = B.dots.p;
  A.ticket = B.ticket.p;
  A.stop = B.stop.p;
  A.step = step;
  return A;
}

template <typename K>
static void gs_launch(Ctx* ctx, const GsBasis& B, K kernel, const GsArgs& A) {
  QD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGsSmem));
  kernel<<<B.grid, kGsThreads, kGsSmem, ctx->stream>>>(A);
  QD_CHECK_LAUNCH();
  QD_LAUNCHED(ctx);
}

template <int RPL, bool kQ>
static void gs_dots(Ctx* ctx, const GsBasis& B, const GsArgs& A, bool upd) {
  if (upd) gs_launch(ctx, B, gs_dots_kernel<RPL, true, kQ>, A);
  else gs_launch(ctx, B, gs_dots_kernel<RPL, false, kQ>, A);
}

static void gs_dots(Ctx* ctx, const GsBasis& B, const GsArgs& A, bool upd) {
  const bool q = B.Vq.p != nullptr;
  if (B.rpl == 4) q ? gs_dots<4, true>(ctx, B, A, upd) : gs_dots<4, false>(ctx, B, A, upd);
  else q ? gs_dots<2, true>(ctx, B, A, upd) : gs_dots<2, false>(ctx, B, A, upd);
}

static void gs_update(Ctx* ctx, GsBasis& B, GsArgs A, int k) {
  A.k = k;
  A.Vk = B.vec(k);
  const bool q = B.Vq.p != nullptr;
  A.Vqk = q ? B.Vq.p + (int64_t)k * B.ld : nullptr;
  if (B.rpl == 4) gs_launch(ctx, B, q ? gs_update_kernel<4, true> : gs_update_kernel<4, false>, A);
  else gs_launch(ctx, B, q ? gs_update_kernel<2, true> : gs_update_kernel<2, false>, A);
}

// w = scl H V_{idx-1}; true with the warps' shares of <V_{idx-1}, w> in B.dots.
template <typename MV>
static bool gs_product(qd_ham* H, const MV* vals, GsBasis& B, int idx) {
  Ctx* ctx = H->ctx;
  const cplx* v = B.vec(idx - 1);
  const double* scl = B.scl.p + idx - 1;
  if (B.dots.p) {
    gs_product_kernel<MV><<<(unsigned)ceil_div(gs_product_warps(B.n), kGsProductThreads / 32), kGsProductThreads, 0,
                            ctx->stream>>>(gs_args(B, idx), H->rowptr.p, H->colidx.p, vals, v, scl, B.w.p,
                            gs_sets(B.n));
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
    return true;
  }
  launch_spmv<MV, cplx>(ctx, H, vals, v, B.w.p, 1.0, nullptr, ham_workspace(H).red_c(0), nullptr, B.stop.p, idx, -1,
                        scl);
  return false;
}

void gs_begin(Ctx* ctx, GsBasis& B, const cplx* psi) {
  QD_CUDA(cudaMemsetAsync(B.stop.p, 0, sizeof(int), ctx->stream));
  GsArgs A = gs_args(B, 0);
  A.src = psi;
  gs_update(ctx, B, A, 0);
}

void gs_step(qd_ham* H, GsBasis& B, int idx, cplx* hcol) {
  Ctx* ctx = H->ctx;
  const bool alpha = (H->flags & QD_HAM_REAL) ? gs_product<double>(H, H->vals_r.p, B, idx)
                                              : gs_product<cplx>(H, H->vals_c.p, B, idx);
  GsArgs A = gs_args(B, idx);
  A.src = B.w.p;
  A.dst = B.w.p;
  A.hcol = hcol;
  A.j1 = idx;
  if (alpha) {
    A.ndots = gs_product_warps(B.n);
    A.j0 = std::max(0, idx - 2);
  } else {
    A.cd = B.coef.p;
    for (int d = 0; d < idx; d += kGsChunk) {
      A.d0 = d;
      A.J = std::min(kGsChunk, idx - d);
      gs_dots(ctx, B, A, false);
    }
    A.cu = B.coef.p;
    A.hadd = true;
  }
  A.cd = B.coef.p + B.vecs;
  for (int d = 0; d < idx; d += kGsChunk) {
    A.d0 = d;
    A.J = std::min(kGsChunk, idx - d);
    gs_dots(ctx, B, A, d == 0);
  }
  A.ndots = 0;
  A.cu = A.cd;
  A.j0 = 0;
  gs_update(ctx, B, A, idx);
}

}  // namespace qd
