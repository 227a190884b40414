// evolve.cu -- Krylov real-time step psi <- exp(-i H h) psi.
//
// Restates ArnoldiSolver<T, herm=0>::evolve (sparse_algorithm.hpp:548-562)
// with expandBasis<0> (:372-393) and updateKrylovRepr (:521-546):
//   v_0 = psi / ||psi||;  for idx = 1 .. m-1:
//     w = H v_{idx-1};  orthogonalise w against v_0 .. v_{idx-1};
//     h_{idx, idx-1} = ||w||;  v_idx = w / ||w||;  stop (keeping the step)
//     when ||w|| < 1e-10;
//   act = number of columns;  psi_out = V[:, :act] exp(-i h K[:act, :act])[:, 0].
// The reference orthogonalises by modified Gram-Schmidt, one dot and one axpy
// per previous vector.  On the device each pass is instead one multi-dot
// kernel (all projections at once) and one update kernel, applied twice
// (classical Gram-Schmidt with reorthogonalisation): the same projector up to
// rounding, with better orthogonality, in 4 launches per step instead of
// 2 * idx.  The small exponential runs on the host (dense.h).  This form serves
// the requests of the serving loop and sectors too large for the persistent
// recurrence (arnres.cu), which takes all other calls.
#include <algorithm>
#include <cstring>
#include <vector>

#include "arnres.cuh"
#include "dense.h"
#include "tridiag.cuh"
#include "evolve.cuh"
#include "krylov.cuh"
#include "spmv.cuh"

namespace qd {

constexpr int kEvThreads = 256;

// Grid of the multi-dot kernels (their per-thread accumulators allow two blocks per SM).
static int ev_grid(Ctx* ctx, int64_t n) {
  const int64_t want = ceil_div(n, kEvThreads * 4);
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 2));
}

// Grid of the streaming kernels (update, norm, scale, combination): eight blocks per SM.
static int ev_stream_grid(Ctx* ctx, int64_t n) {
  const int64_t want = ceil_div(n, kEvThreads);
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 8));
}

__device__ __forceinline__ bool ev_stopped(const int* stop, int step) {
  const int st = *stop;
  return st != 0 && st < step;
}

// out[j] = <V_j, w> for j < J (J <= 32): w staged in shared memory tile by tile
// and a warp per basis vector inside a tile (two accumulators per lane, four
// loads of V_j in flight), so a thread holds one complex accumulator pair, not
// J, and six blocks fit an SM.  Each tile's warp sums are added to the block's
// partial in tile order and the blocks' partials in block order: deterministic.
constexpr int kDotTile = 2048;  // complex elements of w per tile (32 KB)

__global__ void __launch_bounds__(kEvThreads) multidot_tile_kernel(int64_t n, const cplx* __restrict__ V, int64_t ld,
                                                                   int J, const cplx* __restrict__ w,
                                                                   cplx* partials, unsigned* ticket, cplx* out,
                                                                   const int* stop, int step) {
  if (ev_stopped(stop, step)) return;
  __shared__ cplx ws[kDotTile];
  __shared__ cplx part[32];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = kEvThreads / 32;
  if (threadIdx.x < 32) part[threadIdx.x] = mkc(0.0, 0.0);
  for (int64_t t0 = (int64_t)blockIdx.x * kDotTile; t0 < n; t0 += (int64_t)gridDim.x * kDotTile) {
    const int tn = (int)std::min<int64_t>(kDotTile, n - t0);
    __syncthreads();  // the previous tile's readers are done (and part is zeroed)
    for (int i = threadIdx.x; i < tn; i += kEvThreads) ws[i] = w[t0 + i];
    __syncthreads();
    for (int j = warp; j < J; j += nw) {
      const cplx* vj = V + (int64_t)j * ld + t0;
      cplx a0 = mkc(0.0, 0.0), a1 = mkc(0.0, 0.0);
      int i = lane;
      for (; i + 96 < tn; i += 128) {
        const cplx x0 = vj[i], x1 = vj[i + 32], x2 = vj[i + 64], x3 = vj[i + 96];
        a0 = vdotfma(x0, ws[i], a0);
        a1 = vdotfma(x1, ws[i + 32], a1);
        a0 = vdotfma(x2, ws[i + 64], a0);
        a1 = vdotfma(x3, ws[i + 96], a1);
      }
      for (; i < tn; i += 32) a0 = vdotfma(vj[i], ws[i], a0);
      const cplx t = warp_sum0(vadd(a0, a1));
      if (lane == 0) part[j] = vadd(part[j], t);  // one warp owns vector j: no race
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) partials[(int64_t)blockIdx.x * 32 + threadIdx.x] = part[threadIdx.x];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < J) {
    cplx t = mkc(0.0, 0.0);
    for (unsigned b = 0; b < gridDim.x; ++b) t = vadd(t, ld_cg(partials + (int64_t)b * 32 + threadIdx.x));
    out[threadIdx.x] = t;
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

// Grid of multidot_tile_kernel: one tile per block at most, up to six blocks per SM.
static int ev_tile_grid(Ctx* ctx, int64_t n) {
  const int64_t want = ceil_div(n, kDotTile);
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 6));
}

// w -= sum_{j<J} c_j V_j;  acc_h[j] += c_j (the Hessenberg column gathers both passes)
__global__ void __launch_bounds__(kEvThreads) gs_update_kernel(int64_t n, const cplx* __restrict__ V, int64_t ld,
                                                               int J, const cplx* c, cplx* __restrict__ w,
                                                               cplx* hcol, int first_pass, const int* stop, int step) {
  if (ev_stopped(stop, step)) return;
  __shared__ cplx s_c[64];
  if (threadIdx.x < J) s_c[threadIdx.x] = c[threadIdx.x];
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x < J)
    hcol[threadIdx.x] = first_pass ? s_c[threadIdx.x] : vadd(hcol[threadIdx.x], s_c[threadIdx.x]);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    cplx wi = w[i];
    int j = 0;
    for (; j + 4 <= J; j += 4) {  // four loads in flight, the updates still in j order
      const cplx v0 = V[(int64_t)j * ld + i], v1 = V[(int64_t)(j + 1) * ld + i];
      const cplx v2 = V[(int64_t)(j + 2) * ld + i], v3 = V[(int64_t)(j + 3) * ld + i];
      wi = vsubmul(wi, s_c[j], v0);
      wi = vsubmul(wi, s_c[j + 1], v1);
      wi = vsubmul(wi, s_c[j + 2], v2);
      wi = vsubmul(wi, s_c[j + 3], v3);
    }
    for (; j < J; ++j) wi = vsubmul(wi, s_c[j], V[(int64_t)j * ld + i]);
    w[i] = wi;
  }
}

__global__ void __launch_bounds__(kEvThreads) ev_norm_kernel(int64_t n, const cplx* __restrict__ w, double* nrm2,
                                                             double* nrm, GridRed<double> red, int* stop, int step) {
  if (ev_stopped(stop, step)) return;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    acc += vnorm2(w[i]);
  double n2 = 0.0;
  if (grid_sum(acc, red, nrm2, &n2) && threadIdx.x == 0) {
    const double nr = sqrt(n2);
    *nrm = nr;
    if (nr < 1e-10 && *stop == 0) *stop = step;  // sparse_algorithm.hpp:387
  }
}

__global__ void __launch_bounds__(kEvThreads) ev_scale_kernel(int64_t n, const cplx* __restrict__ w,
                                                              const double* nrm, cplx* __restrict__ vout,
                                                              const int* stop, int step) {
  if (ev_stopped(stop, step)) return;
  const double inv = 1.0 / *nrm;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    vout[i] = vscale(inv, w[i]);
}

__global__ void __launch_bounds__(kEvThreads) ev_init_kernel(int64_t n, const cplx* psi, const double* nrm2,
                                                             cplx* v0) {
  const double inv = 1.0 / sqrt(*nrm2);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v0[i] = vscale(inv, psi[i]);
}

__global__ void __launch_bounds__(kEvThreads) ev_norm_only_kernel(int64_t n, const cplx* psi, double* nrm2,
                                                                  GridRed<double> red) {
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    acc += vnorm2(psi[i]);
  grid_sum(acc, red, nrm2);
}

// out = sum_{j<a} e_j V_j
__global__ void __launch_bounds__(kEvThreads) ev_combine_kernel(int64_t n, const cplx* __restrict__ V, int64_t ld,
                                                                int a, const cplx* e, cplx* __restrict__ out) {
  __shared__ cplx s_e[64];
  if (threadIdx.x < a) s_e[threadIdx.x] = e[threadIdx.x];
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    cplx acc = mkc(0.0, 0.0);
    int j = 0;
    for (; j + 4 <= a; j += 4) {  // four loads in flight, the sum still in j order
      const cplx v0 = V[(int64_t)j * ld + i], v1 = V[(int64_t)(j + 1) * ld + i];
      const cplx v2 = V[(int64_t)(j + 2) * ld + i], v3 = V[(int64_t)(j + 3) * ld + i];
      acc = vfma(s_e[j], v0, acc);
      acc = vfma(s_e[j + 1], v1, acc);
      acc = vfma(s_e[j + 2], v2, acc);
      acc = vfma(s_e[j + 3], v3, acc);
    }
    for (; j < a; ++j) acc = vfma(s_e[j], V[(int64_t)j * ld + i], acc);
    out[i] = acc;
  }
}

void launch_ev_combine(Ctx* ctx, int64_t n, const cplx* V, int64_t ld, int a, const cplx* e, cplx* out) {
  ev_combine_kernel<<<ev_stream_grid(ctx, n), kEvThreads, 0, ctx->stream>>>(n, V, ld, a, e, out);
  QD_CHECK_LAUNCH();
  QD_LAUNCHED(ctx);
}

void ArnoldiBuffers::drop_graph() {
  if (steps_exec) cudaGraphExecDestroy(steps_exec);
  steps_exec = nullptr;
  steps_m = steps_kind = 0;
  steps_variant = -1;
  steps_seen = -1;
}

void ArnoldiBuffers::ensure(int64_t n_, int m_, int grid, cudaStream_t stream) {
  if (n_ == n && m_ == m && grid <= grid_cap) return;
  drop_graph();  // the buffers move
  n = n_;
  m = m_;
  ld = (n + 31) / 32 * 32;
  grid_cap = std::max(grid, 1);
  V.alloc((size_t)(m + 1) * ld);
  w.alloc(ld);
  proj.alloc(64);
  hcol.alloc((size_t)(m + 1) * 64);
  nrm.alloc(m + 2);
  nrm2.alloc(m + 2);
  stop.alloc(1);
  e.alloc(64);
  partials.alloc((size_t)grid_cap * 32);
  rpart.alloc(kMaxGrid);
  tickets.alloc(4);
  QD_CUDA(cudaMemsetAsync(tickets.p, 0, 4 * sizeof(unsigned), stream));
}

template <typename MV>
static void arnoldi_steps(qd_ham* H, const MV* vals, ArnoldiBuffers& B, int steps) {
  Ctx* ctx = H->ctx;
  Workspace& W = ham_workspace(H);
  const int64_t n = B.n;
  const int gs = ev_stream_grid(ctx, n), gt = ev_tile_grid(ctx, n);
  for (int idx = 1; idx <= steps; ++idx) {
    const cplx* vprev = B.V.p + (int64_t)(idx - 1) * B.ld;
    launch_spmv<MV, cplx>(ctx, H, vals, vprev, B.w.p, 1.0, nullptr, W.red_c(0), nullptr, B.stop.p, idx, -1);
    cplx* hcol = B.hcol.p + (int64_t)(idx - 1) * 64;
    for (int pass = 0; pass < 2; ++pass) {
      multidot_tile_kernel<<<gt, kEvThreads, 0, ctx->stream>>>(n, B.V.p, B.ld, idx, B.w.p, B.partials.p,
                                                               B.tickets.p, B.proj.p, B.stop.p, idx);
      QD_CHECK_LAUNCH();
      QD_LAUNCHED(ctx);
      gs_update_kernel<<<gs, kEvThreads, 0, ctx->stream>>>(n, B.V.p, B.ld, idx, B.proj.p, B.w.p, hcol, pass == 0,
                                                            B.stop.p, idx);
      QD_CHECK_LAUNCH();
      QD_LAUNCHED(ctx);
    }
    ev_norm_kernel<<<gs, kEvThreads, 0, ctx->stream>>>(n, B.w.p, B.nrm2.p + idx, B.nrm.p + idx,
                                                        GridRed<double>{B.rpart.p, B.tickets.p + 1}, B.stop.p, idx);
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
    ev_scale_kernel<<<gs, kEvThreads, 0, ctx->stream>>>(n, B.w.p, B.nrm.p + idx, B.V.p + (int64_t)idx * B.ld,
                                                         B.stop.p, idx);
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
  }
}

void arnoldi_evolve(qd_ham* H, const cplx* psi_in, cplx* psi_out, double h, int m, int* act_out) {
  Ctx* ctx = H->ctx;
  QD_REQUIRE(m >= 2 && m <= 33, QD_ERR_UNSUPPORTED, "Krylov dimension m must be in 2..33");
  const int64_t n = H->dim;
  if (arn_res_fits(H, m - 1)) {
    if (!H->arn_ev) H->arn_ev.reset(new ArnRes());
    if (arn_res_evolve(H, *H->arn_ev, psi_in, psi_out, h, m - 1, act_out)) return;
  }
  if (!H->arnoldi) H->arnoldi.reset(new ArnoldiBuffers());
  ArnoldiBuffers& B = *H->arnoldi;
  const int g = ev_grid(ctx, n);
  B.ensure(n, m, std::max(g, ev_tile_grid(ctx, n)), ctx->stream);
  // v_0 = psi / ||psi||
  ev_norm_only_kernel<<<g, kEvThreads, 0, ctx->stream>>>(n, psi_in, B.nrm2.p, GridRed<double>{B.rpart.p, B.tickets.p + 1});
  QD_CHECK_LAUNCH();
  QD_LAUNCHED(ctx);
  ev_init_kernel<<<g, kEvThreads, 0, ctx->stream>>>(n, psi_in, B.nrm2.p, B.V.p);
  QD_CHECK_LAUNCH();
  QD_LAUNCHED(ctx);
  QD_CUDA(cudaMemsetAsync(B.stop.p, 0, sizeof(int), ctx->stream));
  const int steps = m - 1;  // updateKrylovRepr(H, kry_dim_rt - 1)
  const bool real = (H->flags & QD_HAM_REAL) != 0;
  auto run_steps = [&]() {
    if (real) arnoldi_steps<double>(H, H->vals_r.p, B, steps);
    else arnoldi_steps<cplx>(H, H->vals_c.p, B, steps);
  };
  const int kind = real ? 1 : 2;
  // one uncaptured run per (m, value type, product kernel) first: the product's workspace and
  // tables are allocated on first use, which a capture does not allow
  const long long key = ((long long)H->spmv_variant << 16) | ((long long)kind << 8) | (long long)m;
  if (H->one_shot || B.steps_seen != key) {  // a served request is solved once: no capture
    run_steps();
    B.steps_seen = key;
  } else {
    const void* vals = real ? (const void*)H->vals_r.p : (const void*)H->vals_c.p;
    if (!B.steps_exec || B.steps_m != m || B.steps_kind != kind || B.steps_variant != H->spmv_variant ||
        B.steps_vals != vals || B.steps_rowptr != (const void*)H->rowptr.p) {
      if (B.steps_exec) cudaGraphExecDestroy(B.steps_exec);
      B.steps_exec = nullptr;
      cudaGraph_t gr = nullptr;
      const int64_t before = ctx->launches;
      QD_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
      try {
        run_steps();
      } catch (...) {
        cudaStreamEndCapture(ctx->stream, &gr);
        if (gr) cudaGraphDestroy(gr);
        ctx->launches = before;
        throw;
      }
      QD_CUDA(cudaStreamEndCapture(ctx->stream, &gr));
      B.steps_kernels = ctx->launches - before;
      ctx->launches = before;
      const cudaError_t e = cudaGraphInstantiate(&B.steps_exec, gr, 0);
      cudaGraphDestroy(gr);
      QD_CUDA(e);
      B.steps_m = m;
      B.steps_kind = kind;
      B.steps_variant = H->spmv_variant;
      B.steps_vals = vals;
      B.steps_rowptr = H->rowptr.p;
    }
    QD_CUDA(cudaGraphLaunch(B.steps_exec, ctx->stream));
    ctx->launches += B.steps_kernels;
  }
  std::vector<cplx> hc((size_t)(m + 1) * 64);
  std::vector<double> nrm(m + 2);
  int stop = 0;
  QD_CUDA(cudaMemcpyAsync(hc.data(), B.hcol.p, hc.size() * sizeof(cplx), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(nrm.data(), B.nrm.p, nrm.size() * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(&stop, B.stop.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  const int act = stop ? stop : steps;  // expandBasis<0> return value
  // K(j, i) = projection of H v_i on v_j (j <= i), K(i+1, i) = ||w_{i+1}||
  dense::Mat A((size_t)act * act, dense::cd(0.0, 0.0));
  for (int i = 0; i < act; ++i) {
    for (int j = 0; j <= i; ++j) {
      const cplx v = hc[(size_t)i * 64 + j];
      A[(size_t)i * act + j] = dense::cd(v.re, v.im);
    }
    if (i + 1 < act) A[(size_t)i * act + i + 1] = nrm[i + 1];
  }
  for (auto& a : A) a *= dense::cd(0.0, -h);  // -i K h
  dense::Mat E;
  QD_REQUIRE(dense::expm(A, act, E), QD_ERR_INVALID, "matrix exponential failed");
  std::vector<cplx> e(act);
  for (int j = 0; j < act; ++j) e[j] = mkc(E[j].real(), E[j].imag());
  QD_CUDA(cudaMemcpyAsync(B.e.p, e.data(), act * sizeof(cplx), cudaMemcpyHostToDevice, ctx->stream));
  launch_ev_combine(ctx, n, B.V.p, B.ld, act, B.e.p, psi_out);
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  if (act_out) *act_out = act;
}

// ---------------------------------------------------------------- Arnoldi ground state
// ArnoldiSolver<T, herm=0>::getGroundState (sparse_algorithm.hpp:564-585) with
// updateKrylovRepr (:521-546) and expandBasis<0> (:372-393): the basis grows by
// full orthogonalisation against every previous vector (here classical
// Gram-Schmidt applied twice, the multi-dot over 32-vector chunks), the breaking
// step (||w|| < 1e-10) counts, and the ground state comes from the reference's
// SelfAdjointEigenSolver on the Arnoldi matrix's lower triangle: the real parts
// of the diagonal <v_i, H v_i> and the sub-diagonal norms, a symmetric
// tridiagonal matrix (for Hermitian H the same matrix as the full projection).
// psi = V[:, :act] z_0 (getState<herm 0>, :447-453).

// w -= sum_{j<J} c_j V_j for any J (coefficients staged 128 at a time);
// hcol[j] (+)= c_j by block 0
__global__ void __launch_bounds__(kEvThreads) gs_update_long_kernel(int64_t n, const cplx* __restrict__ V,
                                                                    int64_t ld, int J, const cplx* c,
                                                                    cplx* __restrict__ w, cplx* hcol, int first_pass,
                                                                    const int* stop, int step) {
  if (ev_stopped(stop, step)) return;
  __shared__ cplx s_c[128];
  if (blockIdx.x == 0)
    for (int j = threadIdx.x; j < J; j += blockDim.x) hcol[j] = first_pass ? c[j] : vadd(hcol[j], c[j]);
  for (int j0 = 0; j0 < J; j0 += 128) {
    const int jc = min(128, J - j0);
    __syncthreads();
    if (threadIdx.x < jc) s_c[threadIdx.x] = c[j0 + threadIdx.x];
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
      cplx wi = w[i];
      const cplx* vp = V + (int64_t)j0 * ld + i;
      int j = 0;
      for (; j + 4 <= jc; j += 4) {  // four loads in flight, the updates still in j order
        const cplx v0 = vp[(int64_t)j * ld], v1 = vp[(int64_t)(j + 1) * ld];
        const cplx v2 = vp[(int64_t)(j + 2) * ld], v3 = vp[(int64_t)(j + 3) * ld];
        wi = vsubmul(wi, s_c[j], v0);
        wi = vsubmul(wi, s_c[j + 1], v1);
        wi = vsubmul(wi, s_c[j + 2], v2);
        wi = vsubmul(wi, s_c[j + 3], v3);
      }
      for (; j < jc; ++j) wi = vsubmul(wi, s_c[j], vp[(int64_t)j * ld]);
      w[i] = wi;
    }
  }
}

// out = sum_{j<a} e_j V_j for any a
__global__ void __launch_bounds__(kEvThreads) ev_combine_long_kernel(int64_t n, const cplx* __restrict__ V, int64_t ld,
                                                                     int a, const cplx* e, cplx* __restrict__ out) {
  __shared__ cplx s_e[128];
  for (int j0 = 0; j0 < a; j0 += 128) {
    const int jc = min(128, a - j0);
    __syncthreads();
    if (threadIdx.x < jc) s_e[threadIdx.x] = e[j0 + threadIdx.x];
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
      cplx acc = (j0 == 0) ? mkc(0.0, 0.0) : out[i];
      const cplx* vp = V + (int64_t)j0 * ld + i;
      int j = 0;
      for (; j + 4 <= jc; j += 4) {  // four loads in flight, the sum still in j order
        const cplx v0 = vp[(int64_t)j * ld], v1 = vp[(int64_t)(j + 1) * ld];
        const cplx v2 = vp[(int64_t)(j + 2) * ld], v3 = vp[(int64_t)(j + 3) * ld];
        acc = vfma(s_e[j], v0, acc);
        acc = vfma(s_e[j + 1], v1, acc);
        acc = vfma(s_e[j + 2], v2, acc);
        acc = vfma(s_e[j + 3], v3, acc);
      }
      for (; j < jc; ++j) acc = vfma(s_e[j], vp[(int64_t)j * ld], acc);
      out[i] = acc;
    }
  }
}

void ArnoldiGround::ensure(int64_t n_, int kdim_, int grid, cudaStream_t stream) {
  if (n_ == n && kdim_ == kdim && grid <= grid_cap) return;
  n = n_;
  kdim = kdim_;
  ld = (n + 31) / 32 * 32;
  ldh = kdim + 1;
  grid_cap = std::max(grid, 1);
  V.alloc((size_t)(kdim + 1) * ld);
  w.alloc(ld);
  proj.alloc(kdim + 1);
  hcol.alloc((size_t)(kdim + 1) * ldh);
  nrm.alloc(kdim + 2);
  nrm2.alloc(kdim + 2);
  stop.alloc(1);
  e.alloc(kdim + 1);
  partials.alloc((size_t)grid_cap * 32);
  rpart.alloc(kMaxGrid);
  tickets.alloc(4);
  QD_CUDA(cudaMemsetAsync(tickets.p, 0, 4 * sizeof(unsigned), stream));
}

template <typename MV>
static void arnoldi_ground_steps(qd_ham* H, const MV* vals, ArnoldiGround& B, int first, int last) {
  Ctx* ctx = H->ctx;
  Workspace& W = ham_workspace(H);
  const int64_t n = B.n;
  const int gs = ev_stream_grid(ctx, n), gt = ev_tile_grid(ctx, n);
  for (int idx = first; idx <= last; ++idx) {
    const cplx* vprev = B.V.p + (int64_t)(idx - 1) * B.ld;
    launch_spmv<MV, cplx>(ctx, H, vals, vprev, B.w.p, 1.0, nullptr, W.red_c(0), nullptr, B.stop.p, idx, -1);
    cplx* hcol = B.hcol.p + (int64_t)(idx - 1) * B.ldh;
    for (int pass = 0; pass < 2; ++pass) {
      for (int j0 = 0; j0 < idx; j0 += 32) {
        multidot_tile_kernel<<<gt, kEvThreads, 0, ctx->stream>>>(n, B.V.p + (int64_t)j0 * B.ld, B.ld,
                                                                 std::min(32, idx - j0), B.w.p, B.partials.p,
                                                                 B.tickets.p, B.proj.p + j0, B.stop.p, idx);
        QD_CHECK_LAUNCH();
        QD_LAUNCHED(ctx);
      }
      gs_update_long_kernel<<<gs, kEvThreads, 0, ctx->stream>>>(n, B.V.p, B.ld, idx, B.proj.p, B.w.p, hcol,
                                                                 pass == 0, B.stop.p, idx);
      QD_CHECK_LAUNCH();
      QD_LAUNCHED(ctx);
    }
    ev_norm_kernel<<<gs, kEvThreads, 0, ctx->stream>>>(n, B.w.p, B.nrm2.p + idx, B.nrm.p + idx,
                                                        GridRed<double>{B.rpart.p, B.tickets.p + 1}, B.stop.p, idx);
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
    ev_scale_kernel<<<gs, kEvThreads, 0, ctx->stream>>>(n, B.w.p, B.nrm.p + idx, B.V.p + (int64_t)idx * B.ld,
                                                         B.stop.p, idx);
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
  }
}

// The persistent form of arnoldi_ground (arnres.cu).  False, with nothing run, when it does not take
// the solve; a solve that it began it also continues.
static bool arnoldi_ground_res(qd_ham* H, cplx* psi, int kdim, int add_dim, bool extend, double* evals_out,
                               qd_lanczos_result* res) {
  Ctx* ctx = H->ctx;
  if (!extend) {
    if (H->arn_gs) H->arn_gs->open = false;
    if (!arn_res_fits(H, kdim)) return false;
    if (!H->arn_gs) H->arn_gs.reset(new ArnRes());
    bool has_imag = false;
    const double n0 = state_norm2_imag(H, psi, &has_imag);
    QD_REQUIRE(n0 > 0.0, QD_ERR_INVALID, "start vector is zero");
    H->arn_gs->act = 0;
    H->arn_gs->broke = false;
    // a real operator keeps a real start vector's Krylov space real
    H->arn_gs->real_start = !has_imag && (H->flags & QD_HAM_REAL);
  } else if (!H->arn_gs || !H->arn_gs->open || H->arn_gs->kdim != kdim) {
    return false;
  }
  ArnRes& B = *H->arn_gs;
  int steps = (add_dim <= 0 || B.act + add_dim > kdim) ? kdim - B.act : add_dim;
  if (B.broke) steps = 0;
  const int act_prev = B.act;
  if (steps > 0) {
    B.open = false;
    if (!arn_res_steps(H, B, psi, kdim, B.real_start, B.act + 1, B.act + steps)) return false;
    B.open = true;
    if (H->arnoldi_gs) H->arnoldi_gs->open = false;
    B.act = B.host.stop ? B.host.stop : B.act + steps;  // expandBasis<0>: the breaking step counts
    B.broke = B.host.stop != 0;
  }
  const int act = B.act;
  QD_REQUIRE(act >= 1, QD_ERR_INVALID, "no Krylov step was run");
  std::vector<double> d(act), e(act), ev(act), y(act);
  for (int i = 0; i < act; ++i) {
    d[i] = B.host.alpha[i + 1];
    e[i] = (i + 1 < act) ? B.host.nrm[i + 1] : 0.0;
  }
  QD_REQUIRE(tridiag_lowest<double>(act, d.data(), e.data(), ev.data(), y.data()) == 0, QD_ERR_INVALID,
             "tridiagonal eigensolver did not converge");
  for (int j = 0; j < act; ++j) y[j] *= B.host.scl[j];
  double* yd = reinterpret_cast<double*>(B.hcol.p);
  QD_CUDA(cudaMemcpyAsync(yd, y.data(), act * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  launch_ritz(ctx, H->dim, B.V.p, B.real_v, B.ld, yd, act, psi);
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  if (evals_out) std::memcpy(evals_out, ev.data(), act * sizeof(double));
  res->act_dim = act;
  res->breakdown = B.broke ? 1 : 0;
  res->matvecs = act - act_prev;
  res->ritz_value = ev[0];
  res->err = std::fabs(ev[0]);
  return true;
}

void arnoldi_ground(qd_ham* H, cplx* psi, int kdim, int add_dim, bool extend, double* evals_out,
                    qd_lanczos_result* res) {
  Ctx* ctx = H->ctx;
  const int64_t n = H->dim;
  QD_REQUIRE(kdim >= 1 && kdim <= 4096, QD_ERR_INVALID, "krylov_dim must be in 1..4096");
  QD_REQUIRE(n >= 1, QD_ERR_INVALID, "empty sector");
  if (arnoldi_ground_res(H, psi, kdim, add_dim, extend, evals_out, res)) return;
  const int g = ev_grid(ctx, n);
  if (extend) {
    QD_REQUIRE(H->arnoldi_gs && H->arnoldi_gs->open && H->arnoldi_gs->kdim == kdim, QD_ERR_INVALID,
               "no open Arnoldi ground-state solve of krylov_dim %d on this operator", kdim);
  } else {
    if (!H->arnoldi_gs) H->arnoldi_gs.reset(new ArnoldiGround());
    ArnoldiGround& B = *H->arnoldi_gs;
    B.ensure(n, kdim, std::max(g, ev_tile_grid(ctx, n)), ctx->stream);
    B.act = 0;
    B.open = true;
    B.broke = false;
    // initKrylov: v_0 = psi / ||psi||
    ev_norm_only_kernel<<<g, kEvThreads, 0, ctx->stream>>>(n, psi, B.nrm2.p, GridRed<double>{B.rpart.p, B.tickets.p + 1});
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
    double n0 = 0.0;
    QD_CUDA(cudaMemcpyAsync(&n0, B.nrm2.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    QD_CUDA(cudaStreamSynchronize(ctx->stream));
    QD_REQUIRE(n0 > 0.0, QD_ERR_INVALID, "start vector is zero");
    ev_init_kernel<<<g, kEvThreads, 0, ctx->stream>>>(n, psi, B.nrm2.p, B.V.p);
    QD_CHECK_LAUNCH();
    QD_LAUNCHED(ctx);
    QD_CUDA(cudaMemsetAsync(B.stop.p, 0, sizeof(int), ctx->stream));
  }
  ArnoldiGround& B = *H->arnoldi_gs;
  // updateKrylovRepr: add_dim = -1 (here <= 0) or past kry_dim -> up to kry_dim
  int steps = (add_dim <= 0 || B.act + add_dim > kdim) ? kdim - B.act : add_dim;
  if (B.broke) steps = 0;  // a space that closed does not grow
  const int first = B.act + 1;
  if (steps > 0) {
    if (H->flags & QD_HAM_REAL)
      arnoldi_ground_steps<double>(H, H->vals_r.p, B, first, B.act + steps);
    else
      arnoldi_ground_steps<cplx>(H, H->vals_c.p, B, first, B.act + steps);
  }
  int stop = 0;
  QD_CUDA(cudaMemcpyAsync(&stop, B.stop.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  const int act_prev = B.act;
  if (steps > 0) {
    B.act = stop ? stop : B.act + steps;  // expandBasis<0>: the breaking step counts
    B.broke = stop != 0;
  }
  const int act = B.act;
  QD_REQUIRE(act >= 1, QD_ERR_INVALID, "no Krylov step was run");
  // lower triangle of KR[:act, :act]: Re <v_i, H v_i> and ||w_{i+1}||
  std::vector<cplx> hc((size_t)act * B.ldh);
  std::vector<double> nrm(act + 1);
  QD_CUDA(cudaMemcpyAsync(hc.data(), B.hcol.p, hc.size() * sizeof(cplx), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(nrm.data(), B.nrm.p, (act + 1) * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  std::vector<double> d(act), e(act), ev(act), y(act);
  for (int i = 0; i < act; ++i) {
    d[i] = hc[(size_t)i * B.ldh + i].re;
    e[i] = (i + 1 < act) ? nrm[i + 1] : 0.0;
  }
  QD_REQUIRE(tridiag_lowest<double>(act, d.data(), e.data(), ev.data(), y.data()) == 0, QD_ERR_INVALID,
             "tridiagonal eigensolver did not converge");
  std::vector<cplx> yc(act);
  for (int j = 0; j < act; ++j) yc[j] = mkc(y[j], 0.0);
  QD_CUDA(cudaMemcpyAsync(B.e.p, yc.data(), act * sizeof(cplx), cudaMemcpyHostToDevice, ctx->stream));
  ev_combine_long_kernel<<<ev_stream_grid(ctx, n), kEvThreads, 0, ctx->stream>>>(n, B.V.p, B.ld, act, B.e.p, psi);
  QD_CHECK_LAUNCH();
  QD_LAUNCHED(ctx);
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  if (evals_out) std::memcpy(evals_out, ev.data(), act * sizeof(double));
  res->act_dim = act;
  res->breakdown = B.broke ? 1 : 0;
  res->matvecs = act - act_prev;
  res->ritz_value = ev[0];
  res->err = std::fabs(ev[0]);
}

void ArnoldiGroundDeleter::operator()(ArnoldiGround* b) const { delete b; }

void ArnResDeleter::operator()(ArnRes* b) const { delete b; }

void ArnoldiDeleter::operator()(ArnoldiBuffers* b) const { delete b; }

}  // namespace qd
