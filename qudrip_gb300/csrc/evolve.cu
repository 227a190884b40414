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
// per previous vector.  On the device a pass projects on all of them at once,
// applied twice (classical Gram-Schmidt with reorthogonalisation, gspass.cu):
// the same projector up to rounding, with better orthogonality, in 4 launches
// per step instead of 2 * idx.  The small exponential runs on the host
// (dense.h).  This form serves the requests of the serving loop and sectors too
// large for the persistent recurrence (arnres.cu), which takes all other calls.
#include <algorithm>
#include <cstring>
#include <vector>

#include "arnres.cuh"
#include "dense.h"
#include "tridiag.cuh"
#include "evolve.cuh"
#include "gspass.cuh"
#include "krylov.cuh"
#include "spmv.cuh"

namespace qd {

constexpr int kEvThreads = 256;

// Grid of the streaming kernels (update, norm, scale, combination): eight blocks per SM.
static int ev_stream_grid(Ctx* ctx, int64_t n) {
  const int64_t want = ceil_div(n, kEvThreads);
  return (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 8));
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

// Columns first .. last of the recurrence on B.
static void arnoldi_steps(qd_ham* H, GsBasis& B, cplx* hcol, int ldh, int first, int last) {
  for (int idx = first; idx <= last; ++idx) gs_step(H, B, idx, hcol + (int64_t)(idx - 1) * ldh);
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
  if (B.basis.ensure(ctx, n, m, (H->flags & QD_HAM_HERMITIAN) && !H->spmv_chosen, !H->one_shot)) B.drop_graph();  // the buffers moved
  if (!B.hcol.p) {
    B.hcol.alloc((size_t)33 * 64);
    B.e.alloc(64);
  }
  gs_begin(ctx, B.basis, psi_in);
  const int steps = m - 1;  // updateKrylovRepr(H, kry_dim_rt - 1)
  const bool real = (H->flags & QD_HAM_REAL) != 0;
  auto run_steps = [&]() { arnoldi_steps(H, B.basis, B.hcol.p, 64, 1, steps); };
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
  std::vector<cplx> hc((size_t)steps * 64);
  std::vector<double> nrm(m), scl(m);
  int stop = 0;
  QD_CUDA(cudaMemcpyAsync(hc.data(), B.hcol.p, hc.size() * sizeof(cplx), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(nrm.data(), B.basis.nrm.p, m * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(scl.data(), B.basis.scl.p, m * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(&stop, B.basis.stop.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
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
  for (int j = 0; j < act; ++j) e[j] = mkc(E[j].real() * scl[j], E[j].imag() * scl[j]);  // V_j is unnormalised
  QD_CUDA(cudaMemcpyAsync(B.e.p, e.data(), act * sizeof(cplx), cudaMemcpyHostToDevice, ctx->stream));
  launch_ev_combine(ctx, n, B.basis.V.p, B.basis.ld, act, B.e.p, psi_out);
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

// The persistent form of arnoldi_ground (arnres.cu).  False, with nothing run, when it does not take
// the solve; a solve that it began it also continues.
static bool arnoldi_ground_res(qd_ham* H, cplx* psi, int kdim, int add_dim, bool extend, double* evals_out,
                               qd_lanczos_result* res) {
  Ctx* ctx = H->ctx;
  if (!extend) {
    if (H->arn_gs) H->arn_gs->open = false;
    if (H->arnoldi_gs) H->arnoldi_gs->open = false;
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
  if (extend) {
    QD_REQUIRE(H->arnoldi_gs && H->arnoldi_gs->open && H->arnoldi_gs->kdim == kdim, QD_ERR_INVALID,
               "no open Arnoldi ground-state solve of krylov_dim %d on this operator", kdim);
  } else {
    if (!H->arnoldi_gs) H->arnoldi_gs.reset(new ArnoldiGround());
    ArnoldiGround& B = *H->arnoldi_gs;
    B.open = false;
    B.basis.ensure(ctx, n, kdim + 1, (H->flags & QD_HAM_HERMITIAN) && !H->spmv_chosen, !H->one_shot);
    if (B.kdim != kdim) {
      B.kdim = 0;
      B.ldh = kdim + 1;
      B.hcol.alloc((size_t)kdim * B.ldh);
      B.e.alloc(kdim + 1);
      B.kdim = kdim;
    }
    B.act = 0;
    B.open = true;
    B.broke = false;
    gs_begin(ctx, B.basis, psi);  // initKrylov: v_0 = psi / ||psi||
    double n0 = 0.0;
    QD_CUDA(cudaMemcpyAsync(&n0, B.basis.nrm.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    QD_CUDA(cudaStreamSynchronize(ctx->stream));
    QD_REQUIRE(n0 > 0.0, QD_ERR_INVALID, "start vector is zero");
  }
  ArnoldiGround& B = *H->arnoldi_gs;
  // updateKrylovRepr: add_dim = -1 (here <= 0) or past kry_dim -> up to kry_dim
  int steps = (add_dim <= 0 || B.act + add_dim > kdim) ? kdim - B.act : add_dim;
  if (B.broke) steps = 0;  // a space that closed does not grow
  const int first = B.act + 1;
  if (steps > 0) arnoldi_steps(H, B.basis, B.hcol.p, B.ldh, first, B.act + steps);
  int stop = 0;
  QD_CUDA(cudaMemcpyAsync(&stop, B.basis.stop.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
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
  std::vector<double> nrm(act + 1), scl(act);
  QD_CUDA(cudaMemcpyAsync(hc.data(), B.hcol.p, hc.size() * sizeof(cplx), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(nrm.data(), B.basis.nrm.p, (act + 1) * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaMemcpyAsync(scl.data(), B.basis.scl.p, act * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  QD_CUDA(cudaStreamSynchronize(ctx->stream));
  std::vector<double> d(act), e(act), ev(act), y(act);
  for (int i = 0; i < act; ++i) {
    d[i] = hc[(size_t)i * B.ldh + i].re;
    e[i] = (i + 1 < act) ? nrm[i + 1] : 0.0;
  }
  QD_REQUIRE(tridiag_lowest<double>(act, d.data(), e.data(), ev.data(), y.data()) == 0, QD_ERR_INVALID,
             "tridiagonal eigensolver did not converge");
  std::vector<cplx> yc(act);
  for (int j = 0; j < act; ++j) yc[j] = mkc(y[j] * scl[j], 0.0);  // V_j is unnormalised
  QD_CUDA(cudaMemcpyAsync(B.e.p, yc.data(), act * sizeof(cplx), cudaMemcpyHostToDevice, ctx->stream));
  ev_combine_long_kernel<<<ev_stream_grid(ctx, n), kEvThreads, 0, ctx->stream>>>(n, B.basis.V.p, B.basis.ld, act, B.e.p, psi);
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
