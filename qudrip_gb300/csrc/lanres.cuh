// lanres.cuh -- the Lanczos recurrence in one persistent launch (lanres.cu).
#pragma once

#include "krylov.cuh"

namespace qd {

// Above this |h| 3 ||H||_inf (a bound of ||h T||_inf, T the Krylov matrix) the exponential is the host's: the
// device's Taylor sub-steps, one for each unit of the norm, take longer than scaling and squaring from about
// here on (a step of m = 32 at dim 3,432: 0.40, 0.72 and 1.96 ms at 64, 256 and 1,000 on the device, 0.63 ms
// with the host's at 1,030).
constexpr double kLanMaxTheta = 256.0;

enum LanForm { kLanLocal = 0, kLanPaige = 1 };

// Steps first .. last of the recurrence on the basis V (V[first - 1] and, past the first step, V[first - 2]
// complete; scl[first - 1] known):
//   kLanLocal  the reference's local orthogonalisation against two vectors (sparse_algorithm.hpp:395-425)
//   kLanPaige  alpha = <v1, H v1>, beta = ||V1|| (Hermitian::LanczosSolver; the Krylov exponential)
// with the stopping rule norm < stop_below (*stop = the step).  `form`: the uniform-coupling form whose
// fixed-point sums the product keeps (real vectors), or null for the FP64 product.  `mf`: the product's
// columns and values from the compiled transitions (kLanLocal; ham_build_matrix_free has run).
template <typename MV, typename VV>
struct LanRun {
  const MV* vals;
  LanForm rule;
  bool mf;
  const FxForm* form;
  VV* V;
  int64_t ld;
  int kdim, first, last;
  double stop_below;
  VV *alpha, *beta;  // alpha[k], beta[k] of step k (beta may be null)
  double *nrm, *scl;
  int* stop;
  int* flags;        // [0] a vector left the fixed-point range, [1] a wait ran out (both 0 before)
  DBuf<double>* slots;
};
template <typename MV, typename VV>
bool lan_res_run(qd_ham* H, const LanRun<MV, VV>& r);

// Sectors of so few rows run on one block, which waits for no other.
constexpr int64_t kLanOneBlock = 64;

// One Krylov step out <- V exp(-i h T) e_0 of dimension kdim (<= 32) from psi; out may be psi.  A run whose wait
// runs out leaves rows of two times in out.  act and the product count are written on the device.  False:
// nothing launched.
template <typename MV>
bool lan_res_evolve(qd_ham* H, const MV* vals, const cplx* psi, cplx* out, cplx* V, int64_t ld, int kdim, double h,
                    int* act, long long* matvecs, int* flags, DBuf<double>* slots);

}  // namespace qd
