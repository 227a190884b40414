// arnres.cuh -- the Arnoldi recurrence in one persistent launch (arnres.cu).
#pragma once

#include "ham.cuh"

namespace qd {

// Most basis vectors the persistent recurrence orthogonalises against.
constexpr int kArnMaxVecs = 96;
// Most Krylov columns whose exponential is formed on the device.
constexpr int kArnMaxExp = 32;

// What the host reads back after a run, and the exchange slots' neighbour (one
// memset prepares both).
struct ArnStatus {
  int abort;      // kXAborted: a bounded wait ran out
  int stop;       // the breaking step (0: none)
  int need_host;  // the exponential is left to the host (its norm is large or not finite)
  int zero;       // the start vector's norm is not positive
  double alpha[kArnMaxVecs + 2];  // real part of <v_i, H v_i> of column i
  double nrm[kArnMaxVecs + 2];    // ||w_idx||, idx = 1 .. (0: the start vector's)
  double scl[kArnMaxVecs + 2];    // basis vector j is scl[j] V[j]
};

// Buffers of the persistent recurrence on one Hamiltonian.
struct ArnRes {
  int64_t n = 0, ld = 0;
  int kdim = 0;        // columns V holds beyond the start
  bool real_v = false; // V holds reals
  int ncl = 0, rows = 0;  // clusters of the grid and rows per block (0: not chosen yet)
  DBuf<char> V;        // (kdim + 1) x ld, unnormalised
  DBuf<cplx> out;      // the evolved state before it replaces the caller's
  DBuf<cplx> hcol;     // Hessenberg column i at i * (kArnMaxVecs + 1)
  DBuf<char> slots;    // ArnStatus, then the exchange slots (gridx.cuh)
  ArnStatus host{};    // the last run's status
  int act = 0;
  bool open = false;   // a solve that a later call may grow
  bool broke = false;  // the last step broke down
  bool real_start = false;
};

// Whether the persistent recurrence takes this operator and Krylov dimension.
bool arn_res_fits(qd_ham* H, int kdim);
// psi_out = V exp(-i h K) e_0 (ArnoldiSolver<T, 0>::evolve); false: not launched.
bool arn_res_evolve(qd_ham* H, ArnRes& B, const cplx* psi_in, cplx* psi_out, double h, int steps, int* act_out);
// Steps first .. last of the ground-state recurrence (first = 1 starts from psi).
bool arn_res_steps(qd_ham* H, ArnRes& B, const cplx* psi, int kdim, bool real_v, int first, int last);

}  // namespace qd
