// gspass.cuh -- Gram-Schmidt passes over a stored Krylov basis (gspass.cu).
#pragma once

#include "ham.cuh"
#include "vec.cuh"

namespace qd {

// A Krylov basis in memory: unnormalised vectors, their scales, and their 55-bit copies with one scale
// per tile of rows.  The copies are optional (twice the basis's memory): without them the passes form
// them again as they load the vectors, with the same results.
struct GsBasis {
  int64_t n = 0, ld = 0;
  int vecs = 0;
  int rpl = 0;          // rows per lane of a tile: tiles of 32 rpl rows
  int64_t ntiles = 0;
  int grid = 0;
  DBuf<cplx> V;         // vecs x ld
  DBuf<int4> Vq;        // the same quantised, or empty
  DBuf<double> u;       // vecs x ntiles scales of the quantised tiles
  DBuf<cplx> w;         // H v
  DBuf<cplx> coef;      // coefficients on the stored vectors: first pass, second pass
  DBuf<double> scl;     // 1 / ||V_j||
  DBuf<double> nrm;     // norms before normalisation
  DBuf<double> dots;    // a Hermitian step's <V, w>, warp by warp of the product; empty: another product
  DBuf<double> partials;
  DBuf<unsigned> ticket;
  DBuf<int> stop;       // first step whose norm fell below 1e-10, 0 while there is none
  cplx* vec(int j) const { return V.p + (int64_t)j * ld; }
  int64_t bytes() const {
    return (int64_t)(V.bytes() + Vq.bytes() + u.bytes() + w.bytes() + coef.bytes() + partials.bytes());
  }
  // True if the buffers moved.
  bool ensure(Ctx* ctx, int64_t n_, int vecs_, bool herm, bool copies);
};

// V_0 = psi, its norm and scale; clears stop.
void gs_begin(Ctx* ctx, GsBasis& B, const cplx* psi);
// V_idx = H v_{idx-1} with its components on V_0 .. V_{idx-1} removed; hcol[j] = <v_j, H v_{idx-1}>.
void gs_step(qd_ham* H, GsBasis& B, int idx, cplx* hcol);

}  // namespace qd
