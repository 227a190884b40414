// mfrow.cuh -- ranking a target state of the compiled transitions (mfree.cu), for the kernels that form a
// row of a product from them.
#pragma once

#include "ham.cuh"

namespace qd {

// What a row needs: its state, the transitions, and the ranking of the sector.
struct MfRows {
  int64_t dim;
  const uint64_t* basis;
  const MfEntry* ent;
  int nent;
  int use_tables;
  MfRank rk;
  SectorView S;
};

inline MfRows mf_rows(const qd_ham* H) {
  MfRows M{};
  M.dim = H->dim;
  M.basis = H->sec->basis.p;
  M.ent = H->mf_ent.p;
  M.nent = H->mf_nent;
  M.use_tables = H->mf_tables ? 1 : 0;
  M.rk = H->mf_rank;
  M.S = H->sec->view;
  return M;
}

// Ranking in 32 bits for registers of at most 32 bits ranked by tables (every model of the configurations):
// states, masks and table entries in 32-bit integers.
struct Mf32 {
  int nf;  // 0: not this form
  int lo[2], k[2], nb[2];
  uint32_t wmask[2];
  uint32_t stride[2];
  int off[2];
  const uint32_t* tab;
};
// The 32-bit form where the register has at most 32 bits, the sector is a product of at most two fields and
// the dimension fits in 32 bits (ham_build_matrix_free has run).
bool mf32_prepare(const qd_ham* H, Mf32& R);

#ifdef __CUDACC__
// The rank of state c into col; false, with no table read, when it is not in the sector (the tables end at k
// set bits).  NF fields, 0: one or two.
template <int NF = 0>
__device__ __forceinline__ bool mf_rank32(const Mf32& R, uint32_t c, uint32_t& col) {
  bool in = __popc((c >> R.lo[0]) & R.wmask[0]) == R.k[0];
  if (NF == 2 || (NF == 0 && R.nf > 1)) in &= __popc((c >> R.lo[1]) & R.wmask[1]) == R.k[1];
  if (!in) return false;
  col = 0;
#pragma unroll
  for (int f = 0; f < (NF ? NF : 2); ++f) {
    if (NF == 0 && f >= R.nf) break;
    const uint32_t v = (c >> R.lo[f]) & R.wmask[f];
    const uint32_t* T = R.tab + R.off[f];
    const int kk = R.k[f] + 1;
    uint32_t a = __ldg(T + (v & 255u) * kk);
    int cb = __popc(v & 255u);
    if (R.nb[f] > 1) {
      a += __ldg(T + (256u + ((v >> 8) & 255u)) * kk + cb);
      cb += __popc((v >> 8) & 255u);
    }
    if (R.nb[f] > 2) {
      a += __ldg(T + (512u + ((v >> 16) & 255u)) * kk + cb);
      cb += __popc((v >> 16) & 255u);
    }
    if (R.nb[f] > 3) a += __ldg(T + (768u + (v >> 24)) * kk + cb);
    col += a * R.stride[f];
  }
  return true;
}

// The rank of state c, A.dim or more when it is not in the sector.
template <typename Args>
__device__ __forceinline__ int64_t mf_rank(const Args& A, uint64_t c) {
  if (!A.use_tables) return sector_rank(A.S, c);
  int64_t r = 0;
  for (int f = 0; f < A.rk.nf; ++f) {
    const int w = A.rk.width[f];
    const uint64_t v = (c >> A.rk.lo[f]) & ((w >= 64) ? ~0ull : ((1ull << w) - 1));
    if (A.rk.is_free[f]) {
      r += (int64_t)v * A.rk.stride[f];
      continue;
    }
    const int k = A.rk.k[f];
    if (__popcll(v) != k) return A.dim;
    const int64_t* T = A.rk.tab + A.rk.off[f];
    int64_t acc = 0;
    int cb = 0;
    for (int b = 0; b < A.rk.nb[f]; ++b) {
      const unsigned byte = (unsigned)(v >> (8 * b)) & 255u;
      acc += __ldg(T + ((int64_t)b * 256 + byte) * (k + 1) + cb);
      cb += __popc(byte);
    }
    r += acc * A.rk.stride[f];
  }
  return r;
}

__device__ __forceinline__ double amp_of(double*, cplx a) { return a.re; }
__device__ __forceinline__ cplx amp_of(cplx*, cplx a) { return a; }
__device__ __forceinline__ double vneg(double a) { return -a; }
__device__ __forceinline__ cplx vneg(cplx a) { return mkc(-a.re, -a.im); }
#endif

}  // namespace qd
