// gridx.cuh -- data and sums across the blocks of one co-resident grid.
//
// The persistent Krylov kernels need a few small sums over the whole grid in
// every step, and the other blocks' rows of the newest vector.  A barrier
// (fence, atomic, poll) before each read costs four dependent trips to L2.
// Here the data is the signal: every slot is written once per launch and holds
// kXEmpty until then, and a reader takes a slot once it is filled.  No fence is
// needed (nothing is inferred about any other word), and nothing is reused, so
// no slot has to be emptied inside the launch: one memset before it fills all
// slots with kXEmptyByte.
//
// A sum over the grid goes through the cluster first: block r of a cluster adds
// its share of the values over the cluster's shared memories, posts them,
// collects the other clusters' and hands the totals to its peers.  With every
// block reading every block's sums the exchange of 60 values took 8,400 cycles
// at 77 blocks and 14,600 at 152 (the polls of one slot by every block queue up
// in L2); through clusters of eight it takes 4,000 at 64 blocks and 4,800 at
// 128, of which two cluster barriers are 1,200.
//
// Every wait is bounded: a thread that runs out of polls raises *abort and goes
// on with what it has, and so does, within 64 polls, every thread that finds it
// raised; the kernel runs to its end without waiting any more and the host
// discards the result.  (No block leaves early: its peers read its shared
// memory.  Within a cluster all blocks see the same sums, so they take the same
// branches even then.)
#pragma once

#include <cooperative_groups.h>

#include "vec.cuh"

namespace qd {

// No value is stored with these bits: as an integer it is below every value that x_sum_int posts,
// and a double that has them is stored with its last bit flipped.
constexpr int kXEmptyByte = 0x80;
constexpr unsigned long long kXEmpty = 0x8080808080808080ull;
constexpr unsigned kXPolls = 1u << 21;  // a second or two of polling
constexpr int kXAborted = 1;

struct GridX {
  int* abort;      // kXAborted once a wait ran out; anything else (kXEmptyByte at launch) before
  unsigned polls;  // poll limit
  int hold;        // test control: block 0 (and its cluster) posts nothing, so every wait runs out
};

__device__ __forceinline__ double x_ld(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void x_st(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool x_is_empty(double v) { return (unsigned long long)__double_as_longlong(v) == kXEmpty; }
__device__ __forceinline__ double x_clean(double v) {
  return x_is_empty(v) ? __longlong_as_double((long long)(kXEmpty ^ 1ull)) : v;
}

// One failed poll of a wait: true when the wait has run out (or another block's has).
__device__ __forceinline__ bool x_spent(const GridX& X, unsigned& polls) {
  if (++polls > X.polls) {
    atomicExch(X.abort, kXAborted);
    return true;
  }
  return (polls & 63u) == 0 && *reinterpret_cast<volatile int*>(X.abort) == kXAborted;
}
__device__ __forceinline__ bool x_wait(const GridX& X, const double* p, double& v) {
  unsigned polls = 0;
  while (x_is_empty(v)) {
    if (x_spent(X, polls)) return false;
    v = x_ld(p);
  }
  return true;
}

// Elements of a vector that other blocks write in this launch: stored clean, taken once filled.
__device__ __forceinline__ void x_put(double* p, double v) { x_st(p, x_clean(v)); }
__device__ __forceinline__ void x_put(cplx* p, cplx v) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(x_clean(v.re)), "d"(x_clean(v.im))
               : "memory");
}
__device__ __forceinline__ double x_peek(const double* p) { return x_ld(p); }
__device__ __forceinline__ cplx x_peek(const cplx* p) {
  cplx v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.re), "=d"(v.im) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool x_filled(double v) { return !x_is_empty(v); }
__device__ __forceinline__ bool x_filled(cplx v) { return !x_is_empty(v.re) && !x_is_empty(v.im); }
// 128-bit integers of magnitude below 2^125 as two words that are never kXEmpty: hi 2^63 + lo, 0 <= lo < 2^63.
struct __align__(16) XInt {
  unsigned long long lo;
  long long hi;
};
__device__ __forceinline__ void x_put(XInt* p, __int128 v) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p),
               "l"((unsigned long long)v & 0x7fffffffffffffffull), "l"((long long)(v >> 63))
               : "memory");
}
__device__ __forceinline__ XInt x_peek(const XInt* p) {
  XInt v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.lo), "=l"(v.hi) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool x_filled(XInt v) { return v.lo != kXEmpty && (unsigned long long)v.hi != kXEmpty; }
__device__ __forceinline__ __int128 x_value(XInt v) { return ((__int128)v.hi << 63) + v.lo; }

template <typename VV>
__device__ __forceinline__ bool x_await(const GridX& X, const VV* p, VV& v) {
  unsigned polls = 0;
  while (!x_filled(v)) {
    if (x_spent(X, polls)) return false;
    v = x_peek(p);
  }
  return true;
}

// out[q] = the sum over the grid of every block's v[q], q < nv <= kXMaxVals, the same bits in every
// block (fixed trees over the cluster's ranks and over the clusters).  kOne: a grid of one block.  v and out
// in shared memory, not overlapping; slots: gridDim.x * nv of them.  v must be complete for all threads, as
// by a block barrier, before the call; out is complete for all threads on return, and v may then be
// written again.  The cluster's size is read, not assumed: a profiler launches a cooperative grid
// without its clusters, and the memory of a rank that does not exist must not be read.
constexpr int kXMaxVals = 256;
template <int CT>  // the cluster's size, 0: any power of two
__device__ __forceinline__ void x_sum_cluster(const GridX& X, double* slots, double* v, int nv, double* out, int size) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int C = CT ? CT : size, tid = threadIdx.x;
  const int rank = (int)cl.block_rank(), ncl = (int)gridDim.x / C, me = (int)blockIdx.x / C;
  const int per = (nv + C - 1) / C;  // values per block
  cl.sync();
  // a value takes C lanes, or a warp where there are many clusters to collect from
  const int L = ncl > 2 * C ? 32 : C;
  const int l = tid & (L - 1);
  for (int g = tid / L; (g & ~(32 / L - 1)) < per; g += blockDim.x / L) {  // whole warps
    const int q = rank * per + g;
    const bool on = g < per && q < nv;
    double a = (on && l < C) ? *cl.map_shared_rank(v + q, l) : 0.0;
#pragma unroll
    for (int o = C / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (ncl > 1) {
      if (on && l == 0 && !(X.hold && me == 0)) x_st(slots + (size_t)me * nv + q, x_clean(a));
      double t = 0.0;
      if (on)
        for (int c = l; c < ncl; c += L) {
          double b = x_ld(slots + (size_t)c * nv + q);
          x_wait(X, slots + (size_t)c * nv + q, b);
          t += b;
        }
      for (int o = L / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      a = t;
    }
    if (on && l < C) *cl.map_shared_rank(out + q, l) = a;
  }
  cl.sync();
}

template <bool kOne>
__device__ __forceinline__ void x_sum(const GridX& X, double* slots, double* v, int nv, double* out) {
  if constexpr (kOne) {
    __syncthreads();
    if (threadIdx.x < nv) out[threadIdx.x] = v[threadIdx.x];
    __syncthreads();
  } else {
    const int size = (int)cooperative_groups::this_cluster().num_blocks();
    if (size == 8) x_sum_cluster<8>(X, slots, v, nv, out, size);
    else if (size == 4) x_sum_cluster<4>(X, slots, v, nv, out, size);
    else x_sum_cluster<0>(X, slots, v, nv, out, size);
  }
}

}  // namespace qd
