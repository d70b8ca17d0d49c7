// rowsolve.cuh -- row sweeps (lines along j, contiguous in memory) staged in
// shared memory: one CTA of NT threads per row.
//
// The chunks of the partition method (linesolve.cuh) make neighbouring
// threads walk stretches of a row a chunk apart, so a load of the row
// generation's stencil touches a sector per lane (26 sectors per request, the
// L1 60% busy). Here the rows are generated with neighbouring threads on
// neighbouring cells, a cell's operands in one round of memory latency, and
// written to shared memory; the chunks are walked there in odd lengths
// (distinct banks) and reduced by shuffles with one barrier (cta_solve), and
// the solution and the segments' ends are emitted with neighbouring threads
// on neighbouring cells. What bounds it is the latency of a row's rounds of
// loads times the rounds of CTAs: the FP64 rows are kept normalised (three
// arrays) so that seven of 1023 cells share an SM and 2047 of them take two
// rounds (four arrays, six rows, three rounds: 0.107 ms, hydraulic). The solve
// itself is a tenth of the time, the rounds of loads half (ablation). On
// 2048x1024, from the chunks in global memory: hydraulic y sweep 0.148 ->
// 0.080 ms (FP64; the FP32 forms' has its own solver, pairgen.cuh); the
// concentration y sweep, whose rows a per-cell kernel wrote to four arrays
// first, 0.126 -> 0.084 in FP64, 0.079 -> 0.062 in FP32, 0.108 -> 0.072 refined.
//
// REFINE: the rows stay in shared memory as they are; the residual is taken
// in FP64 and the correction solved from them again.
#pragma once

#include <climits>
#include <type_traits>

#include "common.cuh"
#include "linesolve.cuh"
#include "partsolve.cuh"

namespace hyd {

// Rows normalised to a unit diagonal (a = A/B, c = C/B, d = D/B: one array
// less) in FP64. In FP32 their rounding would add to the result's error (the
// concentration's 2.0e-7 -> 2.5e-7 against 64 bits after ten steps), and the
// fourth array costs no resident CTA.
template <class Gen>
constexpr bool row_normal() {
  return sizeof(typename Gen::Real) == 8;
}

// The separators' reduction of the plain FP32 form is done in FP64: its levels are
// what the chunks in global memory did not have as many of, and in FP32 they
// added to the result's error (the concentration against 64 bits after 20 steps of
// 64x32 1.0e-7 -> 1.9e-7 of its norm, 256x128 1.3e-7 -> 1.6e-7; so 0.8e-7 and
// 1.0e-7), for no time that shows: 64 against 62..64 us, 2048x1024. (The refined
// form's correction takes the error out anyway.)
template <class Gen>
using reduce_t = std::conditional_t<Gen::REFINE, typename Gen::Real, double>;

// arrays of a row's cells in shared memory: a, c, d or A, C, D, B; with
// refinement also v', c' and the first solution
template <class Gen>
constexpr int row_arrays() {
  return Gen::REFINE ? 7 : (row_normal<Gen>() ? 3 : 4);
}

template <class Gen>
inline size_t row_smem(int ncells) {
  return (size_t)row_arrays<Gen>() * ncells * sizeof(typename Gen::Real);
}

// CTAs per SM the kernel is compiled for: registers of 72 per thread in FP64,
// 64 in FP32
template <class R, int NT>
constexpr int row_min_blocks() {
  constexpr int b = (sizeof(R) == 8 ? 896 : 1024) / NT;
  return b < 1 ? 1 : (b > 24 ? 24 : b);
}

// [p, p + n) towards L2, in whole 16-byte units (p is inside an array, and so
// is what follows it)
template <class T>
__device__ __forceinline__ void prefetch_l2(const T* p, int n) {
  const uintptr_t a = (uintptr_t)p & ~(uintptr_t)15;
  const unsigned bytes = (unsigned)(((uintptr_t)(p + n) - a) & ~(uintptr_t)15);
  if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(bytes) : "memory");
}

// The segment a walk over increasing positions is at, held in registers: the
// first one that ends (END: its last cell, else its last unknown) at or after
// the position.
template <bool END>
struct SegWalk {
  int si = -1, lo = 0, hi = -1;
  SegD d;
  __device__ bool at(const LineSeg& LS, int pos) {
    while (hi < pos) {
      if (++si < LS.nseg) {
        d = LS.s[si];
        lo = END ? d.first : d.off;
        hi = END ? d.last : d.rend;
      } else {
        lo = hi = INT_MAX;
      }
    }
    return lo <= pos;
  }
};

// Line blockIdx.x of member blockIdx.y.
template <class Gen, int NT, int BATCH>
__global__ void __launch_bounds__(NT, row_min_blocks<typename Gen::Real, NT>())
    k_row_solve(Gen G0, Batch<typename Gen::Real> bt) {
  step_begin<BATCH>();
  using R = typename Gen::Real;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LineSeg LS;
  __shared__ reduce_t<Gen> blk[NT / 32 + 1][8];
  auto solve = [&](const Gen& G) {
    const int tid = threadIdx.x, nc = G.cells_per_line(), lp = G.line_pos(blockIdx.x);
    R* rA = reinterpret_cast<R*>(smem_raw);
    R* rC = rA + nc;
    R* rD = rC + nc;
    R* rB = rD + nc;  // (where the rows are not normalised)
    // the row's own new field rows towards L2 at once, so that the rounds of
    // loads after the first find them there (0.115 -> 0.107 ms, hydraulic)
    if (tid == 0) G.prefetch(lp);
    // the first cell's operands and the segment table in one round
    typename Gen::Ops o;
    if (tid < nc) o = G.load(lp, tid + 2);
    for (int e = tid; e < SEG + 1; e += NT) G.load_segment(LS, blockIdx.x, e);
    __syncthreads();
    SegWalk<false> w;
    for (int c = tid; c < nc;) {
      const int pos = c + 2;
      R A = 0, B = 1, C = 0, D = 0;
      if (w.at(LS, pos)) {
        G.row(w.d, lp, pos, o, A, B, C, D);
        G.keep(w.d, lp, pos, o);
        if constexpr (row_normal<Gen>()) {
          const R m = R(1) / B;
          A *= m;
          C *= m;
          D *= m;
        }
      }
      rA[c] = A;
      rC[c] = C;
      rD[c] = D;
      if constexpr (!row_normal<Gen>()) rB[c] = B;
      c += NT;
      if (c < nc) o = G.load(lp, c + 2);
    }
    __syncthreads();
    R* X = rD;
    if constexpr (!Gen::REFINE) {
      cta_solve<R, NT>(rA, rC, rD, nc, blk, [&](int q, R& A, R& B, R& C, R& D) {
        A = rA[q];
        B = row_normal<Gen>() ? R(1) : rB[q];
        C = rC[q];
        D = rD[q];
      });
    } else {
      R* wV = rB + nc;
      R* wC = wV + nc;
      X = wC + nc;
      auto rows = [&](int q, R& A, R& B, R& C, R& D) {
        A = rA[q];
        B = rB[q];
        C = rC[q];
        D = rD[q];
      };
      cta_solve<R, NT>(wV, wC, X, nc, blk, rows);
      __syncthreads();
      for (int c = tid; c < nc; c += NT) {
        const double xm = c > 0 ? X[c - 1] : R(0), xp = c + 1 < nc ? X[c + 1] : R(0);
        rD[c] = (R)((double)rD[c] - (double)rA[c] * xm - (double)rB[c] * (double)X[c] -
                    (double)rC[c] * xp);
      }
      __syncthreads();
      cta_solve<R, NT>(wV, wC, rD, nc, blk, rows);
    }
    __syncthreads();
    // the solution at position p
    auto value = [&](int p) {
      if constexpr (Gen::REFINE) return (double)X[p - 2] + (double)rD[p - 2];
      else return (double)rD[p - 2];
    };
    SegWalk<true> e;
    for (int pos = tid + 2; pos < nc + 2; pos += NT)
      if (e.at(LS, pos)) G.emit_cell(e.d, lp, pos, value);
  };
  if constexpr ((BATCH & 1) != 0) {
    Gen Gm = G0;
    Gm.bind(bt.S[blockIdx.y], bt.c[blockIdx.y]);
    solve(Gm);
  } else {
    solve(G0);
  }
}

}  // namespace hyd
