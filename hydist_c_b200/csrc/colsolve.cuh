// colsolve.cuh -- column sweeps (lines along i) staged in shared memory: one
// CTA of NT threads per L adjacent columns (a 32-byte sector of them).
//
// As the row sweeps (rowsolve.cuh), with L systems interleaved: cell r of
// column l at r*L + l, generated with neighbouring threads on neighbouring
// cells of a row, L at a time, and the CTAs all move down their columns
// together, so that the SMs read a few rows of each field at a time, where a
// thread per chunk of a column walks rows all over every field. In the solve
// thread k*L + l takes chunk k of column l; a warp reduces its 32/L chunks per column by shuffles,
// the warps' last separators are solved by one warp per column. (What it
// takes on which meshes, against the chunks in global memory: sweep.cu.)
#pragma once

#include "common.cuh"
#include "linesolve.cuh"
#include "partsolve.cuh"
#include "rowsolve.cuh"

namespace hyd {

template <class Gen, int L>
inline size_t col_smem(int ncells) {
  return (size_t)row_arrays<Gen>() * ncells * L * sizeof(typename Gen::Real);
}

// what the warps give each other in a solve of L interleaved systems
template <class T, int NT, int L>
struct ColShared {
  T blk[7][L][NT / 32 + 1];
  T x[L][NT / 32];
};

// tile_reduce of L interleaved systems, one chunk per thread.
template <class T, int NT, int L>
__device__ __forceinline__ void cols_reduce(const ChunkEnds<T>& e, ColShared<T, NT, L>& sh, T& x, T& xl) {
  constexpr unsigned full = 0xffffffffu;
  constexpr int W = NT / 32, NC = 32 / L;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l = lane % L, k = lane / L;  // column, chunk within the warp
  const T nyF = __shfl_down_sync(full, e.yF, L), nvF = __shfl_down_sync(full, e.vF, L),
          nwF = __shfl_down_sync(full, e.wF, L);
  const T ra = e.as * e.vL, rb = e.bs + e.as * e.wL, rd = e.ds - e.as * e.yL;
  const bool lastk = k == NC - 1;
  const T cs = lastk ? T(0) : e.cs;
  const T inv = T(1) / (rb + cs * nvF);
  T a = ra * inv, c = cs * nwF * inv, d = (rd - cs * nyF) * inv;
  // (the warp's last chunk per column holds its separator, completed below)
  if (lastk) a = c = d = 0;
#pragma unroll
  for (int st = 1; st < NC; st <<= 1) pcr_level(a, c, d, st * L, k >= st, k + st < NC - 1);
  {
    const T ap = __shfl_up_sync(full, a, L), cp = __shfl_up_sync(full, c, L), dp = __shfl_up_sync(full, d, L);
    if (k == 0) {
      sh.blk[0][l][warp] = e.yF + e.wF * d;
      sh.blk[1][l][warp] = e.vF - e.wF * a;
      sh.blk[2][l][warp] = -e.wF * c;
    }
    if (lastk) {
      sh.blk[3][l][warp] = -ra * ap;
      sh.blk[4][l][warp] = rb - ra * cp;
      sh.blk[5][l][warp] = e.cs;
      sh.blk[6][l][warp] = rd - ra * dp;
    }
  }
  __syncthreads();
  // the warps' separators of column col, lane w the one of warp w
  for (int col = warp; col < L; col += W) {
    T A = 0, B = 1, C = 0, D = 0;
    if (lane < W) {
      A = sh.blk[3][col][lane];
      B = sh.blk[4][col][lane];
      C = sh.blk[5][col][lane];
      D = sh.blk[6][col][lane];
      if (lane + 1 < W) {
        B += C * sh.blk[1][col][lane + 1];
        D -= C * sh.blk[0][col][lane + 1];
        C *= sh.blk[2][col][lane + 1];
      } else {
        C = 0;
      }
    }
    const T m = T(1) / B;
    A *= m;
    C *= m;
    D *= m;
#pragma unroll
    for (int st = 1; st < W; st <<= 1) pcr_level(A, C, D, st, lane >= st, lane + st < W);
    if (lane < W) sh.x[col][lane] = D;
  }
  __syncthreads();
  const T XL = warp > 0 ? sh.x[l][warp - 1] : T(0), XR = sh.x[l][warp];
  x = lastk ? XR : d - a * XL - c * XR;
  xl = __shfl_up_sync(full, x, L);
  if (k == 0) xl = XL;
}

// cta_solve of L interleaved systems of n rows each
template <class T, int NT, int L, class W, class Row>
__device__ __forceinline__ void cols_solve(T* oV, T* oC, T* X, int n, ColShared<W, NT, L>& sh, Row row) {
  const int l = threadIdx.x % L, t = threadIdx.x / L;
  int S = (n + NT / L - 1) / (NT / L);
  S = (S < 3 ? 3 : S) | 1;
  const int P = max(1, n / S), q0 = t * S;
  const int nu = t < P ? (t == P - 1 ? n - q0 : S) : 0;
  ChunkEnds<T> e;
  T cp = 0, yp = 0, vp = 0;
  for (int s = 0; s < nu - 1; ++s) {
    const int o = (q0 + s) * L + l;
    T A, B, C, D;
    row(o, A, B, C, D);
    const T m = T(1) / (s == 0 ? B : B - A * cp);
    yp = (s == 0 ? D : D - A * yp) * m;
    vp = (s == 0 ? -A : -A * vp) * m;
    cp = C * m;
    oC[o] = cp;
    X[o] = yp;
    oV[o] = vp;
    e.yF += e.wF * yp;
    e.vF += e.wF * vp;
    e.wF *= -cp;
  }
  if (nu > 0) row((q0 + nu - 1) * L + l, e.as, e.bs, e.cs, e.ds);
  e.yL = yp;
  e.vL = vp;
  e.wL = -cp;
  W wx, wxl;
  cols_reduce<W, NT, L>(ends_as<W>(e), sh, wx, wxl);
  const T x = (T)wx, xl = (T)wxl;
  if (nu > 0) {
    X[(q0 + nu - 1) * L + l] = x;
    T xn = x;
#pragma unroll 4
    for (int q = q0 + nu - 2; q >= q0; --q) {
      const int o = q * L + l;
      const T xq = X[o] + oV[o] * xl - oC[o] * xn;
      X[o] = xq;
      xn = xq;
    }
  }
}

// Columns blockIdx.x*L .. + L - 1 of member blockIdx.y.
template <class Gen, int NT, int L, int BATCH>
__global__ void __launch_bounds__(NT, 1024 / NT < 1 ? 1 : (sizeof(typename Gen::Real) == 8 && NT < 1024 ? 768 : 1024) / NT)
    k_col_solve(Gen G0, Batch<typename Gen::Real> bt) {
  step_begin<BATCH>();
  using R = typename Gen::Real;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ LineSeg seg[L];
  __shared__ ColShared<reduce_t<Gen>, NT, L> sh;
  auto solve = [&](const Gen& G) {
    const int tid = threadIdx.x, nc = G.cells_per_line(), l = tid % L, r0 = tid / L;
    const int line = blockIdx.x * L + l;
    const bool act = line < G.lines();
    const int lp = G.line_pos(line);
    R* rA = reinterpret_cast<R*>(smem_raw);
    R* rC = rA + nc * L;
    R* rD = rC + nc * L;
    R* rB = rD + nc * L;  // (where the rows are not normalised)
    typename Gen::Ops o;
    if (act && r0 < nc) o = G.load(lp, r0 + 2);
    for (int e = tid; e < L * (SEG + 1); e += NT)
      G.load_segment(seg[e / (SEG + 1)], blockIdx.x * L + e / (SEG + 1), e % (SEG + 1));
    __syncthreads();
    const LineSeg& LS = seg[l];
    SegWalk<false> w;
    for (int r = r0; r < nc;) {
      const int pos = r + 2, q = r * L + l;
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
      rA[q] = A;
      rC[q] = C;
      rD[q] = D;
      if constexpr (!row_normal<Gen>()) rB[q] = B;
      r += NT / L;
      if (act && r < nc) o = G.load(lp, r + 2);
    }
    __syncthreads();
    R* X = rD;
    if constexpr (!Gen::REFINE) {
      cols_solve<R, NT, L>(rA, rC, rD, nc, sh, [&](int q, R& A, R& B, R& C, R& D) {
        A = rA[q];
        B = row_normal<Gen>() ? R(1) : rB[q];
        C = rC[q];
        D = rD[q];
      });
    } else {
      R* wV = rB + nc * L;
      R* wC = wV + nc * L;
      X = wC + nc * L;
      auto rows = [&](int q, R& A, R& B, R& C, R& D) {
        A = rA[q];
        B = rB[q];
        C = rC[q];
        D = rD[q];
      };
      cols_solve<R, NT, L>(wV, wC, X, nc, sh, rows);
      __syncthreads();
      for (int r = r0; r < nc; r += NT / L) {
        const int q = r * L + l;
        const double xm = r > 0 ? X[q - L] : R(0), xp = r + 1 < nc ? X[q + L] : R(0);
        rD[q] = (R)((double)rD[q] - (double)rA[q] * xm - (double)rB[q] * (double)X[q] -
                    (double)rC[q] * xp);
      }
      __syncthreads();
      cols_solve<R, NT, L>(wV, wC, rD, nc, sh, rows);
    }
    __syncthreads();
    auto value = [&](int p) {
      const int q = (p - 2) * L + l;
      if constexpr (Gen::REFINE) return (double)X[q] + (double)rD[q];
      else return (double)rD[q];
    };
    SegWalk<true> e;
    for (int pos = r0 + 2; pos < nc + 2; pos += NT / L)
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
