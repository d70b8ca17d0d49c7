// partsolve.cuh -- partition-method solve of one tridiagonal system held in
// shared memory by a warp or by a CTA.
//
// Rows r = 0..n-1: A_r x_{r-1} + B_r x_r + C_r x_{r+1} = D_r, A_0 = C_{n-1} = 0.
// The system is cut into chunks of S unknowns (the last chunk takes the
// remainder, so every chunk has at least 2); chunk k belongs to thread k:
//   pass A  forward elimination of the chunk's interior keeping the spike of
//           the previous chunk's separator: x_r = y'_r + v'_r x_L - c'_r x_{r+1},
//           (c', y', v') written over the rows in place; the chunk's last
//           unknown is its separator. The first interior row in terms of both
//           neighbouring separators is accumulated on the way;
//   reduce  the separators form a tridiagonal system of one unknown per
//           chunk, solved by cyclic reduction with shuffles: over a warp's
//           chunks, and in a CTA then over its warps' last separators;
//   pass C  back substitution, x written over D.
// So that the chunks a warp walks in step fall on different banks, a CTA's are
// of odd length (bulk_chunk); the warp solver pads instead, row q at q + q/S.
#pragma once

#include <cuda_runtime.h>

namespace hyd {

// q + q / S of q = t0, t0 + dt, t0 + 2 dt, ... without a division per step:
// carries the quotient and remainder of q / S.
struct PartStrideIdx {
  int q, qd, qr, dd, dr, S;
  __device__ PartStrideIdx(int t0, int dt, int S_) : q(t0), qd(t0 / S_), qr(t0 % S_), dd(dt / S_), dr(dt % S_), S(S_) {}
  __device__ int idx() const { return q + qd; }
  __device__ void next(int dt) {
    q += dt;
    qd += dd;
    qr += dr;
    if (qr >= S) {
      qr -= S;
      ++qd;
    }
  }
};

struct PartGeom {
  int S;       // unknowns per chunk (>= 2)
  int nchunk;  // chunks, <= threads
  int stride;  // elements per row array
};

// Upper bound of part_geom(n, threads).stride over all lengths <= nmax
// (the stride itself is not monotonic in n): sizes shared memory for a band.
__host__ __device__ inline int part_stride_bound(int nmax, int threads) {
  return nmax + (nmax / 2 < threads ? nmax / 2 : threads) + 2;
}

__host__ __device__ inline PartGeom part_geom(int n, int threads) {
  PartGeom g;
  g.S = (n + threads - 1) / threads;
  if (g.S < 2) g.S = 2;
  g.nchunk = n / g.S;
  if (g.nchunk < 1) g.nchunk = 1;
  g.stride = n + n / g.S + 2;
  return g;
}

// Chunk k's forward elimination. Writes (c', y', v') over (C, D, A) of the
// interior rows and returns the separator row and the chunk's couplings:
// tri = (yF, vF, wF, yL, vL, wL): first interior unknown = yF + vF x_L + wF x_sep,
// last interior unknown = yL + vL x_L + wL x_sep.
// Index of row q0 + s of chunk k (q0 = k*S): k*(S+1) + s, one more once s
// reaches S (only the last chunk is that long).
__device__ __forceinline__ int part_chunk_idx(int k, int S, int s) {
  return k * (S + 1) + s + (s >= S ? 1 : 0);
}

template <class T>
__device__ __forceinline__ void part_forward(T* rA, T* rB, T* rC, T* rD, int q0, int nu, int S,
                                             T sep[4], T tri[6]) {
  T cp = 0, yp = 0, vp = 0;
  T Pk = 1, fy = 0, fv = 0;
  const int k = q0 / S;
  for (int s = 0; s < nu; ++s) {
    const int o = part_chunk_idx(k, S, s);
    const T A = rA[o], B = rB[o], C = rC[o], D = rD[o];
    if (s == nu - 1) {
      sep[0] = A;
      sep[1] = B;
      sep[2] = C;
      sep[3] = D;
    } else {
      if (s == 0) {
        const T m = T(1) / B;
        cp = C * m;
        yp = D * m;
        vp = -A * m;
      } else {
        const T m = T(1) / (B - A * cp);
        yp = (D - A * yp) * m;
        vp = -A * vp * m;
        cp = C * m;
      }
      rC[o] = cp;
      rD[o] = yp;
      rA[o] = vp;
      fy += Pk * yp;
      fv += Pk * vp;
      Pk *= -cp;
    }
  }
  tri[0] = fy;
  tri[1] = fv;
  tri[2] = Pk;
  tri[3] = yp;
  tri[4] = vp;
  tri[5] = -cp;
}

template <class T>
__device__ __forceinline__ void part_back(T* rA, T* rC, T* rD, int q0, int nu, int S, T xl, T xr) {
  const int k = q0 / S;
  rD[part_chunk_idx(k, S, nu - 1)] = xr;
  T xn = xr;
  for (int t = nu - 2; t >= 0; --t) {
    const int o = part_chunk_idx(k, S, t);
    const T x = rD[o] + rA[o] * xl - rC[o] * xn;
    rD[o] = x;
    xn = x;
  }
}

// the odd chunk length of a system of n rows on NT threads (at least 3)
__device__ __forceinline__ int bulk_chunk(int n, int NT) {
  int S = (n + NT - 1) / NT;
  if (S < 3) S = 3;
  return S | 1;
}

// A chunk after its rows' forward elimination: its separator row, its first
// interior unknown in terms of both neighbouring separators (yF, vF, wF) and
// its last one (yL, vL, wL).
template <class T>
struct ChunkEnds {
  T as = 0, bs = 1, cs = 0, ds = 0;
  T yF = 0, vF = 0, wF = 1, yL = 0, vL = 0, wL = 0;
};

// the same in another type
template <class W, class T>
__device__ __forceinline__ ChunkEnds<W> ends_as(const ChunkEnds<T>& e) {
  return ChunkEnds<W>{(W)e.as, (W)e.bs, (W)e.cs, (W)e.ds, (W)e.yF, (W)e.vF, (W)e.wF, (W)e.yL, (W)e.vL, (W)e.wL};
}

// Eliminates rows q0 .. q0 + nu - 1 (row(q, A, B, C, D) gives row q); where KEEP,
// (v', c', y') go to oV, oC, oY, which may be the rows' own arrays.
template <bool KEEP, class T, class Row>
__device__ __forceinline__ ChunkEnds<T> chunk_forward(T* oV, T* oC, T* oY, int q0, int nu, Row row) {
  ChunkEnds<T> e;
  T cp = 0, yp = 0, vp = 0;
  for (int s = 0; s < nu - 1; ++s) {
    T A, B, C, D;
    row(q0 + s, A, B, C, D);
    if (s == 0) {
      const T m = T(1) / B;
      cp = C * m;
      yp = D * m;
      vp = -A * m;
    } else {
      const T m = T(1) / (B - A * cp);
      yp = (D - A * yp) * m;
      vp = -A * vp * m;
      cp = C * m;
    }
    if constexpr (KEEP) {
      oC[q0 + s] = cp;
      oY[q0 + s] = yp;
      oV[q0 + s] = vp;
    }
    e.yF += e.wF * yp;
    e.vF += e.wF * vp;
    e.wF *= -cp;
  }
  if (nu > 0) row(q0 + nu - 1, e.as, e.bs, e.cs, e.ds);
  e.yL = yp;
  e.vL = vp;
  e.wL = -cp;
  return e;
}

// One level of parallel cyclic reduction on normalised rows (unit diagonal:
// one reciprocal a level): a, c, d of this lane against the lanes st below
// and above, where up / dn. A coupling with no partner stays: it is to the
// unknown beyond the lanes' end.
template <class T>
__device__ __forceinline__ void pcr_level(T& a, T& c, T& d, int st, bool up, bool dn) {
  constexpr unsigned full = 0xffffffffu;
  T am = __shfl_up_sync(full, a, st), cm = __shfl_up_sync(full, c, st), dm = __shfl_up_sync(full, d, st);
  T an = __shfl_down_sync(full, a, st), cn = __shfl_down_sync(full, c, st), dn_ = __shfl_down_sync(full, d, st);
  const T au = up ? a : T(0), cd = dn ? c : T(0);
  const T r = T(1) / (T(1) - au * cm - cd * an);
  d = (d - au * dm - cd * dn_) * r;
  a = (up ? -a * am : a) * r;
  c = (dn ? -c * cn : c) * r;
}

// A tile's separators, one per thread of NT: each warp reduces the chunks of
// its lanes by shuffles, lanes 0..30 to x = d - a XL - c XR (XL, XR the
// previous and this warp's last separators: a coupling out of the warp stays
// in its row), then every warp solves the warps' last separators, one lane
// each, by shuffles again: one barrier, against two per level of a reduction
// over the CTA in shared memory (16 of them for 256 chunks).
// blk: NT / 32 rows of 8 values. FULL: the whole tile is solved here; x and xl
// come back as this chunk's and the previous chunk's separators. Otherwise
// the tile's last separator is the tile's own unknown and tile[0..6] gets the
// first unknown's e0 + e1 XL + e2 X and the row A XL + B X + cs x_next = D
// (written by thread 0).
template <class T, int NT, bool FULL>
__device__ __forceinline__ void tile_reduce(const ChunkEnds<T>& e, T (*blk)[8], T& x, T& xl, T* tile) {
  constexpr unsigned full = 0xffffffffu;
  constexpr int W = NT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const T nyF = __shfl_down_sync(full, e.yF, 1), nvF = __shfl_down_sync(full, e.vF, 1),
          nwF = __shfl_down_sync(full, e.wF, 1);
  const T ra = e.as * e.vL, rb = e.bs + e.as * e.wL, rd = e.ds - e.as * e.yL;
  T a, c, d;
  {
    // (lane 31's own next chunk is another warp's, or none)
    const T cs = lane < 31 ? e.cs : T(0);
    const T inv = T(1) / (rb + cs * nvF);
    a = ra * inv;
    c = cs * nwF * inv;
    d = (rd - cs * nyF) * inv;
    // (it holds the warp's separator, whose row is completed below)
    if (W > 1 && lane == 31) a = c = d = 0;
  }
  if constexpr (W == 1) {
    // one warp: lane 31 is an unknown like the others, nothing lies beyond
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) pcr_level(a, c, d, st, lane >= st, lane + st < 32);
    x = d;
    xl = __shfl_up_sync(full, x, 1);
    if (lane == 0) xl = 0;
    return;
  }
#pragma unroll
  for (int st = 1; st < 32; st <<= 1) pcr_level(a, c, d, st, lane >= st, lane + st < 31);
  {
    const T a30 = __shfl_up_sync(full, a, 1), c30 = __shfl_up_sync(full, c, 1), d30 = __shfl_up_sync(full, d, 1);
    if (lane == 0) {
      blk[warp][0] = e.yF + e.wF * d;
      blk[warp][1] = e.vF - e.wF * a;
      blk[warp][2] = -e.wF * c;
    }
    if (lane == 31) {
      blk[warp][3] = -ra * a30;
      blk[warp][4] = rb - ra * c30;
      blk[warp][5] = e.cs;
      blk[warp][6] = rd - ra * d30;
    }
  }
  __syncthreads();
  // the warps' separators: lane l takes warp l's (not the tile's last one
  // where that is the tile's unknown)
  constexpr int V = FULL ? W : W - 1;
  T A = 0, B = 1, C = 0, D = 0;
  if (lane < V) {
    A = blk[lane][3];
    B = blk[lane][4];
    C = blk[lane][5];
    D = blk[lane][6];
    if (lane + 1 < W) {
      B += C * blk[lane + 1][1];
      D -= C * blk[lane + 1][0];
      C *= blk[lane + 1][2];
    } else {
      C = 0;
    }
  }
  {
    const T inv = T(1) / B;
    A *= inv;
    C *= inv;
    D *= inv;
  }
#pragma unroll
  for (int st = 1; st < V; st <<= 1) pcr_level(A, C, D, st, lane >= st, lane + st < V);
  if constexpr (FULL) {
    T XL = __shfl_sync(full, D, warp > 0 ? warp - 1 : 0);
    if (warp == 0) XL = 0;
    const T XR = __shfl_sync(full, D, warp);
    x = lane == 31 ? XR : d - a * XL - c * XR;
    xl = __shfl_up_sync(full, x, 1);
    if (lane == 0) xl = XL;
  } else if (warp == 0) {
    const T Av = __shfl_sync(full, A, V - 1), Cv = __shfl_sync(full, C, V - 1), Dv = __shfl_sync(full, D, V - 1);
    if (lane == 0) {
      tile[0] = blk[0][0] + blk[0][2] * D;
      tile[1] = blk[0][1] - blk[0][2] * A;
      tile[2] = -blk[0][2] * C;
      tile[3] = -blk[V][3] * Av;
      tile[4] = blk[V][4] - blk[V][3] * Cv;
      tile[5] = blk[V][5];
      tile[6] = blk[V][6] - blk[V][3] * Dv;
    }
  }
}

// The partition solve of n rows in shared memory by the NT threads of a CTA,
// the solution in X: row(q, A, B, C, D) gives row q, (v', c') are kept in oV and
// oC (all three may be the rows' own A, C, D arrays). The reduction is done in
// blk's type W.
template <class T, int NT, class W, class Row>
__device__ __forceinline__ void cta_solve(T* oV, T* oC, T* X, int n, W (*blk)[8], Row row) {
  const int tid = threadIdx.x, S = bulk_chunk(n, NT), P = max(1, n / S);
  const int q0 = tid * S;
  const int nu = tid < P ? (tid == P - 1 ? n - q0 : S) : 0;
  const ChunkEnds<T> e = chunk_forward<true>(oV, oC, X, q0, nu, row);
  W wx, wxl;
  tile_reduce<W, NT, true>(ends_as<W>(e), blk, wx, wxl, nullptr);
  const T x = (T)wx, xl = (T)wxl;
  if (nu > 0) {
    X[q0 + nu - 1] = x;
    T xn = x;
#pragma unroll 4
    for (int q = q0 + nu - 2; q >= q0; --q) {
      const T xq = X[q] + oV[q] * xl - oC[q] * xn;
      X[q] = xq;
      xn = xq;
    }
  }
}

// Reduced-system work space of a CTA of NT threads: what each warp's first
// and last chunks give the others (tile_reduce).
template <class T, int NT>
struct PartCtaShared {
  T blk[NT / 32][8];
};

// Warp-wide solve (all 32 lanes call it; the rows are in the warp's slice of
// shared memory). The reduced system is solved with shuffles.
template <class T>
__device__ void part_solve_warp(T* rA, T* rB, T* rC, T* rD, const PartGeom& g, int n, int lane) {
  const unsigned full = 0xffffffffu;
  const int k = lane, P = g.nchunk, S = g.S;
  const int q0 = k * S;
  const int nu = k < P ? ((k == P - 1) ? n - q0 : S) : 0;
  T sep[4] = {0, 1, 0, 0}, tri[6] = {0, 0, 1, 0, 0, 0};
  if (k < P) part_forward(rA, rB, rC, rD, q0, nu, S, sep, tri);
  const T yF = __shfl_down_sync(full, tri[0], 1);
  const T vF = __shfl_down_sync(full, tri[1], 1);
  const T wF = __shfl_down_sync(full, tri[2], 1);
  T ra = 0, rb = 1, rc = 0, rd = 0;
  if (k < P) {
    const bool nx = k + 1 < P;
    ra = sep[0] * tri[4];
    rb = sep[1] + sep[0] * tri[5] + sep[2] * (nx ? vF : T(0));
    rc = sep[2] * (nx ? wF : T(0));
    rd = sep[3] - sep[0] * tri[3] - sep[2] * (nx ? yF : T(0));
  }
  // (rows normalised to a unit diagonal: one reciprocal per level)
  const T inv = T(1) / rb;
  T a = ra * inv, c = rc * inv, d = rd * inv;
  for (int st = 1; st < P; st <<= 1) {
    const T am = __shfl_up_sync(full, a, st), cm = __shfl_up_sync(full, c, st), dm = __shfl_up_sync(full, d, st);
    const T an = __shfl_down_sync(full, a, st), cn = __shfl_down_sync(full, c, st), dn = __shfl_down_sync(full, d, st);
    const T au = k >= st ? a : T(0), cd = k + st < P ? c : T(0);
    const T r = T(1) / (T(1) - au * cm - cd * an);
    d = (d - au * dm - cd * dn) * r;
    a = -au * am * r;
    c = -cd * cn * r;
  }
  const T xs = d;
  const T xl = __shfl_up_sync(full, xs, 1);
  if (k < P) part_back(rA, rC, rD, q0, nu, S, k > 0 ? xl : T(0), xs);
  __syncwarp();
}

}  // namespace hyd
