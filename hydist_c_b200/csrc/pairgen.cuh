// pairgen.cuh -- the hydraulic line systems of the FP32 forms, as the reference
// has them: two unknowns per cell, level and velocity interleaved, solved in
// single precision by the chunked line solver (linesolve.cuh).
//
// The FP64 sweeps eliminate the levels first and solve staged lines (sweep.cu).
// In single precision that is another rounding, and rounding is not all it
// changes: beside a dry cell the momentum row takes its one-sided second
// difference only where the cross velocity has the right sign (assembly.cuh:
// vtb < 0, utb > 0 ...), so where that velocity passes through zero an error of
// 1e-7 switches a term of full size on or off; the cell jumps by up to 9e-3 of the
// velocities' scale and its neighbours follow. Of 12000 channels of 128x48, thirty
// steps each, held against FP64, 12 jumped by more than 8e-4 here, 9 refined, 8
// and 5 when solved for the velocities' changes in staged lines (which errs less
// elsewhere, 3e-7 against 5.5e-7), mostly not the same ones. Neither rounding is
// the right one in such a cell, so the FP32 forms keep this one: the rows, the
// chunks and the order of operations, of which a faster solver has to give the
// same bits. What it costs, x + y sweep against the staged lines: 2048x1024 105 +
// 122 us against 93 + 72, refined 158 + 205 against 119 + 81; 1024x512 48 + 40
// against 37 + 21, refined 71 + 48 against 40 + 25; 256x128 37 + 25 against 21 + 17;
// a whole step of 64x32 109 us against 52, of 100x4000 354 against 93.
#pragma once

#include "assembly.cuh"
#include "common.cuh"
#include "linesolve.cuh"

namespace hyd {

// REF: refine each line solve once with an FP64 residual
template <int DIR, bool REF>
struct PairGen {
  using R = float;
  using Real = R;
  static constexpr bool REFINE = REF;
  // the rows are generated from the stencils: the refinement keeps them
  static constexpr bool ROWS_AGAIN = false;
  static constexpr int AUX = 0;  // the emitter needs nothing but the solution
  // c', y', v', with refinement the rows A, B, C, D
  static constexpr int SCRATCH_ARRAYS = REFINE ? 7 : 3;
  static constexpr int UPC = 2;
  static constexpr int DIRECTION = DIR;
  // x sweeps (columns, 4 adjacent per warp) run faster with two CTAs per SM
  // despite the register cap, and so do the plain y sweeps; the refined y
  // sweeps slower
  static constexpr int MIN_BLOCKS = (DIR == 0 || !REF) ? 2 : 1;
  StateT<R> S;
  CoefT<R> c;
  R* scratch;
  R f4;
  // lines lp0 .. lp0 + nl - 1: columns 2..M (x) / rows 2..N (y), or the
  // narrow-channel ranges (StateT::x_lo, x_hi, y_lo)
  int lp0, nl;

  __host__ __device__ void bind(const StateT<R>& s, const CoefT<R>& cc) {
    S = s;
    c = cc;
    f4 = DIR == 0 ? 2 * cc.g * cc.dTchia2dX : 2 * cc.g * cc.dTchia2dY;
  }
  __device__ int lines() const { return nl; }
  __device__ int cells_per_line() const { return DIR == 0 ? S.N - 1 : S.M - 1; }
  __device__ int unknowns_per_line() const { return 2 * cells_per_line(); }
  __device__ int end_pos() const { return DIR == 0 ? S.N : S.M; }
  // field index of position p on line position lp
  __device__ int at(int lp, int p) const { return DIR == 0 ? p * S.W + lp : lp * S.W + p; }
  // the preindex values of a cell, from its stencil (computed where the
  // walker reaches the cell: a separate per-cell pass writing them to HBM
  // ahead of the sweep costs more in traffic and a launch than it saves)
  __device__ PreT<R> pre(int lp, int p) const {
    return DIR == 0 ? pre_x(S, c, p, lp) : pre_y(S, c, lp, p);
  }
  __device__ R* vel() const { return DIR == 0 ? S.tu : S.tv; }
  // the VZ extraction reaches columns j <= N only (UVZSolver_multithread.cpp:851)
  __device__ bool extract_ok(int p) const { return DIR == 0 ? true : p <= S.N; }

  __device__ void load_segment(LineSeg& LS, int line, int s) const {
    const bool ok = line < lines();
    const int lp = line + lp0;
    if (s == SEG) {
      LS.nseg = ok ? (DIR == 0 ? S.mocj[lp] : S.moci[lp]) : 0;
      return;
    }
    if (!ok) return;
    const int n = DIR == 0 ? S.mocj[lp] : S.moci[lp];
    if (s >= n) return;
    const int w = S.W;
    SegD& d = LS.s[s];
    int first, last;
    bool br1, br2;
    bool q1, q2;
    if (DIR == 0) {
      first = S.dauj[lp * SEG + s];
      last = S.cuoij[lp * SEG + s];
      // locate_segment_u (support_funcs.cpp:845-851)
      br1 = (first > 2) || ((first == 2) && ((S.h[1 * w + lp] + S.h[1 * w + lp - 1]) * 0.5 == c.NANGDAY));
      br2 = (last < S.N) || ((last == S.N) && ((S.h[S.N * w + lp] + S.h[S.N * w + lp - 1]) * 0.5 == c.NANGDAY));
      q1 = S.bienQ[2] != 0;
      q2 = S.bienQ[3] != 0;
    } else {
      first = S.daui[lp * SEG + s];
      last = S.cuoii[lp * SEG + s];
      // locate_segment_v (support_funcs.cpp:823-826)
      br1 = (first > 2) || ((first == 2) && ((S.h[lp * w + first - 1] + S.h[(lp - 1) * w + first - 1]) * 0.5 == c.NANGDAY));
      br2 = (last < S.M) || ((last == S.M) && ((S.h[lp * w + last] + S.h[(lp - 1) * w + last]) * 0.5 == c.NANGDAY));
      q1 = S.bienQ[1] != 0;
      q2 = S.bienQ[0] != 0;
    }
    const LineSys L = line_sys(first, last, br1, br2, q1, q2, end_pos());
    d.first = first;
    d.last = last;
    d.off = L.off;
    d.rend = L.off + L.sn;
    d.br1 = br1;
    d.br2 = br2;
    d.ran = L.ran;
    d.qfirst = L.qfirst;
    d.last_kind = (unsigned char)L.last_kind;
    d.xq_first = q1;
    d.xq_last = q2;
  }

  // Generates the rows of the line system cell by cell (two unknowns per cell).
  struct Walker {
    int lp, si, pos, prev;
    bool in;
    PreT<R> Pc, Pn;
    MomT<R> Mi;
    __device__ void init(const PairGen& G, const LineSeg& LS, int line, int c0) {
      lp = line + G.lp0;
      si = 0;
      prev = -10;
      in = false;
    }
    __device__ void cell(const PairGen& G, const LineSeg& LS, int c) {
      pos = c + 2;
      while (si < LS.nseg && LS.s[si].last < pos) ++si;
      in = si < LS.nseg && LS.s[si].first <= pos;
      if (!in) {
        prev = -10;
        return;
      }
      const SegD& d = LS.s[si];
      if (prev == pos - 1 && pos > d.first) Pc = Pn;
      else Pc = G.pre(lp, pos);
      if (pos + 1 <= d.last) Pn = G.pre(lp, pos + 1);
      else Pn = Pc;
      if (pos <= d.last - 1 || pos == d.first) Mi = abcd(Pc, Pn, pos, d.first, d.last, G.f4, d.br1, d.br2);
      else Mi = MomT<R>{0, 0, 0, 0};
      prev = pos;
    }
    __device__ void row(const PairGen& G, const LineSeg& LS, int e, R& A, R& B, R& C,
                        R& D) const {
      if (!in) {
        A = 0; B = 1; C = 0; D = 0;
        return;
      }
      G.rows_in(LS.s[si], lp, pos, Pc, Pn, Mi, e, A, B, C, D);
    }
  };

  // Row 2*pos + e of the line system at line position lp, for a cell pos of
  // segment d with its preindex values Pc, those of the next cell Pn (Pc at
  // the segment's last cell) and its momentum coefficients Mi.
  __device__ void rows_in(const SegD& d, int lp, int pos, const PreT<R>& Pc, const PreT<R>& Pn,
                          const MomT<R>& Mi, int e, R& A, R& B, R& C, R& D) const {
    const int r = 2 * pos + e;
    if (r < d.off || r > d.rend) {
      A = 0; B = 1; C = 0; D = 0;
      return;
    }
    const bool even = (r & 1) == 0;
    if ((bool)d.ran == even) {
      const PreT<R>& P = d.ran ? Pc : Pn;
      A = P.a2; B = 1; C = P.c2; D = P.d2;
    } else {
      A = Mi.a1; B = Mi.b1; C = Mi.c1; D = Mi.d1;
    }
    if (r == d.off) {
      if (d.ran) {
        if (d.qfirst) {
          const R ub = DIR == 0 ? S.ubt[lp] : S.vbd[lp];
          D = Pc.d2 - Pc.a2 * ub;
        } else {
          D = Pc.d2;
        }
      } else {
        const R TZ_l = R(S.tz[at(lp, d.first)]);
        D = Mi.d1 - Mi.a1 * TZ_l;
      }
      A = 0;  // the system starts here
    }
    if (r == d.rend) {
      const PreT<R>& PL = (pos == d.last) ? Pc : Pn;
      if (d.last_kind == 1) {
        const R ub = DIR == 0 ? S.ubp[lp] : S.vbt[lp];
        A = PL.a2; B = 1; D = PL.d2 - PL.c2 * ub;
      } else if (d.last_kind == 2) {
        const R TZ_r = R(S.tz[at(lp, d.last)]);
        A = Mi.a1; B = Mi.b1; D = Mi.d1 - Mi.c1 * TZ_r;
      } else {
        A = PL.a2; B = 1; D = PL.d2;
      }
      C = 0;  // and ends here
    }
  }

  // (the refinement reads the stored rows: no cursor over them)
  struct RowCursor {
    __device__ void init(const PairGen&, const LineSeg&, int) {}
    __device__ void row(const PairGen&, const LineSeg&, int, R&, R&, R&, R&) {}
  };

  // Writes each solved unknown to t_z / t_u (t_v) as the extraction does.
  // FWD: the unknowns come in increasing order (init_fwd), else decreasing.
  struct Emitter {
    int lp, si;
    __device__ void init(const PairGen& G, const LineSeg& LS, int line) {
      lp = line + G.lp0;
      si = LS.nseg - 1;
    }
    __device__ void init_fwd(const PairGen& G, const LineSeg& LS, int line) {
      lp = line + G.lp0;
      si = -1;
    }
    template <bool FWD = false>
    __device__ void emit(const PairGen& G, const LineSeg& LS, double* xlast, int q, double x, double,
                         R) {
      const int r = q + 4, pos = r >> 1;
      if constexpr (FWD) {
        while (si + 1 < LS.nseg && LS.s[si + 1].first <= pos) ++si;
      } else {
        while (si >= 0 && LS.s[si].first > pos) --si;
      }
      if (si < 0) return;
      G.store_in(LS.s[si], xlast + si, lp, q, x);
    }
  };

  // The extraction of unknown q (row q + 4) of segment d on line position
  // lp; the segment's last row also goes to *xl for the end fix-up.
  __device__ void store_in(const SegD& d, double* xl, int lp, int q, double x) const {
    const int r = q + 4, pos = r >> 1;
    if (pos > d.last || r < d.off || r > d.rend) return;
    if (r == d.rend) *xl = x;
    R* v = vel_ptr();
    if (d.ran) {
      const int i = r >> 1;
      if (i < d.last && extract_ok(i)) {
        if (r & 1) v[at(lp, i)] = x;
        else S.tz[at(lp, i)] = x;
      }
    } else {
      if (r == 2 * d.first) {
        if (extract_ok(d.first)) v[at(lp, d.first)] = x;
      } else {
        const int i = (r + 1) >> 1;
        if (i > d.first && i < d.last && extract_ok(i)) {
          if (r & 1) S.tz[at(lp, i)] = x;
          else v[at(lp, i)] = x;
        }
      }
    }
  }

  // Segment ends (_uzSolver_extract_solution :558-601 / _vzSolver_ :488-536).
  __device__ void fixup(const LineSeg& LS, const double* xlast, int line, int s) const {
    const SegD& d = LS.s[s];
    const int lp = line + lp0, first = d.first, last = d.last;
    R* vel = vel_ptr();
    double* tz = S.tz;
    if (first < last && extract_ok(first)) {
      if (d.br1) {
        vel[at(lp, first - 1)] = 0;
      } else if (d.xq_first && first == 2) {
        vel[at(lp, first - 1)] = DIR == 0 ? S.ubt[lp] : S.vbd[lp];
      } else {
        const PreT<R> Pf = pre(lp, first);
        vel[at(lp, first - 1)] = (Pf.d2 - tz[at(lp, first)] - Pf.c2 * vel[at(lp, first)]) / Pf.a2;
      }
    }
    if (!extract_ok(last)) return;
    const double xl = (d.rend >= d.off) ? xlast[s] : 0.0;
    if (d.br2) {
      vel[at(lp, last)] = 0;
      tz[at(lp, last)] = xl;
    } else if (d.xq_last && last == end_pos()) {
      vel[at(lp, last)] = DIR == 0 ? S.ubp[lp] : S.vbt[lp];
      tz[at(lp, last)] = xl;
    } else {
      const PreT<R> Pl = pre(lp, last);
      vel[at(lp, last)] = (Pl.d2 - Pl.a2 * vel[at(lp, last - 1)] - tz[at(lp, last)]) / Pl.c2;
    }
  }
  __device__ R* vel_ptr() const { return DIR == 0 ? S.tu : S.tv; }
};

}  // namespace hyd
