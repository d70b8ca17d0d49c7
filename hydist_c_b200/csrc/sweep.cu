// sweep.cu -- the ADI line sweeps: what they solve, and which solver takes them.
//
// The FP64 form's hydraulic sweeps (the FP32 forms': pairgen.cuh).
// HydroGen<0> is the x sweep (UZ half-step: lines are columns j, cells run
// along i, unknowns u_i); HydroGen<1> is the y sweep (VZ half-step: lines are
// rows i, cells along j, unknowns v_j). Both generate the rows of the
// velocities alone (the reference's interleaved z, u system with its
// continuity rows eliminated, make_row) on the fly (assembly.cuh) and write
// the extraction of UZSolver_extract_solution / VZSolver_extract_solution
// (UVZSolver_multithread.cpp:472-603) directly from the solution, each cell's
// level by its continuity row: against the interleaved system on 2048x1024
// (FP64, the same chunked solver) x 0.151 -> 0.111 ms, y 0.172 -> 0.148.
#include <algorithm>

#include "assembly.cuh"
#include "common.cuh"
#include "hydro.cuh"
#include "colsolve.cuh"
#include "linesolve.cuh"
#include "pairgen.cuh"
#include "rowsolve.cuh"
#include "sediment_cell.cuh"

namespace hyd {

template <int DIR>
struct HydroGen {
  using R = double;
  using Real = R;
  static constexpr bool REFINE = false, ROWS_AGAIN = false;
  static constexpr int UPC = 1;
  static constexpr int AUX = 3;  // c', y', v', then the emitter's value
  static constexpr int SCRATCH_ARRAYS = AUX + 1;
  static constexpr int DIRECTION = DIR;
  // resident CTAs per SM the chunked row solver is compiled for (two, with
  // their register cap, are slower)
  static constexpr int MIN_BLOCKS = 1;
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
  __device__ int unknowns_per_line() const { return cells_per_line(); }
  __device__ int end_pos() const { return DIR == 0 ? S.N : S.M; }
  // field index of position p on line position lp
  __device__ int at(int lp, int p) const { return DIR == 0 ? p * S.W + lp : lp * S.W + p; }
  // the VZ extraction reaches columns j <= N only (UVZSolver_multithread.cpp:851)
  __device__ bool extract_ok(int p) const { return DIR == 0 ? true : p <= S.N; }

  __device__ int segments(int lp) const { return DIR == 0 ? S.mocj[lp] : S.moci[lp]; }
  // segment s of line position lp (false if the line has no such segment;
  // count and ends in one round of latency)
  __device__ bool segment(int lp, int s, SegD& d) const {
    const int n = segments(lp);
    const int first = (DIR == 0 ? S.dauj : S.daui)[lp * SEG + s];
    const int last = (DIR == 0 ? S.cuoij : S.cuoii)[lp * SEG + s];
    if (s >= n) return false;
    const int w = S.W;
    bool br1, br2;
    bool q1, q2;
    if (DIR == 0) {
      // locate_segment_u (support_funcs.cpp:845-851)
      br1 = (first > 2) || ((first == 2) && ((S.h[1 * w + lp] + S.h[1 * w + lp - 1]) * 0.5 == c.NANGDAY));
      br2 = (last < S.N) || ((last == S.N) && ((S.h[S.N * w + lp] + S.h[S.N * w + lp - 1]) * 0.5 == c.NANGDAY));
      q1 = S.bienQ[2] != 0;
      q2 = S.bienQ[3] != 0;
    } else {
      // locate_segment_v (support_funcs.cpp:823-826)
      br1 = (first > 2) || ((first == 2) && ((S.h[lp * w + first - 1] + S.h[(lp - 1) * w + first - 1]) * 0.5 == c.NANGDAY));
      br2 = (last < S.M) || ((last == S.M) && ((S.h[lp * w + last] + S.h[(lp - 1) * w + last]) * 0.5 == c.NANGDAY));
      q1 = S.bienQ[1] != 0;
      q2 = S.bienQ[0] != 0;
    }
    const LineSys L = line_sys(first, last, br1, br2, q1, q2, end_pos());
    d.first = first;
    d.last = last;
    d.off = first;
    d.rend = last - 1;
    d.br1 = br1;
    d.br2 = br2;
    d.ran = L.ran;
    d.qfirst = L.qfirst;
    d.last_kind = (unsigned char)L.last_kind;
    d.xq_first = q1;
    d.xq_last = q2;
    return true;
  }
  __device__ void load_segment(LineSeg& LS, int line, int s) const {
    const bool ok = line < lines();
    if (s == SEG) LS.nseg = ok ? segments(line_pos(line)) : 0;
    else if (ok) segment(line_pos(line), s, LS.s[s]);
  }

  // One cell's continuity values: depth at its velocity point, level, and the
  // cross-line flux w (continuity: z_new = z - w + k (Ha_{-} a_{-} - Ha a)).
  struct Cont {
    R H, w;
    double z;
  };
  __device__ R depth(int g) const { return DIR == 0 ? S.Htdu[g] : S.Htdv[g]; }
  __device__ Cont cont(int g) const {
    return Cont{depth(g), DIR == 0 ? flux_x(S, c, g) : flux_y(S, c, g), S.z[g]};
  }
  // the prescribed velocities beyond the line's first and last cells
  __device__ R q_first(int lp) const { return DIR == 0 ? S.ubt[lp] : S.vbd[lp]; }
  __device__ R q_last(int lp) const { return DIR == 0 ? S.ubp[lp] : S.vbt[lp]; }

  // The row of the velocity a_pos of cell pos, first <= pos < last of segment
  // d: the momentum row with the levels of the cells pos and pos + 1 replaced
  // by their continuity rows,
  //   (f1 + e Ha_{-}) a_{-} + (f2 - 2 e Ha) a + (f3 + e Ha_{+}) a_{+}
  //     = f5 + f4 (d2_{+} - d2),   e = f4 k, d2 = z - w,
  // which is what eliminating the z unknowns of the reference's interleaved
  // system (_calculate_abcd + _calculate_matrix_coeff, UVZSolver_
  // multithread.cpp:280-470) leaves: its f1/a2 and f3/c2 terms cancel. Half
  // the unknowns, and one division per cell instead of four. Ends: a solid or
  // discharge end prescribes the velocity beyond it; at an open end (level
  // given) the reference keeps the substituted f1/a2 (f3/c2) term.
  __device__ void make_row(const SegD& d, int lp, int pos, MomF<R> m, R Hm, const Cont& c0,
                           const Cont& c1, R& A, R& B, R& C, R& D) const {
    const R kk = DIR == 0 ? c.dTchia2dX : c.dTchia2dY, e = f4 * kk;
    const bool at0 = pos == d.first, at1 = pos == d.last - 1;
    if (d.last - 1 <= d.first) m.f1 = m.f3 = 0;  // a two-cell segment
    A = m.f1 + e * Hm;
    B = m.f2 - 2 * e * c0.H;
    C = m.f3 + e * c1.H;
    const R dd = R(c1.z - c0.z) - (c1.w - c0.w);
    D = m.f5 + f4 * dd;
    if (at0) {
      if (d.qfirst) {
        D -= A * q_first(lp);
      } else if (!d.ran) {
        // level given at the first cell
        const double zl = S.tz[at(lp, pos)];
        const R ra = -m.f1 / (kk * Hm);
        B = m.f2 - (ra * kk + e) * c0.H;
        D = m.f5 + f4 * (R(c1.z - zl) - c1.w) - ra * (R(c0.z - zl) - c0.w);
      }
      A = 0;
    }
    if (at1) {
      if (d.last_kind == 1) {
        D -= C * q_last(lp);
      } else if (d.last_kind == 2) {
        const double zr = S.tz[at(lp, d.last)];
        const R rc = m.f3 / (kk * c1.H);
        B += (f4 + rc) * kk * c0.H;
        // (between two given levels one velocity alone: the reference's last
        // row overwrites the first level's term)
        if (at0 && !d.ran) D = m.f5 + f4 * R(zr);
        else D += (f4 + rc) * (R(zr - c1.z) + c1.w);
      }
      C = 0;
    }
  }

  // a cell's operands and row for the staged row solver (rowsolve.cuh); load
  // is in bounds for every cell of the mesh, wet or not
  struct Ops {
    R Hm;
    Cont c0, c1;
    MomF<R> m;
  };
  __device__ int line_pos(int line) const { return line + lp0; }
  __device__ Ops load(int lp, int pos) const {
    Ops o;
    const int g = at(lp, pos), s = DIR == 0 ? S.W : 1;
    o.Hm = depth(g - s);
    o.c0 = cont(g);
    o.c1 = cont(g + s);
    o.m = DIR == 0 ? mom_x(S, c, pos, lp) : mom_y(S, c, lp, pos);
    return o;
  }
  __device__ void row(const SegD& d, int lp, int pos, const Ops& o, R& A, R& B, R& C, R& D) const {
    make_row(d, lp, pos, o.m, o.Hm, o.c0, o.c1, A, B, C, D);
  }
  // the part of a cell's new level that does not depend on the solution is
  // kept where the level goes, if the emission will write it there (nothing
  // reads t_z in between: the given levels are at cells that are not written)
  __device__ bool level_out(const SegD& d, int pos) const {
    return (pos > d.first || d.ran) && extract_ok(pos);
  }
  __device__ void keep(const SegD& d, int lp, int pos, const Ops& o) const {
    if (level_out(d, pos)) S.tz[at(lp, pos)] = o.c0.z - o.c0.w;
  }
  __device__ void prefetch(int lp) const {
    const int w = S.W;
    const size_t r = (size_t)lp * w;
    prefetch_l2(S.u + r, w);
    prefetch_l2(S.v + r + 2 * w, w);
    prefetch_l2(S.Hmoi + r + w, w);
    prefetch_l2(S.Htdu + r, w);
    prefetch_l2(S.Htdv + r, w);
    prefetch_l2(S.visco + r, w);
    prefetch_l2(S.Ky1 + r, w);
    prefetch_l2(S.Tsyw + r, w);
    prefetch_l2(S.z + r, w);
  }
  // Writes what the sweep gives at cell pos, first <= pos <= last, of segment
  // d: velocity and level, and beyond the first and at the last cell what
  // fixup does. value(p): the solved velocity of cell p.
  template <class V>
  __device__ void emit_cell(const SegD& d, int lp, int pos, V value) const {
    const int g = at(lp, pos), s = DIR == 0 ? S.W : 1;
    if (!extract_ok(pos)) return;
    R* v = vel_ptr();
    if (pos < d.last) {
      const R x = value(pos);
      v[g] = x;
      if (level_out(d, pos)) {
        const R xm = pos > d.first ? value(pos - 1) : (d.qfirst ? q_first(lp) : 0.0);
        const R kk = DIR == 0 ? c.dTchia2dX : c.dTchia2dY;
        S.tz[g] = S.tz[g] + kk * (depth(g - s) * xm - depth(g) * x);
      }
      if (pos == d.first) end_first(d, lp, x);
    } else {
      const bool two = d.last > d.first;
      const R x = two ? value(pos - 1) : 0.0;
      end_last(d, lp, x, two ? x : v[g - s]);
    }
  }

  // Generates the rows of the line system cell by cell.
  struct Walker {
    int lp, si, pos, prev;
    bool in;
    R Hm, aux;  // depth before c0; the level without the solution's part
    Cont c0, c1;
    MomF<R> m;
    __device__ void init(const HydroGen& G, const LineSeg& LS, int line, int first_cell) {
      lp = line + G.lp0;
      si = 0;
      prev = -10;
      in = false;
    }
    __device__ void cell(const HydroGen& G, const LineSeg& LS, int cc) {
      pos = cc + 2;
      while (si < LS.nseg && LS.s[si].last <= pos) ++si;
      in = si < LS.nseg && LS.s[si].first <= pos;
      if (!in) {
        prev = -10;
        return;
      }
      if (prev == pos - 1) {
        Hm = c0.H;
        c0 = c1;
      } else {
        Hm = G.depth(G.at(lp, pos - 1));
        c0 = G.cont(G.at(lp, pos));
      }
      c1 = G.cont(G.at(lp, pos + 1));
      m = DIR == 0 ? mom_x(G.S, G.c, pos, lp) : mom_y(G.S, G.c, lp, pos);
      prev = pos;
      aux = c0.z - c0.w;
    }
    __device__ void row(const HydroGen& G, const LineSeg& LS, int, R& A, R& B, R& C, R& D) const {
      if (!in) {
        A = 0; B = 1; C = 0; D = 0;
        return;
      }
      G.make_row(LS.s[si], lp, pos, m, Hm, c0, c1, A, B, C, D);
    }
  };

  // Writes each solved velocity and its cell's level to t_u (t_v) / t_z as
  // the extraction does; the unknowns come in decreasing order.
  struct Emitter {
    int lp, si;
    __device__ void init(const HydroGen& G, const LineSeg& LS, int line) {
      lp = line + G.lp0;
      si = LS.nseg - 1;
    }
    // unknown q with value x, the one before it xm, its cell's aux
    __device__ void emit(const HydroGen& G, const LineSeg& LS, double* xlast, int q, double x,
                         double xm, R aux) {
      const int pos = q + 2;
      while (si >= 0 && LS.s[si].first > pos) --si;
      if (si < 0) return;
      G.store_in(LS.s[si], xlast + si, lp, pos, x, xm, aux);
    }
  };

  // The extraction of the velocity x of cell pos of segment d on line position
  // lp, and of the cell's level by continuity (the first cell's where it is
  // not given); the segment's last velocity also goes to *xl for the end
  // fix-up. aux: the level without the solution's part.
  __device__ void store_in(const SegD& d, double* xl, int lp, int pos, double x, double xm,
                           R aux) const {
    if (pos >= d.last) return;
    const int g = at(lp, pos);
    if (pos == d.last - 1) *xl = x;
    if (!extract_ok(pos)) return;
    vel_ptr()[g] = x;
    if (pos > d.first || d.ran) {
      if (pos == d.first) xm = d.qfirst ? q_first(lp) : 0.0;
      const R kk = DIR == 0 ? c.dTchia2dX : c.dTchia2dY;
      S.tz[g] = aux + kk * (depth(DIR == 0 ? g - S.W : g - 1) * xm - depth(g) * x);
    }
  }

  // Segment ends (_uzSolver_extract_solution :558-601 / _vzSolver_ :488-536):
  // the velocity beyond the first cell, x the first cell's ...
  __device__ void end_first(const SegD& d, int lp, R x) const {
    R* vel = vel_ptr();
    const int first = d.first;
    if (d.br1) {
      vel[at(lp, first - 1)] = 0;
    } else if (d.xq_first && first == 2) {
      vel[at(lp, first - 1)] = q_first(lp);
    } else {
      const double kk = DIR == 0 ? c.dTchia2dX : c.dTchia2dY;
      const Cont cf = cont(at(lp, first));
      vel[at(lp, first - 1)] = ((cf.z - cf.w) - S.tz[at(lp, first)] - kk * cf.H * x) /
                               (-kk * depth(at(lp, first - 1)));
    }
  }
  // ... and the last cell's velocity and level; x the solved velocity before
  // it (0 where none was solved), v1 that velocity as t_u (t_v) holds it
  __device__ void end_last(const SegD& d, int lp, double x, R v1) const {
    R* vel = vel_ptr();
    double* tz = S.tz;
    const int first = d.first, last = d.last;
    const double kk = DIR == 0 ? c.dTchia2dX : c.dTchia2dY;
    const Cont cl = cont(at(lp, last));
    const double d2 = cl.z - cl.w;
    // the value of the reference system's last row: the last cell's level, the
    // last velocity where that level is given, 0 where no row was solved
    double xl = 0.0;
    if (last > first) {
      xl = d.last_kind == 2 ? x
                            : d2 + kk * depth(at(lp, last - 1)) * x -
                                  (d.last_kind == 1 ? kk * cl.H * q_last(lp) : 0.0);
    } else if (d.ran && d.last_kind != 2) {
      xl = d2 - (d.last_kind == 1 ? kk * cl.H * q_last(lp) : 0.0);
    }
    if (d.br2) {
      vel[at(lp, last)] = 0;
      tz[at(lp, last)] = xl;
    } else if (d.xq_last && last == end_pos()) {
      vel[at(lp, last)] = q_last(lp);
      tz[at(lp, last)] = xl;
    } else {
      vel[at(lp, last)] = (d2 + kk * depth(at(lp, last - 1)) * v1 - tz[at(lp, last)]) / (kk * cl.H);
    }
  }
  // both ends of segment s (after the emission)
  __device__ void fixup(const LineSeg& LS, const double* xlast, int line, int s) const {
    const SegD& d = LS.s[s];
    const int lp = line + lp0;
    if (d.first < d.last && extract_ok(d.first)) end_first(d, lp, vel_ptr()[at(lp, d.first)]);
    if (extract_ok(d.last)) end_last(d, lp, d.last > d.first ? xlast[s] : 0.0, vel_ptr()[at(lp, d.last - 1)]);
  }
  __device__ R* vel_ptr() const { return DIR == 0 ? S.tu : S.tv; }
};

// the kernel's shared-memory limit, raised once per device
template <class Gen, int P, int L>
static size_t prepare(int dev) {
  const size_t smem = line_smem<typename Gen::Real, P, L>(Gen::REFINE);
  static bool attr[64] = {};
  if (dev < 64 && !attr[dev]) {
    cudaFuncSetAttribute(k_line_solve<Gen, P, L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)smem);
    attr[dev] = true;
  }
  return smem;
}

template <class Gen, int P, int L = LPB>
static void launch_gen(const Gen& G, cudaStream_t st, int grid, int line0, int ngroups,
                       const Batch<typename Gen::Real>& b = {}, int gpm = 0) {
  int dev = 0;
  cudaGetDevice(&dev);
  const size_t smem = prepare<Gen, P, L>(dev);
  if (b.n > 0) {
    static bool attr[64] = {};
    if (dev < 64 && !attr[dev]) {
      cudaFuncSetAttribute(k_line_solve<Gen, P, L, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem);
      attr[dev] = true;
    }
    k_line_solve<Gen, P, L, 1><<<grid, L * P, smem, st>>>(G, line0, ngroups, b, gpm);
  } else {
    k_line_solve<Gen, P, L><<<grid, L * P, smem, st>>>(G, line0, ngroups, b, 0);
  }
}

// Threads per row of the staged row solver: a warp for the shortest rows, else 5
// to 9 cells each (odd chunks), more on rows of over 4608 cells (512 threads: 19
// in FP64, 29 in FP32, 17 refined at the longest).
static int row_threads(int ncells) {
  return ncells <= 160 ? 32 : ncells <= 352 ? 64 : ncells <= 1152 ? 128 : ncells <= 2304 ? 256 : 512;
}

// Shared memory a CTA may have, queried once per device.
static int smem_optin() {
  static int optin[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 0;
  if (!optin[dev]) cudaDeviceGetAttribute(&optin[dev], cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return optin[dev];
}

// The staged row solver takes rows that one CTA's shared memory holds (beside
// its tables): 9344 cells in FP64, 14016 in FP32, 8009 refined. Longer ones keep
// the chunked solver with its scratch in global memory.
template <class Gen>
static bool row_fits(int ncells) {
  return row_smem<Gen>(ncells) + 8192 <= (size_t)smem_optin();
}

template <class Gen, int NT, int BATCH>
static void launch_row_nt(const Gen& G, int ncells, int lines, cudaStream_t st,
                          const Batch<typename Gen::Real>& b) {
  int dev = 0;
  cudaGetDevice(&dev);
  static bool attr[64] = {};
  if (dev < 64 && !attr[dev]) {
    cudaFuncSetAttribute(k_row_solve<Gen, NT, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         smem_optin() - 8192);
    attr[dev] = true;
  }
  const dim3 grid(lines, std::max(b.n, 1));
  const size_t smem = row_smem<Gen>(ncells);
  if constexpr ((BATCH & 2) != 0) launch_dependent(k_row_solve<Gen, NT, BATCH>, grid, NT, smem, st, G, b);
  else k_row_solve<Gen, NT, BATCH><<<grid, NT, smem, st>>>(G, b);
}

template <class Gen, int NT>
static void launch_row_b(const Gen& G, int ncells, int lines, cudaStream_t st,
                         const Batch<typename Gen::Real>& b) {
  const bool dep = dependent_launches(G.S, b);
  if (b.n > 0 && dep) launch_row_nt<Gen, NT, 3>(G, ncells, lines, st, b);
  else if (b.n > 0) launch_row_nt<Gen, NT, 1>(G, ncells, lines, st, b);
  else if (dep) launch_row_nt<Gen, NT, 2>(G, ncells, lines, st, b);
  else launch_row_nt<Gen, NT, 0>(G, ncells, lines, st, b);
}

template <class Gen>
static void launch_rows(const Gen& G, int ncells, int lines, cudaStream_t st,
                        const Batch<typename Gen::Real>& b) {
  switch (row_threads(ncells)) {
    case 32: return launch_row_b<Gen, 32>(G, ncells, lines, st, b);
    case 64: return launch_row_b<Gen, 64>(G, ncells, lines, st, b);
    case 128: return launch_row_b<Gen, 128>(G, ncells, lines, st, b);
    case 256: return launch_row_b<Gen, 256>(G, ncells, lines, st, b);
    default: return launch_row_b<Gen, 512>(G, ncells, lines, st, b);
  }
}

// The staged column solver takes columns of up to COL_MAX cells, a 32-byte
// sector of them per CTA (4 in FP64 and refined, 8 in FP32; 1100 cells take 106
// KB in FP64, 141 in FP32, 123 refined). Hydraulic x sweep, chunked -> staged: 64x32
// 50 -> 13 us, 256x128 31 -> 19, 512x256 32 -> 23, 1024x512 58 -> 42 (FP64); at
// 2048x1024 its 196 KB of rows in one CTA per SM lose (111 -> 220, two columns per
// CTA 168), so longer columns keep the chunks. (Where one round of CTAs takes all
// columns it wins further on, hydraulic and concentration 1300x300 70 -> 48 and 48 ->
// 42, refined 50 -> 37; in FP32 the line lies at 1300, 1500x300 40 -> 58.)
//
// Groups of four that leave a second round of CTAs not nearly full go to the chunks
// too, from 640 cells on, refined (two CTAs an SM up to about there) from 850 on. 590
// and 600 columns (148 and 150 groups on 148 SMs), staged / chunked, us: 620 cells
// hydraulic 29/46, 44/48, concentration 25/40, 40/40, refined 25/35, 27/35; 700
// cells 33/50, 52/50, 29/42, 46/42, 29/38, 31/39; 800 cells refined 31/42, 37/42;
// 900 cells 42/58, 66/58, 37/48, 62/48, 46/44, 64/44; 1100 cells with 900 columns
// 80/72, 76/64, 68/52. A step of two members of 1024x512 (256 groups) 465 -> 457 us; with
// more rounds the tail is a smaller part: six members of 900x200 (300 groups) 585
// against 607, three of 1101x500 (375) 713 against 744, eight of 1024x512 1584
// against 1596.
constexpr int COL_MAX = 1100;
template <class Gen>
constexpr int col_tail() {
  return Gen::REFINE ? 850 : 640;
}
template <class Gen>
constexpr int col_group() {
  return sizeof(typename Gen::Real) == 8 || Gen::REFINE ? 4 : 8;
}
template <class Gen>
static bool cols_fit(const StateT<typename Gen::Real>& S, int ncells, int lines, int members) {
  if (ncells > COL_MAX) return false;
  const long long groups = (long long)cdiv(lines, col_group<Gen>()) * std::max(members, 1);
  const int nsm = S.lslots / 2;
  return col_group<Gen>() != 4 || ncells <= col_tail<Gen>() || groups <= nsm || groups > 2 * nsm;
}

template <class Gen, int NT, int L, int BATCH>
static void launch_col_nt(const Gen& G, int ncells, int lines, cudaStream_t st,
                          const Batch<typename Gen::Real>& b) {
  int dev = 0;
  cudaGetDevice(&dev);
  static bool attr[64] = {};
  if (dev < 64 && !attr[dev]) {
    cudaFuncSetAttribute(k_col_solve<Gen, NT, L, BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)col_smem<Gen, L>(COL_MAX));
    attr[dev] = true;
  }
  const dim3 grid(cdiv(lines, L), std::max(b.n, 1));
  const size_t smem = col_smem<Gen, L>(ncells);
  if constexpr ((BATCH & 2) != 0)
    launch_dependent(k_col_solve<Gen, NT, L, BATCH>, grid, NT, smem, st, G, b);
  else
    k_col_solve<Gen, NT, L, BATCH><<<grid, NT, smem, st>>>(G, b);
}

// Threads of a column group: about eight cells each, four on short columns
// (where the rounds of loads, not their number, count).
template <class Gen, int L, int BATCH>
static void launch_col_l(const Gen& G, int ncells, int lines, cudaStream_t st,
                         const Batch<typename Gen::Real>& b) {
  const int cells = ncells * L;
  if (cells <= 512) launch_col_nt<Gen, 128, L, BATCH>(G, ncells, lines, st, b);
  else if (cells <= 1536) launch_col_nt<Gen, 256, L, BATCH>(G, ncells, lines, st, b);
  else if (L < 8 || cells <= 4096) launch_col_nt<Gen, 512, L, BATCH>(G, ncells, lines, st, b);
  else if constexpr (L == 8) launch_col_nt<Gen, 1024, L, BATCH>(G, ncells, lines, st, b);
}

template <class Gen, int L>
static void launch_cols(const Gen& G, int ncells, int lines, cudaStream_t st,
                        const Batch<typename Gen::Real>& b) {
  const bool dep = dependent_launches(G.S, b);
  if (b.n > 0 && dep) launch_col_l<Gen, L, 3>(G, ncells, lines, st, b);
  else if (b.n > 0) launch_col_l<Gen, L, 1>(G, ncells, lines, st, b);
  else if (dep) launch_col_l<Gen, L, 2>(G, ncells, lines, st, b);
  else launch_col_l<Gen, L, 0>(G, ncells, lines, st, b);
}

// Launches a sweep over `lines` lines and returns the number of launches: rows
// by the staged row solver, columns by the staged column solver, what these do
// not take by the chunked one, whose launch walks the line groups of every
// member of a batch (its persistent grid takes them in member order).
template <class Gen>
static int launch_lines(const Gen& G, int ncells, int lines, cudaStream_t st,
                        const Batch<typename Gen::Real>& b) {
  if constexpr (Gen::DIRECTION == 1) {
    if (row_fits<Gen>(ncells)) {
      launch_rows(G, ncells, lines, st, b);
      return 1;
    }
    const int groups = cdiv(lines, LPB);
    const long long total = (long long)groups * std::max(b.n, 1);
    launch_gen<Gen, 128>(G, st, (int)std::min<long long>(total, G.S.lslots), 0, (int)total, b,
                         b.n > 0 ? groups : 0);
    return 1;
  } else {
    if (cols_fit<Gen>(G.S, ncells, lines, b.n)) {
      launch_cols<Gen, col_group<Gen>()>(G, ncells, lines, st, b);
      return 1;
    }
    // groups of 8 adjacent columns of 128 chunks, one CTA of 1024 threads
    // per SM (a group's scratch slot is two of the 4-line slots)
    const int g8 = cdiv(lines, XPB);
    const long long total = (long long)g8 * std::max(b.n, 1);
    launch_gen<Gen, 128, XPB>(G, st, (int)std::min<long long>(total, G.S.lslots / 2), 0, (int)total, b,
                              b.n > 0 ? g8 : 0);
    return 1;
  }
}

// The FP32 forms' hydraulic sweeps: chunks per line, as many as keep at least
// four cells per chunk (of 128, 64, 32, 16, 4 or 1), so that no chunk of a short
// line is empty or holds its separator alone.
static int pair_chunks(int ncells) {
  int P = 128;
  while (P > 1 && ncells < P * 4) P >>= 1;
  return P == 8 ? 4 : P == 2 ? 1 : P;
}

// Groups of L lines of P chunks, a CTA each; a group of eight takes two of the
// scratch's 4-line slots. The scratch holds StateT::lslots slots of lines of
// 2*max(M, N) unknowns, so a sweep of shorter lines has proportionally more.
// Only the solvers of fewer than 128 chunks (smaller CTAs, more of them resident
// per SM) use them: their grid may then exceed the CTAs resident at once. (For
// the 128-chunk solvers the persistent grid of lslots CTAs measured as fast or
// faster.)
template <class Gen, int P, int L>
static int launch_pairs_p(const Gen& G, int ncells, int chunks, cudaStream_t st, const Batch<float>& b) {
  const int groups = cdiv(G.nl, L);
  const long long total = (long long)groups * std::max(b.n, 1);
  int slots = G.S.lslots;
  if (chunks < 128) slots *= std::max(1, std::max(G.S.M, G.S.N) / ncells);
  launch_gen<Gen, P, L>(G, st, (int)std::min<long long>(total, slots * LPB / L), 0, (int)total, b,
                        b.n > 0 ? groups : 0);
  return 1;
}

// Groups of eight lines where a line has 64 or 128 chunks (columns 64: only
// refined), else of four. On 2048x1024 (128 chunks of columns and rows), four ->
// eight: x refined 0.216 -> 0.154 ms, y 0.130 -> 0.121; the refined rows, alone, as
// 64 chunks 0.210 -> 0.204 (as 128 in a batch).
template <int DIR, bool REF>
static int launch_pairs(const StateT<float>& S, const CoefT<float>& c, cudaStream_t st,
                        const Batch<float>& b) {
  using Gen = PairGen<DIR, REF>;
  Gen G;
  G.bind(S, c);
  G.scratch = S.lscratch;
  G.lp0 = DIR == 0 ? S.x_lo : S.y_lo;
  G.nl = DIR == 0 ? S.x_hi - S.x_lo + 1 : S.N - S.y_lo + 1;
  if (G.nl <= 0) return 0;
  const int ncells = DIR == 0 ? S.N - 1 : S.M - 1, P = pair_chunks(ncells);
  switch (P) {
    case 128:
      if constexpr (DIR == 1 && REF) {
        if (b.n > 0) return launch_pairs_p<Gen, 128, LPB>(G, ncells, P, st, b);
        return launch_pairs_p<Gen, 64, XPB>(G, ncells, P, st, b);
      } else {
        return launch_pairs_p<Gen, 128, XPB>(G, ncells, P, st, b);
      }
    case 64: return launch_pairs_p<Gen, 64, (DIR == 1 || REF) ? XPB : LPB>(G, ncells, P, st, b);
    case 32: return launch_pairs_p<Gen, 32, LPB>(G, ncells, P, st, b);
    case 16: return launch_pairs_p<Gen, 16, LPB>(G, ncells, P, st, b);
    case 4: return launch_pairs_p<Gen, 4, LPB>(G, ncells, P, st, b);
    default: return launch_pairs_p<Gen, 1, LPB>(G, ncells, P, st, b);
  }
}

template <int DIR>
static int launch_dir(const State& S, const Coef& c, cudaStream_t st, const Batch<double>& b) {
  HydroGen<DIR> G;
  G.bind(S, c);
  G.scratch = S.lscratch;
  G.lp0 = DIR == 0 ? S.x_lo : S.y_lo;
  G.nl = DIR == 0 ? S.x_hi - S.x_lo + 1 : S.N - S.y_lo + 1;
  if (G.nl <= 0) return 0;
  return launch_lines(G, DIR == 0 ? S.N - 1 : S.M - 1, G.nl, st, b);
}

// ---------------------------------------------------------------------
// Concentration sweeps: one unknown per cell, cells first+1..last-1 of each
// wet segment of at least three cells (Scan_FSj / Scan_FSi,
// sediment_transport.cpp:51-164, 204-313; extraction :167-201, 316-349).
// DIR 0: columns j = 3..M-1 along i; DIR 1: rows i = 3..N-1 along j.
template <int DIR, class R, bool REF = false>
struct FSGen {
  using Real = R;
  static constexpr bool REFINE = REF;
  // the rows are in StateT::pre (k_fs_rows): the refinement reads them again
  static constexpr bool ROWS_AGAIN = true;
  static constexpr int AUX = 0;  // the emitter needs nothing but the solution
  static constexpr int SCRATCH_ARRAYS = REFINE ? 4 : 3;
  static constexpr int UPC = 1;
  static constexpr int DIRECTION = DIR;
  static constexpr int MIN_BLOCKS = 2;  // in both precisions
  StateT<R> S;
  CoefT<R> c;
  R* scratch;

  __host__ __device__ void bind(const StateT<R>& s, const CoefT<R>& cc) {
    S = s;
    c = cc;
  }
  __device__ int lines() const { return DIR == 0 ? S.M - 3 : S.N - 3; }
  __device__ int cells_per_line() const { return DIR == 0 ? S.N - 1 : S.M - 1; }
  __device__ int unknowns_per_line() const { return cells_per_line(); }
  __device__ int at(int lp, int p) const { return DIR == 0 ? p * S.W + lp : lp * S.W + p; }
  __device__ const R* vel() const { return DIR == 0 ? S.tu : S.tv; }

  __device__ int segments(int lp) const { return DIR == 0 ? S.mocj[lp] : S.moci[lp]; }
  // segment s of line position lp (false if the line has no such segment)
  __device__ bool segment(int lp, int s, SegD& d) const {
    const int n = segments(lp);
    const int first = (DIR == 0 ? S.dauj : S.daui)[lp * SEG + s];
    const int last = (DIR == 0 ? S.cuoij : S.cuoii)[lp * SEG + s];
    if (s >= n) return false;
    const int w = S.W;
    bool br1, br2;
    if (DIR == 0) {
      br1 = (first > 2) || ((first == 2) && ((S.h[1 * w + lp] + S.h[1 * w + lp - 1]) * 0.5 == c.NANGDAY));
      br2 = (last < S.N) || ((last == S.N) && ((S.h[S.N * w + lp] + S.h[S.N * w + lp - 1]) * 0.5 == c.NANGDAY));
    } else {
      br1 = (first > 2) || ((first == 2) && ((S.h[lp * w + first - 1] + S.h[(lp - 1) * w + first - 1]) * 0.5 == c.NANGDAY));
      br2 = (last < S.M) || ((last == S.M) && ((S.h[lp * w + last] + S.h[(lp - 1) * w + last]) * 0.5 == c.NANGDAY));
    }
    d.first = first;
    d.last = last;
    d.off = first + 1;
    d.rend = last - 1;  // rend < off: no interior row, nothing solved
    d.br1 = br1;
    d.br2 = br2;
    d.ran = d.qfirst = d.last_kind = d.xq_first = d.xq_last = 0;
    return true;
  }
  __device__ void load_segment(LineSeg& LS, int line, int s) const {
    const bool ok = line < lines();
    if (s == SEG) LS.nseg = ok ? segments(line_pos(line)) : 0;
    else if (ok) segment(line_pos(line), s, LS.s[s]);
  }

  // a cell's row for the staged row solver (rowsolve.cuh), from the fields
  struct Ops {
    R A, B, C, D;
  };
  __device__ int line_pos(int line) const { return line + 3; }
  __device__ Ops load(int lp, int pos) const {
    Ops o;
    if (DIR == 0) fs_row<0>(S, c, pos, lp, o.A, o.B, o.C, o.D);
    else fs_row<1>(S, c, lp, pos, o.A, o.B, o.C, o.D);
    return o;
  }
  __device__ void row(const SegD& d, int lp, int pos, const Ops& o, R& A, R& B, R& C, R& D) const {
    A = o.A;
    B = o.B;
    C = o.C;
    D = o.D;
    end_rows(d, lp, pos, A, B, C, D);
  }
  __device__ void keep(const SegD&, int, int, const Ops&) const {}
  __device__ void prefetch(int lp) const {
    const int w = S.W;
    const size_t r = (size_t)lp * w;
    prefetch_l2(S.Hmoi + r + 2 * w, w);
    prefetch_l2(S.FS + r + w, w);
    prefetch_l2(S.VTH + r, w);
    prefetch_l2(S.Fw + r, w);
    prefetch_l2(S.tv + r, w);
    prefetch_l2(S.Htdv + r, w);
    prefetch_l2(S.Ky + r, w);
    prefetch_l2(S.tu + r, w);
    prefetch_l2(S.Htdu + r, w);
    prefetch_l2(S.Kx + r, w);
  }
  // the value stored for a solved concentration
  __device__ R stored(double x) const { return (x < 0) ? c.NDnen : (R)x; }
  // Writes tFS at cell pos, first <= pos <= last, of segment d, the ends as
  // fixup does. value(p): the solved concentration of cell p.
  template <class V>
  __device__ void emit_cell(const SegD& d, int lp, int pos, V value) const {
    if (d.rend < d.off) return;
    const R* v = vel();
    const int g = at(lp, pos);
    if (pos == d.first)
      S.tFS[g] = (d.br1 || v[g] == 0) ? stored(value(pos + 1)) : S.FS[g];
    else if (pos == d.last)
      S.tFS[g] = (d.br2 || v[g] == 0) ? stored(value(pos - 1)) : S.FS[g];
    else
      S.tFS[g] = stored(value(pos));
  }

  // Walks a chunk cell by cell; the rows come from k_fs_rows (one coalesced
  // per-cell pass ahead of the sweep), only the segment ends are set here.
  struct Walker {
    int lp, si, pos;
    bool in;
    __device__ void init(const FSGen& G, const LineSeg& LS, int line, int c0) {
      lp = line + 3;
      si = 0;
      in = false;
    }
    __device__ void cell(const FSGen& G, const LineSeg& LS, int cc) {
      pos = cc + 2;
      while (si < LS.nseg && LS.s[si].last < pos) ++si;
      in = si < LS.nseg && LS.s[si].off <= pos && pos <= LS.s[si].rend;
    }
    __device__ void row(const FSGen& G, const LineSeg& LS, int, R& A, R& B, R& C, R& D) const {
      if (!in) {
        A = 0; B = 1; C = 0; D = 0;
        return;
      }
      G.row_in(LS.s[si], lp, pos, A, B, C, D);
    }
  };

  // The row of cell pos of line position lp inside segment d: as k_fs_rows
  // wrote it, then the segment's end conditions.
  __device__ void row_in(const SegD& d, int lp, int pos, R& A, R& B, R& C, R& D) const {
    load_row(lp, pos, A, B, C, D);
    end_rows(d, lp, pos, A, B, C, D);
  }
  __device__ void load_row(int lp, int pos, R& A, R& B, R& C, R& D) const {
    const size_t n = (size_t)S.W * S.H;
    const R* q = S.pre + at(lp, pos);
    A = q[0];
    B = q[n];
    C = q[2 * n];
    D = q[3 * n];
  }
  __device__ void end_rows(const SegD& d, int lp, int pos, R& A, R& B, R& C, R& D) const {
    const R* v = vel();
    if (pos == d.first + 1) {
      // the velocity at the segment's first cell is the previous cell's
      if (d.br1 || v[at(lp, d.first)] == 0) B = B + A;
      else D = D - A * S.FS[at(lp, d.first)];
      A = 0;
    }
    if (pos == d.last - 1) {
      // '&&' in the i-sweep (sediment_transport.cpp:304), '||' in the j-sweep (:153)
      const bool zero = v[at(lp, d.last)] == 0;
      if (DIR == 0 ? (d.br2 && zero) : (d.br2 || zero)) B = B + C;
      else D = D - C * S.FS[at(lp, d.last)];
      C = 0;
    }
  }

  // The rows of a line again, unknown by unknown in decreasing order (the
  // refinement's residuals): the same values the Walker gave pass A.
  struct RowCursor {
    int lp, si;
    __device__ void init(const FSGen& G, const LineSeg& LS, int line) {
      lp = line + 3;
      si = LS.nseg - 1;
    }
    __device__ void row(const FSGen& G, const LineSeg& LS, int q, R& A, R& B, R& C, R& D) {
      const int pos = q + 2;
      while (si >= 0 && LS.s[si].first > pos) --si;
      if (si < 0 || pos < LS.s[si].off || pos > LS.s[si].rend) {
        A = 0; B = 1; C = 0; D = 0;
        return;
      }
      G.row_in(LS.s[si], lp, pos, A, B, C, D);
    }
  };

  // FWD: the unknowns come in increasing order (init_fwd), else decreasing.
  struct Emitter {
    int lp, si;
    __device__ void init(const FSGen& G, const LineSeg& LS, int line) {
      lp = line + 3;
      si = LS.nseg - 1;
    }
    __device__ void init_fwd(const FSGen& G, const LineSeg& LS, int line) {
      lp = line + 3;
      si = -1;
    }
    template <bool FWD = false>
    __device__ void emit(const FSGen& G, const LineSeg& LS, double* xlast, int q, double x, double,
                         R) {
      const int pos = q + 2;
      if constexpr (FWD) {
        while (si + 1 < LS.nseg && LS.s[si + 1].first <= pos) ++si;
      } else {
        while (si >= 0 && LS.s[si].first > pos) --si;
      }
      if (si < 0) return;
      const SegD& d = LS.s[si];
      if (pos < d.off || pos > d.rend) return;
      G.S.tFS[G.at(lp, pos)] = G.stored(x);
    }
  };

  __device__ void fixup(const LineSeg& LS, const double* xlast, int line, int s) const {
    const SegD& d = LS.s[s];
    if (d.rend < d.off) return;
    const int lp = line + 3;
    const R* v = vel();
    R* tFS = S.tFS;
    tFS[at(lp, d.first)] = (d.br1 || v[at(lp, d.first)] == 0) ? tFS[at(lp, d.first + 1)]
                                                               : S.FS[at(lp, d.first)];
    tFS[at(lp, d.last)] = (d.br2 || v[at(lp, d.last)] == 0) ? tFS[at(lp, d.last - 1)]
                                                             : S.FS[at(lp, d.last)];
  }
};

// whether the concentration sweep forms its rows itself (else k_fs_rows
// writes them ahead of it)
template <class R>
bool fs_rows_in_sweep(const StateT<R>& S, int dir, const Batch<R>& b) {
  if constexpr (sizeof(R) == 4) {
    if (S.refine && dir == 0) return cols_fit<FSGen<0, R, true>>(S, S.N - 1, S.M - 3, b.n);
    if (S.refine) return row_fits<FSGen<1, R, true>>(S.M - 1);
  }
  if (dir == 0) return cols_fit<FSGen<0, R, false>>(S, S.N - 1, S.M - 3, b.n);
  return row_fits<FSGen<1, R, false>>(S.M - 1);
}

template <class R>
int launch_fs_sweep(const StateT<R>& S, const CoefT<R>& c, int dir, cudaStream_t st,
                    const Batch<R>& b) {
  const int ncells = dir == 0 ? S.N - 1 : S.M - 1;
  const int lines = dir == 0 ? S.M - 3 : S.N - 3;
  if (lines <= 0) return 0;
  if constexpr (sizeof(R) == 4) {
    if (S.refine && dir == 0)
      return launch_lines(FSGen<0, R, true>{S, c, S.lscratch}, ncells, lines, st, b);
    if (S.refine) return launch_lines(FSGen<1, R, true>{S, c, S.lscratch}, ncells, lines, st, b);
  }
  if (dir == 0) return launch_lines(FSGen<0, R, false>{S, c, S.lscratch}, ncells, lines, st, b);
  return launch_lines(FSGen<1, R, false>{S, c, S.lscratch}, ncells, lines, st, b);
}

template <class R>
int launch_sweep(const StateT<R>& S, const CoefT<R>& c, int dir, cudaStream_t st,
                 const Batch<R>& b) {
  if constexpr (sizeof(R) == 4) {
    if (S.refine && dir == 0) return launch_pairs<0, true>(S, c, st, b);
    if (S.refine) return launch_pairs<1, true>(S, c, st, b);
    if (dir == 0) return launch_pairs<0, false>(S, c, st, b);
    return launch_pairs<1, false>(S, c, st, b);
  } else {
    if (dir == 0) return launch_dir<0>(S, c, st, b);
    return launch_dir<1>(S, c, st, b);
  }
}

template bool fs_rows_in_sweep<double>(const StateT<double>&, int, const Batch<double>&);
template bool fs_rows_in_sweep<float>(const StateT<float>&, int, const Batch<float>&);
template int launch_sweep<double>(const StateT<double>&, const CoefT<double>&, int, cudaStream_t,
                                  const Batch<double>&);
template int launch_sweep<float>(const StateT<float>&, const CoefT<float>&, int, cudaStream_t,
                                 const Batch<float>&);
template int launch_fs_sweep<double>(const StateT<double>&, const CoefT<double>&, int, cudaStream_t,
                                     const Batch<double>&);
template int launch_fs_sweep<float>(const StateT<float>&, const CoefT<float>&, int, cudaStream_t,
                                    const Batch<float>&);

}  // namespace hyd
