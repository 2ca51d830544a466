// The line-preconditioned predictor solve, in the precision T of its inner
// iteration (float: the mixed form, gw_cg_mixed.cu; double: the FP64 line
// form, gw_cg_line64.cu): inner preconditioned CG inside FP64 defect
// correction on the true residual.
//
//   x = the assembly's starting iterate (h^n, or its extrapolation)
//   repeat (outer sweep o = 0, 1, ...):
//     x <- x + S d;  r = b - A x  in FP64 with the FP64 coefficients
//     stop when ||r||_2 <= outer_rtol ||b||_2 (after at least one
//     correction: a start passing the test is not accurate enough)
//     solve (S A S) d = S r approximately in T: CG preconditioned by the exact
//     solve of each column's vertical tridiagonal block (line Jacobi along k),
//     stopped at inner_rtol of the initial preconditioned norm (z'r)^(1/2)
//
// The line preconditioner follows the thin-layer anisotropy of the head
// system (dz << dx makes the vertical legs 10^2-10^3 times the lateral ones):
// it solves the dominant couplings exactly and cuts the inner iteration count
// by an order of magnitude against point Jacobi.  Every iterate that leaves
// the solve is an FP64 vector whose FP64 residual met outer_rtol, so the
// solution's accuracy is set by the FP64 sweep, not by T's arithmetic.
//
// S is the square root of the column factor's pivots (gw_linesolve.cuh), so
// one array l is both the vertical block and its factor and the iteration
// reads l, gx, gy where the unscaled form read diag, gx, gy, gz, 1/d and l.
// LPC lanes own a column, E cells each, in both passes of an iteration:
//   pass A: p = z + bc p_old (at the cell's column and its four neighbours'),
//           w = A p with the block as Lh (Lh' p), p'w; every second
//           iteration d += the last two al p;
//   pass B: r -= al w, z = (Lh Lh')^-1 r, z'r;
// with a grid barrier that sums (grid_sum) after each.  Words of T per cell and
// iteration: A reads z, p_old, gx, gy, l, writes p, w, and half the time reads
// d and the p before p_old and writes d; B reads r, w, l, writes r, z: 13.5
// (54 B in FP32) against 16 unscaled with d updated every iteration.
//
// Measured against the unscaled form (cells by the flat index in pass A,
// unpadded columns), both with the present barrier: 64x64x128 mixed 11.5 ->
// 10.1 us an iteration, 256x256x128 117 -> 98 us; whole solves of few
// iterations 128x128x200 0.72 -> 0.35 ms, 128x128x199 0.84 -> 0.45 ms, 24x20x300
// 0.27 -> 0.13 ms, the batched solve of a 24-member ensemble 4.1 -> 2.4 ms.  At
// 256x256x128 it moves 54 B a cell and iteration through HBM at 5.1 TB/s:
// latency of the 16 warps an SM at 128 registers holds.  28 warps at 72
// registers took 95 us an iteration but spilled the FP64 sweep, 3.7 ms in the
// ensemble's solve; tiles of 4 x 4 columns a block (for L1 hits in j) took 105 us.
#pragma once

#include "gw_coop.cuh"
#include "gw_internal.h"
#include "gw_linefactor.cuh"

namespace fgw {

using namespace coop;

constexpr int kLineBlock = 512;

template <typename T>
struct LineArgs {
  Dims d;
  const double *diag, *gxp, *gyp, *gzp, *b;
  double *x0, *x1;           // iterate ping-pong (x0 holds the start at entry)
  LineVecs<T> v;
  double* part;              // kRedSlots x G
  CgState* st;
  double outer_rtol, inner_rtol, atol;
  int max_inner, max_outer, max_total;
  int variant;               // batched solves: the member's line_variant
  Peers peers;               // batched solves: the launch's members
};

// The inner solve's correction not yet in x: d (when set) plus the last one or
// two updates e1 p1 + e2 p2.
template <typename T>
struct Pending {
  const T *p1, *p2;
  T e1, e2;
  bool dset;
};

// The words of a warp's own columns held in shared memory, W of them in this
// order; W = 0 for chunked columns and domains too large.
enum LineOwn { kLineW = 0, kLineR, kLineL, kLineGym, kLineGxm, kLineGx, kLineGy };

// WATCH: in a batched launch.
template <typename T, int LPC, int E, bool DEEP, int W = 0, bool WATCH = false>
struct LineSolve {
  static constexpr int kCols = 32 / LPC;
  static_assert(W == 0 || (E == 4 && !DEEP), "one quad a lane");

  // This thread's quad of a word for its m-th column (own: the block's words,
  // `per` columns a warp).
  struct Own {
    Quad<T>* q;
    int per;
    __device__ __forceinline__ Quad<T>& at(int word, int m) const {
      return q[(word * per + m) * kLineBlock + threadIdx.x];
    }
  };
  template <int WORD>
  __device__ static __forceinline__ void ld_own(const Own& own, int m, const T* p, int n,
                                                T (&v)[E]) {
    if constexpr (W > WORD) {
      const Quad<T> t = own.at(WORD, m);
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = t.v[e];
    } else {
      ld_cells<E>(p, n, v);
    }
  }
  template <int WORD>
  __device__ static __forceinline__ void st_own(const Own& own, int m, T* p, int n,
                                                const T (&v)[E]) {
    if constexpr (W > WORD) own.at(WORD, m) = Quad<T>{{v[0], v[1], v[2], v[3]}};
    else st_cells<E>(p, n, v);
  }
  // A leg: from shared memory, or (the solve's first pass A) from its array
  // into it.
  template <int WORD>
  __device__ static __forceinline__ void ld_leg(const Own& own, int m, bool fill, const T* p, int n,
                                                T (&v)[E]) {
    if constexpr (W > WORD) {
      if (fill) {
        ld_cells<E>(p, n, v);
        own.at(WORD, m) = Quad<T>{{v[0], v[1], v[2], v[3]}};
        return;
      }
    }
    ld_own<WORD>(own, m, p, n, v);
  }

  // A lane's place in its column: the column, its neighbours' strides and the
  // lane's first cell.
  struct Place {
    long long cp, cu;  // column offsets: padded (T) and FP64 arrays
    int k0, n, q;      // first cell, cells in the padded column, lane in column
  };

  __device__ static __forceinline__ bool place(const LineArgs<T>& a, int base, int kb, Place& p) {
    const Dims& d = a.d;
    const int lane = threadIdx.x & 31;
    p.q = lane % LPC;
    const int c = base + lane / LPC;
    const bool act = c < d.nx * d.ny;
    const int j = act ? c / d.nx : 0, i = act ? c - j * d.nx : 0;
    const long long col = col2(d, j + 1, i + 1);
    const int nzp = line_nzp(d.nz);
    p.cp = col * nzp;
    p.cu = col * d.nz;
    p.k0 = kb + p.q * E;
    p.n = act ? max(0, min(E, nzp - p.k0)) : 0;
    return act;
  }

  // S d + pending at the lane's cells of the column at padded offset cp.
  __device__ static __forceinline__ void corrected(const LineArgs<T>& a, const Pending<T>& pd,
                                                   const double* xo, long long cp, long long cu,
                                                   int k0, int n, bool even, bool first,
                                                   double (&xv)[E]) {
    const int nz = a.d.nz;
    ld_x(xo + cu + k0, min(n, nz - k0), even, xv);
    if (first) return;
    T s[E], c[E], p[E];
    ld_cells<E>(a.v.s + cp + k0, n, s);
    ld_cells<E>(pd.p1 + cp + k0, n, p);
    if (pd.dset) {
      ld_cells<E>(a.v.d + cp + k0, n, c);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) c[e] = T(0);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) c[e] += pd.e1 * p[e];
    if (pd.e2 != T(0)) {
      ld_cells<E>(pd.p2 + cp + k0, n, p);
#pragma unroll
      for (int e = 0; e < E; ++e) c[e] += pd.e2 * p[e];
    }
#pragma unroll
    for (int e = 0; e < E; ++e) xv[e] += static_cast<double>(s[e]) * static_cast<double>(c[e]);
  }

  // n cells of an FP64 array (column pitch nz: pairs only where nz is even).
  __device__ static __forceinline__ void ld_x(const double* p, int n, bool even, double (&v)[E]) {
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = 0.0;
    if (even) {
#pragma unroll
      for (int e = 0; e < E; e += 2) {
        if (e < n) {
          const double2 t = *reinterpret_cast<const double2*>(p + e);
          v[e] = t.x;
          v[e + 1] = t.y;
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e < n) v[e] = p[e];
    }
  }
  __device__ static __forceinline__ void st_x(double* p, int n, bool even, const double (&v)[E]) {
    if (even) {
#pragma unroll
      for (int e = 0; e < E; e += 2)
        if (e < n) *reinterpret_cast<double2*>(p + e) = make_double2(v[e], v[e + 1]);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (e < n) p[e] = v[e];
    }
  }

  // z = (Lh Lh')^-1 r of the column whose lane cells are r (chunked: y goes
  // through z, the chunks forward then backward); z'r accumulated in FP64.
  __device__ static __forceinline__ void solve_store(T* __restrict__ z, const T (&l)[E],
                                                     const T (&r)[E], const Place& p, double& zr) {
    T lm = __shfl_up_sync(kFull, l[E - 1], 1, LPC);
    if (p.q == 0) lm = T(0);
    T y[E], zv[E];
    line_forward<LPC, E>(l, lm, r, T(0), p.q, y);
    line_backward<LPC, E>(l, y, T(0), p.q, zv);
    st_cells<E>(z + p.cp + p.k0, p.n, zv);
#pragma unroll
    for (int e = 0; e < E; ++e) zr += static_cast<double>(zv[e]) * static_cast<double>(r[e]);
  }
  // The chunked column's solve: the forward sweep chunk by chunk as r is made
  // (y through z, its last value carried; z'r = y'y), then the backward one.
  __device__ static __forceinline__ void deep_forward(const LineArgs<T>& a, const Place& p,
                                                      const T (&r)[E], T& carry, double& zr) {
    T l[E], y[E];
    ld_cells<E>(a.v.l + p.cp + p.k0, p.n, l);
    T lm = __shfl_up_sync(kFull, l[E - 1], 1, LPC);
    if (p.q == 0) lm = p.k0 > 0 ? a.v.l[p.cp + p.k0 - 1] : T(0);
    line_forward<LPC, E>(l, lm, r, carry, p.q, y);
    st_cells<E>(a.v.z + p.cp + p.k0, p.n, y);
    carry = __shfl_sync(kFull, y[E - 1], LPC - 1, LPC);
#pragma unroll
    for (int e = 0; e < E; ++e) zr += static_cast<double>(y[e]) * static_cast<double>(y[e]);
  }
  __device__ static __forceinline__ void deep_backward(const LineArgs<T>& a, int base) {
    const int nzp = line_nzp(a.d.nz), chunk = LPC * E;
    T carry = T(0);
    for (int kb = (nzp - 1) / chunk * chunk; kb >= 0; kb -= chunk) {
      Place p;
      place(a, base, kb, p);
      T l[E], y[E], z[E];
      ld_cells<E>(a.v.l + p.cp + p.k0, p.n, l);
      ld_cells<E>(a.v.z + p.cp + p.k0, p.n, y);
      line_backward<LPC, E>(l, y, carry, p.q, z);
      st_cells<E>(a.v.z + p.cp + p.k0, p.n, z);
      carry = __shfl_sync(kFull, z[0], 0, LPC);
    }
  }

  // Outer sweep over a warp's columns: x_new = x + S (d + pending), r = S (b -
  // A x_new), z; on the first (nothing pending, x_new = x) also the scaled
  // lateral legs and b'b.
  template <bool FIRST>
  __device__ static __forceinline__ void outer(const LineArgs<T>& a, const Own& own, const Pending<T>& pd,
                                               const double* xo, double* xn, int gwarp, int nwarp,
                                               double& bb, double& rn2, double& zr) {
    const Dims& d = a.d;
    const int nz = d.nz, nzp = line_nzp(nz);
    const bool even = (nz & 1) == 0;
    const long long sxp = nzp, syp = static_cast<long long>(d.nx2) * nzp, sx = d.sx, sy = d.sy;
    const double *const b = a.b, *const diag = a.diag, *const gxp = a.gxp, *const gyp = a.gyp,
                 *const gzp = a.gzp;
    int m = 0;
    for (int base = gwarp * kCols; base < d.nx * d.ny; base += nwarp * kCols, ++m) {
      T carry = T(0);
      for (int kb = 0; kb < (DEEP ? nzp : 1); kb += LPC * E) {
        Place p;
        place(a, base, kb, p);
        const int n = p.n, nx = min(n, nz - p.k0);
        const long long cp = p.cp, cu = p.cu, f = cu + p.k0;
        const int k0 = p.k0;
        double xc[E], xw[E], xe[E], xs[E], xnn[E];
        corrected(a, pd, xo, cp, cu, k0, n, even, FIRST, xc);
        corrected(a, pd, xo, cp - sxp, cu - sx, k0, n, even, FIRST, xw);
        corrected(a, pd, xo, cp + sxp, cu + sx, k0, n, even, FIRST, xe);
        corrected(a, pd, xo, cp - syp, cu - sy, k0, n, even, FIRST, xs);
        corrected(a, pd, xo, cp + syp, cu + sy, k0, n, even, FIRST, xnn);
        double xu = __shfl_up_sync(kFull, xc[E - 1], 1, LPC);
        double xd = __shfl_down_sync(kFull, xc[0], 1, LPC);
        if (DEEP) {  // the chunk's edge lanes take the neighbouring chunks' cells
          const auto at = [&](int k) {
            double v = xo[cu + k];
            if (!FIRST) {
              T c = pd.dset ? a.v.d[cp + k] : T(0);
              c += pd.e1 * pd.p1[cp + k];
              if (pd.e2 != T(0)) c += pd.e2 * pd.p2[cp + k];
              v += static_cast<double>(a.v.s[cp + k]) * static_cast<double>(c);
            }
            return v;
          };
          if (p.q == 0) xu = (n > 0 && k0 > 0) ? at(k0 - 1) : 0.0;
          if (p.q == LPC - 1) xd = (n > 0 && k0 + E < nz) ? at(k0 + E) : 0.0;
        }
        double g[E], g2[E], bv[E], ax[E];
        ld_x(gyp + f - sy, nx, even, g);
        ld_x(gxp + f - sx, nx, even, g2);
#pragma unroll
        for (int e = 0; e < E; ++e) ax[e] = g[e] * xs[e] + g2[e] * xw[e];
        ld_x(gzp + f, nx, even, g);
        ld_x(diag + f, nx, even, g2);
        double gu = __shfl_up_sync(kFull, g[E - 1], 1, LPC);
        if (p.q == 0) gu = (DEEP && n > 0 && k0 > 0) ? gzp[f - 1] : 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
          ax[e] += (e == 0 ? gu : g[e > 0 ? e - 1 : 0]) * (e == 0 ? xu : xc[e > 0 ? e - 1 : 0]);
          ax[e] += g2[e] * xc[e];
          ax[e] += g[e] * (e + 1 < E ? xc[e + 1 < E ? e + 1 : e] : xd);
        }
        ld_x(gxp + f, nx, even, g);
        ld_x(gyp + f, nx, even, g2);
        ld_x(b + f, nx, even, bv);
        T s[E], r[E];
        ld_cells<E>(a.v.s + cp + k0, n, s);
        if (FIRST) {  // scaled lateral legs
          T se[E], sn[E], lg[E];
          ld_cells<E>(a.v.s + cp + sxp + k0, n, se);
          ld_cells<E>(a.v.s + cp + syp + k0, n, sn);
#pragma unroll
          for (int e = 0; e < E; ++e)
            lg[e] = static_cast<T>(g[e] * static_cast<double>(s[e]) * static_cast<double>(se[e]));
          st_cells<E>(a.v.gx + cp + k0, n, lg);
#pragma unroll
          for (int e = 0; e < E; ++e)
            lg[e] = static_cast<T>(g2[e] * static_cast<double>(s[e]) * static_cast<double>(sn[e]));
          st_cells<E>(a.v.gy + cp + k0, n, lg);
        } else {
          st_x(xn + f, nx, even, xc);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
          ax[e] += g[e] * xe[e];
          ax[e] += g2[e] * xnn[e];
          const double rr = e < nx ? bv[e] - ax[e] : 0.0;
          if (FIRST) bb += bv[e] * bv[e];
          rn2 += rr * rr;
          r[e] = static_cast<T>(static_cast<double>(s[e]) * rr);
        }
        st_own<kLineR>(own, m, a.v.r + cp + k0, n, r);
        if (!DEEP) {
          T l[E];
          ld_leg<kLineL>(own, m, FIRST, a.v.l + cp + k0, n, l);
          solve_store(a.v.z, l, r, p, zr);
        } else {
          deep_forward(a, p, r, carry, zr);
        }
      }
      if (DEEP) deep_backward(a, base);
    }
  }

  // Pass A.  FIRST: p = z.  YUP: d takes the two pending updates (al1 of
  // p_old, al2 of the p in p_new's buffer; DNEW: d = al1 p_old, not read).
  template <bool FIRST, bool YUP, bool DNEW>
  __device__ static __forceinline__ double pass_a(const LineArgs<T>& a, const Own& own, bool fill, T bc, T al1, T al2,
                                                  const T* pold, T* pnew, int gwarp, int nwarp) {
    const Dims& d = a.d;
    const int nzp = line_nzp(d.nz);
    const long long sxp = nzp, syp = static_cast<long long>(d.nx2) * nzp;
    const T *const zv = a.v.z, *const gxv = a.v.gx, *const gyv = a.v.gy, *const lv = a.v.l;
    T *const dv = a.v.d, *const wv = a.v.w;
    double pw = 0.0;
    int m = 0;
    for (int base = gwarp * kCols; base < d.nx * d.ny; base += nwarp * kCols, ++m) {
      for (int kb = 0; kb < (DEEP ? nzp : 1); kb += LPC * E) {
        Place p;
        place(a, base, kb, p);
        const int n = p.n;
        const long long c = p.cp + p.k0;
        T P[E], po[E], l[E], w[E];
        ld_cells<E>(zv + c, n, P);
        if (!FIRST) ld_cells<E>(pold + c, n, po);
        ld_own<kLineL>(own, m, lv + c, n, l);
        // The four lateral neighbours, two directions at a time.
        T za[E], pa[E], ga[E], zb[E], pb[E], gb[E];
        ld_cells<E>(zv + c - syp, n, za);
        if (!FIRST) ld_cells<E>(pold + c - syp, n, pa);
        ld_leg<kLineGym>(own, m, fill, gyv + c - syp, n, ga);
        ld_cells<E>(zv + c - sxp, n, zb);
        if (!FIRST) ld_cells<E>(pold + c - sxp, n, pb);
        ld_leg<kLineGxm>(own, m, fill, gxv + c - sxp, n, gb);
#pragma unroll
        for (int e = 0; e < E; ++e) {
          w[e] = ga[e] * (FIRST ? za[e] : za[e] + bc * pa[e]);
          w[e] += gb[e] * (FIRST ? zb[e] : zb[e] + bc * pb[e]);
        }
        ld_cells<E>(zv + c + sxp, n, za);
        if (!FIRST) ld_cells<E>(pold + c + sxp, n, pa);
        ld_leg<kLineGx>(own, m, fill, gxv + c, n, ga);
        ld_cells<E>(zv + c + syp, n, zb);
        if (!FIRST) ld_cells<E>(pold + c + syp, n, pb);
        ld_leg<kLineGy>(own, m, fill, gyv + c, n, gb);
        T dd[E], pp[E];
        if (YUP && !DNEW) {
          ld_cells<E>(dv + c, n, dd);
          ld_cells<E>(pnew + c, n, pp);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) {
          w[e] += ga[e] * (FIRST ? za[e] : za[e] + bc * pa[e]);
          w[e] += gb[e] * (FIRST ? zb[e] : zb[e] + bc * pb[e]);
          if (!FIRST) P[e] = P[e] + bc * po[e];
        }
        // The column's block as Lh (Lh' p): u_k = p_k + l_k p_{k+1},
        // w_k += u_k + l_{k-1} u_{k-1}.
        T pn = __shfl_down_sync(kFull, P[0], 1, LPC);
        T lm = __shfl_up_sync(kFull, l[E - 1], 1, LPC);
        if (DEEP && p.q == LPC - 1) {
          const long long f = c + E;
          pn = (n > 0 && p.k0 + E < nzp) ? (FIRST ? zv[f] : zv[f] + bc * pold[f]) : T(0);
        }
        if (p.q == LPC - 1 && !DEEP) pn = T(0);
        T u[E];
#pragma unroll
        for (int e = 0; e < E; ++e) u[e] = P[e] + l[e] * (e + 1 < E ? P[e + 1 < E ? e + 1 : e] : pn);
        T um = __shfl_up_sync(kFull, u[E - 1], 1, LPC);
        if (p.q == 0) {
          lm = T(0);
          um = T(0);
          if (DEEP && n > 0 && p.k0 > 0) {
            lm = lv[c - 1];
            um = (FIRST ? zv[c - 1] : zv[c - 1] + bc * pold[c - 1]) + lm * P[0];
          }
        }
#pragma unroll
        for (int e = 0; e < E; ++e)
          w[e] += u[e] + (e == 0 ? lm : l[e > 0 ? e - 1 : 0]) * (e == 0 ? um : u[e > 0 ? e - 1 : 0]);
        st_cells<E>(pnew + c, n, P);
        st_own<kLineW>(own, m, wv + c, n, w);
        if (YUP) {
#pragma unroll
          for (int e = 0; e < E; ++e)
            dd[e] = DNEW ? al1 * po[e] : dd[e] + (al1 * po[e] + al2 * pp[e]);
          st_cells<E>(dv + c, n, dd);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) pw += static_cast<double>(P[e]) * static_cast<double>(w[e]);
      }
    }
    return pw;
  }

  // Pass B, kPassB columns of a warp at a time: three loads a cell leave too
  // few bytes in flight one column after the other.
  static constexpr int kPassB = DEEP || sizeof(T) > 4 || W > kLineL ? 1 : 16 / E;
  __device__ static __forceinline__ double pass_b(const LineArgs<T>& a, const Own& own, T al, int gwarp, int nwarp) {
    const Dims& d = a.d;
    const int nzp = line_nzp(d.nz), ncols = d.nx * d.ny, step = nwarp * kCols;
    const T *const wv = a.v.w, *const lv = a.v.l;
    T *const rv = a.v.r, *const zv = a.v.z;
    double zr = 0.0;
    int m = 0;
    for (int base = gwarp * kCols; base < ncols; base += kPassB * step, m += kPassB) {
      if constexpr (DEEP) {
        T carry = T(0);
        for (int kb = 0; kb < nzp; kb += LPC * E) {
          Place p;
          place(a, base, kb, p);
          const long long c = p.cp + p.k0;
          T w[E], r[E];
          ld_cells<E>(wv + c, p.n, w);
          ld_cells<E>(rv + c, p.n, r);
#pragma unroll
          for (int e = 0; e < E; ++e) r[e] -= al * w[e];
          st_cells<E>(rv + c, p.n, r);
          deep_forward(a, p, r, carry, zr);
        }
        deep_backward(a, base);
      } else {
        Place p[kPassB];
        T w[kPassB][E], r[kPassB][E], l[kPassB][E];
#pragma unroll
        for (int u = 0; u < kPassB; ++u) {
          place(a, base + u * step, 0, p[u]);
          const long long c = p[u].cp + p[u].k0;
          ld_own<kLineW>(own, m + u, wv + c, p[u].n, w[u]);
          ld_own<kLineR>(own, m + u, rv + c, p[u].n, r[u]);
          ld_own<kLineL>(own, m + u, lv + c, p[u].n, l[u]);
        }
#pragma unroll
        for (int u = 0; u < kPassB; ++u) {
          if (u > 0 && base + u * step >= ncols) break;
#pragma unroll
          for (int e = 0; e < E; ++e) r[u][e] -= al * w[u][e];
          st_own<kLineR>(own, m + u, rv + p[u].cp + p[u].k0, p[u].n, r[u]);
          solve_store(zv, l[u], r[u], p[u], zr);
        }
      }
    }
    return zr;
  }

  __device__ static __forceinline__ void run(const LineArgs<T>& a, const int bid, const int G,
                                             Quad<T>* words = nullptr, int per = 0) {
    const Own own{words, per};
    const int gwarp = bid * (kLineBlock / 32) + (threadIdx.x >> 5), nwarp = G * (kLineBlock / 32);
    unsigned epoch = 0;
    double bnorm = 0.0, rnorm = 0.0;
    int total = 0, outers = 0, reason = 0, cur = 0;  // x is in x1 when cur
    Pending<T> pd{a.v.p0, a.v.p1, T(0), T(0), false};
    for (int o = 0;; ++o) {
      double s[3] = {0.0, 0.0, 0.0};
      if (o == 0) {
        outer<true>(a, own, pd, a.x0, a.x1, gwarp, nwarp, s[2], s[0], s[1]);
        if (!grid_sum<kLineBlock, WATCH>(s, a.part, bid, G, epoch, a.st, a.peers)) return;
        bnorm = sqrt(s[2]);
      } else {
        outer<false>(a, own, pd, cur ? a.x1 : a.x0, cur ? a.x0 : a.x1, gwarp, nwarp, s[2], s[0], s[1]);
        double s2[2] = {s[0], s[1]};
        if (!grid_sum<kLineBlock, WATCH>(s2, a.part, bid, G, epoch, a.st, a.peers)) return;
        s[0] = s2[0];
        s[1] = s2[1];
        cur ^= 1;
      }
      rnorm = sqrt(s[0]);
      double beta = s[1];
      const double zn0 = sqrt(beta);
      if (!isfinite(rnorm)) {
        reason = -9;
        break;
      }
      // The start is never returned unrefined, even where it meets the test.
      if (o > 0 && rnorm <= fmax(a.outer_rtol * bnorm, a.atol)) {
        reason = (rnorm < a.atol) ? 3 : 2;
        break;
      }
      if (outers >= a.max_outer || total >= a.max_total) {
        reason = -3;
        break;
      }
      ++outers;
      // Each inner solve reduces its start by inner_rtol, the last one only as
      // far as the outer target needs.  The margin of 5: (z'r)^(1/2) weighs the
      // stiff cells less than ||r|| does, and the trajectory's error should be
      // no larger than with the ||z|| test and a margin of 2 that this replaces
      // (one word a cell less); 2 left the head of ten 512x512x128 steps 1.02e-8
      // off the tight FP64 solve against 7.4e-9.
      const double need = (rnorm > 0.0) ? 0.2 * a.outer_rtol * bnorm / rnorm : a.inner_rtol;
      const double itol = fmax(a.inner_rtol, need) * zn0;
      double betaold = 1.0;
      T al = T(0), al1 = T(0);  // the last two steps' lengths
      int done = -1;            // the last iteration whose length is known
      for (int i = 0; i < a.max_inner && total < a.max_total; ++i) {
        if (beta == 0.0 || (i > 0 && beta * betaold <= 0.0)) break;
        const T bc = (i == 0) ? T(0) : static_cast<T>(beta / betaold);
        const T* pold = (i & 1) ? a.v.p1 : a.v.p0;
        T* pnew = (i & 1) ? a.v.p0 : a.v.p1;
        double s1[1];
        if (i == 0) s1[0] = pass_a<true, false, false>(a, own, o == 0, bc, al, al1, pold, pnew, gwarp, nwarp);
        else if (i == 1) s1[0] = pass_a<false, true, true>(a, own, false, bc, al, al1, pold, pnew, gwarp, nwarp);
        else if (i & 1) s1[0] = pass_a<false, true, false>(a, own, false, bc, al, al1, pold, pnew, gwarp, nwarp);
        else s1[0] = pass_a<false, false, false>(a, own, false, bc, al, al1, pold, pnew, gwarp, nwarp);
        if (!grid_sum<kLineBlock, WATCH>(s1, a.part, bid, G, epoch, a.st, a.peers)) return;
        const double dpi = s1[0];
        if (!(dpi > 0.0)) {  // inner breakdown: keep d, the FP64 sweep decides
          if (i & 1) done = -2;  // this pass applied every update
          break;
        }
        al1 = al;
        al = static_cast<T>(beta / dpi);
        betaold = beta;
        done = i;
        ++total;
        double sb[1] = {pass_b(a, own, al, gwarp, nwarp)};
        if (!grid_sum<kLineBlock, WATCH>(sb, a.part, bid, G, epoch, a.st, a.peers)) return;
        beta = sb[0];
        if (sqrt(beta) <= itol) break;
      }
      // What the outer sweep still has to add: d as far as an odd iteration's
      // pass A wrote it, then the update of iteration `done` and, where
      // `done` is even, of the one before.
      pd.dset = done >= 1 || done == -2;
      // (Without an update, e1 = 0 multiplies the scaling: p0 and p1 may still
      // hold an earlier solve's infinities.)
      pd.p1 = done < 0 ? a.v.s : (done & 1) ? a.v.p0 : a.v.p1;
      pd.p2 = (done & 1) ? a.v.p1 : a.v.p0;
      pd.e1 = done >= 0 ? al : T(0);
      pd.e2 = (done >= 2 && !(done & 1)) ? al1 : T(0);
    }
    // The corrector reads x0.
    if (cur) {
      const long long stride = static_cast<long long>(G) * blockDim.x;
      for (long long c = bid * static_cast<long long>(blockDim.x) + threadIdx.x; c < a.d.ncell;
           c += stride)
        a.x0[c] = a.x1[c];
    }
    if (bid == 0 && threadIdx.x == 0) {
      a.st->dp = rnorm;
      a.st->rnorm0 = bnorm;
      a.st->its = total;
      a.st->reason = reason;
      a.st->outer = outers;
    }
  }
};

// Columns a warp takes of the domain on G blocks, and the words of them that
// shared memory holds: within kLineOwnBytes, which leaves L1 the rest.
constexpr size_t kLineOwnBytes = 144 * 1024;
template <typename T>
inline int line_words(const Device& D, int variant, int G, int* per) {
  const int cols = line_cols(variant) * (kLineBlock / 32) * G;
  *per = (D.d.nx * D.d.ny + cols - 1) / cols;
  const size_t word = sizeof(Quad<T>) * kLineBlock * static_cast<size_t>(*per);
  return 7 * word <= kLineOwnBytes ? 7 : 3 * word <= kLineOwnBytes ? 3 : 0;
}

}  // namespace fgw
