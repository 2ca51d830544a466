// The predictor's linear solve on the B200: Jacobi-preconditioned conjugate
// gradients on the matrix-free 7-point head system, with the algorithm and
// stopping rule of PETSc's KSPCG as the reference configures it
// (src/core/LinearSystem.cpp:147-151, -gw_pc_type jacobi lane): x0 = 0,
// z = r .* (1 / diag), Hestenes-Stiefel recurrences beta = z'r,
// p = z + (beta / beta_old) p, alpha = beta / p'Ap, convergence on the
// preconditioned norm ||z|| <= max(rtol ||D^-1 b||, atol), divergence at
// 1e5 ||D^-1 b||, non-finite norms, indefinite matrix / preconditioner and
// max_iterations.  (A diagonal entry that is not positive, which no physical
// data gives, ends as a non-finite norm.)
//
// The recurrences run on the system scaled to a unit diagonal: with
// S = D^(-1/2), Jacobi-preconditioned CG on A x = b is plain CG on
// (S A S) y = S b, x = S y, step for step (r' = S r, p' = S^-1 p, and z'r is
// r'.r'), so the diagonal and z drop out of the iteration.
//
// One persistent cooperative launch runs the whole solve.  It scales the legs
// in place, then per iteration:
//   phase A: p_new = r + b p_old (for the seven stencil points), w = A p_new,
//            partial p'w; every second iteration y += the last two a p;
//   grid barrier that sums the partials (grid_sum);
//   phase B: r -= a w, partials r'r and ||S r||^2 = ||D^-1 r||^2 (unscaled);
//   the same barrier; convergence test.
// Every thread takes two consecutive cells (cg64v_body), with 16-byte pair
// loads (ld_far for the neighbours' pairs where nz is odd).
// Per cell and iteration this moves 12.5 FP64 words (100 B): phase A reads r,
// p_old, gxp, gyp, gzp and writes p_new, w, and half the time reads y and the
// p before p_old (in p_new's buffer) and writes y; phase B reads r, w, s and
// writes r.  Unscaled, with x updated every iteration and z stored, it was 16.
// Neighbour reads are served by L1/L2 because the grid-stride sweep keeps all
// resident blocks inside a few j-rows of each other.
//
// Small domains at the usual tolerances run the one-barrier form of the same
// iteration (cg64_one_body).
//
// A thread's cells stay its own for the whole solve, so the words only it
// reads can stay in shared memory (cg64_words: as many of w, y, s and the legs
// as the domain's size leaves room for).  512x512x128 (no room) 692 -> 571 us an
// iteration, 131x113x127 (w) 48.2 -> 35.8, 64x64x128 (four) 12.7 -> 11.0.
//
// The grid barrier's wait is bounded: one that gives up (arrive_and_wait) sets
// CgState::err, and every block leaves at its next barrier, so a launch that
// lost co-residency ends with an error status instead of hanging.
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstring>

#include "gw_coop.cuh"
#include "gw_internal.h"

namespace fgw {

namespace {

using namespace coop;

struct Cg64Args {
  Dims d;
  const double *diag, *b;
  double *gxp, *gyp, *gzp;       // scaled in place
  double *x, *r, *z, *p0, *p1, *w;  // x holds y and z holds s until the end
  double* bw;                       // b's array, free once r is made
  double* part;  // kRedSlots x G (read only behind the write of the same barrier)
  CgState* st;
  double rtol, atol;
  int maxit;
  int variant;  // batched solves: 1 = 16-byte pair accesses (nz even), 0 = separate loads
  Peers peers;  // batched solves: the launch's members
};

// Up to this many pairs one block solves alone, without the grid barrier.
constexpr long long kCgAlone = 2 * kCgBlock;

__device__ inline int sgn(double v) { return (v > 0.0) - (v < 0.0); }

// Two consecutive cells per thread, moved as 16-byte pairs: cell 0 of every
// array is 16-byte aligned, so a thread's own pairs are.  Its i and j
// neighbours' are with ALIGNED (nz even); otherwise see ld_far, and an odd
// cell count leaves a last cell that one thread takes alone (cg64_cell_*).
__device__ inline double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ inline void st2(double* p, double a, double b) {
  *reinterpret_cast<double2*>(p) = make_double2(a, b);
}
// Pairs a whole number of columns away from a thread's own: with nz odd they
// may start on an odd cell and are two loads, without asking (a branch on the
// parity took a 256x256x127 iteration from 160 to 204 us: it parts the loads).
// One aligned load and a shuffle from the lane before would halve the loads,
// but a shuffle holds up the loads behind it: 436 us.  With a thread's own
// pairs as two loads as well it was 247 us.
template <bool ALIGNED>
__device__ inline double2 ld_far(const double* p) {
  if (ALIGNED) return ld2(p);
  return make_double2(p[0], p[1]);
}

// The steps of one cell alone (the order of terms of the pair code), for the
// last cell of an odd count.
__device__ inline void cg64_cell_init(const Cg64Args& a, long long c, double& rr, double& zz) {
  const double s = 1.0 / sqrt(a.diag[c]);
  const double r = s * a.b[c];
  a.x[c] = 0.0;
  a.p0[c] = 0.0;
  a.r[c] = r;
  a.z[c] = s;
  a.gxp[c] *= s / sqrt(a.diag[c + a.d.sx]);
  a.gyp[c] *= s / sqrt(a.diag[c + a.d.sy]);
  a.gzp[c] *= s / sqrt(a.diag[c + 1]);
  rr += r * r;
  zz += (s * r) * (s * r);
}
__device__ inline void cg64_cell_stencil(const Cg64Args& a, long long c, bool first, bool yup,
                                         double bc, double al1, double al2, const double* pold,
                                         double* pnew, double& pw) {
  const long long sx = a.d.sx, sy = a.d.sy;
  const auto pv = [&](long long m) { return first ? a.r[m] : a.r[m] + bc * pold[m]; };
  const double pc = pv(c);
  double wv = a.gyp[c - sy] * pv(c - sy);
  wv += a.gxp[c - sx] * pv(c - sx);
  wv += a.gzp[c - 1] * pv(c - 1);
  wv += pc;
  wv += a.gzp[c] * pv(c + 1);
  wv += a.gxp[c] * pv(c + sx);
  wv += a.gyp[c] * pv(c + sy);
  if (yup) a.x[c] += al1 * pold[c] + al2 * pnew[c];
  pnew[c] = pc;
  a.w[c] = wv;
  pw += pc * wv;
}
__device__ inline void cg64_cell_update(const Cg64Args& a, long long c, double al, double& rr,
                                        double& zz) {
  const double r = a.r[c] - al * a.w[c];
  const double z = a.z[c] * r;
  a.r[c] = r;
  rr += r * r;
  zz += z * z;
}

// After a solve that met a NaN or an overflow: the arrays of the assembly that
// the solve wrote, cleared.  The assembly rewrites the interior's before every
// solve, but never the ghost columns', where a scaled leg (0 / sqrt(NaN)) or
// the one-barrier form's scratch would keep the NaN for every later step.
__device__ inline void cg64_clear(const Cg64Args& a, long long t0, long long stride) {
  for (long long c = t0; c < a.d.ncell; c += stride) {
    a.gxp[c] = 0.0;
    a.gyp[c] = 0.0;
    a.gzp[c] = 0.0;
    a.bw[c] = 0.0;
  }
}

// The words of a thread's own cells held in shared memory, by what keeping
// each saves in traffic: W of them, in this order.
enum OwnWord { kOwnW = 0, kOwnY = 1, kOwnS = 2, kOwnGym = 3, kOwnGxm = 4, kOwnGx = 5, kOwnGy = 6 };

// Phase A over a block's cells.  FIRST: p_new = r, p_old is not read, and the
// legs held on chip are filled.  YUP: y takes the two pending updates.
template <bool ALIGNED, int W, bool FIRST, bool YUP>
__device__ __forceinline__ double cg64_phase_a(const Cg64Args& a, double2* __restrict__ own,
                                               const int words, double bc, double al1, double al2,
                                               const double* pold, double* pnew, long long t0,
                                               long long stride) {
  const long long N2 = a.d.ncell / 2, sx = a.d.sx, sy = a.d.sy;
  // Local copies: a batched solve's record lies in shared memory, and a store
  // through any of its pointers would have every pointer read again.
  const double *const r = a.r, *const gxp = a.gxp, *const gyp = a.gyp, *const gzp = a.gzp;
  double *const x = a.x, *const w = a.w;
  double pw = 0.0;
  int o = threadIdx.x;
  for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
    const long long c = 2 * q;
    const auto chip = [&](int word) -> double2& { return own[word * words + o]; };
    const auto leg = [&](int word, const double* g) {
      if (W > word && !FIRST) return chip(word);
      const double2 v = ld_far<ALIGNED>(g);
      if (W > word) chip(word) = v;
      return v;
    };
    const double2 zero = make_double2(0.0, 0.0);
    const double2 rc = ld2(r + c);
    const double2 pc = FIRST ? zero : ld2(pold + c);
    const double2 rxm = ld_far<ALIGNED>(r + c - sx), rxp = ld_far<ALIGNED>(r + c + sx);
    const double2 rym = ld_far<ALIGNED>(r + c - sy), ryp = ld_far<ALIGNED>(r + c + sy);
    const double2 pxm = FIRST ? zero : ld_far<ALIGNED>(pold + c - sx);
    const double2 pxp = FIRST ? zero : ld_far<ALIGNED>(pold + c + sx);
    const double2 pym = FIRST ? zero : ld_far<ALIGNED>(pold + c - sy);
    const double2 pyp = FIRST ? zero : ld_far<ALIGNED>(pold + c + sy);
    const double rkm = r[c - 1], rkp = r[c + 2];
    const double pkm = FIRST ? 0.0 : pold[c - 1], pkp = FIRST ? 0.0 : pold[c + 2];
    const double2 gx = leg(kOwnGx, gxp + c), gxm = leg(kOwnGxm, gxp + c - sx);
    const double2 gy = leg(kOwnGy, gyp + c), gym = leg(kOwnGym, gyp + c - sy);
    const double2 gz = ld2(gzp + c);
    const double gzm = gzp[c - 1];
    double2 y = zero, pp = zero;
    if (YUP) {
      y = W > kOwnY ? chip(kOwnY) : ld2(x + c);
      pp = ld2(pnew + c);
    }
    const double P0 = rc.x + bc * pc.x, P1 = rc.y + bc * pc.y;
    double w0 = gym.x * (rym.x + bc * pym.x);
    w0 += gxm.x * (rxm.x + bc * pxm.x);
    w0 += gzm * (rkm + bc * pkm);
    w0 += P0;
    w0 += gz.x * P1;
    w0 += gx.x * (rxp.x + bc * pxp.x);
    w0 += gy.x * (ryp.x + bc * pyp.x);
    double w1 = gym.y * (rym.y + bc * pym.y);
    w1 += gxm.y * (rxm.y + bc * pxm.y);
    w1 += gz.x * P0;
    w1 += P1;
    w1 += gz.y * (rkp + bc * pkp);
    w1 += gx.y * (rxp.y + bc * pxp.y);
    w1 += gy.y * (ryp.y + bc * pyp.y);
    st2(pnew + c, P0, P1);
    if (W > kOwnW) chip(kOwnW) = make_double2(w0, w1);
    else st2(w + c, w0, w1);
    if (YUP) {
      y.x += al1 * pc.x + al2 * pp.x;
      y.y += al1 * pc.y + al2 * pp.y;
      if (W > kOwnY) chip(kOwnY) = y;
      else st2(x + c, y.x, y.y);
    }
    pw += P0 * w0;
    pw += P1 * w1;
  }
  return pw;
}

// W words of every own cell in shared memory (own, `words` pairs apart).
// WATCH: in a batched launch.
template <bool ALIGNED, int W, bool WATCH = false>
__device__ __forceinline__ void cg64v_body(const Cg64Args& a, const int bid, const int G,
                                           double2* __restrict__ own, const int words) {
  const long long N2 = a.d.ncell / 2, sx = a.d.sx, sy = a.d.sy;
  // The last cell of an odd count, taken by the grid's last thread.
  const bool tail = !ALIGNED && (a.d.ncell & 1) && bid == G - 1 &&
                    threadIdx.x == blockDim.x - 1;
  const long long ct = a.d.ncell - 1;
  const long long stride = static_cast<long long>(G) * blockDim.x;
  const long long t0 = bid * static_cast<long long>(blockDim.x) + threadIdx.x;
  unsigned epoch = 0;
  double *const gxp = a.gxp, *const gyp = a.gyp, *const gzp = a.gzp, *const ra = a.r,
               *const xa = a.x, *const wa = a.w, *const sa = a.z;
  const double *const diag = a.diag, *const b = a.b;

  // Scale: s, r = S b, the legs in place (only their own cell's thread reads
  // or writes them here); y = 0, p_(-1) = 0.
  double rr = 0.0, zz = 0.0;
  int o = threadIdx.x;
  for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
    const long long c = 2 * q;
    const double2 bv = ld2(b + c), dg = ld2(diag + c);
    const double2 dx = ld_far<ALIGNED>(diag + c + sx), dy = ld_far<ALIGNED>(diag + c + sy);
    const double dz = diag[c + 2];
    const double2 gx = ld2(gxp + c), gy = ld2(gyp + c);
    const double2 gz = ld2(gzp + c);
    const double s0 = 1.0 / sqrt(dg.x), s1 = 1.0 / sqrt(dg.y);
    const double r0 = s0 * bv.x, r1 = s1 * bv.y;
    st2(gxp + c, gx.x * (s0 / sqrt(dx.x)), gx.y * (s1 / sqrt(dx.y)));
    st2(gyp + c, gy.x * (s0 / sqrt(dy.x)), gy.y * (s1 / sqrt(dy.y)));
    st2(gzp + c, gz.x * (s0 * s1), gz.y * (s1 / sqrt(dz)));
    st2(ra + c, r0, r1);
    st2(a.p0 + c, 0.0, 0.0);
    if (W > kOwnS) own[kOwnS * words + o] = make_double2(s0, s1);
    else st2(sa + c, s0, s1);
    if (W > kOwnY) own[kOwnY * words + o] = make_double2(0.0, 0.0);
    else st2(xa + c, 0.0, 0.0);
    const double z0 = s0 * r0, z1 = s1 * r1;
    rr += r0 * r0;
    rr += r1 * r1;
    zz += z0 * z0;
    zz += z1 * z1;
  }
  if (tail) cg64_cell_init(a, ct, rr, zz);
  double s2[2] = {zz, rr};
  if (!grid_sum<kCgBlock, WATCH>(s2, a.part, bid, G, epoch, a.st, a.peers)) return;
  double dp = sqrt(s2[0]);
  double beta = s2[1];
  const double rnorm0 = dp;
  const double ttol = fmax(a.rtol * rnorm0, a.atol);
  int reason = 0, its = 0;
  const auto test = [&](double rn) {
    if (!isfinite(rn)) reason = -9;
    else if (rn <= ttol) reason = (rn < a.atol) ? 3 : 2;
    else if (rn >= 1.0e5 * rnorm0) reason = -4;
  };
  test(dp);
  double betaold = 1.0, dpi = 0.0, dpiold = 0.0;
  double al = 0.0, al1 = 0.0;  // a of the last two iterations
  int i = 0, done = -1;        // done: the last iteration with an update pending
  while (reason == 0) {
    its = i + 1;
    if (beta == 0.0) {
      reason = 3;
      break;
    }
    if (i > 0 && beta * betaold < 0.0) {
      reason = -8;
      break;
    }
    const double bc = (i == 0) ? 0.0 : beta / betaold;
    const double* pold = (i & 1) ? a.p1 : a.p0;
    double* pnew = (i & 1) ? a.p0 : a.p1;
    double pw;
    if (i == 0)
      pw = cg64_phase_a<ALIGNED, W, true, false>(a, own, words, bc, al, al1, pold, pnew, t0, stride);
    else if (i & 1)
      pw = cg64_phase_a<ALIGNED, W, false, true>(a, own, words, bc, al, al1, pold, pnew, t0, stride);
    else
      pw = cg64_phase_a<ALIGNED, W, false, false>(a, own, words, bc, al, al1, pold, pnew, t0, stride);
    if (tail) cg64_cell_stencil(a, ct, i == 0, (i & 1) != 0, bc, al, al1, pold, pnew, pw);
    double s1[1] = {pw};
    if (!grid_sum<kCgBlock, WATCH>(s1, a.part, bid, G, epoch, a.st, a.peers)) return;
    dpiold = dpi;
    dpi = s1[0];
    betaold = beta;
    if (dpi == 0.0 || (i > 0 && sgn(dpi) * sgn(dpiold) < 0)) {
      reason = -10;
      break;
    }
    al1 = al;
    al = beta / dpi;
    done = i;
    rr = 0.0;
    zz = 0.0;
    o = threadIdx.x;
    for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
      const long long c = 2 * q;
      const double2 r = ld2(ra + c);
      const double2 w = W > kOwnW ? own[kOwnW * words + o] : ld2(wa + c);
      const double2 s = W > kOwnS ? own[kOwnS * words + o] : ld2(sa + c);
      const double r0 = r.x - al * w.x, r1 = r.y - al * w.y;
      st2(ra + c, r0, r1);
      const double z0 = s.x * r0, z1 = s.y * r1;
      rr += r0 * r0;
      rr += r1 * r1;
      zz += z0 * z0;
      zz += z1 * z1;
    }
    if (tail) cg64_cell_update(a, ct, al, rr, zz);
    s2[0] = zz;
    s2[1] = rr;
    if (!grid_sum<kCgBlock, WATCH>(s2, a.part, bid, G, epoch, a.st, a.peers)) return;
    dp = sqrt(s2[0]);
    test(dp);
    if (reason != 0) break;
    beta = s2[1];
    ++i;
    if (i >= a.maxit) {
      reason = -3;
      break;
    }
  }
  if (reason == -10 && (its & 1) == 0) done = -1;  // the last phase A applied every update
  // x = S y with the pending updates: iteration `done`'s and, where its own
  // phase A did not apply the one before (even), that one's.
  const double e1 = done < 0 ? 0.0 : al, e2 = (done > 0 && !(done & 1)) ? al1 : 0.0;
  const double* pl = (done & 1) ? a.p0 : a.p1;
  const double* pv = (done & 1) ? a.p1 : a.p0;
  const auto fin = [&](double s, double y, long long c) {
    if (done >= 0) y += e1 * pl[c];
    if (e2 != 0.0) y += e2 * pv[c];
    xa[c] = s * y;
  };
  o = threadIdx.x;
  for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
    const long long c = 2 * q;
    const double2 s = W > kOwnS ? own[kOwnS * words + o] : ld2(sa + c);
    const double2 y = W > kOwnY ? own[kOwnY * words + o] : ld2(xa + c);
    fin(s.x, y.x, c);
    fin(s.y, y.y, c + 1);
  }
  if (tail) fin(sa[ct], xa[ct], ct);
  if (reason == -9) cg64_clear(a, t0, stride);
  if (bid == 0 && threadIdx.x == 0) {
    a.st->dp = dp;
    a.st->rnorm0 = rnorm0;
    a.st->its = its;
    a.st->reason = reason;
    a.st->outer = 1;
  }
}

// ---------------------------------------------------------------- one barrier an iteration
// The same CG with one reduction an iteration (G. Meurant, "Multitasking the
// conjugate gradient method on the CRAY X-MP/48", Parallel Computing 5, 1987;
// its stability in T. Chen and E. Carson, "Predict-and-recompute conjugate
// gradient variants", SIAM J. Sci. Comput. 42, 2020): with w = A p,
//   a = r'r / p'w,  r -= a w,  y += a p,  p = r + b p,  w = A p,
// where b is predicted, ||r - a w||^2 = a^2 w'w - r'r, while a takes the r'r
// that the pass summed.  So one pass and one barrier do what the stencil and
// the update pass do.  A neighbour's new p is taken from its old r, w and p
// (three vectors read where p alone needs two, all three in two buffers), which
// costs a large domain more traffic than the barrier costs it; y must fit in
// shared memory beside its thread.
// r follows A p itself, so the residual stays as true as the two-barrier
// form's.  (The form of Chronopoulos and Gear carries A p by a recurrence, whose
// drift a nearly singular system magnifies: the mean head of a closed saturated
// 40x40x40 box at specific storage 1e-9 moved by 5e-6 m in a step, 7e-8 here and
// with two barriers.  An iteration of 64x64x128 took 9.8 us in it as well, one of
// 48x48x100 7.0 against 7.5, of 97x61x75 12.1 against 11.9.)
enum OneWord { kOneY = 0, kOneS, kOneGym, kOneGxm, kOneGx, kOneGy, kOneWords };

// START: w = A r alone.  FIRST: the old p is the old r.
template <bool ALIGNED, int W, bool START, bool FIRST>
__device__ __forceinline__ void cg64_one_pass(const Cg64Args& a, double2* own, const int words,
                                              double al, double be, const double* ro,
                                              const double* wo, const double* po, double* rn,
                                              double* wn, double* pn, long long t0,
                                              long long stride, double& rr, double& zz, double& pw,
                                              double& ww) {
  const long long N2 = a.d.ncell / 2, sx = a.d.sx, sy = a.d.sy;
  int o = threadIdx.x;
  for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
    const long long c = 2 * q;
    const auto chip = [&](int word) -> double2& { return own[word * words + o]; };
    const auto leg = [&](int word, const double* g) {
      if (W > word && !START) return chip(word);
      const double2 v = ld_far<ALIGNED>(g);
      if (W > word) chip(word) = v;
      return v;
    };
    // (r - al w) + be p of a pair (START: r)
    const auto next2 = [&](long long m) {
      double2 r = ld_far<ALIGNED>(ro + m);
      if (START) return r;
      const double2 w = ld_far<ALIGNED>(wo + m), p = FIRST ? r : ld_far<ALIGNED>(po + m);
      r.x = (r.x - al * w.x) + be * p.x;
      r.y = (r.y - al * w.y) + be * p.y;
      return r;
    };
    const auto next1 = [&](long long m) {
      return START ? ro[m] : (ro[m] - al * wo[m]) + be * (FIRST ? ro[m] : po[m]);
    };
    const double2 pym = next2(c - sy), pxm = next2(c - sx);
    const double2 pxp = next2(c + sx), pyp = next2(c + sy);
    const double pkm = next1(c - 1), pkp = next1(c + 2);
    const double2 gx = leg(kOneGx, a.gxp + c), gxm = leg(kOneGxm, a.gxp + c - sx);
    const double2 gy = leg(kOneGy, a.gyp + c), gym = leg(kOneGym, a.gyp + c - sy);
    const double2 gz = ld2(a.gzp + c);
    const double gzm = a.gzp[c - 1];
    double2 p = ld2(ro + c);
    if (!START) {
      const double2 w = ld2(wo + c), pp = FIRST ? p : ld2(po + c);
      const double2 r = make_double2(p.x - al * w.x, p.y - al * w.y);
      double2 y = FIRST ? make_double2(0.0, 0.0) : chip(kOneY);
      y.x += al * pp.x;
      y.y += al * pp.y;
      chip(kOneY) = y;
      p.x = r.x + be * pp.x;
      p.y = r.y + be * pp.y;
      st2(rn + c, r.x, r.y);
      st2(pn + c, p.x, p.y);
      const double2 S = W > kOneS ? chip(kOneS) : ld2(a.z + c);
      const double z0 = S.x * r.x, z1 = S.y * r.y;
      rr += r.x * r.x;
      rr += r.y * r.y;
      zz += z0 * z0;
      zz += z1 * z1;
    }
    double w0 = gym.x * pym.x;
    w0 += gxm.x * pxm.x;
    w0 += gzm * pkm;
    w0 += p.x;
    w0 += gz.x * p.y;
    w0 += gx.x * pxp.x;
    w0 += gy.x * pyp.x;
    double w1 = gym.y * pym.y;
    w1 += gxm.y * pxm.y;
    w1 += gz.x * p.x;
    w1 += p.y;
    w1 += gz.y * pkp;
    w1 += gx.y * pxp.y;
    w1 += gy.y * pyp.y;
    st2(wn + c, w0, w1);
    pw += p.x * w0;
    pw += p.y * w1;
    ww += w0 * w0;
    ww += w1 * w1;
  }
}

template <bool ALIGNED, int W>
__device__ __forceinline__ void cg64_one_body(const Cg64Args& a, const int bid, const int G,
                                              double2* own, const int words) {
  static_assert(W >= 1, "y stays with its thread");
  const long long N2 = a.d.ncell / 2, sx = a.d.sx, sy = a.d.sy, ct = a.d.ncell - 1;
  // The last cell of an odd count, taken by the grid's last thread, with its
  // own y and s in registers.
  const bool tail = !ALIGNED && (a.d.ncell & 1) && bid == G - 1 && threadIdx.x == blockDim.x - 1;
  const long long stride = static_cast<long long>(G) * blockDim.x;
  const long long t0 = bid * static_cast<long long>(blockDim.x) + threadIdx.x;
  double* const rb[2] = {a.r, a.p0};
  double* const wb[2] = {a.w, a.p1};
  double* const pb[2] = {a.bw, a.x};
  unsigned epoch = 0;

  double rr = 0.0, zz = 0.0, pw = 0.0, ww = 0.0, ty = 0.0, ts = 0.0;
  int o = threadIdx.x;
  for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
    const long long c = 2 * q;
    const double2 bv = ld2(a.b + c), dg = ld2(a.diag + c);
    const double2 dx = ld_far<ALIGNED>(a.diag + c + sx), dy = ld_far<ALIGNED>(a.diag + c + sy);
    const double dz = a.diag[c + 2];
    const double2 gx = ld2(a.gxp + c), gy = ld2(a.gyp + c);
    const double2 gz = ld2(a.gzp + c);
    const double s0 = 1.0 / sqrt(dg.x), s1 = 1.0 / sqrt(dg.y);
    const double r0 = s0 * bv.x, r1 = s1 * bv.y;
    st2(a.gxp + c, gx.x * (s0 / sqrt(dx.x)), gx.y * (s1 / sqrt(dx.y)));
    st2(a.gyp + c, gy.x * (s0 / sqrt(dy.x)), gy.y * (s1 / sqrt(dy.y)));
    st2(a.gzp + c, gz.x * (s0 * s1), gz.y * (s1 / sqrt(dz)));
    st2(a.r + c, r0, r1);
    if (W > kOneS) own[kOneS * words + o] = make_double2(s0, s1);
    else st2(a.z + c, s0, s1);
    const double z0 = s0 * r0, z1 = s1 * r1;
    rr += r0 * r0;
    rr += r1 * r1;
    zz += z0 * z0;
    zz += z1 * z1;
    own[kOneY * words + o] = make_double2(0.0, 0.0);
  }
  if (tail) {
    ts = 1.0 / sqrt(a.diag[ct]);
    const double r = ts * a.b[ct];
    a.r[ct] = r;
    a.gxp[ct] *= ts / sqrt(a.diag[ct + sx]);
    a.gyp[ct] *= ts / sqrt(a.diag[ct + sy]);
    a.gzp[ct] *= ts / sqrt(a.diag[ct + 1]);
    rr += r * r;
    zz += (ts * r) * (ts * r);
  }
  double v2[2] = {zz, rr};
  if (!grid_sum<kCgBlock, false>(v2, a.part, bid, G, epoch, a.st, a.peers)) return;
  double dp = sqrt(v2[0]), gamma = v2[1];
  const double rnorm0 = dp;
  const double ttol = fmax(a.rtol * rnorm0, a.atol);
  int reason = 0, its = 0;
  const auto test = [&](double rn) {
    if (!isfinite(rn)) reason = -9;
    else if (rn <= ttol) reason = (rn < a.atol) ? 3 : 2;
    else if (rn >= 1.0e5 * rnorm0) reason = -4;
  };
  test(dp);
  // The tail cell's share of a pass, on the buffers the pairs use.
  const auto tail_cell = [&](bool start, bool first, double al, double be, const double* ro,
                             const double* wo, const double* po, double* rn, double* wn,
                             double* pn) {
    const auto nx = [&](long long m) {
      return start ? ro[m] : (ro[m] - al * wo[m]) + be * (first ? ro[m] : po[m]);
    };
    double p = ro[ct];
    if (!start) {
      const double pp = first ? p : po[ct], r = p - al * wo[ct];
      ty += al * pp;
      p = r + be * pp;
      rn[ct] = r;
      pn[ct] = p;
      rr += r * r;
      zz += (ts * r) * (ts * r);
    }
    double wv = a.gyp[ct - sy] * nx(ct - sy);
    wv += a.gxp[ct - sx] * nx(ct - sx);
    wv += a.gzp[ct - 1] * nx(ct - 1);
    wv += p;
    wv += a.gzp[ct] * nx(ct + 1);
    wv += a.gxp[ct] * nx(ct + sx);
    wv += a.gyp[ct] * nx(ct + sy);
    wn[ct] = wv;
    pw += p * wv;
    ww += wv * wv;
  };
  if (reason == 0) {  // p = r, w = A p
    cg64_one_pass<ALIGNED, W, true, false>(a, own, words, 0.0, 0.0, rb[0], nullptr, nullptr,
                                           nullptr, wb[0], nullptr, t0, stride, rr, zz, pw, ww);
    if (tail) tail_cell(true, false, 0.0, 0.0, rb[0], nullptr, nullptr, nullptr, wb[0], nullptr);
    double v1[2] = {pw, ww};
    if (!grid_sum<kCgBlock, false>(v1, a.part, bid, G, epoch, a.st, a.peers)) return;
    pw = v1[0];
    ww = v1[1];
  }
  double dpi = 0.0, dpiold = 0.0;
  int i = 0;
  while (reason == 0) {
    its = i + 1;
    if (gamma == 0.0) {
      reason = 3;
      break;
    }
    dpiold = dpi;
    dpi = pw;
    if (dpi == 0.0 || (i > 0 && sgn(dpi) * sgn(dpiold) < 0)) {
      reason = -10;
      break;
    }
    const double al = gamma / dpi;
    const double be = fmax(al * al * ww - gamma, 0.0) / gamma;
    const int f = i & 1;
    rr = zz = pw = ww = 0.0;
    if (i == 0)
      cg64_one_pass<ALIGNED, W, false, true>(a, own, words, al, be, rb[f], wb[f], pb[f], rb[1 - f],
                                             wb[1 - f], pb[1 - f], t0, stride, rr, zz, pw, ww);
    else
      cg64_one_pass<ALIGNED, W, false, false>(a, own, words, al, be, rb[f], wb[f], pb[f],
                                              rb[1 - f], wb[1 - f], pb[1 - f], t0, stride, rr, zz,
                                              pw, ww);
    if (tail)
      tail_cell(false, i == 0, al, be, rb[f], wb[f], pb[f], rb[1 - f], wb[1 - f], pb[1 - f]);
    double v4[4] = {zz, rr, pw, ww};
    if (!grid_sum<kCgBlock, false>(v4, a.part, bid, G, epoch, a.st, a.peers)) return;
    dp = sqrt(v4[0]);
    test(dp);
    if (reason != 0) break;
    gamma = v4[1];
    pw = v4[2];
    ww = v4[3];
    ++i;
    if (i >= a.maxit) {
      reason = -3;
      break;
    }
  }
  o = threadIdx.x;
  for (long long q = t0; q < N2; q += stride, o += kCgBlock) {
    const long long c = 2 * q;
    const double2 s = W > kOneS ? own[kOneS * words + o] : ld2(a.z + c);
    const double2 y = own[kOneY * words + o];
    st2(a.x + c, s.x * y.x, s.y * y.y);
  }
  if (tail) a.x[ct] = ts * ty;
  if (reason == -9) cg64_clear(a, t0, stride);
  if (bid == 0 && threadIdx.x == 0) {
    a.st->dp = dp;
    a.st->rnorm0 = rnorm0;
    a.st->its = its;
    a.st->reason = reason;
    a.st->outer = 1;
  }
}

// 128 registers a thread: at an 80-register cap (768 threads per SM) the
// kernel spilled and the 512x512x128 FP64 solve took 251 ms against 236.
template <bool ALIGNED, int W>
__global__ void __launch_bounds__(kCgBlock, 1) k_cg64(Cg64Args a, int words) {
  extern __shared__ double2 own[];
  cg64v_body<ALIGNED, W>(a, blockIdx.x, gridDim.x, own, words);
}

template <bool ALIGNED, int W>
__global__ void __launch_bounds__(kCgBlock, 1) k_cg64_one(Cg64Args a, int words) {
  extern __shared__ double2 own[];
  cg64_one_body<ALIGNED, W>(a, blockIdx.x, gridDim.x, own, words);
}

// One cooperative launch over several domains: instance i owns
// first[i+1] - first[i] block slots and runs its own solve on them, in the
// paired or the separate-load two-cell form by its `variant`; each block takes the next
// slot from `queue` (zeroed before the launch) until all are handed out, the
// instances' slots in queue order (`order`, slot offsets `ofirst`), so a
// block whose instance has converged goes on to a waiting instance.  The
// slot's index within its instance, not the block, fixes the block's share
// of the instance's cells.
__global__ void __launch_bounds__(kCgBlock, 1)
    k_cg64_batch(const Cg64Args* __restrict__ tab, const int* __restrict__ first, int n,
                 int* queue, const int* __restrict__ order, const int* __restrict__ ofirst) {
  __shared__ Cg64Args sa;
  __shared__ int sb, sg, slot;
  for (;;) {
    if (threadIdx.x == 0) {
      slot = atomicAdd(queue, 1);
      if (slot < first[n]) {
        const int q = instance_of(ofirst, n, slot);
        const int i = order[q];
        sa = tab[i];
        sb = slot - ofirst[q];
        sg = first[i + 1] - first[i];
      }
    }
    __syncthreads();
    if (slot >= first[n]) break;
    if (sa.variant) {
      cg64v_body<true, 0, true>(sa, sb, sg, nullptr, 0);
    } else {
      cg64v_body<false, 0, true>(sa, sb, sg, nullptr, 0);
    }
    __syncthreads();  // every thread is done with sa before the next slot's
  }
}

}  // namespace

// One block per SM; as few as hold a pair of cells a thread, and one alone
// (no grid barrier) up to kCgAlone pairs.
int cg64_grid(int sm_count, long long ncell) {
  const long long pairs = ncell / 2;
  if (pairs <= kCgAlone) return 1;
  return static_cast<int>(std::min<long long>((pairs + kCgBlock - 1) / kCgBlock, sm_count));
}

namespace {

Cg64Args make_cg64_args(const Device& D, double rtol, double atol, int maxit) {
  Cg64Args a;
  a.d = D.d;
  a.diag = D.diag;
  a.gxp = D.gxp;
  a.gyp = D.gyp;
  a.gzp = D.gzp;
  a.b = D.rhs;
  a.bw = D.rhs;
  a.x = D.x;
  a.r = D.r;
  a.z = D.z;
  a.p0 = D.p0;
  a.p1 = D.p1;
  a.w = D.w;
  a.part = D.cgpart;
  a.st = &D.out->cg;
  a.rtol = rtol;
  a.atol = atol;
  a.maxit = maxit;
  return a;
}

}  // namespace

namespace {

// Shared-memory words of the own cells at `pairs` pairs a thread: the largest
// built variant within kOwnBytes.  Half the SM's 256 KB stays L1, which serves
// the stencil's neighbours: with 208 KB taken the 131x113x127 iteration was
// 54.8 us against 37.0 with 104 KB and 40.5 with none (64x64x128: 224 KB 11.5,
// 128 KB 10.9, none 11.4; 101x55x25, 56 KB: 5 % of a coupled pass).
constexpr size_t kOwnBytes = 128 * 1024;
int cg64_words(long long pairs) {
  const long long fit = kOwnBytes / (pairs * kCgBlock * sizeof(double2));
  return fit >= 7 ? 7 : fit >= 4 ? 4 : fit >= 2 ? 2 : fit >= 1 ? 1 : 0;
}

// Solves at least this loose, of at most this many pairs a thread on more than
// one block, take one barrier an iteration (us an iteration, two barriers
// against one: 32x32x50 7.2 / 5.7, 101x55x25 7.7 / 6.1, 48x48x100 8.7 / 7.5,
// 64x64x128 11.0 / 9.8, 97x61x75 12.6 / 11.9, 80x83x103 with five pairs 14.6 /
// 14.1).  Beyond, the third vector's traffic outweighs the barrier (81x80x127
// with six 18.4 / 18.8, 90x90x128 with eight 15.6 / 17.2).  Tighter solves keep
// two: the predicted b has an error of eps r'r / (the next r'r).
constexpr double kOneBarrierRtol = 1.0e-10;
constexpr long long kOneBarrierPairs = 5;

using Cg64Kernel = void (*)(Cg64Args, int);
template <bool ALIGNED>
Cg64Kernel cg64_one_kernel(int w) {
  return w == 7 ? k_cg64_one<ALIGNED, 7> : w == 4 ? k_cg64_one<ALIGNED, 4>
                                                  : k_cg64_one<ALIGNED, 2>;
}
template <bool ALIGNED>
Cg64Kernel cg64_kernel(int w) {
  return w == 7 ? k_cg64<ALIGNED, 7> : w == 4 ? k_cg64<ALIGNED, 4> : w == 2 ? k_cg64<ALIGNED, 2>
       : w == 1 ? k_cg64<ALIGNED, 1> : k_cg64<ALIGNED, 0>;
}

}  // namespace

cudaError_t launch_cg64(Device& D, double rtol, double atol, int maxit, bool clear) {
  if (clear) cudaMemsetAsync(&D.out->cg, 0, sizeof(CgState), D.stream);
  Cg64Args a = make_cg64_args(D, rtol, atol, maxit);
  const long long threads = static_cast<long long>(D.cg_grid) * kCgBlock;
  const long long pairs = std::max<long long>(1, (D.d.ncell / 2 + threads - 1) / threads);
  const int w = cg64_words(pairs);
  int words = static_cast<int>(pairs * kCgBlock);
  const bool even = D.d.nz % 2 == 0, one = w >= 2 && pairs <= kOneBarrierPairs &&
                                         D.cg_grid > 1 && rtol >= kOneBarrierRtol;
  const size_t smem = (one ? std::min<int>(w, kOneWords) : w) * words * sizeof(double2);
  const Cg64Kernel k = one ? (even ? cg64_one_kernel<true>(w) : cg64_one_kernel<false>(w))
                           : (even ? cg64_kernel<true>(w) : cg64_kernel<false>(w));
  const void* kern = reinterpret_cast<const void*>(k);
  const cudaError_t e = raise_smem_limit(kern, smem);
  if (e != cudaSuccess) return e;
  void* args[] = {&a, &words};
  ++D.launches;
  return cudaLaunchCooperativeKernel(kern, dim3(D.cg_grid), dim3(kCgBlock), args, smem, D.stream);
}

size_t cg64_args_bytes() { return sizeof(Cg64Args); }

void cg64_fill_args(const Device& D, const SolveParams& p, int variant, const Peers& peers,
                    void* dst) {
  Cg64Args a = make_cg64_args(D, p.rtol, p.atol, p.maxit);
  a.variant = variant;
  a.peers = peers;
  std::memcpy(dst, &a, sizeof(a));
}

const void* cg64_batch_kernel() { return reinterpret_cast<const void*>(k_cg64_batch); }

}  // namespace fgw
