// The per-column factorization of the line preconditioner's vertical blocks,
// LPC lanes of a warp per column: the pivots d_k of T = L D L^T in FP64, and
// from them the scaling s_k = d_k^(-1/2) and the scaled factor
// l_k = e_k s_k s_{k+1} (e the vertical leg) in the precision T of the inner
// iteration, in the padded column layout of gw_linesolve.cuh.
//
// The pivot recurrence d_k = a_k - e_{k-1}^2 / d_{k-1} is the Moebius map of
// the matrix M_k = [[a_k, -e_{k-1}^2], [1, 0]] acting on (numerator,
// denominator).  A lane composes its E matrices, a Hillis-Steele scan composes
// the lanes', and each lane replays the recurrence itself from its exclusive
// prefix.  Products are rescaled by their largest entry every four cells and
// at every scan step (the map is projective), so nothing overflows.
#pragma once

#include "gw_internal.h"
#include "gw_linesolve.cuh"

namespace fgw {

struct M2 {
  double a, b, c, d;  // [[a, b], [c, d]]
};

__device__ inline M2 m2_scaled(M2 r) {
  const double s = fmax(fmax(fabs(r.a), fabs(r.b)), fmax(fabs(r.c), fabs(r.d)));
  if (s > 0.0 && isfinite(s)) {
    const double is = 1.0 / s;
    r.a *= is;
    r.b *= is;
    r.c *= is;
    r.d *= is;
  }
  return r;
}
__device__ inline M2 m2_mul(const M2& x, const M2& y) {  // x * y
  return M2{x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c,
            x.c * y.b + x.d * y.d};
}

// The columns of blocks bid of G: s and l of every interior column.  DEEP:
// columns in chunks of LPC E cells (LPC = 32), the recurrence and the last
// cell carried from chunk to chunk.
template <typename T, int LPC, int E, bool DEEP>
__device__ __forceinline__ void line_factor_body(const Dims& d, const double* diag, const double* gzp,
                                                 T* __restrict__ s_out, T* __restrict__ l_out,
                                                 const int bid, const int G) {
  constexpr int kCols = 32 / LPC;
  const int lane = threadIdx.x & 31, q = lane % LPC, nz = d.nz, nzp = line_nzp(nz);
  const int ncols = d.nx * d.ny, warps = G * (blockDim.x >> 5);
  for (int base = (bid * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kCols; base < ncols;
       base += warps * kCols) {
    const int c2 = base + lane / LPC;
    const bool act = c2 < ncols;
    const long long col = act ? col2(d, c2 / d.nx + 1, c2 % d.nx + 1) : 0;
    const double* const av = diag + col * nz;
    const double* const ev = gzp + col * nz;
    double n0 = 1.0, m0 = 0.0, slast = 0.0;  // (n, m) and s of the cell before the chunk
    for (int kb = 0; kb < (DEEP ? nz : 1); kb += LPC * E) {
      const int k0 = kb + q * E;
      double a[E], e2[E], el[E];  // diag, e_{k-1}^2, e_k
      const double ep0 = (act && k0 > 0 && k0 < nz) ? ev[k0 - 1] : 0.0;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const bool in = act && k0 + e < nz;
        a[e] = in ? av[k0 + e] : 1.0;
        el[e] = in ? ev[k0 + e] : 0.0;
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const double ep = e == 0 ? ep0 : el[e - 1];
        e2[e] = ep * ep;
      }
      M2 L{1.0, 0.0, 0.0, 1.0};
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (k0 + e < nz) L = m2_mul(M2{a[e], -e2[e], 1.0, 0.0}, L);
        if (e % 4 == 3) L = m2_scaled(L);
      }
#pragma unroll
      for (int off = 1; off < LPC; off <<= 1) {
        const M2 p{__shfl_up_sync(kFull, L.a, off, LPC), __shfl_up_sync(kFull, L.b, off, LPC),
                   __shfl_up_sync(kFull, L.c, off, LPC), __shfl_up_sync(kFull, L.d, off, LPC)};
        if (q >= off) L = m2_scaled(m2_mul(L, p));
      }
      M2 X{__shfl_up_sync(kFull, L.a, 1, LPC), __shfl_up_sync(kFull, L.b, 1, LPC),
           __shfl_up_sync(kFull, L.c, 1, LPC), __shfl_up_sync(kFull, L.d, 1, LPC)};
      if (q == 0) X = M2{1.0, 0.0, 0.0, 1.0};
      double dp = (X.a * n0 + X.b * m0) / (X.c * n0 + X.d * m0);  // d_{k0-1}; unused at k = 0
      double s[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const double dk = (k0 + e == 0) ? a[e] : a[e] - e2[e] / dp;
        // A pivot that is not positive (no SPD block): the diagonal's scaling.
        s[e] = rsqrt((dk > 0.0 && isfinite(dk)) ? dk : a[e]);
        dp = dk;
      }
      const double snext = __shfl_down_sync(kFull, s[0], 1, LPC);
      T so[E], lo[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const bool in = k0 + e < nz;
        so[e] = in ? static_cast<T>(s[e]) : T(0);
        const double sn = e + 1 < E ? s[e + 1 < E ? e + 1 : e] : snext;
        // The last lane's last leg follows with the next chunk's first pivot.
        lo[e] = (k0 + e + 1 < nz && (e + 1 < E || q + 1 < LPC)) ? static_cast<T>(el[e] * s[e] * sn)
                                                                : T(0);
      }
      const int n = act ? max(0, min(E, nzp - k0)) : 0;
      T* const lc = l_out + col * nzp;
      st_cells<E>(s_out + col * nzp + k0, n, so);
      st_cells<E>(lc + k0, n, lo);
      if (DEEP) {
        __syncwarp();
        if (q == 0 && kb > 0 && act) lc[kb - 1] = static_cast<T>(ep0 * slast * s[0]);
        slast = __shfl_sync(kFull, s[E - 1], 31);
        // (n, m) of the chunk's last cell (dp = n / m there).
        n0 = __shfl_sync(kFull, dp, 31);
        m0 = 1.0;
      }
    }
  }
}

// The FP32 factorization of one domain from its step record, by its depth.
__device__ __forceinline__ void line_factor_any(const StepArgs& a, const int bid, const int G) {
  switch (line_variant(a.d.nz)) {
    case 0: line_factor_body<float, 8, 4, false>(a.d, a.diag, a.gzp, a.s32, a.l32, bid, G); break;
    case 1: line_factor_body<float, 16, 4, false>(a.d, a.diag, a.gzp, a.s32, a.l32, bid, G); break;
    case 2: line_factor_body<float, 32, 4, false>(a.d, a.diag, a.gzp, a.s32, a.l32, bid, G); break;
    case 3: line_factor_body<float, 32, 8, false>(a.d, a.diag, a.gzp, a.s32, a.l32, bid, G); break;
    default: line_factor_body<float, 32, 8, true>(a.d, a.diag, a.gzp, a.s32, a.l32, bid, G);
  }
}

}  // namespace fgw
