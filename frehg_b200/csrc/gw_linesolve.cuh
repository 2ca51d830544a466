// Columns of the line-preconditioned solves (gw_cg_line.cuh): their layout,
// the accesses to it and the column solve, in the precision T of the inner
// iteration (FP32 for the mixed form, FP64 for the FP64 line form).
//
// The inner system is scaled by the square roots of the column factor's
// pivots: with A's column blocks T = L D L^T and S = D^(-1/2),
//   S T S = Lh Lh^T,  Lh unit lower bidiagonal, subdiagonal l = S L S^-1's,
// so one array l holds the factor and the block at once (unit pivots; the
// block's diagonal is 1 + l_{k-1}^2, its legs l_k) and the iteration reads
// three coefficients a cell (l, gx, gy) where the unscaled one read six.
//
// Layout.  Column c of a T array starts at c * nzp, nzp = nz rounded up to 4,
// so every column starts on a 16-byte boundary whatever nz; the padding holds
// zero legs and zero vectors, which every operation keeps.  LPC lanes of a
// warp own a column (32 / LPC columns a warp), lane q of it E consecutive
// cells; columns deeper than 32 E are taken in chunks of 32 E (DEEP).
#pragma once

#include <type_traits>

namespace fgw {

constexpr unsigned kFull = 0xffffffffu;

__host__ __device__ inline int line_nzp(int nz) { return (nz + 3) & ~3; }

// How a column of nz cells is taken: 8, 16 or 32 lanes of four cells (one
// 16-byte FP32 access) up to 128, 32 lanes of eight up to 256, chunks beyond.
constexpr int kLineDeep = 4;
__host__ __device__ inline int line_variant(int nz) {
  return nz <= 32 ? 0 : nz <= 64 ? 1 : nz <= 128 ? 2 : nz <= 256 ? 3 : kLineDeep;
}
// Columns a warp takes at once in a variant.
__host__ __device__ inline int line_cols(int variant) {
  return variant == 0 ? 4 : variant == 1 ? 2 : 1;
}

__device__ inline float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
__device__ inline double fma_t(double a, double b, double c) { return fma(a, b, c); }

// Four consecutive cells at a 16-byte (FP64: 32-byte) boundary.
template <typename T>
struct alignas(4 * sizeof(T) < 16 ? 4 * sizeof(T) : 16) Quad {
  T v[4];
};
__device__ inline Quad<float> ld_quad(const float* p) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  return Quad<float>{{t.x, t.y, t.z, t.w}};
}
__device__ inline Quad<double> ld_quad(const double* p) {
  const double2 a = *reinterpret_cast<const double2*>(p);
  const double2 b = *reinterpret_cast<const double2*>(p + 2);
  return Quad<double>{{a.x, a.y, b.x, b.y}};
}
__device__ inline void st_quad(float* p, const Quad<float>& q) {
  *reinterpret_cast<float4*>(p) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]);
}
__device__ inline void st_quad(double* p, const Quad<double>& q) {
  *reinterpret_cast<double2*>(p) = make_double2(q.v[0], q.v[1]);
  *reinterpret_cast<double2*>(p + 2) = make_double2(q.v[2], q.v[3]);
}

// A lane's E cells from p (its first cell), n of them (a multiple of 4, 0 when
// the lane has none) in the column; the rest 0.
template <int E, typename T>
__device__ inline void ld_cells(const T* p, int n, T (&v)[E]) {
#pragma unroll
  for (int e = 0; e < E; e += 4) {
    Quad<T> q{{T(0), T(0), T(0), T(0)}};
    if (e < n) q = ld_quad(p + e);
#pragma unroll
    for (int u = 0; u < 4; ++u) v[e + u] = q.v[u];
  }
}
template <int E, typename T>
__device__ inline void st_cells(T* p, int n, const T (&v)[E]) {
#pragma unroll
  for (int e = 0; e < E; e += 4)
    if (e < n) st_quad(p + e, Quad<T>{{v[e], v[e + 1], v[e + 2], v[e + 3]}});
}

// Forward sweep y_k = r_k - l_{k-1} y_{k-1} over the column (or chunk): an
// affine map of the predecessor a cell; a lane composes its E maps, a
// Hillis-Steele scan over the column's LPC lanes composes the lanes', and
// each lane replays its cells from its exclusive prefix.  lm is l of the cell
// before the lane's first (0 at the column's first); `carry` the y before
// the chunk.
template <int LPC, int E, typename T>
__device__ inline void line_forward(const T (&l)[E], T lm, const T (&r)[E], T carry, int q,
                                    T (&y)[E]) {
  T A = T(1), B = T(0);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const T a = -(e == 0 ? lm : l[e - 1]);
    B = fma_t(a, B, r[e]);
    A *= a;
  }
#pragma unroll
  for (int off = 1; off < LPC; off <<= 1) {
    const T Ap = __shfl_up_sync(kFull, A, off, LPC);
    const T Bp = __shfl_up_sync(kFull, B, off, LPC);
    if (q >= off) {
      B = fma_t(A, Bp, B);
      A *= Ap;
    }
  }
  const T Ax = __shfl_up_sync(kFull, A, 1, LPC);
  const T Bx = __shfl_up_sync(kFull, B, 1, LPC);
  T v = (q == 0) ? carry : fma_t(Ax, carry, Bx);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    v = fma_t(-(e == 0 ? lm : l[e - 1]), v, r[e]);
    y[e] = v;
  }
}

// Backward sweep z_k = y_k - l_k z_{k+1}; `carry` the z after the chunk.
template <int LPC, int E, typename T>
__device__ inline void line_backward(const T (&l)[E], const T (&y)[E], T carry, int q, T (&z)[E]) {
  T C = T(1), D = T(0);
#pragma unroll
  for (int e = E - 1; e >= 0; --e) {
    D = fma_t(-l[e], D, y[e]);
    C *= -l[e];
  }
#pragma unroll
  for (int off = 1; off < LPC; off <<= 1) {
    const T Cn = __shfl_down_sync(kFull, C, off, LPC);
    const T Dn = __shfl_down_sync(kFull, D, off, LPC);
    if (q + off < LPC) {
      D = fma_t(C, Dn, D);
      C *= Cn;
    }
  }
  const T Cx = __shfl_down_sync(kFull, C, 1, LPC);
  const T Dx = __shfl_down_sync(kFull, D, 1, LPC);
  T v = (q == LPC - 1) ? carry : fma_t(Cx, carry, Dx);
#pragma unroll
  for (int e = E - 1; e >= 0; --e) {
    v = fma_t(-l[e], v, y[e]);
    z[e] = v;
  }
}

}  // namespace fgw
