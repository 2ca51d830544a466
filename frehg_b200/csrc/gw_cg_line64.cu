// The FP64 line form of the predictor solve: the mixed form's algorithm
// (gw_cg_line.cuh) with every inner vector and coefficient in FP64.  It exists
// to measure what FP32 buys the mixed form: the two differ only in the inner
// precision, so their ratio is the precision's share and the ratio of this
// form to the Jacobi FP64 form (PETSc's x0 = 0, point Jacobi) the algorithm's.
//
// Columns of nz <= 256 cells; four cells a lane throughout (eight FP64 cells a
// lane spill), so columns past 128 cells go in two chunks.
#include <algorithm>

#include "gw_cg_line.cuh"

namespace fgw {

namespace {

template <int LPC, bool DEEP, int W>
__global__ void __launch_bounds__(kLineBlock, 1) k_cg_line64(LineArgs<double> a, int per) {
  extern __shared__ __align__(16) char own[];
  LineSolve<double, LPC, 4, DEEP, W>::run(a, blockIdx.x, gridDim.x,
                                          reinterpret_cast<Quad<double>*>(own), per);
}

using Line64Kernel = void (*)(LineArgs<double>, int);
template <int W>
Line64Kernel line64_kernel(int variant) {
  return variant == 0 ? k_cg_line64<8, false, W> : variant == 1 ? k_cg_line64<16, false, W>
                                                                : k_cg_line64<32, false, W>;
}

template <int LPC, bool DEEP>
__global__ void __launch_bounds__(256) k_line_factor64(Dims d, const double* __restrict__ diag,
                                                       const double* __restrict__ gzp, double* s,
                                                       double* l) {
  line_factor_body<double, LPC, 4, DEEP>(d, diag, gzp, s, l, blockIdx.x, gridDim.x);
}

}  // namespace

cudaError_t launch_line_factor64(Device& D) {
  const int variant = line_variant(D.d.nz);
  if (variant == kLineDeep) return cudaErrorInvalidValue;
  const auto k = variant == 0 ? k_line_factor64<8, false> : variant == 1 ? k_line_factor64<16, false>
               : variant == 2 ? k_line_factor64<32, false> : k_line_factor64<32, true>;
  k<<<line_factor_blocks(D), 256, 0, D.stream>>>(D.d, D.diag, D.gzp, D.line64.s, D.line64.l);
  ++D.launches;
  return cudaGetLastError();
}

cudaError_t launch_cg_line64(Device& D, double atol, int maxit, double outer_rtol,
                             int max_outer, bool clear) {
  const int variant = line_variant(D.d.nz);
  if (variant == kLineDeep) return cudaErrorInvalidValue;
  const int G = line_grid(D, variant);
  int per = 0, w = 0;
  Line64Kernel k = k_cg_line64<32, true, 0>;
  if (variant < 3) {
    w = line_words<double>(D, variant, G, &per);
    k = w == 7 ? line64_kernel<7>(variant) : w == 3 ? line64_kernel<3>(variant)
                                                    : line64_kernel<0>(variant);
  }
  const size_t smem = sizeof(Quad<double>) * kLineBlock * static_cast<size_t>(w) * per;
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  if (clear) cudaMemsetAsync(&D.out->cg, 0, sizeof(CgState), D.stream);
  LineArgs<double> a;
  a.d = D.d;
  a.diag = D.diag;
  a.gxp = D.gxp;
  a.gyp = D.gyp;
  a.gzp = D.gzp;
  a.b = D.rhs;
  a.x0 = D.x;
  a.x1 = D.xalt;
  a.v = D.line64;
  a.part = D.cgpart;
  a.st = &D.out->cg;
  a.outer_rtol = outer_rtol;
  a.inner_rtol = 1.0e-4;  // the mixed form's inner reduction
  a.atol = atol;
  a.max_inner = maxit;
  a.max_outer = max_outer;
  a.max_total = maxit;
  a.variant = variant;
  void* args[] = {&a, &per};
  ++D.launches;
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k), dim3(G), dim3(kLineBlock),
                                     args, smem, D.stream);
}

}  // namespace fgw
