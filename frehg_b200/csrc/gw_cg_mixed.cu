// Mixed-precision predictor solve: FP32 inner line-preconditioned CG inside
// FP64 defect correction on the true residual (gw_cg_line.cuh), its column
// factorization (gw_linefactor.cuh), and both batched over many domains.
#include <algorithm>
#include <cstring>

#include "gw_cg_line.cuh"

namespace fgw {

namespace {

constexpr int kFactorBlock = 256;

template <int LPC, int E, bool DEEP>
__global__ void __launch_bounds__(kFactorBlock) k_line_factor(Dims d,
                                                              const double* __restrict__ diag,
                                                              const double* __restrict__ gzp,
                                                              float* s, float* l) {
  line_factor_body<float, LPC, E, DEEP>(d, diag, gzp, s, l, blockIdx.x, gridDim.x);
}

using FactorKernel = void (*)(Dims, const double*, const double*, float*, float*);
FactorKernel factor_kernel(int variant) {
  static const FactorKernel table[] = {k_line_factor<8, 4, false>, k_line_factor<16, 4, false>,
                                       k_line_factor<32, 4, false>, k_line_factor<32, 8, false>,
                                       k_line_factor<32, 8, true>};
  return table[variant];
}

template <int LPC, int E, bool DEEP, int W>
__global__ void __launch_bounds__(kLineBlock, 1) k_cg_mixed(LineArgs<float> a, int per) {
  extern __shared__ __align__(16) char own[];
  LineSolve<float, LPC, E, DEEP, W>::run(a, blockIdx.x, gridDim.x,
                                         reinterpret_cast<Quad<float>*>(own), per);
}

using MixedKernel = void (*)(LineArgs<float>, int);
template <int W>
MixedKernel mixed_kernel(int variant) {
  return variant == 0 ? k_cg_mixed<8, 4, false, W> : variant == 1 ? k_cg_mixed<16, 4, false, W>
                                                                  : k_cg_mixed<32, 4, false, W>;
}

// One cooperative launch over several domains of every column variant:
// instance i owns first[i+1] - first[i] block slots and runs its own solve in
// its `variant`; the blocks take the slots from `queue` in queue order (as
// k_cg64_batch).  One launch for all variants, so they share the device
// instead of following one another.
__global__ void __launch_bounds__(kLineBlock, 1)
    k_cg_mixed_batch(const LineArgs<float>* __restrict__ tab, const int* __restrict__ first, int n,
                     int* queue, const int* __restrict__ order, const int* __restrict__ ofirst) {
  __shared__ LineArgs<float> sa;
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
    switch (sa.variant) {
      case 0: LineSolve<float, 8, 4, false, 0, true>::run(sa, sb, sg); break;
      case 1: LineSolve<float, 16, 4, false, 0, true>::run(sa, sb, sg); break;
      case 2: LineSolve<float, 32, 4, false, 0, true>::run(sa, sb, sg); break;
      case 3: LineSolve<float, 32, 8, false, 0, true>::run(sa, sb, sg); break;
      default: LineSolve<float, 32, 8, true, 0, true>::run(sa, sb, sg); break;
    }
    __syncthreads();  // every thread is done with sa before the next slot's
  }
}

LineArgs<float> make_mixed_args(const Device& D, double atol, int maxit, double outer_rtol,
                                int max_outer) {
  LineArgs<float> a;
  a.d = D.d;
  a.diag = D.diag;
  a.gxp = D.gxp;
  a.gyp = D.gyp;
  a.gzp = D.gzp;
  a.b = D.rhs;
  a.x0 = D.x;
  a.x1 = D.xalt;
  a.v = D.line32;
  a.part = D.cgpart;
  a.st = &D.out->cg;
  a.outer_rtol = outer_rtol;
  // Reduction asked of every inner solve but the last: 1e-4 minimised the
  // total inner iterations of the two corrections on slab crops (96^2 and
  // 128^2 x 128 systems: 22, 24, 18 against 24, 26, 20 at 1e-5).
  a.inner_rtol = 1.0e-4;
  a.atol = atol;
  a.max_inner = maxit;
  a.max_outer = max_outer;
  a.max_total = maxit;
  a.variant = line_variant(D.d.nz);
  return a;
}

}  // namespace

// Deepest columns the mixed form takes.
constexpr int kMixedMaxNz = 4096;

int line_block() { return kLineBlock; }

// Blocks of a line solve: a warp a column (or a few shallow ones) and eight
// warps a block before the next, at most one block per SM.
int line_grid(const Device& D, int variant) {
  const long long warps = (static_cast<long long>(D.d.nx) * D.d.ny + line_cols(variant) - 1) /
                          line_cols(variant);
  if (warps <= kLineBlock / 32) return 1;
  return static_cast<int>(std::min<long long>((warps + 7) / 8, D.sm_count));
}

cudaError_t launch_line_factor(Device& D) {
  factor_kernel(line_variant(D.d.nz))<<<line_factor_blocks(D), kFactorBlock, 0, D.stream>>>(
      D.d, D.diag, D.gzp, D.line32.s, D.line32.l);
  ++D.launches;
  return cudaGetLastError();
}

cudaError_t launch_cg_mixed(Device& D, double rtol, double atol, int maxit, double outer_rtol,
                            int max_outer, bool clear) {
  (void)rtol;
  if (D.d.nz > kMixedMaxNz) return cudaErrorInvalidValue;
  const int variant = line_variant(D.d.nz), G = line_grid(D, variant);
  int per = 0, w = 0;
  MixedKernel k = k_cg_mixed<32, 8, true, 0>;
  if (variant == 3) {
    k = k_cg_mixed<32, 8, false, 0>;
  } else if (variant < 3) {
    w = line_words<float>(D, variant, G, &per);
    k = w == 7 ? mixed_kernel<7>(variant) : w == 3 ? mixed_kernel<3>(variant)
                                                   : mixed_kernel<0>(variant);
  }
  const size_t smem = sizeof(Quad<float>) * kLineBlock * static_cast<size_t>(w) * per;
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void*>(k), smem);
  if (e != cudaSuccess) return e;
  if (clear) cudaMemsetAsync(&D.out->cg, 0, sizeof(CgState), D.stream);
  LineArgs<float> a = make_mixed_args(D, atol, maxit, outer_rtol, max_outer);
  void* args[] = {&a, &per};
  ++D.launches;
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k), dim3(G), dim3(kLineBlock),
                                     args, smem, D.stream);
}

// ---------------------------------------------------------------- batched solves
int mixed_variant(const Device& D, bool tiled) { return tiled ? kLineDeep : line_variant(D.d.nz); }

size_t mixed_args_bytes() { return sizeof(LineArgs<float>); }

void mixed_fill_args(const Device& D, const SolveParams& p, int variant, const Peers& peers,
                     void* dst) {
  LineArgs<float> a = make_mixed_args(D, p.atol, p.maxit, p.outer_rtol, p.max_outer);
  a.variant = variant;
  a.peers = peers;
  std::memcpy(dst, &a, sizeof(a));
}

const void* mixed_batch_kernel() { return reinterpret_cast<const void*>(k_cg_mixed_batch); }

// ---------------------------------------------------------------- batched line factor
namespace {

__global__ void __launch_bounds__(kFactorBlock) k_line_factor_batch(const StepArgs* tab,
                                                                    const int* first, int n) {
  __shared__ StepArgs sa;
  __shared__ int si;
  if (threadIdx.x == 0) si = instance_of(first, n, blockIdx.x);
  __syncthreads();
  const unsigned long long* src = reinterpret_cast<const unsigned long long*>(tab + si);
  unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sa);
  for (int w = threadIdx.x; w < static_cast<int>(sizeof(StepArgs) / 8); w += blockDim.x)
    dst[w] = src[w];
  const int bid = blockIdx.x - first[si], G = first[si + 1] - first[si];
  __syncthreads();
  line_factor_any(sa, bid, G);
}

}  // namespace

int line_factor_blocks(const Device& D) {
  const int cols = line_cols(line_variant(D.d.nz)) * (kFactorBlock / 32);
  const long long n = static_cast<long long>(D.d.nx) * D.d.ny;
  return static_cast<int>(std::min<long long>((n + cols - 1) / cols, 16LL * D.sm_count));
}

cudaError_t launch_line_factor_batch(const PhaseTables& t, cudaStream_t s) {
  k_line_factor_batch<<<t.grid_factor, kFactorBlock, 0, s>>>(t.tab, t.first_factor, t.n);
  return cudaGetLastError();
}

}  // namespace fgw
