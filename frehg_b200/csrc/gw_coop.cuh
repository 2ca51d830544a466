// Device helpers shared by the cooperative solver kernels: the bounded grid
// barrier with its fixed-order (deterministic) grid sums.
#pragma once

#include "gw_internal.h"

namespace fgw {
namespace coop {

// Threads of a solve block, one block per SM (128 registers a thread): half
// the blocks of two 256-thread ones at a barrier for the same threads.  A
// 64x64x128 mixed iteration takes 11.6 us against 14.0, FP64 12.7 against 13.1.
constexpr int kCgBlock = 512;

// Polls after which a barrier's wait gives up: 14 s at 0.32 us a poll.  In a
// batched launch a domain's first blocks may wait for the rest of another
// domain's whole solve, however long that is, before theirs are handed out:
// their limit starts over while any domain of the launch arrives at a barrier.
constexpr long long kSpinLimit = 45000000LL;

// Reduction slots of a solve on G blocks: two generations of kRedVals values,
// one double per block each, at the head of a solve's `part` array.
constexpr int kRedVals = 4;
constexpr int kRedSlots = 2 * kRedVals;
static_assert(kRedSlots == kSolveSlots, "the solves' slot allocation");

__device__ inline int ld_relaxed_int(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline void red_add(unsigned* p, unsigned v) {
  asm volatile("red.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ inline double ld_relaxed_f64(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline void st_relaxed_f64(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ inline void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

__device__ inline double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Thread 0's part of a grid barrier: counts the block in on `arrived` and polls
// it up to `want` (which may wrap: the two differ by less than 2^31), with the
// block's writes released before and the others' acquired after.  Gives up
// past kSpinLimit polls, or when another block has, by setting *err.  With
// WATCH the limit starts over when one of the launch's domains, peers, has
// arrived somewhere since the last limit (the code of it cost a solve of one
// domain registers: 131x113x127 35.5 -> 37.2 us an iteration).
template <bool WATCH>
__device__ inline int arrive_and_wait(unsigned* arrived, unsigned want, int* err,
                                      const Peers& peers) {
  fence_gpu();
  red_add(arrived, 1u);
  int ok = 1;
  long long spins = 0;
  unsigned seen = 0u;
  while (static_cast<int>(ld_relaxed_u32(arrived) - want) < 0) {
    ++spins;
    if (WATCH && spins > kSpinLimit) {
      unsigned now = 0u;
      for (int i = 0; i < peers.n; ++i) now += ld_relaxed_u32(&peers.states[i]->arrived);
      if (now != seen) spins = 0;
      seen = now;
    }
    if (spins > kSpinLimit || ((spins & 1023) == 0 && ld_relaxed_int(err) != 0)) {
      atomicExch(err, 1);
      ok = 0;
      break;
    }
  }
  fence_gpu();
  return ok;
}

// Grid barrier without a sum.  False when it gave up; the block then leaves.
__device__ inline bool grid_barrier(unsigned* arrived, unsigned want, int* err) {
  __shared__ int good;
  __syncthreads();
  if (threadIdx.x == 0) good = arrive_and_wait<false>(arrived, want, err, Peers{});
  __syncthreads();
  return good != 0;
}

// Sum of a block's N warp sums, pairwise (a chain of 16 additions is 0.15 us).
template <int N>
__device__ inline double tree_sum(const double* w) {
  double t[N];
#pragma unroll
  for (int q = 0; q < N; ++q) t[q] = w[q];
#pragma unroll
  for (int m = 1; m < N; m <<= 1) {
#pragma unroll
    for (int q = 0; q + m < N; q += 2 * m) t[q] += t[q + m];
  }
  return t[0];
}

// Grid barrier and sum in one exchange, for a cooperative (co-resident)
// launch of BLOCK threads a block: v[n] <- the sum of every thread's v[n]
// over the G blocks, the same bits in every thread (fixed order: lanes, warps,
// then blocks by stripes of the block's threads).  Writes made before the call
// by any thread of the G blocks are visible after it.
//
// Thread 0 publishes the block's sums, counts the block in on CgState::arrived
// (it only grows: generation e is complete at e G) and polls that one word;
// then the block reads the G sums.  Two generations of slots suffice: a block
// writes generation e + 2 only after all have arrived at e + 1, so have read e.
// Measured per iteration (two barriers) against a barrier with two block sums,
// a counter, a generation word polled with __nanosleep and two rounds of
// partials: 64x64x128 FP64 16.6 -> 12.7 us, mixed 17.8 -> 11.6 us.  Polling the
// sums themselves as their own flags saves a round trip, but every block then
// polls G words: 22.5 us for the FP64 iteration (at 296 blocks).
//
// WATCH: a batched launch, whose domains are `peers`.
// The wait is bounded (arrive_and_wait): when it gives up thread 0 sets
// CgState::err and every block returns false here or at its next call, and
// leaves the kernel.
template <int BLOCK, bool WATCH, int NV>
__device__ __forceinline__ bool grid_sum(double (&v)[NV], double* slots, const int bid,
                                         const int G, unsigned& epoch, CgState* st,
                                         const Peers& peers) {
  static_assert(NV <= kRedVals, "slots");
  constexpr int kWarps = BLOCK / 32;
  __shared__ double sh[NV][kWarps];
  __shared__ double sw[NV][kWarps];
  __shared__ int good;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    v[n] = warp_sum(v[n]);
    if (lane == 0) sh[n][wid] = v[n];
  }
  __syncthreads();
  if (G > 1) {
    double* const gen = slots + static_cast<long long>(epoch & 1u) * kRedVals * G;
    ++epoch;
    if (wid == 0) {
      if (lane < NV) {
        const double s = tree_sum<kWarps>(sh[lane]);
        st_relaxed_f64(gen + static_cast<long long>(lane) * G + bid, s);
      }
      __syncwarp();
      if (lane == 0) {
        good = arrive_and_wait<WATCH>(&st->arrived, epoch * static_cast<unsigned>(G), &st->err,
                                      peers);
      }
    }
    __syncthreads();
    if (!good) return false;
#pragma unroll
    for (int n = 0; n < NV; ++n) v[n] = 0.0;
    for (int b = threadIdx.x; b < G; b += BLOCK) {
#pragma unroll
      for (int n = 0; n < NV; ++n) v[n] += ld_relaxed_f64(gen + static_cast<long long>(n) * G + b);
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      v[n] = warp_sum(v[n]);
      if (lane == 0) sw[n][wid] = v[n];
    }
    __syncthreads();
#pragma unroll
    for (int n = 0; n < NV; ++n) v[n] = tree_sum<kWarps>(sw[n]);
  } else {
#pragma unroll
    for (int n = 0; n < NV; ++n) v[n] = tree_sum<kWarps>(sh[n]);
    __syncthreads();
  }
  return true;
}

// The member of a batched launch whose block range [first[i], first[i+1])
// holds block b (first has n + 1 ascending entries).
__device__ inline int instance_of(const int* first, int n, int b) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first[mid] <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

}  // namespace coop
}  // namespace fgw
