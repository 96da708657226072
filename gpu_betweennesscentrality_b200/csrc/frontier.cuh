// frontier.cuh -- frontier lists of the shortest-path sweeps (sssp.cu, core.cuh) in vertex order.
#pragma once

#include <cuda_runtime.h>

namespace qbc {
namespace {

constexpr unsigned kSweepFull = 0xffffffffu;
constexpr int kSortBuckets = 4096;  // shared-memory counters of the whole graph's frontier ordering
constexpr int kSortMinLen = 1024;   // shorter lists are visited as they are

// Exclusive scan of c[0..len) in place (len <= BUCKETS), whole CTA; red holds 33 ints.
template <int THREADS, int BUCKETS>
__device__ __forceinline__ void cta_exclusive_scan(int *c, int len, int *red) {
  constexpr int per = (BUCKETS + THREADS - 1) / THREADS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = tid * per;
  int local = 0;
#pragma unroll
  for (int k = 0; k < per; k++) local += (b + k < len) ? c[b + k] : 0;
  int x = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kSweepFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) red[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int t = lane < THREADS / 32 ? red[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(kSweepFull, t, o);
      if (lane >= o) t += y;
    }
    red[lane] = t;  // inclusive warp totals
  }
  __syncthreads();
  int run = x - local + (warp > 0 ? red[warp - 1] : 0);
#pragma unroll
  for (int k = 0; k < per; k++)
    if (b + k < len) {
      const int v = c[b + k];
      c[b + k] = run;
      run += v;
    }
  __syncthreads();
}

// Frontier ordering: a list of vertices is rewritten into `out` grouped by v >> shift (a counting
// sort, CTA-wide), so that a pass visits the frontier in vertex-id order.  Near lists and Kahn
// waves are bands of the graph; in id order consecutive visits share record lines, and the rows
// above and below are visited soon after, while their lines are still in L1/L2.
template <int THREADS, int BUCKETS, class IN, class OUT>
__device__ __forceinline__ void order_frontier(int shift, int buckets, IN in, int len, OUT out, int *hist, int *red) {
  const int tid = threadIdx.x;
  for (int i = tid; i < buckets; i += THREADS) hist[i] = 0;
  __syncthreads();
  for (int i = tid; i < len; i += THREADS) atomicAdd(hist + (in(i) >> shift), 1);
  __syncthreads();
  cta_exclusive_scan<THREADS, BUCKETS>(hist, buckets, red);
  for (int i = tid; i < len; i += THREADS) {
    const int v = in(i);
    out(atomicAdd(hist + (v >> shift), 1)) = v;
  }
  __syncthreads();
}

}  // namespace
}  // namespace qbc
