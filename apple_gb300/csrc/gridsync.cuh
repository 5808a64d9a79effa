// Barrier and deterministic sums across the CTAs of a cooperative launch.
//
// The barrier is a counter of arrivals: CTA thread 0 adds one and polls until
// every CTA has arrived `round` times.  The wait is bounded: after about two
// seconds it gives up, the caller reports a device error and returns.  The
// last CTA to leave the kernel resets the counters for the next launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk.cuh"
#include "reduce.cuh"

namespace agb {

struct GridBar {
  unsigned* counters;  // [0] arrivals, [1] exits; zero before the first launch
  unsigned n;          // CTAs
  unsigned round;      // barriers passed

  // every thread of the CTA calls it; false when the wait gave up
  __device__ __forceinline__ bool sync() {
    __shared__ int s_ok;
    ++round;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&counters[0], 1u);
      const unsigned want = round * n;
      const uint64_t t0 = global_ns();
      bool ok = true;
      for (;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counters) : "memory");
        if (v >= want) break;
        if (global_ns() - t0 > 2000000000ull) {
          ok = false;
          break;
        }
      }
      s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
  }

  // every CTA once, after its last sync()
  __device__ __forceinline__ void leave() {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&counters[1], 1u) == n - 1u) {
      counters[0] = 0u;
      counters[1] = 0u;
    }
  }
};

// The CTA's sums of N quantities into part[k * n + block]: float-float warp
// trees for the quantities in FF, plain ones for the others, then the warps
// in order (as block_reduce).
template <int N, unsigned FF, class R>
__device__ __forceinline__ void cta_partials(Acc<R> (&a)[N], Acc<R>* scratch, AccStore<R>* part, int n) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    if ((FF >> k) & 1u) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) a[k].add(a[k].shfl_down(off));
    } else {
      a[k].warp_plain_sum();
    }
  }
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) scratch[warp * N + k] = a[k];
  }
  __syncthreads();
  if (threadIdx.x < N) {
    Acc<R> s = scratch[threadIdx.x];
    for (int w = 1; w < nw; ++w) s.add(scratch[w * N + threadIdx.x]);
    part[(size_t)threadIdx.x * n + blockIdx.x] = acc_store(s);
  }
}

// After a barrier: the sums over all CTAs, in every CTA.  Warp w adds
// quantities w, w + nw, ...; tot is complete after the closing __syncthreads.
template <int N, class R>
__device__ __forceinline__ void grid_totals(const AccStore<R>* part, int n, double* tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = warp; k < N; k += nw) {
    Acc<R> s{};
#pragma unroll 4
    for (int b = lane; b < n; b += 32) s.add(acc_load<R>(part + (size_t)k * n + b));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s.add(s.shfl_down(off));
    if (lane == 0) tot[k] = s.value();
  }
  __syncthreads();
}

}  // namespace agb
