// Barrier and deterministic sums across the CTAs of a cooperative launch.
//
// The barrier is a counter of arrivals: CTA thread 0 adds one and polls until
// every CTA has arrived `round` times.  The wait is bounded: at its limit it
// polls once more and gives up; its CTA leaves, and the others' next waits give
// up too.  The counter of CTAs that left also counts those that gave up, so the
// last one to leave learns of it, after everything the others wrote; it resets
// the counters for the next launch.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "bulk.cuh"
#include "reduce.cuh"

namespace agb {

// words of `counters`, zero before the first launch
constexpr int kArrived = 0, kLeft = 1, kPlaceWord = 2;
constexpr unsigned kGaveUp = 1u << 16;  // in kLeft, above the CTAs that left

struct GridBar {
  unsigned* counters;
  int words;           // reset by the last CTA to leave
  uint64_t limit;      // of a wait, ns
  unsigned n;          // CTAs
  unsigned round;      // barriers passed
  bool gave_up;        // thread 0: its wait ran out

  // every thread of the CTA calls it; what the CTA wrote before is visible to
  // the others after their wait().  Work that needs nothing from them can go
  // between arrive() and wait().
  __device__ __forceinline__ void arrive() {
    ++round;
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(&counters[kArrived], 1u);
    }
  }

  // wait until every CTA has arrived; false when the wait gave up
  __device__ __forceinline__ bool wait() {
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
      const unsigned want = round * n;
      const uint64_t t0 = global_ns();
      bool ok = true;
      for (;;) {
        const bool late = global_ns() - t0 >= limit;  // read before the load, which may come long after it
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counters + kArrived) : "memory");
        if ((int)(v - want) >= 0) break;  // the counter may wrap
        if (late) {
          ok = false;
          gave_up = true;
          break;
        }
      }
      s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
  }

  // every CTA once, after its last wait(), whether that gave up or not; true
  // in thread 0 of the last CTA when a wait gave up anywhere
  __device__ __forceinline__ bool leave() {
    __syncthreads();
    if (threadIdx.x != 0) return false;
    __threadfence();
    const unsigned before = atomicAdd(&counters[kLeft], gave_up ? 1u + kGaveUp : 1u);
    if (before % kGaveUp != n - 1u) return false;
    for (int k = 0; k < words; ++k) counters[k] = 0u;
    if (before < kGaveUp && !gave_up) return false;
    __threadfence();  // what the others wrote comes before what the caller reports
    return true;
  }
};

// The CTA's sum of each of N quantities into part[k * n + block].  x: the
// thread's terms; lo: the low word of quantity LO (float-float), or unused
// with LO < 0.  The terms go through shared memory (`rows`: N + 1 rows of
// THREADS reals) so that one warp adds one quantity, instead of every warp
// reducing all N by shuffles, in float-float from the threads' terms on.
// (Same-sign sums in plain FP32 above the threads had several times the
// rounding error and were no faster: 14.0 us an iteration of the 5k-tet cube.)
template <int N, int LO, int THREADS, class R>
__device__ __forceinline__ void cta_partials(const R (&x)[N], R lo, R* rows, AccStore<R>* part, int n, int block) {
  constexpr int NW = THREADS / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) rows[k * THREADS + threadIdx.x] = x[k];
  if constexpr (LO >= 0) rows[N * THREADS + threadIdx.x] = lo;
  __syncthreads();
  for (int k = warp; k < N; k += NW) {
    const R* row = rows + k * THREADS;
    Acc<R> s{};
#pragma unroll 4
    for (int j = 0; j < NW; ++j) s.add(row[lane + 32 * j]);
    if (k == LO) {
      R l = R(0);
#pragma unroll 4
      for (int j = 0; j < NW; ++j) l += rows[N * THREADS + lane + 32 * j];
      s.add(l);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s.add(s.shfl_down(off));
    if (lane == 0) part[(size_t)k * n + block] = acc_store(s);
  }
}

// After a barrier: the sums over all CTAs in every CTA, into shared tot: a
// warp per quantity (its KPW quantities interleaved, so that their loads are
// in flight together); complete after the closing __syncthreads.
template <int N, int THREADS, class R>
__device__ __forceinline__ void grid_totals(const AccStore<R>* part, int n, Acc<R>* tot) {
  constexpr int NW = THREADS / 32, KPW = (N + NW - 1) / NW, U = 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Acc<R> s[KPW] = {};
  for (int b0 = lane; b0 < n; b0 += 32 * U) {
    Acc<R> v[KPW][U] = {};
#pragma unroll
    for (int j = 0; j < KPW; ++j)
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (warp + j * NW < N && b0 + 32 * q < n)
          v[j][q] = acc_load<R>(part + (size_t)(warp + j * NW) * n + b0 + 32 * q);
#pragma unroll
    for (int j = 0; j < KPW; ++j)
#pragma unroll
      for (int q = 0; q < U; ++q) s[j].add(v[j][q]);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int j = 0; j < KPW; ++j) s[j].add(s[j].shfl_down(off));
  }
#pragma unroll
  for (int j = 0; j < KPW; ++j)
    if (lane == 0 && warp + j * NW < N) tot[warp + j * NW] = s[j];
  __syncthreads();
}

// The work item of this CTA when the first `whole` of n items are large: the
// first CTA to arrive on an SM takes the next large one, a second CTA there
// the next of the others, so that no SM holds two large items while another
// holds none.  counters[kPlaceWord] and the next: items taken; those after:
// CTAs on each SM (kPlaceWords words in all, zero before the launch).
// Called by one thread.
constexpr int kPlaceSms = 256;
constexpr int kPlaceWords = 2 + kPlaceSms;

__device__ __forceinline__ int place_cta(unsigned* counters, int whole, int n) {
  unsigned sm;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
  counters += kPlaceWord;
  const bool first = atomicAdd(&counters[2 + (sm & (kPlaceSms - 1))], 1u) == 0u;
  if (first) {
    const int k = (int)atomicAdd(&counters[0], 1u);
    if (k < whole) return k;
    return min(whole + (int)atomicAdd(&counters[1], 1u), n - 1);
  }
  const int k = (int)atomicAdd(&counters[1], 1u);
  if (whole + k < n) return whole + k;
  return min((int)atomicAdd(&counters[0], 1u), n - 1);
}

}  // namespace agb
