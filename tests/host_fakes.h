// A host-only stand-in for the CUDA runtime and the kernel launchers, for C++
// programs that link the package's host code (capi.cpp, prep.cpp) alone:
// device memory is host memory, launches are counted or checked by the
// program, and the allocation that is number `fail_at` from now on fails.
#pragma once

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <vector>

#include "apple_gb300.h"
#include "kernels.h"
#include "solver.h"

namespace fake {
inline std::set<void*> live;
inline int fail_at = 0;  // 1: the next allocation fails; 0: none does
inline int sms = 152;
inline cudaError_t alloc(void** p, size_t n) {
  if (fail_at > 0 && --fail_at == 0) return cudaErrorMemoryAllocation;
  *p = malloc(n);
  memset(*p, 0x5a, n);
  live.insert(*p);
  return cudaSuccess;
}
inline cudaError_t release(void* p) {
  if (p && !live.erase(p)) {
    printf("freed twice\n");
    exit(99);
  }
  free(p);
  return cudaSuccess;
}
}  // namespace fake

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return fake::alloc(p, n); }
cudaError_t cudaFree(void* p) { return fake::release(p); }
cudaError_t cudaFreeHost(void* p) { return fake::release(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? fake::sms : 1;
  return cudaSuccess;
}
}

namespace agb {
int unpack_blocks(int n) { return (n + 255) / 256; }
int solver_vertex_blocks(int n) { return (n + 255) / 256; }
cudaError_t solver_prepare_kernels(int) { return cudaSuccess; }
cudaError_t cg_prepare_kernels(int) { return cudaSuccess; }
}  // namespace agb

// a grid of n x n x n cells, five tets each, E and nu alike
struct FakeMesh {
  std::vector<double> points, mu, lam;
  std::vector<int32_t> cells;
  explicit FakeMesh(int n) {
    auto id = [n](int i, int j, int k) { return (i * (n + 1) + j) * (n + 1) + k; };
    for (int i = 0; i <= n; ++i)
      for (int j = 0; j <= n; ++j)
        for (int k = 0; k <= n; ++k) points.insert(points.end(), {(double)i, (double)j, (double)k});
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        for (int k = 0; k < n; ++k) {
          int v[8];
          for (int c = 0; c < 8; ++c) v[c] = id(i + (c >> 2), j + ((c >> 1) & 1), k + (c & 1));
          static const int even[5][4] = {{0, 4, 2, 1}, {3, 1, 2, 7}, {5, 4, 1, 7}, {6, 2, 4, 7}, {1, 2, 4, 7}};
          static const int odd[5][4] = {{1, 0, 5, 3}, {2, 3, 6, 0}, {4, 5, 0, 6}, {7, 6, 3, 5}, {0, 3, 6, 5}};
          for (int t = 0; t < 5; ++t)
            for (int c = 0; c < 4; ++c) cells.push_back(v[((i + j + k) & 1 ? odd : even)[t][c]]);
        }
    mu.assign(cells.size() / 4, 1.0);
    lam.assign(cells.size() / 4, 2.0);
  }
  int n_points() const { return (int)points.size() / 3; }
  int n_cells() const { return (int)cells.size() / 4; }
};
