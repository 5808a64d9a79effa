// Shared by the resident kernels (solver_resident.cu, adjoint_resident.cu):
// every tile stays on one CTA for a whole run, two tiles per SM, cooperative
// launch.
#pragma once

#include "gridsync.cuh"
#include "pdl.cuh"
#include "solver.h"
#include "tile.cuh"

namespace agb {

static_assert(kResidentCounters == kPlaceWord + kPlaceWords, "barrier and placement");

// Warps per tile (two tiles per SM): 8 in FP32; FP64 is bound by its
// arithmetic pipe, which 8 warps per SM fill: 4.  Meshes with fewer tiles
// than CTAs are cut finer first (split_tiles in prep.cpp): a whole tile's
// groups are issue-bound on one SM while others idle.
template <class R>
constexpr int kResidentWarps = sizeof(R) == 4 ? 8 : 4;

// loads that see what other CTAs wrote before a barrier
template <class R>
__device__ __forceinline__ V4<R> ldcg4(const V4<R>* p);
template <>
__device__ __forceinline__ V4<float> ldcg4<float>(const V4<float>* p) {
  const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
  return V4<float>{v.x, v.y, v.z, v.w};
}
template <>
__device__ __forceinline__ V4<double> ldcg4<double>(const V4<double>* p) {
  const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  return V4<double>{a.x, a.y, b.x, b.y};
}

// Element records kept in shared memory (FP32): the float4 streams of the
// tile, [stream][element], and its groups' first elements.  A barrier's
// acquire leaves nothing in L1, so every pass would fetch them from L2.
template <int MAT>
constexpr int kRecStreams = MAT == AGB_STABLE_NEO_HOOKEAN_MUSCLE ? 5 : 3;

template <int MAT>
size_t records_bytes(const ResidentPlan& p) {
  return (size_t)p.max_elems * kRecStreams<MAT> * sizeof(float4) + ((size_t)p.max_groups + 1) * sizeof(int);
}

template <int MAT>
__device__ __forceinline__ void keep_records(const FemView& fv, int tile, int max_elems, float4* srec, int* sgrp,
                                             int tid, int threads) {
  const int e0 = fv.tile_estart[tile], ne = fv.tile_estart[tile + 1] - e0;
  const int gs = fv.tile_gstart[tile], ge = fv.tile_gstart[tile + 1];
  const float4* rec = static_cast<const float4*>(fv.rec);
  const float4* act = static_cast<const float4*>(fv.act);
  const size_t nc = (size_t)fv.n_cells;
  for (int i = tid; i < ne; i += threads) {
#pragma unroll
    for (int k = 0; k < 3; ++k) srec[(size_t)k * max_elems + i] = __ldg(rec + k * nc + e0 + i);
#pragma unroll
    for (int k = 3; k < kRecStreams<MAT>; ++k) srec[(size_t)k * max_elems + i] = __ldg(act + (k - 3) * nc + e0 + i);
  }
  for (int i = tid; i <= ge - gs; i += threads) sgrp[i] = fv.group_estart[gs + i] - e0;
}

// The record of this lane in warp group q, and the group's size: from shared
// memory (REC) or from global memory.
template <class R, int MAT, bool REC>
struct GroupLoader {
  const FemView& fv;
  int gs, max_elems;
  const float4* srec;
  const int* sgrp;
  __device__ __forceinline__ void operator()(int q, int& n, ElemGeo<R>& geo, uint32_t& ids) const {
    const int lane = threadIdx.x & 31;
    if constexpr (REC) {
      const int e0 = sgrp[q - gs];
      n = sgrp[q - gs + 1] - e0;
      if (lane >= n) return;
      const float4* r = srec + e0 + lane;
      const float4 A = r[0], B = r[max_elems], C = r[2 * max_elems];
      geo.D[0][0] = A.x; geo.D[0][1] = A.y; geo.D[0][2] = A.z;
      geo.D[1][0] = A.w; geo.D[1][1] = B.x; geo.D[1][2] = B.y;
      geo.D[2][0] = B.z; geo.D[2][1] = B.w; geo.D[2][2] = C.x;
      geo.mu = C.y;
      geo.lam = C.z;
      ids = __float_as_uint(C.w);
      if constexpr (kRecStreams<MAT> == 5) {
        const float4 s0 = r[3 * max_elems], s1 = r[4 * max_elems];
        geo.S[0] = s0.x; geo.S[1] = s0.y; geo.S[2] = s0.z;
        geo.S[3] = s0.w; geo.S[4] = s1.x; geo.S[5] = s1.y;
      }
    } else {
      const int e0 = fv.group_estart[q];
      n = fv.group_estart[q + 1] - e0;
      if (lane < n) load_elem_m<R, MAT>(fv, e0 + lane, geo, ids);
    }
  }
};

// The first shape (1: FP32 records in shared memory; 2, or 1 in FP64: not)
// whose CTAs fit the device at once, into p->shape; 0 if none
// does (too many tiles, or tiles with too many elements).
template <class ShapeOf>
cudaError_t choose_shape(const SolveArgs& a, ResidentPlan* p, ShapeOf shape_of) {
  p->shape = 0;
  if (a.fv.n_tiles == 0 || a.fv.n_tiles > kResidentMaxTiles) return cudaSuccess;
  int dev = 0, sms = 0, coop = 0, limit = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess || !coop) return e;
  const int shapes = a.precision == AGB_F64 ? 1 : 2;
  for (int k = 1; k <= shapes; ++k) {
    ResidentPlan q = *p;
    q.shape = k;
    const auto sh = shape_of(q);
    if (sh.smem + 8 * 1024 > (size_t)limit) continue;  // beside the kernel's static arrays
    int occ = 0;
    e = allow_max_smem(sh.kernel);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, sh.kernel, sh.threads, sh.smem);
    if (e != cudaSuccess) return e;
    if ((int64_t)sh.blocks <= (int64_t)occ * sms) {
      p->shape = k;
      return cudaSuccess;
    }
  }
  return cudaSuccess;
}

template <class... P, class... A>
cudaError_t launch_cooperative(void (*k)(P...), int blocks, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace agb
