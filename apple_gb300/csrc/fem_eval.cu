// Evaluation API kernels: the five WarpPotential methods as one fused,
// tiled pass over the mesh (warp/fem/_base.py:243-383).
//
// One CTA per tile: the tile's vertices (<= kTileVerts) are staged in
// shared memory straight from the caller's arrays, and each warp evaluates
// conflict-free groups of the tile's elements.  The element-to-vertex scatter
// (the reference's 4 x vec3 global atomics per tet, _base.py:288-289,
// 321-322, 348-349) becomes plain read-modify-writes of the warp's private
// shared-memory accumulator; each tile writes one slot per vertex that a
// vertex pass sums in a fixed order.  Scalar outputs (energy, p^T H p) are
// reduced in float-float and finished by the last block, replacing the
// single-address scalar atomics of _base.py:261, 381.  Every output is
// bitwise reproducible.
#include <algorithm>

#include "kernels.h"
#include "pdl.cuh"
#include "tile.cuh"

namespace agb {

namespace {

// The NVEC vectors requested (of gradient, diagonal, product, in that order)
// as 3 NVEC reals per vertex: NVEC 1: one V4 (last lane unused); 2: V4 + V2;
// 3: two V4 and one real.  The accumulators and the slots share this layout.
template <int NVEC>
struct VecLayout {
  static constexpr int n4 = NVEC == 3 ? 2 : (NVEC ? 1 : 0);
  static constexpr int n2 = NVEC == 2 ? 1 : 0;
  static constexpr int n1 = NVEC == 3 ? 1 : 0;
  static constexpr int reals = 4 * n4 + 2 * n2 + n1;
};

// arrays of `n` entries each: n4 of V4, then n2 of V2, then n1 of R
template <class R, int NVEC>
struct VecArrays {
  using L = VecLayout<NVEC>;
  unsigned char* base;
  size_t n;
  __device__ __forceinline__ V4<R>* v4(int j) const { return reinterpret_cast<V4<R>*>(base) + j * n; }
  __device__ __forceinline__ V2<R>* v2() const { return reinterpret_cast<V2<R>*>(base + n * L::n4 * sizeof(V4<R>)); }
  __device__ __forceinline__ R* v1() const {
    return reinterpret_cast<R*>(base + n * (L::n4 * sizeof(V4<R>) + L::n2 * sizeof(V2<R>)));
  }
  __device__ __forceinline__ void load(size_t i, R (&x)[9]) const {
    if constexpr (NVEC >= 1) {
      const V4<R> a = v4(0)[i];
      x[0] = a.x;
      x[1] = a.y;
      x[2] = a.z;
      if constexpr (NVEC >= 2) x[3] = a.w;
    }
    if constexpr (NVEC == 2) {
      const V2<R> b = v2()[i];
      x[4] = b.x;
      x[5] = b.y;
    }
    if constexpr (NVEC == 3) {
      const V4<R> b = v4(1)[i];
      x[4] = b.x;
      x[5] = b.y;
      x[6] = b.z;
      x[7] = b.w;
      x[8] = v1()[i];
    }
  }
  __device__ __forceinline__ void store(size_t i, const R (&x)[9]) const {
    if constexpr (NVEC >= 1) v4(0)[i] = V4<R>{x[0], x[1], x[2], NVEC >= 2 ? x[3] : R(0)};
    if constexpr (NVEC == 2) v2()[i] = V2<R>{x[4], x[5]};
    if constexpr (NVEC == 3) {
      v4(1)[i] = V4<R>{x[4], x[5], x[6], x[7]};
      v1()[i] = x[8];
    }
  }
};

// staging: (x y z p.x) and, with p, (p.y p.z) per vertex
template <class R>
constexpr size_t eval_stage_bytes() {
  return (size_t)kTileVerts * (sizeof(V4<R>) + sizeof(V2<R>));
}
template <class R, int NVEC>
constexpr size_t eval_smem_bytes(int warps) {
  return eval_stage_bytes<R>() + (size_t)warps * kTileVerts * VecLayout<NVEC>::reals * sizeof(R);
}

// Bound: the shared-memory pipe and latency in FP32 (staging, gathers and
// read-modify-writes of 3 NVEC reals per corner), the FP64 pipe in FP64.  The
// records of a warp's next batch of elements (a warp group) are loaded while
// the current one computes.
// MAXT 128 (FP32): four warps per tile and five CTAs per SM, for meshes with
// enough tiles to fill the SMs; MAXT 512 (FP64: 256): up to 16 (8) warps per
// tile (blockDim), for meshes with fewer tiles than SMs, where one tile's
// serial chain of batches is the whole pass (eval_warps below).
// A call for scalars alone runs the NVEC 1 kernel without its accumulators:
// with the vector branches compiled in, the invariants are formed the same
// way, and the energy and p^T H p have the same element values whatever else
// is asked for.
// Measured, all five quantities on the 1.5M-tet grid in FP32: the call 90 us
// (170 us with shared-memory float atomics on one accumulator, a packing pass
// and separate zeroing).
// PACK (FP64): a batch is 32 consecutive elements, scattered group by group.
// FP64 pays for idle lanes, and the warp groups of small tiles are half empty
// (10 elements a group with 64 elements a tile, 27 with 256).  All five
// quantities of 138k tets in FP64: 254 us against 482 by groups with 64
// elements a tile, 207 against 238 with 256, 184.5 against 183.5 with the
// default tiles; ARAP 568 against 1,481, 541 against 671, 595 against 595.
// FemView::packed chooses.
template <class R, int MAT, int NVEC, int MAXT, bool PACK>
__global__ void __launch_bounds__(MAXT, MAXT == 128 ? 5 : 1) fem_eval_kernel(
    FemView fv, unsigned flags, const R* __restrict__ u, const R* __restrict__ p,
    const int32_t* __restrict__ p_slot, const int32_t* __restrict__ slot_of_tv, void* __restrict__ slots,
    int n_slots, AccStore<R>* __restrict__ partials, unsigned* counter, double* energy, double* quad, int assign) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V4<R>* sx = reinterpret_cast<V4<R>*>(smem_raw);
  V2<R>* sq = reinterpret_cast<V2<R>*>(sx + kTileVerts);
  unsigned char* acc = smem_raw + eval_stage_bytes<R>();
  constexpr size_t kAccBytes = (size_t)kTileVerts * VecLayout<NVEC>::reals * sizeof(R);
  __shared__ Acc<R> red[(MAXT / 32) * 2];

  const bool do_fun = flags & AGB_FUN, do_grad = flags & AGB_GRAD, do_diag = flags & AGB_HESS_DIAG;
  const bool do_prod = flags & AGB_HESS_PROD, do_quad = flags & AGB_HESS_QUAD;
  const bool need_p = do_prod || do_quad, vectors = do_grad || do_diag || do_prod;

  const int tile = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int gs = fv.tile_gstart[tile], gend = fv.tile_gstart[tile + 1];
  // the warp's batches of elements, b = g, g + warps, ... below ge
  const int ea = PACK ? fv.group_estart[gs] : 0, eb = PACK ? fv.group_estart[gend] : 0;
  const int ge = PACK ? (eb - ea + 31) / 32 : gend;
  auto batch = [&](int b, int& e0, int& count) {
    e0 = PACK ? ea + 32 * b : fv.group_estart[b];
    count = PACK ? min(32, eb - e0) : fv.group_estart[b + 1] - e0;
  };
  int g = (PACK ? 0 : gs) + warp, e0 = 0, n = 0, h = gs;  // h (PACK): the group of the batch's first element
  ElemGeo<R> geo;
  uint32_t ids = 0;
  if (g < ge) {
    batch(g, e0, n);
    if (lane < n) load_elem_m<R, MAT>(fv, e0 + lane, geo, ids);
  }
  const int vs = fv.tile_vstart[tile], nv = fv.tile_vstart[tile + 1] - vs;
  pdl_trigger();
  for (int i = threadIdx.x; i < nv; i += blockDim.x) {
    const size_t k = 3 * (size_t)fv.tv_user[vs + i];
    V4<R> a{u[k], u[k + 1], u[k + 2], R(0)};
    if (need_p) {
      if (p_slot) {  // p over the free components
        const int32_t s0 = p_slot[k], s1 = p_slot[k + 1], s2 = p_slot[k + 2];
        a.w = s0 >= 0 ? p[s0] : R(0);
        sq[i] = V2<R>{s1 >= 0 ? p[s1] : R(0), s2 >= 0 ? p[s2] : R(0)};
      } else {
        a.w = p[k];
        sq[i] = V2<R>{p[k + 1], p[k + 2]};
      }
    }
    sx[i] = a;
  }
  if (vectors) {
    V4<R>* z = reinterpret_cast<V4<R>*>(acc);
    const int nz = (int)(warps * kAccBytes / sizeof(V4<R>));
    for (int i = threadIdx.x; i < nz; i += blockDim.x) z[i] = V4<R>{R(0), R(0), R(0), R(0)};
  }
  __syncthreads();

  const VecArrays<R, NVEC> my{acc + warp * kAccBytes, (size_t)kTileVerts};
  Acc<R> sums[2] = {};
  while (g < ge) {
    const int gn = g + warps;
    int e0n = 0, nn = 0;
    ElemGeo<R> geon;
    uint32_t idsn = 0;
    if (gn < ge) {
      batch(gn, e0n, nn);
      if (lane < nn) load_elem_m<R, MAT>(fv, e0n + lane, geon, idsn);
    }
    // PACK: the end of the group that the batch begins in, and of the next one
    int end0 = 0, end1 = 0;
    if (PACK && vectors) {
      while (fv.group_estart[h + 1] <= e0) ++h;
      end0 = fv.group_estart[h + 1];
      end1 = fv.group_estart[min(h + 2, gend)];
    }
    const int l[4] = {corner(ids, 0), corner(ids, 1), corner(ids, 2), corner(ids, 3)};
    // f[q]: corner values of the q-th requested vector
    R f[NVEC][4][3];
    if (lane < n) {
      R G[3][3], dF[3][3];
      if (need_p) {
        dir_gradients(sx, sq, l, geo.D, G, dF);
      } else {
        vec_gradient(sx, l, geo.D, G);
      }
      add_act<MAT>(geo, G);
      // which vector each f[q] holds: with one or two requested the choice is
      // uniform over the launch
      auto fill = [&](auto grad, auto diag, auto prod) {
        if constexpr (NVEC == 1) {
          if (do_grad)
            grad(f[0]);
          else if (do_diag)
            diag(f[0]);
          else if (do_prod)
            prod(f[0]);
        } else if constexpr (NVEC == 2) {
          if (do_grad)
            grad(f[0]);
          else
            diag(f[0]);
          if (do_prod)
            prod(f[1]);
          else
            diag(f[1]);
        } else {
          grad(f[0]);
          diag(f[1]);
          prod(f[2]);
        }
      };
      auto clamp = [](R(&h)[4][3]) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int c = 0; c < 3; ++c) h[a][c] = clamp0(h[a][c]);
      };
      if constexpr (snh_family(MAT)) {
        SnhPoint<R> s;
        snh_prepare(G, s);
        SnhDir<R> d;
        if (need_p) snh_dir(s, dF, d);
        if (do_fun) sums[0].add(snh_energy(s, geo.mu, geo.lam));
        if (do_quad) sums[1].add(clamp0(snh_hess_quad(s, d, geo.mu, geo.lam)));
        fill(
            [&](R(&h)[4][3]) {
              R P[3][3];
              snh_pk1(s, geo.mu, geo.lam, P);
              corner_vjp(P, geo.D, h);
            },
            [&](R(&h)[4][3]) {
              snh_hess_diag(s, geo.D, geo.mu, geo.lam, h);
              clamp(h);
            },
            [&](R(&h)[4][3]) {
              R M[3][3];
              snh_hess_prod(s, d, dF, geo.mu, geo.lam, M);
              corner_vjp(M, geo.D, h);
            });
      } else {
        const R jm1 = (G[0][0] + G[1][1] + G[2][2]) + inv2(G) + det3(G);
        Svd<R> sv;
        svd_rv(G, jm1, sv);
        R lk[3];
        arap_lambdas(sv, lk);
        if (do_fun) sums[0].add(arap_energy(sv, geo.mu));
        if (do_quad) sums[1].add(clamp0(arap_hess_quad(sv, lk, dF, geo.mu)));
        fill(
            [&](R(&h)[4][3]) {
              R P[3][3];
              arap_pk1(sv, geo.mu, P);
              corner_vjp(P, geo.D, h);
            },
            [&](R(&h)[4][3]) {
              arap_hess_diag(sv, lk, geo.D, geo.mu, h);
              clamp(h);
            },
            [&](R(&h)[4][3]) {
              R M[3][3];
              arap_hess_prod(sv, lk, dF, geo.mu, M);
              corner_vjp(M, geo.D, h);
            });
      }
    }
    if (vectors) {
      // corner k of a group's lanes is a distinct vertex for every lane
      auto scatter = [&](bool mine) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          __syncwarp();
          if (mine) {
            R x[9];
            my.load(l[k], x);
#pragma unroll
            for (int q = 0; q < NVEC; ++q)
#pragma unroll
              for (int c = 0; c < 3; ++c) x[3 * q + c] += f[q][k][c];
            my.store(l[k], x);
          }
        }
        __syncwarp();
      };
      if constexpr (PACK) {
        const int e = e0 + lane;
        scatter(lane < n && e < end0);
        for (int q = h + 1, from = end0, to = end1; from < e0 + n; ++q) {
          scatter(lane < n && e >= from && e < to);
          from = to;
          to = fv.group_estart[min(q + 2, gend)];
        }
      } else {
        scatter(lane < n);
      }
    }
    g = gn;
    e0 = e0n;
    n = nn;
    geo = geon;
    ids = idsn;
  }
  if (vectors) {
    __syncthreads();
    const VecArrays<R, NVEC> out{(unsigned char*)slots, (size_t)n_slots};
    for (int i = threadIdx.x; i < nv; i += blockDim.x) {
      R x[9];
      VecArrays<R, NVEC>{acc, (size_t)kTileVerts}.load(i, x);
      for (int w = 1; w < warps; ++w) {
        R y[9];
        VecArrays<R, NVEC>{acc + w * kAccBytes, (size_t)kTileVerts}.load(i, y);
#pragma unroll
        for (int c = 0; c < 3 * NVEC; ++c) x[c] += y[c];
      }
      out.store(slot_of_tv[vs + i], x);
    }
  }

  if (do_fun || do_quad) {
    double tot[2];
    if (grid_reduce<2, R>(sums, partials, counter, gridDim.x, red, tot) && threadIdx.x == 0) {
      if (do_fun) *energy = assign ? tot[0] : *energy + tot[0];
      if (do_quad) *quad = assign ? tot[1] : *quad + tot[1];
    }
  }
}

constexpr int kUnpackThreads = 256;

// The vertex pass: a vertex's slots (contiguous, fixed order), the external
// force, and one write per requested vector in the caller's order.  Bound by
// the latency of offsets -> slots -> output, so a dependent launch reads the
// offsets before the element pass ends.
template <class R, int NVEC>
__global__ void __launch_bounds__(kUnpackThreads) unpack_kernel(
    int n, const int32_t* __restrict__ uoi, const int32_t* __restrict__ off, const void* __restrict__ slots,
    int n_slots, R* o0, R* o1, R* o2, const int32_t* __restrict__ out_slot, int assign, int force_grad,
    int force_fun, const V4<R>* __restrict__ force, const R* __restrict__ u, AccStore<R>* partials,
    unsigned* counter, double* energy) {
  __shared__ Acc<R> red[kUnpackThreads / 32];
  const VecArrays<R, NVEC> in{(unsigned char*)slots, (size_t)n_slots};
  Acc<R> ext[1] = {};
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int s0 = 0, s1 = 0, user = 0;
  if (i < n) {
    user = uoi[i];
    s0 = off[i];
    s1 = off[i + 1];
  }
  pdl_wait();
  while (i < n) {
    const size_t k = 3 * (size_t)user;
    V4<R> f{R(0), R(0), R(0), R(0)};
    if (force_grad || force_fun) f = ldg4(force + i);
    if constexpr (NVEC > 0) {
      R x[9];
#pragma unroll
      for (int c = 0; c < 3 * NVEC; ++c) x[c] = R(0);
      for (int s = s0; s < s1; ++s) {
        R y[9];
        in.load(s, y);
#pragma unroll
        for (int c = 0; c < 3 * NVEC; ++c) x[c] += y[c];
      }
      if (force_grad) {  // the gradient, when requested, is the first vector
        x[0] -= f.x;
        x[1] -= f.y;
        x[2] -= f.z;
      }
      R* const outs[3] = {o0, o1, o2};
      int64_t at[3] = {(int64_t)k, (int64_t)k + 1, (int64_t)k + 2};
      if (out_slot) {  // outputs over the free components
#pragma unroll
        for (int c = 0; c < 3; ++c) at[c] = out_slot[k + c];
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (at[c] < 0) continue;
#pragma unroll
        for (int q = 0; q < NVEC; ++q)
          outs[q][at[c]] = assign ? x[3 * q + c] : outs[q][at[c]] + x[3 * q + c];
      }
    }
    if (force_fun) ext[0].add(-(f.x * u[k] + f.y * u[k + 1] + f.z * u[k + 2]));
    i += gridDim.x * blockDim.x;
    if (i < n) {
      user = uoi[i];
      s0 = off[i];
      s1 = off[i + 1];
    }
  }
  if (force_fun) {
    double tot[1];
    if (grid_reduce<1, R>(ext, partials, counter, gridDim.x, red, tot) && threadIdx.x == 0) *energy += tot[0];
  }
}

int popcount3(unsigned vec) { return (int)((vec & 1u) + ((vec >> 1) & 1u) + ((vec >> 2) & 1u)); }

// the vectors among the flags, as a 3-bit mask (gradient, diagonal, product)
unsigned vec_mask(unsigned flags) {
  return (flags & AGB_GRAD ? 1u : 0u) | (flags & AGB_HESS_DIAG ? 2u : 0u) | (flags & AGB_HESS_PROD ? 4u : 0u);
}

// Warps per tile.  With at least two tiles per SM, four (five CTAs per SM
// keep the SM busy, and fewer accumulator copies are summed); below that the
// SMs have room, and in FP32 more warps shorten each tile's chain of groups: 8
// up to two tiles per SM, 16 up to one.  FP64 tiles arrive cut (eval_view):
// four warps, which fill the pipe, so that two CTAs share an SM, and 8 up to
// one tile per SM or for ARAP's scalars and single vectors, where the SVDs wait
// rather than compute (the energy of 138k tets with 384 elements a tile 343 us,
// 433 with four; the gradient with 192 elements 341 and 381).  All five
// quantities of 138k tets in FP64: 245 us with 214 whole tiles of 8 warps, 184
// us with 275 pieces of 4.
int eval_warps(int precision, const FemView& fv, int nvec) {
  if (precision == AGB_F64) return fv.n_tiles > kSMs && (nvec > 1 || fv.material != AGB_ARAP) ? 4 : 8;
  return fv.n_tiles > 2 * kSMs ? 4 : (fv.n_tiles > kSMs ? 8 : 16);
}

// No more warps than the largest tile has batches: the others' accumulators
// would be cleared and summed and take the shared memory and, in FP64, the
// registers of further CTAs.  Packed batches are dealt out evenly.
int used_warps(int warps, const FemView& fv) {
  if (fv.max_batches < 1) return 1;
  if (!fv.packed) return std::min(warps, fv.max_batches);
  const int rounds = (fv.max_batches + warps - 1) / warps;
  return (fv.max_batches + rounds - 1) / rounds;
}

template <class R, int MAT, int NVEC, int MAXT, bool PACK>
cudaError_t eval_launch(const FemView& fv, int warps, unsigned flags, const void* u, const void* p,
                        const int32_t* p_slot, const int32_t* slot_of_tv, void* slots, int32_t n_slots,
                        void* partials, unsigned* counter, double* energy, double* quad, int assign, cudaStream_t s) {
  const bool vectors = flags & (AGB_GRAD | AGB_HESS_DIAG | AGB_HESS_PROD);
  if (vectors || sizeof(R) == 8) warps = used_warps(warps, fv);
  const size_t smem = vectors ? eval_smem_bytes<R, NVEC>(warps) : eval_stage_bytes<R>();
  if (smem + 1024 > 48 * 1024) {  // with its static arrays above the default limit the kernel has to opt in
    const cudaError_t e = allow_max_smem(fem_eval_kernel<R, MAT, NVEC, MAXT, PACK>);
    if (e != cudaSuccess) return e;
  }
  fem_eval_kernel<R, MAT, NVEC, MAXT, PACK><<<fv.n_tiles, 32 * warps, smem, s>>>(
      fv, flags, (const R*)u, (const R*)p, p_slot, slot_of_tv, slots, n_slots, (AccStore<R>*)partials, counter, energy,
      quad, assign);
  return cudaGetLastError();
}

template <class R, int MAT, int NVEC, class... A>
cudaError_t eval_warps_of(const FemView& fv, int warps, A... args) {
  if constexpr (sizeof(R) == 8) {
    if constexpr (MAT != AGB_ARAP) {  // ARAP is always packed
      if (!fv.packed) return eval_launch<R, MAT, NVEC, 256, false>(fv, warps, args...);
    }
    return eval_launch<R, MAT, NVEC, 256, true>(fv, warps, args...);
  } else {
    return warps == 4 ? eval_launch<R, MAT, NVEC, 128, false>(fv, warps, args...)
                      : eval_launch<R, MAT, NVEC, 512, false>(fv, warps, args...);
  }
}

template <class R, int MAT, class... A>
cudaError_t eval_vectors(int nvec, const FemView& fv, A... args) {
  switch (nvec) {
    case 0:
    case 1: return eval_warps_of<R, MAT, 1>(fv, args...);
    case 2: return eval_warps_of<R, MAT, 2>(fv, args...);
    default: return eval_warps_of<R, MAT, 3>(fv, args...);
  }
}

template <class R, class... A>
cudaError_t eval_material(int nvec, const FemView& fv, A... args) {
  if (fv.material == AGB_ARAP) return eval_vectors<R, AGB_ARAP>(nvec, fv, args...);
  if (fv.material == AGB_STABLE_NEO_HOOKEAN_MUSCLE)
    return eval_vectors<R, AGB_STABLE_NEO_HOOKEAN_MUSCLE>(nvec, fv, args...);
  return eval_vectors<R, AGB_STABLE_NEO_HOOKEAN>(nvec, fv, args...);
}

template <class R, int NVEC>
cudaError_t unpack_launch(int n, const int32_t* uoi, const int32_t* off, const void* slots, int32_t n_slots,
                          unsigned flags, void* grad, void* diag, void* prod, const int32_t* out_slot, int assign,
                          const void* force, const void* u, void* partials, unsigned* counter, double* energy,
                          cudaStream_t s) {
  R* outs[3] = {nullptr, nullptr, nullptr};
  int k = 0;
  if (flags & AGB_GRAD) outs[k++] = (R*)grad;
  if (flags & AGB_HESS_DIAG) outs[k++] = (R*)diag;
  if (flags & AGB_HESS_PROD) outs[k++] = (R*)prod;
  const int force_grad = force && (flags & AGB_GRAD) ? 1 : 0, force_fun = force && (flags & AGB_FUN) ? 1 : 0;
  return launch_pdl(unpack_kernel<R, NVEC>, dim3(unpack_blocks(n)), dim3(kUnpackThreads), 0, s, n, uoi, off, slots,
                    n_slots, outs[0], outs[1], outs[2], out_slot, assign, force_grad, force_fun, (const V4<R>*)force,
                    (const R*)u, (AccStore<R>*)partials, counter, energy);
}

template <class R, class... A>
cudaError_t unpack_vectors(int nvec, A... args) {
  switch (nvec) {
    case 0: return unpack_launch<R, 0>(args...);
    case 1: return unpack_launch<R, 1>(args...);
    case 2: return unpack_launch<R, 2>(args...);
    default: return unpack_launch<R, 3>(args...);
  }
}

}  // namespace

int unpack_blocks(int n_points) {
  int b = (n_points + kUnpackThreads - 1) / kUnpackThreads;
  return b < 1 ? 1 : (b > 1216 ? 1216 : b);
}

cudaError_t launch_fem_eval(int precision, const FemView& fv, unsigned flags, const void* u, const void* p,
                            const int32_t* p_slot, const int32_t* slot_of_tv, void* slots, int32_t n_slots,
                            void* partials, unsigned* counter, double* energy, double* quad, int assign,
                            cudaStream_t stream) {
  if (fv.n_tiles == 0) return cudaSuccess;
  const int nvec = popcount3(vec_mask(flags)), warps = eval_warps(precision, fv, nvec);
  if (precision == AGB_F64)
    return eval_material<double>(nvec, fv, warps, flags, u, p, p_slot, slot_of_tv, slots, n_slots, partials, counter,
                                 energy, quad, assign, stream);
  return eval_material<float>(nvec, fv, warps, flags, u, p, p_slot, slot_of_tv, slots, n_slots, partials, counter,
                              energy, quad, assign, stream);
}

cudaError_t launch_unpack(int precision, int n, const int32_t* uoi, const int32_t* off, const void* slots,
                          int32_t n_slots, unsigned flags, void* grad, void* diag, void* prod,
                          const int32_t* out_slot, int assign, const void* force, const void* u, void* partials,
                          unsigned* counter, double* energy, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  const int nvec = popcount3(vec_mask(flags));
  if (precision == AGB_F64)
    return unpack_vectors<double>(nvec, n, uoi, off, slots, n_slots, flags, grad, diag, prod, out_slot, assign, force,
                                  u, partials, counter, energy, stream);
  return unpack_vectors<float>(nvec, n, uoi, off, slots, n_slots, flags, grad, diag, prod, out_slot, assign, force, u,
                               partials, counter, energy, stream);
}

// ---------------------------------------------------------------------------
// muscle activation: the records' D A and the offset stream S = sym(a) of
// every element, from D in FP64 (rounded once, as at set-up).  A fit sets new
// activations on every evaluation, so the product runs here and not on the
// host: D is read and the records are written once each, coalesced; only the
// 48-byte activation rows are gathered (cells in the caller's order).
// Measured on 138,240 cells in FP32: set_activation, energy, gradient and
// diagonal, and the three VJPs together take 286 us; with host loops and
// whole-record uploads in place of this kernel they took 4,697 us (743 with
// the evaluation of that time).
// ---------------------------------------------------------------------------
template <class R>
__global__ void __launch_bounds__(256) muscle_records_kernel(int n, const int32_t* __restrict__ elem_user,
                                                             const double* __restrict__ D,
                                                             const double* __restrict__ act_user, R* __restrict__ rec,
                                                             R* __restrict__ act) {
  const size_t N = (size_t)n;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const double2* row = reinterpret_cast<const double2*>(act_user + 6 * (size_t)elem_user[e]);
    const double2 a01 = row[0], a23 = row[1], a45 = row[2];
    const double a[6] = {a01.x, a01.y, a23.x, a23.y, a45.x, a45.y};
    const double A[3][3] = {{1.0 + a[0], a[3], a[4]}, {a[3], 1.0 + a[1], a[5]}, {a[4], a[5], 1.0 + a[2]}};
    double DA[9];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const double d0 = D[(3 * r) * N + e], d1 = D[(3 * r + 1) * N + e], d2 = D[(3 * r + 2) * N + e];
#pragma unroll
      for (int j = 0; j < 3; ++j) DA[3 * r + j] = fma(d2, A[2][j], fma(d1, A[1][j], d0 * A[0][j]));
    }
    if constexpr (sizeof(R) == 4) {
      float4* r4 = reinterpret_cast<float4*>(rec);
      r4[e] = make_float4((float)DA[0], (float)DA[1], (float)DA[2], (float)DA[3]);
      r4[N + e] = make_float4((float)DA[4], (float)DA[5], (float)DA[6], (float)DA[7]);
      reinterpret_cast<float*>(r4 + 2 * N + e)[0] = (float)DA[8];  // mu', lambda' and the ids stay
      float4* s4 = reinterpret_cast<float4*>(act);
      s4[e] = make_float4((float)a[0], (float)a[1], (float)a[2], (float)a[3]);
      s4[N + e] = make_float4((float)a[4], (float)a[5], 0.f, 0.f);
    } else {
#pragma unroll
      for (int k = 0; k < 9; ++k) rec[k * N + e] = DA[k];
#pragma unroll
      for (int k = 0; k < 6; ++k) act[k * N + e] = a[k];
    }
  }
}

cudaError_t launch_muscle_records(int precision, int n, const int32_t* elem_user, const double* D,
                                  const double* act_user, void* rec, void* act, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const int blocks = std::min((n + 255) / 256, 152 * 8);  // 8 resident 256-thread CTAs on each of the 152 SMs
  if (precision == AGB_F64)
    muscle_records_kernel<double><<<blocks, 256, 0, s>>>(n, elem_user, D, act_user, (double*)rec, (double*)act);
  else
    muscle_records_kernel<float><<<blocks, 256, 0, s>>>(n, elem_user, D, act_user, (float*)rec, (float*)act);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// free/fixed DOF maps (forward/dof_map/_dof_map.py:30-50): one gather each,
// with coalesced writes; to_full reads a full-length slot map (free index or
// -1) instead of scattering the free and the fixed values separately
// ---------------------------------------------------------------------------
template <class R>
__global__ void dof_to_free_kernel(int64_t n, const int64_t* __restrict__ idx, const R* __restrict__ full,
                                   R* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = full[idx[i]];
}

template <class R>
__global__ void dof_to_full_kernel(int64_t n, const int32_t* __restrict__ slot, const R* __restrict__ free_in,
                                   const R* __restrict__ fill, R* __restrict__ out) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
    const int32_t k = slot[j];
    out[j] = k >= 0 ? free_in[k] : (fill ? fill[j] : R(0));
  }
}

static int dof_blocks(int64_t n) {
  const int64_t b = (n + 255) / 256;
  const int64_t cap = 152 * 8;  // 8 resident 256-thread CTAs on each of the 152 SMs
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

cudaError_t launch_dof_to_free(int precision, int64_t n, const int64_t* idx, const void* full, void* out,
                               cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (precision == AGB_F64)
    dof_to_free_kernel<double><<<dof_blocks(n), 256, 0, s>>>(n, idx, (const double*)full, (double*)out);
  else
    dof_to_free_kernel<float><<<dof_blocks(n), 256, 0, s>>>(n, idx, (const float*)full, (float*)out);
  return cudaGetLastError();
}

cudaError_t launch_dof_to_full(int precision, int64_t n, const int32_t* slot, const void* free_in,
                               const void* fill, void* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (precision == AGB_F64)
    dof_to_full_kernel<double><<<dof_blocks(n), 256, 0, s>>>(n, slot, (const double*)free_in,
                                                            (const double*)fill, (double*)out);
  else
    dof_to_full_kernel<float><<<dof_blocks(n), 256, 0, s>>>(n, slot, (const float*)free_in,
                                                           (const float*)fill, (float*)out);
  return cudaGetLastError();
}

}  // namespace agb
