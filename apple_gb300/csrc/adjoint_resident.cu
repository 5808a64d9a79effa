// Adjoint CG of a small or medium mesh in one cooperative launch.
//
// The three-kernel iteration (adjoint.cu) is bound by its launches and serial
// tails on meshes of a few hundred tiles; here every tile stays on a resident
// CTA (as in solver_resident.cu) and three grid barriers separate the passes:
//
//   element   p = z + beta p_prev per tile vertex; H_e p -> slots
//   -- barrier --
//   vertex 1  32 consecutive vertices per warp: q = sum of slots (masked), p . q
//   -- barrier: p . q, alpha --
//   vertex 2  lam += alpha p, r -= alpha q, z = M^-1 r (stored); r . z and r . r
//   -- barrier: sums, beta, convergence --
//
// x, the element records and p stay in shared memory for the whole solve, and
// lam, r, p and M^-1 of a vertex with its thread; z, the slots and the
// partials pass through L2.
//
// A CG amplifies rounding where H is nearly singular, so every FP32 sum keeps
// the three-kernel iteration's order and the results its bits: four
// accumulator copies per tile, each adding the groups of one residue class in
// order (two warps take turns on a copy, so that eight can compute), slots in
// CSR order, and plain 32-vertex warp sums for r . z and r . r; the sums above
// those are float-float, whose order does not reach the FP32 scalars.
//
// Measured: 40 iterations with the material gradients on 138,240 tets 723 us
// against 1,105, on 5,000 tets 553 against 952 (FP32, the same bits); 30 FP64
// iterations on 40,000 tets 2,365 against 2,744.  Above two tiles per SM the
// tiles do not fit at once and the three-kernel iteration runs.
#include <math.h>

#include <algorithm>

#include "resident.cuh"
#include "solver.h"
#include "solver_common.cuh"

namespace agb {

namespace {

constexpr int kCopies = 4;      // accumulator copies per tile (adjoint.cu: kCgWarps)
constexpr int kCgCap = 256;     // vertices per CTA in the vertex passes: at most 8 chunks of 32
// kept per vertex of the vertex passes: p, lam, r, M^-1, q, mask
constexpr int kCgWords = 16;

template <class R>
constexpr size_t cg_resident_smem() {
  return (size_t)kTileVerts * ((kCopies + 2) * sizeof(V4<R>) + sizeof(V2<R>) + 2 * sizeof(int)) +
         (size_t)kCgCap * (kCgWords * sizeof(R) + 2 * sizeof(int));
}

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <class R, int MAT, int NW, bool REC>
__global__ void __launch_bounds__(32 * NW, 2) cg_resident_kernel(CgArgs c, int max_elems, void* part_p, void* part_v,
                                                                unsigned* counters, uint64_t wait_ns) {
  constexpr int T = 32 * NW, TURNS = NW / kCopies, kSlotBatch = 4;
  static_assert(TURNS == 1 || TURNS == 2, "one or two warps per accumulator copy");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V4<R>* sh = reinterpret_cast<V4<R>*>(smem_raw);  // x hi, x lo.x
  V4<R>* sp = sh + kTileVerts;                     // p
  V4<R>* acc = sp + kTileVerts;                    // [copy][vertex]
  V2<R>* sl = reinterpret_cast<V2<R>*>(acc + kCopies * kTileVerts);  // x lo.y, lo.z
  R* vw = reinterpret_cast<R*>(sl + kTileVerts);
  int* vi = reinterpret_cast<int*>(vw + kCgWords * kCgCap);  // tile vertices: vertex, slot
  int* vo = vi + 2 * kTileVerts;                             // pass vertices: first and end slot
  float4* srec = reinterpret_cast<float4*>(vo + 2 * kCgCap);
  int* sgrp = reinterpret_cast<int*>(srec + (size_t)kRecStreams<MAT> * max_elems);
  __shared__ Acc<R> red[NW * 2];
  __shared__ Acc<R> tot[2];
  __shared__ CgState cs;
  __shared__ R s_alpha, s_beta;
  __shared__ int s_end;
  auto word = [&](int w, int j) -> R& { return vw[w * kCgCap + j]; };
  constexpr int P = 0, LAM = 3, RES = 6, MINV = 9, Q = 12, MASK = 15;

  if (c.cs->done) return;
  const SolveArgs& a = c.a;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, tile = blockIdx.x;
  const int copy = warp % kCopies, turn = warp / kCopies;
  const int gs = a.fv.tile_gstart[tile], ge = a.fv.tile_gstart[tile + 1];
  const int rounds = (ge - gs + NW - 1) / NW;
  const int vs = a.fv.tile_vstart[tile], nv = a.fv.tile_vstart[tile + 1] - vs;
  const int n = a.n_points, chunks = (n + 31) / 32;
  const int mine = (chunks - tile + (int)gridDim.x - 1) / (int)gridDim.x;  // chunks tile, tile + grid, ...
  if (tid == 0) cs = *c.cs;
  GridBar bar{counters, kResidentCounters, wait_ns, gridDim.x, 0, false};
  V4<R>* slots = (V4<R>*)a.slots;
  V4<R>* Z = (V4<R>*)c.q;  // z = M^-1 r of the current residual
  for (int i = tid; i < nv; i += T) {
    const int v = a.fv.tv_vid[vs + i];
    vi[i] = v;
    vi[kTileVerts + i] = a.slot_of_tv[vs + i];
    const V4<R> x = ((const V4<R>*)a.xa)[2 * v], xl = ((const V4<R>*)a.xa)[2 * v + 1];
    sh[i] = V4<R>{x.x, x.y, x.z, xl.x};
    sl[i] = V2<R>{xl.y, xl.z};
    const V4<R> m = ((const V4<R>*)c.minv)[v], r = ((const V4<R>*)c.res)[v];
    // the first p: z + 0 p_prev
    sp[i] = V4<R>{add_rn(mul_rn(m.x, r.x), R(0)), add_rn(mul_rn(m.y, r.y), R(0)), add_rn(mul_rn(m.z, r.z), R(0)), R(0)};
  }
  for (int k = warp; k < mine; k += NW) {
    const int j = 32 * k + lane, v = 32 * (tile + k * (int)gridDim.x) + lane;
    if (v >= n) continue;
    vo[j] = a.off[v];
    vo[kCgCap + j] = a.off[v + 1];
    const V4<R> m4 = ((const V4<R>*)c.minv)[v], r4 = ((const V4<R>*)c.res)[v];
    const R m[3] = {m4.x, m4.y, m4.z}, r[3] = {r4.x, r4.y, r4.z};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      word(P + d, j) = add_rn(mul_rn(m[d], r[d]), R(0));
      word(LAM + d, j) = R(0);
      word(RES + d, j) = r[d];
      word(MINV + d, j) = m[d];
    }
    word(MASK, j) = ((const V4<R>*)a.xa)[2 * v].w;
  }
  if constexpr (REC) keep_records<MAT>(a.fv, tile, max_elems, srec, sgrp, threadIdx.x, blockDim.x);
  const GroupLoader<R, MAT, REC> load{a.fv, gs, max_elems, srec, sgrp};
  __syncthreads();

  bool ok = true;
  for (;;) {
    // ---- element ----
    for (int w = 0; w < kCopies; ++w)
      for (int i = tid; i < nv; i += T) acc[w * kTileVerts + i] = V4<R>{R(0), R(0), R(0), R(0)};
    int g = gs + warp, ng = 0;
    ElemGeo<R> geo;
    uint32_t ids = 0;
    if (!REC && g < ge) load(g, ng, geo, ids);
    __syncthreads();
    {
      V4<R>* my = acc + copy * kTileVerts;
      for (int round = 0; round < rounds; ++round) {
        const int gn = g + NW;
        int nn = 0;
        ElemGeo<R> geon;
        uint32_t idsn = 0;
        if constexpr (REC) {
          ng = 0;
          if (g < ge) load(g, ng, geo, ids);
        } else if (gn < ge) {
          load(gn, nn, geon, idsn);
        }
        const int l[4] = {corner(ids, 0), corner(ids, 1), corner(ids, 2), corner(ids, 3)};
        R f[4][3];
        if (lane < ng) {
          R G[3][3], dF[3][3], M[3][3];
          pair_gradient(sh, sl, l, geo.D, G);
          vec_gradient(sp, l, geo.D, dF);
          add_act<MAT>(geo, G);
          if constexpr (snh_family(MAT)) {
            SnhPoint<R> s;
            snh_prepare(G, s);
            SnhDir<R> d;
            snh_dir(s, dF, d);
            snh_hess_prod(s, d, dF, geo.mu, geo.lam, M);
          } else {
            const R jm1 = (G[0][0] + G[1][1] + G[2][2]) + inv2(G) + det3(G);
            Svd<R> sv;
            svd_rv(G, jm1, sv);
            R lk[3];
            arap_lambdas(sv, lk);
            arap_hess_prod(sv, lk, dF, geo.mu, M);
          }
          corner_vjp(M, geo.D, f);
        }
        // the copy's groups in order: turn 0's, then turn 1's of this round
        if constexpr (TURNS == 2) {
          if (turn == 1)
            bar_sync(1 + copy, 64);
          else if (round > 0)
            bar_sync(1 + kCopies + copy, 64);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          __syncwarp();
          if (lane < ng) {
            V4<R> q = my[l[k]];
            q.x += f[k][0];
            q.y += f[k][1];
            q.z += f[k][2];
            my[l[k]] = q;
          }
        }
        __syncwarp();
        if constexpr (TURNS == 2) bar_arrive(turn == 0 ? 1 + copy : 1 + kCopies + copy, 64);
        g = gn;
        if constexpr (!REC) {
          ng = nn;
          geo = geon;
          ids = idsn;
        }
      }
      if constexpr (TURNS == 2) {
        if (turn == 0 && rounds > 0) bar_sync(1 + kCopies + copy, 64);
      }
    }
    __syncthreads();
    for (int i = tid; i < nv; i += T) {
      V4<R> q = acc[i];
#pragma unroll
      for (int w = 1; w < kCopies; ++w) {
        const V4<R> r = acc[w * kTileVerts + i];
        q.x += r.x;
        q.y += r.y;
        q.z += r.z;
      }
      slots[2 * (size_t)vi[kTileVerts + i]] = V4<R>{q.x, q.y, q.z, R(0)};
    }
    bar.arrive();
    if (!(ok = bar.wait())) break;

    // ---- vertex 1: q, p . q ----
    {
      Acc<R> s[1] = {};
      for (int k = warp; k < mine; k += NW) {
        const int j = 32 * k + lane, v = 32 * (tile + k * (int)gridDim.x) + lane;
        if (v >= n) continue;
        const int mask = (int)word(MASK, j);
        R q[3] = {R(0), R(0), R(0)};
        for (int b = vo[j]; b < vo[kCgCap + j]; b += kSlotBatch) {
          V4<R> t[kSlotBatch];
#pragma unroll
          for (int m = 0; m < kSlotBatch; ++m)
            if (b + m < vo[kCgCap + j]) t[m] = ldcg4(slots + 2 * (size_t)(b + m));
#pragma unroll
          for (int m = 0; m < kSlotBatch; ++m)
            if (b + m < vo[kCgCap + j]) {
              q[0] += t[m].x;
              q[1] += t[m].y;
              q[2] += t[m].z;
            }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if ((mask >> d) & 1) q[d] = R(0);
          word(Q + d, j) = q[d];
        }
        s[0].add(word(P, j) * q[0] + word(P + 1, j) * q[1] + word(P + 2, j) * q[2]);
      }
      block_reduce<1, 0x1u, R>(s, red);
      if (tid == 0) ((AccStore<R>*)part_p)[tile] = acc_store(s[0]);
    }
    bar.arrive();
    if (!(ok = bar.wait())) break;
    grid_totals<1, T, R>((const AccStore<R>*)part_p, gridDim.x, tot);
    if (warp == 0) {
      const double pq = tot[0].value();
      const bool pos = positive_finite(pq);  // else H is not positive definite along p, or NaN
      const double al = pos ? cs.rz / pq : 0.0;
      if (lane == 0) {
        if (!pos) {
          cs.done = 1;
          cs.result = finite_bits(pq) ? AGB_LINE_SEARCH_FAILED : AGB_NAN_ENCOUNTERED;
        }
        cs.alpha = al;
        s_alpha = to_real<R>(al);
      }
    }
    __syncthreads();
    if (cs.done) break;

    // ---- vertex 2: lam, r, z, r . z, r . r ----
    {
      const R alpha = s_alpha;
      Acc<R> s[2] = {};
      for (int k = warp; k < mine; k += NW) {
        const int j = 32 * k + lane, v = 32 * (tile + k * (int)gridDim.x) + lane;
        Acc<R> t[2] = {};
        if (v < n) {
          R r[3], z[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            word(LAM + d, j) = fma_rn(alpha, word(P + d, j), word(LAM + d, j));
            r[d] = fma_rn(-alpha, word(Q + d, j), word(RES + d, j));
            word(RES + d, j) = r[d];
            z[d] = mul_rn(word(MINV + d, j), r[d]);
          }
          t[0].add(r[0] * z[0] + r[1] * z[1] + r[2] * z[2]);
          t[1].add(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
          Z[v] = V4<R>{z[0], z[1], z[2], R(0)};
        }
        t[0].warp_plain_sum();
        t[1].warp_plain_sum();
        s[0].add(t[0]);
        s[1].add(t[1]);
      }
      if (lane == 0) {
        red[2 * warp] = s[0];
        red[2 * warp + 1] = s[1];
      }
      __syncthreads();
      if (tid < 2) {
        Acc<R> b = red[tid];
        for (int w = 1; w < NW; ++w) b.add(red[2 * w + tid]);
        ((AccStore<R>*)part_v)[(size_t)tid * gridDim.x + tile] = acc_store(b);
      }
    }
    bar.arrive();
    if (!(ok = bar.wait())) break;
    grid_totals<2, T, R>((const AccStore<R>*)part_v, gridDim.x, tot);
    if (warp == 0) {
      const double rz = tot[0].value();
      const double b = cs.rz > 0.0 ? rz / cs.rz : 0.0;
      __syncwarp();
      if (lane == 0) {
        cs.beta = b;
        cs.rz = rz;
        s_beta = to_real<R>(b);
      }
    } else if (warp == 1) {
      const double rr = tot[1].value();
      const double rn = sqrt(rr);
      const bool small = rn <= fmax(cs.atol, cs.rtol * sqrt(cs.rr0));
      __syncwarp();
      if (lane == 0) {
        cs.rr = rr;
        cs.iter += 1;
        cs.pbuf ^= 1;
        if (!finite_bits(rn)) {
          cs.done = 1;
          cs.result = AGB_NAN_ENCOUNTERED;
        } else if (small) {
          cs.done = 1;
          cs.result = AGB_PRIMARY_SUCCESS;
        } else if (cs.iter >= cs.max_iter) {
          cs.done = 1;
          cs.result = AGB_MAX_STEPS_REACHED;
        }
        s_end = cs.done || cs.iter >= cs.iter_limit;
      }
    }
    __syncthreads();
    if (s_end) break;
    // the next p, of the tile's vertices and of this thread's
    const R beta = s_beta;
    for (int i = tid; i < nv; i += T) {
      const V4<R> z = ldcg4(Z + vi[i]), po = sp[i];
      sp[i] = V4<R>{fma_rn(beta, po.x, z.x), fma_rn(beta, po.y, z.y), fma_rn(beta, po.z, z.z), R(0)};
    }
    for (int k = warp; k < mine; k += NW) {
      const int j = 32 * k + lane;
      if (32 * (tile + k * (int)gridDim.x) + lane >= n) continue;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        word(P + d, j) = fma_rn(beta, word(P + d, j), mul_rn(word(MINV + d, j), word(RES + d, j)));
    }
  }

  if (ok) {
    for (int k = warp; k < mine; k += NW) {
      const int j = 32 * k + lane, v = 32 * (tile + k * (int)gridDim.x) + lane;
      if (v < n) ((V4<R>*)c.lam)[v] = V4<R>{word(LAM, j), word(LAM + 1, j), word(LAM + 2, j), R(0)};
    }
    if (tile == 0 && tid == 0) *c.cs = cs;
  }
  if (bar.leave()) {  // a barrier gave up
    c.cs->done = 1;
    c.cs->result = AGB_E_DEVICE;
  }
}

using CgKernel = void (*)(CgArgs, int, void*, void*, unsigned*, uint64_t);

struct Shape {
  CgKernel kernel;
  int blocks, threads;
  size_t smem;
};

template <class R, int MAT, bool REC>
Shape shape(const ResidentPlan& p, int n_tiles) {
  constexpr int NW = kResidentWarps<R>;
  size_t smem = cg_resident_smem<R>();
  if (REC) smem += records_bytes<MAT>(p);
  // up to one tile per SM: more shared memory than half an SM's, so that no
  // two CTAs share an SM while others idle
  if (n_tiles <= p.sms) smem = std::max(smem, (size_t)120 * 1024);
  return Shape{cg_resident_kernel<R, MAT, NW, REC>, n_tiles, 32 * NW, smem};
}

template <int MAT>
Shape shape_of(int precision, const ResidentPlan& p, int nt) {
  if (precision == AGB_F64) return shape<double, MAT, false>(p, nt);
  return p.shape == 1 ? shape<float, MAT, true>(p, nt) : shape<float, MAT, false>(p, nt);
}

Shape shape_of(const SolveArgs& a, const ResidentPlan& p) {
  if (a.fv.material == AGB_ARAP) return shape_of<AGB_ARAP>(a.precision, p, a.fv.n_tiles);
  if (a.fv.material == AGB_STABLE_NEO_HOOKEAN_MUSCLE)
    return shape_of<AGB_STABLE_NEO_HOOKEAN_MUSCLE>(a.precision, p, a.fv.n_tiles);
  return shape_of<AGB_STABLE_NEO_HOOKEAN>(a.precision, p, a.fv.n_tiles);
}

}  // namespace

cudaError_t cg_resident_prepare(const SolveArgs& a, ResidentPlan* p) {
  p->shape = 0;
  // every chunk of 32 vertices needs a place (a point that no cell uses may
  // leave more vertices than tiles hold)
  if (a.fv.n_tiles == 0 || (a.n_points + 31) / 32 > (int64_t)a.fv.n_tiles * (kCgCap / 32)) return cudaSuccess;
  return choose_shape(a, p, [&](const ResidentPlan& q) { return shape_of(a, q); });
}

cudaError_t launch_cg_resident(const CgArgs& c, const ResidentPlan& p, void* part_p, void* part_v, unsigned* counters,
                               cudaStream_t s) {
  if (!p.shape) return cudaErrorInvalidValue;
  const Shape sh = shape_of(c.a, p);
  return launch_cooperative(sh.kernel, sh.blocks, sh.threads, sh.smem, s, c, p.max_elems, part_p, part_v, counters,
                            p.wait_ns);
}

}  // namespace agb
