// PNCG iterations of a small or medium mesh in one cooperative launch.
//
// A mesh of a few hundred tiles has too little work per pass to cover the
// fixed costs of the three-kernel iteration (solver.cu): a launch, a drain, a
// completion counter and a one-thread scalar tail per pass.  Here every tile
// stays on one resident CTA for the whole run, three grid barriers separate
// the passes, and all CTAs sum the partials and take the scalar decisions
// themselves (the same numbers in the same order, so they agree bit for bit;
// one CTA deciding and publishing took 2 us more per decision):
//
//   direction   the CTA's tile vertices read (g, d), form p = -P g + beta
//               p_prev; per element p^T H_e p and the line-search polynomial
//   -- barrier: sums, alpha_0, Armijo step t --
//   gradient    x <- x + t p; forces and clamped diagonal -> slots
//   -- barrier --
//   vertex      one of the tiles that hold a vertex sums its slots, writes
//               (g, d) and adds the 12 dot products
//   -- barrier: sums, beta, preconditioner mean, termination --
//
// Every tile keeps x (hi + lo), p, x_ref and the previous g of its vertices in
// shared memory between iterations and updates x and p itself (each tile that
// holds a vertex computes the same values); only (g, d), the slots and the
// partials pass through L2.  The run ends at the iteration limit, at
// termination or when a reference-state refresh is due; the vertex state and
// SolverState are then written back, so a run cut into pieces continues bit
// for bit.
//
// Measured (40 iterations with the reset and the refreshes): 5,000-tet cube in
// FP32 807 us against 1,371 with the three-kernel loop, 138,240 tets 1,139
// against 1,968; 20 iterations of 138,240 tets in FP64 3,955 against 7,303.
// An iteration of the cube takes 15.7 us, of which the three barriers are 4,
// the element groups 3, the sums 1.3 and the two decisions 2.5.
#include <math.h>

#include <algorithm>

#include "gridsync.cuh"
#include "resident.cuh"
#include "solver.h"
#include "solver_common.cuh"

namespace agb {

namespace {

constexpr int kStateWords = (int)(sizeof(SolverState) / 4);

// per-vertex words kept between iterations: x hi, x lo, p, previous g, mask,
// and with the reference-state correction x_ref
template <bool DELTA>
constexpr int kVertexWords = DELTA ? 16 : 13;

// the accumulators' space also takes the block sums' rows (13 per thread)
template <class R, bool DELTA>
constexpr size_t resident_smem(int nw) {
  return (size_t)kTileVerts *
         ((size_t)(nw + 1) * (sizeof(V4<R>) + sizeof(V2<R>)) + kVertexWords<DELTA> * sizeof(R) + 4 * sizeof(int));
}

// REC: the tile's element records stay in shared memory after the first read;
// otherwise each group's records are loaded one group ahead.
//
// SHARE: how tiles share an SM.  kTwoCtas, FP32: two CTAs of a tile each, which
// run apart between the barriers (as halves of one CTA 108k tets took 1,117
// against 1,086 us, 138k 1,158 against 1,144).  kTwoTiles, FP64 with more tiles
// than SMs: the halves of one CTA hold a tile each, paired by their size.  The
// SM has one FP64 pipe (19 cycles per warp instruction from four warps on), and
// the CTA takes the grid's sums and the decisions once: with the vertex sums
// packed (below) 138k tets 4,153 -> 3,955 us for 20 iterations, 80k 5,910 ->
// 5,297 for 40.  kAlone, FP64 with at most a tile per SM.
enum Share { kAlone, kTwoCtas, kTwoTiles };

template <class R, int MAT, bool DELTA, int NW, bool REC, Share SHARE>
__global__ void __launch_bounds__(32 * NW * (SHARE == kTwoTiles ? 2 : 1), SHARE == kTwoCtas ? 2 : 1)
    solver_resident_kernel(SolveArgs a, int max_elems, int tile_smem, int whole, const int32_t* __restrict__ order,
                           void* part_d, void* part_v, unsigned* counters, uint64_t wait_ns) {
  constexpr int T = 32 * NW, ND = 6, NVT = 12, kSlotBatch = 4;  // T threads per tile
  constexpr int TILES = SHARE == kTwoTiles ? 2 : 1, TC = T * TILES;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int half = TILES == 2 ? (int)threadIdx.x / T : 0;
  V4<R>* s4 = reinterpret_cast<V4<R>*>(smem_raw + (size_t)half * tile_smem);  // staging
  V4<R>* acc4 = s4 + kTileVerts;                            // [warp][vertex]: gx gy gz dx
  V2<R>* s2 = reinterpret_cast<V2<R>*>(acc4 + NW * kTileVerts);
  V2<R>* acc2 = s2 + kTileVerts;                            // [warp][vertex]: dy dz
  R* vw = reinterpret_cast<R*>(acc2 + NW * kTileVerts);     // kept vertex words, [word][vertex]
  int* vi = reinterpret_cast<int*>(vw + kVertexWords<DELTA> * kTileVerts);  // vertex, slot, first and end slot
  float4* srec = reinterpret_cast<float4*>(vi + 4 * kTileVerts);  // REC: [stream][element]
  int* sgrp = reinterpret_cast<int*>(srec + (size_t)kRecStreams<MAT> * max_elems);  // REC: group starts
  // the block sums' terms, in the first tile's accumulators while no accumulation runs
  R* const rows = reinterpret_cast<R*>(reinterpret_cast<V4<R>*>(smem_raw) + kTileVerts);
  static_assert(NW * kTileVerts * sizeof(V4<R>) >= (NVT + 1) * TC * sizeof(R), "rows fit the accumulators");
  __shared__ Acc<R> tot[NVT];
  __shared__ SolverState sst;
  __shared__ uint8_t s_own[TILES][kTileVerts];  // the tile vertices that this tile sums
  __shared__ int s_owned[TILES][NW];
  uint8_t* const own = s_own[half];
  R* const xh = vw;
  R* const xl = vw + 3 * kTileVerts;
  R* const vp = vw + 6 * kTileVerts;
  R* const vg = vw + 9 * kTileVerts;
  R* const vmask = vw + 12 * kTileVerts;
  R* const xr = vw + 13 * kTileVerts;  // DELTA only

  if (a.st->done) return;
  const int tid = (int)threadIdx.x - half * T, warp = tid >> 5, lane = tid & 31;  // within the tile's threads
  int tile = blockIdx.x;
  if constexpr (SHARE == kTwoCtas) {
    __shared__ int s_tile;
    if (whole > 0) {
      if (threadIdx.x == 0) s_tile = place_cta(counters, whole, gridDim.x);
      __syncthreads();
      tile = s_tile;
    }
  } else if constexpr (SHARE == kTwoTiles) {
    tile = order[2 * blockIdx.x + half];  // -1: the half takes part in the CTA's sums and barriers only
  }
  const int gs = tile < 0 ? 0 : a.fv.tile_gstart[tile], ge = tile < 0 ? 0 : a.fv.tile_gstart[tile + 1];
  const int vs = tile < 0 ? 0 : a.fv.tile_vstart[tile], nv = tile < 0 ? 0 : a.fv.tile_vstart[tile + 1] - vs;
  const int me = SHARE == kTwoCtas ? tile : (int)blockIdx.x;  // the place of the CTA's partials
  GridBar bar{counters, kResidentCounters, wait_ns, gridDim.x, 0, false};
  if (threadIdx.x < kStateWords) ((uint32_t*)&sst)[threadIdx.x] = ((const uint32_t*)a.st)[threadIdx.x];
  __syncthreads();
  const V4<R>* XA = (const V4<R>*)a.xa;
  V4<R>* GD = (V4<R>*)a.gd;
  V4<R>* slots = (V4<R>*)a.slots;
  {
    const V4<R>* P = p_prev<R>(a, sst.pbuf);
    for (int i = tid; i < nv; i += T) {
      const int v = a.fv.tv_vid[vs + i], sl = a.slot_of_tv[vs + i];
      const int s0 = a.off[v], s1 = a.off[v + 1];
      vi[i] = v;
      vi[kTileVerts + i] = sl;
      // one of the tiles that hold a vertex owns it, spread over its slots
      vi[2 * kTileVerts + i] = s0;
      vi[3 * kTileVerts + i] = sl == s0 + v % (s1 - s0) ? s1 : s0;
      const V4<R> x = XA[2 * v], l = XA[2 * v + 1], p = P[v];
      xh[i] = x.x;
      xh[kTileVerts + i] = x.y;
      xh[2 * kTileVerts + i] = x.z;
      vmask[i] = x.w;
      xl[i] = l.x;
      xl[kTileVerts + i] = l.y;
      xl[2 * kTileVerts + i] = l.z;
      vp[i] = p.x;
      vp[kTileVerts + i] = p.y;
      vp[2 * kTileVerts + i] = p.z;
      if constexpr (DELTA) {
        const V4<R> r = ((const V4<R>*)a.xref)[v];
        xr[i] = r.x;
        xr[kTileVerts + i] = r.y;
        xr[2 * kTileVerts + i] = r.z;
      }
    }
  }
  // FP64 sums its vertices without the gaps that other tiles' ones leave in the
  // warps (FP32 takes a tile's vertices in one turn anyhow)
  constexpr bool PACK = sizeof(R) == 8;
  int n_own = PACK ? 0 : nv;
  for (int i0 = 0; PACK && i0 < kTileVerts; i0 += T) {  // both halves take every turn
    const int i = i0 + tid;
    const bool mine = i < nv && vi[2 * kTileVerts + i] != vi[3 * kTileVerts + i];  // this thread's own stores
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (lane == 0) s_owned[half][warp] = __popc(m);
    __syncthreads();
    int k = n_own + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < NW; ++w) {
      if (w < warp) k += s_owned[half][w];
      n_own += s_owned[half][w];
    }
    if (mine) own[k] = (uint8_t)i;
    __syncthreads();
  }
  if (REC && tile >= 0) keep_records<MAT>(a.fv, tile, max_elems, srec, sgrp, tid, T);
  const GroupLoader<R, MAT, REC> load_group{a.fv, gs, max_elems, srec, sgrp};
  // The accumulators are cleared while a barrier is waited for: those that
  // the block sums' rows overlay after the direction pass, the others after
  // the vertex pass.
  constexpr int kRowCopies = (int)(((NVT + 1) * TC * sizeof(R) + kTileVerts * sizeof(V4<R>) - 1) /
                                   (kTileVerts * sizeof(V4<R>)));
  auto zero4 = [&](int w) {
    for (int i = tid; i < nv; i += T) acc4[w * kTileVerts + i] = V4<R>{R(0), R(0), R(0), R(0)};
  };
  auto zero_rest = [&]() {
    for (int w = kRowCopies; w < NW; ++w) zero4(w);
    for (int w = 0; w < NW; ++w)
      for (int i = tid; i < nv; i += T) acc2[w * kTileVerts + i] = V2<R>{R(0), R(0)};
  };
  zero_rest();
  __syncthreads();  // every thread has read sst.pbuf; records and groups are in place
  if (threadIdx.x == 0) sst.refresh = 0;  // the refresh passes, if any, ran after the last vertex pass

  bool ok = true;
  for (;;) {
    // ---- direction ----
    __syncthreads();
    {
      const R beta = to_real<R>(sst.beta), inv_mean = to_real<R>(sst.inv_mean);
      for (int i = tid; i < nv; i += T) {
        const int v = vi[i];
        const V4<R> g = ldcg4(GD + 2 * v), d = ldcg4(GD + 2 * v + 1);
        const V4<R> po{vp[i], vp[kTileVerts + i], vp[2 * kTileVerts + i], R(0)};
        R p[3];
        pdir(g, d, po, beta, inv_mean, p);
        vg[i] = g.x;
        vg[kTileVerts + i] = g.y;
        vg[2 * kTileVerts + i] = g.z;
        vp[i] = p[0];
        vp[kTileVerts + i] = p[1];
        vp[2 * kTileVerts + i] = p[2];
        s4[i] = V4<R>{xh[i], xh[kTileVerts + i], xh[2 * kTileVerts + i], p[0]};
        s2[i] = V2<R>{p[1], p[2]};
      }
    }
    int g = gs + warp, n = 0;
    ElemGeo<R> geo;
    uint32_t ids = 0;
    if (!REC && g < ge) load_group(g, n, geo, ids);
    __syncthreads();
    {
      R plain[ND] = {};
      Acc<R> c2acc = {};
      while (g < ge) {
        const int gn = g + NW;
        int nn = 0;
        ElemGeo<R> geon;
        uint32_t idsn = 0;
        if constexpr (REC)
          load_group(g, n, geo, ids);
        else if (gn < ge)
          load_group(gn, nn, geon, idsn);
        if (lane < n) {
          const int l[4] = {corner(ids, 0), corner(ids, 1), corner(ids, 2), corner(ids, 3)};
          R G[3][3], dF[3][3];
          dir_gradients(s4, s2, l, geo.D, G, dF);
          add_act<MAT>(geo, G);
          SnhPoint<R> s;
          snh_prepare(G, s);
          SnhDir<R> d;
          snh_dir(s, dF, d);
          plain[0] += clamp0(snh_hess_quad(s, d, geo.mu, geo.lam));
          R c[5];
          snh_poly(s, d, geo.mu, geo.lam, c);
          c2acc.add(c[0]);
#pragma unroll
          for (int m = 1; m < 5; ++m) plain[1 + m] += c[m];
        }
        g = gn;
        if constexpr (!REC) {
          n = nn;
          geo = geon;
          ids = idsn;
        }
      }
      R lo = R(0);
      if constexpr (sizeof(R) == 4) {
        plain[1] = c2acc.hi;
        lo = c2acc.lo;
      } else {
        plain[1] = c2acc.v;
      }
      cta_partials<ND, sizeof(R) == 4 ? 1 : -1, TC, R>(plain, lo, rows, (AccStore<R>*)part_d, gridDim.x, me);
    }
    bar.arrive();
    for (int w = 0; w < kRowCopies; ++w) zero4(w);
    if (!(ok = bar.wait())) break;
    // the gradient pass's first record, in flight during the decision
    g = gs + warp;
    n = 0;
    if (!REC && g < ge) load_group(g, n, geo, ids);
    grid_totals<ND, TC, R>((const AccStore<R>*)part_d, gridDim.x, tot);
    if (threadIdx.x < 32) dir_decide<MAT, R>(&sst, tot);
    __syncthreads();
    const R t = to_real<R>(sst.t);

    // ---- gradient at x + t p ----
    {
      for (int i = tid; i < nv; i += T) {
        R h[3], l[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          h[c] = xh[c * kTileVerts + i];
          l[c] = xl[c * kTileVerts + i];
          pair_add(h[c], l[c], mul_rn(t, vp[c * kTileVerts + i]));
          xh[c * kTileVerts + i] = h[c];
          xl[c * kTileVerts + i] = l[c];
        }
        if constexpr (DELTA) {
          const R r[3] = {xr[i], xr[kTileVerts + i], xr[2 * kTileVerts + i]};
          s4[i] = V4<R>{r[0], r[1], r[2], add_rn(sub_rn(h[0], r[0]), l[0])};
          s2[i] = V2<R>{add_rn(sub_rn(h[1], r[1]), l[1]), add_rn(sub_rn(h[2], r[2]), l[2])};
        } else {
          s4[i] = V4<R>{h[0], h[1], h[2], l[0]};
          s2[i] = V2<R>{l[1], l[2]};
        }
      }
    }
    __syncthreads();
    {
      V4<R>* my4 = acc4 + warp * kTileVerts;
      V2<R>* my2 = acc2 + warp * kTileVerts;
      while (g < ge) {
        const int gn = g + NW;
        int nn = 0;
        ElemGeo<R> geon;
        uint32_t idsn = 0;
        if constexpr (REC)
          load_group(g, n, geo, ids);
        else if (gn < ge)
          load_group(gn, nn, geon, idsn);
        const int l[4] = {corner(ids, 0), corner(ids, 1), corner(ids, 2), corner(ids, 3)};
        R f[4][3], hd[4][3];
        if (lane < n) {
          R G[3][3], P[3][3];
          if constexpr (DELTA) {
            R dG[3][3];
            delta_gradient(s4, s2, l, geo.D, G, dG);
            add_act<MAT>(geo, G);
            SnhPoint<R> s, sn;
            snh_prepare(G, s);
            snh_pk1_delta(s, dG, geo.mu, geo.lam, P, sn);
            corner_vjp(P, geo.D, f);
            snh_hess_diag(sn, geo.D, geo.mu, geo.lam, hd);
          } else {
            pair_gradient(s4, s2, l, geo.D, G);
            add_act<MAT>(geo, G);
            SnhPoint<R> s;
            snh_prepare(G, s);
            snh_pk1(s, geo.mu, geo.lam, P);
            corner_vjp(P, geo.D, f);
            snh_hess_diag(s, geo.D, geo.mu, geo.lam, hd);
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          __syncwarp();
          if (lane < n) {
            const int v = l[k];
            V4<R> q4 = my4[v];
            V2<R> q2 = my2[v];
            q4.x += f[k][0];
            q4.y += f[k][1];
            q4.z += f[k][2];
            q4.w += clamp0(hd[k][0]);
            q2.x += clamp0(hd[k][1]);
            q2.y += clamp0(hd[k][2]);
            my4[v] = q4;
            my2[v] = q2;
          }
        }
        __syncwarp();
        g = gn;
        if constexpr (!REC) {
          n = nn;
          geo = geon;
          ids = idsn;
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < nv; i += T) {
      V4<R> q4 = acc4[i];
      V2<R> q2 = acc2[i];
#pragma unroll
      for (int w = 1; w < NW; ++w) {
        const V4<R> r4 = acc4[w * kTileVerts + i];
        const V2<R> r2 = acc2[w * kTileVerts + i];
        q4.x += r4.x;
        q4.y += r4.y;
        q4.z += r4.z;
        q4.w += r4.w;
        q2.x += r2.x;
        q2.y += r2.y;
      }
      const size_t sl = 2 * (size_t)vi[kTileVerts + i];
      slots[sl] = V4<R>{q4.x, q4.y, q4.z, R(0)};
      slots[sl + 1] = V4<R>{q4.w, q2.x, q2.y, R(0)};
    }
    bar.arrive();
    if (!(ok = bar.wait())) break;

    // ---- vertex ----
    {
      R s[NVT] = {};
      for (int k = tid; k < n_own; k += T) {
        const int i = PACK ? own[k] : k, s0 = vi[2 * kTileVerts + i], s1 = vi[3 * kTileVerts + i];
        if (s0 == s1) continue;  // another tile's vertex
        const int v = vi[i];
        V4<R> r{}, f{};
        if constexpr (DELTA) r = ldg4((const V4<R>*)a.gref + v);
        if (a.force) f = ldg4((const V4<R>*)a.force + v);
        R ss[3] = {R(0), R(0), R(0)}, ds[3] = {R(0), R(0), R(0)};
        for (int b = s0; b < s1; b += kSlotBatch) {  // a batch of slots in flight together
          V4<R> sg[kSlotBatch], sd[kSlotBatch];
#pragma unroll
          for (int q = 0; q < kSlotBatch; ++q)
            if (b + q < s1) {
              sg[q] = ldcg4(slots + 2 * (size_t)(b + q));
              sd[q] = ldcg4(slots + 2 * (size_t)(b + q) + 1);
            }
#pragma unroll
          for (int q = 0; q < kSlotBatch; ++q)
            if (b + q < s1) {
              ss[0] += sg[q].x;
              ss[1] += sg[q].y;
              ss[2] += sg[q].z;
              ds[0] += sd[q].x;
              ds[1] += sd[q].y;
              ds[2] += sd[q].z;
            }
        }
        R xn[3], p[3], gn[3], dn[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xn[c] = xh[c * kTileVerts + i] + xl[c * kTileVerts + i];
          p[c] = vp[c * kTileVerts + i];
        }
        const V4<R> go{vg[i], vg[kTileVerts + i], vg[2 * kTileVerts + i], R(0)};
        vertex_terms<R, DELTA>(a.force != nullptr, (int)vmask[i], xn, p, go, r, f, ss, ds, gn, dn, s);
        GD[2 * v] = V4<R>{gn[0], gn[1], gn[2], R(0)};
        GD[2 * v + 1] = V4<R>{dn[0], dn[1], dn[2], R(0)};
      }
      cta_partials<NVT, -1, TC, R>(s, R(0), rows, (AccStore<R>*)part_v, gridDim.x, me);
    }
    bar.arrive();
    zero_rest();
    if (!(ok = bar.wait())) break;
    grid_totals<NVT, TC, R>((const AccStore<R>*)part_v, gridDim.x, tot);
    vertex_decide<R>(&sst, tot);
    __syncthreads();
    if (sst.done || sst.iter >= sst.iter_limit || sst.refresh) break;
  }

  if (ok) {
    V4<R>* X = (V4<R>*)a.xa;
    V4<R>* P = p_prev<R>(a, sst.pbuf);  // the last direction, flipped to p_prev by the decision
    if (tile == 0 && tid < kStateWords) ((uint32_t*)a.st)[tid] = ((const uint32_t*)&sst)[tid];
    for (int i = tid; i < nv; i += T) {
      if (vi[2 * kTileVerts + i] == vi[3 * kTileVerts + i]) continue;
      const int v = vi[i];
      X[2 * v] = V4<R>{xh[i], xh[kTileVerts + i], xh[2 * kTileVerts + i], vmask[i]};
      X[2 * v + 1] = V4<R>{xl[i], xl[kTileVerts + i], xl[2 * kTileVerts + i], R(0)};
      P[v] = V4<R>{vp[i], vp[kTileVerts + i], vp[2 * kTileVerts + i], R(0)};
    }
  }
  if (bar.leave()) {  // a barrier gave up: the solve stops with a device error
    a.st->error = 3;
    a.st->done = 1;
  }
}

using ResidentKernel = void (*)(SolveArgs, int, int, int, const int32_t*, void*, void*, unsigned*, uint64_t);

struct Shape {
  ResidentKernel kernel;
  int blocks, threads;
  size_t smem;
  int tile_smem;
};

template <class R, int MAT, bool DELTA, int NW, bool REC>
Shape shape(const ResidentPlan& p, int n_tiles) {
  size_t smem = resident_smem<R, DELTA>(NW);
  if (REC) smem += records_bytes<MAT>(p);
  smem = (smem + 15) & ~(size_t)15;
  if constexpr (sizeof(R) == 4) {
    return Shape{solver_resident_kernel<R, MAT, DELTA, NW, REC, kTwoCtas>, n_tiles, 32 * NW, smem, 0};
  } else if (n_tiles > p.sms) {
    return Shape{solver_resident_kernel<R, MAT, DELTA, NW, REC, kTwoTiles>, p.sms, 64 * NW, 2 * smem, (int)smem};
  } else {
    // more shared memory than half an SM's: no two CTAs share an SM while others idle
    return Shape{solver_resident_kernel<R, MAT, DELTA, NW, REC, kAlone>, n_tiles, 32 * NW,
                 std::max(smem, (size_t)120 * 1024), 0};
  }
}

template <int MAT, bool DELTA>
Shape shape_f32(const ResidentPlan& p, int nt) {
  constexpr int W = kResidentWarps<float>;
  return p.shape == 1 ? shape<float, MAT, DELTA, W, true>(p, nt) : shape<float, MAT, DELTA, W, false>(p, nt);
}

Shape shape_of(const SolveArgs& a, const ResidentPlan& p) {
  constexpr int SNH = AGB_STABLE_NEO_HOOKEAN, MU = AGB_STABLE_NEO_HOOKEAN_MUSCLE;
  const bool mu = a.fv.material == MU;
  const int nt = a.fv.n_tiles;
  if (a.precision == AGB_F64)
    return mu ? shape<double, MU, false, kResidentWarps<double>, false>(p, nt)
              : shape<double, SNH, false, kResidentWarps<double>, false>(p, nt);
  if (a.delta) return mu ? shape_f32<MU, true>(p, nt) : shape_f32<SNH, true>(p, nt);
  return mu ? shape_f32<MU, false>(p, nt) : shape_f32<SNH, false>(p, nt);
}

}  // namespace

// Above two tiles per SM the three-kernel iteration is the faster one: with
// four 4-warp CTAs per SM this kernel took 2.46 against 2.23 ms on 245,760 tets
// (376 tiles) and 2.88 against 2.55 ms on 400,000 (592 tiles), for 40
// iterations and the reset.
cudaError_t resident_prepare(const SolveArgs& a, ResidentPlan* p) {
  p->shape = 0;
  if (!snh_family(a.fv.material)) return cudaSuccess;
  return choose_shape(a, p, [&](const ResidentPlan& q) { return shape_of(a, q); });
}

cudaError_t launch_resident(const SolveArgs& a, const ResidentPlan& p, void* part_d, void* part_v, unsigned* counters,
                            cudaStream_t s) {
  if (!p.shape) return cudaErrorInvalidValue;
  const Shape sh = shape_of(a, p);
  return launch_cooperative(sh.kernel, sh.blocks, sh.threads, sh.smem, s, a, p.max_elems, sh.tile_smem, p.whole,
                            p.order, part_d, part_v, counters, p.wait_ns);
}

}  // namespace agb
