// stage_cns.cuh -- the compressible Navier-Stokes stage on Morton tiles staged
// into shared memory, and its launches (host tables: h3c_stage_cns.cu).
//
// hom3's CNS flux is AUSM plus a three-point viscous flux
// (src/solver/fv/cns/physics.hpp:155-161, 305-338) whose transverse
// derivatives average the central slopes of the two face cells
// (surface_slope / slope, src/solver/fv/solver.hpp:596-678).  The per-cell
// kernel evaluates every face twice and reads slopes that a separate pass
// wrote for every cell.  Here a block owns a 256-cell tile at a time:
//
//  1. copies (as in h3c_stage_halo.cu): the tile's state and neighbour slots
//     by cp.async.bulk, the halo cells' state by cp.async: the first layer
//     (the tile's face neighbours) and the second (the cells the first
//     layer's slopes read: edge-diagonal neighbours of the tile);
//  2. primitive variables and slopes of the tile and first-layer cells,
//     computed once into shared memory (a ghost's slopes -- its boundary or
//     periodic partner cell's, with the walls' sign rule -- from a ghost-only
//     slope pass run before the stage);
//  3. fluxes direction by direction, each face once (the plus face is
//     published for the neighbour's minus face, as in the Euler tile kernel);
//     every face is the same F(l, r) evaluation and each cell sums
//     F(minus) - F(plus) in hom3's order, so the results are bit-identical to
//     the per-cell kernel;
//  4. the update and the fused CFL minimum.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#define H3C_DEVICE_FUNCTIONS_ONLY
#include "fv_kernels.cuh"
#include "stage_cns.hpp"
#include "async_copy.cuh"
#include "launch.hpp"

namespace h3c {

// Slopes of the ghost cells: the ghost branch of k_slopes (a ghost takes its
// boundary cell's central slope, a periodic ghost its partner's, with the
// walls' sign flip of tangential velocity slopes: boundary_condition.hpp:63-67,
// cns/boundary_conditions.hpp:143-147, 230-234), same arithmetic.
template <int ND>
__global__ void __launch_bounds__(kBlock) k_ghost_slopes(const double* q, Geometry g, GhostTables gt,
                                                         double* __restrict__ gsl, long long ngl) {
  constexpr int NV = ND + 2;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ld = g.ld;
  int b = -1, dg = 0, wall = 0, nb[2 * ND];
  if (i < gt.ng) {
    const BcParam& B = gt.bcs[load_here(gt.bc_own + i)];
    wall = load_here(&B.wall);
    dg = load_here(gt.pos + i) >> 1;
    b = load_here(&B.kind) == BC_PERIODIC ? load_here(gt.partner + i) : load_here(gt.bndry + i);
    if (b >= 0) {
#pragma unroll
      for (int p = 0; p < 2 * ND; ++p) nb[p] = load_here(g.nbr + p * ld + b);
    }
  }
  chain_begin();
  if (b < 0) return;
  const double h2 = 2. * g.len[g.lvl[b]];
#pragma unroll
  for (int sd = 0; sd < ND; ++sd) {
    const int m = nb[2 * sd], p = nb[2 * sd + 1];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      double s = (q[v * ld + p] - q[v * ld + m]) / h2;
      if (wall && v < ND && sd != dg) s = -s;
      gsl[(sd * NV + v) * ngl + i] = s;
    }
  }
}

#ifndef H3C_CNS_MINB
#define H3C_CNS_MINB 2  // blocks per SM the CNS tile kernel is register-budgeted for
#endif

// AUSM (euler/physics.hpp:276-293) with the splits' supersonic branches off
// the common path: the same values as ausm (fv_kernels.cuh).  The brick
// variant takes it; the general one was not measured with it and keeps ausm.
template <class R, int ND>
__device__ __forceinline__ void ausm_subsonic_first(const Prim<R, ND>& L, const Prim<R, ND>& Rt, int d, R* f) {
  const R ML = L.M[d], MR = Rt.M[d];
  const R tl = (ML + R(1)) * (ML + R(1)), tr = (MR + R(-1)) * (MR + R(-1));
  R mi = R(0.25) * tl + R(-0.25) * tr;
  R pl = (R(0.25) * tl) * (R(2) - ML), pr = (R(0.25) * tr) * (R(2) + MR);
  if (beyond_one(ML) || beyond_one(MR)) {
    mi = m_int<R>(R(1), ML) + m_int<R>(R(-1), MR);
    pl = p_int<R>(R(1), ML);
    pr = p_int<R>(R(-1), MR);
  }
  const R pi = pl * L.p + pr * Rt.p;
  const bool left = mi >= R(0);
  const R a = left ? L.a : Rt.a;
#pragma unroll
  for (int v = 0; v < ND + 1; ++v) f[v] = ((left ? L.q[v] : Rt.q[v]) * a) * mi;
  f[ND + 1] = (((left ? L.q[ND + 1] + L.p : Rt.q[ND + 1] + Rt.p)) * a) * mi;
#pragma unroll
  for (int v = 0; v < ND; ++v)
    if (v == d) f[v] = f[v] + pi;
}

// cell_dt of CNS (fv_kernels.cuh) over a warp's cells: per lane a value whose
// minimum over the warp is the cells' minimum, to the bit.  On one level the
// convective part falls as the wave speed grows, division by division, so the
// warp's least is that of its largest wave speed; and the viscous part, three
// divisions and a square root more, is left out where it cannot be the
// smaller one for any cell: an estimate by reciprocals (within a few ulp,
// against a margin of 1e-9) of the warp's largest decides.  A cell that is no
// physical state, or has no wave speed or estimate, sends its warp to cell_dt
// in every cell (a NaN state's time step lies below zero, and a maximum drops
// it).  128^3 Taylor-Green, second RK2 stage: 347.6 us with both parts in
// every cell; 336.8 without cell_dt as the other branch, 1% more with it.
template <int ND>
__device__ __forceinline__ long long cns_warp_dt(const double* q, bool live, double h, const PhysConst& pc, bool& bad) {
  Prim<double, ND> P;
  const double kInf = __longlong_as_double(0x7ff0000000000000LL);
  double S = -1.7976931348623157e308, est = S;
  if (live) {
#pragma unroll
    for (int v = 0; v < ND + 2; ++v) P.q[v] = q[v];
    make_prim<double, ND>(P, pc.gamma, pc.gm1);
    bad = !(P.q[ND] > 0.0 && P.q[ND + 1] > 0.0 && P.p > 0.0);
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const double cand = fabs(P.u[d]) + P.a;
      S = (S < cand) ? cand : S;
    }
    const double rinv = nr_rcp(P.q[ND]);
    const double T = pc.gamma * P.p * rinv;
    est = (T * (T * nr_rsqrt(T))) * pc.sOverTrefP1 * nr_rcp(T + pc.sOverTref) * rinv;
    if (bad || !(S > 0.0) || !(est > 0.0)) est = kInf;  // cell_dt decides
  }
  for (int w = 16; w > 0; w >>= 1) {
    S = fmax(S, __shfl_xor_sync(0xffffffffu, S, w));
    est = fmax(est, __shfl_xor_sync(0xffffffffu, est, w));
  }
  // dt_v = cflv h / (2 S_visc), S_visc = coeff max(1 / Re0, 1 / (Re0 Pr0 gm1)), coeff = est / h
  const double worst = est * fmax(1.0, nr_rcp(pc.Pr0 * pc.gm1)) * nr_rcp(pc.Re0 * h);
  const bool convective = S > 0.0 && pc.cflv * S > (2.0 + 1e-9) * pc.cfl * worst;  // the same in every lane
  if (!convective && !live) return kOrdMax;
  const double dt = convective ? pc.cfl * h / S : cell_dt<ND, CNS>(q, h, pc);
  return isnan(dt) ? kOrdMax : dbl_to_ord(dt);
}

// BRICK: constant row strides, and the minus faces on the tile's border come
// from its list, evaluated before the direction loop by whole warps and
// handed over through shared memory.  Left to their cells they are a sixth of
// the tile's face evaluations, but in divergent branches of half the warps
// and directions: 12 of a tile's 36 warp-wide evaluations, against 4 of 28.
template <int ND, class R, int MODE, bool FUSE, bool BRICK>
__global__ void __launch_bounds__(kHaloTile, H3C_CNS_MINB)
    k_stage_cns_halo(const double* qin, double* out, Geometry g, CnsHaloGeom ch, PhysConst pc,
                     const Scalars* sc, long long* dtmin, int* status) {
  constexpr int NV = ND + 2, NP = 2 * ND, TB = kHaloTile;
  constexpr int NPR = NV + ND + 2;  // q[nv], M[nd], p, a
  constexpr int SV = kCnsSlopeVars<ND>;
  constexpr int NSL = ND * SV;      // slopes [sd][v], v <= nd
  constexpr int KH = kHaloMaxSlots / kHaloTile;
  constexpr bool LIP = cns_land_in_prims<R, ND>();
  const HaloGeom& hg = ch.h;
  constexpr int NB = kCnsBorder<ND>;
  const int S1 = BRICK ? TB + kCnsBrickH1<ND> : TB + ch.h1max;
  const int S = TB + hg.hmax, S2 = S - TB - ch.h1max;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem);
  double* fx = reinterpret_cast<double*>(smem + 16);                              // [NV][TB]
  R* pr = reinterpret_cast<R*>(fx + NV * TB);                                     // [NPR][S1]
  R* sl = pr + (size_t)NPR * S1;                                                  // [NSL][S1]
  R* bm = sl + (size_t)NSL * S1;                                                  // [NV][NB]
  double* land = reinterpret_cast<double*>(bm + (BRICK ? NV * NB : 0));           // FP32: [NV][S]
  double* land2 = land;                                                           // FP64: [NV][S2]
  unsigned short* ln = reinterpret_cast<unsigned short*>(land + (LIP ? (size_t)NV * S2 : (size_t)NV * S));  // [2][NP][TB]
  const int tid = threadIdx.x;
  const long long ld = g.ld;
  const R gamma = (R)pc.gamma, gm1 = (R)pc.gm1;
  const double h = g.len[0];  // single-level grid
  const double h2 = 2. * h;
  const R hr = (R)h;

  // where the state of slot s (tile, first or second layer) lands
  auto qslot = [&](int v, int s) -> double* {
    if (LIP) return s < S1 ? reinterpret_cast<double*>(pr) + v * S1 + s : land2 + (size_t)v * S2 + (s - S1);
    return land + (size_t)v * S + s;
  };

  long long tile = blockIdx.x;
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncthreads();

  // halo cells (layer 1 then layer 2) of tile t this thread copies
  auto fetch_ids = [&](long long t, int* hid, int& o0, int& nh1) -> int {
    o0 = load_here(hg.halo_off + t);
    const int nh = load_here(hg.halo_off + t + 1) - o0;
    nh1 = load_here(ch.h1end + t) - o0;
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      const int hh = tid + k * TB;
      hid[k] = hh < nh ? load_here(hg.halo_ids + o0 + hh) : 0;
    }
    return nh;
  };
  auto issue = [&](long long t, int buf, const int* hid, int nh) {
    if (tid == 0) {
      const long long c0 = t * TB;
      const long long te = min(c0 + TB, instance_end(g, tile_instance(g, t)));
      const unsigned ncp = (unsigned)((te - c0 + 15) & ~15LL);
      fence_proxy_async();
      mbar_expect_tx(bar, ncp * (8u * NV + 2u * NP));
#pragma unroll
      for (int v = 0; v < NV; ++v) bulk_g2s(qslot(v, 0), qin + v * ld + c0, ncp * 8u, bar);
#pragma unroll
      for (int p = 0; p < NP; ++p) bulk_g2s(ln + (buf * NP + p) * TB, hg.lnb + p * ld + c0, ncp * 2u, bar);
    }
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      const int hh = tid + k * TB;
      if (hh < nh) {
        const long long n = hid[k];
#pragma unroll
        for (int v = 0; v < NV; ++v) cp_async8(qslot(v, TB + hh), qin + v * ld + n);
      }
    }
    cp_async_commit();
  };
  // primitive variables of a state (make_prim, euler/physics.hpp:83-125) into slot s;
  // in FP64 the state rows already hold q
  auto store_prim = [&](const double* q, int s) {
    Prim<R, ND> P;
#pragma unroll
    for (int v = 0; v < NV; ++v) P.q[v] = (R)q[v];
    make_prim<R, ND>(P, gamma, gm1);
    if (!LIP) {
#pragma unroll
      for (int v = 0; v < NV; ++v) pr[v * S1 + s] = P.q[v];
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) pr[(NV + d) * S1 + s] = P.M[d];
    pr[(NV + ND) * S1 + s] = P.p;
    pr[(NV + ND + 1) * S1 + s] = P.a;
  };
  auto load_prim_s = [&](int s, int d, Prim<R, ND>& P) {
#pragma unroll
    for (int v = 0; v < NV; ++v) P.q[v] = pr[v * S1 + s];
#pragma unroll
    for (int e = 0; e < ND; ++e) P.M[e] = e == d ? pr[(NV + e) * S1 + s] : R(0);
#pragma unroll
    for (int e = 0; e < ND; ++e) P.u[e] = R(0);  // not read by the AUSM and viscous fluxes
    P.p = pr[(NV + ND) * S1 + s];
    P.a = pr[(NV + ND + 1) * S1 + s];
  };
  // the transverse slopes (sd != d, v <= nd) the viscous flux of direction d
  // reads, in the [sd][v] layout (v < nv) the viscous flux indexes
  auto load_slopes = [&](int s, int d, R* out_) {
#pragma unroll
    for (int sd = 0; sd < ND; ++sd)
#pragma unroll
      for (int v = 0; v < NV; ++v)
        out_[sd * NV + v] = (sd != d && v < SV) ? sl[(sd * SV + v) * S1 + s] : R(0);
  };
  // central slopes of slot s from its face-neighbour slots m, p along sd
  auto store_slopes = [&](int s, int sd, int m, int p) {
#pragma unroll
    for (int v = 0; v < SV; ++v) sl[(sd * SV + v) * S1 + s] = (R)((*qslot(v, p) - *qslot(v, m)) / h2);
  };
  // the face flux F(l, r): AUSM + three-point viscous (cns/physics.hpp:155-161)
  auto face = [&](const Prim<R, ND>& L, const Prim<R, ND>& Rt, const R* sL, const R* sR, int d, R* f) {
    if (BRICK) ausm_subsonic_first<R, ND>(L, Rt, d, f);
    else ausm<R, ND>(L, Rt, d, f);
    R fv[NV];
    viscous<R, ND>(L, Rt, sL, sR, d, hr, pc, fv);
#pragma unroll
    for (int v = 0; v < NV; ++v) f[v] = f[v] + fv[v];
  };

  int hid[KH];
  int o0 = 0, nh1 = 0, nh = 0;
  if (tile < g.ntiles) nh = fetch_ids(tile, hid, o0, nh1);
  chain_begin();
  const double k = sc->dt / h;  // single grids only
  if (tile >= g.ntiles) return;
  issue(tile, 0, hid, nh);

  for (int it = 0; tile < g.ntiles; tile += gridDim.x, ++it) {
    const int buf = LIP ? 0 : (it & 1);
    const long long next = tile + gridDim.x;
    const long long c0 = tile * TB, c = c0 + tid;
    const int inst = tile_instance(g, tile);
    const long long te = min(c0 + (long long)TB, instance_end(g, inst));
    const bool live = c < te;
    if (MODE != 0 && live) prefetch_row_l2<NV>(g.q0, ld, c);  // the start state, read at the update

    const bool ok = mbar_wait_bounded(bar, (unsigned)(it & 1));
    cp_async_wait_all();
    if (!__syncthreads_and(ok)) {
      if (tid == 0) {
        flag_timeout(sc, status);
        // the block keeps its shared memory while its copies may still land there, for a second bounded wait
        mbar_wait_bounded(bar, (unsigned)(it & 1));
      }
      return;
    }

    // ---- primitives and slopes of the own cell and the layer-1 cells ----
    const unsigned short* L = ln + buf * NP * TB;
    if (live) {
      double qc[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) qc[v] = *qslot(v, tid);
      store_prim(qc, tid);
#pragma unroll
      for (int sd = 0; sd < ND; ++sd) store_slopes(tid, sd, L[(2 * sd) * TB + tid], L[(2 * sd + 1) * TB + tid]);
    }
#pragma unroll
    for (int k = 0; k < KH; ++k) {
      const int hh = tid + k * TB;
      if (hh < nh1) {
        const int s = TB + hh;
        double qh[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) qh[v] = *qslot(v, s);
        store_prim(qh, s);
        const long long n = hid[k];
        if (n >= g.n_int) {  // a ghost: the ghost-slope pass
#pragma unroll
          for (int sd = 0; sd < ND; ++sd)
#pragma unroll
            for (int v = 0; v < SV; ++v)
              sl[(sd * SV + v) * S1 + s] = (R)ch.gsl[(sd * NV + v) * ch.ngl + (n - g.n_int)];
        } else {
#pragma unroll
          for (int sd = 0; sd < ND; ++sd) {
            const unsigned short m = __ldg(ch.hnb + (size_t)(o0 + hh) * NP + 2 * sd);
            const unsigned short p = __ldg(ch.hnb + (size_t)(o0 + hh) * NP + 2 * sd + 1);
            if (m != 0xffff) store_slopes(s, sd, m, p);
          }
        }
      }
    }
    const unsigned bsel = BRICK && live ? __ldg(ch.bsel + c) : 0;  // per direction 1 + this cell's place in the list
    unsigned entry = ~0u;
    if (BRICK && tid < NB) entry = __ldg(ch.blist + tile * NB + tid);
    __syncthreads();  // primitives and slopes complete

    int hid_n[KH], o0_n = 0, nh1_n = 0, nh_n = 0;
    if (!LIP) {  // FP32: the next tile lands in its own area while this one's fluxes run
      if (next < g.ntiles) {
        nh_n = fetch_ids(next, hid_n, o0_n, nh1_n);
        issue(next, buf ^ 1, hid_n, nh_n);
      }
    }

    // ---- bricks: the minus faces on the tile's border (a warp's entries share their direction) ----
    if (BRICK && entry != ~0u) {
      const int cs = entry & 0xff, m = (entry >> 8) & 0xfff, de = entry >> 20;
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        if (de != d) continue;
        Prim<R, ND> Pc, Pn;
        load_prim_s(cs, d, Pc);
        load_prim_s(m, d, Pn);
        R slc[ND * NV], sn[ND * NV];
        load_slopes(cs, d, slc);
        load_slopes(m, d, sn);
        R f[NV];
        face(Pn, Pc, sn, slc, d, f);
#pragma unroll
        for (int v = 0; v < NV; ++v) bm[v * NB + tid] = f[v];
      }
    }

    // ---- fluxes, direction by direction ----
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      if (live) {
        Prim<R, ND> Pc, Pn;
        load_prim_s(tid, d, Pc);
        const int p = L[(2 * d + 1) * TB + tid];
        load_prim_s(p, d, Pn);
        R slc[ND * NV], sn[ND * NV];
        load_slopes(tid, d, slc);
        load_slopes(p, d, sn);
        R f[NV];
        face(Pc, Pn, slc, sn, d, f);
#pragma unroll
        for (int v = 0; v < NV; ++v) fx[v * TB + tid] = (double)f[v];
      }
      __syncthreads();  // this direction's plus faces are published
      if (live) {
        const int m = L[(2 * d) * TB + tid];
        double fm[NV];
        if (BRICK) {
          const int b = (bsel >> (8 * d)) & 0xff;
#pragma unroll
          for (int v = 0; v < NV; ++v) fm[v] = b ? (double)bm[v * NB + b - 1] : fx[v * TB + m];
        } else if (m < TB && L[(2 * d + 1) * TB + m] == tid) {
#pragma unroll
          for (int v = 0; v < NV; ++v) fm[v] = fx[v * TB + m];
        } else {
          Prim<R, ND> Pc, Pn;
          load_prim_s(tid, d, Pc);
          load_prim_s(m, d, Pn);
          R slc[ND * NV], sn[ND * NV];
          load_slopes(tid, d, slc);
          load_slopes(m, d, sn);
          R f[NV];
          face(Pn, Pc, sn, slc, d, f);
#pragma unroll
          for (int v = 0; v < NV; ++v) fm[v] = (double)f[v];
        }
        // the own plus flux as published (a rounded value: no FMA with this sum, as in the per-cell kernel)
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] = acc[v] + (fm[v] - fx[v * TB + tid]);
      }
      __syncthreads();  // the next direction rewrites the plus faces
    }

    // ---- update and the next step's CFL minimum ----
    bool bad = false;
    double o[NV];
    if (live) {
      double qc[NV], qo[NV];  // FP32: the landing area already holds the next tile
#pragma unroll
      for (int v = 0; v < NV; ++v) qc[v] = LIP ? *qslot(v, tid) : qin[v * ld + c];
      if (MODE != 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) qo[v] = g.q0[v * ld + c];
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) o[v] = rk_combine<MODE>(MODE == 0 ? 0.0 : qo[v], qc[v], k * acc[v]);
#pragma unroll
      for (int v = 0; v < NV; ++v) out[v * ld + c] = o[v];
    }
    if (FUSE) {
      const long long ord = cns_warp_dt<ND>(o, live, h, pc, bad);
      flag_bad_state(bad, sc, inst);
      block_min_atomic(ord, dtmin);
    }
    if (LIP) {  // FP64: the next tile lands where this one's primitives were
      __syncthreads();
      if (next < g.ntiles) {
        nh = fetch_ids(next, hid, o0, nh1);
        issue(next, 0, hid, nh);
      }
    } else {
      nh = nh_n;
      o0 = o0_n;
      nh1 = nh1_n;
#pragma unroll
      for (int k = 0; k < KH; ++k) hid[k] = hid_n[k];
    }
  }
}

// ---------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------
namespace {

template <int ND, class R, int MODE, bool FUSE, bool BRICK>
int cprep_one(size_t smem) {
  auto k = k_stage_cns_halo<ND, R, MODE, FUSE, BRICK>;
  // the opt-in limit (less the kernel's static arrays), not this grid's size: several solvers
  // share the kernel and its attribute
  int dev = 0, optin = 0;
  cudaFuncAttributes fa{};
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
      cudaFuncGetAttributes(&fa, k) != cudaSuccess || (size_t)optin < smem + fa.sharedSizeBytes ||
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes) !=
          cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, kHaloTile, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return nb;
}
// the least over the variants the solver launches
template <int ND, class R, int MODE, bool BRICK>
int cprep_f(size_t smem) {
  return std::min(cprep_one<ND, R, MODE, false, BRICK>(smem), cprep_one<ND, R, MODE, true, BRICK>(smem));
}
template <int ND, class R, bool BRICK>
int cprep_m(unsigned modes, size_t smem) {
  int n = 1 << 30;
  if (modes & 1u) n = std::min(n, cprep_f<ND, R, 0, BRICK>(smem));
  if (modes & 4u) n = std::min(n, cprep_f<ND, R, 2, BRICK>(smem));
  if (modes & 8u) n = std::min(n, cprep_f<ND, R, 3, BRICK>(smem));
  if (modes & 16u) n = std::min(n, cprep_f<ND, R, 4, BRICK>(smem));
  return n;
}
template <int ND, class R>
int cprep(unsigned modes, size_t smem, bool brick) {
  return brick ? cprep_m<ND, R, true>(modes, smem) : cprep_m<ND, R, false>(modes, smem);
}

template <int ND, class R, int MODE, bool FUSE>
void claunch_b(const CnsLaunch& a) {
  const auto k = a.h.blist ? k_stage_cns_halo<ND, R, MODE, FUSE, true> : k_stage_cns_halo<ND, R, MODE, FUSE, false>;
  // Chained (launch.hpp) where blocks take few tiles: 64^3 FP32 1141 -> 1106 us per 10 steps.  On long runs of
  // tiles per block the early start is worth nothing, and blocks that find an SM still taken by the kernel
  // before finish last (128^3, 28 tiles per block: 3205 -> 3245 us per 4 steps).
  if (a.g.ntiles <= 8LL * a.grid)
    launch_chain(k, a.grid, kHaloTile, a.smem, a.st, a.qin, a.out, a.g, a.h, a.pc, a.sc, a.dtmin, a.status);
  else
    k<<<a.grid, kHaloTile, a.smem, a.st>>>(a.qin, a.out, a.g, a.h, a.pc, a.sc, a.dtmin, a.status);
}
template <int ND, class R, int MODE>
void claunch_f(bool fuse, const CnsLaunch& a) {
  if (fuse) claunch_b<ND, R, MODE, true>(a);
  else claunch_b<ND, R, MODE, false>(a);
}
template <int ND, class R>
void claunch_m(int mode, bool fuse, const CnsLaunch& a) {
  switch (mode) {
    case 0: claunch_f<ND, R, 0>(fuse, a); break;
    case 2: claunch_f<ND, R, 2>(fuse, a); break;
    case 3: claunch_f<ND, R, 3>(fuse, a); break;
    default: claunch_f<ND, R, 4>(fuse, a); break;
  }
}

}  // namespace

template <int ND, class R>
int cns_prepare_v(unsigned modes, size_t smem, bool brick) {
  return cprep<ND, R>(modes, smem, brick);
}

template <int ND, class R>
void cns_stage_v(int mode, bool fuse, const GhostTables& gt, double* gsl, const CnsLaunch& a) {
  if (gt.ng > 0) {
    const unsigned nb = (unsigned)((gt.ng + kBlock - 1) / kBlock);
    launch_chain(k_ghost_slopes<ND>, nb, kBlock, 0, a.st, a.qin, a.g, gt, gsl, a.h.ngl);
  }
  claunch_m<ND, R>(mode, fuse, a);
}

}  // namespace h3c
