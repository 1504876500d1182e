// h3c_stage_split.cu -- the Euler/AUSM stage on Morton tiles with the flux
// splits precomputed per cell (the default Euler stage).
//
// AUSM (src/solver/fv/euler/physics.hpp:276-325) is a sum of a left and a
// right split: m = M+(L) + M-(R), p = P+(L) p_L + P-(R) p_R, and the flux is
// m theta_upwind + p e_d.  M+-, P+- p and theta depend on one cell only.  So
// a block of 256 threads, which owns a 256-cell tile of the Morton order
// (8x8x4 cells in 3D, 16x16 in 2D), first computes them once per cell into
// shared memory -- for its own cells along every direction, for the cells
// around the tile (the halo, listed at set-up per cell, direction and side)
// only the split their one face reads -- and after a single barrier every
// cell sums its 2 nd faces: per face two additions, one upwind choice of a
// shared-memory slot, and one product per variable.
//
// The kernel it replaced as the default (k_stage_ausm) evaluated each in-tile
// face once and handed the flux over, which took two more barriers and 30 KB
// of flux rows, and its border cells -- a third of an 8x8x4 brick's faces --
// recomputed the neighbour's primitive state in divergent branches (20.7 of
// 32 lanes active; 27.5-28.5 here).  1,448,336-cell 3D tree, RK2, microseconds per
// stage with the events' overhead (about 4), same GPU: FP64 98.6 / 111.2
// before, 84.1 / 105.0 here; FP32 fluxes 86.3 / 101.5 before, 70.0 / 82.1
// here; 24 2D grids of 2.3 M cells, FP32 fluxes: 85.0 / 99.1 before,
// 67.9 / 80.3 here.
//
// What bounds it: the pipe of shared memory and L1 in FP64 (59-63% of its
// peak by ncu), and in both the latency of the gathers ahead of the one barrier at
// 24-32 warps per SM.  At four blocks shared memory takes nearly the whole
// L1, so a register spilled on the common path costs an L2 round trip.  Hence
// the FP64 halo states land in shared memory by 8-byte asynchronous copies
// (no registers held in flight), and the neighbour slots are loaded only
// before the barrier.  Kept out, measured on the same tree (FP64): both
// states through registers 96 / 110; own theta in registers 89 / 110; halo
// slots ordered against bank conflicts 100 / 116 (conflicts fell by a
// quarter, but the gathers touched twice the lines).
#include <cuda_runtime.h>

#include <algorithm>

#define H3C_DEVICE_FUNCTIONS_ONLY
#include "fv_kernels.cuh"
#include "stage_split.hpp"
#include "launch.hpp"
#include "async_copy.cuh"

namespace h3c {

namespace {

template <class R> struct Pair;
template <> struct Pair<double> { using T = double2; };
template <> struct Pair<float> { using T = float2; };

// Shared rows over tile and halo slots: theta in pairs (two rows of pairs),
// then the splits (M, P) as pairs -- [2 nd][256] of the tile (M+ of each
// direction, then M-), and one per halo entry -- and what is left over (3D:
// theta_E; FP32: the pressure) in one row of singles or pairs.  The number of
// halo slots is a compile-time constant so that every row lies at a constant
// distance (an 8x8x4 brick has 256 halo cells, a 16x16 one 64; tiles at level
// jumps and at ragged edges more): four FP32 blocks still share an SM.
template <int ND, class R>
__host__ __device__ constexpr int split_slots() {
  return ND == 3 ? 384 : 256;
}
template <int ND, class R>
__host__ __device__ constexpr int split_extra() {  // R values per slot beyond the four paired thetas
  return (ND == 3 ? 1 : 0) + (sizeof(R) == 4 ? 1 : 0);
}
template <int ND, class R>
__host__ __device__ constexpr size_t split_layout_bytes() {
  return sizeof(R) * ((size_t)(4 + split_extra<ND, R>()) * (kHaloTile + split_slots<ND, R>()) +
                      2 * ((size_t)2 * ND * kHaloTile + split_slots<ND, R>()));
}

// Blocks per SM the kernel is register-budgeted for: four (64 registers), but
// three (80) in 3D FP64, where the coarse/fine path holds both sides' fluxes
// and 64 registers spilled 80-104 bytes: 97.7 / 111.4 us against 84.1 / 105.0
// (three blocks also leave 58 KB of L1 to the re-read of the state).  FP32
// at three blocks: 80.6 / 91.0 against 70.0 / 82.1.
template <int ND, class R>
__host__ __device__ constexpr int split_minb() {
  return ND == 3 && sizeof(R) == 8 ? 3 : 4;
}

// element `c` of a row of doubles: row pointers are the same for the whole
// grid, and cells number below 2^29 (the halo ids), so the byte offset is one
// 32-bit register
__device__ __forceinline__ const double* at32(const double* row, unsigned c) {
  return reinterpret_cast<const double*>(reinterpret_cast<const char*>(row) + c * 8u);
}
__device__ __forceinline__ double* at32(double* row, unsigned c) {
  return reinterpret_cast<double*>(reinterpret_cast<char*>(row) + c * 8u);
}

}  // namespace

template <int ND, class R, int MODE, bool HANG, bool FUSE>
__global__ void __launch_bounds__(kHaloTile, split_minb<ND, R>())
    k_stage_split(const double* qin, double* out, Geometry g, SplitGeom sg, PhysConst pc,
                  const Scalars* sc, long long* dtmin) {
  constexpr int NV = ND + 2, NP = 2 * ND, NS = 1 << (ND - 1), TB = kHaloTile;
  constexpr int HM = split_slots<ND, R>(), S = TB + HM;
  constexpr double W = ND == 2 ? 0.5 : 0.25;
  constexpr bool F32 = sizeof(R) == 4;
  constexpr int EX = split_extra<ND, R>();
  using P2 = typename Pair<R>::T;
  extern __shared__ __align__(16) unsigned char smem[];
  P2* const thA = reinterpret_cast<P2*>(smem);  // theta 0, 1
  P2* const thB = thA + S;                      // theta 2, 3
  P2* const sp = thB + S;                       // splits: [2 ND][TB] | [HM]
  R* const ex = reinterpret_cast<R*>(sp + 2 * ND * TB + HM);
  __shared__ double skdt[kMaxLevels];  // dt / length of each level
  const int tid = threadIdx.x;
  const long long ld = g.ld;
  const R gamma = (R)pc.gamma, gm1 = (R)pc.gm1;
  chain_begin();

  // theta of the state in P.q into slot s; P keeps p, a and the Mach numbers
  auto store_theta = [&](int s, Prim<R, ND>& P) {
    make_prim<R, ND>(P, gamma, gm1);
    thA[s] = P2{P.q[0] * P.a, P.q[1] * P.a};
    const R thE = (P.q[ND + 1] + P.p) * P.a;
    thB[s] = P2{P.q[2] * P.a, ND == 3 ? P.q[3] * P.a : thE};
    if (EX == 2) reinterpret_cast<P2*>(ex)[s] = P2{thE, P.p};
    else if (EX == 1) ex[s] = F32 ? P.p : thE;
  };
  // split pair of a cell on its left (s = 1) or right (s = -1) side of a face, |M| <= 1: the subsonic
  // branches of m_int and p_int.  FP64 keeps P p (the face then only adds); FP32 keeps P alone and the
  // face forms P p with the roundings of ausm_face.
  auto split_sub = [&](R s, R M, R p) -> P2 {
    const R t = (M + s) * (M + s);
    const R ps = (R(0.25) * t) * (R(2) - s * M);
    return P2{(s * R(0.25)) * t, F32 ? ps : ps * p};
  };
  // the general pair; callers take it for a warp's supersonic cells only
  auto split = [&](R s, R M, R p) -> P2 {
    const R ps = p_int<R>(s, M);
    return P2{m_int<R>(s, M), F32 ? ps : ps * p};
  };
  // FP64: a state lands in its slot's theta row by 8-byte asynchronous copies (no registers held while in flight)
  auto land = [&](int s, unsigned n) {
    double* a = reinterpret_cast<double*>(thA + s);
    double* b = reinterpret_cast<double*>(thB + s);
    cp_async8(a, at32(qin, n));
    cp_async8(a + 1, at32(qin + ld, n));
    cp_async8(b, at32(qin + 2 * ld, n));
    cp_async8(b + 1, at32(qin + 3 * ld, n));
    if (ND == 3) cp_async8(ex + s, at32(qin + 4 * ld, n));
  };
  auto landed = [&](int s, Prim<R, ND>& P) {
    const P2 a = thA[s], b = thB[s];
    P.q[0] = a.x;
    P.q[1] = a.y;
    P.q[2] = b.x;
    P.q[3] = b.y;
    if (ND == 3) P.q[NV - 1] = ex[s];
  };
  auto fetch = [&](unsigned n, double* q) {
#pragma unroll
    for (int v = 0; v < NV; ++v) q[v] = *at32(qin + v * ld, n);
  };

  for (long long tile = blockIdx.x; tile < g.ntiles; tile += gridDim.x) {
    const unsigned c = (unsigned)(tile * TB) + tid;
    const int inst = tile_instance(g, tile);
    const bool live = c < (unsigned)min(tile * TB + TB, instance_end(g, inst));
    const int o0 = __ldg(sg.h.halo_off + tile);
    const int nh = min(__ldg(sg.h.halo_off + tile + 1) - o0, HM);  // entries beyond HM: read where a face needs them
    int hid = tid < nh ? __ldg(sg.h.halo_ids + o0 + tid) : 0;
    double q[NV];
    if (live) fetch(c, q);
    if (live) {
      if (ND == 3) asm volatile("prefetch.global.L2 [%0];" ::"l"(sg.pack3 + c));
      else asm volatile("prefetch.global.L2 [%0];" ::"l"(sg.pack2 + c));
      if (MODE != 0) {  // the start state, read at the update
#pragma unroll
        for (int v = 0; v < NV; ++v) asm volatile("prefetch.global.L2 [%0];" ::"l"(at32(g.q0 + v * ld, c)));
      }
    }
    if (tid < kMaxLevels) skdt[tid] = sc[inst].dt / g.len[tid];

    // ---- theta and splits of the own cell and of the halo entries ----
    auto own_cell = [&](Prim<R, ND>& P) {
      store_theta(tid, P);
      bool super = false;
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        sp[d * TB + tid] = split_sub(R(1), P.M[d], P.p);
        sp[(ND + d) * TB + tid] = split_sub(R(-1), P.M[d], P.p);
        super |= beyond_one(P.M[d]);
      }
      if (super) {
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          sp[d * TB + tid] = split(R(1), P.M[d], P.p);
          sp[(ND + d) * TB + tid] = split(R(-1), P.M[d], P.p);
        }
      }
    };
    auto halo_cell = [&](int h, int id, Prim<R, ND>& P) {
      store_theta(TB + h, P);
      const int dir = halo_dir(id);
      R M = P.M[0];
#pragma unroll
      for (int d = 1; d < ND; ++d) M = dir == d ? P.M[d] : M;
      const R sd = halo_plus(id) ? R(-1) : R(1);
      sp[2 * ND * TB + h] = split_sub(sd, M, P.p);
      if (beyond_one(M)) sp[2 * ND * TB + h] = split(sd, M, P.p);
    };
    if (F32) {
      Prim<R, ND> P;
      if (live) {
#pragma unroll
        for (int v = 0; v < NV; ++v) P.q[v] = (R)q[v];
      }
      if (tid < nh) fetch(hid & kHaloCellMask, q);
      if (live) own_cell(P);
      for (int h = tid; h < nh; h += TB) {
        if (h != tid) {
          hid = __ldg(sg.h.halo_ids + o0 + h);
          fetch(hid & kHaloCellMask, q);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v) P.q[v] = (R)q[v];
        halo_cell(h, hid, P);
      }
    } else {
      const int h2 = tid + TB;
      int hid2 = 0;
      if (tid < nh) land(TB + tid, hid & kHaloCellMask);
      if (HM > TB && h2 < nh) {
        hid2 = __ldg(sg.h.halo_ids + o0 + h2);
        land(TB + h2, hid2 & kHaloCellMask);
      }
      Prim<R, ND> P;
      if (live) {
#pragma unroll
        for (int v = 0; v < NV; ++v) P.q[v] = (R)q[v];
        own_cell(P);
      }
      cp_async_wait_all();  // a thread reads only what it copied itself
      if (tid < nh) {
        landed(TB + tid, P);
        halo_cell(tid, hid, P);
      }
      if (HM > TB && h2 < nh) {
        landed(TB + h2, P);
        halo_cell(h2, hid2, P);
      }
    }
    uint4 pk = make_uint4(0, 0, 0, 0);
    int lev = 0;
    if (live) {
      if (ND == 3) {
        pk = load_here(sg.pack3 + c);
        lev = pk.w & 0xffff;
      } else {
        const uint2 t = __ldg(sg.pack2 + c);
        pk.x = t.x;
        pk.y = t.y;
        lev = g.lvl[c];
      }
    }
    __syncthreads();

    // ---- faces: AUSM flux (euler/physics.hpp:276-293) from both sides' splits and pressures and the upwind theta ----
    auto pressure_sum = [&](P2 l, P2 r, R pl, R pr) -> R {
      if (F32) return (R)fmaf((float)l.y, (float)pl, __fmul_rn((float)r.y, (float)pr));
      return l.y + r.y;
    };
    // component v of the flux: rounded products, so that equal faces cancel exactly
    auto term = [&](int v, int d, const R* th, R mi, R pi) -> double {
      if (v == d) return F32 ? (double)fmaf((float)th[v], (float)mi, (float)pi) : fma((double)th[v], (double)mi, (double)pi);
      return F32 ? (double)__fmul_rn((float)th[v], (float)mi) : __dmul_rn((double)th[v], (double)mi);
    };
    auto load_theta = [&](int s, R* th) {
      const P2 a = thA[s], b = thB[s];
      th[0] = a.x;
      th[1] = a.y;
      th[2] = b.x;
      th[3] = b.y;
      if (ND == 3) th[NV - 1] = EX == 2 ? reinterpret_cast<const P2*>(ex)[s].x : ex[s];
    };
    auto pressure = [&](int s) -> R {  // FP32 only
      if (!F32) return R(0);
      return EX == 2 ? reinterpret_cast<const P2*>(ex)[s].y : ex[s];
    };
    // slot and split pair index of the neighbour across position 2 d + side
    auto slot_of = [&](int p) -> int {
      const unsigned w = p < 2 ? pk.x : p < 4 ? pk.y : pk.z;
      return (p & 1) ? (int)(w >> 16) : (int)(w & 0xffff);
    };
    auto split_at = [&](int s, int row) -> P2 { return sp[s + (s < TB ? row * TB : 2 * ND * TB - TB)]; };

    long long ord = kOrdMax;
    bool bad = false;
    if (live) {
      double acc[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] = 0.0;
      unsigned deferred = 0;
      const R po = pressure(tid);
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        const int sm = slot_of(2 * d), sq = slot_of(2 * d + 1);
        // a coarse/fine group (slots have kGroupBit) or an entry that is not in shared memory: the rolled loop below
        if (sm >= S || sq >= S) {
          deferred |= 1u << d;
          continue;
        }
        R th[NV];
        double fm[NV];
        {
          const P2 l = split_at(sm, d), r = sp[(ND + d) * TB + tid];
          const R mi = l.x + r.x;
          const R pi = pressure_sum(l, r, pressure(sm), po);
          load_theta(mi >= R(0) ? sm : tid, th);
#pragma unroll
          for (int v = 0; v < NV; ++v) fm[v] = term(v, d, th, mi, pi);
        }
        const P2 l = sp[d * TB + tid], r = split_at(sq, ND + d);
        const R mi = l.x + r.x;
        const R pi = pressure_sum(l, r, po, pressure(sq));
        load_theta(mi >= R(0) ? tid : sq, th);
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] = acc[v] + (fm[v] - term(v, d, th, mi, pi));
      }
      if (deferred) {
        // directions with a coarse/fine group on a side: W times the sum over the fine cells j of
        // F(minus, j) - F(plus, j), where a side without a group gives its one flux every time -- exactly
        // zero in a uniform flow, and no more registers than the loop above (the sums of both sides kept
        // apart made the common path spill: FP64 108 / 134 us)
        const int gbase = HANG ? __ldg(sg.h.grp_off + tile) : 0;
        const unsigned short* slots = ND == 3 ? reinterpret_cast<const unsigned short*>(sg.pack3 + c)
                                              : reinterpret_cast<const unsigned short*>(sg.pack2 + c);
#pragma unroll 1
        for (int d = 0; d < ND; ++d) {
          if (!((deferred >> d) & 1u)) continue;
          const int s0[2] = {__ldg(slots + 2 * d), __ldg(slots + 2 * d + 1)};
          const bool any = HANG && ((s0[0] | s0[1]) & kGroupBit);
          const int cnt = any ? NS : 1;
          const double w = any ? W : 1.0;  // a power of two: its products are exact
#pragma unroll 1
          for (int j = 0; j < cnt; ++j) {
            double fm[NV];
#pragma unroll
            for (int side = 0; side < 2; ++side) {
              const bool plus = side;
              const bool grp = HANG && (s0[side] & kGroupBit);
              const int s = grp ? __ldg(sg.h.grp + (size_t)(gbase + (s0[side] & ~kGroupBit)) * NS + j) : s0[side];
              const P2 own = sp[(plus ? d : ND + d) * TB + tid];
              P2 nb;
              R th[NV], pn, mi;
              if (s < S) {
                nb = split_at(s, plus ? ND + d : d);
                pn = pressure(s);
                mi = plus ? own.x + nb.x : nb.x + own.x;
                load_theta((mi >= R(0)) == plus ? tid : s, th);
              } else {
                Prim<R, ND> P;
                load_prim<R, ND>(P, qin, ld, __ldg(sg.h.halo_ids + o0 + (s - TB)) & kHaloCellMask, gamma, gm1);
                R M = P.M[0];
#pragma unroll
                for (int e = 1; e < ND; ++e) M = d == e ? P.M[e] : M;
                nb = split(plus ? R(-1) : R(1), M, P.p);
                pn = P.p;
                mi = plus ? own.x + nb.x : nb.x + own.x;
                if ((mi >= R(0)) == plus) {
                  load_theta(tid, th);
                } else {
#pragma unroll
                  for (int v = 0; v < ND + 1; ++v) th[v] = P.q[v] * P.a;
                  th[ND + 1] = (P.q[ND + 1] + P.p) * P.a;
                }
              }
              // FP32: the product that is rounded first is the right cell's, in a group the own cell's
              const R pi = plus && !grp ? pressure_sum(own, nb, po, pn) : pressure_sum(nb, own, pn, po);
#pragma unroll
              for (int v = 0; v < NV; ++v) {
                double f = term(v, -1, th, mi, pi);
                if (v < ND) f = v == d ? term(v, v, th, mi, pi) : f;
                if (!plus) fm[v] = f;
                else acc[v] = fma(w, fm[v] - f, acc[v]);
              }
            }
          }
        }
      }
      // ---- update and the next step's CFL minimum ----
      double qo[NV];
      if (MODE != 0) {
#pragma unroll
        for (int v = 0; v < NV; ++v) qo[v] = *at32(g.q0 + v * ld, c);
      }
      const double k = skdt[lev];
      double o[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v)
        o[v] = rk_combine<MODE>(MODE == 0 ? 0.0 : qo[v], *at32(qin + v * ld, c), k * acc[v]);
#pragma unroll
      for (int v = 0; v < NV; ++v) *at32(out + v * ld, c) = o[v];
      if (FUSE) {
        const double cd = cell_dt<ND, EULER>(o, g.len[lev], pc, nullptr, &bad);
        if (!isnan(cd)) ord = dbl_to_ord(cd);
      }
    }
    if (FUSE) {
      flag_bad_state(bad, sc, inst);
      block_min_atomic(ord, per_instance(dtmin, inst));
    }
    if (gridDim.x < g.ntiles) __syncthreads();  // the next tile rewrites the shared rows
  }
}

__global__ void __launch_bounds__(kBlock) k_split_pack(int nd, const unsigned short* __restrict__ lnb,
                                                       const unsigned char* __restrict__ lvl, long long ld,
                                                       long long n, uint4* pack3, uint2* pack2) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  unsigned w[3] = {0, 0, 0};
  for (int p = 0; p < 2 * nd; ++p) w[p >> 1] |= (unsigned)lnb[p * ld + c] << (16 * (p & 1));
  if (nd == 3) pack3[c] = make_uint4(w[0], w[1], w[2], lvl[c]);
  else pack2[c] = make_uint2(w[0], w[1]);
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
size_t split_pack_bytes(int nd, long long n) { return (size_t)n * (nd == 3 ? sizeof(uint4) : sizeof(uint2)); }

void split_pack(int nd, const unsigned short* lnb, const unsigned char* lvl, long long ld, long long n, void* pack,
                cudaStream_t st) {
  const unsigned nb = (unsigned)std::max<long long>(1, (n + kBlock - 1) / kBlock);
  k_split_pack<<<nb, kBlock, 0, st>>>(nd, lnb, lvl, ld, n, (uint4*)pack, (uint2*)pack);
}

int split_halo_slots(int nd) { return nd == 2 ? split_slots<2, double>() : split_slots<3, double>(); }

size_t split_smem_bytes(int nd, bool mixed) {
  if (nd == 2) return mixed ? split_layout_bytes<2, float>() : split_layout_bytes<2, double>();
  return mixed ? split_layout_bytes<3, float>() : split_layout_bytes<3, double>();
}

namespace {

template <int ND, class R, int MODE, bool HANG, bool FUSE>
bool sprep_one(size_t smem) {
  auto k = k_stage_split<ND, R, MODE, HANG, FUSE>;
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
    return false;
  }
  return true;
}
template <int ND, class R, int MODE>
bool sprep_m(size_t smem, bool hang) {
  return hang ? sprep_one<ND, R, MODE, true, false>(smem) && sprep_one<ND, R, MODE, true, true>(smem)
              : sprep_one<ND, R, MODE, false, false>(smem) && sprep_one<ND, R, MODE, false, true>(smem);
}
template <int ND, class R>
bool sprep(size_t smem, unsigned modes, bool hang) {
  return (!(modes & 1u) || sprep_m<ND, R, 0>(smem, hang)) && (!(modes & 4u) || sprep_m<ND, R, 2>(smem, hang)) &&
         (!(modes & 8u) || sprep_m<ND, R, 3>(smem, hang)) && (!(modes & 16u) || sprep_m<ND, R, 4>(smem, hang));
}

struct SplitLaunch {
  const double* qin;
  double* out;
  const Geometry& g;
  const SplitGeom& h;
  const PhysConst& pc;
  const Scalars* sc;
  long long* dtmin;
  unsigned grid;
  size_t smem;
  cudaStream_t st;
};
template <int ND, class R, int MODE, bool HANG>
void slaunch_f(bool fuse, const SplitLaunch& a) {
  launch_chain(fuse ? k_stage_split<ND, R, MODE, HANG, true> : k_stage_split<ND, R, MODE, HANG, false>, a.grid,
               kHaloTile, a.smem, a.st, a.qin, a.out, a.g, a.h, a.pc, a.sc, a.dtmin);
}
template <int ND, class R, int MODE>
void slaunch_h(bool hang, bool fuse, const SplitLaunch& a) {
  if (hang) slaunch_f<ND, R, MODE, true>(fuse, a);
  else slaunch_f<ND, R, MODE, false>(fuse, a);
}
template <int ND, class R>
void slaunch_m(int mode, bool hang, bool fuse, const SplitLaunch& a) {
  switch (mode) {
    case 0: slaunch_h<ND, R, 0>(hang, fuse, a); break;
    case 2: slaunch_h<ND, R, 2>(hang, fuse, a); break;
    case 3: slaunch_h<ND, R, 3>(hang, fuse, a); break;
    default: slaunch_h<ND, R, 4>(hang, fuse, a); break;
  }
}

}  // namespace

// 48 KB are a block's without an opt-in: only 3D FP64 (56 KB) needs one, for
// the variants the solver launches (each is loaded by its first call, which
// for all 16 of a dimension and precision took a first grid 2 ms).
bool split_prepare(int nd, bool mixed, unsigned modes, bool hang, size_t smem) {
  constexpr size_t kFree = 48 * 1024, kStatic = 1024;  // the kernel's static arrays are smaller
  if (smem + kStatic <= kFree) return true;
  if (nd == 2) return mixed ? sprep<2, float>(smem, modes, hang) : sprep<2, double>(smem, modes, hang);
  return mixed ? sprep<3, float>(smem, modes, hang) : sprep<3, double>(smem, modes, hang);
}

void split_stage(int nd, bool mixed, int mode, bool hang, bool fuse, const double* qin, double* out,
                 const Geometry& g, const SplitGeom& h, const PhysConst& pc, const Scalars* sc, long long* dtmin,
                 unsigned grid, size_t smem, cudaStream_t st) {
  const SplitLaunch a{qin, out, g, h, pc, sc, dtmin, grid, smem, st};
  if (nd == 2) {
    if (mixed) slaunch_m<2, float>(mode, hang, fuse, a);
    else slaunch_m<2, double>(mode, hang, fuse, a);
  } else {
    if (mixed) slaunch_m<3, float>(mode, hang, fuse, a);
    else slaunch_m<3, double>(mode, hang, fuse, a);
  }
}

}  // namespace h3c
