// h3c_stage_cns.cu -- host side of the CNS tile stage (stage_cns.cuh): its
// set-up tables and the dispatch on dimension.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#define H3C_DEVICE_FUNCTIONS_ONLY
#include "fv_kernels.cuh"
#include "stage_cns.hpp"

namespace h3c {

bool halo_build_cns(int nd, long long ld, long long n_int, long long ntiles, const std::vector<long long>& tile_end,
                    const int* nbr, CnsHaloHost& H) {
  const int NP = 2 * nd, TB = kHaloTile;
  H.base.lnb.assign((size_t)NP * ld, 0);
  const int NB = nd == 3 ? kCnsBorder<3> : kCnsBorder<2>, H1 = nd == 3 ? kCnsBrickH1<3> : kCnsBrickH1<2>;
  std::vector<std::vector<int>> l1s(ntiles), l2s(ntiles);
  std::vector<std::vector<unsigned short>> hns(ntiles);
  H.bsel.assign(ld, 0);
  H.blist.assign((size_t)std::max<long long>(ntiles, 1) * NB, ~0u);
  std::atomic<bool> ok{true}, brick{true};
  auto work = [&](long long t0, long long t1) {
    std::vector<int> l1, l2;
    std::vector<unsigned char> need;
    for (long long t = t0; t < t1 && ok.load(std::memory_order_relaxed); ++t) {
      const long long c0 = t * TB, ce = tile_end[t];
      auto outside = [&](long long v) { return v < c0 || v >= ce; };
      l1.clear();
      for (long long c = c0; c < ce; ++c)
        for (int p = 0; p < NP; ++p) {
          const long long v = nbr[p * ld + c];
          if (v < 0) {  // CNS grids have no coarse/fine faces: every neighbour is a cell
            ok = false;
            return;
          }
          if (outside(v)) l1.push_back((int)v);
        }
      std::sort(l1.begin(), l1.end());
      l1.erase(std::unique(l1.begin(), l1.end()), l1.end());
      auto idx1 = [&](long long v) { return (long long)(std::lower_bound(l1.begin(), l1.end(), (int)v) - l1.begin()); };
      // slope directions each layer-1 cell needs: every direction but the ones it is a face neighbour across
      need.assign(l1.size(), 0);
      for (long long c = c0; c < ce; ++c)
        for (int p = 0; p < NP; ++p) {
          const long long v = nbr[p * ld + c];
          if (outside(v)) need[idx1(v)] |= (unsigned char)(((1 << nd) - 1) & ~(1 << (p >> 1)));
        }
      auto in_l1 = [&](long long v) { return std::binary_search(l1.begin(), l1.end(), (int)v); };
      l2.clear();
      for (size_t i = 0; i < l1.size(); ++i) {
        if (l1[i] >= n_int) continue;  // ghost: slopes from the ghost pass
        for (int sd = 0; sd < nd; ++sd) {
          if (!((need[i] >> sd) & 1)) continue;
          for (int side = 0; side < 2; ++side) {
            const long long v = nbr[(2 * sd + side) * ld + l1[i]];
            if (v < 0) {
              ok = false;
              return;
            }
            if (outside(v) && !in_l1(v)) l2.push_back((int)v);
          }
        }
      }
      std::sort(l2.begin(), l2.end());
      l2.erase(std::unique(l2.begin(), l2.end()), l2.end());
      if ((int)(l1.size() + l2.size()) > kHaloMaxSlots) {
        ok = false;
        return;
      }
      auto slot = [&](long long v) -> unsigned short {
        if (!outside(v)) return (unsigned short)(v - c0);
        auto it1 = std::lower_bound(l1.begin(), l1.end(), (int)v);
        if (it1 != l1.end() && *it1 == v) return (unsigned short)(TB + (it1 - l1.begin()));
        return (unsigned short)(TB + l1.size() + (std::lower_bound(l2.begin(), l2.end(), (int)v) - l2.begin()));
      };
      for (long long c = c0; c < ce; ++c)
        for (int p = 0; p < NP; ++p) H.base.lnb[(size_t)p * ld + c] = slot(nbr[p * ld + c]);
      // the border list (brick grids): minus faces that no plus face of the tile covers, whole warps per direction
      int nb = 0;
      for (int d = 0; d < nd && brick.load(std::memory_order_relaxed); ++d) {
        nb = (nb + 31) / 32 * 32;
        for (long long c = c0; c < ce; ++c) {
          const long long v = nbr[(2 * d) * ld + c];
          if (!outside(v) && nbr[(2 * d + 1) * ld + v] == c) continue;
          if (nb >= NB || !outside(v)) {
            brick = false;
            break;
          }
          H.blist[(size_t)t * NB + nb] = (unsigned)(c - c0) | ((unsigned)H.base.lnb[(size_t)(2 * d) * ld + c] << 8) |
                                            ((unsigned)d << 20);
          H.bsel[c] |= (unsigned)(nb + 1) << (8 * d);
          ++nb;
        }
      }
      std::vector<unsigned short>& hn = hns[t];
      hn.assign(l1.size() * NP, 0xffff);
      for (size_t i = 0; i < l1.size(); ++i) {
        if (l1[i] >= n_int) continue;
        for (int p = 0; p < NP; ++p)
          if ((need[i] >> (p >> 1)) & 1) hn[i * NP + p] = slot(nbr[p * ld + l1[i]]);
      }
      l1s[t] = l1;
      l2s[t] = l2;
    }
  };
  const int nthr = std::max(1, std::min<int>((int)std::thread::hardware_concurrency(), 16));
  std::vector<std::thread> pool;
  const long long per = (ntiles + nthr - 1) / nthr;
  for (int i = 0; i < nthr; ++i) {
    const long long a = i * per, b = std::min(ntiles, a + per);
    if (a < b) pool.emplace_back(work, a, b);
  }
  for (auto& th : pool) th.join();
  if (!ok) return false;
  HaloHost& B = H.base;
  B.off.assign(ntiles + 1, 0);
  B.goff.assign(ntiles + 1, 0);
  H.h1end.assign(std::max<long long>(ntiles, 1), 0);
  size_t nids = 0;
  int mx = 0, mx1 = 0;
  for (long long t = 0; t < ntiles; ++t) {
    const int n1 = (int)l1s[t].size(), n2 = (int)l2s[t].size();
    H.h1end[t] = (int)(nids + n1);
    nids += n1 + n2;
    B.off[t + 1] = (int)nids;
    mx = std::max(mx, n1 + n2);
    mx1 = std::max(mx1, n1);
  }
  B.ids.resize(std::max<size_t>(nids, 1));
  H.hnb.assign(std::max<size_t>(nids, 1) * NP, 0xffff);
  for (long long t = 0; t < ntiles; ++t) {
    std::copy(l1s[t].begin(), l1s[t].end(), B.ids.begin() + B.off[t]);
    std::copy(l2s[t].begin(), l2s[t].end(), B.ids.begin() + B.off[t] + l1s[t].size());
    std::copy(hns[t].begin(), hns[t].end(), H.hnb.begin() + (size_t)B.off[t] * NP);
  }
  B.grp.assign(1, 0);
  B.max_halo = mx;
  B.mean_halo = ntiles ? (double)nids / ntiles : 0.0;
  B.hmax = std::max(32, (mx + 31) / 32 * 32);
  H.h1max = std::max(32, (mx1 + 31) / 32 * 32);
  H.brick = brick && H.h1max <= H1;
  return true;
}

size_t cns_halo_smem_bytes(int nd, bool mixed, int hmax, int h1max, bool brick) {
  if (brick) {  // rows as long as a brick's, the second layer's landing as wide as this grid's
    const int h1 = nd == 3 ? kCnsBrickH1<3> : kCnsBrickH1<2>;
    hmax += h1 - h1max;
    h1max = h1;
  }
  if (nd == 2) return mixed ? cns_layout_bytes<float, 2>(hmax, h1max, brick) : cns_layout_bytes<double, 2>(hmax, h1max, brick);
  return mixed ? cns_layout_bytes<float, 3>(hmax, h1max, brick) : cns_layout_bytes<double, 3>(hmax, h1max, brick);
}

int cns_halo_prepare(int nd, bool mixed, unsigned modes, size_t smem, bool brick) {
  if (nd == 2) return mixed ? cns_prepare_v<2, float>(modes, smem, brick) : cns_prepare_v<2, double>(modes, smem, brick);
  return mixed ? cns_prepare_v<3, float>(modes, smem, brick) : cns_prepare_v<3, double>(modes, smem, brick);
}

void cns_halo_stage(int nd, bool mixed, int mode, bool fuse, const double* qin, double* out, const Geometry& g,
                    const GhostTables& gt, const CnsHaloGeom& h, const PhysConst& pc, const Scalars* sc,
                    long long* dtmin, int* status, int grid, size_t smem, cudaStream_t st, double* gsl) {
  const CnsLaunch a{qin, out, g, h, pc, sc, dtmin, status, grid, smem, st};
  if (nd == 2) {
    if (mixed) cns_stage_v<2, float>(mode, fuse, gt, gsl, a);
    else cns_stage_v<2, double>(mode, fuse, gt, gsl, a);
  } else {
    if (mixed) cns_stage_v<3, float>(mode, fuse, gt, gsl, a);
    else cns_stage_v<3, double>(mode, fuse, gt, gsl, a);
  }
}

}  // namespace h3c
