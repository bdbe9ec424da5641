// dg_launch.cuh -- host-side launch of the beam-search kernel instantiations.
#pragma once
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "dg_search_cta.cuh"

namespace dg {

struct LaunchInfo {
  int grid = 0;
  int blocks_per_sm = 0;
  uint32_t smem = 0;
};

// Launch geometry: as many resident CTAs as shared memory and registers allow
// on every SM, never more than the queries need.
// Resident blocks per SM of (device, kernel, shared-memory size), and the
// largest dynamic shared memory already granted to (device, kernel): the
// attribute and occupancy queries run once, not on every launch (a serving
// loop launches thousands of small batches per second).
struct LaunchGeometry {
  std::mutex mu;
  std::unordered_map<const void *, int> sms, optin;                  // per device (key: device id)
  std::unordered_map<uint64_t, int> granted;                           // (device, kernel) -> smem
  std::unordered_map<uint64_t, std::unordered_map<uint32_t, int>> nb;  // (device, kernel) -> smem -> blocks
};
inline LaunchGeometry &launch_geometry() {
  static LaunchGeometry g;
  return g;
}

// `queries` per CTA of `warps` warps, Ly.total bytes of shared memory each.
template <typename K>
DgStatus launch_persistent(K kernel, const SearchArgs &a, const WarpLayout &Ly, uint32_t warps, uint32_t queries,
                           cudaStream_t st, LaunchInfo *info) {
  const uint32_t smem = Ly.total * queries;
  int dev = 0;
  DG_CUDA(cudaGetDevice(&dev));
  LaunchGeometry &G = launch_geometry();
  const void *kp = reinterpret_cast<const void *>(kernel);
  const uint64_t key = (reinterpret_cast<uint64_t>(kp) << 8) ^ (uint64_t)dev;
  const void *dkey = reinterpret_cast<const void *>((uintptr_t)dev + 1);
  int sms = 0, nb = 0;
  {
    std::lock_guard<std::mutex> lk(G.mu);
    auto s_it = G.sms.find(dkey);
    if (s_it == G.sms.end()) {
      int m = 0, o = 0;
      DG_CUDA(cudaDeviceGetAttribute(&o, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
      DG_CUDA(cudaDeviceGetAttribute(&m, cudaDevAttrMultiProcessorCount, dev));
      G.optin[dkey] = o;
      s_it = G.sms.emplace(dkey, m).first;
    }
    sms = s_it->second;
    if (std::max(smem, a.limit_smem) > (uint32_t)G.optin[dkey])
      return fail(DG_ENOTSUP, "search state does not fit in shared memory (beam/quantizer too large)");
    int &gr = G.granted[key];
    if ((int)smem > gr) {
      DG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      gr = (int)smem;
    }
    auto &per = G.nb[key];
    const uint32_t okey = smem * 8u + warps;
    auto n_it = per.find(okey);
    if (n_it == per.end()) {
      int v = 0;
      DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kernel, 32 * (int)warps, smem));
      n_it = per.emplace(okey, v).first;
    }
    nb = n_it->second;
  }
  if (nb <= 0) return fail(DG_ENOTSUP, "search kernel cannot be resident on an SM");
  if (a.occ_pct > 0 && a.occ_pct < 100) nb = std::max(1, (int)((nb * a.occ_pct + 99) / 100));
  int grid = nb * sms;
  const int need = (int)((a.nq + queries - 1) / queries);
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  kernel<<<grid, 32 * warps, smem, st>>>(a, Ly);
  DG_CUDA(cudaGetLastError());
  if (info) {
    info->grid = grid;
    info->blocks_per_sm = nb;
    info->smem = smem;
  }
  return DG_OK;
}

template <int NW, int TRAV, int MET, int LPR>
DgStatus launch_cta(const SearchArgs &a, const WarpLayout &Ly, bool tc, bool filt, cudaStream_t st, LaunchInfo *info) {
  if constexpr (TRAV == TRAV_BF16) {
    if (tc) return launch_persistent(beam_search_cta_kernel<NW, TRAV, MET, LPR, true, false>, a, Ly, NW, 1, st, info);
  }
  return filt ? launch_persistent(beam_search_cta_kernel<NW, TRAV, MET, LPR, false, true>, a, Ly, NW, 1, st, info)
              : launch_persistent(beam_search_cta_kernel<NW, TRAV, MET, LPR, false, false>, a, Ly, NW, 1, st, info);
}

// The CTA-per-query kernel (cta), or the register-list kernel (unfiltered, one
// seed, beams up to 64).  BF16 rows: beams up to 64 without a filter take the
// tensor-core distances of the register-list kernel in both (tc), so that a
// search returns the same bits at every batch size.
template <int TRAV, int MET, int LPR>
DgStatus launch_trav(const SearchArgs &a, const WarpLayout &Ly, uint32_t cta, bool tc, bool filt, cudaStream_t st,
                     LaunchInfo *info) {
  constexpr int F = 8;  // lanes per FP32 row in the rerank gather
  if (!cta) {
    const uint32_t wpb = (a.wpb == 1 || a.wpb == 2) ? a.wpb : 4u;
    return launch_persistent(beam_search_kernel<TRAV, MET, LPR, F>, a, Ly, wpb, wpb, st, info);
  }
  return cta == 1   ? launch_cta<1, TRAV, MET, LPR>(a, Ly, tc, filt, st, info)
         : cta == 2 ? launch_cta<2, TRAV, MET, LPR>(a, Ly, tc, filt, st, info)
         : cta == 8 ? launch_cta<8, TRAV, MET, LPR>(a, Ly, tc, filt, st, info)
                    : launch_cta<4, TRAV, MET, LPR>(a, Ly, tc, filt, st, info);
}

template <int TRAV, int LPR>
DgStatus launch_met(const SearchArgs &a, const WarpLayout &Ly, int met, uint32_t cta, bool tc, bool filt,
                    cudaStream_t st, LaunchInfo *info) {
  switch (met) {
    case MET_L2: return launch_trav<TRAV, MET_L2, LPR>(a, Ly, cta, tc, filt, st, info);
    case MET_DOT: return launch_trav<TRAV, MET_DOT, LPR>(a, Ly, cta, tc, filt, st, info);
    default: return launch_trav<TRAV, MET_COS, LPR>(a, Ly, cta, tc, filt, st, info);
  }
}

// One entry per traversal kind, defined in its own translation unit.
DgStatus launch_search_f32(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                           bool filt, cudaStream_t st, LaunchInfo *info);
DgStatus launch_search_bf16(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                            bool filt, cudaStream_t st, LaunchInfo *info);
DgStatus launch_search_f16(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                           bool filt, cudaStream_t st, LaunchInfo *info);
DgStatus launch_search_int8(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                            bool filt, cudaStream_t st, LaunchInfo *info);
DgStatus launch_search_pq(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                          bool filt, cudaStream_t st, LaunchInfo *info);
DgStatus launch_search_rabitq(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                              bool filt, cudaStream_t st, LaunchInfo *info);
DgStatus launch_search_fp8(const SearchArgs &a, const WarpLayout &Ly, int met, int lpr, uint32_t cta, bool tc,
                           bool filt, cudaStream_t st, LaunchInfo *info);

}  // namespace dg
