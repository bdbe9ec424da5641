// dg_vamana.cu -- build_vamana_graph (diskann-rs src/lib.rs:774-1073) on the GPU.
//
// Each refinement pass of the reference reads a snapshot of the graph, so it
// is data parallel over nodes:
//   1. k_build_search: one warp per node runs the three greedy searches
//      (medoid + two random seeds, src/lib.rs:823-844) on the snapshot and
//      writes the node's candidate pool (current neighbours + the three
//      working sets) as (distance, id) keys;
//   2. k_prune: one block per node sorts and de-duplicates the pool and runs
//      robust_prune (src/lib.rs:977-1034) with the candidate rows staged in
//      shared memory;
//   3. symmetrisation (src/lib.rs:868-904): in-degree count, prefix sum,
//      incoming lists, distances, and k_prune again.
// The random draws use the counter-based stream shared with the oracle, so a
// GPU build equals the oracle build whenever distances are exact (integer
// valued data), which the tests check.
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dg_index.h"
#include "dg_search_cta.cuh"

namespace dg {

constexpr int kPruneThreads = 256;
constexpr int kPruneSortCap = 2048;  // pools up to this size are sorted in shared memory
constexpr int kPruneTileBytes = 64 * 1024;

// --------------------------------------------------------------- bootstrap
// src/lib.rs:786-799: `target` distinct random neighbours != i, in draw order.
__global__ void k_bootstrap(uint64_t n, uint32_t R, uint32_t target, uint64_t seed, uint32_t *graph) {
  const int lane = threadIdx.x & 31;
  const uint64_t gw = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t i = gw; i < n; i += nw) {
    uint32_t *row = graph + i * R;
    uint32_t have = 0;
    for (uint64_t t0 = 0; have < target; t0 += 32) {
      const uint32_t x = (uint32_t)range_of(rand4(seed, 0, i, t0 + lane), n);
      bool ok = x != (uint32_t)i;
      // first occurrence within this batch of draws
      const uint32_t same = __match_any_sync(kFull, x);
      if (__ffs(same) - 1 != lane) ok = false;
      // not accepted by an earlier batch
      for (uint32_t j = 0; j < have && ok; ++j)
        if (row[j] == x) ok = false;
      const uint32_t m = __ballot_sync(kFull, ok);
      const uint32_t pos = have + __popc(m & ((1u << lane) - 1u));
      if (ok && pos < target) row[pos] = x;
      have = min(target, have + (uint32_t)__popc(m));
      __syncwarp();
    }
    for (uint32_t j = target + lane; j < R; j += 32) row[j] = DG_PAD;
  }
}

// -------------------------------------------------------- build searches
struct BuildArgs {
  uint64_t n;
  uint32_t d, dpad, R, Lb, medoid, pass;
  uint64_t seed;
  int32_t metric;
  const float *vf;      // [n][dpad]
  const uint16_t *vb;   // [n][dpad] bf16 (only when every value is bf16-exact)
  const float *vbn;     // [n] squared norms of the bf16 rows (tensor-core distances)
  const uint32_t *graph;  // snapshot [n][R]
  uint32_t hbits, hB;     // visited table: log2 words, id bits
  uint64_t u0, u1;        // node range of this chunk
  uint32_t cw;            // candidate slots per node (R + 3*Lb)
  uint64_t *cand;         // [(u1-u0)][cw]
  uint32_t *cand_cnt;     // [(u1-u0)]
};

// Distances of a warp's cnt <= 32 candidates to the node's own row (qs).  TC:
// integer-valued rows whose sums are exact in any order, x.q on the tensor
// cores (the query is its own high half, hi; the low half is zero) and
// |x|^2 + |q|^2 - 2 x.q in integers.
template <int ELEM, int MET, int LPR, bool TC>
__device__ __forceinline__ float build_dist(const BuildArgs &a, const float *qs, const uint16_t *hi, float qq,
                                            uint32_t cand, int cnt, int lane) {
  if constexpr (TC) {
    const float xx = MET == MET_L2 && lane < cnt ? __ldg(a.vbn + cand) : 0.0f;
    const float dot = bf16_dot_mma(a.vb, a.dpad, hi, cand, cnt, lane);
    const float v = MET == MET_L2 ? (float)((int)xx + (int)qq - 2 * (int)dot) : dot;
    return finish_metric(MET, a.metric == DG_L2, v, 0.0f, 0.0f);
  } else if constexpr (ELEM == 1) {
    return rows_distance<LPR, 1, MET>(reinterpret_cast<const uint8_t *>(a.vb), a.dpad * 2, (a.dpad / 8) / LPR, qs,
                                      cand, cnt, lane, a.metric == DG_L2, qq);
  } else {
    return rows_distance<LPR, 0, MET>(reinterpret_cast<const uint8_t *>(a.vf), a.dpad * 4, (a.dpad / 4) / LPR, qs,
                                      cand, cnt, lane, a.metric == DG_L2, qq);
  }
}

// Shared memory of one warp's searches: list, new keys, staged candidates,
// visited table, the node's row (f32, and its BF16 halves), bitmap and count.
struct BuildLayout {
  uint32_t list, surv, stage, hash, qf, hi, ctl, total;
};
static BuildLayout build_layout(uint32_t Lb, uint32_t R, uint32_t hbits, uint32_t dpad, bool tc) {
  BuildLayout L{};
  uint32_t o = 0;
  L.list = o; o += align16(std::max(Lb, 2u) * 8);
  L.surv = o; o += cta_surv_bytes(32);
  L.stage = o; o += align16(R * 4);
  L.hash = o; o += (1u << hbits) * 4;
  L.qf = o; o += dpad * 4;
  L.hi = o; o += tc ? dpad * 4 : 0;
  L.ctl = o; o += (32 + 4) * 4;
  L.total = align16(o);
  return L;
}

// One warp per node: its current neighbours with their distances, then three
// greedy searches, each on a list merged in place (cta_merge, one warp).
// 25k nodes x 128, R = 64, beam 128: 24 ms per pass with a second copy of the
// list, entry-by-entry merges and FMA distances.  Five CTAs per SM leave 96
// registers, of which FMA distances of FP32 rows spill 144-224 bytes.
template <int ELEM, int MET, int LPR, bool TC>
__global__ void __launch_bounds__(128, 5) k_build_search(BuildArgs a, BuildLayout Ly) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t *wsm = smem + (size_t)warp * Ly.total;
  uint64_t *W = reinterpret_cast<uint64_t *>(wsm + Ly.list);
  uint32_t *stage = reinterpret_cast<uint32_t *>(wsm + Ly.stage);
  const Visited vt{reinterpret_cast<uint32_t *>(wsm + Ly.hash), a.hbits, a.hB};
  float *qs = reinterpret_cast<float *>(wsm + Ly.qf);
  uint16_t *hi = reinterpret_cast<uint16_t *>(wsm + Ly.hi);
  uint32_t *map = reinterpret_cast<uint32_t *>(wsm + Ly.ctl), *cnt_s = map + 32;
  CtaList lists[2];
  lists[0] = CtaList{W, 0, (int)a.Lb, reinterpret_cast<uint64_t *>(wsm + Ly.surv),
                     reinterpret_cast<uint16_t *>(wsm + Ly.surv + align16(32 * 8)), map};
  map[lane] = 0u;
  if (lane == 0) *cnt_s = 0u;
  const uint64_t gw = blockIdx.x * (uint64_t)(blockDim.x >> 5) + warp;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t u = a.u0 + gw; u < a.u1; u += nw) {
    uint64_t *out = a.cand + (u - a.u0) * a.cw;
    for (uint32_t i = lane; i < a.dpad; i += 32) {
      qs[i] = a.vf[u * a.dpad + i];
      if (TC) {
        hi[i] = a.vb[u * a.dpad + i];
        hi[a.dpad + i] = 0;
      }
    }
    __syncwarp();
    float qq = TC && MET == MET_L2 ? __ldg(a.vbn + u) : 0.0f;
    if (MET == MET_COS) {
      for (uint32_t i = lane; i < a.dpad; i += 32) qq = fmaf(qs[i], qs[i], qq);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) qq += __shfl_xor_sync(kFull, qq, o);
    }
    uint32_t nout = 0;
    // current neighbours with their distances (src/lib.rs:818-822)
    {
      const uint32_t *row = a.graph + u * a.R;
      for (uint32_t j0 = 0; j0 < a.R; j0 += 32) {
        const uint32_t j = j0 + lane;
        const uint32_t nb = j < a.R ? row[j] : DG_PAD;
        const bool ok = nb != DG_PAD;
        const uint32_t m = __ballot_sync(kFull, ok);
        const int cnt = __popc(m);
        if (!cnt) continue;
        if (ok) stage[__popc(m & ((1u << lane) - 1u))] = nb;
        __syncwarp();
        const uint32_t c = lane < cnt ? stage[lane] : 0u;
        const float dd = build_dist<ELEM, MET, LPR, TC>(a, qs, hi, qq, c, cnt, lane);
        if (lane < cnt) out[nout + lane] = make_key(dd, c);
        nout += cnt;
        __syncwarp();
      }
    }
    // three greedy searches (greedy_search, src/lib.rs:921-973)
    const uint32_t seeds[3] = {a.medoid, (uint32_t)range_of(rand4(a.seed, a.pass + 1, u, 0), a.n),
                               (uint32_t)range_of(rand4(a.seed, a.pass + 1, u, 1), a.n)};
    for (int s = 0; s < 3; ++s) {
      vt.clear(lane);
      __syncwarp();
      int &wsize = lists[0].size, next = 0, ns = 1;
      wsize = 0;
      if (lane == 0) {
        stage[0] = seeds[s];
        vt.test_and_set(seeds[s]);
      }
      __syncwarp();
      while (true) {
        for (int g0 = 0; g0 < ns; g0 += 32) {
          const int cnt = min(32, ns - g0);
          const uint32_t c = lane < cnt ? stage[g0 + lane] : DG_PAD;
          const float dd = build_dist<ELEM, MET, LPR, TC>(a, qs, hi, qq, c, cnt, lane);
          const uint64_t key = lane < cnt ? make_key(dd, c) : kKeyInvalid;
          const uint64_t thr = wsize >= (int)a.Lb ? strip_flag(W[a.Lb - 1]) : kKeyInvalid;
          cta_survive<1>(lists[0], key, key < thr, cnt_s, lane);
          __syncwarp();
          const int nk[2] = {(int)*cnt_s, 0};
          if (nk[0] > 0) {
            cta_merge<1, 1>(lists, nk, lane, next);
            if (lane == 0) *cnt_s = 0u;
            __syncwarp();
          }
        }
        int idx = -1;
        for (int base = next; base < wsize; base += 32) {
          const int i = base + lane;
          const uint32_t m = __ballot_sync(kFull, i < wsize && !key_expanded(W[i]));
          if (m) {
            idx = base + __ffs(m) - 1;
            break;
          }
        }
        if (idx < 0) break;
        const uint64_t best = W[idx];
        if (wsize >= (int)a.Lb && key_dist(best) >= key_dist(W[a.Lb - 1])) break;
        __syncwarp();
        if (lane == 0) W[idx] = best | 1ull;
        next = idx + 1;
        const uint32_t *row = a.graph + (size_t)key_id(best) * a.R;
        const uint32_t n0 = (uint32_t)lane < a.R ? __ldg(row + lane) : DG_PAD;
        const uint32_t n1 = (uint32_t)lane + 32 < a.R ? __ldg(row + lane + 32) : DG_PAD;
        ns = 0;
        for (uint32_t j0 = 0; j0 < a.R; j0 += 32) {
          const uint32_t j = j0 + lane;
          const uint32_t nb = j0 == 0 ? n0 : j0 == 32 ? n1 : (j < a.R ? __ldg(row + j) : DG_PAD);
          bool ok = nb != DG_PAD && nb < a.n;
          if (ok) ok = !vt.test_and_set(nb);
          const uint32_t m = __ballot_sync(kFull, ok);
          if (ok) stage[ns + __popc(m & ((1u << lane) - 1u))] = nb;
          ns += __popc(m);
        }
        __syncwarp();
      }
      for (int i = lane; i < wsize; i += 32) out[nout + i] = strip_flag(W[i]);
      nout += wsize;
      __syncwarp();
    }
    if (lane == 0) a.cand_cnt[u - a.u0] = nout;
    __syncwarp();
  }
}

// ------------------------------------------------------------------- prune
struct PruneArgs {
  uint64_t u0, nodes;
  const uint64_t *keys;     // candidate keys
  const uint64_t *off;      // per-node offset into keys (nodes entries) or null (fixed stride)
  uint64_t stride;          // fixed stride when off is null
  const uint32_t *cnt;      // per-node count
  uint64_t *gsort;          // global sort scratch for oversized pools: [gridDim][gcap]
  uint32_t gcap;
  const float *vf;
  const uint16_t *vb;
  uint32_t d, dpad, R;
  float alpha;
  int32_t metric;
  uint32_t tile_rows;
  uint32_t *out;            // [n][R]
  uint32_t skip;            // k_prune: pools of up to this many entries are k_prune_small's
};

// Distance between candidate rows j and i (rows staged in `tile` when < tile_rows).
template <int ELEM, int MET>
__device__ __forceinline__ float pair_dist(const PruneArgs &a, const uint32_t *tile, uint32_t tw,
                                           uint32_t j, uint32_t idj, uint32_t i, uint32_t idi) {
  float ab = 0.0f, aa = 0.0f, bb = 0.0f;
  const uint32_t words = ELEM == 1 ? a.dpad / 2 : a.dpad;
  const uint32_t *rj = j < a.tile_rows ? tile + (size_t)j * tw
                                       : (ELEM == 1 ? reinterpret_cast<const uint32_t *>(a.vb + (size_t)idj * a.dpad)
                                                    : reinterpret_cast<const uint32_t *>(a.vf + (size_t)idj * a.dpad));
  const uint32_t *ri = i < a.tile_rows ? tile + (size_t)i * tw
                                       : (ELEM == 1 ? reinterpret_cast<const uint32_t *>(a.vb + (size_t)idi * a.dpad)
                                                    : reinterpret_cast<const uint32_t *>(a.vf + (size_t)idi * a.dpad));
  for (uint32_t t = 0; t < words; ++t) {
    const uint32_t wj = rj[t], wi = ri[t];
    if (ELEM == 1) {
      const float xj0 = __uint_as_float(wj << 16), xj1 = __uint_as_float(wj & 0xffff0000u);
      const float xi0 = __uint_as_float(wi << 16), xi1 = __uint_as_float(wi & 0xffff0000u);
      if (MET == MET_L2) {
        const float t0 = xj0 - xi0, t1 = xj1 - xi1;
        ab = fmaf(t0, t0, ab);
        ab = fmaf(t1, t1, ab);
      } else {
        ab = fmaf(xj0, xi0, ab);
        ab = fmaf(xj1, xi1, ab);
        if (MET == MET_COS) {
          aa = fmaf(xj0, xj0, aa); aa = fmaf(xj1, xj1, aa);
          bb = fmaf(xi0, xi0, bb); bb = fmaf(xi1, xi1, bb);
        }
      }
    } else {
      const float xj = __uint_as_float(wj), xi = __uint_as_float(wi);
      if (MET == MET_L2) {
        const float t0 = xj - xi;
        ab = fmaf(t0, t0, ab);
      } else {
        ab = fmaf(xj, xi, ab);
        if (MET == MET_COS) {
          aa = fmaf(xj, xj, aa);
          bb = fmaf(xi, xi, bb);
        }
      }
    }
  }
  // metric_eval(X[j], X[i]) of the reference's prune_neighbors
  return finish_metric(MET, a.metric == DG_L2, ab, aa, bb);
}

template <int ELEM, int MET>
__global__ void __launch_bounds__(kPruneThreads) k_prune(PruneArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint64_t *skeys = reinterpret_cast<uint64_t *>(smem);               // kPruneSortCap
  float *occ = reinterpret_cast<float *>(skeys + kPruneSortCap);        // kPruneSortCap
  uint8_t *sel = reinterpret_cast<uint8_t *>(occ + kPruneSortCap);      // kPruneSortCap
  uint32_t *tile = reinterpret_cast<uint32_t *>(sel + kPruneSortCap);
  __shared__ uint32_t s_m, s_np;
  __shared__ uint32_t s_out[kStageCap];
  const int tid = threadIdx.x;
  const uint32_t words = ELEM == 1 ? a.dpad / 2 : a.dpad;
  const uint32_t tw = words + 1;  // odd stride: rows land in distinct banks
  for (uint64_t b = blockIdx.x; b < a.nodes; b += gridDim.x) {
    const uint64_t u = a.u0 + b;
    const uint64_t off = a.off ? a.off[b] : b * a.stride;
    const uint32_t c = a.cnt[b];
    if (c <= a.skip) continue;
    const uint64_t *src = a.keys + off;
    // sort the pool (self removed) in shared memory, or in global scratch when large
    uint32_t p2 = 1;
    while (p2 < c) p2 <<= 1;
    uint64_t *K = p2 <= (uint32_t)kPruneSortCap ? skeys : a.gsort + (size_t)blockIdx.x * a.gcap;
    for (uint32_t i = tid; i < p2; i += blockDim.x) {
      uint64_t k = i < c ? strip_flag(src[i]) : kKeyInvalid;
      if (k != kKeyInvalid && key_id(k) == (uint32_t)u) k = kKeyInvalid;
      K[i] = k;
    }
    __syncthreads();
    for (uint32_t k = 2; k <= p2; k <<= 1) {
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {
        for (uint32_t i = tid; i < p2; i += blockDim.x) {
          const uint32_t l = i ^ j;
          if (l > i) {
            const uint64_t x = K[i], y = K[l];
            const bool up = (i & k) == 0;
            if ((x > y) == up) {
              K[i] = y;
              K[l] = x;
            }
          }
        }
        __syncthreads();
      }
    }
    // de-duplicate (same id => same key) and compact, keeping order
    if (tid == 0) {
      uint32_t m = 0;
      uint64_t prev = kKeyInvalid;
      for (uint32_t i = 0; i < p2; ++i) {
        const uint64_t k = K[i];
        if (k == kKeyInvalid) break;
        if (k == prev) continue;
        prev = k;
        K[m++] = k;
      }
      s_m = m;
      s_np = 0;
    }
    __syncthreads();
    const uint32_t m = s_m;
    // per-candidate state lives in shared memory for the first kPruneSortCap
    // candidates; larger pools keep it next to their keys in global scratch
    float *O = m <= (uint32_t)kPruneSortCap ? occ : reinterpret_cast<float *>(a.gsort + (size_t)blockIdx.x * a.gcap + a.gcap / 2);
    uint8_t *S = m <= (uint32_t)kPruneSortCap ? sel : reinterpret_cast<uint8_t *>(O + a.gcap / 2);
    for (uint32_t i = tid; i < m; i += blockDim.x) {
      O[i] = 0.0f;
      S[i] = 0;
    }
    // stage candidate rows
    const uint32_t rows = min(m, a.tile_rows);
    for (uint32_t e = tid; e < rows * words; e += blockDim.x) {
      const uint32_t r = e / words, t = e % words;
      const uint32_t id = key_id(K[r]);
      tile[(size_t)r * tw + t] = ELEM == 1 ? reinterpret_cast<const uint32_t *>(a.vb + (size_t)id * a.dpad)[t]
                                           : __float_as_uint(a.vf[(size_t)id * a.dpad + t]);
    }
    __syncthreads();
    // robust_prune (src/lib.rs:977-1034)
    const float alpha = fmaxf(a.alpha, 1.0f);
    float cur_alpha = 1.0f;
    uint32_t np = 0;
    // Every thread takes the same decisions from S/O: the flag of the entry
    // being decided is written only after the barrier that ends its selection,
    // and each pass ends with a barrier, so no thread can read a flag in the
    // middle of its update and skip a barrier the others wait at.
    while (cur_alpha <= alpha && np < a.R) {
      for (uint32_t i = 0; i < m; ++i) {
        if (np >= a.R) break;
        if (S[i] || O[i] > cur_alpha) continue;
        const uint32_t idi = key_id(K[i]);
        if (tid == 0) s_out[np] = idi;
        ++np;
        for (uint32_t j = i + 1 + tid; j < m; j += blockDim.x) {
          if (S[j] || O[j] > alpha) continue;
          const uint64_t kj = K[j];
          const float djk = pair_dist<ELEM, MET>(a, tile, tw, j, key_id(kj), i, idi);
          O[j] = djk == 0.0f ? __int_as_float(0x7f800000) : fmaxf(O[j], __fdiv_rn(key_dist(kj), djk));
        }
        __syncthreads();
        if (tid == 0) S[i] = 1;
      }
      __syncthreads();
      cur_alpha = __fmul_rn(cur_alpha, 1.2f);
    }
    if (tid == 0) {
      for (uint32_t i = 0; i < m && np < a.R; ++i)
        if (!S[i]) {
          S[i] = 1;
          s_out[np++] = key_id(K[i]);
        }
      s_np = np;
    }
    __syncthreads();
    uint32_t *row = a.out + u * a.R;
    for (uint32_t j = tid; j < a.R; j += blockDim.x) row[j] = j < s_np ? s_out[j] : DG_PAD;
    __syncthreads();
  }
}

// ------------------------------------------------- pools of up to 512 entries
// k_prune for the usual pools.  robust_prune walks the sorted pool and needs,
// for every entry it keeps, the distances from it to all later entries; one
// kept entry at a time leaves a chain of 128 FMAs, a division and a barrier
// per entry (13 ms per pass of 25k nodes x 128).  Here the next eligible
// entries are taken as a batch, all their distances are computed at once, and
// the walk through the batch then only compares: an entry that the batch
// itself occludes is dropped there, as it would have been.
//   TC (integer-valued rows whose sums stay below 2^24, so that any order of
//   summation gives the same bits): batches of 16 on the tensor cores, x.y as
//   BF16 mma with rows and columns read in the same permuted order of
//   coordinates, |x|^2 + |y|^2 - 2 x.y in integers;
//   otherwise batches of 4, a thread per later entry with one FMA chain per
//   batch entry in coordinate order, as pair_dist.
constexpr int kSmallPool = 512;

template <bool TC>
constexpr int prune_batch() { return TC ? 16 : 4; }

// Row stride of the staged rows in 16-byte units: 4 modulo 8 (TC: the four
// chunks of two rows that a quarter warp reads fall in distinct banks), or odd
// (a row per lane).
__host__ __device__ inline uint32_t prune_stride16(uint32_t chunks, bool tc) {
  return tc ? chunks + ((12u - (chunks & 7u)) & 7u) : chunks | 1u;
}

// The ratio kd / d of an occlusion test.  It is only ever compared with alpha
// and with the walk's thresholds 1, 1.2, 1.44, ... up to alpha, so the
// approximate quotient (2 ulp for |d| in [2^-126, 2^126]) stands in for the
// rounded one wherever both lie on the same side of each of them; within 8 ulp
// of one, for extreme divisors, and for alpha above 8 (more than 12
// thresholds), the rounded quotient is taken.  (The rounded division is a call
// of some 280 cycles here; it was two thirds of a pruned node's time.)
__device__ __forceinline__ float prune_ratio(float kd, float d, float alpha) {
  const float r = __fdividef(kd, d), ad = fabsf(d);
  bool exact = !(ad > 1e-30f && ad < 1e30f) || fabsf(r - 1.0f) <= 1e-6f || fabsf(r - 1.2f) <= 1.2e-6f ||
               fabsf(r - alpha) <= 1e-6f * alpha || alpha > 8.0f;
  if (alpha > 1.2f && alpha <= 8.0f)
    for (float t = 1.2f; t <= alpha; t = __fmul_rn(t, 1.2f)) exact |= fabsf(r - t) <= 1e-6f * t;
  if (!exact) return r;
  return d == 0.0f ? __int_as_float(0x7f800000) : __fdiv_rn(kd, d);
}

struct PruneSmem {
  uint64_t ka[kSmallPool], kb[kSmallPool];
  float occ[kSmallPool];
  int norm[kSmallPool];
  float D[16][kSmallPool + 4];  // (padded: the tensor-core stores are conflict-free)
  uint32_t out[kStageCap];
  int bi[16];       // the batch: pool positions
  int nb, cursor;   // its size, where the next one starts
  uint32_t selected;  // which of the batch stay
  float ratio[16][17];  // [q][l]: occlusion of batch entry l by entry q < l
  uint32_t cnt[8];
  uint8_t sel[kSmallPool];
};

template <int ELEM, int MET, bool TC>
__global__ void __launch_bounds__(kPruneThreads, 2) k_prune_small(PruneArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  PruneSmem &P = *reinterpret_cast<PruneSmem *>(smem);
  uint4 *tile = reinterpret_cast<uint4 *>(smem + ((sizeof(PruneSmem) + 15) & ~(size_t)15));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int B = prune_batch<TC>();
  const uint32_t chunks = ELEM == 1 ? a.dpad / 8 : a.dpad / 4, ts = prune_stride16(chunks, TC);
  const uint8_t *rows = ELEM == 1 ? reinterpret_cast<const uint8_t *>(a.vb) : reinterpret_cast<const uint8_t *>(a.vf);
  for (uint64_t b = blockIdx.x; b < a.nodes; b += gridDim.x) {
    const uint64_t u = a.u0 + b;
    const uint32_t c = a.cnt[b];
    if (c > (uint32_t)kSmallPool) continue;
    const uint64_t *src = a.keys + (a.off ? a.off[b] : b * a.stride);
    // ---- sort (self removed): every warp sorts 64 keys in registers (entries
    // lane and lane + 32 of its run), then each key's place is its rank in its
    // own run plus the keys before it in the other runs
    const uint32_t runs = (c + 63) / 64;
    uint64_t k0 = kKeyInvalid, k1 = kKeyInvalid;
    {
      const uint32_t i0 = 64 * warp + lane, i1 = i0 + 32;
      if (i0 < c) k0 = strip_flag(src[i0]);
      if (i1 < c) k1 = strip_flag(src[i1]);
      if (k0 != kKeyInvalid && key_id(k0) == (uint32_t)u) k0 = kKeyInvalid;
      if (k1 != kKeyInvalid && key_id(k1) == (uint32_t)u) k1 = kKeyInvalid;
    }
    if ((uint32_t)warp < runs) {
      k0 = warp_sort_keys(k0, lane);
      k1 = shfl64(warp_sort_keys(k1, lane), 31 - lane);  // descending: k0 then k1 is bitonic
      if (k1 < k0) {
        const uint64_t t = k0;
        k0 = k1;
        k1 = t;
      }
#pragma unroll
      for (int j = 16; j > 0; j >>= 1) {
        const uint64_t o0 = shfl_xor64(k0, j), o1 = shfl_xor64(k1, j);
        const bool low = (lane & j) == 0;
        k0 = (o0 < k0) == low ? o0 : k0;
        k1 = (o1 < k1) == low ? o1 : k1;
      }
      P.ka[64 * warp + lane] = k0;
      P.ka[64 * warp + 32 + lane] = k1;
    }
    __syncthreads();
    if ((uint32_t)warp < runs) {
      int p0 = lane, p1 = lane + 32;
      for (uint32_t r = 0; r < runs; ++r) {
        if (r == (uint32_t)warp) continue;
        const uint64_t *run = P.ka + 64 * r;
        // keys of run r before mine; equal keys of an earlier run go first
        const uint64_t b0 = k0 + (r < (uint32_t)warp ? 1u : 0u), b1 = k1 + (r < (uint32_t)warp ? 1u : 0u);
        int q0 = 0, q1 = 0;
#pragma unroll
        for (int step = 32; step > 0; step >>= 1) {
          q0 += run[q0 + step - 1] < b0 ? step : 0;
          q1 += run[q1 + step - 1] < b1 ? step : 0;
        }
        p0 += q0 + (q0 == 63 && run[63] < b0);
        p1 += q1 + (q1 == 63 && run[63] < b1);
      }
      if (k0 != kKeyInvalid) P.kb[p0] = k0;
      if (k1 != kKeyInvalid) P.kb[p1] = k1;
    }
    // ---- de-duplicate (same id => same key), keeping order: kb[0 .. valid) -> ka
    const int valid = __syncthreads_count(k0 != kKeyInvalid) + __syncthreads_count(k1 != kKeyInvalid);
    uint32_t keep[2];
    uint64_t mine[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = 64 * warp + 32 * h + lane;
      mine[h] = i < valid ? P.kb[i] : kKeyInvalid;
      keep[h] = __ballot_sync(kFull, i < valid && (i == 0 || P.kb[i - 1] != mine[h]));
    }
    if (lane == 0) P.cnt[warp] = __popc(keep[0]) + __popc(keep[1]);
    __syncthreads();
    int before = 0, m = 0;
    for (int w = 0; w < 8; ++w) {
      before += w < warp ? (int)P.cnt[w] : 0;
      m += (int)P.cnt[w];
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if ((keep[h] >> lane) & 1u) P.ka[before + (h ? __popc(keep[0]) : 0) + __popc(keep[h] & lanemask_lt(lane))] = mine[h];
    }
    const uint64_t *K = P.ka;
    for (int i = tid; i < m; i += kPruneThreads) {
      P.occ[i] = 0.0f;
      P.sel[i] = 0;
    }
    __syncthreads();
    // ---- stage rows (and, TC, their squared norms)
    const int staged = min(m, (int)a.tile_rows);
#pragma unroll 8
    for (uint32_t e = tid; e < staged * chunks; e += kPruneThreads) {
      const uint32_t r = e / chunks, t = e - r * chunks;
      cp_async16(tile + r * ts + t, reinterpret_cast<const uint4 *>(rows) + (size_t)key_id(K[r]) * chunks + t, 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    auto row_of = [&](int j) -> const uint4 * {
      return j < staged ? tile + (size_t)j * ts : reinterpret_cast<const uint4 *>(rows) + (size_t)key_id(K[j]) * chunks;
    };
    if (TC) {
      const uint32_t quad = 0xfu << (lane & 28);  // (quads leave the loop at different times)
      for (int j = 8 * warp + (lane >> 2); j < m; j += 64) {  // four lanes per row
        const uint4 *x = row_of(j);
        float s2 = 0.0f;
        for (uint32_t t = lane & 3; t < chunks; t += 4) {
          float v[8];
          Chunk<1>::unpack(x[t], v);
#pragma unroll
          for (int e = 0; e < 8; ++e) s2 = fmaf(v[e], v[e], s2);
        }
        s2 += __shfl_xor_sync(quad, s2, 1);
        s2 += __shfl_xor_sync(quad, s2, 2);
        if ((lane & 3) == 0) P.norm[j] = (int)s2;
      }
    }
    // ---- robust_prune (src/lib.rs:977-1034)
    const float alpha = fmaxf(a.alpha, 1.0f);
    float cur_alpha = 1.0f;
    uint32_t np = 0;
    while (cur_alpha <= alpha && np < a.R) {
      int from = 0;
      while (np < a.R) {
        __syncthreads();  // occlusion and selection of the previous batch (and the norms) are in place
        if (warp == 0) {
          int nb = 0, at = m;
          for (int base = from; base < m && nb < B; base += 32) {
            const int i = base + lane;
            const bool ok = i < m && !P.sel[i] && P.occ[i] <= cur_alpha;
            const uint32_t mk = __ballot_sync(kFull, ok);
            const int rank = nb + __popc(mk & lanemask_lt(lane));
            if (ok && rank < B) P.bi[rank] = i;
            const uint32_t last = __ballot_sync(kFull, ok && rank == B - 1);
            if (last) at = base + __ffs(last);
            nb = min(B, nb + __popc(mk));
          }
          if (lane == 0) {
            P.nb = nb;
            P.cursor = at;
          }
        }
        __syncthreads();
        const int nb = P.nb, next = P.cursor;
        if (nb == 0) break;
        const int j0 = P.bi[0] + 1;
        // ---- distances from the batch to every later entry that can still be kept
        if (TC) {
          const int g = lane >> 2, t = lane & 3;
          const uint4 *col0 = row_of(P.bi[min(g, nb - 1)]), *col1 = row_of(P.bi[min(g + 8, nb - 1)]);
          const bool wide = nb > 8;
          int cn[4];  // squared norms of this lane's columns 2t, 2t + 1 (+ 8)
#pragma unroll
          for (int e = 0; e < 4; ++e) cn[e] = MET == MET_L2 ? P.norm[P.bi[min(2 * t + (e & 1) + (e >> 1) * 8, nb - 1)]] : 0;
          for (int jt = (j0 & ~15) + 16 * warp; jt < m; jt += 16 * 8) {
            const uint4 *r0 = row_of(min(jt + g, m - 1)), *r1 = row_of(min(jt + g + 8, m - 1));
            float d0[4] = {}, d1[4] = {};
#pragma unroll 4
            for (uint32_t ch = t; ch < chunks; ch += 4) {
              const uint4 x0 = r0[ch], x1 = r1[ch], y0 = col0[ch];
              mma_bf16_16x8x16(d0, x0.x, x1.x, x0.y, x1.y, y0.x, y0.y);
              mma_bf16_16x8x16(d0, x0.z, x1.z, x0.w, x1.w, y0.z, y0.w);
              if (wide) {
                const uint4 y1 = col1[ch];
                mma_bf16_16x8x16(d1, x0.x, x1.x, x0.y, x1.y, y1.x, y1.y);
                mma_bf16_16x8x16(d1, x0.z, x1.z, x0.w, x1.w, y1.z, y1.w);
              }
            }
            // lane (g, t): rows jt + g, jt + g + 8 x columns 2t, 2t + 1 (+ 8)
            const int rn[2] = {MET == MET_L2 && jt + g < m ? P.norm[jt + g] : 0,
                               MET == MET_L2 && jt + g + 8 < m ? P.norm[jt + g + 8] : 0};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int col = 2 * t + (e & 1) + (e >= 4 ? 8 : 0), j = jt + g + ((e & 2) ? 8 : 0);
              if (col < nb && j < m) {
                const float dot = e < 4 ? d0[e] : d1[e & 3];
                float v = dot;
                if (MET == MET_L2) v = (float)(rn[(e >> 1) & 1] + cn[(e & 1) + (e >> 2) * 2] - 2 * (int)dot);
                P.D[col][j] = finish_metric(MET, a.metric == DG_L2, v, 0.0f, 0.0f);
              }
            }
          }
        } else {
          const uint4 *col[B];
#pragma unroll
          for (int q = 0; q < B; ++q) col[q] = row_of(P.bi[min(q, nb - 1)]);
          for (int j = j0 + tid; j < m; j += kPruneThreads) {
            if (P.sel[j] || P.occ[j] > alpha) continue;
            const uint4 *x = row_of(j);
            constexpr int E = Chunk<ELEM>::EPC;
            float ab[B], aa = 0.0f, bb[B];
#pragma unroll
            for (int q = 0; q < B; ++q) ab[q] = bb[q] = 0.0f;
            for (uint32_t ch = 0; ch < chunks; ++ch) {
              float xv[E];
              Chunk<ELEM>::unpack(x[ch], xv);
              if (MET == MET_COS) {
#pragma unroll
                for (int e = 0; e < E; ++e) aa = fmaf(xv[e], xv[e], aa);
              }
#pragma unroll
              for (int q = 0; q < B; ++q) {
                float yv[E];
                Chunk<ELEM>::unpack(col[q][ch], yv);
#pragma unroll
                for (int e = 0; e < E; ++e) {
                  if (MET == MET_L2) {
                    const float df = xv[e] - yv[e];
                    ab[q] = fmaf(df, df, ab[q]);
                  } else {
                    ab[q] = fmaf(xv[e], yv[e], ab[q]);
                    if (MET == MET_COS) bb[q] = fmaf(yv[e], yv[e], bb[q]);
                  }
                }
              }
            }
#pragma unroll
            for (int q = 0; q < B; ++q)
              if (q < nb) P.D[q][j] = finish_metric(MET, a.metric == DG_L2, ab[q], aa, bb[q]);
          }
        }
        __syncthreads();
        // ---- which of the batch stay: the occlusions inside the batch, a thread
        // each, then warp 0 walks through them (lane l is entry l)
        if (tid < B * B) {
          const int q = tid / B, l = tid % B;
          if (q < l && l < nb) {
            const int i = P.bi[l];
            P.ratio[q][l] = prune_ratio(key_dist(K[i]), P.D[q][i], alpha);
          }
        }
        __syncthreads();
        if (warp == 0) {
          const int l = min(lane, nb - 1), iq = P.bi[l];
          float oq = P.occ[iq], rt[B];
#pragma unroll
          for (int q = 0; q < B; ++q) rt[q] = q < l && lane < nb ? P.ratio[q][l] : 0.0f;
          uint32_t sel = 0, kept = 0;
#pragma unroll
          for (int q = 0; q < B; ++q) {
            if (q < nb && np + kept < a.R && __shfl_sync(kFull, oq, q) <= cur_alpha) {
              sel |= 1u << q;
              ++kept;
              oq = fmaxf(oq, rt[q]);
            }
          }
          if (lane < nb && ((sel >> lane) & 1u)) P.out[np + __popc(sel & lanemask_lt(lane))] = key_id(K[iq]);
          if (lane == 0) P.selected = sel;
        }
        __syncthreads();
        const uint32_t selected = P.selected, count = __popc(selected);
        // ---- occlusion of the later entries by the kept ones
        for (int j = j0 + tid; j < m; j += kPruneThreads) {
          float o = P.occ[j];
          if (P.sel[j] || o > alpha) continue;
          const float kj = key_dist(K[j]);
#pragma unroll
          for (int q = 0; q < B; ++q)
            if (((selected >> q) & 1u) && P.bi[q] < j) o = fmaxf(o, prune_ratio(kj, P.D[q][j], alpha));
          P.occ[j] = o;
        }
        __syncthreads();  // (selection flags are read above)
        if (warp == 0 && lane < nb && ((selected >> lane) & 1u)) P.sel[P.bi[lane]] = 1;
        np += count;
        from = next;
      }
      cur_alpha = __fmul_rn(cur_alpha, 1.2f);
    }
    __syncthreads();
    // ---- fill with the nearest entries not kept
    if (warp == 0) {
      for (int base = 0; base < m && np < a.R; base += 32) {
        const int i = base + lane;
        const bool ok = i < m && !P.sel[i];
        const uint32_t mk = __ballot_sync(kFull, ok);
        const uint32_t at = np + __popc(mk & lanemask_lt(lane));
        if (ok && at < a.R) P.out[at] = key_id(K[i]);
        np = min(a.R, np + (uint32_t)__popc(mk));
      }
      __syncwarp();  // the entries above are other lanes'
      for (uint32_t j = lane; j < a.R; j += 32) a.out[u * a.R + j] = j < np ? P.out[j] : DG_PAD;
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------- symmetrisation
__global__ void k_degrees(const uint32_t *g, uint64_t n, uint32_t R, uint32_t *outdeg, uint32_t *indeg) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n * R;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = g[e];
    if (v != DG_PAD) {
      atomicAdd(indeg + v, 1u);
      atomicAdd(outdeg + e / R, 1u);
    }
  }
}
__global__ void k_pool_sizes(const uint32_t *outdeg, const uint32_t *indeg, uint64_t n, uint64_t *sz) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    sz[i] = (uint64_t)outdeg[i] + indeg[i];
}
// pool ids of node u: its outgoing list, then everyone pointing at u
__global__ void k_fill_pools(const uint32_t *g, uint64_t n, uint32_t R, const uint64_t *off,
                             const uint32_t *outdeg, uint32_t *cursor, uint32_t *pool_ids) {
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n * R;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = g[e];
    if (v == DG_PAD) continue;
    const uint64_t u = e / R;
    pool_ids[off[u] + (e % R)] = v;  // outgoing lists are packed at the row front
    const uint32_t pos = atomicAdd(cursor + v, 1u);
    pool_ids[off[v] + outdeg[v] + pos] = (uint32_t)u;
  }
}
// distances of every pool entry to its node (warp per node)
template <int ELEM, int MET, int LPR>
__global__ void k_pool_keys(const float *vf, const uint16_t *vb, uint64_t n, uint32_t dpad, int metric,
                            const uint64_t *off, const uint32_t *pool_ids, uint64_t *keys, uint32_t *cnt) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  extern __shared__ __align__(16) float qsm[];
  float *qs = qsm + (size_t)warp * dpad;
  const uint64_t gw = blockIdx.x * (uint64_t)(blockDim.x >> 5) + warp;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t u = gw; u < n; u += nw) {
    for (uint32_t i = lane; i < dpad; i += 32) qs[i] = vf[u * dpad + i];
    __syncwarp();
    float qq = 0.0f;
    if (MET == MET_COS) {
      for (uint32_t i = lane; i < dpad; i += 32) qq = fmaf(qs[i], qs[i], qq);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) qq += __shfl_xor_sync(kFull, qq, o);
    }
    const uint64_t b = off[u], e = off[u + 1];
    for (uint64_t g0 = b; g0 < e; g0 += 32) {
      const int c = (int)((e - g0) < 32 ? (e - g0) : 32);
      const uint32_t id = lane < c ? pool_ids[g0 + lane] : 0u;
      const float dd = rows_distance<LPR, ELEM == 1 ? 1 : 0, MET>(
          ELEM == 1 ? reinterpret_cast<const uint8_t *>(vb) : reinterpret_cast<const uint8_t *>(vf),
          ELEM == 1 ? dpad * 2 : dpad * 4, ELEM == 1 ? (dpad / 8) / LPR : (dpad / 4) / LPR, qs, id, c, lane,
          metric == DG_L2, qq);
      if (lane < c) keys[g0 + lane] = make_key(dd, id);
    }
    if (lane == 0) cnt[u] = (uint32_t)(e - b);
    __syncwarp();
  }
}

// What the build may assume of the values: out[0] bit 0 set when one is not
// exact in BF16, bit 1 when one is not an integer; out[1], out[2]: ordered bits
// of the largest and of the smallest.
__global__ void k_value_range(const float *v, uint64_t total, uint32_t *out) {
  uint32_t f = 0, hi = 0, lo = 0xffffffffu;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float x = v[i];
    f |= __uint_as_float(__float_as_uint(x) & 0xffff0000u) != x ? 1u : 0u;
    f |= x != rintf(x) ? 2u : 0u;
    hi = max(hi, ordered_bits(x));
    lo = min(lo, ordered_bits(x));
  }
  f = __reduce_or_sync(kFull, f);
  hi = __reduce_max_sync(kFull, hi);
  lo = __reduce_min_sync(kFull, lo);
  if ((threadIdx.x & 31) == 0) {
    if (f) atomicOr(out, f);
    atomicMax(out + 1, hi);
    atomicMin(out + 2, lo);
  }
}

static uint32_t id_bits(uint64_t n) {
  uint32_t b = 1;
  while (b < 32 && (1ull << b) < n) ++b;
  return b;
}

template <int ELEM, int MET>
static DgStatus run_build(const BuildArgs &base, float *vf, uint16_t *vb, bool tc, uint32_t *g0, uint32_t *g1,
                          float alpha, cudaStream_t st, uint32_t **result) {
  const uint64_t n = base.n;
  const uint32_t R = base.R, dpad = base.dpad;
  constexpr int LPR = ELEM == 1 ? 4 : 8;
  int dev = 0, sms = 0;
  DG_CUDA(cudaGetDevice(&dev));
  DG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // candidate pools of the search phase, processed in node chunks
  const uint32_t cw = R + 3 * base.Lb;
  const uint64_t chunk = std::min<uint64_t>(n, 1ull << 18);
  uint64_t *cand = nullptr;
  uint32_t *ccnt = nullptr;
  DG_CUDA(cudaMallocAsync(&cand, chunk * cw * 8, st));
  DG_CUDA(cudaMallocAsync(&ccnt, chunk * 4, st));
  // prune geometry
  const uint32_t words = ELEM == 1 ? dpad / 2 : dpad;
  uint32_t tile_rows = (uint32_t)(kPruneTileBytes / ((words + 1) * 4));
  if (tile_rows < 1) tile_rows = 1;
  const size_t psmem = (size_t)kPruneSortCap * (8 + 4 + 1) + (size_t)tile_rows * (words + 1) * 4;
  auto prune_k = k_prune<ELEM, MET>;
  DG_CUDA(cudaFuncSetAttribute(prune_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psmem));
  int pblocks = 0;
  DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pblocks, prune_k, kPruneThreads, psmem));
  const int pgrid = std::max(1, pblocks) * sms;
  // pools of up to kSmallPool entries: two CTAs per SM, the rest of whose shared
  // memory stages rows
  void (*small_k)(PruneArgs) = k_prune_small<ELEM, MET, false>;
  if constexpr (ELEM == 1 && MET != MET_COS)
    if (tc) small_k = k_prune_small<ELEM, MET, true>;
  const uint32_t row16 = prune_stride16(ELEM == 1 ? dpad / 8 : dpad / 4, tc);
  const size_t fixed = (sizeof(PruneSmem) + 15) & ~(size_t)15;
  const uint32_t small_rows = (uint32_t)std::min<size_t>(kSmallPool, (112 * 1024 - fixed) / (row16 * 16));
  const size_t ssmem = fixed + (size_t)small_rows * row16 * 16;
  DG_CUDA(cudaFuncSetAttribute(small_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssmem));
  auto prune = [&](PruneArgs p, uint64_t nodes, uint64_t largest) -> DgStatus {
    PruneArgs q = p;
    q.tile_rows = small_rows;
    small_k<<<(int)std::min<uint64_t>(2ull * sms, nodes), kPruneThreads, ssmem, st>>>(q);
    DG_CUDA(cudaGetLastError());
    if (largest > (uint64_t)kSmallPool) {
      p.skip = kSmallPool;
      prune_k<<<(int)std::min<uint64_t>(pgrid, nodes), kPruneThreads, psmem, st>>>(p);
      DG_CUDA(cudaGetLastError());
    }
    return DG_OK;
  };
  // search kernel geometry
  // (a larger visited table for beams above 128 leaves two CTAs per SM instead of
  // four or five; a forgotten id costs its distance again.  Searches of 20k real
  // rows x 128, R = 64, 2^12 / 2^11 words: beam 200 121 / 58 ms, 256 149 / 84, 400
  // 249 / 141, 800 517 / 403; integer rows, beam 256, 77 / 46)
  const uint32_t hbits = base.Lb <= 64 ? 10 : 11;
  const BuildLayout Ly = build_layout(base.Lb, R, hbits, dpad, tc);
  void (*sk)(BuildArgs, BuildLayout) = k_build_search<ELEM, MET, LPR, false>;
  if constexpr (ELEM == 1 && MET != MET_COS)
    if (tc) sk = k_build_search<ELEM, MET, LPR, true>;
  // (accepted or refused by the state of a two-list search, as ever)
  const uint32_t lcap = base.Lb <= 64 ? 64 : base.Lb <= 256 ? 256 : 1024;
  const WarpLayout limit = warp_layout(ELEM == 1 ? TRAV_BF16 : TRAV_F32, lcap, false, base.Lb <= 128 ? hbits : 12, dpad,
                                       0, 0, 0);
  DG_CUDA(cudaFuncSetAttribute(sk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)std::max(limit.total * 4, Ly.total * 4)));
  int sblocks = 0;
  DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sblocks, sk, 128, Ly.total * 4));
  if (sblocks < 1) return fail(DG_ENOTSUP, "build search state does not fit in shared memory");
  // symmetrisation buffers
  uint32_t *outdeg = nullptr, *indeg = nullptr, *cursor = nullptr, *pool_ids = nullptr, *pcnt = nullptr;
  uint64_t *psz = nullptr, *poff = nullptr, *pkeys = nullptr;
  DG_CUDA(cudaMallocAsync(&outdeg, n * 4, st));
  DG_CUDA(cudaMallocAsync(&indeg, n * 4, st));
  DG_CUDA(cudaMallocAsync(&cursor, n * 4, st));
  DG_CUDA(cudaMallocAsync(&pcnt, n * 4, st));
  DG_CUDA(cudaMallocAsync(&psz, (n + 1) * 8, st));
  DG_CUDA(cudaMallocAsync(&poff, (n + 1) * 8, st));
  DG_CUDA(cudaMallocAsync(&pool_ids, n * R * 2 * 4, st));
  DG_CUDA(cudaMallocAsync(&pkeys, n * R * 2 * 8, st));
  size_t scan_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, psz, poff, n + 1, st);
  void *scan_tmp = nullptr;
  DG_CUDA(cudaMallocAsync(&scan_tmp, scan_bytes, st));
  // global sort scratch for pools above the shared-memory capacity
  const uint32_t gcap = (uint32_t)std::max<uint64_t>(4096, 2 * (uint64_t)(cw + 2 * R));
  uint64_t *gsort = nullptr;
  // sized generously: pools larger than this are clipped by a pre-check below
  uint32_t gcap_sym = gcap;
  uint32_t *cur = g0, *nxt = g1;
  for (uint32_t pass = 0; pass < 2; ++pass) {
    BuildArgs a = base;
    a.pass = pass;
    a.graph = cur;
    a.hbits = hbits;
    a.hB = std::max(id_bits(n), hbits);
    a.cw = cw;
    a.cand = cand;
    a.cand_cnt = ccnt;
    for (uint64_t u0 = 0; u0 < n; u0 += chunk) {
      a.u0 = u0;
      a.u1 = std::min(n, u0 + chunk);
      const uint64_t nodes = a.u1 - a.u0;
      const int grid = (int)std::min<uint64_t>((uint64_t)sblocks * sms, (nodes + 3) / 4);
      sk<<<grid, 128, Ly.total * 4, st>>>(a, Ly);
      DG_CUDA(cudaGetLastError());
      PruneArgs p{};
      p.u0 = u0;
      p.nodes = nodes;
      p.keys = cand;
      p.off = nullptr;
      p.stride = cw;
      p.cnt = ccnt;
      p.vf = vf;
      p.vb = vb;
      p.d = base.d;
      p.dpad = dpad;
      p.R = R;
      p.alpha = alpha;
      p.metric = base.metric;
      p.tile_rows = tile_rows;
      p.out = nxt;
      if (cw > (uint32_t)kPruneSortCap) {
        if (!gsort) DG_CUDA(cudaMallocAsync(&gsort, (size_t)pgrid * gcap * 8, st));
        p.gsort = gsort;
        p.gcap = gcap;
      }
      DgStatus ps = prune(p, nodes, cw);
      if (ps != DG_OK) return ps;
    }
    // symmetrise: union of outgoing and incoming, distances, prune into `cur`
    DG_CUDA(cudaMemsetAsync(outdeg, 0, n * 4, st));
    DG_CUDA(cudaMemsetAsync(indeg, 0, n * 4, st));
    DG_CUDA(cudaMemsetAsync(cursor, 0, n * 4, st));
    DG_CUDA(cudaMemsetAsync(psz, 0, (n + 1) * 8, st));
    k_degrees<<<sms * 8, 256, 0, st>>>(nxt, n, R, outdeg, indeg);
    k_pool_sizes<<<sms * 8, 256, 0, st>>>(outdeg, indeg, n, psz);
    cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, psz, poff, n + 1, st);
    k_fill_pools<<<sms * 8, 256, 0, st>>>(nxt, n, R, poff, outdeg, cursor, pool_ids);
    const int kw = 4;
    k_pool_keys<ELEM, MET, LPR><<<sms * 16, kw * 32, kw * dpad * 4, st>>>(vf, vb, n, dpad, base.metric, poff,
                                                                         pool_ids, pkeys, pcnt);
    DG_CUDA(cudaGetLastError());
    // the largest pool decides whether global sort scratch is needed
    uint32_t max_in = 0;
    {
      std::vector<uint32_t> hin(n);
      DG_CUDA(cudaMemcpyAsync(hin.data(), indeg, n * 4, cudaMemcpyDeviceToHost, st));
      DG_CUDA(cudaStreamSynchronize(st));
      for (uint32_t v : hin) max_in = std::max(max_in, v);
    }
    uint64_t maxpool = (uint64_t)R + max_in;
    PruneArgs p{};
    p.u0 = 0;
    p.nodes = n;
    p.keys = pkeys;
    p.off = poff;
    p.cnt = pcnt;
    p.vf = vf;
    p.vb = vb;
    p.d = base.d;
    p.dpad = dpad;
    p.R = R;
    p.alpha = alpha;
    p.metric = base.metric;
    p.tile_rows = tile_rows;
    p.out = cur;
    if (maxpool > (uint64_t)kPruneSortCap) {
      uint32_t need = 1;
      while (need < maxpool) need <<= 1;
      need = std::max<uint32_t>(need * 2, 4096);  // keys, then occlusion + flags
      if (need > gcap_sym || !gsort) {
        if (gsort) DG_CUDA(cudaFreeAsync(gsort, st));
        gcap_sym = need;
        DG_CUDA(cudaMallocAsync(&gsort, (size_t)pgrid * gcap_sym * 8, st));
      }
      p.gsort = gsort;
      p.gcap = gcap_sym;
    }
    DgStatus ps = prune(p, n, maxpool);
    if (ps != DG_OK) return ps;
  }
  DG_CUDA(cudaStreamSynchronize(st));
  cudaFreeAsync(cand, st);
  cudaFreeAsync(ccnt, st);
  cudaFreeAsync(outdeg, st);
  cudaFreeAsync(indeg, st);
  cudaFreeAsync(cursor, st);
  cudaFreeAsync(pcnt, st);
  cudaFreeAsync(psz, st);
  cudaFreeAsync(poff, st);
  cudaFreeAsync(pool_ids, st);
  cudaFreeAsync(pkeys, st);
  cudaFreeAsync(scan_tmp, st);
  if (gsort) cudaFreeAsync(gsort, st);
  *result = cur;
  return DG_OK;
}

}  // namespace dg

using namespace dg;

extern "C" DgStatus dg_build_vamana(const float *X, uint64_t n, uint32_t dim, int32_t metric, uint32_t R,
                                    uint32_t build_beam, float alpha, uint64_t seed, uint32_t medoid,
                                    int32_t device, uint32_t *out_adjacency) {
  if (!X || !out_adjacency || n == 0 || dim == 0) return fail(DG_EINVAL, "bad build arguments");
  if (n >= (1ull << 31)) return fail(DG_EINVAL, "num_vectors must be < 2^31");
  if (R == 0 || R > (uint32_t)kStageCap) return fail(DG_EINVAL, "max_degree must be in [1, 256]");
  if (build_beam == 0 || build_beam > 1024) return fail(DG_EINVAL, "build_beam_width must be in [1, 1024]");
  if (medoid >= n) return fail(DG_EINVAL, "medoid out of range");
  if (metric < DG_L2SQ || metric > DG_DOT) return fail(DG_EINVAL, "unknown metric");
  // the relaxed passes multiply their threshold until it exceeds alpha, which it
  // never does when both are infinite; the largest float keeps the same entries
  // (what the pass at infinity would add, the fill adds in the same order)
  alpha = std::min(alpha, 3.402823466e38f);
  DG_CUDA(cudaSetDevice(device));
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  const uint32_t dpad = dpad_of(dim);
  float *vf = nullptr;
  uint16_t *vb = nullptr;
  uint32_t *g0 = nullptr, *g1 = nullptr;
  uint32_t *flag = nullptr;
  float *vbn = nullptr;
  DgStatus s = DG_OK;
  if (cudaMallocAsync(&vf, n * dpad * 4, st) != cudaSuccess || cudaMallocAsync(&g0, n * R * 4, st) != cudaSuccess ||
      cudaMallocAsync(&g1, n * R * 4, st) != cudaSuccess || cudaMallocAsync(&flag, 12, st) != cudaSuccess)
    s = fail(DG_ENOMEM, "build staging");
  if (s == DG_OK) s = upload_rows_f32(X, n, dim, dpad, vf, st);
  bool exact_bf16 = false, tc = false;
  if (s == DG_OK) {
    // BF16 rows carry the same values when every coordinate is bf16-exact
    // (integer data in [-256, 256], BF16-stored embeddings): half the gather bytes.
    uint32_t hf[3] = {0u, 0u, 0xffffffffu};
    cudaMemcpyAsync(flag, hf, 12, cudaMemcpyHostToDevice, st);
    k_value_range<<<148 * 8, 256, 0, st>>>(vf, n * dpad, flag);
    hf[0] = 3u;
    cudaMemcpyAsync(hf, flag, 12, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    exact_bf16 = !(hf[0] & 1u) && metric != DG_COSINE;
    // integers whose sums of products and of squared differences stay below
    // 2^24: every partial sum is exact, so the order of summation is free and
    // the tensor cores return the FMA chain's bits
    auto value = [](uint32_t o) {
      const uint32_t b = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
      float f;
      std::memcpy(&f, &b, 4);
      return (double)f;
    };
    const double hi = value(hf[1]), lo = value(hf[2]), mx = std::max(std::fabs(hi), std::fabs(lo));
    tc = exact_bf16 && !(hf[0] & 2u) && (double)dim * mx * mx < 16777216.0 &&
         (double)dim * (hi - lo) * (hi - lo) < 16777216.0;
    if (exact_bf16) {
      if (cudaMallocAsync(&vb, n * dpad * 2, st) != cudaSuccess || cudaMallocAsync(&vbn, n * 4, st) != cudaSuccess)
        s = fail(DG_ENOMEM, "build staging");
      else
        s = encode_bf16_device(vf, n, dpad, vb, st, tc ? vbn : nullptr);
    }
  }
  if (s == DG_OK) {
    const uint32_t target = (uint32_t)std::min<uint64_t>(std::max<uint32_t>(R / 2, 2u), n - 1);
    k_bootstrap<<<148 * 8, 256, 0, st>>>(n, R, target, seed, g0);
    if (cudaGetLastError() != cudaSuccess) s = fail(DG_EDEVICE, "bootstrap launch");
  }
  uint32_t *result = nullptr;
  if (s == DG_OK) {
    BuildArgs a{};
    a.n = n;
    a.d = dim;
    a.dpad = dpad;
    a.R = R;
    a.Lb = build_beam;
    a.medoid = medoid;
    a.seed = seed;
    a.metric = metric;
    a.vf = vf;
    a.vb = vb;
    a.vbn = vbn;
    const int met = metric == DG_DOT ? MET_DOT : metric == DG_COSINE ? MET_COS : MET_L2;
    if (exact_bf16) {
      s = met == MET_DOT ? run_build<1, MET_DOT>(a, vf, vb, tc, g0, g1, alpha, st, &result)
                         : run_build<1, MET_L2>(a, vf, vb, tc, g0, g1, alpha, st, &result);
    } else {
      s = met == MET_DOT   ? run_build<0, MET_DOT>(a, vf, vb, tc, g0, g1, alpha, st, &result)
          : met == MET_COS ? run_build<0, MET_COS>(a, vf, vb, tc, g0, g1, alpha, st, &result)
                           : run_build<0, MET_L2>(a, vf, vb, tc, g0, g1, alpha, st, &result);
    }
  }
  if (s == DG_OK) {
    if (cudaMemcpyAsync(out_adjacency, result, n * R * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      s = fail(DG_EDEVICE, std::string("build failed: ") + cudaGetErrorString(cudaGetLastError()));
  }
  if (vf) cudaFreeAsync(vf, st);
  if (vb) cudaFreeAsync(vb, st);
  if (vbn) cudaFreeAsync(vbn, st);
  if (g0) cudaFreeAsync(g0, st);
  if (g1) cudaFreeAsync(g1, st);
  if (flag) cudaFreeAsync(flag, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}
