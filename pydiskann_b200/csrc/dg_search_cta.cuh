// dg_search_cta.cuh -- beam search with one CTA of NW warps per query.
//
// The warp-per-query kernel keeps a list of up to 64 entries in one warp's
// registers and fills the GPU with 24 queries per SM.  Wider beams, filtered
// searches and small batches take this kernel: the list (up to 1024 entries)
// lives in shared memory and is merged in place, and the warps of a CTA share
// one query's state.  Warp 0 picks the node to expand and stages its unvisited
// neighbours, each warp takes its share of them through row gather and
// distance, so the gathers of one expansion are all in flight at once, and all
// threads merge the surviving keys into the list.  Results are those of
// search_one_reg: the same distances (same summation order per row), the same
// L smallest (distance, id) pairs after every expansion, the same stopping
// rules and, at one size of the visited table, the same counts.
//
// What bounds it is the chain of one expansion, not bandwidth (cycles on one
// 8-warp CTA of the 100k x 128 FP32 search, beam 128: neighbour list and visited
// test 1120, row distances 1160, merge 720, selection 300; DRAM 6 %, issue 35 %
// in a filtered batch).  Against the kernel before it (one warp per query, two
// copies of the list in shared memory, merged entry by entry): one query of that
// search 547 -> 345 us; 4000 768-d int8 cosine queries with beams up to 256 16.9
// -> 6.7 ms; 5000 PQ queries, beam 128, 7.7 -> 2.6 ms; 500 filtered queries,
// k = 100, 16.4 -> 7.9 ms; 2000 filtered queries, k = 10, 5.9 -> 4.1 ms.
#pragma once
#include "dg_search_kernel.cuh"

namespace dg {

constexpr uint32_t kCtaOps = 16;  // filter programs up to this long are staged in shared memory

// Words of the control block: staged candidates (or kCtaStop), keys surviving
// for the list and for the result list, the query index, then a bitmap of the
// list slots that new keys take (and one of the result list's).
enum CtaCtl { CTL_NS = 0, CTL_CNT = 1, CTL_CNTR = 2, CTL_Q = 3, CTL_MAP = 4, CTL_WORDS = CTL_MAP + 32 };
constexpr uint32_t kCtaStop = 0xffffffffu;

// One survivor buffer: up to `degree` keys, then their list positions (u16).
__host__ __device__ inline uint32_t cta_surv_bytes(uint32_t degree) {
  const uint32_t n = degree < 2 ? 2 : degree;
  return align16(n * 8) + align16(n * 2);
}

// Shared-memory carve-up of one query: the list (w0, wcap keys), the keys that
// enter it after one expansion (w1; then those of the result list), the result
// list (res, rcap keys, filtered searches), the staged candidates, the visited
// table (the rerank's keys reuse it), the query and the quantizer state, the
// staged filter program (cstage), the control block (aux).
inline WarpLayout cta_layout(int trav, uint32_t wcap, uint32_t rcap, uint32_t rerank_keys, bool filt, uint32_t hbits,
                             uint32_t dpad, uint32_t pq_M, uint32_t pq_K, uint32_t rq_padded, bool decode,
                             uint32_t degree) {
  const WarpLayout B = warp_layout(trav, 64, false, hbits, dpad, pq_M, pq_K, rq_padded, decode, degree, true);
  const uint32_t prov_bytes = B.aux - B.prov;
  WarpLayout L{};
  uint32_t o = 0;
  L.w0 = o; o += align16(std::max(wcap, 2u) * 8);
  L.w1 = o; o += cta_surv_bytes(degree) * (filt ? 2 : 1);
  L.res = o; o += align16(rcap * 8);
  L.stage = o; o += align16(std::max(degree, 2u) * 4);
  L.hash = o; o += std::max((1u << hbits) * 4, align16(rerank_keys * 8));
  L.qf = o; o += align16(dpad * 4);
  L.prov = o; o += prov_bytes;
  L.cstage = o; o += filt ? align16(kCtaOps * (uint32_t)sizeof(DgFilterOp)) : 0;
  L.aux = o; o += align16((CTL_WORDS + (filt ? 32 : 0)) * 4);
  L.total = align16(o);
  return L;
}

// Barrier of one query's warps.
template <int NW>
__device__ __forceinline__ void cta_sync() {
  if (NW == 1) __syncwarp();
  else __syncthreads();
}
template <int NW>
__device__ __forceinline__ int cta_sync_count(bool v) {
  if (NW != 1) return __syncthreads_count(v);
  const int n = __popc(__ballot_sync(kFull, v));
  __syncwarp();  // (a ballot orders no memory)
  return n;
}

// Candidates a warp takes at a time.  8 long rows of an eighth, or 16, keep a quarter (an eighth, a half) of
// an expansion in flight at once.  32 where a lane scores a whole code, and
// for a warp that has the expansion to itself, unless its rows are long (8
// lanes per row): two tiles of 16 short rows wait for memory once, not twice
// (300k x 128, beam 100, 6000 queries, 16 -> 32: int8 2436 -> 1619 us; but FP32
// rows of 512 bytes 2466 -> 2576, F16 2524 -> 2730).
template <int NW, int TRAV, int LPR, bool TC>
constexpr int cta_batch() {
  if (TRAV == TRAV_PQ || TRAV == TRAV_RABITQ) return 32;
  const bool rows = TRAV == TRAV_F32 || TRAV == TRAV_F16 || (TRAV == TRAV_BF16 && !TC);
  if (NW == 8 && rows && LPR == 8) return 8;
  return NW == 1 && !(rows && LPR == 8) ? 32 : 16;
}

// Distances of a warp's cnt <= B candidates (lane j holds cand).
template <int B, int TRAV, int MET, int LPR, bool TC>
__device__ __forceinline__ float cta_distance(const SearchArgs &a, uint8_t *sm, const WarpLayout &Ly, uint32_t cand,
                                              int cnt, int lane, float qq) {
  const float *qs = reinterpret_cast<const float *>(sm + Ly.qf);
  const bool sq = a.metric == DG_L2;
  if constexpr (B == 32) {
    return batch_distance<TRAV, MET, LPR, TC>(a, sm, Ly, cand, cnt, lane, qq);
  } else if constexpr (TRAV == TRAV_F32) {
    return rows_distance_few<B == 8 ? 2 : LPR / 2, LPR, 0, MET>(reinterpret_cast<const uint8_t *>(a.vec_f32), a.dpad * 4, (a.dpad / 4) / LPR,
                                        qs, cand, cnt, lane, sq, qq);
  } else if constexpr (TRAV == TRAV_BF16 && !TC) {
    return rows_distance_few<B == 8 ? 2 : LPR / 2, LPR, 1, MET>(reinterpret_cast<const uint8_t *>(a.vec_bf16), a.dpad * 2,
                                        (a.dpad / 8) / LPR, qs, cand, cnt, lane, sq, qq);
  } else if constexpr (TRAV == TRAV_F16) {
    const float *qx = MET == MET_L2 ? reinterpret_cast<const float *>(sm + Ly.prov) : qs;
    return rows_distance_few<B == 8 ? 2 : LPR / 2, LPR, 2, MET>(a.codes, a.code_stride, (a.code_stride / 16) / LPR, qx, cand, cnt, lane, sq,
                                        qq);
  } else {
    return batch_distance<TRAV, MET, LPR, TC, true>(a, sm, Ly, cand, cnt, lane, qq);
  }
}

// lower_bound_smem by eight-way steps: the seven probes of a step are
// independent loads, so a 1024-entry list costs four shared-memory round trips.
__device__ __forceinline__ int lower_bound8(const uint64_t *a, int n, uint64_t key) {
  int lo = 0;
  for (int step = n <= 8 ? 1 : n <= 64 ? 8 : n <= 512 ? 64 : 512; step > 0; step >>= 3) {
    int add = 0;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
      const int at = lo + i * step - 1;
      add += at < n && a[at] < key;
    }
    lo += add * step;
    if (step == 1) lo += lo < n && a[lo] < key;  // the eighth of the last eight
  }
  return lo;
}

// One sorted list of a query (at most 1024 keys) and the keys about to enter it.
struct CtaList {
  uint64_t *p;         // the list
  int size, cap;
  uint64_t *key;       // new keys, each below the full list's last and not listed
  uint16_t *pos;       // their positions in the list (lower bounds)
  uint32_t *map;       // 32 words, zero between merges
};

// A lane's key enters `L` unless it is already listed or not below a full
// list's last: recorded with its position (cnt: the shared number of records).
// With few warps per query instructions are what a search waits for, and the
// binary search has fewer; with more, its chain of loads is.
template <int NW>
__device__ __forceinline__ void cta_survive(const CtaList &L, uint64_t key, bool want, uint32_t *cnt, int lane) {
  if (!__any_sync(kFull, want)) return;
  int pos = 0;
  if (want) {
    pos = NW > 2 ? lower_bound8(L.p, L.size, key) : lower_bound_smem(L.p, L.size, key);
    want = pos < L.cap && !(pos < L.size && strip_flag(L.p[pos]) == key);
  }
  const uint32_t m = __ballot_sync(kFull, want);
  if (!m) return;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(cnt, (uint32_t)__popc(m));
  at = __shfl_sync(kFull, at, 0) + __popc(m & lanemask_lt(lane));
  if (want) {
    L.key[at] = key;
    L.pos[at] = (uint16_t)pos;
  }
}

// The slot a new key takes: its position plus its rank among the new keys of
// this batch (each thread has one), marked in the bitmap.  Returns the slot
// (cap or above: dropped); dup: an equal key marked it first.
__device__ __forceinline__ int cta_slot(const CtaList &L, int b0, int nb, int t, bool &dup) {
  dup = false;
  if (t >= nb) return 1 << 20;
  const uint64_t *sv = L.key + b0;
  const uint64_t u = sv[t];
  int rank = 0;
#pragma unroll 4
  for (int i = 0; i < nb; ++i) rank += sv[i] < u;
  if (u == kKeyInvalid) return 1 << 20;
  const int slot = L.pos[b0 + t] + rank;
  if (slot < L.cap) dup = (atomicOr(L.map + (slot >> 5), 1u << (slot & 31)) >> (slot & 31)) & 1u;
  return slot;
}

// Merges the s new keys of each list into it, in place, by all NW warps of the
// query.  A new key's slot is its position in the list plus its rank among the
// new keys; the slots go to a bitmap, and the entry that ends in any other
// slot o is the one at o less the number of new slots below o.  Slots are
// rewritten in rounds of 32 NW E from the last one down to the first that
// changes, all reads of a round before its writes (an entry only moves up, so
// later rounds read nothing that earlier ones wrote); the new keys are written
// last.  Keys that repeat within the batch (a neighbour listed twice) are
// dropped, in a slow path.  All threads see the same lists before and after;
// first: the smallest slot that changed in lists[0], or unchanged.
template <int NW, int NL>
__device__ __forceinline__ void cta_merge(CtaList (&lists)[2], const int (&s)[2], int tid, int &first) {
  constexpr int T = 32 * NW, E = NW == 1 ? 4 : 2;
  const int lane = tid & 31, warp = tid >> 5;
  const int smax = NL == 2 ? max(s[0], s[1]) : s[0];
  for (int b0 = 0; b0 < smax; b0 += T) {
    int slot[NL], nb[NL];
    bool dup = false, d[NL];
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      nb[l] = max(0, min(T, s[l] - b0));
      if (b0 > 0 && tid < nb[l]) {  // a second batch: the list has grown
        CtaList &L = lists[l];
        const int p = lower_bound8(L.p, L.size, L.key[b0 + tid]);
        if (p >= L.cap || (p < L.size && strip_flag(L.p[p]) == L.key[b0 + tid])) L.key[b0 + tid] = kKeyInvalid;
        L.pos[b0 + tid] = (uint16_t)min(p, 65535);
      }
    }
    if (b0 > 0) cta_sync<NW>();
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      slot[l] = cta_slot(lists[l], b0, nb[l], tid, d[l]);
      dup |= d[l];
    }
    // drop the repeats and place the rest again; the ranks they inflated may
    // have hidden others past the capacity, so until none is left
    while (cta_sync_count<NW>(dup) > 0) {
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        if (d[l]) lists[l].key[b0 + tid] = kKeyInvalid;
        if (warp == 0) lists[l].map[lane] = 0u;
      }
      cta_sync<NW>();
      dup = false;
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        slot[l] = cta_slot(lists[l], b0, nb[l], tid, d[l]);
        dup |= d[l];
      }
    }
    uint32_t word[NL], below[NL];  // lane w: word w of the bitmap, set bits of the words before it
    int lo[NL], hi[NL], na[NL];
    int rounds = 0;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      word[l] = lists[l].map[lane];
      uint32_t incl = __popc(word[l]);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
      }
      below[l] = incl - __popc(word[l]);
      na[l] = (int)__shfl_sync(kFull, incl, 31);
      const uint32_t nz = __ballot_sync(kFull, word[l] != 0u);
      lo[l] = nz ? __ffs(nz) - 1 : 32;  // first word that changes
      if (l == 0 && nz) first = min(first, 32 * lo[l] + __ffs(__shfl_sync(kFull, word[l], lo[l] & 31)) - 1);
      lists[l].size = min(lists[l].cap, lists[l].size + na[l]);
      hi[l] = na[l] ? (lists[l].size - 1) >> 5 : -1;
      rounds = max(rounds, (hi[l] - lo[l] + NW * E) / (NW * E));
    }
    for (int r = 0; r < rounds; ++r) {
      uint64_t e[NL][E];
      bool put[NL][E];
#pragma unroll
      for (int l = 0; l < NL; ++l)
#pragma unroll
        for (int c = 0; c < E; ++c) {
          const int w = hi[l] - (r * E + c) * NW - warp;  // this warp's word of 32 slots
          const uint32_t m = __shfl_sync(kFull, word[l], w & 31), bl = __shfl_sync(kFull, below[l], w & 31);
          const int o = 32 * w + lane;
          put[l][c] = w >= lo[l] && o < lists[l].size && !((m >> lane) & 1u);
          if (put[l][c]) e[l][c] = lists[l].p[o - (int)(bl + __popc(m & lanemask_lt(lane)))];
        }
      cta_sync<NW>();
#pragma unroll
      for (int l = 0; l < NL; ++l)
#pragma unroll
        for (int c = 0; c < E; ++c) {
          const int w = hi[l] - (r * E + c) * NW - warp;
          if (put[l][c]) lists[l].p[32 * w + lane] = e[l][c];
        }
    }
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      if (slot[l] < lists[l].cap) lists[l].p[slot[l]] = lists[l].key[b0 + tid];
      if (warp == 0 && na[l]) lists[l].map[lane] = 0u;
    }
    cta_sync<NW>();
  }
}

template <int NW, int TRAV, int MET, int LPR, bool TC, bool FILT>
__device__ inline void search_cta(const SearchArgs &a, uint32_t q, uint8_t *sm, const WarpLayout &Ly, int tid) {
  constexpr int T = 32 * NW;
  const int warp = NW == 1 ? 0 : tid >> 5, lane = tid & 31;
  uint64_t *W = reinterpret_cast<uint64_t *>(sm + Ly.w0);
  uint64_t *RES = reinterpret_cast<uint64_t *>(sm + Ly.res);
  uint32_t *stage = reinterpret_cast<uint32_t *>(sm + Ly.stage);
  uint32_t *ctl = reinterpret_cast<uint32_t *>(sm + Ly.aux);
  float *qs = reinterpret_cast<float *>(sm + Ly.qf);
  const Visited vt{reinterpret_cast<uint32_t *>(sm + Ly.hash), a.hbits, a.hB};

  const uint32_t L = a.perL ? a.perL[q] : a.L;
  const uint32_t k = a.perK ? a.perK[q] : a.k;
  const bool use_rerank = TRAV != TRAV_F32 && a.rerank > 0;
  const uint32_t search_k = use_rerank ? max(a.rerank, k) : k;

  // per-query filter program
  QueryCtx qc{a.fops, a.fnops};
  if (FILT && a.foffs) {
    qc.fops = a.fops + a.foffs[q];
    qc.fnops = a.foffs[q + 1] - a.foffs[q];
  }
  const bool labeled = FILT && qc.fnops > 0;
  const bool tombed = FILT && a.tomb != nullptr;
  const bool filtered = labeled || tombed;
  uint32_t working = L, max_iter = 0xffffffffu;
  if (labeled) {  // src/filtered.rs:35-56, src/incremental.rs:1048-1062
    working = max(L * 4, k * 10);
    max_iter = working * 2;
  } else if (tombed) {  // tombstone_config (src/incremental.rs:505-516)
    working = max(L * 2, search_k + min(a.ntomb, L));
    max_iter = working * 2;
  }
  const bool two = a.seed2 != DG_PAD && a.seed2 != a.medoid;
  if (two) working = max(working, 2u);  // both seeds enter w (src/lib.rs:218-229)
  working = min(working, (Ly.w1 - Ly.w0) / 8);  // (the layout holds it; this bounds the writes)

  // ---- query into shared memory (zero padded), visited table, filter program
  const float *qg = a.Q + (size_t)q * a.d;
  for (uint32_t i = tid; i < a.dpad; i += T) qs[i] = i < a.d ? qg[i] : 0.0f;
  vt.clear(tid, T);
  if (FILT && labeled && qc.fnops <= kCtaOps) {
    uint64_t *dst = reinterpret_cast<uint64_t *>(sm + Ly.cstage);
    const uint64_t *src = reinterpret_cast<const uint64_t *>(qc.fops);
    for (uint32_t i = tid; i < qc.fnops * (uint32_t)(sizeof(DgFilterOp) / 8); i += T) dst[i] = src[i];
    qc.fops = reinterpret_cast<const DgFilterOp *>(dst);
  }
  cta_sync<NW>();
  float qq = 0.0f;
  if (MET == MET_COS) qq = query_norm2<TRAV>(qs, a.d, lane);
  if (TRAV == TRAV_PQ) {
    float *lut = reinterpret_cast<float *>(sm + Ly.prov);
    if (MET == MET_L2) build_pq_lut(a, qs, lut, tid, T);
    else build_pq_ip_lut(a, qs, lut, tid, T);
  } else if (warp == 0) {
    prepare_query<TRAV, MET>(a, sm, Ly, qs, lane);
  }

  // a result must be live (UnifiedView::is_live, src/incremental.rs:463-470) and match
  auto allow = [&](uint32_t id) -> bool {
    if (a.tomb && ((__ldg(a.tomb + (id >> 5)) >> (id & 31)) & 1u)) return false;
    if (!labeled) return true;
    const uint64_t *row = a.labels + (size_t)id * a.nf;
    if (a.nf > 4) return filter_eval(qc.fops, qc.fnops, a.fpool, row, a.nf);
    uint64_t l[4];  // the whole row at once
#pragma unroll
    for (uint32_t f = 0; f < 4; ++f) l[f] = f < a.nf ? __ldg(row + f) : 0ull;
    return filter_eval_by(qc.fops, qc.fnops, a.fpool, a.nf, [&](uint32_t f) {
      return f == 0 ? l[0] : f == 1 ? l[1] : f == 2 ? l[2] : l[3];
    });
  };

  // ---- seeds: the medoid, and the delta layer's entry point of a base + delta
  // index (src/incremental.rs:383-392), staged as the first candidates
  CtaList lists[2];
  const uint32_t nsv = max(a.R, 2u);
#pragma unroll
  for (int l = 0; l < (FILT ? 2 : 1); ++l) {
    uint8_t *sv = sm + Ly.w1 + l * cta_surv_bytes(a.R);
    lists[l] = CtaList{l ? RES : W, 0, l ? (int)search_k : (int)working, reinterpret_cast<uint64_t *>(sv),
                       reinterpret_cast<uint16_t *>(sv + align16(nsv * 8)), ctl + CTL_MAP + 32 * l};
  }
  const int &wsize = lists[0].size, &rsize = lists[1].size;
  if (!FILT) lists[1].size = 0;
  int next = 0;                    // every list entry below it is expanded (warp 0)
  uint32_t n_exp = 0, n_dist = 0;  // warp 0's
  if (tid == 0) {
    stage[0] = a.medoid;
    vt.test_and_set(a.medoid);
    if (two) {
      stage[1] = a.seed2;
      vt.test_and_set(a.seed2);
    }
    ctl[CTL_NS] = two ? 2u : 1u;
    ctl[CTL_CNT] = ctl[CTL_CNTR] = 0u;
  }
  for (int i = tid; i < (FILT ? 64 : 32); i += T) ctl[CTL_MAP + i] = 0u;
  if (warp == 0) n_dist = two ? 2u : 1u;
  cta_sync<NW>();  // candidates, quantizer state

  while (true) {
    const int ns = (int)ctl[CTL_NS];
    // ---- this warp's share of the candidates, B at a time: distances; keys
    // that can enter the list (or, matching, the result list) survive
    const uint64_t thr = wsize >= (int)working ? strip_flag(W[working - 1]) : kKeyInvalid;
    const uint64_t rthr = !filtered ? 0ull : rsize >= (int)search_k ? RES[search_k - 1] : kKeyInvalid;
    const int share = (ns + NW - 1) / NW, g1 = min(ns, (warp + 1) * share);
    constexpr int B = cta_batch<NW, TRAV, LPR, TC>();
    for (int g0 = warp * share; g0 < g1; g0 += B) {
      const int cnt = min(B, g1 - g0);
      const uint32_t cand = lane < cnt ? stage[g0 + lane] : DG_PAD;
      // the label row is on its way under the distances
      if (FILT && labeled && lane < cnt)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.labels + (size_t)cand * a.nf));
      float d = cta_distance<B, TRAV, MET, LPR, TC>(a, sm, Ly, cand, cnt, lane, qq);
      if (TRAV != TRAV_F32 && a.code_limit < a.n && lane < cnt && cand >= a.code_limit)
        d = exact_row_distance<MET>(a, qs, cand, qq);
      const uint64_t key = lane < cnt ? make_key(d, cand) : kKeyInvalid;
      cta_survive<NW>(lists[0], key, key < thr, ctl + CTL_CNT, lane);
      if (FILT && filtered)
        cta_survive<NW>(lists[1], key, lane < cnt && key < rthr && allow(cand), ctl + CTL_CNTR, lane);
    }
    cta_sync<NW>();  // every warp's survivors are in place
    const int s[2] = {(int)ctl[CTL_CNT], FILT ? (int)ctl[CTL_CNTR] : 0};
    if (FILT && s[1] > 0) cta_merge<NW, 2>(lists, s, tid, next);
    else if (s[0] > 0) cta_merge<NW, 1>(lists, s, tid, next);

    // ---- warp 0: the first unexpanded entry (the frontier minimum), the
    // stopping rules, its unvisited neighbours
    if (warp == 0) {
      int idx = -1;
      for (int base = next; base < wsize; base += 32) {
        const int i = base + lane;
        const uint32_t m = __ballot_sync(kFull, i < wsize && !key_expanded(W[i]));
        if (m) {
          idx = base + __ffs(m) - 1;
          break;
        }
      }
      bool stop = idx < 0;
      const uint64_t best = stop ? 0ull : W[idx];
      const float bd = key_dist(best);
      if (filtered && !stop) {
        stop = n_exp >= max_iter;  // src/lib.rs:237-240
        if (rsize >= (int)search_k && search_k > 0) {  // :242-251
          const float worst = key_dist(RES[search_k - 1]);
          if (worst >= 0.0f && bd > __fmul_rn(worst, 1.5f)) stop = true;
        }
      }
      if (!stop && wsize >= (int)working && bd >= key_dist(W[working - 1])) stop = true;  // :253-259
      uint32_t staged = kCtaStop;
      if (!stop) {
        next = idx + 1;
        ++n_exp;
        staged = (uint32_t)stage_neighbours(a, a.adj + (size_t)key_id(best) * a.R, vt, stage, lane);
        n_dist += staged;
      }
      if (lane == 0) {
        if (!stop) W[idx] = best | 1ull;
        ctl[CTL_NS] = staged;
        ctl[CTL_CNT] = ctl[CTL_CNTR] = 0u;  // (still to be read only where both are zero: merges end with a barrier)
      }
    }
    cta_sync<NW>();  // candidates
    if (ctl[CTL_NS] == kCtaStop) break;
  }

  // ---- results: the first k of the list, or its first max(rerank, k) reranked
  // with exact FP32 distances (a stable sort, src/quantized.rs:110-121)
  const uint64_t *src = filtered ? RES : W;
  const int have = filtered ? rsize : wsize;
  uint32_t *oid = a.out_ids + (size_t)q * a.k;
  float *od = a.out_d + (size_t)q * a.k;
  int count;
  if (use_rerank) {
    uint64_t *tmp = reinterpret_cast<uint64_t *>(sm + Ly.hash);
    const int nr = min(have, (int)search_k);
    for (int g0 = 16 * warp; g0 < nr; g0 += 16 * NW) {
      const int cnt = min(16, nr - g0);
      const uint32_t cand = lane < cnt ? key_id(src[g0 + lane]) : 0u;
      const float d = rows_distance_few<4, 8, 0, MET>(reinterpret_cast<const uint8_t *>(a.vec_f32), a.dpad * 4,
                                                 (a.dpad / 4) / 8, qs, cand, cnt, lane, a.metric == DG_L2, qq);
      if (lane < cnt) tmp[g0 + lane] = make_key_payload(d, (uint32_t)(g0 + lane));
    }
    cta_sync<NW>();
    count = min(nr, (int)k);
    for (int i = tid; i < nr; i += T) {
      const uint64_t u = tmp[i];
      int rank = 0;
      for (int j = 0; j < nr; ++j) rank += tmp[j] < u;
      if (rank < count) {
        oid[rank] = key_id(src[i]);
        od[rank] = key_dist(u);
      }
    }
  } else {
    count = min(have, (int)k);
    for (int i = tid; i < count; i += T) {
      oid[i] = key_id(src[i]);
      od[i] = key_dist(src[i]);
    }
  }
  for (int i = count + tid; i < (int)a.k; i += T) {
    oid[i] = DG_PAD;
    od[i] = __int_as_float(0x7f800000);
  }
  if (tid == 0) {
    a.out_cnt[q] = (uint32_t)count;
    if (a.out_stats) {
      a.out_stats[2 * q] = n_exp;
      a.out_stats[2 * q + 1] = n_dist;
    }
  }
}

// 20 warps per SM leave 96 registers (8 warps per query: 128).  They are not
// enough for every form: per thread, BF16 rows with a filter spill 128-264 bytes
// at 1 to 4 warps, without one 24-128; int8 codes 48-76 and 116-176.
template <int NW, int TRAV, int MET, int LPR, bool TC, bool FILT>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? 2 : 20 / NW) beam_search_cta_kernel(SearchArgs a, WarpLayout Ly) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t *ctl = reinterpret_cast<uint32_t *>(smem + Ly.aux);
  while (true) {
    if (threadIdx.x == 0) ctl[CTL_Q] = atomicAdd(a.counter, 1u);
    cta_sync<NW>();
    uint32_t q = ctl[CTL_Q];
    if (q >= a.nq) break;
    if (a.perm) q = __ldg(a.perm + q);
    search_cta<NW, TRAV, MET, LPR, TC, FILT>(a, q, smem, Ly, threadIdx.x);
    cta_sync<NW>();  // the query's shared state is free
  }
}

}  // namespace dg
