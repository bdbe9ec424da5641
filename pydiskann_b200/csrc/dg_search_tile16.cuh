// dg_search_tile16.cuh -- distances of at most 16 candidate rows by one warp,
// as the CTA-per-query search takes them: a quarter of one expansion's
// neighbours, all of whose loads should be in flight at once.
#pragma once
#include "dg_search.cuh"

namespace dg {

// 16-byte loads in flight per lane: kTileLoads, spread over the row slots of
// rows_distance_few or over the two rows of a tensor-core tile (4 KB per warp).
// Rows of four rounds and more have the rest asked for in L2 at the same time,
// so that only their first round waits for DRAM; shorter ones lose more to the
// extra requests (300k rows, beam 100, 6000 queries, with / without: FP32 256-d
// 3500 / 3891 us, FP32 128-d 2419 / 2283; BF16 256-d, beam 200, 5593 / 5346).
constexpr int kTileLoads = 8;

// Asks L2 for bytes [from, to) of this lane's row (both multiples of 16).
__device__ __forceinline__ void prefetch_row(const uint8_t *row, uint32_t from, uint32_t to) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row + from), "r"(to - from));
}

// rows_distance for at most S * 32 / LPR candidates: S row slots instead of
// LPR, kTileLoads / S 16-byte rounds of each in flight.  Every row is summed in the order of
// rows_distance (per lane over its chunks, then over lanes 4, 2, 1 apart), so
// the distances are the same bits.
template <int S, int LPR, int ELEM, int MET>
__device__ __forceinline__ float rows_distance_few(const uint8_t *__restrict__ rows, uint32_t stride, int loads,
                                                 const float *qs, uint32_t cand, int cnt, int lane, bool sqrt_l2,
                                                 float qq) {
  constexpr int RPI = 32 / LPR;
  constexpr int EPC = Chunk<ELEM>::EPC;
  constexpr int U = kTileLoads / S;  // rounds in flight
  const int g = lane / LPR, r = lane % LPR;
  if (loads > 3 * U && lane < cnt) prefetch_row(rows + (size_t)cand * stride, U * LPR * 16, loads * LPR * 16);
  float sa[S], sb[S];
  uint32_t ids[S];
#pragma unroll
  for (int i = 0; i < S; ++i) {
    sa[i] = sb[i] = 0.0f;
    const int c = i * RPI + g;
    const uint32_t id = __shfl_sync(kFull, cand, c & 31);
    ids[i] = c < cnt ? id : DG_PAD;
  }
  for (int t = 0; t < loads; t += U) {
    uint4 v[U][S];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < S; ++i)
        if (ids[i] != DG_PAD && t + u < loads)
          v[u][i] = ldg_row<ELEM == 0>(reinterpret_cast<const uint4 *>(rows + (size_t)ids[i] * stride) + r +
                                       LPR * (t + u));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (t + u >= loads) break;
      const int chunk = r + LPR * (t + u);
      float2 q2[EPC / 2];
#pragma unroll
      for (int e = 0; e < EPC / 2; ++e) q2[e] = reinterpret_cast<const float2 *>(qs + chunk * EPC)[e];
#pragma unroll
      for (int i = 0; i < S; ++i) {
        if (ids[i] != DG_PAD) {
          const float2 neg1 = make_float2(-1.0f, -1.0f);
          float x[EPC];
          Chunk<ELEM>::unpack(v[u][i], x);
          float2 pa = make_float2(0.0f, 0.0f), pb = make_float2(0.0f, 0.0f);
#pragma unroll
          for (int e = 0; e < EPC / 2; ++e) {
            const float2 x2 = make_float2(x[2 * e], x[2 * e + 1]);
            if (MET == MET_L2) {
              const float2 df = __ffma2_rn(q2[e], neg1, x2);
              pa = __ffma2_rn(df, df, pa);
            } else {
              pa = __ffma2_rn(x2, q2[e], pa);
              if (MET == MET_COS) pb = __ffma2_rn(x2, x2, pb);
            }
          }
          sa[i] += pa.x + pa.y;
          if (MET == MET_COS) sb[i] += pb.x + pb.y;
        }
      }
    }
  }
  // lanes LPR / 2 .. S apart first, then the transposed reduction over the S slots
  auto reduce = [&](float (&p)[S]) {
#pragma unroll
    for (int o = LPR / 2; o >= S; o >>= 1)
#pragma unroll
      for (int i = 0; i < S; ++i) p[i] += __shfl_xor_sync(kFull, p[i], o);
    return transpose_reduce<S>(p, lane);
  };
  float a = reduce(sa), b = 0.0f;
  if (MET == MET_COS) b = reduce(sb);
  const int srcl = (lane % RPI) * LPR + ((lane / RPI) & (LPR - 1));
  a = __shfl_sync(kFull, a, srcl);
  if (MET == MET_COS) b = __shfl_sync(kFull, b, srcl);
  return finish_metric(MET, sqrt_l2, a, b, qq);
}

// The 16-row tile of the tensor-core distances (int8_l2_mma, int8_dot_mma,
// bf16_dot_mma, fp8_dot_mma), same lane layout and the same order of the
// accumulations, with several 16-byte chunks of each of a lane's two rows in
// flight.  `col`: this lane's column of B holds a query column (at pq; zero
// otherwise); step(u, x0, x1, q) accumulates chunk step u's two row chunks.
template <typename Step>
__device__ __forceinline__ void mma16_chunks(const uint8_t *__restrict__ rows, uint32_t stride, const uint4 *pq,
                                             bool col, uint32_t cand, int cnt, int lane, Step step) {
  constexpr int U = kTileLoads / 2;  // chunk steps in flight
  const int g = lane >> 2, t = lane & 3;
  const int nch = (int)(stride >> 4), J = (nch + 3) >> 2;
  if (J > 3 * U && lane < cnt) prefetch_row(rows + (size_t)cand * stride, U * 64, stride);
  const uint32_t id0 = __shfl_sync(kFull, cand, 0);
  uint32_t i0 = __shfl_sync(kFull, cand, g), i1 = __shfl_sync(kFull, cand, g + 8);
  i0 = g < cnt ? i0 : id0;
  i1 = g + 8 < cnt ? i1 : id0;
  const uint4 *r0 = reinterpret_cast<const uint4 *>(rows + (size_t)i0 * stride);
  const uint4 *r1 = reinterpret_cast<const uint4 *>(rows + (size_t)i1 * stride);
  const uint4 z = make_uint4(0, 0, 0, 0);
  for (int j0 = 0; j0 < J; j0 += U) {
    uint4 x[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int ch = t + 4 * (j0 + u);
      const bool ok = ch < nch;
      x[u][0] = ok ? __ldg(r0 + ch) : z;
      x[u][1] = ok ? __ldg(r1 + ch) : z;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int ch = t + 4 * (j0 + u);
      if (j0 + u < J) step(u, x[u][0], x[u][1], ch < nch && col ? pq[ch] : z);
    }
  }
}

// int8_l2_mma, int8_dot_mma, bf16_dot_mma and fp8_dot_mma for at most 16
// candidates (lane j: candidate j).
__device__ __forceinline__ uint32_t int8_l2_mma16(const SearchArgs &a, const uint8_t *qcode, uint32_t qn,
                                                  uint32_t cand, int cnt, int lane) {
  const uint32_t xn = lane < cnt ? __ldg(a.i8_norm + cand) : 0u;
  int c[4] = {0, 0, 0, 0};
  mma16_chunks(a.codes, a.code_stride, reinterpret_cast<const uint4 *>(qcode), true, cand, cnt, lane,
               [&](int, const uint4 &x0, const uint4 &x1, const uint4 &q) {
                 mma_u8_16x8x32(c, x0.x, x1.x, x0.y, x1.y, q.x, q.y);
                 mma_u8_16x8x32(c, x0.z, x1.z, x0.w, x1.w, q.z, q.w);
               });
  const int src = (lane & 7) << 2;
  const int d0 = __shfl_sync(kFull, c[0], src), d1 = __shfl_sync(kFull, c[2], src);
  return qn + xn - 2u * (uint32_t)((lane & 15) < 8 ? d0 : d1);
}

__device__ __forceinline__ double int8_dot_mma16(const SearchArgs &a, const uint8_t *qdig, uint32_t dstride,
                                                 uint32_t cand, int cnt, int lane) {
  const int g = lane >> 2;
  int c[4] = {0, 0, 0, 0};
  mma16_chunks(a.codes, a.code_stride, reinterpret_cast<const uint4 *>(qdig + (size_t)(g & 3) * dstride), g < 4, cand,
               cnt, lane, [&](int, const uint4 &x0, const uint4 &x1, const uint4 &q) {
                 mma_u8s8_16x8x32(c, x0.x, x1.x, x0.y, x1.y, q.x, q.y);
                 mma_u8s8_16x8x32(c, x0.z, x1.z, x0.w, x1.w, q.z, q.w);
               });
  const int s0 = (lane & 7) << 2;
  const bool hi = (lane & 15) >= 8;
  const int e0 = __shfl_sync(kFull, c[0], s0), e1 = __shfl_sync(kFull, c[1], s0);
  const int e2 = __shfl_sync(kFull, c[2], s0), e3 = __shfl_sync(kFull, c[3], s0);
  const int f0 = __shfl_sync(kFull, c[0], s0 + 1), f1 = __shfl_sync(kFull, c[1], s0 + 1);
  const int f2 = __shfl_sync(kFull, c[2], s0 + 1), f3 = __shfl_sync(kFull, c[3], s0 + 1);
  return (double)(hi ? e2 : e0) * 16777216.0 + (double)(hi ? e3 : e1) * 65536.0 + (double)(hi ? f2 : f0) * 256.0 +
         (double)(hi ? f3 : f1);
}

__device__ __forceinline__ float bf16_dot_mma16(const SearchArgs &a, const uint16_t *qhl, uint32_t cand, int cnt,
                                                int lane) {
  const int g = lane >> 2;
  float c[2][4] = {};  // even and odd chunk steps
  mma16_chunks(reinterpret_cast<const uint8_t *>(a.vec_bf16), a.dpad * 2,
               reinterpret_cast<const uint4 *>(qhl + (g == 1 ? a.dpad : 0)), g < 2, cand, cnt, lane,
               [&](int u, const uint4 &x0, const uint4 &x1, const uint4 &q) {
                 mma_bf16_16x8x16(c[u & 1], x0.x, x1.x, x0.y, x1.y, q.x, q.y);
                 mma_bf16_16x8x16(c[u & 1], x0.z, x1.z, x0.w, x1.w, q.z, q.w);
               });
  const float a0 = __fadd_rn(__fadd_rn(c[0][0], c[1][0]), __fadd_rn(c[0][1], c[1][1]));
  const float a1 = __fadd_rn(__fadd_rn(c[0][2], c[1][2]), __fadd_rn(c[0][3], c[1][3]));
  const int src = (lane & 7) << 2;
  const float e0 = __shfl_sync(kFull, a0, src), e1 = __shfl_sync(kFull, a1, src);
  return (lane & 15) < 8 ? e0 : e1;
}

__device__ __forceinline__ float fp8_dot_mma16(const SearchArgs &a, const uint8_t *qhl, uint32_t cand, int cnt,
                                               int lane) {
  const int g = lane >> 2;
  float c[4] = {};
  mma16_chunks(a.vec_fp8, a.dpad, reinterpret_cast<const uint4 *>(qhl + (g == 1 ? a.dpad : 0)), g < 2, cand, cnt,
               lane, [&](int, const uint4 &x0, const uint4 &x1, const uint4 &q) {
                 mma_e4m3_16x8x32(c, x0.x, x1.x, x0.y, x1.y, q.x, q.y);
                 mma_e4m3_16x8x32(c, x0.z, x1.z, x0.w, x1.w, q.z, q.w);
               });
  const int src = (lane & 7) << 2;
  const float d0 = __shfl_sync(kFull, fmaf(c[1], 0.0625f, c[0]), src);
  const float d1 = __shfl_sync(kFull, fmaf(c[3], 0.0625f, c[2]), src);
  return (lane & 15) < 8 ? d0 : d1;
}

}  // namespace dg
