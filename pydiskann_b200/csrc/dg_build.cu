// dg_build.cu -- encoders, medoid, PQ training and exact kNN on the GPU.
#include <algorithm>
#include <cmath>
#include <vector>

#include "dg_index.h"
#include "dg_search.cuh"

namespace dg {

// ------------------------------------------------------------ row encoders
__global__ void k_bf16(const float *v, uint64_t total, uint16_t *out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = __bfloat16_as_ushort(__float2bfloat16_rn(v[i]));
}
__global__ void k_f16(const float *v, uint64_t total, uint16_t *out) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = __half_as_ushort(__float2half_rn(v[i]));
}
// Int8Quantizer::encode (src/sq.rs:208-220)
__global__ void k_int8(const float *v, uint64_t n, uint32_t d, uint32_t dpad, float inv, float beta,
                       uint8_t *out, uint32_t stride) {
  const uint64_t total = n * stride;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t r = i / stride;
    const uint32_t c = (uint32_t)(i % stride);
    out[i] = c < d ? int8_code(v[r * dpad + c], inv, beta) : 0;
  }
}
// FP8 rows: per vector s = max|x| / 448 (1 for a zero vector), codes
// e4m3(x / s) rounded to nearest even with saturation, and |s * e4m3(x / s)|^2
// summed in coordinate order.  One thread per vector.
__global__ void k_fp8(const float *v, uint64_t n, uint32_t d, uint32_t dpad, uint8_t *codes, float2 *sn) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
    const float *x = v + r * dpad;
    float mx = 0.0f;
    for (uint32_t i = 0; i < d; ++i) mx = fmaxf(mx, fabsf(x[i]));
    const float s = mx > 0.0f ? __fdiv_rn(mx, 448.0f) : 1.0f;
    uint8_t *c = codes + r * dpad;
    float nn = 0.0f;
    for (uint32_t i = 0; i < dpad; ++i) {
      const __nv_fp8_storage_t e = i < d ? __nv_cvt_float_to_fp8(__fdiv_rn(x[i], s), __NV_SATFINITE, __NV_E4M3) : 0;
      c[i] = e;
      const float xv = __fmul_rn(s, __half2float(__half(__nv_cvt_fp8_to_halfraw(e, __NV_E4M3))));
      nn = __fadd_rn(nn, __fmul_rn(xv, xv));
    }
    sn[r] = make_float2(s, nn);
  }
}
// Sum of squared codes of every int8 row (padding bytes are zero).
__global__ void k_int8_norm(const uint8_t *codes, uint64_t n, uint32_t stride, uint32_t *out, uint32_t *sums) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
    const uint4 *row = reinterpret_cast<const uint4 *>(codes + r * stride);
    uint32_t s = 0, t = 0;
    for (uint32_t c = 0; c < stride / 16; ++c) {
      const uint4 v = row[c];
      s = __dp4a(v.x, v.x, s);
      s = __dp4a(v.y, v.y, s);
      s = __dp4a(v.z, v.z, s);
      s = __dp4a(v.w, v.w, s);
      t = __dp4a(v.x, 0x01010101u, t);
      t = __dp4a(v.y, 0x01010101u, t);
      t = __dp4a(v.z, 0x01010101u, t);
      t = __dp4a(v.w, 0x01010101u, t);
    }
    out[r] = s;
    if (sums) sums[r] = t;
  }
}
// ProductQuantizer::encode (src/pq.rs:122-149): argmin with strict '<', each
// distance summed in coordinate order.  Row i's code of subspace m goes to
// codes[i * row_step + m * sub_step].  Any subspace width.
__global__ void k_pq_encode(const float *v, uint64_t n, uint32_t dpad, uint32_t M, uint32_t K,
                            uint32_t ds, const float *cb, uint8_t *codes, uint64_t row_step, uint64_t sub_step) {
  const uint32_t m = blockIdx.y;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float *sub = v + i * dpad + m * ds;
    float best = 3.402823466e38f;
    uint32_t bc = 0;
    for (uint32_t c = 0; c < K; ++c) {
      const float *cen = cb + ((size_t)m * K + c) * ds;
      float acc = 0.0f;
      for (uint32_t j = 0; j < ds; ++j) {
        float t = __fsub_rn(sub[j], __ldg(cen + j));
        acc = __fadd_rn(acc, __fmul_rn(t, t));
      }
      if (acc < best) {
        best = acc;
        bc = c;
      }
    }
    codes[i * row_step + m * sub_step] = (uint8_t)bc;
  }
}

// The same for the usual widths: the subspace's codebook sits in shared
// memory, two centroids interleaved, and a thread holds two sub-vectors in
// registers, so that each load of a centroid pair serves four distances (a
// subtraction, a multiplication and an addition per coordinate, each rounded
// once, in coordinate order: the same bits.  Packed two-wide forms were
// contracted to FMAs, which changed one code in eight million).  Bound by FP32
// issue; the kernel above
// re-reads the sub-vector and the centroid for every term (200k rows, M = 16,
// K = 256, 8 wide: 24 ms).
template <int DS>
__global__ void __launch_bounds__(256) k_pq_nearest(const float *__restrict__ v, uint64_t n, uint32_t stride,
                                                    uint32_t K, const float *__restrict__ cb, uint8_t *codes,
                                                    uint64_t row_step, uint64_t sub_step) {
  __shared__ __align__(16) float2 cs[128 * DS];  // [pair of centroids][coordinate]
  const uint32_t m = blockIdx.y, pairs = (K + 1) / 2;
  const float inf = __int_as_float(0x7f800000);
  for (uint32_t e = threadIdx.x; e < pairs * DS; e += blockDim.x) {
    const uint32_t c = 2 * (e / DS), j = e % DS;
    const float *p = cb + ((size_t)m * K + c) * DS + j;
    cs[e] = make_float2(p[0], c + 1 < K ? p[DS] : inf);  // (an infinite distance is never the smallest)
  }
  __syncthreads();
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i0 < n; i0 += 2 * step) {
    const uint64_t i1 = i0 + step < n ? i0 + step : i0;
    const float *x0 = v + i0 * stride + m * DS, *x1 = v + i1 * stride + m * DS;
    float a[DS], b[DS];
    if (DS % 4 == 0) {  // stride and the subspace's offset are then multiples of 16 bytes
#pragma unroll
      for (int j = 0; j < DS / 4; ++j) {
        reinterpret_cast<float4 *>(a)[j] = __ldg(reinterpret_cast<const float4 *>(x0) + j);
        reinterpret_cast<float4 *>(b)[j] = __ldg(reinterpret_cast<const float4 *>(x1) + j);
      }
    } else {
#pragma unroll
      for (int j = 0; j < DS; ++j) {
        a[j] = __ldg(x0 + j);
        b[j] = __ldg(x1 + j);
      }
    }
    float best0 = 3.402823466e38f, best1 = best0;
    uint32_t c0 = 0, c1 = 0;
    for (uint32_t c = 0; c < pairs; ++c) {
      float2 s0 = make_float2(0.0f, 0.0f), s1 = s0;
#pragma unroll
      for (int j = 0; j < DS; ++j) {
        const float2 cv = cs[c * DS + j];
        const float t0 = __fsub_rn(a[j], cv.x), t1 = __fsub_rn(a[j], cv.y);
        const float u0 = __fsub_rn(b[j], cv.x), u1 = __fsub_rn(b[j], cv.y);
        s0.x = __fadd_rn(s0.x, __fmul_rn(t0, t0));
        s0.y = __fadd_rn(s0.y, __fmul_rn(t1, t1));
        s1.x = __fadd_rn(s1.x, __fmul_rn(u0, u0));
        s1.y = __fadd_rn(s1.y, __fmul_rn(u1, u1));
      }
      if (s0.x < best0) { best0 = s0.x; c0 = 2 * c; }
      if (s0.y < best0) { best0 = s0.y; c0 = 2 * c + 1; }
      if (s1.x < best1) { best1 = s1.x; c1 = 2 * c; }
      if (s1.y < best1) { best1 = s1.y; c1 = 2 * c + 1; }
    }
    codes[i0 * row_step + m * sub_step] = (uint8_t)c0;
    codes[i1 * row_step + m * sub_step] = (uint8_t)c1;
  }
}

// Codes of n rows (rows `stride` floats apart) by the kernel for this width.
static DgStatus pq_codes(const float *v, uint64_t n, uint32_t stride, uint32_t M, uint32_t K, uint32_t ds,
                         const float *cb, uint8_t *codes, uint64_t row_step, uint64_t sub_step, cudaStream_t st) {
  // float4 loads need rows of whole 16-byte blocks
  const bool wide = ds % 4 != 0 || (stride % 4 == 0 && (reinterpret_cast<uintptr_t>(v) & 15) == 0);
  const dim3 grid((unsigned)std::min<uint64_t>((n + 511) / 512, 4096), M), block(256);
  auto fast = [&](auto kern) { kern<<<grid, block, 0, st>>>(v, n, stride, K, cb, codes, row_step, sub_step); };
  switch (wide ? ds : 0) {
    case 2: fast(k_pq_nearest<2>); break;
    case 4: fast(k_pq_nearest<4>); break;
    case 6: fast(k_pq_nearest<6>); break;
    case 8: fast(k_pq_nearest<8>); break;
    case 10: fast(k_pq_nearest<10>); break;
    case 12: fast(k_pq_nearest<12>); break;
    case 16: fast(k_pq_nearest<16>); break;
    default:
      k_pq_encode<<<dim3((unsigned)std::min<uint64_t>((n + 127) / 128, 4096), M), 128, 0, st>>>(
          v, n, stride, M, K, ds, cb, codes, row_step, sub_step);
  }
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}

// RaBitQ encode_with (src/rabitq.rs:136-149,240-256), one warp per vector.
__global__ void k_rabitq_encode(const float *v, uint64_t n, uint32_t d, uint32_t dpad, uint32_t P,
                                const float *cen, const float *signs, uint8_t *codes,
                                uint32_t stride) {
  extern __shared__ __align__(16) float rbuf[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *r = rbuf + (size_t)warp * P;
  const uint64_t gw = blockIdx.x * (uint64_t)(blockDim.x >> 5) + warp;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
  for (uint64_t row = gw; row < n; row += nw) {
    const float *x = v + row * dpad;
    for (uint32_t i = lane; i < P; i += 32) r[i] = i < d ? __fsub_rn(x[i], cen[i]) : 0.0f;
    __syncwarp();
    float s = 0.0f;
    if (lane == 0)
      for (uint32_t i = 0; i < P; ++i) s = __fadd_rn(s, __fmul_rn(r[i], r[i]));
    const float norm = __shfl_sync(kFull, __fsqrt_rn(s), 0);
    if (norm > 0.0f)
      for (uint32_t i = lane; i < P; i += 32) r[i] = __fdiv_rn(r[i], norm);
    __syncwarp();
    for (int rd = 0; rd < 3; ++rd) {
      for (uint32_t i = lane; i < P; i += 32) r[i] = __fmul_rn(r[i], signs[rd * P + i]);
      __syncwarp();
      for (uint32_t h = 1; h < P; h *= 2) {
        for (uint32_t t = lane; t < P / 2; t += 32) {
          const uint32_t j = (t / h) * 2 * h + (t % h);
          const float a = r[j], b = r[j + h];
          r[j] = __fadd_rn(a, b);
          r[j + h] = __fsub_rn(a, b);
        }
        __syncwarp();
      }
    }
    uint8_t *code = codes + row * stride;
    for (uint32_t wd = 0; wd < P / 64; ++wd) {
      const bool b0 = r[wd * 64 + lane] > 0.0f, b1 = r[wd * 64 + 32 + lane] > 0.0f;
      const uint32_t lo = __ballot_sync(kFull, b0), hi = __ballot_sync(kFull, b1);
      if (lane == 0) {
        uint32_t *w = reinterpret_cast<uint32_t *>(code + wd * 8);
        w[0] = lo;
        w[1] = hi;
      }
    }
    if (lane == 0) {  // sequential sum of |x| in coordinate order, as the oracle
      float ip = 0.0f;
      for (uint32_t i = 0; i < P; ++i) ip = __fadd_rn(ip, fabsf(r[i]));
      ip = __fdiv_rn(ip, __fsqrt_rn((float)P));
      const float fac = ip > 0.0f ? __fdiv_rn(norm, ip) : 0.0f;
      float *tail = reinterpret_cast<float *>(code + P / 8);
      tail[0] = __fmul_rn(norm, norm);
      tail[1] = fac;
    }
    __syncwarp();
  }
}

// Squared norm of every decoded PQ code (ProductQuantizer::decode,
// src/pq.rs:151-160): the |x|^2 term of the cosine metric over codes, summed
// in coordinate order as angular() does.  One thread per vector.
__global__ void k_pq_dnorm2(const uint8_t *codes, uint64_t n, uint32_t stride, uint32_t M, uint32_t K,
                            uint32_t ds, const float *cb, float *out) {
  for (uint64_t row = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; row < n;
       row += (uint64_t)gridDim.x * blockDim.x) {
    const uint8_t *code = codes + row * stride;
    float bb = 0.0f;
    for (uint32_t m = 0; m < M; ++m) {
      const float *c = cb + ((size_t)m * K + code[m]) * ds;
      for (uint32_t j = 0; j < ds; ++j) bb = __fadd_rn(bb, __fmul_rn(c[j], c[j]));
    }
    out[row] = bb;
  }
}

// Squared norm of every decoded RaBitQ code (src/rabitq.rs:224-238): signs
// +-1/sqrt(P), three inverse rounds (Hadamard, then sign flip), then
// c + |v-c| * r over the first d coordinates, summed in coordinate order.
// One warp per vector.
__global__ void k_rq_dnorm2(const uint8_t *codes, uint64_t n, uint32_t stride, uint32_t d, uint32_t P,
                            const float *cen, const float *signs, float *out) {
  extern __shared__ __align__(16) float rbuf[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float *r = rbuf + (size_t)warp * P;
  const uint64_t gw = blockIdx.x * (uint64_t)(blockDim.x >> 5) + warp;
  const uint64_t nw = (uint64_t)gridDim.x * (blockDim.x >> 5);
  const float inv = __fdiv_rn(1.0f, __fsqrt_rn((float)P));
  for (uint64_t row = gw; row < n; row += nw) {
    const uint8_t *code = codes + row * stride;
    for (uint32_t i = lane; i < P; i += 32) r[i] = ((code[i >> 3] >> (i & 7)) & 1u) ? inv : -inv;
    __syncwarp();
    for (int rd = 2; rd >= 0; --rd) {
      for (uint32_t h = 1; h < P; h *= 2) {
        for (uint32_t t = lane; t < P / 2; t += 32) {
          const uint32_t j = (t / h) * 2 * h + (t % h);
          const float a = r[j], b = r[j + h];
          r[j] = __fadd_rn(a, b);
          r[j + h] = __fsub_rn(a, b);
        }
        __syncwarp();
      }
      for (uint32_t i = lane; i < P; i += 32) r[i] = __fmul_rn(r[i], signs[rd * P + i]);
      __syncwarp();
    }
    if (lane == 0) {
      const float norm = __fsqrt_rn(*reinterpret_cast<const float *>(code + P / 8));
      float bb = 0.0f;
      for (uint32_t i = 0; i < d; ++i) {
        const float o = __fadd_rn(cen[i], __fmul_rn(norm, r[i]));
        bb = __fadd_rn(bb, __fmul_rn(o, o));
      }
      out[row] = bb;
    }
    __syncwarp();
  }
}

__global__ void k_count(const uint64_t *labels, uint64_t n, uint32_t nf, const DgFilterOp *ops,
                        uint32_t nops, const uint64_t *pool, unsigned long long *count) {
  unsigned long long c = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    c += filter_eval(ops, nops, pool, labels + i * nf, nf) ? 1 : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, c);
}

static int grid_for(uint64_t work, int threads) {
  uint64_t g = (work + threads - 1) / threads;
  return (int)std::min<uint64_t>(std::max<uint64_t>(g, 1), 148ull * 64);
}

// Squared norm of every BF16 row, summed in coordinate order in FP32.
__global__ void k_bf16_norms(const uint16_t *rows, uint64_t n, uint32_t dpad, float *out) {
  for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
    const uint16_t *x = rows + r * dpad;
    float s2 = 0.0f;
    for (uint32_t i = 0; i < dpad; ++i) {
      const float v = __uint_as_float((uint32_t)x[i] << 16);
      s2 = __fadd_rn(s2, __fmul_rn(v, v));
    }
    out[r] = s2;
  }
}

DgStatus encode_bf16_device(const float *vec, uint64_t n, uint32_t dpad, uint16_t *out, cudaStream_t st,
                            float *norms) {
  k_bf16<<<grid_for(n * dpad, 256), 256, 0, st>>>(vec, n * dpad, out);
  DG_CUDA(cudaGetLastError());
  if (norms) {
    k_bf16_norms<<<grid_for(n, 128), 128, 0, st>>>(out, n, dpad, norms);
    DG_CUDA(cudaGetLastError());
  }
  return DG_OK;
}
DgStatus encode_f16_device(const float *vec, uint64_t n, uint32_t dpad, uint16_t *out, cudaStream_t st) {
  k_f16<<<grid_for(n * dpad, 256), 256, 0, st>>>(vec, n * dpad, out);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
DgStatus encode_int8_device(const float *vec, uint64_t n, uint32_t d, uint32_t dpad, float scale,
                            float offset, uint8_t *codes, uint32_t stride, cudaStream_t st) {
  const float inv = 1.0f / scale;  // same f32 expressions as Int8Quantizer::encode
  const float beta = -offset / scale;
  k_int8<<<grid_for(n * stride, 256), 256, 0, st>>>(vec, n, d, dpad, inv, beta, codes, stride);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
DgStatus encode_fp8_device(const float *vec, uint64_t n, uint32_t d, uint32_t dpad, uint8_t *codes,
                           float2 *sn, cudaStream_t st) {
  k_fp8<<<grid_for(n, 128), 128, 0, st>>>(vec, n, d, dpad, codes, sn);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
DgStatus int8_norms_device(const uint8_t *codes, uint64_t n, uint32_t stride, uint32_t *out, uint32_t *sums,
                           cudaStream_t st) {
  k_int8_norm<<<grid_for(n, 256), 256, 0, st>>>(codes, n, stride, out, sums);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
DgStatus encode_pq_device(const float *vec, uint64_t n, uint32_t d, uint32_t dpad, uint32_t M,
                          uint32_t K, const float *cb, uint8_t *codes, uint32_t stride,
                          cudaStream_t st) {
  return pq_codes(vec, n, dpad, M, K, d / M, cb, codes, stride, 1, st);
}
DgStatus encode_rabitq_device(const float *vec, uint64_t n, uint32_t d, uint32_t dpad, uint32_t P,
                              const float *centroid, const float *signs, uint8_t *codes,
                              uint32_t stride, cudaStream_t st) {
  const int warps = 4;
  const size_t smem = (size_t)warps * P * 4;
  DG_CUDA(cudaFuncSetAttribute(k_rabitq_encode, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int blocks = (int)std::min<uint64_t>((n + warps - 1) / warps, 148ull * 16);
  k_rabitq_encode<<<blocks, warps * 32, smem, st>>>(vec, n, d, dpad, P, centroid, signs, codes, stride);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
DgStatus decoded_norms_device(const DgIndex *idx, float *out, cudaStream_t st) {
  if (idx->quant == DG_Q_PQ) {
    k_pq_dnorm2<<<grid_for(idx->n, 128), 128, 0, st>>>(idx->codes, idx->n, idx->code_stride, idx->pq_M,
                                                       idx->pq_K, idx->d / idx->pq_M, idx->pq_cb, out);
  } else {
    const int warps = 4;
    const uint32_t P = idx->rq_padded;
    const size_t smem = (size_t)warps * P * 4;
    DG_CUDA(cudaFuncSetAttribute(k_rq_dnorm2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int blocks = (int)std::min<uint64_t>((idx->n + warps - 1) / warps, 148ull * 16);
    k_rq_dnorm2<<<blocks, warps * 32, smem, st>>>(idx->codes, idx->n, idx->code_stride, idx->d, P,
                                                  idx->rq_centroid, idx->rq_signs, out);
  }
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}
DgStatus count_matching_device(const uint64_t *labels, uint64_t n, uint32_t nf,
                               const DgFilterOp *ops, uint32_t nops, const uint64_t *pool,
                               unsigned long long *count, cudaStream_t st) {
  k_count<<<grid_for(n, 256), 256, 0, st>>>(labels, n, nf, ops, nops, pool, count);
  DG_CUDA(cudaGetLastError());
  return DG_OK;
}

// ------------------------------------------------------------------ medoid
// calculate_medoid (src/lib.rs:748-768): centroid summed in f64 and rounded
// once to f32, f64 distances, lowest index on ties (same as the oracle).
__global__ void k_colsum(const float *v, uint64_t n, uint32_t d, uint32_t dpad, double *sums) {
  for (uint32_t c = threadIdx.x; c < d; c += blockDim.x) {
    double acc = 0.0;
    for (uint64_t r = blockIdx.x; r < n; r += gridDim.x) acc += (double)v[r * dpad + c];
    atomicAdd(sums + c, acc);
  }
}
__device__ __forceinline__ unsigned long long ordered_u64(double x) {
  unsigned long long u = (unsigned long long)__double_as_longlong(x);
  return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ double medoid_metric(const float *x, const float *c, uint32_t d, int metric) {
  if (metric == DG_L2SQ || metric == DG_L2) {
    double s = 0.0;
    for (uint32_t j = 0; j < d; ++j) {
      double t = __dsub_rn((double)c[j], (double)x[j]);
      s = __dadd_rn(s, __dmul_rn(t, t));
    }
    return s;
  }
  double ab = 0.0, aa = 0.0, bb = 0.0;
  for (uint32_t j = 0; j < d; ++j) {
    ab = __dadd_rn(ab, __dmul_rn((double)c[j], (double)x[j]));
    aa = __dadd_rn(aa, __dmul_rn((double)c[j], (double)c[j]));
    bb = __dadd_rn(bb, __dmul_rn((double)x[j], (double)x[j]));
  }
  if (metric == DG_COSINE) return (aa == 0.0 || bb == 0.0) ? 1.0 : 1.0 - ab / (sqrt(aa) * sqrt(bb));
  return 1.0 - ab;
}
__global__ void k_medoid_min(const float *v, uint64_t n, uint32_t d, uint32_t dpad, const float *c,
                             int metric, unsigned long long *best) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    atomicMin(best, ordered_u64(medoid_metric(v + i * dpad, c, d, metric)));
}
__global__ void k_medoid_arg(const float *v, uint64_t n, uint32_t d, uint32_t dpad, const float *c,
                             int metric, const unsigned long long *best, unsigned long long *arg) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    if (ordered_u64(medoid_metric(v + i * dpad, c, d, metric)) == *best) atomicMin(arg, (unsigned long long)i);
}

DgStatus medoid_device(const float *vec, uint64_t n, uint32_t d, uint32_t dpad, int metric,
                       uint32_t *out, cudaStream_t st) {
  double *sums = nullptr;
  float *cen = nullptr;
  unsigned long long *best = nullptr;
  DG_CUDA(cudaMallocAsync(&sums, d * 8, st));
  DG_CUDA(cudaMallocAsync(&cen, d * 4, st));
  DG_CUDA(cudaMallocAsync(&best, 16, st));
  DG_CUDA(cudaMemsetAsync(sums, 0, d * 8, st));
  k_colsum<<<(unsigned)std::min<uint64_t>(n, 1024), 128, 0, st>>>(vec, n, d, dpad, sums);
  std::vector<double> hs(d);
  DG_CUDA(cudaMemcpyAsync(hs.data(), sums, d * 8, cudaMemcpyDeviceToHost, st));
  DG_CUDA(cudaStreamSynchronize(st));
  std::vector<float> hc(d);
  for (uint32_t j = 0; j < d; ++j) hc[j] = (float)(hs[j] / (double)n);
  DG_CUDA(cudaMemcpyAsync(cen, hc.data(), d * 4, cudaMemcpyHostToDevice, st));
  unsigned long long init[2] = {~0ull, ~0ull};
  DG_CUDA(cudaMemcpyAsync(best, init, 16, cudaMemcpyHostToDevice, st));
  k_medoid_min<<<grid_for(n, 256), 256, 0, st>>>(vec, n, d, dpad, cen, metric, best);
  k_medoid_arg<<<grid_for(n, 256), 256, 0, st>>>(vec, n, d, dpad, cen, metric, best, best + 1);
  unsigned long long res[2];
  DG_CUDA(cudaMemcpyAsync(res, best, 16, cudaMemcpyDeviceToHost, st));
  DG_CUDA(cudaStreamSynchronize(st));
  cudaFreeAsync(sums, st);
  cudaFreeAsync(cen, st);
  cudaFreeAsync(best, st);
  *out = (uint32_t)res[1];
  return DG_OK;
}

// -------------------------------------------------------------- exact kNN
// Brute force with FP64 accumulation.  A block holds 8 queries (one per
// warp); base rows stream through shared memory 32 at a time and each warp
// keeps its k best (distance, id) keys with the same merge as the search.
constexpr int kKnnWarps = 8;
__global__ void __launch_bounds__(256) k_exact_knn(const float *X, uint64_t n, uint32_t d, uint32_t dpad,
                                                   const float *Q, uint32_t nq, uint32_t k, int metric,
                                                   uint32_t kcap, uint32_t *out_ids, float *out_d) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rs = d + 1;  // padded row stride (bank-conflict free)
  float *tile = reinterpret_cast<float *>(sm);
  float *qsm = tile + 32 * rs;
  uint64_t *lists = reinterpret_cast<uint64_t *>(sm + align16((32 * rs + kKnnWarps * d) * 4));
  uint64_t *L0 = lists + (size_t)warp * (2 * kcap + 32);
  uint64_t *L1 = L0 + kcap;
  uint64_t *cst = L1 + kcap;
  const uint32_t q = blockIdx.x * kKnnWarps + warp;
  const bool active = q < nq;
  for (uint32_t j = lane; j < d; j += 32) qsm[warp * d + j] = active ? Q[(size_t)q * d + j] : 0.0f;
  double qq = 0.0;
  for (uint32_t j = 0; j < d; ++j) qq += (double)qsm[warp * d + j] * (double)qsm[warp * d + j];
  int size = 0, cur = 0;
  uint64_t *Ls[2] = {L0, L1};
  for (uint64_t base = 0; base < n; base += 32) {
    __syncthreads();
    const uint32_t rows = (uint32_t)((n - base) < 32 ? (n - base) : 32);
    for (uint32_t e = threadIdx.x; e < rows * d; e += blockDim.x) {
      const uint32_t r = e / d, c = e % d;
      tile[r * rs + c] = X[(base + r) * dpad + c];
    }
    __syncthreads();
    if (!active) continue;
    uint64_t key = kKeyInvalid;
    if ((uint32_t)lane < rows) {
      const float *x = tile + lane * rs;
      const float *qv = qsm + warp * d;
      double v;
      if (metric == DG_L2SQ || metric == DG_L2) {
        double s = 0.0;
        for (uint32_t j = 0; j < d; ++j) {
          double t = (double)qv[j] - (double)x[j];
          s = fma(t, t, s);
        }
        v = metric == DG_L2 ? sqrt(s) : s;
      } else {
        double ab = 0.0, bb = 0.0;
        for (uint32_t j = 0; j < d; ++j) {
          ab = fma((double)qv[j], (double)x[j], ab);
          bb = fma((double)x[j], (double)x[j], bb);
        }
        v = metric == DG_COSINE ? ((qq == 0.0 || bb == 0.0) ? 1.0 : 1.0 - ab / (sqrt(qq) * sqrt(bb)))
                                : 1.0 - ab;
      }
      key = make_key((float)v, (uint32_t)(base + lane));
    }
    // skip the merge when no lane beats the current k-th
    const bool maybe = key != kKeyInvalid && (size < (int)k || key < Ls[cur][k - 1]);
    if (!__any_sync(kFull, maybe)) continue;
    const int nc = prepare_batch(key, Ls[cur], size, (int)k, cst, lane);
    if (nc > 0) {
      size = merge_keys(Ls[cur], size, Ls[cur ^ 1], (int)k, cst, nc, lane);
      cur ^= 1;
    }
  }
  if (!active) return;
  for (int i = lane; i < (int)k; i += 32) {
    out_ids[(size_t)q * k + i] = i < size ? key_id(Ls[cur][i]) : DG_PAD;
    out_d[(size_t)q * k + i] = i < size ? key_dist(Ls[cur][i]) : __int_as_float(0x7f800000);
  }
}

// Tiled form for k <= kKnnTileK: a CTA takes 64 queries and a slice of the
// rows, 64 at a time; each thread owns a 4 x 4 tile of (query, row) pairs in
// FP64 registers, fed from shared memory that holds 16 coordinates of both
// sides as doubles (converted once per CTA instead of once per pair).  Every
// pair is summed in coordinate order with one rounding per operation, as the
// kernel above does, so the results are the same bits.  The distances of a
// tile go through shared memory to the warps, each keeping the k best keys of
// eight queries; entries beyond the smallest k-th distance any slice has seen
// (qthr) are dropped before insertion, and k_knn_merge joins the slices' lists.
// Bound by the FP64 pipe: a subtraction and an FMA per coordinate and pair,
// 1.4 ms for 1000 queries x 100k x 128 at 64 lanes per SM; the kernel above ran
// 125 CTAs of 8 warps and converted both operands of every pair.
constexpr int kKnnT = 64, kKnnJ = 16, kKnnTileK = 128;
constexpr int kKnnS = kKnnT + 2;  // row of 64 doubles, padded

template <bool L2>
__global__ void __launch_bounds__(256, 2) k_knn_tiled(const float *__restrict__ X, uint64_t n, uint32_t d,
                                                      uint32_t dpad, const float *__restrict__ Q, uint32_t nq,
                                                      uint32_t k, int metric, uint32_t kcap, uint64_t rows_per_slice,
                                                      uint32_t *qthr, uint64_t *part, uint32_t *part_cnt) {
  extern __shared__ __align__(16) uint8_t sm[];
  double *xs = reinterpret_cast<double *>(sm);                        // [kKnnJ][kKnnS]
  double *qs = xs + kKnnJ * kKnnS;                                    // [kKnnJ][kKnnS]
  float *dist = reinterpret_cast<float *>(qs + kKnnJ * kKnnS);        // [kKnnT queries][kKnnT + 1 rows]
  uint64_t *cst = reinterpret_cast<uint64_t *>(sm + align16(2 * kKnnJ * kKnnS * 8 + kKnnT * (kKnnT + 1) * 4));  // [8][32]
  uint64_t *lists = cst + 8 * 32;                                     // [kKnnT][2][kcap]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = tid & 15, ty = tid >> 4;  // rows tx + 16 i, queries ty + 16 i
  const uint32_t q0 = blockIdx.x * kKnnT;
  const uint64_t x0 = blockIdx.y * rows_per_slice, x1 = min(n, x0 + rows_per_slice);
  // loads: thread t takes coordinates 4 (t % 4) .. +3 of row / query t / 4
  const int lr = tid >> 2, lc = (tid & 3) * 4;
  int cur[8] = {}, size[8] = {};  // this warp's queries 8 warp + u
  for (uint64_t base = x0; base < x1; base += kKnnT) {
    double s[4][4], nx[4], nq_[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      nx[i] = nq_[i] = 0.0;
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.0;
    }
    float4 xv, qv;
    auto fetch = [&](uint32_t j0) {
      xv = qv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (base + lr < x1 && j0 + lc < dpad) xv = __ldg(reinterpret_cast<const float4 *>(X + (base + lr) * dpad + j0 + lc));
      if (q0 + lr < nq) {
        const float *q = Q + (size_t)(q0 + lr) * d + j0 + lc;
        if (j0 + lc < d) qv.x = __ldg(q);
        if (j0 + lc + 1 < d) qv.y = __ldg(q + 1);
        if (j0 + lc + 2 < d) qv.z = __ldg(q + 2);
        if (j0 + lc + 3 < d) qv.w = __ldg(q + 3);
      }
    };
    fetch(0);
    for (uint32_t j0 = 0; j0 < d; j0 += kKnnJ) {
      __syncthreads();  // the previous chunk (and the previous tile's distances) are consumed
      const float xa[4] = {xv.x, xv.y, xv.z, xv.w}, qa[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        xs[(lc + e) * kKnnS + lr] = (double)xa[e];
        qs[(lc + e) * kKnnS + lr] = (double)qa[e];
      }
      __syncthreads();
      if (j0 + kKnnJ < d) fetch(j0 + kKnnJ);  // in flight under the arithmetic
#pragma unroll 4
      for (int j = 0; j < kKnnJ; ++j) {
        double xr[4], qr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          xr[i] = xs[j * kKnnS + tx + 16 * i];
          qr[i] = qs[j * kKnnS + ty + 16 * i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (L2) {
              const double t = qr[i] - xr[c];
              s[i][c] = fma(t, t, s[i][c]);
            } else {
              s[i][c] = fma(qr[i], xr[c], s[i][c]);
            }
          }
          if (!L2) {
            nx[i] = fma(xr[i], xr[i], nx[i]);
            nq_[i] = fma(qr[i], qr[i], nq_[i]);
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        double v = s[i][c];
        if (L2) {
          if (metric == DG_L2) v = sqrt(v);
        } else if (metric == DG_COSINE) {
          v = (nq_[i] == 0.0 || nx[c] == 0.0) ? 1.0 : 1.0 - v / (sqrt(nq_[i]) * sqrt(nx[c]));
        } else {
          v = 1.0 - v;
        }
        dist[(ty + 16 * i) * (kKnnT + 1) + tx + 16 * c] = (float)v;
      }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t ql = 8 * warp + u, q = q0 + ql;
      if (q >= nq) break;
      uint64_t *const bufs[2] = {lists + (size_t)ql * 2 * kcap, lists + (size_t)ql * 2 * kcap + kcap};
      const uint32_t tb = *reinterpret_cast<volatile uint32_t *>(qthr + q);
      const uint64_t worst = size[u] >= (int)k ? bufs[cur[u]][k - 1] : kKeyInvalid;
      uint64_t key[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint64_t r = base + lane + 32 * h;
        key[h] = r < x1 ? make_key(dist[ql * (kKnnT + 1) + lane + 32 * h], (uint32_t)r) : kKeyInvalid;
        if (key_hi(key[h]) > tb || key[h] >= worst) key[h] = kKeyInvalid;
      }
      if (!__any_sync(kFull, key[0] != kKeyInvalid || key[1] != kKeyInvalid)) continue;
      insert_batch(key[0], bufs, cur[u], size[u], (int)k, cst + 32 * warp, lane);
      insert_batch(key[1], bufs, cur[u], size[u], (int)k, cst + 32 * warp, lane);
      if (size[u] >= (int)k && lane == 0) {
        const uint32_t nb = key_hi(bufs[cur[u]][k - 1]);
        if (nb < tb) atomicMin(qthr + q, nb);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const uint32_t ql = 8 * warp + u, q = q0 + ql;
    if (q >= nq) break;
    const uint64_t *l = lists + (size_t)ql * 2 * kcap + (size_t)cur[u] * kcap;
    const size_t at = (size_t)blockIdx.y * nq + q;
    for (int i = lane; i < size[u]; i += 32) part[at * k + i] = l[i];
    if (lane == 0) part_cnt[at] = (uint32_t)size[u];
  }
}

// The k smallest keys of a query's slice lists (a warp per query).
__global__ void __launch_bounds__(128) k_knn_merge(const uint64_t *part, const uint32_t *part_cnt, uint32_t slices,
                                                   uint32_t nq, uint32_t k, uint32_t *out_ids, float *out_d) {
  __shared__ uint64_t buf[4][2][kKnnTileK];
  __shared__ uint64_t cst[4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint64_t *const bufs[2] = {buf[warp][0], buf[warp][1]};
  for (uint32_t q = blockIdx.x * 4 + warp; q < nq; q += gridDim.x * 4) {
    int cur = 0, size = 0;
    for (uint32_t sl = 0; sl < slices; ++sl) {
      const size_t at = (size_t)sl * nq + q;
      const uint32_t c = part_cnt[at];
      for (uint32_t j0 = 0; j0 < c; j0 += 32) {
        const uint32_t j = j0 + lane;
        insert_batch(j < c ? part[at * k + j] : kKeyInvalid, bufs, cur, size, (int)k, cst[warp], lane);
      }
    }
    for (int i = lane; i < (int)k; i += 32) {
      out_ids[(size_t)q * k + i] = i < size ? key_id(bufs[cur][i]) : DG_PAD;
      out_d[(size_t)q * k + i] = i < size ? key_dist(bufs[cur][i]) : __int_as_float(0x7f800000);
    }
    __syncwarp();
  }
}

// Launches the tiled kNN: the rows are cut into the number of slices that costs
// the busiest of the resident CTAs (2 per SM for k up to 64, 1 above, whose lists
// take 128 KB) least, as far as the slices' lists stay within kKnnPartBytes.  A
// tile takes about 5.5 + 0.11 dim us; filling the lists of a slice's 64 queries
// 12 k us more, whatever its length, so that long lists want few slices (100k
// rows, 10k queries, k = 100, 16 / 3 slices: 8-d 51.6 / 30.5 ms, 32-d 51.4 / 31.9;
// 20k x 128-d queries, k = 64, 16 / 4: 85.9 / 61.5).
constexpr size_t kKnnPartBytes = (size_t)256 << 20;
static DgStatus knn_tiled(const float *v, uint64_t n, uint32_t dim, uint32_t dpad, const float *q, uint32_t nq,
                          uint32_t k, int metric, uint32_t *oi, float *od, cudaStream_t st) {
  int dev = 0, sms = 0;
  DG_CUDA(cudaGetDevice(&dev));
  DG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  uint32_t kcap = 16;
  while (kcap < k) kcap <<= 1;
  const size_t smem = align16(2 * kKnnJ * kKnnS * 8 + kKnnT * (kKnnT + 1) * 4) + 8 * 32 * 8 + (size_t)kKnnT * 2 * kcap * 8;
  const bool l2 = metric == DG_L2SQ || metric == DG_L2;
  auto kern = l2 ? k_knn_tiled<true> : k_knn_tiled<false>;
  int per_sm = 0;
  DG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  DG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem));
  const uint64_t qb = (nq + kKnnT - 1) / kKnnT, tiles = (n + kKnnT - 1) / kKnnT;
  const uint64_t slots = (uint64_t)std::max(1, per_sm) * sms;
  const uint64_t most = std::min({tiles, 4 * slots, (uint64_t)(kKnnPartBytes / std::max<size_t>((size_t)nq * k * 8, 1))});
  const double fill = 12.0 * k / (5.5 + 0.11 * dim);  // in tiles
  double best = 1e300;
  uint64_t slices = 1;
  for (uint64_t s = 1; s <= most; ++s) {
    const double cost = (double)((qb * s + slots - 1) / slots) * ((double)((tiles + s - 1) / s + 2) + fill);
    if (cost < best) {
      best = cost;
      slices = s;
    }
  }
  const uint64_t rows = (tiles + slices - 1) / slices * kKnnT;
  slices = (n + rows - 1) / rows;
  uint32_t *thr = nullptr, *pc = nullptr;
  uint64_t *part = nullptr;
  if (cudaMallocAsync(&thr, (size_t)nq * 4, st) != cudaSuccess ||
      cudaMallocAsync(&pc, (size_t)slices * nq * 4, st) != cudaSuccess ||
      cudaMallocAsync(&part, (size_t)slices * nq * k * 8, st) != cudaSuccess) {
    for (void *p : {(void *)thr, (void *)pc, (void *)part})
      if (p) cudaFreeAsync(p, st);
    cudaGetLastError();
    return fail(DG_ENOMEM, "exact knn staging");
  }
  DgStatus s = DG_OK;
  cudaError_t e = cudaMemsetAsync(thr, 0xff, (size_t)nq * 4, st);
  if (e == cudaSuccess) {
    kern<<<dim3((unsigned)qb, (unsigned)slices), 256, smem, st>>>(v, n, dim, dpad, q, nq, k, metric, kcap, rows, thr,
                                                                  part, pc);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    k_knn_merge<<<(unsigned)std::min<uint32_t>((nq + 3) / 4, 148 * 16), 128, 0, st>>>(part, pc, (uint32_t)slices, nq, k,
                                                                                   oi, od);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) s = cuda_fail(e, "exact knn launch");
  cudaFreeAsync(thr, st);
  cudaFreeAsync(pc, st);
  cudaFreeAsync(part, st);
  return s;
}

// Whether the tiled kernel takes a call (the same results either way).  Its
// tiles halve and better the FP64 time of a pair, 0.4 ps x dim on the whole GPU;
// its slices and 64-query barriers make a list entry dearer, by 22 ns at 100k rows
// and about in proportion to the root of their number.  So few coordinates, few
// rows and long lists favour one list per query, once there are enough queries to
// fill the GPU that way (ms, one list / tiles; 10k queries x 100k rows: 8-d, k = 10
// 10.0 / 10.2, k = 100 15.6 / 31.4; 32-d, k = 32 24.8 / 19.4, k = 100 28.1 / 33.4;
// 128-d, k = 128 86 / 53; 10k rows: 32-d, k = 10 3.3 / 3.5, k = 100 4.9 / 10.7; 1000
// queries x 100k rows: 8-d, k = 128 6.7 / 7.4, 16-d 7.8 / 7.4, 32-d 11.0 / 8.3; 500
// queries: 8-d 6.6 / 4.6).  Lists above kKnnTileK do not fit a tile CTA; above
// 1024 coordinates tiles always win.
static bool knn_by_tiles(uint64_t n, uint32_t dim, uint32_t nq, uint32_t k) {
  if (k > (uint32_t)kKnnTileK) return false;
  return nq <= (dim < 16 ? 512u : 1024u) || dim > 1024 || 200.0 * k <= dim * std::sqrt((double)n);
}

// ------------------------------------------------------------ PQ training
// ProductQuantizer::train (src/pq.rs:51-119): per subspace, k-means++ seeding
// then Lloyd iterations; empty clusters restart from a random training point.
// One seeding step of every subspace (grid.y): distances to the newest seed
// lower mind (the first step, c_new = 1, starts it), and the last block of a
// subspace to finish draws seed c_new with probability proportional to mind:
// the first point whose running sum of mind (FP64) reaches u * total.  A block
// covers kSeedPts points; its partial sums let the last block find the drawn
// point in two scans.  One launch per seed; before, an update kernel and a
// 1024-thread pick whose thread 0 added the partial sums one by one took
// 31 + 61 us for 50k points x 16 subspaces.
constexpr int kSeedPts = 1024;

// Inclusive running sums over the 256 threads of a block (s: 8 doubles).
__device__ __forceinline__ double block_scan256(double v, double *s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += t;
  }
  __syncthreads();  // s may still be read from the previous scan
  if (lane == 31) s[warp] = v;
  __syncthreads();
  double before = 0.0;
  for (int w = 0; w < warp; ++w) before += s[w];
  return before + v;
}

__global__ void __launch_bounds__(256) k_seed_step(const float *__restrict__ S, uint32_t ns, uint32_t d, uint32_t ds,
                                                   float *cb, uint32_t K, uint32_t c_new, float *mind, double *part,
                                                   unsigned int *done, uint64_t seed) {
  __shared__ double scan[8];
  __shared__ unsigned int s_pick;
  const uint32_t m = blockIdx.y, nblk = gridDim.x;
  const float *cen = cb + ((size_t)m * K + c_new - 1) * ds;
  float *md = mind + (size_t)m * ns;
  double *pm = part + (size_t)m * nblk;
  const bool vec = ds % 4 == 0 && d % 4 == 0;
  double sum = 0.0;
#pragma unroll
  for (int u = 0; u < kSeedPts / 256; ++u) {
    const uint32_t i = blockIdx.x * kSeedPts + u * 256 + threadIdx.x;
    if (i >= ns) break;
    const float *x = S + (size_t)i * d + m * ds;
    float acc = 0.0f;
    if (vec) {
      for (uint32_t j = 0; j < ds; j += 4) {
        const float4 xv = __ldg(reinterpret_cast<const float4 *>(x + j));
        const float xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float t = __fsub_rn(xs[e], cen[j + e]);
          acc = __fadd_rn(acc, __fmul_rn(t, t));
        }
      }
    } else {
      for (uint32_t j = 0; j < ds; ++j) {
        const float t = __fsub_rn(x[j], cen[j]);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
      }
    }
    const float v = fminf(c_new == 1 ? 3.402823466e38f : md[i], acc);
    md[i] = v;
    sum += (double)v;
  }
  const double incl = block_scan256(sum, scan);
  __threadfence();  // this block's mind before its mark
  if (threadIdx.x == 255) pm[blockIdx.x] = incl;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_pick = atomicAdd(done + m, 1u);
  __syncthreads();
  if (s_pick != nblk - 1) return;
  // the last block of the subspace: the total, then the block and the point
  __threadfence();
  double tot = 0.0;
  for (uint32_t b = threadIdx.x; b < nblk; b += 256) tot += __ldcg(pm + b);
  tot = block_scan256(tot, scan);
  __syncthreads();
  if (threadIdx.x == 255) scan[0] = tot;
  if (threadIdx.x == 0) s_pick = ns - 1;
  __syncthreads();
  tot = scan[0];
  __syncthreads();
  if (tot <= 0.0) {
    if (threadIdx.x == 0) s_pick = (uint32_t)range_of(rand4(seed, 0x6b6e, m, c_new), ns);
  } else {
    const double u = (double)(rand4(seed, 0x6b6d, m, c_new) >> 11) * (1.0 / 9007199254740992.0);
    const double thr = u * tot;
    // running sums over blocks, then over the points of the block that reaches thr
    double base = 0.0;
    uint32_t blk = nblk;  // (none: the last point)
    for (uint32_t b0 = 0; b0 < nblk && blk == nblk; b0 += 256) {
      const uint32_t b = b0 + threadIdx.x;
      const double v = b < nblk ? __ldcg(pm + b) : 0.0;
      const double c = base + block_scan256(v, scan);
      __shared__ uint32_t s_first;
      __shared__ double s_base;
      if (threadIdx.x == 0) s_first = 0xffffffffu;
      __syncthreads();
      if (b < nblk && c >= thr) atomicMin(&s_first, b);
      __syncthreads();
      if (s_first != 0xffffffffu ? b == s_first : threadIdx.x == 255) s_base = s_first != 0xffffffffu ? c - v : c;
      __syncthreads();
      base = s_base;
      if (s_first != 0xffffffffu) blk = s_first;
      __syncthreads();
    }
    if (blk < nblk) {
      if (threadIdx.x == 0) s_pick = min(ns, (blk + 1) * (uint32_t)kSeedPts) - 1;
      __syncthreads();
      double v[kSeedPts / 256], s4 = 0.0;
#pragma unroll
      for (int e = 0; e < kSeedPts / 256; ++e) {  // four consecutive points per thread
        const uint32_t i = blk * kSeedPts + threadIdx.x * (kSeedPts / 256) + e;
        v[e] = i < ns ? (double)__ldcg(md + i) : 0.0;
        s4 += v[e];
      }
      double c = base + block_scan256(s4, scan) - s4;
#pragma unroll
      for (int e = 0; e < kSeedPts / 256; ++e) {
        const uint32_t i = blk * kSeedPts + threadIdx.x * (kSeedPts / 256) + e;
        c += v[e];
        if (i < ns && c >= thr) {
          atomicMin(&s_pick, i);
          break;
        }
      }
    }
  }
  __syncthreads();
  const uint32_t chosen = s_pick;
  for (uint32_t j = threadIdx.x; j < ds; j += 256)
    cb[((size_t)m * K + c_new) * ds + j] = S[(size_t)chosen * d + m * ds + j];
  if (threadIdx.x == 0) done[m] = 0u;
}

// Sums and counts of the points of each cluster (codes: [M][ns]).  A block
// sorts the numbers of kAccPts points of one subspace by code in shared memory
// (counting sort), then a warp adds up one cluster's points, lanes over points
// and coordinates, so that each block adds to a cluster's sums once.  Adding
// every point's coordinates to global memory took 6.4 ms per iteration for 50k
// points x 16 subspaces x 8 (FP64 atomics on 2048 addresses per subspace).
constexpr int kAccPts = 2048;
__global__ void __launch_bounds__(256) k_cluster_sums(const float *__restrict__ S, uint32_t ns, uint32_t d,
                                                      uint32_t ds, uint32_t K, const uint8_t *__restrict__ codes,
                                                      double *sums, unsigned int *counts) {
  __shared__ uint32_t start[257], fill[256];
  __shared__ uint16_t order[kAccPts];
  const uint32_t m = blockIdx.y, p0 = blockIdx.x * kAccPts, np = min((uint32_t)kAccPts, ns - p0);
  const uint8_t *cm = codes + (size_t)m * ns + p0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  fill[threadIdx.x] = 0u;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < np; i += 256) atomicAdd(fill + cm[i], 1u);
  __syncthreads();
  if (warp == 0) {  // exclusive prefix of the 256 counts, eight per lane
    uint32_t c[8], sum = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      c[e] = sum;
      sum += fill[8 * lane + e];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, o);
      if (lane >= o) incl += t;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) start[8 * lane + e] = incl - sum + c[e];
    if (lane == 31) start[256] = incl;
  }
  __syncthreads();
  fill[threadIdx.x] = start[threadIdx.x];
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < np; i += 256) order[atomicAdd(fill + cm[i], 1u)] = (uint16_t)i;
  __syncthreads();
  // lanes: `w` coordinates (a power of two) x 32 / w points
  uint32_t w = 1;
  while (w < ds && w < 32) w <<= 1;
  const uint32_t jl = lane & (w - 1), pl = lane / w, pn = 32 / w;
  for (uint32_t c = warp; c < K; c += 8) {
    const uint32_t b = start[c], e = start[c + 1];
    if (b == e) continue;
    for (uint32_t j0 = 0; j0 < ds; j0 += w) {
      double acc = 0.0;
      if (j0 + jl < ds)
        for (uint32_t i = b + pl; i < e; i += pn) acc += (double)__ldg(S + (size_t)(p0 + order[i]) * d + m * ds + j0 + jl);
      for (uint32_t o = w; o < 32; o <<= 1) acc += __shfl_xor_sync(kFull, acc, o);
      if (pl == 0 && j0 + jl < ds) atomicAdd(sums + ((size_t)m * K + c) * ds + j0 + jl, acc);
    }
    if (lane == 0) atomicAdd(counts + (size_t)m * K + c, e - b);
  }
}
__global__ void k_update(const float *S, uint32_t ns, uint32_t d, uint32_t M, uint32_t ds, float *cb,
                         uint32_t K, const double *sums, const unsigned int *counts, uint64_t seed,
                         uint32_t iter) {
  const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= M * K) return;
  const uint32_t m = e / K, c = e % K;
  const unsigned int cnt = counts[e];
  if (cnt > 0) {
    for (uint32_t j = 0; j < ds; ++j) cb[(size_t)e * ds + j] = (float)(sums[(size_t)e * ds + j] / (double)cnt);
  } else {
    const uint32_t r = (uint32_t)range_of(rand4(seed, 0x6b6f + iter, m, c), ns);
    for (uint32_t j = 0; j < ds; ++j) cb[(size_t)e * ds + j] = S[(size_t)r * d + m * ds + j];
  }
}

}  // namespace dg

using namespace dg;

extern "C" {

DgStatus dg_medoid(const float *X, uint64_t n, uint32_t dim, int32_t metric, int32_t device,
                   uint32_t *out_medoid) {
  if (!X || !out_medoid || n == 0 || dim == 0) return fail(DG_EINVAL, "bad medoid arguments");
  DG_CUDA(cudaSetDevice(device));
  const uint32_t dpad = dpad_of(dim);
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  float *v = nullptr;
  DgStatus s = DG_OK;
  if (cudaMallocAsync(&v, n * dpad * 4, st) != cudaSuccess) s = fail(DG_ENOMEM, "medoid staging");
  if (s == DG_OK) s = upload_rows_f32(X, n, dim, dpad, v, st);
  if (s == DG_OK) s = medoid_device(v, n, dim, dpad, metric, out_medoid, st);
  if (v) cudaFreeAsync(v, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}

DgStatus dg_fp8_encode(const float *X, uint64_t n, uint32_t dim, int32_t device, uint8_t *out_codes,
                       float *out_scales) {
  if (!X || !out_codes || !out_scales) return fail(DG_EINVAL, "null argument");
  if (n == 0 || dim == 0) return DG_OK;
  DG_CUDA(cudaSetDevice(device));
  const uint32_t dpad = dpad_of(dim);
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  float *v = nullptr;
  uint8_t *codes = nullptr;
  float2 *sn = nullptr;
  DgStatus s = DG_OK;
  if (cudaMallocAsync(&v, n * dpad * 4, st) != cudaSuccess || cudaMallocAsync(&codes, n * dpad, st) != cudaSuccess ||
      cudaMallocAsync(&sn, n * sizeof(float2), st) != cudaSuccess)
    s = fail(DG_ENOMEM, "fp8 encode staging");
  if (s == DG_OK) s = upload_rows_f32(X, n, dim, dpad, v, st);
  if (s == DG_OK) s = encode_fp8_device(v, n, dim, dpad, codes, sn, st);
  if (s == DG_OK && cudaMemcpy2DAsync(out_codes, dim, codes, dpad, dim, n, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    s = fail(DG_EDEVICE, "code download");
  if (s == DG_OK && cudaMemcpy2DAsync(out_scales, 4, sn, sizeof(float2), 4, n, cudaMemcpyDeviceToHost, st) !=
                        cudaSuccess)
    s = fail(DG_EDEVICE, "scale download");
  cudaStreamSynchronize(st);
  if (v) cudaFreeAsync(v, st);
  if (codes) cudaFreeAsync(codes, st);
  if (sn) cudaFreeAsync(sn, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}

DgStatus dg_pq_encode(const float *X, uint64_t n, uint32_t dim, uint32_t M, uint32_t K,
                      const float *codebooks, int32_t device, uint8_t *out_codes) {
  if (!X || !codebooks || !out_codes) return fail(DG_EINVAL, "null argument");
  if (M == 0 || dim % M) return fail(DG_EINVAL, "dimension not divisible by num_subspaces");
  if (K == 0 || K > 256) return fail(DG_EINVAL, "num_centroids must be in [1, 256]");
  DG_CUDA(cudaSetDevice(device));
  const uint32_t dpad = dpad_of(dim);
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  float *v = nullptr, *cb = nullptr;
  uint8_t *codes = nullptr;
  DgStatus s = DG_OK;
  const size_t cbb = (size_t)M * K * (dim / M) * 4;
  if (cudaMallocAsync(&v, n * dpad * 4, st) != cudaSuccess || cudaMallocAsync(&cb, cbb, st) != cudaSuccess ||
      cudaMallocAsync(&codes, n * M, st) != cudaSuccess)
    s = fail(DG_ENOMEM, "pq encode staging");
  if (s == DG_OK) s = upload_rows_f32(X, n, dim, dpad, v, st);
  if (s == DG_OK && cudaMemcpyAsync(cb, codebooks, cbb, cudaMemcpyHostToDevice, st) != cudaSuccess)
    s = fail(DG_EDEVICE, "codebook upload");
  if (s == DG_OK) s = encode_pq_device(v, n, dim, dpad, M, K, cb, codes, M, st);
  if (s == DG_OK && cudaMemcpyAsync(out_codes, codes, n * M, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    s = fail(DG_EDEVICE, "code download");
  cudaStreamSynchronize(st);
  if (v) cudaFreeAsync(v, st);
  if (cb) cudaFreeAsync(cb, st);
  if (codes) cudaFreeAsync(codes, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}

DgStatus dg_rabitq_encode(const float *X, uint64_t n, uint32_t dim, uint32_t padded, const float *centroid,
                          const float *signs, int32_t device, uint8_t *out_codes) {
  if (!X || !centroid || !signs || !out_codes) return fail(DG_EINVAL, "null argument");
  if (padded < 64 || (padded & (padded - 1)) || padded < dim) return fail(DG_EINVAL, "bad padded dimension");
  if (n == 0) return DG_OK;
  DG_CUDA(cudaSetDevice(device));
  const uint32_t dpad = dpad_of(dim), cs = padded / 8 + 8;
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  float *v = nullptr, *cen = nullptr, *sg = nullptr;
  uint8_t *codes = nullptr;
  DgStatus s = DG_OK;
  if (cudaMallocAsync(&v, n * dpad * 4, st) != cudaSuccess || cudaMallocAsync(&cen, (size_t)dim * 4, st) != cudaSuccess ||
      cudaMallocAsync(&sg, (size_t)3 * padded * 4, st) != cudaSuccess ||
      cudaMallocAsync(&codes, n * cs, st) != cudaSuccess)
    s = fail(DG_ENOMEM, "rabitq encode staging");
  if (s == DG_OK) s = upload_rows_f32(X, n, dim, dpad, v, st);
  if (s == DG_OK && (cudaMemcpyAsync(cen, centroid, (size_t)dim * 4, cudaMemcpyHostToDevice, st) != cudaSuccess ||
                     cudaMemcpyAsync(sg, signs, (size_t)3 * padded * 4, cudaMemcpyHostToDevice, st) != cudaSuccess))
    s = fail(DG_EDEVICE, "rabitq parameter upload");
  if (s == DG_OK) s = encode_rabitq_device(v, n, dim, dpad, padded, cen, sg, codes, cs, st);
  if (s == DG_OK && cudaMemcpyAsync(out_codes, codes, n * cs, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    s = fail(DG_EDEVICE, "code download");
  cudaStreamSynchronize(st);
  for (void *p : {(void *)v, (void *)cen, (void *)sg, (void *)codes})
    if (p) cudaFreeAsync(p, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}

DgStatus dg_pq_train(const float *X, uint64_t n, uint32_t dim, uint32_t M, uint32_t K,
                     uint32_t iterations, uint64_t sample, uint64_t seed, int32_t device,
                     float *out_codebooks) {
  if (!X || !out_codebooks || n == 0) return fail(DG_EINVAL, "No vectors to train on");
  if (K > 256) return fail(DG_EINVAL, "num_centroids " + std::to_string(K) + " exceeds 256 (codes are u8)");
  if (M == 0 || dim % M)
    return fail(DG_EINVAL, "Dimension " + std::to_string(dim) + " not divisible by num_subspaces " +
                               std::to_string(M));
  if (K == 0) return fail(DG_EINVAL, "num_centroids must be >= 1");
  DG_CUDA(cudaSetDevice(device));
  const uint32_t ds = dim / M;
  // training sample (src/pq.rs:75-82): `sample` distinct rows drawn by a
  // seeded partial Fisher-Yates shuffle when the set is larger
  std::vector<uint64_t> rows;
  if (sample > 0 && n > sample) {
    std::vector<uint64_t> perm(n);
    for (uint64_t i = 0; i < n; ++i) perm[i] = i;
    for (uint64_t i = 0; i < sample; ++i) {
      uint64_t j = i + (uint64_t)(((unsigned __int128)rand4(seed, 0x7371, i, 0) * (n - i)) >> 64);
      std::swap(perm[i], perm[j]);
    }
    rows.assign(perm.begin(), perm.begin() + sample);
  } else {
    rows.resize(n);
    for (uint64_t i = 0; i < n; ++i) rows[i] = i;
  }
  const uint32_t ns = (uint32_t)rows.size();
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  float *S = nullptr, *cb = nullptr, *mind = nullptr;
  double *sums = nullptr, *part = nullptr;
  unsigned int *counts = nullptr, *done = nullptr;
  uint8_t *codes = nullptr;
  DgStatus s = DG_OK;
  const size_t cbn = (size_t)M * K * ds;
  const uint32_t nblk = (ns + kSeedPts - 1) / kSeedPts;
  if (cudaMallocAsync(&S, (size_t)ns * dim * 4, st) != cudaSuccess || cudaMallocAsync(&cb, cbn * 4, st) != cudaSuccess ||
      cudaMallocAsync(&mind, (size_t)M * ns * 4, st) != cudaSuccess ||
      cudaMallocAsync(&sums, cbn * 8, st) != cudaSuccess ||
      cudaMallocAsync(&counts, (size_t)M * K * 4, st) != cudaSuccess ||
      cudaMallocAsync(&part, (size_t)M * nblk * 8, st) != cudaSuccess ||
      cudaMallocAsync(&done, (size_t)M * 4, st) != cudaSuccess ||
      cudaMallocAsync(&codes, (size_t)M * ns, st) != cudaSuccess)
    s = fail(DG_ENOMEM, "pq training staging");
  if (s == DG_OK) s = upload_rows_f32(X, ns, dim, dim, S, st, rows.data());
  if (s == DG_OK) {
    // k-means++ seeding (src/pq.rs:301-341)
    cudaMemsetAsync(done, 0, (size_t)M * 4, st);
    const uint32_t keff = std::min<uint32_t>(K, ns);
    std::vector<float> hcb(cbn);
    for (uint32_t m = 0; m < M; ++m) {
      const uint32_t first = (uint32_t)(((unsigned __int128)rand4(seed, 0x6b6c, m, 0) * ns) >> 64);
      const float *x = X + rows[first] * dim + m * ds;
      std::copy(x, x + ds, hcb.begin() + (size_t)m * K * ds);
    }
    cudaMemcpyAsync(cb, hcb.data(), cbn * 4, cudaMemcpyHostToDevice, st);
    for (uint32_t c = 1; c < keff; ++c)
      k_seed_step<<<dim3(nblk, M), 256, 0, st>>>(S, ns, dim, ds, cb, K, c, mind, part, done, seed);
    // replicate when K exceeds the sample (src/pq.rs:344-350)
    if (keff < K) {
      cudaMemcpyAsync(hcb.data(), cb, cbn * 4, cudaMemcpyDeviceToHost, st);
      cudaStreamSynchronize(st);
      for (uint32_t m = 0; m < M; ++m)
        for (uint32_t c = keff; c < K; ++c)
          std::copy(hcb.begin() + ((size_t)m * K + c % keff) * ds, hcb.begin() + ((size_t)m * K + c % keff) * ds + ds,
                    hcb.begin() + ((size_t)m * K + c) * ds);
      cudaMemcpyAsync(cb, hcb.data(), cbn * 4, cudaMemcpyHostToDevice, st);
    }
    // Lloyd iterations (src/pq.rs:353-408)
    for (uint32_t it = 0; it < iterations && s == DG_OK; ++it) {
      cudaMemsetAsync(sums, 0, cbn * 8, st);
      cudaMemsetAsync(counts, 0, (size_t)M * K * 4, st);
      s = pq_codes(S, ns, dim, M, K, ds, cb, codes, 1, ns, st);
      k_cluster_sums<<<dim3((ns + kAccPts - 1) / kAccPts, M), 256, 0, st>>>(S, ns, dim, ds, K, codes, sums, counts);
      k_update<<<(M * K + 255) / 256, 256, 0, st>>>(S, ns, dim, M, ds, cb, K, sums, counts, seed, it);
    }
    if (cudaMemcpyAsync(out_codebooks, cb, cbn * 4, cudaMemcpyDeviceToHost, st) != cudaSuccess)
      s = fail(DG_EDEVICE, "codebook download");
    if (cudaStreamSynchronize(st) != cudaSuccess) s = fail(DG_EDEVICE, cudaGetErrorString(cudaGetLastError()));
  }
  if (S) cudaFreeAsync(S, st);
  if (cb) cudaFreeAsync(cb, st);
  if (mind) cudaFreeAsync(mind, st);
  if (sums) cudaFreeAsync(sums, st);
  if (counts) cudaFreeAsync(counts, st);
  if (part) cudaFreeAsync(part, st);
  if (done) cudaFreeAsync(done, st);
  if (codes) cudaFreeAsync(codes, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}

DgStatus dg_exact_knn(const float *X, uint64_t n, uint32_t dim, const float *Q, uint32_t nq,
                      uint32_t k, int32_t metric, int32_t device, uint32_t *out_ids,
                      float *out_dists) {
  if (!X || !Q || !out_ids || !out_dists || n == 0 || dim == 0) return fail(DG_EINVAL, "bad arguments");
  if (k == 0 || k > 1024) return fail(DG_EINVAL, "k must be in [1, 1024]");
  DG_CUDA(cudaSetDevice(device));
  const uint32_t dpad = dpad_of(dim);
  cudaStream_t st;
  DG_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
  float *v = nullptr, *q = nullptr, *od = nullptr;
  uint32_t *oi = nullptr;
  DgStatus s = DG_OK;
  if (cudaMallocAsync(&v, n * dpad * 4, st) != cudaSuccess || cudaMallocAsync(&q, (size_t)nq * dim * 4, st) != cudaSuccess ||
      cudaMallocAsync(&oi, (size_t)nq * k * 4, st) != cudaSuccess ||
      cudaMallocAsync(&od, (size_t)nq * k * 4, st) != cudaSuccess)
    s = fail(DG_ENOMEM, "exact knn staging");
  if (s == DG_OK) s = upload_rows_f32(X, n, dim, dpad, v, st);
  if (s == DG_OK) cudaMemcpyAsync(q, Q, (size_t)nq * dim * 4, cudaMemcpyHostToDevice, st);
  bool tiled = s == DG_OK && knn_by_tiles(n, dim, nq, k);
  if (tiled && (s = knn_tiled(v, n, dim, dpad, q, nq, k, metric, oi, od, st)) == DG_ENOMEM) {
    tiled = false;  // the partial lists do not fit beside the rows: the other kernel needs none
    s = DG_OK;
  }
  if (s == DG_OK && !tiled) {  // 8 queries per CTA, one list each
    uint32_t kcap = 32;
    while (kcap < k) kcap <<= 1;
    const size_t smem = align16((32 * (dim + 1) + kKnnWarps * dim) * 4) + (size_t)kKnnWarps * (2 * kcap + 32) * 8;
    if (cudaFuncSetAttribute(k_exact_knn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      s = fail(DG_ENOTSUP, "exact knn tile does not fit in shared memory");
    if (s == DG_OK) {
      k_exact_knn<<<(nq + kKnnWarps - 1) / kKnnWarps, 256, smem, st>>>(v, n, dim, dpad, q, nq, k, metric, kcap, oi, od);
      if (cudaGetLastError() != cudaSuccess) s = fail(DG_EDEVICE, "exact knn launch");
    }
  }
  if (s == DG_OK) {
    cudaMemcpyAsync(out_ids, oi, (size_t)nq * k * 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(out_dists, od, (size_t)nq * k * 4, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) s = fail(DG_EDEVICE, "exact knn failed");
  }
  if (v) cudaFreeAsync(v, st);
  if (q) cudaFreeAsync(q, st);
  if (oi) cudaFreeAsync(oi, st);
  if (od) cudaFreeAsync(od, st);
  cudaStreamSynchronize(st);
  cudaStreamDestroy(st);
  return s;
}

}  // extern "C"
