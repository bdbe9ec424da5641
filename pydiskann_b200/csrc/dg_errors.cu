// dg_errors.cu -- per-thread error text, status helpers, the row padding
// rule and the padded row upload, shared by the search library (libdgann) and the index-construction
// library (libdgbuild).
#include <algorithm>
#include <cstring>
#include <exception>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "dg_index.h"

namespace dg {

static thread_local std::string g_err;

void set_error(const std::string &msg) { g_err = msg; }
DgStatus fail(DgStatus st, const std::string &msg) {
  g_err = msg;
  return st;
}
DgStatus cuda_fail(cudaError_t e, const char *what) {
  g_err = std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? DG_ENOMEM : DG_EDEVICE;
}

// Rows are padded to a multiple of 32 dimensions: every 16-byte chunk
// geometry of the gather kernels then divides the row exactly.
uint32_t dpad_of(uint32_t d) { return (d + 31u) & ~31u; }

// Pinned staging of large uploads from pageable memory: kUpThreads threads copy
// pieces of kUpPiece bytes into page-locked buffers (two each) and send them
// from there, so that the host copies run in parallel and overlap the
// transfers; the driver's own staging runs on one thread at 11 GB/s.  The
// buffers (16 MB) are page-locked once per process, since locking them costs
// as much as an upload of 50 MB, and given back when it ends; one upload uses
// them at a time, a concurrent one takes the plain copy.
constexpr int kUpThreads = 4, kUpBufs = 2;
constexpr size_t kUpPiece = 2u << 20, kUpMin = 4u << 20;
struct UploadPool {
  std::mutex mu;
  uint8_t *mem = nullptr;
  ~UploadPool() {
    if (mem) cudaFreeHost(mem);
  }
};
static UploadPool &upload_pool() {
  static UploadPool p;
  return p;
}

// Rows of d floats into rows of dpad floats, zero padded (a strided copy of
// short rows runs at a few GB/s: 400k x 100, 30 ms).
__global__ void k_pad_rows(const float *__restrict__ src, uint64_t n, uint32_t d, uint32_t dpad, float4 *dst) {
  const uint32_t q = dpad / 4;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < n * q; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t r = e / q;
    const uint32_t c = 4 * (uint32_t)(e - r * q);
    const float *x = src + r * d + c;
    dst[e] = make_float4(c < d ? x[0] : 0.0f, c + 1 < d ? x[1] : 0.0f, c + 2 < d ? x[2] : 0.0f, c + 3 < d ? x[3] : 0.0f);
  }
}

// Rows i of `host` (or rows[i], when given), d floats each, to dev with rows
// dpad floats apart (padding zero).  A pageable source has been read when this
// returns; one that the caller page-locked is read in stream order.
DgStatus upload_rows_f32(const float *host, uint64_t n, uint32_t d, uint32_t dpad, float *dev, cudaStream_t st,
                         const uint64_t *rows) {
  const size_t row = (size_t)d * sizeof(float);
  int device = 0;
  DG_CUDA(cudaGetDevice(&device));
  UploadPool &pool = upload_pool();
  std::unique_lock<std::mutex> lk(pool.mu, std::defer_lock);
  bool staged = n * row >= kUpMin && row <= kUpPiece;
  if (staged && !rows) {  // page-locked by the caller: the transfer reads it directly
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, host) != cudaSuccess) cudaGetLastError();
    else staged = at.type == cudaMemoryTypeUnregistered;
  }
  staged = staged && lk.try_lock();
  if (staged && !pool.mem &&
      cudaHostAlloc((void **)&pool.mem, kUpThreads * kUpBufs * kUpPiece, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    pool.mem = nullptr;
    staged = false;
  }
  uint8_t *landing = nullptr;  // padded rows: pieces land here and are spread by k_pad_rows, in stream order
  if (staged && d != dpad &&
      cudaMallocAsync((void **)&landing, kUpThreads * kUpBufs * kUpPiece, st) != cudaSuccess) {
    cudaGetLastError();  // (a device full but for the rows: the strided copy needs no room)
    landing = nullptr;
    staged = false;
  }
  if (!staged) {
    std::vector<float> gathered;
    if (rows) {
      gathered.resize(n * d);
      for (uint64_t i = 0; i < n; ++i) std::memcpy(gathered.data() + i * d, host + rows[i] * d, row);
      host = gathered.data();
    }
    if (d == dpad) {
      DG_CUDA(cudaMemcpyAsync(dev, host, n * row, cudaMemcpyHostToDevice, st));
    } else {
      DG_CUDA(cudaMemsetAsync(dev, 0, n * dpad * sizeof(float), st));
      DG_CUDA(cudaMemcpy2DAsync(dev, dpad * sizeof(float), host, row, row, n, cudaMemcpyHostToDevice, st));
    }
    if (rows) DG_CUDA(cudaStreamSynchronize(st));  // the gathered copy goes now
    return DG_OK;
  }
  const uint64_t per = kUpPiece / row, pieces = (n + per - 1) / per;
  cudaError_t err[kUpThreads] = {};
  auto work = [&](int t) {
    cudaError_t e = cudaSetDevice(device);
    cudaEvent_t sent[kUpBufs] = {};
    for (int b = 0; b < kUpBufs && e == cudaSuccess; ++b) e = cudaEventCreateWithFlags(&sent[b], cudaEventDisableTiming);
    int b = 0;
    for (uint64_t p = t; p < pieces && e == cudaSuccess; p += kUpThreads, b = (b + 1) % kUpBufs) {
      uint8_t *buf = pool.mem + (size_t)(t * kUpBufs + b) * kUpPiece;
      const uint64_t r0 = p * per, m = std::min<uint64_t>(per, n - r0);
      e = cudaEventSynchronize(sent[b]);  // its previous piece has left
      if (e != cudaSuccess) break;
      if (rows)
        for (uint64_t i = 0; i < m; ++i) std::memcpy(buf + i * row, host + rows[r0 + i] * d, row);
      else
        std::memcpy(buf, host + r0 * d, m * row);
      float *to = landing ? (float *)(landing + (size_t)(t * kUpBufs + b) * kUpPiece) : dev + r0 * d;
      e = cudaMemcpyAsync(to, buf, m * row, cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess && landing) {
        k_pad_rows<<<(unsigned)std::min<uint64_t>((m * (dpad / 4) + 255) / 256, 1024), 256, 0, st>>>(
            to, m, d, dpad, reinterpret_cast<float4 *>(dev + r0 * dpad));
        e = cudaGetLastError();
      }
      if (e == cudaSuccess) e = cudaEventRecord(sent[b], st);
    }
    for (cudaEvent_t ev : sent)
      if (ev) {
        const cudaError_t w = cudaEventSynchronize(ev);
        if (e == cudaSuccess) e = w;
        cudaEventDestroy(ev);
      }
    err[t] = e;
  };
  std::thread helpers[kUpThreads];
  int started = 1;
  try {
    for (; started < kUpThreads; ++started) helpers[started] = std::thread(work, started);
  } catch (const std::exception &) {  // no more threads: their pieces are sent below
  }
  work(0);
  for (int t = started; t < kUpThreads; ++t) work(t);
  for (int t = 1; t < started; ++t) helpers[t].join();
  if (landing) cudaFreeAsync(landing, st);
  for (cudaError_t e : err)
    if (e != cudaSuccess) return cuda_fail(e, "row upload");
  return DG_OK;
}

}  // namespace dg

extern "C" {
const char *dg_last_error(void) { return dg::g_err.c_str(); }
int32_t dg_version(void) { return DGANN_VERSION; }
}
