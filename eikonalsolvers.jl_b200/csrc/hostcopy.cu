// Large results to pageable host memory, and arrays whose host side is row-major.
//
// What bounds such a copy is the host: one thread of the driver copies out of its own pinned
// buffer and takes the page faults of a fresh destination. Here several threads do, each with
// two pinned slots of its own, the next chunk crossing the bus while it copies the last one. A
// row-major destination (the layout of NumPy's default) is gathered by a kernel straight into
// the slot: the strided reads hit L2, where a transpose on the host reads a cache line per value.
// Measured with 16 host cores: the 134 MB of a 256^3 gradient 26 -> 5 ms; a 200^3 grid to row-major
// 41 ms (copy, then NumPy's transpose) -> 5 ms. Slots of 0.5, 1 and 2 MB differ by less than the runs
// do, and the smallest cost the first call of a context least (3.3, 4.8, 6.7 ms).
#include <atomic>
#include <cstring>
#include <memory>
#include <new>
#include <thread>

#include "runtime.hpp"

namespace eik {

constexpr size_t HOST_COPY_MIN = (size_t)8 << 20;

// out[q] = value at position o0 + q of column-major grids of n nodes, one after another, each gone through in
// row-major order (last axis fastest).
__global__ void rows_kernel(const double* grids, double* out, int nd, int n0, int n1, int n2, unsigned long long n,
                            unsigned long long o0, unsigned cnt) {
  for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < cnt; q += gridDim.x * blockDim.x) {
    const unsigned long long s = (o0 + q) / n, o = o0 + q - s * n;
    const double* t = grids + s * n;
    if (nd == 2) {
      out[q] = t[o / n1 + (unsigned long long)n0 * (o % n1)];
    } else {
      const unsigned long long k = o % n2, r = o / n2;
      out[q] = t[r / n1 + (unsigned long long)n0 * (r % n1 + (unsigned long long)n1 * k)];
    }
  }
}

// out[l] (column-major) = rows at the same node of a row-major grid.
__global__ void columns_kernel(const double* rows, double* out, int nd, int n0, int n1, int n2, unsigned long long n) {
  for (unsigned long long l = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; l < n;
       l += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long i = l % n0, r = l / n0;
    out[l] = nd == 2 ? rows[r + (unsigned long long)n1 * i]
                     : rows[r / n1 + (unsigned long long)n2 * (r % n1 + (unsigned long long)n1 * i)];
  }
}

void launch_columns(const GridDesc& g, const double* rows, double* out, cudaStream_t st) {
  columns_kernel<<<1184, 256, 0, st>>>(rows, out, g.nd, g.n[0], g.n[1], g.n[2], (unsigned long long)npts(g));
}

static bool ring_ready(eik_ctx* ctx) {
  HostRing& h = ctx->ring;
  if (!ctx->host_ring) return false;
  if (h.buf) return true;
  if (cudaMallocHost(&h.buf, HOST_SLOTS * HOST_SLOT) != cudaSuccess) {
    h.buf = nullptr;
    cudaGetLastError();
    return false;
  }
  for (auto& e : h.ev)
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      free_ring(h);
      cudaGetLastError();
      return false;
    }
  return true;
}

void free_ring(HostRing& h) {
  for (auto& e : h.ev) {
    if (e) cudaEventDestroy(e);
    e = nullptr;
  }
  if (h.buf) cudaFreeHost(h.buf);
  h.buf = nullptr;
}

// nsrc arrays of n doubles by chunks through the ring; rows: row-major at the destination. A chunk takes
// the values of as many arrays as a slot holds: one or more to each array, thousands of small grids were
// thousands of launches and events (beyond the solve, 16x16 x 3000 24 -> 3.9 ms, 24x24 x 2000 16 -> 3.0).
static int copy_chunks(eik_ctx* ctx, double* const* dst, const double* src, int64_t nsrc, unsigned long long n,
                       const GridDesc* rows, cudaStream_t st) {
  CUDA_OK(ctx, cudaStreamSynchronize(st));  // the threads would spin while the solve runs
  const unsigned long long per = HOST_SLOT / sizeof(double), total = n * (unsigned long long)nsrc,
                           nchunk = (total + per - 1) / per;
  std::atomic<unsigned long long> next{0};
  std::atomic<int> bad{(int)cudaSuccess};
  auto count = [&](unsigned long long c) { return (unsigned)std::min<unsigned long long>(per, total - c * per); };
  auto deliver = [&](unsigned long long c, const double* slot) {
    for (unsigned long long q = c * per, end = q + count(c); q < end;) {
      const unsigned long long s = q / n, o = q - s * n, len = std::min(n - o, end - q);
      std::memcpy(dst[s] + o, slot, sizeof(double) * (size_t)len);
      slot += len;
      q += len;
    }
  };
  auto work = [&](int w) noexcept {
    cudaError_t e = cudaSetDevice(ctx->device);
    bool have = false;
    unsigned long long last = 0;  // chunk in this worker's other slot, if it has one
    for (int k = 0; e == cudaSuccess && bad.load() == (int)cudaSuccess; k++) {
      const unsigned long long c = next.fetch_add(1);
      const int s = 2 * w + (k & 1);
      if (c < nchunk) {
        char* slot = ctx->ring.buf + (size_t)s * HOST_SLOT;
        if (rows)
          rows_kernel<<<64, 256, 0, st>>>(src, reinterpret_cast<double*>(slot), rows->nd, rows->n[0], rows->n[1],
                                          rows->n[2], n, c * per, count(c));
        else
          cudaMemcpyAsync(slot, src + c * per, sizeof(double) * count(c), cudaMemcpyDeviceToHost, st);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaEventRecord(ctx->ring.ev[s], st);
      }
      if (have && e == cudaSuccess) {
        e = cudaEventSynchronize(ctx->ring.ev[s ^ 1]);
        if (e == cudaSuccess) deliver(last, reinterpret_cast<double*>(ctx->ring.buf + (size_t)(s ^ 1) * HOST_SLOT));
      }
      have = c < nchunk;
      last = c;
      if (!have) break;
    }
    if (e != cudaSuccess) bad.store((int)e);
  };
  const int workers = (int)std::min<unsigned long long>(HOST_SLOTS / 2, nchunk);
  std::thread more[HOST_SLOTS / 2];
  try {
    for (int w = 1; w < workers; w++) more[w] = std::thread(work, w);
  } catch (...) {
    // no more threads to be had: the ones there are take all chunks
  }
  work(0);
  for (auto& t : more)
    if (t.joinable()) t.join();
  CUDA_OK(ctx, cudaStreamSynchronize(st));
  CUDA_OK(ctx, (cudaError_t)bad.load());
  return EIK_OK;
}

int copy_out(eik_ctx* ctx, double* dst, const double* src, unsigned long long n, cudaStream_t st) {
  const size_t bytes = sizeof(double) * (size_t)n;
  // small copies: below 8 MB the driver's own takes about 1 ms, less than making the ring costs the first
  // call; pinned memory takes the copy as it is
  bool plain = bytes < HOST_COPY_MIN || ctx->capturing;
  if (!plain) {
    cudaPointerAttributes at;
    plain = cudaPointerGetAttributes(&at, dst) != cudaSuccess || at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
  }
  if (!plain && ring_ready(ctx)) return copy_chunks(ctx, &dst, src, 1, n, nullptr, st);
  CUDA_OK(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
  return EIK_OK;
}

int copy_rows_out(eik_ctx* ctx, double* const* dst, const double* src, int64_t nsrc, const GridDesc& g, cudaStream_t st) {
  const unsigned long long n = (unsigned long long)npts(g);
  // the ring is made once a context has brought back as much as repays it: making it costs 3 to 6 ms, and the
  // way below 4 ms more than the ring's for 8 MB (first call of a context, 64x64 x 200, 6.6 MB: 8.6 -> 4.1 ms,
  // 300x220 x 8, 4.2 MB: 9.8 -> 6.4)
  ctx->rows_bytes += sizeof(double) * n * (unsigned long long)nsrc;
  if (ctx->rows_bytes >= HOST_COPY_MIN && ring_ready(ctx)) return copy_chunks(ctx, dst, src, nsrc, n, &g, st);
  // or no pinned memory to be had: 8 MB of grids (at least one) at a time to pageable memory, reordered there
  const int64_t group = std::max<int64_t>(1, std::min<int64_t>(nsrc, (int64_t)(HOST_COPY_MIN / sizeof(double) / n)));
  std::unique_ptr<double[]> tmp(new (std::nothrow) double[(size_t)n * (size_t)group]);
  if (!tmp) return fail(ctx, EIK_ERR_CUDA, "no host memory to reorder grids of %llu nodes", n);
  const size_t n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  for (int64_t s0 = 0; s0 < nsrc; s0 += group) {
    const int64_t m = std::min(group, nsrc - s0);
    CUDA_OK(ctx, cudaMemcpyAsync(tmp.get(), src + (size_t)s0 * n, sizeof(double) * (size_t)n * (size_t)m,
                                 cudaMemcpyDeviceToHost, st));
    CUDA_OK(ctx, cudaStreamSynchronize(st));
    for (int64_t s = 0; s < m; s++) {
      const double* t = tmp.get() + (size_t)s * n;
      double* out = dst[s0 + s];
      for (size_t i = 0; i < n0; i++)
        for (size_t j = 0; j < n1; j++)
          for (size_t k = 0; k < n2; k++) *out++ = t[i + n0 * (j + n1 * k)];
    }
  }
  return EIK_OK;
}

}  // namespace eik
