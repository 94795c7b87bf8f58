// Context, error handling and small shared services of the C ABI (include/qgpu.h).
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <list>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "qgpu_internal.cuh"

qg_status qg_cuda_fail(qg_context ctx, cudaError_t e, const char *what) {
  if (ctx) {
    char buf[512];
    std::snprintf(buf, sizeof(buf), "%s: %s (%s)", what, cudaGetErrorName(e), cudaGetErrorString(e));
    ctx->last_error = buf;
  }
  cudaGetLastError();  // clear a non-sticky error
  return e == cudaErrorMemoryAllocation ? QG_ERR_OOM : QG_ERR_CUDA;
}

qg_status qg_check_launch(qg_context ctx, const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return qg_cuda_fail(ctx, e, what);
  return QG_OK;
}

// Read and clear the device error word (synchronises the stream).
qg_status qg_check_device_error(qg_context ctx, const char *what) {
  unsigned int h = 0, zero = 0;
  cudaError_t e = cudaMemcpyAsync(&h, ctx->d_err, 4, cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(ctx->d_err, &zero, 4, cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return qg_cuda_fail(ctx, e, what);
  if (h & QG_DEVERR_TIMEOUT) {
    ctx->last_error = std::string(what) + ": bounded wait on a bulk copy gave up";
    return QG_ERR_TIMEOUT;
  }
  if (h & QG_DEVERR_PROBE) {
    ctx->last_error = std::string(what) + ": hash probe limit reached";
    return QG_ERR_TIMEOUT;
  }
  if (h & (QG_DEVERR_TABLE_FULL | QG_DEVERR_OVERFLOW)) {
    ctx->last_error = std::string(what) + ": device table or list full";
    return QG_ERR_TABLE_FULL;
  }
  return QG_OK;
}

// ------------------------------------------------------------------ device memory

#define QG_POOL_BYTES ((size_t)1 << 30)  // kept per context
#define QG_POOL_BLOCK ((size_t)1 << 29)  // the largest block kept

struct QgPool {
  std::mutex m;
  bool open = true;
  int device = 0;
  size_t held = 0;
  std::list<std::pair<void *, size_t>> idle;  // oldest first

  // give idle blocks back until at most `most` bytes are held (m locked)
  void shrink(size_t most) {
    while (!idle.empty() && held > most) {
      cudaFree(idle.front().first);
      held -= idle.front().second;
      idle.pop_front();
    }
  }
};

namespace {
std::mutex g_live_m;
// every block handed out: its pool and its size
std::unordered_map<void *, std::pair<std::shared_ptr<QgPool>, size_t>> g_live;
std::vector<std::weak_ptr<QgPool>> g_pools;

std::vector<std::shared_ptr<QgPool>> pools_of(int device) {
  std::lock_guard<std::mutex> l(g_live_m);
  std::vector<std::shared_ptr<QgPool>> out;
  for (auto &w : g_pools)
    if (auto p = w.lock())
      if (p->device == device) out.push_back(p);
  return out;
}

void drain_pools(int device) {
  for (auto &q : pools_of(device)) {
    std::lock_guard<std::mutex> l(q->m);
    q->shrink(0);
  }
}

// cudaMalloc, tried again without what the pools of the device hold
cudaError_t malloc_or_drain(qg_context ctx, void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  drain_pools(ctx->device);
  return cudaMalloc(p, bytes);
}
}  // namespace

cudaError_t qg_malloc_bytes(qg_context ctx, void **p, size_t bytes) {
  *p = nullptr;
  if (!bytes) return cudaSuccess;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (!ctx || !ctx->pool || cudaStreamIsCapturing(ctx->stream, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return cudaMalloc(p, bytes);
  }
  const size_t need = (bytes + 511) & ~(size_t)511;
  size_t got = need;
  {
    std::lock_guard<std::mutex> l(ctx->pool->m);
    auto best = ctx->pool->idle.end();
    for (auto it = ctx->pool->idle.begin(); it != ctx->pool->idle.end(); ++it)
      if (it->second >= need && it->second <= need + need / 8 + 4096 &&
          (best == ctx->pool->idle.end() || it->second < best->second))
        best = it;
    if (best != ctx->pool->idle.end()) {
      *p = best->first;
      got = best->second;
      ctx->pool->held -= got;
      ctx->pool->idle.erase(best);
    }
  }
  if (!*p) {
    const cudaError_t e = malloc_or_drain(ctx, p, need);
    if (e != cudaSuccess) {
      *p = nullptr;
      return e;
    }
  }
  std::lock_guard<std::mutex> l(g_live_m);
  g_live[*p] = {ctx->pool, got};
  return cudaSuccess;
}

cudaError_t qg_free(void *p) {
  if (!p) return cudaSuccess;
  std::shared_ptr<QgPool> pool;
  size_t size = 0;
  {
    std::lock_guard<std::mutex> l(g_live_m);
    auto it = g_live.find(p);
    if (it != g_live.end()) {
      pool = it->second.first;
      size = it->second.second;
      g_live.erase(it);
    }
  }
  if (!pool || size > QG_POOL_BLOCK) return cudaFree(p);
  std::lock_guard<std::mutex> l(pool->m);
  if (!pool->open) return cudaFree(p);
  pool->shrink(QG_POOL_BYTES - size);
  pool->idle.emplace_back(p, size);
  pool->held += size;
  return cudaSuccess;
}

cudaError_t qg_free_now(void *p) {
  if (!p) return cudaSuccess;
  {
    std::lock_guard<std::mutex> l(g_live_m);
    g_live.erase(p);
  }
  return cudaFree(p);
}

// of the current device, which is `device`
static cudaError_t memory_of(int device, size_t *free_bytes, size_t *total_bytes) {
  cudaError_t e = cudaMemGetInfo(free_bytes, total_bytes);
  if (e != cudaSuccess) return e;
  for (auto &q : pools_of(device)) {
    std::lock_guard<std::mutex> l(q->m);
    *free_bytes += q->held;
  }
  return cudaSuccess;
}

cudaError_t qg_mem_info(qg_context ctx, size_t *free_bytes, size_t *total_bytes) {
  return memory_of(ctx->device, free_bytes, total_bytes);
}

// the device for the time of a call
struct OnDevice {
  int before = -1;
  cudaError_t e;
  explicit OnDevice(int device) {
    e = cudaGetDevice(&before);
    if (e == cudaSuccess && before != device) e = cudaSetDevice(device);
  }
  ~OnDevice() {
    if (before >= 0) cudaSetDevice(before);
  }
};

extern "C" qg_status qg_device_memory(int device, int64_t *free_bytes, int64_t *total_bytes) {
  if (!free_bytes || !total_bytes) return QG_ERR_ARG;
  OnDevice on(device);
  size_t fr = 0, tot = 0;
  if (on.e != cudaSuccess || memory_of(device, &fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return QG_ERR_CUDA;
  }
  *free_bytes = (int64_t)fr;
  *total_bytes = (int64_t)tot;
  return QG_OK;
}

extern "C" qg_status qg_trim(int device) {
  OnDevice on(device);
  if (on.e != cudaSuccess) {
    cudaGetLastError();
    return QG_ERR_CUDA;
  }
  drain_pools(device);
  return QG_OK;
}

cudaError_t qg_upload(qg_context ctx, void *dst, const void *src, size_t bytes) {
  cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream);
  return e == cudaSuccess ? cudaStreamSynchronize(ctx->stream) : e;
}

qg_status qg_ensure_scratch(qg_context ctx, size_t bytes) {
  if (ctx->scratch_bytes >= bytes) return QG_OK;
  cudaStreamSynchronize(ctx->stream);
  cudaFree(ctx->d_scratch);
  ctx->d_scratch = nullptr;
  ctx->scratch_bytes = 0;
  size_t b = bytes < 65536 ? 65536 : bytes;
  QG_CUDA(ctx, malloc_or_drain(ctx, (void **)&ctx->d_scratch, b));
  ctx->scratch_bytes = b;
  return QG_OK;
}

qg_status qg_ensure_pinned(qg_context ctx, size_t bytes) {
  if (ctx->pinned_bytes >= bytes) return QG_OK;
  cudaFreeHost(ctx->h_pinned);
  ctx->h_pinned = nullptr;
  ctx->pinned_bytes = 0;
  QG_CUDA(ctx, cudaMallocHost(&ctx->h_pinned, bytes));
  ctx->pinned_bytes = bytes;
  return QG_OK;
}

extern "C" qg_status qg_init(int device, qg_context *out) {
  if (!out) return QG_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0 || device < 0 || device >= ndev) {
    cudaGetLastError();
    return QG_ERR_CUDA;
  }
  qg_context ctx = new qg_context_s();
  ctx->device = device;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
  ctx->own_stream = true;
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_err, 4);
  if (e == cudaSuccess) e = cudaMemset(ctx->d_err, 0, 4);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) {
    qg_cuda_fail(ctx, e, "qg_init");
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    cudaFree(ctx->d_err);
    delete ctx;
    return QG_ERR_CUDA;
  }
  ctx->pool = std::make_shared<QgPool>();
  ctx->pool->device = device;
  {
    std::lock_guard<std::mutex> l(g_live_m);
    g_pools.erase(std::remove_if(g_pools.begin(), g_pools.end(), [](const std::weak_ptr<QgPool> &w) { return w.expired(); }),
                  g_pools.end());
    g_pools.push_back(ctx->pool);
  }
  *out = ctx;
  return QG_OK;
}

extern "C" qg_status qg_finalize(qg_context ctx) {
  if (!ctx) return QG_OK;
  cudaStreamSynchronize(ctx->stream);
  {
    std::lock_guard<std::mutex> l(ctx->pool->m);
    ctx->pool->open = false;
    ctx->pool->shrink(0);
  }
  cudaFree(ctx->d_err);
  cudaFree(ctx->d_scratch);
  cudaFreeHost(ctx->h_pinned);
  qg_free_now(ctx->d_io);
  if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
  return QG_OK;
}

extern "C" qg_status qg_set_stream(qg_context ctx, void *stream) {
  if (!ctx) return QG_ERR_ARG;
  cudaStreamSynchronize(ctx->stream);
  if (stream) {
    if (ctx->own_stream) cudaStreamDestroy(ctx->stream);
    ctx->stream = (cudaStream_t)stream;
    ctx->own_stream = false;
  } else if (!ctx->own_stream) {
    QG_CUDA(ctx, cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
    ctx->own_stream = true;
  }
  return QG_OK;
}

extern "C" void *qg_get_stream(qg_context ctx) { return ctx ? (void *)ctx->stream : nullptr; }

extern "C" const char *qg_last_error(qg_context ctx) { return ctx ? ctx->last_error.c_str() : "no context"; }

extern "C" int64_t qg_launch_count(qg_context ctx) { return ctx ? ctx->launches : 0; }

extern "C" qg_status qg_synchronize(qg_context ctx) {
  if (!ctx) return QG_ERR_ARG;
  QG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return qg_check_device_error(ctx, "qg_synchronize");
}
