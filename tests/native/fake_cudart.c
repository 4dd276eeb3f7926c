/* A CUDA runtime without a GPU, preloaded in front of the real one: memory is
 * host memory, kernels do nothing, and every call of interest is a line of
 * the file $FAKE_CUDART_LOG.  $FAKE_CAPACITY: bytes a device holds (what is
 * allocated and what its pools keep; past it allocations fail).
 * $FAKE_CLUSTERS: clusters a device holds at once. */
#define _GNU_SOURCE
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <cuda_runtime_api.h>

static int device = 0;
static FILE* out = NULL;

static void note(const char* fmt, ...) {
  if (!out) {
    const char* path = getenv("FAKE_CUDART_LOG");
    if (!path || !(out = fopen(path, "a"))) return;
  }
  va_list ap;
  va_start(ap, fmt);
  vfprintf(out, fmt, ap);
  va_end(ap);
  fputc('\n', out);
  fflush(out);
}

static long long number(const char* name, long long otherwise) {
  const char* v = getenv(name);
  return v ? atoll(v) : otherwise;
}

/* ---- memory */

struct pool {
  size_t keep, used, held; /* held: mapped, used among it */
  int dev;
};
struct block {
  void* p;
  size_t n;
  struct pool* pool;
  int dev;
};
static struct block blocks[4096];
static size_t taken[64]; /* mapped bytes of each device */

static int room(int dev, size_t n) { return taken[dev] + n <= (size_t)number("FAKE_CAPACITY", 1ll << 40); }

static cudaError_t keep_block(void** p, size_t n, struct pool* pool, int dev) {
  for (int i = 0; i < 4096; ++i)
    if (!blocks[i].p) {
      blocks[i].p = *p = calloc(n ? n : 1, 1);
      blocks[i].n = n;
      blocks[i].pool = pool;
      blocks[i].dev = dev;
      return cudaSuccess;
    }
  return cudaErrorMemoryAllocation;
}
static struct block* find(void* p) {
  for (int i = 0; i < 4096; ++i)
    if (blocks[i].p == p) return &blocks[i];
  return NULL;
}

cudaError_t cudaMalloc(void** p, size_t n) {
  const int ok = room(device, n);
  note("malloc %zu dev %d %s", n, device, ok ? "ok" : "full");
  if (!ok) return cudaErrorMemoryAllocation;
  taken[device] += n;
  return keep_block(p, n, NULL, device);
}
cudaError_t cudaFree(void* p) {
  struct block* b = p ? find(p) : NULL;
  if (!b) return p ? cudaErrorInvalidValue : cudaSuccess;
  taken[b->dev] -= b->n;
  free(b->p);
  memset(b, 0, sizeof *b);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* out_pool, const struct cudaMemPoolProps* props) {
  struct pool* q = calloc(1, sizeof *q);
  q->dev = props->location.id;
  note("pool dev %d", q->dev);
  *out_pool = (cudaMemPool_t)q;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t pool, enum cudaMemPoolAttr attr, void* v) {
  if (attr == cudaMemPoolAttrReleaseThreshold) ((struct pool*)pool)->keep = *(unsigned long long*)v;
  return cudaSuccess;
}
static void pool_shrink(struct pool* q, size_t keep) {
  const size_t want = q->used > keep ? q->used : keep;
  if (q->held > want) {
    taken[q->dev] -= q->held - want;
    q->held = want;
  }
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep) {
  note("trim %zu", keep);
  pool_shrink((struct pool*)pool, keep);
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
  (void)s;
  struct pool* q = (struct pool*)pool;
  if (q->used + n > q->held) {
    const size_t more = q->used + n - q->held;
    if (!room(q->dev, more)) {
      note("pool_malloc %zu dev %d full", n, q->dev);
      return cudaErrorMemoryAllocation;
    }
    taken[q->dev] += more;
    q->held += more;
  }
  q->used += n;
  note("pool_malloc %zu dev %d ok", n, q->dev);
  return keep_block(p, n, q, q->dev);
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  (void)s;
  struct block* b = p ? find(p) : NULL;
  if (!b || !b->pool) return cudaErrorInvalidValue;
  b->pool->used -= b->n;
  pool_shrink(b->pool, b->pool->keep);
  note("pool_free %zu held %zu", b->n, b->pool->held);
  free(b->p);
  memset(b, 0, sizeof *b);
  return cudaSuccess;
}

/* ---- copies */

cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) {
  (void)k;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) {
  (void)st;
  if (k == cudaMemcpyHostToDevice) note("upload %zu", n);
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind k) {
  (void)k;
  for (size_t i = 0; i < h; ++i) memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}

/* ---- devices, streams, events */

cudaError_t cudaSetDevice(int d) {
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr attr, int d) {
  (void)d;
  *v = attr == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
  *least = 0;
  *greatest = -5;
  return cudaSuccess;
}
static cudaError_t handle(void** h) {
  *h = malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  (void)f;
  return handle((void**)s);
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int p) {
  (void)f, (void)p;
  return handle((void**)s);
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  (void)s;
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned f) {
  (void)s, (void)e, (void)f;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) {
  (void)f;
  return handle((void**)e);
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  (void)e, (void)s;
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }

/* ---- kernels */

cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  (void)f;
  note("attribute %d %d dev %d", (int)a, v, device);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void* f, const cudaLaunchConfig_t* cfg) {
  (void)f, (void)cfg;
  *n = (int)number("FAKE_CLUSTERS", 10);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem, cudaStream_t s) {
  (void)f, (void)args, (void)s;
  note("launch %u x %u smem %zu dev %d", g.x, b.x, smem, device);
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void* f, void** args) {
  (void)f, (void)args;
  note("cluster_launch %u x %u dev %d", cfg->gridDim.x, cfg->blockDim.x, device);
  return cudaSuccess;
}
