// The library's device memory (csrc/gvr_pool.cpp) against a CUDA runtime made
// of counters: what happens to memory when calls are refused, without a GPU.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

#include "../ascent_gb300/csrc/gvr_internal.h"

namespace {
struct Pool {
  uint64_t keep = 0;
  size_t used = 0, free = 0;   // bytes handed out, and held free
};
struct Block {
  Pool *pool;   // nullptr: cudaMalloc's
  size_t bytes;
};
size_t capacity = 1 << 20;     // of the device
bool capturing = false;        // a capture that refuses unsafe calls
bool device_sync_seen = false;
int trims = 0;
cudaError_t last = cudaSuccess;
std::set<Pool *> pools;
std::map<void *, Block> blocks;

size_t reserved()
{
  size_t n = 0;
  for (Pool *p : pools) n += p->used + p->free;
  for (auto &b : blocks)
    if (!b.second.pool) n += b.second.bytes;
  return n;
}

cudaError_t fail(cudaError_t e)
{
  last = e;
  return e;
}

int checks_failed = 0;
#define CHECK(x)                                                     \
  do {                                                               \
    if (!(x)) {                                                      \
      std::printf("line %d: %s\n", __LINE__, #x);                    \
      ++checks_failed;                                               \
    }                                                                \
  } while (0)
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaDeviceSynchronize() { device_sync_seen = true; return capturing ? fail(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return capturing ? fail(cudaErrorStreamCaptureUnsupported) : cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s)
{
  *s = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n)
{
  if (capturing) return fail(cudaErrorStreamCaptureUnsupported);
  if (reserved() + n > capacity) return fail(cudaErrorMemoryAllocation);
  blocks[*p = std::malloc(1)] = {nullptr, n};
  return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
  if (!p) return cudaSuccess;
  if (capturing) return fail(cudaErrorStreamCaptureUnsupported);
  CHECK(blocks.count(p) && !blocks[p].pool);
  blocks.erase(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *out, const cudaMemPoolProps *)
{
  Pool *p = new Pool;
  pools.insert(p);
  *out = (cudaMemPool_t)p;
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void *v)
{
  if (a == cudaMemPoolAttrReleaseThreshold) ((Pool *)p)->keep = *(uint64_t *)v;
  return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr, void *v)
{
  *(uint64_t *)v = ((Pool *)p)->used + ((Pool *)p)->free;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t n)
{
  ++trims;
  Pool *q = (Pool *)p;
  const size_t keep = n > q->used ? n - q->used : 0;
  if (q->free > keep) q->free = keep;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t)
{
  Pool *q = (Pool *)pool;
  if (q->free >= n) q->free -= n;
  else if (reserved() + n > capacity) return fail(cudaErrorMemoryAllocation);
  q->used += n;
  blocks[*p = std::malloc(1)] = {q, n};
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **, size_t, cudaStream_t) { return fail(cudaErrorInvalidValue); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t)
{
  CHECK(blocks.count(p) && blocks[p].pool);
  Pool *q = blocks[p].pool;
  q->used -= blocks[p].bytes;
  q->free += blocks[p].bytes;
  blocks.erase(p);
  return cudaSuccess;
}
}

namespace gvr {
int set_error(int code, const std::string &) { return code; }
int cuda_error(cudaError_t, const char *) { return GVR_ERR_CUDA; }
}  // namespace gvr

using namespace gvr;

// Memory whose wait is refused is kept, and freed after the next wait that is
// not, whether a free's, an allocation's or a trim's; no error is left behind.
static void refused_wait(int then)
{
  void *a, *b, *c;
  CHECK(device_alloc(&a, 1000) == cudaSuccess && device_alloc(&b, 2000) == cudaSuccess);
  CHECK(device_alloc(&c, 3000) == cudaSuccess);
  capturing = true;
  void *ab[3] = {a, nullptr, b};
  CHECK(device_free(ab, 3) == cudaErrorStreamCaptureUnsupported);
  CHECK(blocks.count(a) && blocks.count(b));
  CHECK(last == cudaSuccess);
  capturing = false;
  if (then == 0) {
    CHECK(device_free(c) == cudaSuccess);
  } else if (then == 1) {
    void *d;
    CHECK(device_alloc(&d, 500) == cudaSuccess);
    CHECK(!blocks.count(a) && !blocks.count(b) && blocks.count(c));
    CHECK(device_free(d) == cudaSuccess && device_free(c) == cudaSuccess);
  } else {
    CHECK(gvr_scratch_trim(0, 0, nullptr) == GVR_OK);
    CHECK(!blocks.count(a) && !blocks.count(b) && blocks.count(c));
    CHECK(device_free(c) == cudaSuccess);
  }
  for (auto &q : blocks) CHECK(!q.second.pool);
  CHECK(!device_sync_seen);   // it would end another thread's capture
}

// An allocation that a capture refuses leaves nothing behind.
static void refused_allocation()
{
  void *a = &a;
  capturing = true;
  CHECK(device_alloc(&a, 1000) != cudaSuccess);
  capturing = false;
  CHECK(a == nullptr);
  for (auto &q : blocks) CHECK(!q.second.pool);
  last = cudaSuccess;
}

// What either pool holds free is given back where the other's allocation does
// not fit, not under capture; and the device's memory is what it was.
static void out_of_memory()
{
  void *a, *s;
  trims = 0;
  CHECK(device_alloc(&a, 800000) == cudaSuccess && device_free(a) == cudaSuccess);
  CHECK(scratch_alloc(&s, 900000, nullptr) == cudaSuccess);   // the scenes' pool made room
  CHECK(trims > 0 && last == cudaSuccess);
  CHECK(scratch_alloc(&a, 900000, nullptr) == cudaErrorMemoryAllocation && blocks.count(s));
  last = cudaSuccess;
  CHECK(cudaFreeAsync(s, nullptr) == cudaSuccess);
  trims = 0;
  CHECK(device_alloc(&a, 700000) == cudaSuccess);             // the scratch pool did
  CHECK(trims > 0 && last == cudaSuccess);
  CHECK(device_alloc(&s, 700000) == cudaErrorMemoryAllocation && s == nullptr);
  last = cudaSuccess;
  CHECK(device_free(a) == cudaSuccess);
  capturing = true;
  trims = 0;
  CHECK(scratch_alloc(&s, 900000, nullptr) == cudaErrorMemoryAllocation && trims == 0);
  capturing = false;
  last = cudaSuccess;
  CHECK(gvr_scratch_trim(0, 0, nullptr) == GVR_OK);
  size_t held = 0;
  for (Pool *p : pools) held += p->used + p->free;
  CHECK(held == 0);
}

// The larger amount where it fits, the smaller where only that does.
static void either_amount()
{
  void *a, *s;
  bool all = false;
  CHECK(scratch_alloc(&s, 600000, 100000, &all, nullptr) == cudaSuccess && all);
  CHECK(cudaFreeAsync(s, nullptr) == cudaSuccess);
  CHECK(device_alloc(&a, 700000) == cudaSuccess);
  CHECK(scratch_alloc(&s, 600000, 100000, &all, nullptr) == cudaSuccess && !all && last == cudaSuccess);
  CHECK(blocks[s].bytes == 100000);
  void *t;
  CHECK(scratch_alloc(&t, 600000, 500000, &all, nullptr) == cudaErrorMemoryAllocation && !all);
  last = cudaSuccess;
  CHECK(cudaFreeAsync(s, nullptr) == cudaSuccess && device_free(a) == cudaSuccess);
}

int main()
{
  for (int then = 0; then < 3; ++then) refused_wait(then);
  refused_allocation();
  out_of_memory();
  either_amount();
  return checks_failed != 0;
}
