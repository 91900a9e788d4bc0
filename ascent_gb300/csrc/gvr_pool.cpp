// gvr_pool.cpp — the library's device memory: a pool for scenes and their
// builds, a pool for the scratch of calls.
#include <mutex>
#include <vector>

#include "gvr_internal.h"

namespace gvr {
namespace {

constexpr int kMaxPoolDevices = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pools[kMaxPoolDevices] = {};         // call scratch
cudaMemPool_t g_scene_pools[kMaxPoolDevices] = {};   // scenes' memory
cudaStream_t g_scene_streams[kMaxPoolDevices] = {};  // its allocations and frees
void *g_anchors[kMaxPoolDevices] = {};               // see wait_for_device
// scenes' memory whose wait was refused; never destroyed, as a scene may be at exit
std::vector<void *> *const g_kept = new std::vector<void *>[kMaxPoolDevices];

// Free memory that a device's scene pool holds on to between scenes, and so
// keeps from the process's other allocators. A scene made for each step of a
// device field: 0.3 ms for 500^3 nodes (0.7 GiB of bricks), 1.1 for 850^3
// (3.2 GiB); of larger ones the pool maps and unmaps what exceeds the limit in
// each step: 3.1 ms for 950^3 (4.5 GiB), 9.6 for 1100^3 (7.0 GiB).
constexpr uint64_t kScenePoolKeep = (uint64_t)4 << 30;

constexpr size_t kAnchorBytes = 256;

// A pool of this library on `device` that keeps up to `keep` free bytes.
cudaError_t make_pool(int device, uint64_t keep, cudaMemPool_t *out)
{
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  cudaMemPool_t created = nullptr;
  cudaError_t e = cudaMemPoolCreate(&created, &props);
  if (e != cudaSuccess) return e;
  if ((e = cudaMemPoolSetAttribute(created, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
    cudaMemPoolDestroy(created);
    return e;
  }
  *out = created;
  return cudaSuccess;
}

// Waits for all work on the current device as cudaFree does, by one. Not by
// cudaDeviceSynchronize, which a capture on any stream of the device refuses,
// whatever its mode and its thread, and which ends that capture: a scene
// destroyed by one thread would break the graph that another one records, this
// library's own in gvr_render_volume_batch among them. cudaFree is refused by
// captures in global mode and by a capture of the calling thread, unless that
// is relaxed, and by no other. 2.0 us where nothing runs, next to a word that
// stays allocated (g_anchors); without that each call maps and unmaps the
// block that the word comes from, 58 us.
cudaError_t wait_for_device()
{
  void *word = nullptr;
  cudaError_t e = cudaMalloc(&word, kAnchorBytes);
  if (e == cudaSuccess) return cudaFree(word);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  return cudaDeviceSynchronize();
}

}  // namespace

cudaError_t device_free(void *const *ptrs, size_t n)
{
  std::vector<void *> list;
  for (size_t i = 0; i < n; ++i)
    if (ptrs[i]) list.push_back(ptrs[i]);
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device < 0 || device >= kMaxPoolDevices) {
    for (void *p : list)
      if ((e = cudaFree(p)) != cudaSuccess) return e;
    return cudaSuccess;
  }
  cudaStream_t stream;
  {
    // what was kept goes too: it is taken before the wait, which so covers it
    std::lock_guard<std::mutex> lock(g_pool_mu);
    list.insert(list.end(), g_kept[device].begin(), g_kept[device].end());
    g_kept[device].clear();
    stream = g_scene_streams[device];
  }
  if (list.empty()) return cudaSuccess;
  e = wait_for_device();
  if (e == cudaSuccess) {
    for (void *p : list) cudaFreeAsync(p, stream);
    e = cudaStreamSynchronize(stream);   // until which the memory counts as used where the pool is trimmed
  } else {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    g_kept[device].insert(g_kept[device].end(), list.begin(), list.end());
  }
  if (e != cudaSuccess) cudaGetLastError();   // not the next launch's
  return e;
}

// Scenes' memory. An in-situ host makes a scene per publish, some 30 buffers
// that cudaMalloc maps and cudaFree unmaps, each call a synchronisation: 3.9
// of the 6.7 ms of a step with 1M new hexahedra, 1.2 of 3.4 ms of one with
// four structured host domains. From a pool they cost a microsecond each; the
// pool gives back what it holds beyond kScenePoolKeep when a scene's memory is
// freed, all of it to gvr_scratch_trim, and when an allocation of either pool
// does not fit. Allocations and frees are made on one stream of the pool's own on
// which nothing runs, and an allocation is waited for, so that the memory may
// be used on any stream and from any thread.
cudaError_t device_alloc(void **ptr, size_t bytes)
{
  *ptr = nullptr;
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device < 0 || device >= kMaxPoolDevices) return cudaMalloc(ptr, bytes);
  cudaMemPool_t pool;
  cudaStream_t stream;
  bool kept;
  {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_scene_streams[device] &&
        (e = cudaStreamCreateWithFlags(&g_scene_streams[device], cudaStreamNonBlocking)) != cudaSuccess)
      return e;
    if (!g_scene_pools[device] && (e = make_pool(device, kScenePoolKeep, &g_scene_pools[device])) != cudaSuccess)
      return e;
    if (!g_anchors[device] && cudaMalloc(&g_anchors[device], kAnchorBytes) != cudaSuccess) {
      g_anchors[device] = nullptr;   // waits are slower until there is one
      cudaGetLastError();
    }
    pool = g_scene_pools[device];
    stream = g_scene_streams[device];
    kept = !g_kept[device].empty();
  }
  if (kept) device_free(nullptr, 0);
  e = cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
  if (e == cudaErrorMemoryAllocation) {
    // what the pools hold free may be what is missing
    cudaGetLastError();
    gvr_scratch_trim(device, 0, nullptr);
    e = cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
  }
  if (e != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) {
    // refused by a capture: nothing has used the memory
    cudaFreeAsync(*ptr, stream);
    *ptr = nullptr;
  }
  return e;
}

// The device's default memory pool gives its free memory back to the
// system at every synchronisation (release threshold 0), so a call that
// allocates tens of MB of scratch and synchronises would map fresh pages
// every time. This library's own pool keeps what it has allocated (up to
// its high-water mark, held until the process exits) and leaves the
// default pool, which other libraries in the process may use, as it is. An
// allocation that does not fit is tried again without what both pools hold
// free, as much as the scenes' pool keeps; not under capture, where the trim's
// waits are refused.
cudaError_t scratch_alloc(void **ptr, size_t bytes, cudaStream_t stream)
{
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device < 0 || device >= kMaxPoolDevices) return cudaMallocAsync(ptr, bytes, stream);
  cudaMemPool_t pool;
  {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    if (!g_pools[device] && (e = make_pool(device, UINT64_MAX, &g_pools[device])) != cudaSuccess) return e;
    pool = g_pools[device];
  }
  e = cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusActive;
  if (e != cudaErrorMemoryAllocation || cudaStreamIsCapturing(stream, &capture) != cudaSuccess ||
      capture != cudaStreamCaptureStatusNone)
    return e;
  cudaGetLastError();
  gvr_scratch_trim(device, 0, nullptr);
  return cudaMallocFromPoolAsync(ptr, bytes, pool, stream);
}

cudaError_t scratch_alloc(void **ptr, size_t bytes, size_t least, bool *all, cudaStream_t stream)
{
  cudaError_t e = scratch_alloc(ptr, bytes, stream);
  *all = e == cudaSuccess;
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  return scratch_alloc(ptr, least, stream);
}

}  // namespace gvr

int gvr_scratch_trim(int device, uint64_t keep_bytes, uint64_t *reserved_out)
{
  using namespace gvr;
  if (device < 0) return set_error(GVR_ERR_INVALID_ARGUMENT, "negative device");
  cudaMemPool_t pool = nullptr, scenes = nullptr;
  bool kept = false;
  if (device < kMaxPoolDevices) {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    pool = g_pools[device];
    scenes = g_scene_pools[device];
    kept = !g_kept[device].empty();
  }
  int current = -1;
  if (kept && cudaGetDevice(&current) == cudaSuccess && current == device) device_free(nullptr, 0);
  uint64_t reserved = 0;
  // what scenes that are gone have left in their pool; what scenes use stays
  if (scenes) {
    const cudaError_t e = cudaMemPoolTrimTo(scenes, (size_t)keep_bytes);
    if (e != cudaSuccess) return cuda_error(e, "cudaMemPoolTrimTo");
  }
  if (pool) {
    // blocks still in use are kept whatever keep_bytes says; memory freed
    // on a stream is returned once that free has completed
    cudaError_t e = cudaMemPoolTrimTo(pool, (size_t)keep_bytes);
    if (e != cudaSuccess) return cuda_error(e, "cudaMemPoolTrimTo");
    e = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved);
    if (e != cudaSuccess) return cuda_error(e, "cudaMemPoolGetAttribute");
  }
  if (reserved_out) *reserved_out = reserved;
  return GVR_OK;
}
