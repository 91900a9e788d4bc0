// gvr_batch.cu — many views in one persistent launch.
#include "gvr_march_device.cuh"

namespace gvr {
namespace {

// Many views in one persistent launch. A device counter hands out work items
// of `tiles_per_item` consecutive 16x16 tiles; items run through every tile
// of view 0, then view 1, ... so neighbouring CTAs share bricks in L2. Each
// tile first builds the bitmask of domains whose projected screen rectangle
// (rects[view * n_domains + d], inclusive pixel bounds, computed on the host)
// touches it, and its rays march only those. The counter only grows: no CTA
// ever waits for another.
template <int PW, int UNROLL, int MINB, int MODE>
__global__ void __launch_bounds__(kThreads, MINB)
batch_kernel(const DomainDev *__restrict__ g_domains, const ViewDev *__restrict__ views,
             const int4 *__restrict__ rects, const __grid_constant__ MarchParams mp, int n_views,
             int tiles_x,
             int tiles_y, int tiles_per_item, const float4 *__restrict__ g_lut,
             float4 *__restrict__ rgba, float *__restrict__ depth,
             unsigned long long *__restrict__ samples, unsigned int *__restrict__ queue)
{
  constexpr int PH = 32 / PW;
  constexpr int PX = kTile / PW;
  extern __shared__ float4 smem[];
  float4 *lut = smem;
  DomainDev *doms = reinterpret_cast<DomainDev *>(smem + mp.lut_size);
  __shared__ unsigned int s_item;
  __shared__ unsigned int s_mask[2];
  __shared__ float s_state[kStateSlots * kThreads];
  const int empties = empties_of(mp);
  for (int i = threadIdx.x; i < mp.lut_size; i += kThreads) lut[i] = g_lut[i];
  {
    const int words = mp.n_domains * (int)(sizeof(DomainDev) / 4);
    const uint32_t *src = reinterpret_cast<const uint32_t *>(g_domains);
    uint32_t *dst = reinterpret_cast<uint32_t *>(doms);
    for (int i = threadIdx.x; i < words; i += kThreads) dst[i] = src[i];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_per_view = tiles_x * tiles_y;
  const long long total_tiles = (long long)tiles_per_view * n_views;
  const long long n_items = (total_tiles + tiles_per_item - 1) / tiles_per_item;
  const int64_t pixels = (int64_t)mp.width * mp.height;
  int count = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(queue, 1u);
    __syncthreads();
    const long long item = s_item;
    if (item >= n_items) break;
    for (int sub = 0; sub < tiles_per_item; ++sub) {
      const long long tile = item * tiles_per_item + sub;
      if (tile >= total_tiles) break;
      const int v = (int)(tile / tiles_per_view);
      const int t = (int)(tile % tiles_per_view);
      const int tx = t % tiles_x, ty = t / tiles_x;
      const int x0 = tx * kTile, y0 = ty * kTile;
      if (warp < 2) {
        const int d = warp * 32 + lane;
        bool hit = false;
        if (d < mp.n_domains) {
          const int4 r = __ldg(rects + (int64_t)v * mp.n_domains + d);
          hit = !(r.z < x0 || r.x > x0 + kTile - 1 || r.w < y0 || r.y > y0 + kTile - 1);
        }
        const unsigned b = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) s_mask[warp] = b;
      }
      __syncthreads();
      const uint64_t mask = ((uint64_t)s_mask[1] << 32) | s_mask[0];
      const int px = x0 + (warp % PX) * PW + (lane % PW);
      const int py = y0 + (warp / PX) * PH + (lane / PW);
      if (px < mp.width && py < mp.height) {
        float4 out;
        float dep;
        count += render_ray<UNROLL, MODE>(doms, mask, views[v], mp, lut, px, py, out, dep, s_state,
                                          empties);
        const int64_t pix = (int64_t)v * pixels + (int64_t)py * mp.width + px;
        rgba[pix] = out;
        depth[pix] = dep;
      }
      __syncthreads();
    }
  }
  if (samples) {
    unsigned long long c = (unsigned long long)count;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0 && c) atomicAdd(samples, c);
  }
}

}  // namespace

namespace {

using BatchFn = void (*)(const DomainDev *, const ViewDev *, const int4 *, const MarchParams, int,
                         int, int, int, const float4 *, float4 *, float *, unsigned long long *,
                         unsigned int *);

BatchFn select_batch(Tuning t, int mode)
{
  t.packet_w = packet_width(t, mode, true, 0);
  if (mode == kMarchHex) return t.packet_w == 4 ? batch_kernel<4, 1, 2, kMarchHex> : batch_kernel<8, 1, 2, kMarchHex>;
  if (mode == kMarchRect)
    return t.packet_w == 4 ? batch_kernel<4, 2, 3, kMarchRect>
                           : (t.packet_w == 16 ? batch_kernel<16, 2, 3, kMarchRect> : batch_kernel<8, 2, 3, kMarchRect>);
  if (mode == kMarchCells)
    return t.packet_w == 4 ? batch_kernel<4, 2, 4, kMarchCells>
                           : (t.packet_w == 16 ? batch_kernel<16, 2, 4, kMarchCells> : batch_kernel<8, 2, 4, kMarchCells>);
  const int u = t.unroll == 1 ? 1 : 2;
  const int m = t.min_blocks == 3 ? 3 : 4;
  switch (t.packet_w) {
    case 4:
      return u == 2 ? (m == 4 ? batch_kernel<4, 2, 4, kMarchUniform> : batch_kernel<4, 2, 3, kMarchUniform>)
                    : (m == 4 ? batch_kernel<4, 1, 4, kMarchUniform> : batch_kernel<4, 1, 3, kMarchUniform>);
    case 16:
      return u == 2 ? (m == 4 ? batch_kernel<16, 2, 4, kMarchUniform> : batch_kernel<16, 2, 3, kMarchUniform>)
                    : (m == 4 ? batch_kernel<16, 1, 4, kMarchUniform> : batch_kernel<16, 1, 3, kMarchUniform>);
    default:
      return u == 2 ? (m == 4 ? batch_kernel<8, 2, 4, kMarchUniform> : batch_kernel<8, 2, 3, kMarchUniform>)
                    : (m == 4 ? batch_kernel<8, 1, 4, kMarchUniform> : batch_kernel<8, 1, 3, kMarchUniform>);
  }
}

}  // namespace

// Resident CTAs of the batch kernel for this launch shape (SMs x CTAs per SM
// from the occupancy calculator), capped by the number of work items. Also
// sets the kernel's dynamic shared-memory limit; call it outside any capture.
cudaError_t batch_grid(const MarchParams &mp, int n_views, const Tuning &tuning, int mode,
                       int *grid)
{
  const size_t smem = sizeof(float4) * mp.lut_size + sizeof(DomainDev) * mp.n_domains;
  BatchFn fn = select_batch(tuning, mode);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(sizeof(float4) * kMaxLut + sizeof(DomainDev) * kMaxDomains));
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per_sm = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kThreads, smem);
  if (e != cudaSuccess) return e;
  const int tiles_x = (mp.width + kTile - 1) / kTile, tiles_y = (mp.height + kTile - 1) / kTile;
  const int tpi = tuning.tiles_per_item > 0 ? tuning.tiles_per_item : 1;
  const long long items = ((long long)tiles_x * tiles_y * n_views + tpi - 1) / tpi;
  *grid = (int)std::max(1ll, std::min<long long>(items, (long long)sms * std::max(per_sm, 1)));
  return cudaSuccess;
}

// Clear the work counter and launch the persistent batch kernel (both stream
// operations, so the pair can be captured into a CUDA graph).
cudaError_t launch_batch(const DomainDev *d_domains, const ViewDev *d_views, const int4 *d_rects,
                         const MarchParams &mp, int n_views, const float4 *d_lut, float4 *d_rgba,
                         float *d_depth, unsigned long long *d_samples, unsigned int *d_queue,
                         const Tuning &tuning, int mode, int grid, cudaStream_t stream)
{
  const size_t smem = sizeof(float4) * mp.lut_size + sizeof(DomainDev) * mp.n_domains;
  BatchFn fn = select_batch(tuning, mode);
  const int tiles_x = (mp.width + kTile - 1) / kTile, tiles_y = (mp.height + kTile - 1) / kTile;
  const int tpi = tuning.tiles_per_item > 0 ? tuning.tiles_per_item : 1;
  cudaError_t e = cudaMemsetAsync(d_queue, 0, sizeof(unsigned int), stream);
  if (e != cudaSuccess) return e;
  fn<<<(unsigned)grid, kThreads, smem, stream>>>(d_domains, d_views, d_rects, mp, n_views, tiles_x,
                                                 tiles_y, tpi, d_lut, d_rgba, d_depth, d_samples,
                                                 d_queue);
  return cudaGetLastError();
}

}  // namespace gvr
