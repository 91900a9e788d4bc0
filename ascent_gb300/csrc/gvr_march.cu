// gvr_march.cu — the march kernel of one view, the choice of its shape, and the
// longest-first tile order.
#include "gvr_march_device.cuh"

namespace gvr {
namespace {

// PW x (32 / PW) pixel packet per warp, 16 x 16 pixels per CTA.
template <int PW, int UNROLL, int MINB, int MODE = kMarchUniform>
__global__ void __launch_bounds__(kThreads, MINB)
march_kernel(const DomainDev *__restrict__ g_domains, const __grid_constant__ ViewDev view,
             const __grid_constant__ MarchParams mp, const float4 *__restrict__ g_lut,
             float4 *__restrict__ rgba, float *__restrict__ depth,
             unsigned long long *__restrict__ samples, const int *__restrict__ order)
{
  constexpr int PH = 32 / PW;
  constexpr int PX = kTile / PW;  // packets per tile row
  const int tiles_x = (mp.width + kTile - 1) / kTile;
  const int tile = order ? __ldg(order + blockIdx.x) : (int)blockIdx.x;
  const int tile_x = tile % tiles_x, tile_y = tile / tiles_x;
  extern __shared__ float4 smem[];
  __shared__ float s_state[kStateSlots * kThreads];
  float4 *lut = smem;
  DomainDev *doms = reinterpret_cast<DomainDev *>(smem + mp.lut_size);
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
  const int px = tile_x * kTile + (warp % PX) * PW + (lane % PW);
  const int py = tile_y * kTile + (warp / PX) * PH + (lane / PW);
  const bool valid = px < mp.width && py < mp.height;
  int count = 0;
  if (valid) {
    const uint64_t all = mp.n_domains >= 64 ? ~0ull : ((1ull << mp.n_domains) - 1ull);
    float4 out;
    float dep;
    count = render_ray<UNROLL, MODE>(doms, all, view, mp, lut, px, py, out, dep, s_state, empties);
    const int64_t pix = (int64_t)py * mp.width + px;
    rgba[pix] = out;
    depth[pix] = dep;
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

using MarchFn = void (*)(const DomainDev *, const ViewDev, const MarchParams, const float4 *,
                         float4 *, float *, unsigned long long *, const int *);

template <int PW, int UNROLL, int MINB>
MarchFn pick() { return march_kernel<PW, UNROLL, MINB>; }

MarchFn select(Tuning t, int mode, int64_t tiles, bool long_steps)
{
  t.packet_w = packet_width(t, mode, false, tiles);
  // Until a shape is set: small frames, whose few warps wait for their loads
  // more than for each other, take four samples per iteration at 3 CTAs per SM
  // (10 to 14% faster at 80 to 1200 tiles, 46.3 -> 41.8 us for the 64^3 field at
  // 512^2); large ones two at 4 (1388 against 1406 us at 4096 tiles).
  if (!t.unroll) {
    t.unroll = mode == kMarchUniform && tiles < kSmallFrame ? 4 : 2;
    t.min_blocks = mode == kMarchUniform && tiles < kSmallFrame ? 3 : 4;
  }
  // the hex path keeps a cell's eight coefficient records in registers: 2 or
  // 3 CTAs per SM (3 spills some 400 bytes and measured 1.5% faster)
  if (mode == kMarchHex) {
    const bool m3 = t.min_blocks >= 4;
    if (t.packet_w == 4) return m3 ? march_kernel<4, 1, 3, kMarchHex> : march_kernel<4, 1, 2, kMarchHex>;
    return m3 ? march_kernel<8, 1, 3, kMarchHex> : march_kernel<8, 1, 2, kMarchHex>;
  }
  // rectilinear domains keep three cells' records in registers besides the
  // ray, which 4 CTAs per SM spill: 502 against 464 us at 3 for the 242 x 200 x
  // 174 nodes at 0.65 cells a step; with two cells a step and more the way from
  // cell to cell waits for its loads, and 4 are faster (241^3 nodes at 1024^2:
  // 618 and 622 us at one cell a step, 425 and 438 at two, 306 and 322 at four,
  // 153 and 170 at 20). The tuning has no say.
  if (mode == kMarchRect) {
    if (long_steps)
      return t.packet_w == 4 ? march_kernel<4, 2, 4, kMarchRect>
                             : (t.packet_w == 16 ? march_kernel<16, 2, 4, kMarchRect> : march_kernel<8, 2, 4, kMarchRect>);
    return t.packet_w == 4 ? march_kernel<4, 2, 3, kMarchRect>
                           : (t.packet_w == 16 ? march_kernel<16, 2, 3, kMarchRect> : march_kernel<8, 2, 3, kMarchRect>);
  }
  // cell-centred ones take 4 (210 against 221 us on two domains of 160 x 144 x
  // 121 cells at 1280 x 720)
  if (mode == kMarchCells)
    return t.packet_w == 4 ? march_kernel<4, 2, 4, kMarchCells>
                           : (t.packet_w == 16 ? march_kernel<16, 2, 4, kMarchCells> : march_kernel<8, 2, 4, kMarchCells>);
  // three and four samples per iteration have kernels only at 3 CTAs per SM
  // (one: four); with 64 registers they spill in the loop (1930 against 1437 us
  // on the 513^3 field) and take two
  if (t.unroll >= 3 && t.min_blocks < 4 && t.packet_w != 16) return t.packet_w == 4 ? pick<4, 4, 3>() : pick<8, 4, 3>();
  const int u = t.unroll == 1 ? 1 : 2;
  const int m = t.min_blocks == 3 ? 3 : 4;
  switch (t.packet_w) {
    case 4:
      return u == 2 ? (m == 4 ? pick<4, 2, 4>() : pick<4, 2, 3>()) : (m == 4 ? pick<4, 1, 4>() : pick<4, 1, 3>());
    case 16:
      return u == 2 ? (m == 4 ? pick<16, 2, 4>() : pick<16, 2, 3>()) : (m == 4 ? pick<16, 1, 4>() : pick<16, 1, 3>());
    default:
      return u == 2 ? (m == 4 ? pick<8, 2, 4>() : pick<8, 2, 3>()) : (m == 4 ? pick<8, 1, 4>() : pick<8, 1, 3>());
  }
}

}  // namespace

cudaError_t launch_march(const DomainDev *d_domains, const ViewDev &view,
                         const MarchParams &mp, const float4 *d_lut, float4 *d_rgba,
                         float *d_depth, unsigned long long *d_samples, const Tuning &tuning,
                         int mode, bool long_steps, const int *d_order, cudaStream_t stream)
{
  const size_t smem = sizeof(float4) * mp.lut_size + sizeof(DomainDev) * mp.n_domains;
  const int64_t tiles = (int64_t)((mp.width + kTile - 1) / kTile) * ((mp.height + kTile - 1) / kTile);
  MarchFn fn = select(tuning, mode, tiles, long_steps);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(sizeof(float4) * kMaxLut + sizeof(DomainDev) * kMaxDomains));
  if (e != cudaSuccess) return e;
  fn<<<(unsigned)tiles, kThreads, smem, stream>>>(d_domains, view, mp, d_lut, d_rgba, d_depth,
                                                  d_samples, d_order);
  count_launch();
  return cudaGetLastError();
}


// Longest-first launch order of the march tiles for one view: the cost of a
// tile is the summed length, through every domain box, of five of its rays
// (its centre and corner pixels); tiles are counting-sorted into 1024 cost
// bins, longest first, so that the last tiles the GPU takes are the short
// ones (longest-processing-time-first list scheduling). Two launches: the
// costs with one thread per tile (keys[t] = the cost's bits, *top = their
// maximum), then one CTA bins, scans and scatters them and clears *top for
// the next view. The order of tiles within a bin is whatever the
// shared-memory atomics give, and no order changes a pixel.
__global__ void __launch_bounds__(256)
tile_cost_kernel(const DomainDev *__restrict__ g_domains, const __grid_constant__ ViewDev view,
                 const __grid_constant__ MarchParams mp, unsigned *__restrict__ keys,
                 unsigned *__restrict__ top)
{
  const int tiles_x = (mp.width + kTile - 1) / kTile;
  const int n = tiles_x * ((mp.height + kTile - 1) / kTile);
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned bits = 0u;
  if (t < n) {
    const int x0 = (t % tiles_x) * kTile, y0 = (t / tiles_x) * kTile;
    const int x1 = min(x0 + kTile - 1, mp.width - 1), y1 = min(y0 + kTile - 1, mp.height - 1);
    const int rx[5] = {(x0 + x1) >> 1, x0, x1, x0, x1};
    const int ry[5] = {(y0 + y1) >> 1, y0, y0, y1, y1};
    float cost = 0.f;
    for (int k = 0; k < 5; ++k) {
      const Ray r = pixel_ray(view, mp, rx[k], ry[k]);
      for (int d = 0; d < mp.n_domains; ++d) {
        float t0, t1;
        if (slab(g_domains[d], r, t0, t1)) cost += t1 - t0;
      }
    }
    cost = cost > 0.f && cost < FLT_MAX ? cost : 0.f;   // NaN and inf cost nothing
    bits = __float_as_uint(cost);
    keys[t] = bits;
  }
  bits = __reduce_max_sync(0xffffffffu, bits);
  if ((threadIdx.x & 31) == 0 && bits) atomicMax(top, bits);
}

__global__ void __launch_bounds__(1024)
tile_order_sort_kernel(const __grid_constant__ MarchParams mp, const unsigned *__restrict__ keys,
                       unsigned *__restrict__ top, int *__restrict__ order)
{
  __shared__ int s_hist[1024];
  __shared__ int s_warp[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tiles_x = (mp.width + kTile - 1) / kTile;
  const int n = tiles_x * ((mp.height + kTile - 1) / kTile);
  s_hist[tid] = 0;
  const float high = __uint_as_float(*top);
  const float scale = high > 0.f ? 1023.f / high : 0.f;
  __syncthreads();
  for (int t = tid; t < n; t += 1024)
    atomicAdd(&s_hist[1023 - min(1023, (int)(__uint_as_float(keys[t]) * scale))], 1);
  __syncthreads();
  // exclusive scan of the 1024 bins, one per thread
  const int v = s_hist[tid];
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = s_warp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    s_warp[lane] = w;
  }
  __syncthreads();
  s_hist[tid] = x - v + (warp ? s_warp[warp - 1] : 0);
  __syncthreads();
  for (int t = tid; t < n; t += 1024) {
    const int bin = 1023 - min(1023, (int)(__uint_as_float(keys[t]) * scale));
    order[atomicAdd(&s_hist[bin], 1)] = t;
  }
  if (tid == 0) *top = 0u;
}

cudaError_t launch_tile_cost_order(const DomainDev *d_domains, const ViewDev &view, const MarchParams &mp,
                                   int *d_order, unsigned *d_keys, unsigned *d_top, cudaStream_t stream)
{
  const int64_t tiles = (int64_t)((mp.width + kTile - 1) / kTile) * ((mp.height + kTile - 1) / kTile);
  if (tiles > kCostOrderTiles) return cudaErrorInvalidValue;
  tile_cost_kernel<<<(unsigned)((tiles + 255) / 256), 256, 0, stream>>>(d_domains, view, mp, d_keys, d_top);
  tile_order_sort_kernel<<<1, 1024, 0, stream>>>(mp, d_keys, d_top, d_order);
  count_launch(2);
  return cudaGetLastError();
}

}  // namespace gvr
