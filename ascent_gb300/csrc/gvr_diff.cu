// gvr_diff.cu — differentiable volume render: forward with transmittance
// checkpoints and its hand-written adjoint.
//
// The render is the single-uniform-domain march of gvr_march_device.cuh (same ray
// model, stepping rule and front-to-back blend) with the two changes a
// gradient needs: the transfer function is looked up with linear
// interpolation (so colour and opacity are differentiable in the scalar),
// and no partial is culled. Inputs are the caller's device buffers: the node
// field in its plain layout (x fastest) and the LUT (n RGBA floats), both
// differentiable.
//
// Forward (training): one thread per ray; it stores the transmittance at the
// start of every kDiffK-sample segment and caches every sample's scalar v_k
// in a workspace ([sample][ray], so that a warp writes contiguous rays).
// Backward: per ray, segments from last to first. A segment's transmittances
// T_k are rebuilt forward from its checkpoint through the cached scalars and
// the LUT — no field loads, and the blend is never inverted — into an
// array of the thread's; then its samples are walked back to front with the
// suffix composite (R', A') of the samples behind them:
//   dL/dc_k = T_k a_k g_rgb,
//   dL/da_k = T_k (g_rgb . (c_k - R'_k) + g_A (1 - A'_k)),
//   R'_{k-1} = a_k c_k + (1 - a_k) R'_k,  A'_{k-1} = a_k + (1 - a_k) A'_k.
// LUT gradients are summed in registers while consecutive samples of a ray
// stay in one LUT interval, then added with two float4 atomics to the CTA's
// private copy in global memory; a last kernel sums the copies. Field
// gradients are
// summed per ray while consecutive samples stay in one cell, then combined
// with the neighbouring lane's sums when both leave the same cell at the
// same step, and added with two float4 atomics per cell into a corner-quad
// buffer that is folded into the node gradient at the end.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "gvr_internal.h"

namespace gvr {
namespace {

constexpr int kDiffK = 64;          // samples per transmittance checkpoint
constexpr int kSub = 8;             // backward: scalars loaded together
constexpr int kMaxDiffViews = 64;
constexpr int kDiffLut = 4096;
constexpr int kSharedTLut = 512;    // backward: transmittances in shared memory up to this LUT

struct DiffViews {
  ViewDev v[kMaxDiffViews];
};

struct DiffGrid {
  int dims[3];
  float origin[3];
  float inv_spacing[3];
  float lo[3];
  float hi[3];
};

struct DiffParams {
  int width;
  int height;
  int n_views;
  int lut_size;
  int n_seg;       // checkpoint segments per ray
  double max_samples;  // of a ray, along the grid's diagonal
  int lut_copies;  // backward: LUT-gradient copies in global memory (CTA c uses c % copies)
  int64_t n_rays;  // views x height x width
  int packets;     // rays numbered by 8 x 4-pixel packets (see ray_number)
  int64_t v_offset;  // start of the per-sample scalar cache in the workspace
  float sample_dist;
  float scalar_min;
  float inv_range;
};

// Corner quads of a field (see gather_quads): a copy per axis along which they
// lie one after the other, and the copy that each view reads.
struct DiffQuads {
  const float4 *copy[3];
  int stride[3][3];   // of the copy along axis f: from a cell to the next in x, y, z
  unsigned char axis[kMaxDiffViews];
};

__device__ __forceinline__ float lerp2(float a, float b, float w) { return fmaf(w, b - a, a); }

// Ray of pixel (px, py) of view v: origin, unit direction, [t0, t1) inside the
// grid; false when the ray misses it.
__device__ __forceinline__ bool diff_ray(const ViewDev &view, const DiffGrid &g, const DiffParams &p,
                                         int px, int py, float o[3], float d[3], float &t0,
                                         float &t1)
{
  const float fx = view.dx_scale * ((float)px - 0.5f * (float)p.width - view.xoff);
  const float fy = view.dy_scale * ((float)py - 0.5f * (float)p.height - view.yoff);
  float dn = 0.f;
  for (int a = 0; a < 3; ++a) {
    d[a] = view.look[a] + view.ru[a] * fx + view.rv[a] * fy;
    dn = fmaf(d[a], d[a], dn);
  }
  const float inv = rsqrtf(dn);
  t0 = 0.f;
  t1 = FLT_MAX;
  for (int a = 0; a < 3; ++a) {
    o[a] = view.origin[a];
    d[a] *= inv;
    if (d[a] != 0.f) {
      const float r = 1.f / d[a];
      float ta = (g.lo[a] - o[a]) * r, tb = (g.hi[a] - o[a]) * r;
      if (ta > tb) { const float t = ta; ta = tb; tb = t; }
      t0 = fmaxf(t0, ta);
      t1 = fminf(t1, tb);
    } else if (o[a] < g.lo[a] || o[a] > g.hi[a]) {
      return false;
    }
  }
  return t1 > t0;
}

// Number of a ray in the workspace: where the image is whole 8 x 4-pixel
// packets, a warp's 32 rays one after the other, so that the scalars it stores
// and loads for a sample are one 128-byte line and not four pieces of rows;
// otherwise the pixels row by row.
__device__ __forceinline__ int64_t ray_number(const DiffParams &p, int v, int px, int py)
{
  if (!p.packets) return ((int64_t)v * p.height + py) * p.width + px;
  const int packet = (py >> 2) * (p.width >> 3) + (px >> 3);
  return (int64_t)v * p.width * p.height + 32 * (int64_t)packet + ((py & 3) * 8 + (px & 7));
}

// Cell (linear index of its corner 000, of type I: int where the field has
// fewer than 2^31 nodes) and trilinear weights of sample t.
template <typename I>
__device__ __forceinline__ I diff_cell(const DiffGrid &g, const float A[3], const float B[3],
                                       float t, float w[3])
{
  int c[3];
  for (int a = 0; a < 3; ++a) {
    const float gg = fmaf(t, B[a], A[a]);
    c[a] = __vimin_s32_relu((int)gg, g.dims[a] - 2);   // max(0, min)
    w[a] = gg - (float)c[a];
  }
  return ((I)c[2] * g.dims[1] + c[1]) * g.dims[0] + c[0];
}

// The 8 corners of the cell at base: (x, y, z) bits of the index are
// (1, 2, 4).
template <typename I>
__device__ __forceinline__ void diff_corners(const float *__restrict__ f, const DiffGrid &g,
                                             I base, float c[8])
{
  const I sy = g.dims[0], sz = (I)g.dims[0] * g.dims[1];
  const float *p = f + base;
  c[0] = __ldg(p);
  c[1] = __ldg(p + 1);
  c[2] = __ldg(p + sy);
  c[3] = __ldg(p + sy + 1);
  p += sz;
  c[4] = __ldg(p);
  c[5] = __ldg(p + 1);
  c[6] = __ldg(p + sy);
  c[7] = __ldg(p + sy + 1);
}

// out[cell] = the corners (x, y), (x+1, y), (x, y+1), (x+1, y+1) of the layer
// z for every node as corner 000 (clamped at the far faces, where no cell
// starts), laid out along axis F: neighbours along F are neighbours in out.
// A block reads a tile of 33 x 33 nodes (F = 2: of two y rows) with lanes
// along x and writes the 32 x 32 quads with lanes along F. HBM-bound at the
// quads' 16 bytes a node: 9 us for 128^3 (32 us when lanes along y also read
// the field that way).
template <int F>
__global__ void __launch_bounds__(256)
gather_quads(const float *__restrict__ f, const DiffGrid g, float4 *__restrict__ out)
{
  constexpr int U = F == 2 ? 2 : 1, T = F == 2 ? 1 : 2;   // the tile's other axis, the blocks'
  __shared__ float tile[F == 2 ? 2 : 1][33][33];
  const int64_t stride[3] = {1, g.dims[0], (int64_t)g.dims[0] * g.dims[1]};
  const int x0 = blockIdx.x * 32;
  for (int t = blockIdx.z; t < g.dims[T]; t += gridDim.z)
    for (int u0 = blockIdx.y * 32; u0 < g.dims[U]; u0 += gridDim.y * 32) {
#pragma unroll
      for (int l = 0; l < (F == 2 ? 2 : 1); ++l) {
        const float *plane = f + min(t + l, g.dims[T] - 1) * stride[T];
        for (int i = threadIdx.y * 32 + threadIdx.x; i < 33 * 33; i += 256) {
          const int r = i / 33, c = i % 33;
          tile[l][r][c] = __ldg(plane + min(u0 + r, g.dims[U] - 1) * stride[U] + min(x0 + c, g.dims[0] - 1));
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = threadIdx.y; i < 32; i += 8) {
        const int r = F == 0 ? i : threadIdx.x, c = F == 0 ? threadIdx.x : i;
        const int x = x0 + c, u = u0 + r;
        if (x < g.dims[0] && u < g.dims[U]) {
          const float4 q = F == 2 ? make_float4(tile[0][r][c], tile[0][r][c + 1], tile[F == 2][r][c], tile[F == 2][r][c + 1])
                                  : make_float4(tile[0][r][c], tile[0][r][c + 1], tile[0][r + 1][c], tile[0][r + 1][c + 1]);
          const int in = F == 0 ? x : u, over = F == 0 ? u : x;   // along F, and the next axis
          out[((int64_t)t * g.dims[F == 0 ? 1 : 0] + over) * g.dims[F] + in] = q;
        }
      }
      __syncthreads();
    }
}

// The 8 corners of sample t's cell, from the quads, and its weights.
__device__ __forceinline__ void quad_corners(const float4 *__restrict__ quads, const int st[3],
                                             const DiffGrid &g, const float A[3], const float B[3],
                                             float t, float c[8], float w[3])
{
  int at = 0;
  for (int a = 0; a < 3; ++a) {
    const float gg = fmaf(t, B[a], A[a]);
    const int i = __vimin_s32_relu((int)gg, g.dims[a] - 2);   // as in diff_cell
    w[a] = gg - (float)i;
    at += i * st[a];
  }
  const float4 lo = __ldg(quads + at), hi = __ldg(quads + at + st[2]);
  c[0] = lo.x; c[1] = lo.y; c[2] = lo.z; c[3] = lo.w;
  c[4] = hi.x; c[5] = hi.y; c[6] = hi.z; c[7] = hi.w;
}

__device__ __forceinline__ float diff_interp(const float c[8], const float w[3])
{
  const float c00 = lerp2(c[0], c[1], w[0]);
  const float c10 = lerp2(c[2], c[3], w[0]);
  const float c01 = lerp2(c[4], c[5], w[0]);
  const float c11 = lerp2(c[6], c[7], w[0]);
  return lerp2(lerp2(c00, c10, w[1]), lerp2(c01, c11, w[1]), w[2]);
}

// Opacity of the linear LUT lookup at scalar v (the w of diff_lut), from the
// LUT's opacity column.
__device__ __forceinline__ float lut_alpha(const float *lut_a, const DiffParams &p, float v)
{
  const float x = __saturatef((v - p.scalar_min) * p.inv_range) * (float)(p.lut_size - 1);
  const int i0 = min((int)x, p.lut_size - 2);
  return lerp2(lut_a[i0], lut_a[i0 + 1], x - (float)i0);
}

// Linear LUT lookup at scalar v; also returns the entry index i0, the weight
// and the difference of entries i0 + 1 and i0.
__device__ __forceinline__ float4 diff_lut(const float4 *lut, const DiffParams &p, float v,
                                           float &s_raw, int &i0, float &wl, float4 &step)
{
  s_raw = (v - p.scalar_min) * p.inv_range;
  const float s = __saturatef(s_raw);
  const float x = s * (float)(p.lut_size - 1);
  i0 = min((int)x, p.lut_size - 2);
  wl = x - (float)i0;
  const float4 a = lut[i0], b = lut[i0 + 1];
  step = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, b.w - a.w);
  return make_float4(fmaf(wl, step.x, a.x), fmaf(wl, step.y, a.y), fmaf(wl, step.z, a.z), fmaf(wl, step.w, a.w));
}

// Blend a sample of scalar v behind acc.
__device__ __forceinline__ void diff_blend(const float4 *lut, const DiffParams &p, float v, float4 &acc)
{
  float s_raw, wl;
  int i0;
  float4 step;
  const float4 c = diff_lut(lut, p, v, s_raw, i0, wl, step);
  const float wa = (1.f - acc.w) * c.w;
  acc.x = fmaf(wa, c.x, acc.x);
  acc.y = fmaf(wa, c.y, acc.y);
  acc.z = fmaf(wa, c.z, acc.z);
  acc.w += wa;
}

// One thread per ray, a warp per 8 x 4-pixel packet. Reading the corners from
// the field is bound by the L1 tags (97% busy): 8 loads a sample, each over as
// many lines as the packet's cells have (y, z) rows, 3 for a packet that lies
// along x and 12 for one across it. With QUADS they are two 16-byte loads from
// the copy that lies along the packet's longer edge, so that the rows are few
// from every side, and four samples' loads are in flight before the first is
// blended (kept cells, which save lines in the other form, would chain the
// loads: 1.2 to 1.6 times slower here; quads in 2 x 2 x 2 blocks, the same from
// every side, cost more index arithmetic: 1.3 times slower). 128^3 field, 16
// views at 256^2, the copies included: 1117 -> 640 us; 4 views 233 -> 182; a
// 64^3 field, 4 views at 96 x 80: 37 -> 27.
template <typename I, bool QUADS>
__global__ void __launch_bounds__(256)
diff_forward(const float *__restrict__ field, const __grid_constant__ DiffQuads quads, const DiffGrid g,
             const DiffViews views, const DiffParams p, const float4 *__restrict__ g_lut,
             float4 *__restrict__ rgba, float *__restrict__ ws)
{
  extern __shared__ float4 lut[];
  for (int i = threadIdx.x; i < p.lut_size; i += blockDim.x) lut[i] = g_lut[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int px = blockIdx.x * 16 + (warp & 1) * 8 + (lane & 7);
  const int py = blockIdx.y * 16 + (warp >> 1) * 4 + (lane >> 3);
  const int v = blockIdx.z;
  if (px >= p.width || py >= p.height) return;
  float o[3], d[3], t0, t1;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (diff_ray(views.v[v], g, p, px, py, o, d, t0, t1)) {
    float A[3], B[3];
    for (int a = 0; a < 3; ++a) {
      A[a] = (o[a] - g.origin[a]) * g.inv_spacing[a];
      B[a] = d[a] * g.inv_spacing[a];
    }
    const int64_t ray = ray_number(p, v, px, py);
    float *check = ws ? ws + ray * p.n_seg : nullptr;     // transmittance at the next segment's start
    float *scalar = ws ? ws + p.v_offset + ray : nullptr; // the next sample's scalar
    if constexpr (QUADS) {
      constexpr int kGroup = 4;   // divides kDiffK
      const int axis = quads.axis[v];
      const float4 *copy = quads.copy[axis];
      const int st[3] = {quads.stride[axis][0], quads.stride[axis][1], quads.stride[axis][2]};
      int k = 0;
      for (; fmaf((float)(k + kGroup - 1), p.sample_dist, t0) < t1; k += kGroup) {
        if (ws && (k % kDiffK) == 0) *check++ = 1.f - acc.w;
        float cc[kGroup][8], w[kGroup][3];
#pragma unroll
        for (int j = 0; j < kGroup; ++j)
          quad_corners(copy, st, g, A, B, fmaf((float)(k + j), p.sample_dist, t0), cc[j], w[j]);
        float val[kGroup];
#pragma unroll
        for (int j = 0; j < kGroup; ++j) {
          val[j] = diff_interp(cc[j], w[j]);
          if (ws) {
            *scalar = val[j];
            scalar += p.n_rays;
          }
        }
#pragma unroll
        for (int j = 0; j < kGroup; ++j) diff_blend(lut, p, val[j], acc);
      }
      for (;; ++k) {   // the ray's last samples
        const float t = fmaf((float)k, p.sample_dist, t0);
        if (!(t < t1)) break;
        if (ws && (k % kDiffK) == 0) *check++ = 1.f - acc.w;
        float cc[8], w[3];
        quad_corners(copy, st, g, A, B, t, cc, w);
        const float val = diff_interp(cc, w);
        if (ws) {
          *scalar = val;
          scalar += p.n_rays;
        }
        diff_blend(lut, p, val, acc);
      }
    } else {
      // corners of the last cell loaded, reused while samples stay in it
      I last = -1;
      float cc[8];
      for (int k = 0;; ++k) {
        const float t = fmaf((float)k, p.sample_dist, t0);
        if (!(t < t1)) break;
        if (ws && (k % kDiffK) == 0) *check++ = 1.f - acc.w;
        float w[3];
        const I base = diff_cell<I>(g, A, B, t, w);
        if (base != last) {
          diff_corners<I>(field, g, base, cc);
          last = base;
        }
        const float val = diff_interp(cc, w);
        if (ws) {
          *scalar = val;
          scalar += p.n_rays;
        }
        diff_blend(lut, p, val, acc);
      }
    }
  }
  rgba[((int64_t)v * p.height + py) * p.width + px] = acc;
}

// Add g8 (the gradients of one cell's eight corners) to the field gradient.
// Warp-aggregated in pairs: lanes 2i and 2i + 1 (neighbouring pixels in x)
// that flush the same cell at the same step add their sums first, the even
// lane the corners of the lower z layer and the odd lane those of the upper, so
// that four values change hands and each lane makes one atomic. Measured
// against pooling whole peer sets (__match_any_sync, then shuffles) and against
// 2x2 / 4x2 pixel groups, pairs were fastest: wider groups cost more shuffles
// than they save atomics. The sums go to the corner-quad buffer gq (one float4
// per cell base: corners (x, y), (x+1, y), (x, y+1), (x+1, y+1) of one z
// layer), so a flush is 16-byte vector atomics, each in one sector; fold_quads
// adds the quads into the node gradient afterwards. Called by all lanes.
template <typename I>
__device__ __forceinline__ void flush_cell(float4 *__restrict__ gq, const DiffGrid &g,
                                           I base, const float g8[8], bool active)
{
  const int lane = threadIdx.x & 31;
  const I mine = active ? base : (I)(-1 - lane);
  const bool pair = __shfl_xor_sync(0xffffffffu, mine, 1) == mine;
  const bool odd = lane & 1;
  float s[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    // what this lane keeps, and what it hands over
    const float keep = odd ? g8[4 + m] : g8[m];
    s[m] = keep + __shfl_xor_sync(0xffffffffu, odd ? g8[m] : g8[4 + m], 1);
  }
  if (!active) return;
  float4 *lower = gq + base, *upper = lower + (I)g.dims[0] * g.dims[1];
  if (pair) {
    atomicAdd(odd ? upper : lower, make_float4(s[0], s[1], s[2], s[3]));
  } else {
    atomicAdd(lower, make_float4(g8[0], g8[1], g8[2], g8[3]));
    atomicAdd(upper, make_float4(g8[4], g8[5], g8[6], g8[7]));
  }
}

// grad[i] += quads whose corners include node i: its own quad's (x, y)
// entry, the (x+1, y) entry of the quad to its left, and so on.
__global__ void fold_quads(const float4 *__restrict__ gq, const DiffGrid g,
                           float *__restrict__ grad)
{
  const int64_t nx = g.dims[0], ny = g.dims[1], n = nx * ny * g.dims[2];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = i % nx, y = (i / nx) % ny;
    float acc = gq[i].x;
    if (x > 0) acc += gq[i - 1].y;
    if (y > 0) acc += gq[i - nx].z;
    if (x > 0 && y > 0) acc += gq[i - nx - 1].w;
    if (acc != 0.f) grad[i] += acc;
  }
}

// Add the register sums of LUT interval li (entries li and li + 1) to this
// CTA's LUT-gradient copy as two float4 atomics, and clear them.
__device__ __forceinline__ void flush_lut4(float *copy, int li, float (&lg)[8])
{
  if (li < 0) return;
  float4 *q = reinterpret_cast<float4 *>(copy + 4 * li);
  atomicAdd(q, make_float4(lg[0], lg[1], lg[2], lg[3]));
  atomicAdd(q + 1, make_float4(lg[4], lg[5], lg[6], lg[7]));
#pragma unroll
  for (int m = 0; m < 8; ++m) lg[m] = 0.f;
}

// A segment's transmittances lie in shared memory where three CTAs per SM still
// fit with them (SHARED_T: 64 KB and 20 bytes per LUT entry each), else in local
// memory, which the L1 does not hold (200 KB per SM): 1930 -> 1856 us for a
// 128^3 field, 16 views at 256^2. What is left is issue (67%) and reductions on
// their way to L2 (L1-to-crossbar requests 58%); four CTAs per SM at 64
// registers ran the same.
template <typename I, bool SHARED_T>
__global__ void __launch_bounds__(256)
diff_backward(const float *__restrict__ field, const DiffGrid g, const DiffViews views,
              const DiffParams p, const float4 *__restrict__ g_lut,
              const float4 *__restrict__ grad_rgba, const float *__restrict__ ws,
              float4 *__restrict__ gq, float *__restrict__ glut_cta)
{
  extern __shared__ float4 smem[];
  float4 *lut = smem;
  // LUT gradient: this CTA's private copy in global memory (L2-resident),
  // two float4 atomics per flushed interval. Measured against 16 padded
  // private copies in shared memory per CTA (8 scalar shared atomics per
  // flush, bank conflicts, 64 KB of shared memory taken from L1): 4.72 vs
  // 5.86 ms for the whole training step.
  float *lut_a = reinterpret_cast<float *>(smem + p.lut_size);  // opacity column
  const int64_t cta = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  float *slg = glut_cta + (cta % p.lut_copies) * 4 * p.lut_size;
  for (int i = threadIdx.x; i < p.lut_size; i += blockDim.x) {
    lut[i] = g_lut[i];
    lut_a[i] = g_lut[i].w;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int px = blockIdx.x * 16 + (warp & 1) * 8 + (lane & 7);
  const int py = blockIdx.y * 16 + (warp >> 1) * 4 + (lane >> 3);
  const int v = blockIdx.z;
  const bool inside = px < p.width && py < p.height;
  float o[3], d[3], t0 = 0.f, t1 = 0.f;
  const bool hit = inside && diff_ray(views.v[v], g, p, min(px, p.width - 1), min(py, p.height - 1),
                                      o, d, t0, t1);
  int n = 0;
  float4 gr = make_float4(0.f, 0.f, 0.f, 0.f);
  float A[3] = {0.f, 0.f, 0.f}, B[3] = {0.f, 0.f, 0.f};
  int64_t ray = 0;
  if (hit) {
    ray = ray_number(p, v, px, py);
    gr = grad_rgba[((int64_t)v * p.height + py) * p.width + px];
    for (int a = 0; a < 3; ++a) {
      A[a] = (o[a] - g.origin[a]) * g.inv_spacing[a];
      B[a] = d[a] * g.inv_spacing[a];
    }
    while (fmaf((float)n, p.sample_dist, t0) < t1) ++n;
  }
  // the warp walks segments in lock step so that lanes can pool their
  // field gradients; lanes with fewer segments idle
  int nseg = hit ? (n + kDiffK - 1) / kDiffK : 0;
  int max_seg = nseg;
  for (int off = 16; off > 0; off >>= 1) max_seg = max(max_seg, __shfl_xor_sync(0xffffffffu, max_seg, off));
  float Rr = 0.f, Rg = 0.f, Rb = 0.f, Ra = 0.f;  // suffix composite behind the sample
  I cur = -1;
  float g8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int li = -1;  // LUT interval of the register sums lg
  float lg[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const float *scalars = ws + p.v_offset + ray;   // sample k's at k * n_rays
  float local_t[SHARED_T ? 1 : kDiffK];
  float *T = SHARED_T ? lut_a + p.lut_size + threadIdx.x : local_t;   // sample j's at j * kStep
  constexpr int kStep = SHARED_T ? 256 : 1;
  for (int sidx = max_seg - 1; sidx >= 0; --sidx) {
    const int k0 = sidx * kDiffK, k1 = sidx < nseg ? min(k0 + kDiffK, n) : k0;
    // transmittance of every sample of the segment, forward from its
    // checkpoint through the cached scalars (no field loads); the scalars
    // are loaded kSub at a time so that their latencies overlap
    if (k1 > k0) {
      float Tr = ws[ray * p.n_seg + sidx];
      const float *at = scalars + (int64_t)k0 * p.n_rays;
      for (int kq = k0; kq < k1; kq += kSub) {
        float vv[kSub];
#pragma unroll
        for (int j = 0; j < kSub; ++j) {
          vv[j] = kq + j < k1 ? *at : 0.f;
          at += p.n_rays;
        }
#pragma unroll
        for (int j = 0; j < kSub; ++j) {
          T[kStep * (kq - k0 + j)] = Tr;
          if (kq + j < k1) Tr *= 1.f - lut_alpha(lut_a, p, vv[j]);
        }
      }
    }
    // walk it back to front, from the warp's last sample in the segment
    // (uniform trip count across the warp); the scalar and transmittance of
    // the next sample are loaded one step ahead
    {
      const int jn = (int)__reduce_max_sync(0xffffffffu, (unsigned)(k1 - k0));
      const float *at = scalars + (int64_t)(k0 + jn - 1) * p.n_rays;
      float v_next = k1 > k0 + jn - 1 ? *at : 0.f;
      float t_next = T[kStep * max(jn - 1, 0)];
      for (int j = jn - 1; j >= 0; --j) {
        const int k = k0 + j;
        const bool on = k < k1;
        const float v_cur = v_next, Tk = t_next;
        if (j > 0) {
          at -= p.n_rays;
          v_next = k - 1 < k1 ? *at : 0.f;
          t_next = T[kStep * (j - 1)];
        }
        I base = -1;
        float w[3] = {0.f, 0.f, 0.f}, dv = 0.f;
        if (on) {
          const float t = fmaf((float)k, p.sample_dist, t0);
          base = diff_cell<I>(g, A, B, t, w);
          float s_raw, wl;
          int i0;
          float4 st;   // d(rgba)/dx, x = s (n - 1)
          const float4 c = diff_lut(lut, p, v_cur, s_raw, i0, wl, st);
          const float ta = Tk * c.w;
          const float dcr = ta * gr.x, dcg = ta * gr.y, dcb = ta * gr.z;
          const float da = Tk * (gr.x * (c.x - Rr) + gr.y * (c.y - Rg) + gr.z * (c.z - Rb) +
                                 gr.w * (1.f - Ra));
          Rr = fmaf(c.w, c.x, (1.f - c.w) * Rr);
          Rg = fmaf(c.w, c.y, (1.f - c.w) * Rg);
          Rb = fmaf(c.w, c.z, (1.f - c.w) * Rb);
          Ra = c.w + (1.f - c.w) * Ra;
          // transfer-function entries i0 and i0 + 1: summed in registers
          // while consecutive samples stay in one LUT interval
          if (i0 != li) {
            flush_lut4(slg, li, lg);
            li = i0;
          }
          const float w0 = 1.f - wl;
          lg[0] = fmaf(w0, dcr, lg[0]);
          lg[1] = fmaf(w0, dcg, lg[1]);
          lg[2] = fmaf(w0, dcb, lg[2]);
          lg[3] = fmaf(w0, da, lg[3]);
          lg[4] = fmaf(wl, dcr, lg[4]);
          lg[5] = fmaf(wl, dcg, lg[5]);
          lg[6] = fmaf(wl, dcb, lg[6]);
          lg[7] = fmaf(wl, da, lg[7]);
          if (s_raw > 0.f && s_raw < 1.f)
            dv = (dcr * st.x + dcg * st.y + dcb * st.z + da * st.w) * (float)(p.lut_size - 1) * p.inv_range;
        }
        // pool the field gradient per cell; flush when a lane changes cell
        const bool change = on && base != cur && cur >= 0;
        flush_cell<I>(gq, g, cur, g8, change);
        if (change) {
#pragma unroll
          for (int m = 0; m < 8; ++m) g8[m] = 0.f;
        }
        if (on) {
          cur = base;
          const float x0 = 1.f - w[0], y0 = 1.f - w[1];
          const float lo = dv * (1.f - w[2]), hi = dv * w[2];
          const float xy[4] = {x0 * y0, w[0] * y0, x0 * w[1], w[0] * w[1]};
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            g8[m] = fmaf(lo, xy[m], g8[m]);
            g8[4 + m] = fmaf(hi, xy[m], g8[4 + m]);
          }
        }
      }
    }
  }
  flush_cell<I>(gq, g, cur, g8, cur >= 0);
  flush_lut4(slg, li, lg);
}

// glut[i] += the CTAs' private LUT-gradient copies, 32 CTAs per thread
__global__ void sum_lut_copies(const float *__restrict__ glut_cta, int64_t n_cta, int n,
                               float *__restrict__ glut)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t c0 = (int64_t)blockIdx.y * 32, c1 = min(c0 + 32, n_cta);
  float acc = 0.f;
  for (int64_t c = c0; c < c1; ++c) acc += glut_cta[c * n + i];
  if (acc != 0.f) atomicAdd(glut + i, acc);
}

int diff_setup(const float *field, const int dims[3], const double origin[3],
               const double spacing[3], const gvr_camera *cameras, int n_views,
               const gvr_render_params *params, DiffGrid &g, DiffViews &views, DiffParams &p)
{
  if (!field || !dims || !origin || !spacing || !cameras || !params)
    return set_error(GVR_ERR_INVALID_ARGUMENT, "NULL argument");
  if (n_views < 1 || n_views > kMaxDiffViews)
    return set_error(GVR_ERR_INVALID_ARGUMENT, "the differentiable render takes 1..64 views");
  if (params->width < 1 || params->height < 1 || params->lut_size < 2 || params->lut_size > kDiffLut)
    return set_error(GVR_ERR_INVALID_ARGUMENT, "bad image size or lut_size (2..4096)");
  if (!(params->sample_dist > 0)) return set_error(GVR_ERR_INVALID_ARGUMENT, "sample_dist must be > 0");
  double diag = 0;
  for (int a = 0; a < 3; ++a) {
    if (dims[a] < 2 || !(spacing[a] > 0))
      return set_error(GVR_ERR_INVALID_ARGUMENT, "dims >= 2 and spacing > 0 required");
    const float o = (float)origin[a], sp = (float)spacing[a];
    g.dims[a] = dims[a];
    g.origin[a] = o;
    g.inv_spacing[a] = 1.f / sp;
    g.lo[a] = o;
    g.hi[a] = (float)((double)o + (double)(dims[a] - 1) * sp);
    diag += (double)(dims[a] - 1) * sp * (double)(dims[a] - 1) * sp;
  }
  for (int v = 0; v < n_views; ++v) make_view(cameras[v], params->width, params->height, &views.v[v]);
  p.width = params->width;
  p.height = params->height;
  p.n_views = n_views;
  p.lut_size = params->lut_size;
  p.sample_dist = params->sample_dist;
  p.scalar_min = params->scalar_min;
  p.inv_range = params->scalar_max > params->scalar_min
                    ? 1.f / (params->scalar_max - params->scalar_min) : 0.f;
  const double max_samples = std::sqrt(diag) / params->sample_dist + 2.0;
  p.n_seg = (int)((max_samples + kDiffK - 1) / kDiffK);
  p.max_samples = max_samples;
  p.lut_copies = 1;
  p.n_rays = (int64_t)n_views * params->width * params->height;
  p.packets = params->width % 8 == 0 && params->height % 4 == 0;
  p.v_offset = p.n_rays * p.n_seg;
  return GVR_OK;
}

// The longer edge of view's packets (8 pixels along its right vector) lies
// along this axis of the grid.
int packet_axis(const ViewDev &view, const DiffGrid &g)
{
  int axis = 0;
  for (int a = 1; a < 3; ++a)
    if (std::fabs(view.ru[a]) * g.inv_spacing[a] > std::fabs(view.ru[axis]) * g.inv_spacing[axis]) axis = a;
  return axis;
}

// Copies the field's corner quads into scratch for the forward's views; false
// where the field is read as it is. In microseconds, a call with copies spends 14
// more on the host (scratch and its end) and 5 a copy, and a copy 4.3 per
// million nodes; the quads give back 0.55 per million samples (counted at the
// diagonal's for every ray) where the samples' throughput bounds the frame and
// 0.08 per sample of a ray where the longest ray does. Over 160 calls of 1 to
// 16 views, 4 to 600 samples, 10^3 to 10^6 nodes, this takes the faster side or
// one within some 10% of it; at 8 samples a node alone the copies cost calls with
// short rays 15 to 25 of 80 us. With 14 samples a node, one view of a 128^3
// field at 256^2, the forward went from 102 to 72 us. Where there are not enough
// samples for a copy per axis all views read the one along x. Not under capture,
// where the scratch would become part of the graph, not beyond 1 GiB, and not
// where that is not to be had.
bool make_quads(const float *field, const DiffGrid &g, const DiffViews &views, const DiffParams &p,
                cudaStream_t st, DiffQuads &quads, float4 **scratch)
{
  const int64_t nodes = (int64_t)g.dims[0] * g.dims[1] * g.dims[2];
  const double gain = std::max(0.55e-6 * (double)p.n_rays * p.max_samples, 0.08 * p.max_samples);
  const auto pays = [&](int copies) { return gain > 14.0 + copies * (5.0 + 4.3e-6 * (double)nodes); };
  if (!pays(1) || nodes > ((int64_t)1 << 26)) return false;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusActive;
  if (cudaStreamIsCapturing(st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) return false;
  bool wanted[3] = {};
  int copies = 0;
  for (int v = 0; v < p.n_views; ++v) {
    quads.axis[v] = (unsigned char)packet_axis(views.v[v], g);
    copies += !wanted[quads.axis[v]];
    wanted[quads.axis[v]] = true;
  }
  if (!pays(copies) || copies * nodes > ((int64_t)1 << 26)) {
    std::fill(quads.axis, quads.axis + p.n_views, 0);
    wanted[0] = true;
    wanted[1] = wanted[2] = false;
    copies = 1;
  }
  if (scratch_alloc((void **)scratch, sizeof(float4) * copies * nodes, st) != cudaSuccess) {
    cudaGetLastError();
    *scratch = nullptr;
    return false;
  }
  float4 *to = *scratch;
  for (int f = 0; f < 3; ++f) {
    if (!wanted[f]) continue;
    const int s = f == 0 ? 1 : 0, t = f == 2 ? 1 : 2;
    quads.copy[f] = to;
    quads.stride[f][f] = 1;
    quads.stride[f][s] = g.dims[f];
    quads.stride[f][t] = g.dims[f] * g.dims[s];
    const int u = f == 2 ? 2 : 1;
    const dim3 grid((g.dims[0] + 31) / 32, std::min((g.dims[u] + 31) / 32, 65535), std::min(g.dims[t], 65535));
    const auto gather = f == 0 ? gather_quads<0> : f == 1 ? gather_quads<1> : gather_quads<2>;
    gather<<<grid, dim3(32, 8), 0, st>>>(field, g, to);
    count_launch();
    to += nodes;
  }
  return true;
}

}  // namespace
}  // namespace gvr

using namespace gvr;

extern "C" {

int gvr_diff_workspace(const int dims[3], const double spacing[3], float sample_dist,
                       int *floats_per_ray)
{
  if (!dims || !spacing || !floats_per_ray || !(sample_dist > 0))
    return set_error(GVR_ERR_INVALID_ARGUMENT, "bad arguments");
  double diag = 0;
  for (int a = 0; a < 3; ++a) diag += (double)(dims[a] - 1) * spacing[a] * (double)(dims[a] - 1) * spacing[a];
  const double max_samples = std::sqrt(diag) / sample_dist + 2.0;
  const int n_seg = (int)((max_samples + kDiffK - 1) / kDiffK);
  *floats_per_ray = n_seg * (1 + kDiffK);
  return GVR_OK;
}

int gvr_diff_render_forward(const float *field, const int dims[3], const double origin[3],
                            const double spacing[3], const gvr_camera *cameras, int n_views,
                            const gvr_render_params *params, const float *lut, float *rgba,
                            float *workspace, void *stream)
{
  DiffGrid g;
  DiffViews views;
  DiffParams p;
  int rc = diff_setup(field, dims, origin, spacing, cameras, n_views, params, g, views, p);
  if (rc != GVR_OK) return rc;
  if (!lut || !rgba) return set_error(GVR_ERR_INVALID_ARGUMENT, "NULL lut or rgba");
  const size_t smem = sizeof(float4) * p.lut_size;
  const bool small = (int64_t)dims[0] * dims[1] * dims[2] < ((int64_t)1 << 31);
  cudaStream_t st = (cudaStream_t)stream;
  DiffQuads quads{};
  float4 *scratch = nullptr;
  const auto forward = make_quads(field, g, views, p, st, quads, &scratch)
                           ? diff_forward<int, true>
                           : small ? diff_forward<int, false> : diff_forward<int64_t, false>;
  cudaError_t e = cudaFuncSetAttribute(forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(sizeof(float4) * kDiffLut));
  if (e == cudaSuccess) {
    dim3 grid((p.width + 15) / 16, (p.height + 15) / 16, n_views);
    forward<<<grid, 256, smem, st>>>(field, quads, g, views, p, (const float4 *)lut, (float4 *)rgba, workspace);
    count_launch();
    e = cudaGetLastError();
  }
  if (scratch) cudaFreeAsync(scratch, st);
  if (e != cudaSuccess) return cuda_error(e, "differentiable forward launch");
  return GVR_OK;
}

int gvr_diff_render_backward(const float *field, const int dims[3], const double origin[3],
                             const double spacing[3], const gvr_camera *cameras, int n_views,
                             const gvr_render_params *params, const float *lut,
                             const float *grad_rgba, const float *workspace, float *grad_field,
                             float *grad_lut, void *stream)
{
  DiffGrid g;
  DiffViews views;
  DiffParams p;
  int rc = diff_setup(field, dims, origin, spacing, cameras, n_views, params, g, views, p);
  if (rc != GVR_OK) return rc;
  if (!lut || !grad_rgba || !workspace || !grad_field || !grad_lut)
    return set_error(GVR_ERR_INVALID_ARGUMENT, "NULL buffer");
  const bool shared_t = p.lut_size <= kSharedTLut;
  // of n LUT entries; the attribute is set to the kernel's largest, whatever other threads launch
  const auto shared_bytes = [&](int n) {
    return (sizeof(float4) + sizeof(float)) * n + (shared_t ? sizeof(float) * 256 * kDiffK : 0);
  };
  const size_t smem = shared_bytes(p.lut_size);
  const bool small = (int64_t)dims[0] * dims[1] * dims[2] < ((int64_t)1 << 31);
  const auto backward = shared_t ? (small ? diff_backward<int, true> : diff_backward<int64_t, true>)
                                 : (small ? diff_backward<int, false> : diff_backward<int64_t, false>);
  cudaError_t e = cudaFuncSetAttribute(backward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)shared_bytes(shared_t ? kSharedTLut : kDiffLut));
  if (e != cudaSuccess) return cuda_error(e, "shared-memory attribute");
  // corner-quad buffer of the field gradient, from the library's pool
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nodes = (int64_t)g.dims[0] * g.dims[1] * g.dims[2];
  float4 *gq = nullptr;
  dim3 grid((p.width + 15) / 16, (p.height + 15) / 16, n_views);
  const int64_t n_cta = (int64_t)grid.x * grid.y * grid.z;
  // one copy per CTA, at most 512 MB of copies (CTAs then share them)
  p.lut_copies = (int)std::max<int64_t>(
      1, std::min<int64_t>(n_cta, ((int64_t)512 << 20) / (16 * (int64_t)p.lut_size)));
  float *glc = nullptr;
  e = scratch_alloc((void **)&gq, sizeof(float4) * nodes, st);
  if (e != cudaSuccess) return cuda_error(e, "allocate gradient quads");
  e = scratch_alloc((void **)&glc, sizeof(float) * 4 * p.lut_size * p.lut_copies, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(glc, 0, sizeof(float) * 4 * p.lut_size * p.lut_copies, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(gq, 0, sizeof(float4) * nodes, st);
  if (e == cudaSuccess) {
    backward<<<grid, 256, smem, st>>>(field, g, views, p, (const float4 *)lut,
                                           (const float4 *)grad_rgba, workspace, gq, glc);
    count_launch();
    sum_lut_copies<<<dim3((4 * p.lut_size + 255) / 256, (unsigned)((p.lut_copies + 31) / 32)), 256, 0,
                     st>>>(glc, p.lut_copies, 4 * p.lut_size, grad_lut);
    count_launch();
    fold_quads<<<(unsigned)std::min<int64_t>((nodes + 255) / 256, 152 * 16), 256, 0, st>>>(gq, g,
                                                                                         grad_field);
    count_launch();
    e = cudaGetLastError();
  }
  cudaFreeAsync(gq, st);
  if (glc) cudaFreeAsync(glc, st);
  if (e != cudaSuccess) return cuda_error(e, "differentiable backward launch");
  return GVR_OK;
}

}  // extern "C"
