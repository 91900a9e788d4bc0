// gvr_march_device.cuh — fused ray march + partial compositing (device code of
// the march, staged and batch kernels).
//
// One thread per ray; a warp marches a 4x8-pixel packet and a CTA a 16x16
// tile, so neighbouring lanes read neighbouring bricks. For every pixel the
// kernel does what the reference spreads over several host passes:
//   - per-domain ray setup and march        (StructuredWrapper::render,
//     VolumeRenderer.cpp:223-284; the march itself is VTK-m's
//     VolumeRendererStructured),
//   - partial extraction with the alpha < alpha_cull drop and depth = the
//     ray's exit distance of the domain    (VolumeRenderer.cpp:262-283),
//   - compositing of the partials of all domains in increasing depth with
//     VolumePartial::blend                  (PartialCompositor.cpp:57-90,
//     331-490; VolumePartial.hpp:86-95),
//   - partials_to_canvas: blend over the cleared canvas and image depth
//     0.5 z/w + 0.49                        (VolumeRenderer.cpp:287-391),
//   - the uint8 round trip of the single-domain path (Image.hpp:102-105,
//     Renderer.cpp:265-283) and the background blend.
// Domains are visited in increasing entry distance along each ray, which for
// disjoint boxes is the order the reference's (pixel, exit depth) sort
// produces, so no partial buffer or sort pass is needed.
#pragma once

#include <algorithm>
#include <cfloat>
#include <type_traits>

#include "gvr_hex_device.cuh"

namespace gvr {
namespace {

constexpr int kTile = kMarchTile;  // CTA tile edge in pixels
constexpr int kThreads = 256; // 8 warps, each a 32-ray packet
// Per-ray compositing state kept in shared memory while a domain is marched
// (rgb, front depth, last entry distance, covered exit, last domain, ray
// end, pixel): parked there rather than in registers, the unrolled march
// loop fits 64 registers (4 CTAs per SM) with little or no spilling.
constexpr int kStateSlots = 11;   // the last one: render_ray_unified's sequence position

struct Ray {
  float o[3];
  float d[3];
};

__device__ __forceinline__ bool slab(const float *lo, const float *hi, const Ray &r, float &t0,
                                     float &t1)
{
  float tmin = 0.f, tmax = FLT_MAX;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if (r.d[a] != 0.f) {
      const float inv = 1.f / r.d[a];
      float ta = (lo[a] - r.o[a]) * inv;
      float tb = (hi[a] - r.o[a]) * inv;
      if (ta > tb) { const float t = ta; ta = tb; tb = t; }
      tmin = fmaxf(tmin, ta);
      tmax = fminf(tmax, tb);
    } else if (r.o[a] < lo[a] || r.o[a] > hi[a]) {
      return false;
    }
  }
  t0 = tmin;
  t1 = tmax;
  return tmax > tmin;
}

__device__ __forceinline__ bool slab(const DomainDev &dm, const Ray &r, float &t0, float &t1)
{
  return slab(dm.lo, dm.hi, r, t0, t1);
}

__device__ __forceinline__ float lerpf(float a, float b, float w)
{
  return fmaf(w, b - a, a);
}

// Nearest LUT entry of a saturated scalar s in [0, 1]: s * (n - 1) <= n - 1
// in float, so (int)(s * nm1) is an index of the table without a clamp
// (the value a clamp to n - 1 would give).
__device__ __forceinline__ float4 lut_nearest(const float4 *lut, float nm1, float s)
{
  return lut[(int)(s * nm1)];
}

__device__ __forceinline__ float4 lut_fetch(const float4 *lut, int n, int filter, float s)
{
  if (filter == GVR_LUT_LINEAR) {
    const float x = s * (float)(n - 1);
    int i0 = min((int)x, n - 2);
    const float w = x - (float)i0;
    const float4 a = lut[i0], b = lut[i0 + 1];
    return make_float4(lerpf(a.x, b.x, w), lerpf(a.y, b.y, w), lerpf(a.z, b.z, w),
                       lerpf(a.w, b.w, w));
  }
  const int i = min((int)(s * (float)(n - 1)), n - 1);
  return lut[i];
}

struct Partial {
  float4 acc;   // premultiplied colour and opacity of the domain's partial
  int count;    // samples the stepping rule took
};

// The colour of a saturated scalar, the filter known at compile time: a branch
// per sample on a uniform value costs four instructions of some ninety.
template <bool LIN>
__device__ __forceinline__ float4 lut_color(const float4 *lut, const MarchParams &mp, float nm1, float s)
{
  return LIN ? lut_fetch(lut, mp.lut_size, GVR_LUT_LINEAR, s) : lut_nearest(lut, nm1, s);
}

// a / b from y = RN(1 / b): the product a y corrected by its residual
// (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000", 1990). Three operations against the eight or so and the
// branch of a general division; b is a cell's width and y is kept with it. The
// quotient is the divide's where 1 / b is a normal number and the residual, down
// to 2^-46 a, keeps its last bit: for b in kByReciprocal and a down to 2^-38 b.
// Domains with other cells divide.
__device__ __forceinline__ float div_by(float a, float b, float y)
{
  const float q = a * y;
  return fmaf(fmaf(-q, b, a), y, q);
}

// Rectilinear domains: steps of so many cells and more do not jump to the end of
// an empty brick, whose few samples are counted one by one.
constexpr float kSkipCells = 2.f;

// Along one axis of a rectilinear domain: where p lies past the node ahead,
// step to the ray's next cell and load its record, without a branch.
__device__ __forceinline__ void next_cell(RectCell &q, int &c, float p, const RectCell *recs)
{
  asm("{\n\t.reg .pred n;\n\t.reg .u64 at;\n\t"
      "setp.gt.f32 n, %6, %3;\n\t"
      "@n add.s32 %5, %5, 1;\n\t"
      "mad.wide.s32 at, %5, 32, %7;\n\t"
      "@n ld.global.nc.v4.f32 {%0, %1, %2, %3}, [at];\n\t"
      "@n ld.global.nc.s32 %4, [at + 16];\n\t}"
      : "+f"(q.x0), "+f"(q.width), "+f"(q.inv_width), "+f"(q.ahead), "+r"(q.share), "+r"(c)
      : "f"(p), "l"(recs));
}

// Along one axis: from a cell whose node ahead p may lie past, to the first
// whose does not. Four nodes are compared at a time, since their loads need
// nothing of each other, and the record is loaded for the cell found alone; the
// lists end in four records that nothing lies past.
__device__ __forceinline__ void far_cell(RectCell &q, int &c, float p, const RectCell *__restrict__ recs, unsigned warp)
{
  bool more = p > q.ahead;
  if (!__any_sync(warp, more)) return;
  const bool moves = more;
  do {
    if (more) {
      const RectCell *at = recs + c;
      const bool a = p > __ldg(&at[1].ahead), b = p > __ldg(&at[2].ahead);
      const bool e = p > __ldg(&at[3].ahead), f = p > __ldg(&at[4].ahead);
      // nodes ascend: as many are passed as there are comparisons that hold
      c += min(1 + a + b + e + f, 4);
      more = f;
    }
  } while (__any_sync(warp, more));
  if (moves) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(recs + c));
    q.x0 = v.x;
    q.width = v.y;
    q.inv_width = v.z;
    q.ahead = v.w;
    q.share = __ldg(&recs[c].share);
  }
  __syncwarp(warp);
}

// March one rectilinear domain (ELEM: a cell-centred field; SH: the brick
// shift of a vertex field, 0 = read it) over [t0, t1) from zero opacity: the
// domain's partial and its sample count. A ray crosses each axis in one
// direction, so per axis only the node ahead is compared with the sample's
// position (both times the direction's sign, so that ahead is always
// greater); the cell's record stays in registers and is reloaded by predicated
// loads when the ray leaves the cell, and the corners (ELEM: the value's LUT
// colour) are loaded only for a new cell.
//
// Instruction-bound, and with it a matter of keeping the warp together: the
// step to the next cell has no branch, and the lanes that came here together
// leave together, voting, while lanes that are done idle. Measured on 242 x
// 200 x 174 nodes at 901 x 677: every sample located anew (compares against
// both nodes, two loads and a division per axis, 330 instructions a sample)
// 763 us; the records with `while (past the node) load the next cell` and a
// return per lane, 15 to 18 of 32 lanes active, 710-983 us; without the
// branches and with the votes 532 us; with a record per direction and a
// brick's number taken from the offset (a division by a constant) instead of
// from three cells, 498 us; with every ray going up a list of its own direction,
// 486 us. Not inlined, so that its registers do not weigh on
// the kernels' uniform-grid loop; the ray comes by value and the result goes
// back by value, so nothing is kept in local memory for the call.
template <bool ELEM, int SH, bool DIVIDE = false>
__device__ __noinline__ Partial march_rect(const DomainDev &dm, const Ray r, float t0, float t1,
                                           const MarchParams &mp, const float4 *lut, float thr)
{
  const float dt = mp.sample_dist;
  const int bsh = SH ? SH : dm.bshift;
  const float nm1 = (float)(mp.lut_size - 1);
  const bool skip = !ELEM && mp.skip_empty && *dm.any_empty;
  const RectCell *__restrict__ recs = dm.cell_rec;
  float sg[3], o[3], d[3];   // direction sign; origin and direction times it
  int c[3];                  // the cell's record in the ray's direction
  RectCell q[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    sg[a] = r.d[a] < 0.f ? -1.f : 1.f;
    o[a] = sg[a] * r.o[a];
    d[a] = sg[a] * r.d[a];
    const RectCell *first = recs + dm.rec_first[a];
    const float p = fmaf(t0, r.d[a], r.o[a]);
    int lo = 0, hi = dm.dims[a] - 1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(&first[mid].x0) <= p) lo = mid; else hi = mid;
    }
    c[a] = dm.rec_first[a] + (sg[a] > 0.f ? lo : rect_list(dm.dims[a]) + dm.dims[a] - 2 - lo);
    const float4 v = __ldg(reinterpret_cast<const float4 *>(recs + c[a]));
    q[a].x0 = v.x;
    q[a].width = v.y;
    q[a].inv_width = v.z;
    q[a].ahead = v.w;
    q[a].share = __ldg(&recs[c[a]].share);
  }
  const float *__restrict__ field = ELEM ? dm.cells : dm.bricks;
  const int bn = SH ? brick_nodes(SH) : brick_nodes(bsh), bn2 = bn * bn;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 col = make_float4(0.f, 0.f, 0.f, 0.f);   // ELEM: the cell's colour
  float lc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int brick = -1;
  bool hidden = false;   // the brick is empty
  bool jumps = skip;
  if (!ELEM && skip) {
    // a brick of many cells to a step holds too few samples to jump over
    float cells = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
      cells = fmaxf(cells, __fdividef(fabsf(r.d[a]) * (float)(dm.dims[a] - 1), dm.hi[a] - dm.lo[a]));
    jumps = cells * dt < kSkipCells;
  }
  using At = typename std::conditional<ELEM, int64_t, int>::type;   // a bricked field holds < 2^31 floats
  At last = -1;
  const unsigned warp = __activemask();
  bool done = false;
  for (int k = 0;;) {
    float t = fmaf((float)k, dt, t0);
    done = done || !(t < t1);
    if (!__any_sync(warp, !done)) return Partial{acc, k};
    t = done ? t0 : t;   // a lane that is done stays in its cells
    float p[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) p[a] = fmaf(t, d[a], o[a]);
    // steps of up to three cells one by one, longer ones four at a time
    for (int hops = 0;; ++hops) {
#pragma unroll
      for (int a = 0; a < 3; ++a) next_cell(q[a], c[a], p[a], recs);
      if (!__any_sync(warp, p[0] > q[0].ahead || p[1] > q[1].ahead || p[2] > q[2].ahead)) break;
      if (hops == 2) {
#pragma unroll
        for (int a = 0; a < 3; ++a) far_cell(q[a], c[a], p[a], recs, warp);
        break;
      }
    }
    At at;
    if (ELEM) at = ((At)q[2].share * (dm.dims[1] - 1) + q[1].share) * (dm.dims[0] - 1) + q[0].share;
    else at = q[0].share + q[1].share + q[2].share;
    int taken = 1;   // samples this turn of the loop passes
    if (at != last) {
      last = at;
      if (ELEM) {
        const float v = __ldg(field + at);
        col = lut_fetch(lut, mp.lut_size, mp.lut_filter, __saturatef((v - mp.scalar_min) * mp.inv_range));
      } else {
        if (skip) {
          const int b = at / brick_floats(SH ? SH : bsh);
          if (b != brick) {
            brick = b;
            hidden = dm.brick_empty[b];
          }
        }
        if (!hidden) {
          const float *f = field + at;
          lc[0] = __ldg(f);
          lc[1] = __ldg(f + 1);
          lc[2] = __ldg(f + bn);
          lc[3] = __ldg(f + bn + 1);
          lc[4] = __ldg(f + bn2);
          lc[5] = __ldg(f + bn2 + 1);
          lc[6] = __ldg(f + bn2 + bn);
          lc[7] = __ldg(f + bn2 + bn + 1);
        }
      }
    }
    if (!ELEM && hidden) {
      // zero opacity over the whole brick: the sample is counted alone, or with
      // fine steps all samples up to one step before the ray leaves the brick
      taken = -1;
      if (jumps) {
        float texit = t1;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (r.d[a] != 0.f) {
            const int n = dm.dims[a] - 1, at0 = c[a] - dm.rec_first[a];
            const bool up = sg[a] > 0.f;
            const int ba = (up ? at0 : rect_list(n + 1) + n - 1 - at0) >> bsh;
            const RectCell *x = recs + dm.rec_first[a] + (up ? min(((ba + 1) << bsh) - 1, n - 1) : ba << bsh);
            texit = fminf(texit, __fdividef((up ? __ldg(&x->ahead) : __ldg(&x->x0)) - r.o[a], r.d[a]));
          }
        }
        taken = -max((int)floorf(__fdividef(texit - t0, dt)) - k, 1);   // negative: none of them is blended
      }
    }
    if (!ELEM && __any_sync(warp, !done && !hidden)) {
      float w[3];
#pragma unroll
      for (int a = 0; a < 3; ++a)
        w[a] = __saturatef(DIVIDE ? fmaf(sg[a], p[a], -q[a].x0) / q[a].width
                                  : div_by(fmaf(sg[a], p[a], -q[a].x0), q[a].width, q[a].inv_width));
      const float c00 = lerpf(lc[0], lc[1], w[0]);
      const float c10 = lerpf(lc[2], lc[3], w[0]);
      const float c01 = lerpf(lc[4], lc[5], w[0]);
      const float c11 = lerpf(lc[6], lc[7], w[0]);
      const float v = lerpf(lerpf(c00, c10, w[1]), lerpf(c01, c11, w[1]), w[2]);
      const float s = __saturatef((v - mp.scalar_min) * mp.inv_range);
      col = mp.lut_filter == GVR_LUT_LINEAR ? lut_fetch(lut, mp.lut_size, GVR_LUT_LINEAR, s)
                                            : lut_nearest(lut, nm1, s);
    }
    if (!done) {
      if (taken > 0) {
        const float wa = (1.f - acc.w) * col.w;
        acc.x = fmaf(wa, col.x, acc.x);
        acc.y = fmaf(wa, col.y, acc.y);
        acc.z = fmaf(wa, col.z, acc.z);
        acc.w += wa;
        done = acc.w >= thr;
      }
      k += abs(taken);
    }
  }
}

// March one uniform domain with a cell-centred field. UNROLL samples are
// located and their cells' values loaded before any of them is blended (a
// sample in the cell of the one before it needs neither load nor LUT lookup);
// latency-bound one sample at a time: 255 us for 41.7M samples of 1280 x 720
// pixels over an opaque canvas, 210 us so.
// I indexes the cells: int below 2^31 of them (155 against 164 us for the same
// frame), which a cell-centred field may exceed in one z layer.
template <int UNROLL, typename I>
__device__ __noinline__ Partial march_cells(const DomainDev &dm, const Ray r, float t0, float t1,
                                            const MarchParams &mp, const float4 *lut, float thr)
{
  const float dt = mp.sample_dist;
  float A[3], B[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    A[a] = (r.o[a] - dm.origin[a]) * dm.inv_spacing[a];
    B[a] = r.d[a] * dm.inv_spacing[a];
  }
  const int cmax[3] = {dm.dims[0] - 2, dm.dims[1] - 2, dm.dims[2] - 2};
  const I sy = dm.dims[0] - 1, sz = sy * (dm.dims[1] - 1);
  const float *__restrict__ cells = dm.cells;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), col = acc;
  I last = -1;
  for (int k = 0;; k += UNROLL) {
    bool ok[UNROLL], fresh[UNROLL];
    float v[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      float t = fmaf((float)(k + u), dt, t0);
      ok[u] = t < t1;
      t = ok[u] ? t : t0;
      int c[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) c[a] = max(0, min((int)fmaf(t, B[a], A[a]), cmax[a]));
      const I at = c[2] * sz + (c[1] * sy + c[0]);
      fresh[u] = at != last;
      v[u] = 0.f;
      if (fresh[u]) v[u] = __ldg(cells + at);
      last = at;
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if (!ok[u]) return Partial{acc, k + u};
      if (fresh[u])
        col = lut_fetch(lut, mp.lut_size, mp.lut_filter, __saturatef((v[u] - mp.scalar_min) * mp.inv_range));
      const float wa = (1.f - acc.w) * col.w;
      acc.x = fmaf(wa, col.x, acc.x);
      acc.y = fmaf(wa, col.y, acc.y);
      acc.z = fmaf(wa, col.z, acc.z);
      acc.w += wa;
      if (acc.w >= thr) return Partial{acc, k + u + 1};
    }
  }
}

// Samples k .. k + UNROLL - 1 of a ray in a uniform vertex domain, whose
// grid-space position at distance t is A + t B: each is located, its cell's
// 8 corners are loaded from the bricks unless the sample before was in the
// same cell (lc, last_off hold that cell's), and v[u] is the trilinear
// value. ok[u]: the sample lies before t1 (and, with LIMIT, its index
// before kend); the cell of one that does not is clamped to the domain like any
// other's, so its loads stay inside. Shared by the per-domain loops and the one-loop
// domain walk, so all of them take the same samples with the same
// arithmetic.
template <int UNROLL, int SH, bool LIMIT>
__device__ __forceinline__ void sample_cells(const float *__restrict__ bricks, const float A[3],
                                             const float B[3], const int cmax[3], int sy, int sz,
                                             int k, int kend, float dt, float t0, float t1,
                                             int &last_off, float lc[8], float v[UNROLL],
                                             bool ok[UNROLL])
{
  constexpr int BC = brick_cells(SH), BN = brick_nodes(SH), BF = brick_floats(SH);
  const float kf = (float)k;
#pragma unroll
  for (int u = 0; u < UNROLL; ++u) {
    const float t = fmaf(kf + (float)u, dt, t0);
    ok[u] = LIMIT ? (k + u < kend && t < t1) : t < t1;
    // brick c >> SH, place c - (c >> SH) * BC in it: the offset is linear in
    // both, so the place needs no operation of its own
    int off = 0;
    float w[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float g = fmaf(t, B[a], A[a]);
      const int c = __vimin_s32_relu((int)g, cmax[a]);   // max(0, min)
      w[a] = g - (float)c;
      const int hi = c >> SH;
      off += a == 0 ? hi * (BF - BC) + c
                    : (a == 1 ? hi * (sy - BC * BN) + c * BN : hi * (sz - BC * BN * BN) + c * (BN * BN));
    }
    if (off != last_off) {
      const float *p = bricks + off;
      lc[0] = __ldg(p);
      lc[1] = __ldg(p + 1);
      lc[2] = __ldg(p + BN);
      lc[3] = __ldg(p + BN + 1);
      lc[4] = __ldg(p + BN * BN);
      lc[5] = __ldg(p + BN * BN + 1);
      lc[6] = __ldg(p + BN * BN + BN);
      lc[7] = __ldg(p + BN * BN + BN + 1);
      last_off = off;
    }
    const float c00 = lerpf(lc[0], lc[1], w[0]);
    const float c10 = lerpf(lc[2], lc[3], w[0]);
    const float c01 = lerpf(lc[4], lc[5], w[0]);
    const float c11 = lerpf(lc[6], lc[7], w[0]);
    v[u] = lerpf(lerpf(c00, c10, w[1]), lerpf(c01, c11, w[1]), w[2]);
  }
}

// Uniform grid, vertex field, no empty bricks: the hot path. UNROLL samples
// are located and their 8 corners loaded before any of them is blended, so
// a warp keeps UNROLL x 8 loads in flight. A sample in the cell of the one
// before it reuses that cell's corners from registers (the same values, so
// the result does not change). Blending stays sequential and stops exactly
// where the one-sample loop stops.
template <int UNROLL, int SH, bool LIN>
__device__ __forceinline__ int march_uniform(const DomainDev &dm, const Ray &r, float t0,
                                             float t1, const MarchParams &mp,
                                             const float4 *lut, float thr, float4 &acc)
{
  const float dt = mp.sample_dist;
  float A[3], B[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    A[a] = (r.o[a] - dm.origin[a]) * dm.inv_spacing[a];
    B[a] = r.d[a] * dm.inv_spacing[a];
  }
  const int cmax[3] = {dm.dims[0] - 2, dm.dims[1] - 2, dm.dims[2] - 2};
  constexpr int BC = brick_cells(SH), BN = brick_nodes(SH), BF = brick_floats(SH);
  const int sy = dm.nbrick[0] * BF;
  const int sz = dm.nbrick[1] * sy;
  const float *__restrict__ bricks = dm.bricks;
  const float nm1 = (float)(mp.lut_size - 1);
  // corners of the last cell loaded (at half-cell spacing about half of the
  // samples fall in the cell of the sample before)
  int last_off = -1;
  float lc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // a whole group at a time while its last sample lies before t1 and no
  // opacity on the way reaches the threshold; the last group sample by sample
  // (samples taken: k + u when sample k + u lies past t1, k + u + 1 when it
  // reached the threshold)
  for (int k = 0;; k += UNROLL) {
    float v[UNROLL];
    bool ok[UNROLL];
    sample_cells<UNROLL, SH, false>(bricks, A, B, cmax, sy, sz, k, 0, dt, t0, t1, last_off, lc, v, ok);
    float4 all = acc;
    float top = -INFINITY;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const float s = __saturatef((v[u] - mp.scalar_min) * mp.inv_range);
      const float4 col = lut_color<LIN>(lut, mp, nm1, s);
      const float wa = (1.f - all.w) * col.w;
      all.x = fmaf(wa, col.x, all.x);
      all.y = fmaf(wa, col.y, all.y);
      all.z = fmaf(wa, col.z, all.z);
      all.w += wa;
      top = u ? fmaxf(top, all.w) : all.w;
    }
    if (ok[UNROLL - 1] && !(top >= thr)) {
      acc = all;
      continue;
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if (!ok[u]) return k + u;
      const float s = __saturatef((v[u] - mp.scalar_min) * mp.inv_range);
      const float4 col = lut_color<LIN>(lut, mp, nm1, s);
      const float wa = (1.f - acc.w) * col.w;
      acc.x = fmaf(wa, col.x, acc.x);
      acc.y = fmaf(wa, col.y, acc.y);
      acc.z = fmaf(wa, col.z, acc.z);
      acc.w += wa;
      if (acc.w >= thr) return k + u + 1;
    }
  }
}

// Uniform grid, vertex field, with empty bricks: the march walks the ray
// brick by brick. Entering a brick it computes the last sample before the
// brick's exit (a whole step inside it); an empty brick's samples up to
// there are counted and jumped over (they would blend with zero opacity),
// and a non-empty brick's samples up to its exit run through the same
// unrolled, corner-reusing loop as march_uniform. Compared with a test per
// sample, the emptiness test and the exit distance are paid once per brick.
template <int UNROLL, int SH>
__device__ __forceinline__ int march_bricks(const DomainDev &dm, const Ray &r, float t0,
                                         float t1, const MarchParams &mp,
                                         const float4 *lut, float thr, float4 &acc)
{
  const float dt = mp.sample_dist;
  float A[3], B[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    A[a] = (r.o[a] - dm.origin[a]) * dm.inv_spacing[a];
    B[a] = r.d[a] * dm.inv_spacing[a];
  }
  const int cmax[3] = {dm.dims[0] - 2, dm.dims[1] - 2, dm.dims[2] - 2};
  constexpr int BC = brick_cells(SH), BN = brick_nodes(SH), BF = brick_floats(SH);
  const int sy = dm.nbrick[0] * BF;
  const int sz = dm.nbrick[1] * sy;
  const float *__restrict__ bricks = dm.bricks;
  const float nm1 = (float)(mp.lut_size - 1);
  int count = 0;
  int last_off = -1;
  float lc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  int k = 0;
  for (;;) {
    const float t = fmaf((float)k, dt, t0);
    if (!(t < t1)) return count;
    int b[3];
    float texit = t1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      b[a] = max(0, min((int)fmaf(t, B[a], A[a]), cmax[a])) >> SH;
      if (B[a] != 0.f) {
        const float edge = B[a] > 0.f ? (float)min((b[a] + 1) * BC, cmax[a] + 1)
                                      : (float)(b[a] * BC);
        texit = fminf(texit, (edge - A[a]) / B[a]);
      }
    }
    // samples k .. kx - 1 lie at least one step before the exit
    const int kx = (int)floorf((texit - t0) / dt);
    if (dm.brick_empty[(b[2] * dm.nbrick[1] + b[1]) * dm.nbrick[0] + b[0]]) {
      const int kn = max(kx, k + 1);  // sample k itself is in the empty brick
      count += kn - k;
      k = kn;
      continue;
    }
    const int kend = max(kx + 1, k + 1);
    for (; k < kend; k += UNROLL) {
      float v[UNROLL];
      bool ok[UNROLL];
      sample_cells<UNROLL, SH, true>(bricks, A, B, cmax, sy, sz, k, kend, dt, t0, t1, last_off, lc, v, ok);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        if (!ok[u]) break;
        ++count;
        const float sc = __saturatef((v[u] - mp.scalar_min) * mp.inv_range);
        float4 col;
        if (mp.lut_filter == GVR_LUT_LINEAR) {
          col = lut_fetch(lut, mp.lut_size, GVR_LUT_LINEAR, sc);
        } else {
          col = lut_nearest(lut, nm1, sc);
        }
        const float wa = (1.f - acc.w) * col.w;
        acc.x = fmaf(wa, col.x, acc.x);
        acc.y = fmaf(wa, col.y, acc.y);
        acc.z = fmaf(wa, col.z, acc.z);
        acc.w += wa;
        if (acc.w >= thr) return count;
      }
    }
    k = kend;
  }
}

// Hexahedral domain: each sample is located by Newton's method in the cell
// of the previous sample (starting from its reference coordinates moved by
// the last Jacobian's image of the ray step); when the
// solution lies outside that cell, the march steps to the face neighbour it
// left through (up to kHexHops cells), and only when that fails walks the
// LBVH. The position coefficients of the current cell stay in registers
// between samples. Samples outside every cell contribute nothing but are
// counted, like the structured stepping rule.
//
// The lanes that came here together meet again after each stage of a sample
// and leave together, lanes that are done idling: 13.9 -> 16.7 of 32 lanes
// active, 5101 -> 5001 us for 8M cells at 1024^2, with the L1 pipe at 75%.
// (One Newton step of every lane per turn, each lane at its own sample, takes
// 17% fewer instructions but 57% more L1 wavefronts, since lanes at different
// depths share no cells: 5266 us.)
__device__ int march_hex(const DomainDev &dm, const Ray &r, float t0, float t1,
                         const MarchParams &mp, const float4 *lut, float thr, float4 &acc)
{
  HexGeom v;
  int cur = -1;
  float rst[3] = {0.5f, 0.5f, 0.5f};
  // change of rst from one sample to the next (J^-1 times the ray step,
  // from the last Newton solve): the next sample's guess
  float drst[3] = {0.f, 0.f, 0.f};
  const float step[3] = {r.d[0] * mp.sample_dist, r.d[1] * mp.sample_dist, r.d[2] * mp.sample_dist};
  const unsigned warp = __activemask();
  bool done = false;
  for (int k = 0;;) {
    const float t = fmaf((float)k, mp.sample_dist, t0);
    done = done || !(t < t1);
    if (!__any_sync(warp, !done)) return k;
    const float p[3] = {fmaf(t, r.d[0], r.o[0]), fmaf(t, r.d[1], r.o[1]), fmaf(t, r.d[2], r.o[2])};
    float g[3] = {rst[0] + drst[0], rst[1] + drst[1], rst[2] + drst[2]};
    const bool in_cell = !done && cur >= 0;
    // Predicted exit: the extrapolated guess is clearly outside the cell,
    // so step to the face neighbour before solving (a cheap divergent
    // branch: eight loads) and let every lane do its one solve together;
    // solving in the old cell first and then in the neighbour costs the
    // warp two solves per step (19.5 vs 14.1 Gsamples/s on a jittered
    // 200^3 mesh). Mispredictions fall through to the stepping below.
    if (in_cell && dm.hex_nbr && !(g[0] > -kHexPredictMargin && g[0] < 1.f + kHexPredictMargin &&
                                   g[1] > -kHexPredictMargin && g[1] < 1.f + kHexPredictMargin &&
                                   g[2] > -kHexPredictMargin && g[2] < 1.f + kHexPredictMargin)) {
      const int face = hex_exit_face(g);
      const int nb = __ldg(dm.hex_nbr + 6 * (int64_t)cur + face);
      if (nb >= 0) {
        cur = nb;
        hex_load(dm, cur, v);
        g[face >> 1] += (face & 1) ? -1.f : 1.f;
      }
    }
    __syncwarp(warp);
    int st = -1;
    if (in_cell) st = hex_newton_status(v, p, g, step, drst, true);
    // left the cell: step to the neighbour across the face it left
    // through (Newton's outside solution names it), a few times at most
    for (int hop = 0; hop < kHexHops && __any_sync(warp, st == 0); ++hop) {
      if (st == 0) {
        int nb = -1;
        if (dm.hex_nbr) {
          const int face = hex_exit_face(g);
          nb = __ldg(dm.hex_nbr + 6 * (int64_t)cur + face);
          // guess: the point's coordinates across a like-oriented face
          if (nb >= 0) g[face >> 1] += (face & 1) ? -1.f : 1.f;
        }
        if (nb < 0) {
          st = -1;
        } else {
          cur = nb;
          hex_load(dm, cur, v);
          g[0] = __saturatef(g[0]);
          g[1] = __saturatef(g[1]);
          g[2] = __saturatef(g[2]);
          st = hex_newton_status(v, p, g, step, drst, true);
        }
      }
      __syncwarp(warp);
    }
    if (st == 1) {
      rst[0] = g[0]; rst[1] = g[1]; rst[2] = g[2];
    } else if (!done) {
      cur = hex_locate(dm, p, rst, v);
      drst[0] = drst[1] = drst[2] = 0.f;
    }
    __syncwarp(warp);
    if (!done) {
      ++k;
      if (cur >= 0) {
        float val;
        if (dm.assoc == GVR_ASSOC_ELEMENT) {
          val = __ldg(dm.cells + cur);
        } else {
          val = hex_value(dm, cur, __saturatef(rst[0]), __saturatef(rst[1]), __saturatef(rst[2]));
        }
        const float s = __saturatef((val - mp.scalar_min) * mp.inv_range);
        const float4 col = lut_fetch(lut, mp.lut_size, mp.lut_filter, s);
        const float wa = (1.f - acc.w) * col.w;
        acc.x = fmaf(wa, col.x, acc.x);
        acc.y = fmaf(wa, col.y, acc.y);
        acc.z = fmaf(wa, col.z, acc.z);
        acc.w += wa;
        done = acc.w >= thr;
      }
    }
  }
}

// Everything one ray does: march the candidate domains (bits of `mask`) in
// increasing exit distance, blend their partials, and finish the pixel
// (image depth, uint8 round trip, background). Returns the samples taken.
// g_state: the CTA's shared-memory slots for the state that must survive
// the march of a domain (kStateSlots words per thread, slot k of thread i
// at g_state[k * kThreads + i]).
// The ray of pixel (px, py): the pinhole model partials_to_canvas inverts
// (VolumeRenderer.cpp:335-344).
__device__ __forceinline__ Ray pixel_ray(const ViewDev &view, const MarchParams &mp, int px, int py)
{
  Ray r;
  const float fx = view.dx_scale * ((float)px - 0.5f * (float)mp.width - view.xoff);
  const float fy = view.dy_scale * ((float)py - 0.5f * (float)mp.height - view.yoff);
  float d[3], dn = 0.f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    d[a] = view.look[a] + view.ru[a] * fx + view.rv[a] * fy;
    dn = fmaf(d[a], d[a], dn);
  }
  const float inv = rsqrtf(dn);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    r.o[a] = view.origin[a];
    r.d[a] = d[a] * inv;
  }
  return r;
}

// Opaque canvas: the ray ends at the world point of the canvas depth
// (MapCanvasToRays: pixel (i, j) at depth d unprojected from NDC
// (2i/W - 1, 2j/H - 1, 2d - 1); FP64, as in the oracle). FLT_MAX where the
// pixel's end lies past `far`, at or past the ray's furthest exit from a domain,
// so that it cuts nothing off: an FP32 estimate less its own error bound (each term of
// a row within 16 units in the last place of the sum of the row's magnitudes)
// shows that for the background and for surfaces behind the volume. The FP64
// pipe issues a warp in some 16 cycles, and the hundred or so FP64 operations
// of the plain form for every pixel were more than half of a 1280 x 720 frame;
// the bound takes 12 multiply-adds on matrices that hold the NDC map, and one
// division. Four cell-centred domains of 160 x 144 x 121 cells in all, in front
// of a canvas: 277 us with the plain form and a sample at a time, 163 us so and
// with four in flight.
__device__ __noinline__ float canvas_ray_end(const ViewDev &view, const MarchParams &mp, int px, int py,
                                             float far)
{
  const float d = mp.canvas_depth[(int64_t)py * mp.width + px];
  {
    const float *U = view.unproject_f;
    float P[4], E[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float a = U[4 * q] * (float)px, b = U[4 * q + 1] * (float)py, c = U[4 * q + 2] * d;
      P[q] = a + b + c + U[4 * q + 3];
      E[q] = 1e-6f * (fabsf(a) + fabsf(b) + fabsf(c) + fabsf(U[4 * q + 3]));
    }
    const float w = fabsf(P[3]);
    if (w > 4.f * E[3]) {
      float d2 = 0.f, err = 0.f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float x = P[a] / P[3];
        const float e = x - view.origin[a];
        d2 = fmaf(e, e, d2);
        err += 1.5f * (E[a] + fabsf(x) * E[3]) / w + 1e-6f * fabsf(view.origin[a]);
      }
      if (sqrtf(d2) * 0.99999f - err > far) return FLT_MAX;
    }
  }
  const double *U = view.unproject;
  double P[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) P[q] = U[4 * q] * px + U[4 * q + 1] * py + U[4 * q + 2] * (double)d + U[4 * q + 3];
  if (P[3] == 0.0) return FLT_MAX;
  const double iw = 1.0 / P[3];
  const double ex = P[0] * iw - view.origin[0], ey = P[1] * iw - view.origin[1],
               ez = P[2] * iw - view.origin[2];
  return (float)sqrt(ex * ex + ey * ey + ez * ez);
}

// Where the canvas ends a ray; FLT_MAX without a canvas, where the ray misses
// the box around all domains, and where the canvas lies past that box. (The
// furthest exit of the domains themselves costs a slab test each: 401 -> 484 us
// for 48 small domains at 1280 x 769, before any sample.)
__device__ __forceinline__ float ray_end(const Ray &r, const ViewDev &view, const MarchParams &mp, int px, int py)
{
  float t0, far;
  if (!mp.canvas_depth || !slab(mp.box_lo, mp.box_hi, r, t0, far)) return FLT_MAX;
  return canvas_ray_end(view, mp, px, py, far);
}

// The pixel's final value from its composited partial (have = whether any
// partial survived the cull): partials_to_canvas over the cleared or opaque
// canvas with the image depth, then the uint8 round trip and background.
__device__ __forceinline__ void finish_pixel(const ViewDev &view, const MarchParams &mp, int px, int py,
                                             bool have, const float crgb[3], float ca, float cdepth,
                                             float4 &out, float &dep)
{
  float4 cin = make_float4(0.f, 0.f, 0.f, 0.f);
  float din = mp.clear_depth;
  if (mp.canvas_depth) {
    const int64_t pix = (int64_t)py * mp.width + px;
    cin = mp.canvas_rgba[pix];
    din = mp.canvas_depth[pix];
  }
  out = cin;
  dep = din;
  if (have) {
    const float om = 1.f - ca;
    out = make_float4(crgb[0] + cin.x * om, crgb[1] + cin.y * om, crgb[2] + cin.z * om,
                      cin.w * om + ca);
    // partials_to_canvas ray rebuild: delta_y runs along ru there
    const float ex = view.dx_scale * (float)(2 * px - mp.width) * 0.5f;
    const float ey = view.dy_scale * (float)(2 * py - mp.height) * 0.5f;
    float q[3], qn = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      q[a] = view.look[a] + view.ru[a] * ex + view.ru[a] * ey;
      qn = fmaf(q[a], q[a], qn);
    }
    const float qi = rsqrtf(qn);
    float pos[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) pos[a] = fmaf(cdepth, q[a] * qi, view.origin[a]);
    const float *M = view.projview;
    const float z = M[8] * pos[0] + M[9] * pos[1] + M[10] * pos[2] + M[11];
    const float wv = M[12] * pos[0] + M[13] * pos[1] + M[14] * pos[2] + M[15];
    dep = 0.5f * (z / wv) + 0.49f;
  }
  if (mp.quantize_uint8) {
    out.x = (float)(unsigned char)fminf(out.x * 255.f, 255.f) * (1.f / 255.f);
    out.y = (float)(unsigned char)fminf(out.y * 255.f, 255.f) * (1.f / 255.f);
    out.z = (float)(unsigned char)fminf(out.z * 255.f, 255.f) * (1.f / 255.f);
    out.w = (float)(unsigned char)fminf(out.w * 255.f, 255.f) * (1.f / 255.f);
    dep = fabsf(dep);
  }
  if (mp.render_bg) {
    const float om = 1.f - out.w;
    out.x = fmaf(mp.bg[0], om, out.x);
    out.y = fmaf(mp.bg[1], om, out.y);
    out.z = fmaf(mp.bg[2], om, out.z);
    out.w = fmaf(mp.bg[3], om, out.w);
  }
}

// render_ray for rays whose domains are all uniform vertex fields in 8^3-cell
// bricks: one loop walks the samples of every domain the ray crosses. A lane
// that reaches the end of a domain (or its opacity threshold) blends that
// domain's partial and sets up the next domain inside the same loop, while
// the other lanes of its warp go on sampling; in the per-domain form a
// lane that left its domain first waits at the end of the domain's loop
// until the last lane of the warp leaves it. Empty bricks are met in the same
// loop too: after a group of samples a lane whose last sample lies in another
// brick than before looks that brick up, and where it is empty passes over
// its samples (and the next bricks' while they are empty), again without the
// other lanes; only the bricks' own loop would make them wait at each brick.
// No lane leaves a group early: a lane that is done takes samples of weight
// zero until all lanes of the warp are done, so that the warp stays together.
// The domain order, the sample positions, the per-domain accumulation and the
// blend are render_ray's and march_uniform's, operation for operation, so
// images are identical.
//
// Bound by instructions and, at a sample per half cell and pixel, as much by
// L1 wavefronts (75% of their peak, 33 a sample of a warp). 64 views at 512^2
// of 37 domains, whose rays cross some six of them: a loop per domain and per
// brick kept 18.4 of 32 lanes active and took 36.6 ms; this one keeps 27.9 and
// takes 23.7. The 513^3 field in 8 domains at 1024^2: 1468 us with branches
// out of the group's samples, 1433 us so.
constexpr int kWalkDomains = 10;   // domains of a ray ordered at a time, 6 bits each in two words

template <int UNROLL, int MODE, bool LIN>
__device__ __forceinline__ int render_ray_unified(const DomainDev *doms, uint64_t mask, const ViewDev &view,
                                                  const MarchParams &mp, const float4 *lut, int px, int py,
                                                  float4 &out, float &dep, float *g_state, bool pass_over)
{
  constexpr int BF = brick_floats(3);
  const Ray r = pixel_ray(view, mp, px, py);
  float *st = g_state + threadIdx.x;
  st[7 * kThreads] = MODE == kMarchUniform ? FLT_MAX : ray_end(r, view, mp, px, py);
  st[8 * kThreads] = __int_as_float(px);
  st[9 * kThreads] = __int_as_float(py);
  st[0 * kThreads] = 0.f;          // composited rgb
  st[1 * kThreads] = 0.f;
  st[2 * kThreads] = 0.f;
  st[3 * kThreads] = 0.f;          // depth of the front partial
  st[5 * kThreads] = -FLT_MAX;     // furthest exit covered
  // the ray's domains in render_ray's order, (entry distance, index)
  // ascending, kWalkDomains at a time: five in each of slots 4 and 6, and in
  // slot 10 the next position, their number << 8, the last of them << 16, and
  // bit 24: there are more
  st[10 * kThreads] = __int_as_float(0xff << 16 | 1 << 24);
  float ca = 0.f;
  bool have = false;
  bool live = true;       // the ray has samples left
  bool fresh = true;      // the next turn starts a domain
  bool started = false;   // a domain has been marched (its partial is pending)
  const unsigned warp = __activemask();
  const float dt = mp.sample_dist;
  const float nm1 = (float)(mp.lut_size - 1);
  float A[3] = {0.f, 0.f, 0.f}, B[3] = {0.f, 0.f, 0.f};
  int cmax[3] = {0, 0, 0};
  int sy = 0, sz = 0;
  const float *__restrict__ bricks = nullptr;
  int hidden = -1;        // the domain if it has empty bricks, else -1
  float bt0 = 0.f, bt1 = 0.f, thr = 2.f;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  int k = 0, count = 0;
  int last_off = 0, brick = -1;
  float lc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (;;) {
    if (fresh) {
      fresh = false;
      if (started && !(acc.w < mp.alpha_cull)) {
        if (!have) {
          st[0 * kThreads] = acc.x; st[1 * kThreads] = acc.y; st[2 * kThreads] = acc.z;
          ca = acc.w;
          st[3 * kThreads] = bt1;
          have = true;
        } else if (ca < 1.f && acc.w != 0.f) {
          const float op = 1.f - ca;
          st[0 * kThreads] = fmaf(op, acc.x, st[0 * kThreads]);
          st[1 * kThreads] = fmaf(op, acc.y, st[1 * kThreads]);
          st[2 * kThreads] = fmaf(op, acc.z, st[2 * kThreads]);
          ca = fminf(fmaf(op, acc.w, ca), 1.f);
        }
      }
      int pos = __float_as_int(st[10 * kThreads]);
      if (!(ca >= mp.early_term) && (pos & 255) >= (pos >> 8 & 255) && (pos >> 24)) {
        // order the next domains: those after the last one taken, sorted by
        // insertion as they are found (indices ascend, so of equal entries the
        // lower index stays first)
        float last_t0 = -FLT_MAX;
        int last_d = -1;
        if ((pos >> 16 & 255) != 255) {
          float t1;
          last_d = pos >> 16 & 255;
          slab(doms[last_d], r, last_t0, t1);
        }
        float at[kWalkDomains];
#pragma unroll
        for (int i = 0; i < kWalkDomains; ++i) at[i] = INFINITY;
        uint64_t ids = 0;
        int found = 0;
        for (uint64_t m = mask; m; m &= m - 1) {
          const int d = __ffsll((long long)m) - 1;
          float t0, t1;
          if (!slab(doms[d], r, t0, t1)) continue;
          if (!(t0 > last_t0 || (t0 == last_t0 && d > last_d))) continue;
          ++found;
          int place = 0;
#pragma unroll
          for (int i = kWalkDomains - 1; i >= 0; --i) {
            place += at[i] <= t0 ? 1 : 0;
            at[i] = fminf(at[i], i > 0 ? fmaxf(at[i > 0 ? i - 1 : 0], t0) : t0);
          }
          if (place < kWalkDomains) {
            const uint64_t low = (1ull << (6 * place)) - 1ull;
            ids = (ids & low) | (uint64_t)d << (6 * place) | (ids & ~low) << 6;
          }
        }
        const int n = min(found, kWalkDomains);
        constexpr int kHalf = 6 * kWalkDomains / 2;
        st[4 * kThreads] = __int_as_float((int)(ids & ((1u << kHalf) - 1u)));
        st[6 * kThreads] = __int_as_float((int)((ids >> kHalf) & ((1u << kHalf) - 1u)));
        pos = n << 8 | (n ? (int)(ids >> (6 * n - 6)) & 63 : 255) << 16 | (found > kWalkDomains ? 1 << 24 : 0);
      }
      const int next = pos & 255;
      st[10 * kThreads] = __int_as_float(pos + 1);
      if (ca >= mp.early_term || next >= (pos >> 8 & 255)) {
        // no more: a place whose samples load nothing
        live = false;
        bt0 = bt1 = 0.f;
        A[0] = A[1] = A[2] = B[0] = B[1] = B[2] = 0.f;
        cmax[0] = cmax[1] = cmax[2] = 0;
        last_off = 0;
      } else {
        const uint32_t word = (uint32_t)__float_as_int(st[(next < kWalkDomains / 2 ? 4 : 6) * kThreads]);
        const int d = (int)((word >> (6 * (next < kWalkDomains / 2 ? next : next - kWalkDomains / 2))) & 63u);
        const DomainDev &dm = doms[d];
        float t0, t1;
        slab(dm, r, t0, t1);
        const float covered = st[5 * kThreads];
        bt0 = fmaxf(t0, covered);
        bt1 = fminf(t1, st[7 * kThreads]);
        st[5 * kThreads] = fmaxf(covered, bt1);
        thr = mp.early_term < 1.f ? (mp.early_term - ca) / (1.f - ca) : 2.f;
        acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          A[a] = (r.o[a] - dm.origin[a]) * dm.inv_spacing[a];
          B[a] = r.d[a] * dm.inv_spacing[a];
          cmax[a] = dm.dims[a] - 2;
        }
        sy = dm.nbrick[0] * BF;
        sz = dm.nbrick[1] * sy;
        bricks = dm.bricks;
        hidden = pass_over && *dm.any_empty ? d : -1;
        k = 0;
        last_off = -1;
        brick = -1;
        started = true;
      }
    }
    if (!__any_sync(warp, live)) break;
    float v[UNROLL];
    bool ok[UNROLL];
    sample_cells<UNROLL, 3, false>(bricks, A, B, cmax, sy, sz, k, 0, dt, bt0, bt1, last_off, lc, v, ok);
    // the whole group if its last sample lies in the domain and no opacity on
    // the way reaches the threshold; otherwise, once per ray and domain, again
    // from the start, sample by sample
    float4 all = acc;
    float top = -INFINITY;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const float sc = __saturatef((v[u] - mp.scalar_min) * mp.inv_range);
      const float4 col = lut_color<LIN>(lut, mp, nm1, sc);
      const float wa = (1.f - all.w) * col.w;
      all.x = fmaf(wa, col.x, all.x);
      all.y = fmaf(wa, col.y, all.y);
      all.z = fmaf(wa, col.z, all.z);
      all.w += wa;
      top = u ? fmaxf(top, all.w) : all.w;
    }
    bool on = ok[UNROLL - 1] && !(top >= thr);
    if (on) {
      acc = all;
      k += UNROLL;
    } else if (live) {
      fresh = true;
      bool more = true;
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        if (more && ok[u]) {
          const float sc = __saturatef((v[u] - mp.scalar_min) * mp.inv_range);
          const float4 col = lut_color<LIN>(lut, mp, nm1, sc);
          const float wa = (1.f - acc.w) * col.w;
          acc.x = fmaf(wa, col.x, acc.x);
          acc.y = fmaf(wa, col.y, acc.y);
          acc.z = fmaf(wa, col.z, acc.z);
          acc.w += wa;
          ++k;
          more = !(acc.w >= thr);
        }
      }
      count += k;
    }
    // an offset is its brick's number times BF and a place below BF in it
    if (on && hidden >= 0 && last_off / BF != brick) {
      brick = last_off / BF;
      const DomainDev &dm = doms[hidden];
      int j = k - 1;      // a sample in `brick`
      while (dm.brick_empty[brick]) {
        // the samples up to one step before the ray leaves the brick lie in it
        const float t = fmaf((float)j, dt, bt0);
        float texit = bt1;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (B[a] != 0.f) {
            const int b = max(0, min((int)fmaf(t, B[a], A[a]), cmax[a])) >> 3;
            const float edge = B[a] > 0.f ? (float)min((b + 1) * 8, cmax[a] + 1) : (float)(b * 8);
            texit = fminf(texit, __fdividef(edge - A[a], B[a]));
          }
        }
        j = max((int)floorf(__fdividef(texit - bt0, dt)), j + 1);
        const float tj = fmaf((float)j, dt, bt0);
        if (!(tj < bt1)) break;
        int b3[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) b3[a] = max(0, min((int)fmaf(tj, B[a], A[a]), cmax[a])) >> 3;
        const int nb = (b3[2] * dm.nbrick[1] + b3[1]) * dm.nbrick[0] + b3[0];
        if (nb == brick) break;
        brick = nb;
      }
      k = max(j, k);
    }
    __syncwarp(warp);
  }
  const float crgb[3] = {st[0], st[kThreads], st[2 * kThreads]};
  const float cdepth = st[3 * kThreads];
  px = __float_as_int(st[8 * kThreads]);
  py = __float_as_int(st[9 * kThreads]);
  finish_pixel(view, mp, px, py, have, crgb, ca, cdepth, out, dep);
  return count;
}

// What a frame does at the empty bricks of uniform vertex domains (in 8^3-cell
// bricks): take their samples like any others', which blend as nothing; pass over
// them in the one-loop walk; pass over them in a loop per domain and brick, the
// domains one by one. empty_limits has the limits and the reasons.
enum { kEmptyTake = 0, kEmptyPass = 1, kEmptyByDomain = 2 };
__device__ __forceinline__ int empties_of(const MarchParams &mp)
{
  const int n = mp.skip_empty ? *mp.n_empty : 0;
  return n >= mp.by_domain_from ? kEmptyByDomain : n >= mp.pass_from ? kEmptyPass : kEmptyTake;
}

// MODE: what the scene holds, and so which march code its kernel carries. The
// calls of the rectilinear and cell-centred loops cost a 64-register kernel
// some 90 bytes of spills, which one of uniform vertex fields does without;
// that one has no canvas either (a canvas takes kMarchCells at least).
template <int UNROLL, int MODE>
__device__ __forceinline__ int render_ray(const DomainDev *doms, uint64_t mask, const ViewDev &view,
                                          const MarchParams &mp, const float4 *lut, int px, int py,
                                          float4 &out, float &dep, float *g_state, int empties)
{
  if (MODE != kMarchHex && mask) {
    // domains that are all uniform vertex fields in 8^3-cell bricks, two or
    // more of them or one with empty bricks to pass over: the one-loop walk (a
    // single domain without has no crossing to wait at, and its own loop keeps
    // fewer values live: 1.39 against 1.49 ms on the 513^3 field as one domain)
    bool walk = empties != kEmptyByDomain && doms[__ffsll((long long)mask) - 1].bshift == 3 &&
                ((mask & (mask - 1)) != 0 || empties == kEmptyPass);
    if (MODE != kMarchUniform)
      for (uint64_t m = mask; m; m &= m - 1) {
        const DomainDev &dm = doms[__ffsll((long long)m) - 1];
        walk = walk && dm.kind == GVR_DOMAIN_UNIFORM && dm.assoc == GVR_ASSOC_VERTEX && dm.bshift == 3;
      }
    if (walk)
      return mp.lut_filter == GVR_LUT_LINEAR
                 ? render_ray_unified<UNROLL, MODE, true>(doms, mask, view, mp, lut, px, py, out, dep, g_state, empties == kEmptyPass)
                 : render_ray_unified<UNROLL, MODE, false>(doms, mask, view, mp, lut, px, py, out, dep, g_state, empties == kEmptyPass);
  }
  int count = 0;
  const Ray r = pixel_ray(view, mp, px, py);
  const float t_max = MODE == kMarchUniform ? FLT_MAX : ray_end(r, view, mp, px, py);

  // Compositing state that lives across the march of a domain is parked in
  // shared memory (one word per thread per slot, st[k * kThreads]), so the
  // march loop gets the registers.
  float *st = g_state + threadIdx.x;
  st[7 * kThreads] = t_max;
  st[8 * kThreads] = __int_as_float(px);
  st[9 * kThreads] = __int_as_float(py);
  st[0 * kThreads] = 0.f;          // composited rgb
  st[1 * kThreads] = 0.f;
  st[2 * kThreads] = 0.f;
  st[3 * kThreads] = 0.f;          // depth of the front partial
  st[4 * kThreads] = -FLT_MAX;     // entry distance of the last domain
  st[5 * kThreads] = -FLT_MAX;     // furthest exit covered
  st[6 * kThreads] = __int_as_float(-1);  // last domain
  float ca = 0.f;
  bool have = false;
  for (;;) {
    if (ca >= mp.early_term) break;
    // Next domain along the ray by (entry distance, index). Domains tile
    // space without overlapping, so each is marched from the furthest exit
    // reached so far: every point of the ray is covered once, also where
    // rounding makes neighbouring intervals overlap (rays lying in a shared
    // face). For disjoint boxes this is the order of the reference's
    // (pixel, depth = exit distance) sort.
    int best = -1;
    float bt0 = FLT_MAX, bt1 = 0.f;
    {
      const float last_t0 = st[4 * kThreads];
      const int last_d = __float_as_int(st[6 * kThreads]);
      for (uint64_t m = mask; m; m &= m - 1) {
        const int dd = __ffsll((long long)m) - 1;
        float t0, t1;
        if (!slab(doms[dd], r, t0, t1)) continue;
        const bool after = t0 > last_t0 || (t0 == last_t0 && dd > last_d);
        const bool before = best < 0 || t0 < bt0;
        if (after && before) { best = dd; bt0 = t0; bt1 = t1; }
      }
    }
    if (best < 0) break;
    st[4 * kThreads] = bt0;
    st[6 * kThreads] = __int_as_float(best);
    {
      const float covered = st[5 * kThreads];
      bt0 = fmaxf(bt0, covered);
      bt1 = fminf(bt1, st[7 * kThreads]);
      st[5 * kThreads] = fmaxf(covered, bt1);
    }
    const float thr = mp.early_term < 1.f ? (mp.early_term - ca) / (1.f - ca) : 2.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const DomainDev &dm = doms[best];
    const bool uniform_vertex =
        MODE == kMarchUniform || (dm.kind == GVR_DOMAIN_UNIFORM && dm.assoc == GVR_ASSOC_VERTEX);
    if (MODE == kMarchHex && dm.kind == GVR_DOMAIN_HEX)
      count += march_hex(dm, r, bt0, bt1, mp, lut, thr, acc);
    else if (uniform_vertex && (!(mp.skip_empty && *dm.any_empty) || (empties == kEmptyTake && dm.bshift == 3))) {
      if (mp.lut_filter == GVR_LUT_LINEAR)
        count += dm.bshift == 3 ? march_uniform<UNROLL, 3, true>(dm, r, bt0, bt1, mp, lut, thr, acc)
               : dm.bshift == 2 ? march_uniform<UNROLL, 2, true>(dm, r, bt0, bt1, mp, lut, thr, acc)
                                : march_uniform<UNROLL, 4, true>(dm, r, bt0, bt1, mp, lut, thr, acc);
      else
        count += dm.bshift == 3 ? march_uniform<UNROLL, 3, false>(dm, r, bt0, bt1, mp, lut, thr, acc)
               : dm.bshift == 2 ? march_uniform<UNROLL, 2, false>(dm, r, bt0, bt1, mp, lut, thr, acc)
                                : march_uniform<UNROLL, 4, false>(dm, r, bt0, bt1, mp, lut, thr, acc);
    } else if (uniform_vertex) {
      // 8^3-cell bricks come here next to other kinds of domains and domain by domain
      count += (MODE != kMarchUniform || empties == kEmptyByDomain) && dm.bshift == 3
                   ? march_bricks<UNROLL, 3>(dm, r, bt0, bt1, mp, lut, thr, acc)
                   : dm.bshift == 2 ? march_bricks<UNROLL, 2>(dm, r, bt0, bt1, mp, lut, thr, acc)
                                    : march_bricks<UNROLL, 4>(dm, r, bt0, bt1, mp, lut, thr, acc);
    }
    else {
      Partial part;
      if (MODE >= kMarchRect && dm.kind == GVR_DOMAIN_RECTILINEAR)
        part = dm.assoc == GVR_ASSOC_ELEMENT ? march_rect<true, 0>(dm, r, bt0, bt1, mp, lut, thr)
               : dm.divide                  ? march_rect<false, 0, true>(dm, r, bt0, bt1, mp, lut, thr)
               : dm.bshift == 3             ? march_rect<false, 3>(dm, r, bt0, bt1, mp, lut, thr)
                                             : march_rect<false, 0>(dm, r, bt0, bt1, mp, lut, thr);
      else
        part = (int64_t)(dm.dims[0] - 1) * (dm.dims[1] - 1) * (dm.dims[2] - 1) < ((int64_t)1 << 31)
                   ? march_cells<4, int>(dm, r, bt0, bt1, mp, lut, thr)
                   : march_cells<4, int64_t>(dm, r, bt0, bt1, mp, lut, thr);
      acc = part.acc;
      count += part.count;
    }
    if (acc.w < mp.alpha_cull) continue;
    if (!have) {
      st[0 * kThreads] = acc.x; st[1 * kThreads] = acc.y; st[2 * kThreads] = acc.z;
      ca = acc.w;
      st[3 * kThreads] = bt1;
      have = true;
    } else if (ca < 1.f && acc.w != 0.f) {
      const float op = 1.f - ca;
      st[0 * kThreads] = fmaf(op, acc.x, st[0 * kThreads]);
      st[1 * kThreads] = fmaf(op, acc.y, st[1 * kThreads]);
      st[2 * kThreads] = fmaf(op, acc.z, st[2 * kThreads]);
      ca = fminf(fmaf(op, acc.w, ca), 1.f);
    }
  }
  const float crgb[3] = {st[0], st[kThreads], st[2 * kThreads]};
  const float cdepth = st[3 * kThreads];
  px = __float_as_int(st[8 * kThreads]);
  py = __float_as_int(st[9 * kThreads]);

  finish_pixel(view, mp, px, py, have, crgb, ca, cdepth, out, dep);
  return count;
}

}  // namespace
}  // namespace gvr
