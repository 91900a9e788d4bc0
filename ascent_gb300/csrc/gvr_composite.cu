// gvr_composite.cu — device partial compositing.
//
// Replaces PartialCompositor<VolumePartial<float>>::composite for partials a
// caller already holds (vtkh/compositing/PartialCompositor.cpp:244-547,
// BlendPartials :57-90, VolumePartial::blend VolumePartial.hpp:53-62). The
// result is the reference's: records ordered by (pixel id, depth) with
// equal keys in input order; pixels with one record are copied, the others
// blended front to back; output = single-record pixels in pixel order, then
// blended pixels in pixel order (composite_partials :422-489). The blend
// uses explicitly rounded FP32 operations (no fused multiply-add), so the
// output is bit-identical to the reference compiled without contraction.
//
// Two ways to group the records by pixel:
//   dense ids (pixel range <= 2 n + 64 Ki, the normal case: ids are y*W+x)
//     a per-pixel histogram whose atomics also hand every record its slot
//     in its pixel's bucket, scans over the pixel range for the bucket
//     offsets and for the output slots, and one thread per pixel that
//     orders its few records by (depth, input index) and blends them;
//   sparse ids
//     a stable device radix sort of 64-bit keys (pixel id, order-preserving
//     depth bits), segment flags and scans, one thread per blended pixel.
// Scratch comes from the library's stream-ordered memory pool
// (scratch_alloc), which keeps its memory between calls.
#include <algorithm>
#include <cstdint>

#include "gvr_internal.h"

namespace gvr {
namespace {

using Partial = gvr_partial;
static_assert(sizeof(Partial) == 24, "VolumePartial<float> layout");

// Unsigned key with the order of float <; -0 and +0 compare equal there, so
// both map to the key of +0 (equal keys keep their input order).
__device__ __forceinline__ uint32_t order_bits(float f)
{
  uint32_t u = __float_as_uint(f);
  if (u == 0x80000000u) u = 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ void blend_into(Partial &r, const Partial &o)
{
  // VolumePartial::blend
  if (r.alpha >= 1.f || o.alpha == 0.f) return;
  const float op = __fsub_rn(1.f, r.alpha);
  r.rgb[0] = __fadd_rn(r.rgb[0], __fmul_rn(op, o.rgb[0]));
  r.rgb[1] = __fadd_rn(r.rgb[1], __fmul_rn(op, o.rgb[1]));
  r.rgb[2] = __fadd_rn(r.rgb[2], __fmul_rn(op, o.rgb[2]));
  r.alpha = __fadd_rn(r.alpha, __fmul_rn(op, o.alpha));
  r.alpha = r.alpha > 1.f ? 1.f : r.alpha;
}

__global__ void key_kernel(const Partial *__restrict__ in, int64_t n, uint64_t *__restrict__ keys,
                           uint32_t *__restrict__ idx)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const Partial p = in[i];
    const uint32_t pid = (uint32_t)p.pixel_id ^ 0x80000000u;  // signed order
    keys[i] = ((uint64_t)pid << 32) | order_bits(p.depth);
    idx[i] = (uint32_t)i;
  }
}

// flags: uniq[i] = 1 for a pixel with one record, multi[i] = 1 for the first
// record of a pixel with several
__global__ void flag_kernel(const uint64_t *__restrict__ keys, int64_t n, uint32_t *__restrict__ uniq,
                            uint32_t *__restrict__ multi)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t pid = (uint32_t)(keys[i] >> 32);
    const bool head = i == 0 || (uint32_t)(keys[i - 1] >> 32) != pid;
    const bool last = i == n - 1 || (uint32_t)(keys[i + 1] >> 32) != pid;
    uniq[i] = head && last;
    multi[i] = head && !last;
  }
}

// Unique and blended pixel counts of the sorted path: last exclusive
// prefix plus last flag.
__global__ void sorted_totals_kernel(const uint32_t *upos, const uint32_t *uniq, const uint32_t *mpos,
                                     const uint32_t *multi, int64_t n, uint32_t *totals)
{
  if (threadIdx.x == 0) {
    totals[0] = upos[n - 1] + uniq[n - 1];
    totals[1] = mpos[n - 1] + multi[n - 1];
  }
}

__global__ void emit_kernel(const Partial *__restrict__ in, const uint64_t *__restrict__ keys,
                            const uint32_t *__restrict__ idx, int64_t n,
                            const uint32_t *__restrict__ upos, const uint32_t *__restrict__ mpos,
                            const uint32_t *__restrict__ uniq, const uint32_t *__restrict__ multi,
                            const uint32_t *__restrict__ totals, Partial *__restrict__ out)
{
  const uint32_t n_unique = totals[0];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (uniq[i]) {
      out[upos[i]] = in[idx[i]];
    } else if (multi[i]) {
      Partial r = in[idx[i]];
      const uint32_t pid = (uint32_t)(keys[i] >> 32);
      for (int64_t j = i + 1; j < n && (uint32_t)(keys[j] >> 32) == pid; ++j) blend_into(r, in[idx[j]]);
      out[n_unique + mpos[i]] = r;
    }
  }
}

// Smallest and largest pixel id, as order-preserving unsigned values
// (mm[0] starts at 0xffffffff, mm[1] at 0).
__global__ void range_kernel(const Partial *__restrict__ in, int64_t n, unsigned *__restrict__ mm)
{
  unsigned lo = 0xffffffffu, hi = 0u;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned u = (unsigned)in[i].pixel_id ^ 0x80000000u;
    lo = min(lo, u);
    hi = max(hi, u);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  // one pair of atomics per block, not per warp (thousands of warps on two
  // addresses serialise at L2)
  __shared__ unsigned slo[32], shi[32];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    slo[w] = lo;
    shi[w] = hi;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = (int)(blockDim.x >> 5);
    lo = threadIdx.x < nw ? slo[threadIdx.x] : 0xffffffffu;
    hi = threadIdx.x < nw ? shi[threadIdx.x] : 0u;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (threadIdx.x == 0) {
      atomicMin(mm, lo);
      atomicMax(mm + 1, hi);
    }
  }
}

// cnt[p] = records of pixel lo + p; pr[i] = {p, record i's slot in its
// bucket} (slots in arrival order; the emit kernel restores input order),
// so that the bucket pass reads 8 bytes per record instead of the 24-byte
// records again. A record whose id lies outside [lo, lo + r) (possible only
// when the caller gave the range) is left out (p = 0xffffffff) and sets
// *bad.
__global__ void count_kernel(const Partial *__restrict__ in, int64_t n, int lo, int64_t r,
                             uint32_t *__restrict__ cnt, uint2 *__restrict__ pr,
                             unsigned *__restrict__ bad)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = (int64_t)in[i].pixel_id - lo;
    if (p < 0 || p >= r) {
      atomicOr(bad, 1u);
      pr[i] = make_uint2(0xffffffffu, 0u);
      continue;
    }
    pr[i] = make_uint2((uint32_t)p, atomicAdd(cnt + p, 1u));
  }
}

__global__ void bucket_kernel(const uint2 *__restrict__ pr, int64_t n, int64_t r,
                              const uint32_t *__restrict__ off, uint32_t *__restrict__ order)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint2 v = pr[i];
    if ((int64_t)v.x >= r) continue;
    order[off[v.x] + v.y] = (uint32_t)i;
  }
}

// Output count of the caller-range path into the caller's device int64:
// -1 when a record's pixel id was outside the given range.
__global__ void count_out_kernel(const uint32_t *__restrict__ totals, const unsigned *__restrict__ bad,
                                 int64_t *__restrict__ n_out)
{
  if (threadIdx.x == 0) *n_out = *bad ? -1 : (int64_t)totals[0] + totals[1];
}

// upos[p] = 1 for pixels with one record, mpos[p] = 1 for pixels with more
// (scanned in place afterwards into output slots).
__global__ void pixel_flag_kernel(const uint32_t *__restrict__ cnt, int64_t r,
                                  uint32_t *__restrict__ upos, uint32_t *__restrict__ mpos)
{
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < r;
       p += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t c = cnt[p];
    upos[p] = c == 1;
    mpos[p] = c > 1;
  }
}

// The three pixel scans of the dense path in one pass over the counts:
// off = exclusive scan of cnt (bucket offsets), upos / mpos = exclusive
// scans of (cnt == 1) / (cnt > 1) (output slots). A tile of kTile3 pixels
// per block writes its local prefixes and its totals; one block scans the
// tile totals (at most kTile3 tiles, so r <= kTile3^2); a last pass adds
// each tile's base. Replaces a copy, a flag kernel and three three-launch
// scans (11 operations) by three launches.
constexpr int kTile3 = 1024;

__device__ __forceinline__ uint3 add3(uint3 a, uint3 b) { return make_uint3(a.x + b.x, a.y + b.y, a.z + b.z); }

// Inclusive block scan of one uint3 per thread (kTile3 threads); returns the
// thread's inclusive prefix, *tot receives the block total.
__device__ __forceinline__ uint3 block_scan3(uint3 v, uint3 *tot)
{
  __shared__ uint3 warp_tot[kTile3 / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint3 x = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint3 y;
    y.x = __shfl_up_sync(0xffffffffu, x.x, o);
    y.y = __shfl_up_sync(0xffffffffu, x.y, o);
    y.z = __shfl_up_sync(0xffffffffu, x.z, o);
    if (lane >= o) x = add3(x, y);
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint3 t = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      uint3 y;
      y.x = __shfl_up_sync(0xffffffffu, t.x, o);
      y.y = __shfl_up_sync(0xffffffffu, t.y, o);
      y.z = __shfl_up_sync(0xffffffffu, t.z, o);
      if (lane >= o) t = add3(t, y);
    }
    warp_tot[lane] = t;
  }
  __syncthreads();
  if (warp > 0) x = add3(x, warp_tot[warp - 1]);
  *tot = warp_tot[kTile3 / 32 - 1];
  return x;
}

__global__ void __launch_bounds__(kTile3)
scan3_tile_kernel(const uint32_t *__restrict__ cnt, int64_t r, uint32_t *__restrict__ off,
                  uint32_t *__restrict__ upos, uint32_t *__restrict__ mpos, uint3 *__restrict__ sums)
{
  const int64_t p = (int64_t)blockIdx.x * kTile3 + threadIdx.x;
  const uint32_t c = p < r ? cnt[p] : 0u;
  const uint3 v = make_uint3(c, c == 1, c > 1);
  uint3 tot;
  const uint3 inc = block_scan3(v, &tot);
  if (p < r) {
    off[p] = inc.x - v.x;
    upos[p] = inc.y - v.y;
    mpos[p] = inc.z - v.z;
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// One block: exclusive scan of the tile totals in place.
__global__ void __launch_bounds__(kTile3) scan3_top_kernel(uint3 *__restrict__ sums, int tiles)
{
  const uint3 v = threadIdx.x < tiles ? sums[threadIdx.x] : make_uint3(0u, 0u, 0u);
  uint3 tot;
  const uint3 inc = block_scan3(v, &tot);
  if (threadIdx.x < tiles) sums[threadIdx.x] = make_uint3(inc.x - v.x, inc.y - v.y, inc.z - v.z);
}

__global__ void __launch_bounds__(kTile3)
scan3_add_kernel(int64_t r, uint32_t *__restrict__ off, uint32_t *__restrict__ upos,
                 uint32_t *__restrict__ mpos, const uint3 *__restrict__ sums)
{
  const int64_t p = (int64_t)blockIdx.x * kTile3 + threadIdx.x;
  if (p >= r) return;
  const uint3 b = sums[blockIdx.x];
  off[p] += b.x;
  upos[p] += b.y;
  mpos[p] += b.z;
}

constexpr int kLocalSort = 32;  // records per pixel ordered in thread-local arrays

__device__ __forceinline__ bool before(uint32_t ka, uint32_t ia, uint32_t kb, uint32_t ib)
{
  return ka < kb || (ka == kb && ia < ib);
}

// One thread per pixel: copy or blend its records in (depth, input index)
// order. totals[0..1] receive the unique and blended pixel counts.
__global__ void pixel_emit_kernel(const Partial *__restrict__ in, const uint32_t *__restrict__ cnt,
                                  const uint32_t *__restrict__ off, const uint32_t *__restrict__ upos,
                                  const uint32_t *__restrict__ mpos, uint32_t *__restrict__ order,
                                  int64_t r, Partial *__restrict__ out, uint32_t *__restrict__ totals)
{
  const uint32_t n_unique = upos[r - 1] + (cnt[r - 1] == 1);
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < r;
       p += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t c = cnt[p];
    if (p == r - 1) {
      totals[0] = n_unique;
      totals[1] = mpos[p] + (c > 1);
    }
    if (c == 0) continue;
    uint32_t *seg = order + off[p];
    if (c == 1) {
      out[upos[p]] = in[seg[0]];
      continue;
    }
    Partial res;
    if (c <= 8) {
      // the common case (one record per partial image, at most 8 images):
      // keys and indices in registers, ordered by Batcher's odd-even merge
      // network for 8 inputs (19 compare-exchanges; padding sorts last)
      uint32_t key[8], idx[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if ((uint32_t)j < c) {
          const uint32_t i = seg[j];
          key[j] = order_bits(in[i].depth);
          idx[j] = i;
        } else {
          key[j] = 0xffffffffu;
          idx[j] = 0xffffffffu;
        }
      }
      auto cx = [&](int a, int b) {
        if (before(key[b], idx[b], key[a], idx[a])) {
          const uint32_t tk = key[a], ti = idx[a];
          key[a] = key[b];
          idx[a] = idx[b];
          key[b] = tk;
          idx[b] = ti;
        }
      };
      cx(0, 1); cx(2, 3); cx(4, 5); cx(6, 7);
      cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7);
      cx(1, 2); cx(5, 6);
      cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7);
      cx(2, 4); cx(3, 5);
      cx(1, 2); cx(3, 4); cx(5, 6);
      res = in[idx[0]];
#pragma unroll
      for (int j = 1; j < 8; ++j)
        if ((uint32_t)j < c) blend_into(res, in[idx[j]]);
    } else if (c <= kLocalSort) {
      uint32_t key[kLocalSort], idx[kLocalSort];
      for (uint32_t j = 0; j < c; ++j) {
        const uint32_t i = seg[j];
        const uint32_t k = order_bits(in[i].depth);
        uint32_t q = j;
        while (q > 0 && before(k, i, key[q - 1], idx[q - 1])) {
          key[q] = key[q - 1];
          idx[q] = idx[q - 1];
          --q;
        }
        key[q] = k;
        idx[q] = i;
      }
      res = in[idx[0]];
      for (uint32_t j = 1; j < c; ++j) blend_into(res, in[idx[j]]);
    } else {
      // rare deep pixels: insertion sort of the bucket in place
      for (uint32_t j = 1; j < c; ++j) {
        const uint32_t i = seg[j];
        const uint32_t k = order_bits(in[i].depth);
        uint32_t q = j;
        while (q > 0) {
          const uint32_t pi = seg[q - 1];
          if (!before(k, i, order_bits(in[pi].depth), pi)) break;
          seg[q] = pi;
          --q;
        }
        seg[q] = i;
      }
      res = in[seg[0]];
      for (uint32_t j = 1; j < c; ++j) blend_into(res, in[seg[j]]);
    }
    out[n_unique + mpos[p]] = res;
  }
}

// ---------------------------------------------------------------------------
// Slots: the dense path while the pixels are no more than twice the records.
// Every pixel has kSlots places for record indices (place s of all pixels
// together: neighbouring records mostly take the same place of neighbouring
// pixels), which a record's atomic on the pixel's count hands out directly, so
// there is no bucket offset to scan for and no second pass over the records
// before they are blended; records beyond the places hang on the pixel in a
// list. Bound by memory: the records
// are read twice, once for their pixel ids (24-byte records, so every sector of
// them) and once to blend, the index places stay in L2. 8 images of 1024^2 at
// 80% cover (6.7M records, 161 MB): the histogram, three scans, bucket and emit
// passes took 150 us of kernels, these three 99: 38 (4.6 TB/s), 7 and 51, the
// last waiting for its records (55 with a barrier between a thread's pixels, 61
// at 3 CTAs per SM, 92 at 5, where it spills).
// ---------------------------------------------------------------------------
constexpr int kSlots = 8;
constexpr int kSlotThreads = 256;
constexpr uint32_t kWarpDeep = 1024;   // records of a pixel that a warp orders alone

// Word-sized loads of a record, or 8-byte ones where the array is aligned.
template <bool WIDE>
__device__ __forceinline__ Partial load_partial(const Partial *__restrict__ p)
{
  Partial r;
  if (WIDE) {
    const uint2 *q = reinterpret_cast<const uint2 *>(p);
    const uint2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    r.pixel_id = (int32_t)a.x;
    r.depth = __uint_as_float(a.y);
    r.rgb[0] = __uint_as_float(b.x);
    r.rgb[1] = __uint_as_float(b.y);
    r.rgb[2] = __uint_as_float(c.x);
    r.alpha = __uint_as_float(c.y);
  } else {
    r = *p;
  }
  return r;
}

// A record outside [lo, lo + r) (possible only when the caller gave the range)
// is left out and sets *bad.
__global__ void __launch_bounds__(256)
slot_kernel(const Partial *__restrict__ in, int64_t n, int lo, int64_t r, uint32_t *__restrict__ cnt,
            uint32_t *__restrict__ place, uint32_t *__restrict__ head, uint32_t *__restrict__ next,
            unsigned *__restrict__ bad)
{
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = (int64_t)__ldg(&in[i].pixel_id) - lo;
    if (p < 0 || p >= r) {
      atomicOr(bad, 1u);
      continue;
    }
    const uint32_t s = atomicAdd(cnt + p, 1u);
    if (s < kSlots) place[s * r + p] = (uint32_t)i;
    else next[i] = atomicExch(head + p, (uint32_t)i + 1u);   // 0 ends a list
  }
}

// Pixels with one record and with more, per tile of ROWS x 256; the CTA that
// finishes last turns the tiles' numbers into exclusive prefixes and writes the
// totals.
template <int ROWS>
__global__ void __launch_bounds__(kSlotThreads)
slot_sums_kernel(const uint32_t *__restrict__ cnt, int64_t r, uint2 *__restrict__ sums, int tiles,
                 unsigned *__restrict__ finished, uint32_t *__restrict__ totals)
{
  __shared__ uint2 part[8];
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned one = 0, more = 0;
  const int64_t p0 = (int64_t)blockIdx.x * (ROWS * kSlotThreads);
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const int64_t p = p0 + q * kSlotThreads + threadIdx.x;
    const uint32_t c = p < r ? cnt[p] : 0u;
    one += c == 1;
    more += c > 1;
  }
  one = __reduce_add_sync(0xffffffffu, one);
  more = __reduce_add_sync(0xffffffffu, more);
  if (lane == 0) part[warp] = make_uint2(one, more);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      one += part[w].x;
      more += part[w].y;
    }
    sums[blockIdx.x] = make_uint2(one, more);
    __threadfence();
    last = atomicAdd(finished, 1u) == (unsigned)tiles - 1u;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  uint2 run = make_uint2(0u, 0u);
  for (int t0 = 0; t0 < tiles; t0 += 256) {
    const int t = t0 + threadIdx.x;
    const uint2 v = t < tiles ? __ldcg(sums + t) : make_uint2(0u, 0u);
    uint2 x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned a = __shfl_up_sync(0xffffffffu, x.x, o), b = __shfl_up_sync(0xffffffffu, x.y, o);
      if (lane >= o) {
        x.x += a;
        x.y += b;
      }
    }
    if (lane == 31) part[warp] = x;
    __syncthreads();
    uint2 base = run;
    for (int w = 0; w < 8; ++w) {
      if (w < warp) {
        base.x += part[w].x;
        base.y += part[w].y;
      }
      run.x += part[w].x;
      run.y += part[w].y;
    }
    if (t < tiles) sums[t] = make_uint2(base.x + x.x - v.x, base.y + x.y - v.y);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    totals[0] = run.x;
    totals[1] = run.y;
  }
}

// Blends a pixel's c records, whose indices are rows[0 .. c - 1].y, in (depth,
// input index) order: by one warp, or by all of a CTA (the last blend by its
// first warp alone). Each record's place is the number of those before it;
// next[] of the pixel's own records, which nothing walks any more, holds the
// order. Every lane of the blending warp gets the result.
template <bool CTA, bool WIDE>
__device__ __forceinline__ Partial blend_deep(const Partial *__restrict__ in, uint2 *rows, uint32_t c, uint32_t *next)
{
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t t = CTA ? threadIdx.x : lane, step = CTA ? kSlotThreads : 32;
  const auto meet = [] {
    if (CTA) __syncthreads();
    else __syncwarp();
  };
  for (uint32_t j = t; j < c; j += step) rows[j].x = order_bits(__ldg(&in[rows[j].y].depth));
  meet();
  for (uint32_t j = t; j < c; j += step) {
    const uint2 mine = rows[j];
    uint32_t rank = 0;
    for (uint32_t q = 0; q < c; ++q) {
      const uint2 o = rows[q];
      rank += before(o.x, o.y, mine.x, mine.y);
    }
    next[rows[rank].y] = mine.y;
  }
  meet();
  Partial res{};
  if (CTA && threadIdx.x >= 32) return res;
  for (uint32_t j0 = 0; j0 < c; j0 += 32) {
    Partial mine{};
    if (j0 + lane < c) mine = load_partial<WIDE>(in + next[rows[j0 + lane].y]);
    const uint32_t m = min(32u, c - j0);
    for (uint32_t k = 0; k < m; ++k) {
      Partial rec;
      rec.pixel_id = __shfl_sync(0xffffffffu, mine.pixel_id, k);
      rec.depth = __shfl_sync(0xffffffffu, mine.depth, k);
#pragma unroll
      for (int a = 0; a < 3; ++a) rec.rgb[a] = __shfl_sync(0xffffffffu, mine.rgb[a], k);
      rec.alpha = __shfl_sync(0xffffffffu, mine.alpha, k);
      if (j0 + k == 0) res = rec;
      else blend_into(res, rec);
    }
  }
  return res;
}

// One thread per pixel: copy its record or blend its records in (depth, input
// index) order. Up to kSlots records are loaded whole, so that each is read
// once, and ordered by Batcher's odd-even merge network (19 exchanges) with
// their colours. Up to kLocalSort are ordered by insertion in local arrays,
// their indices, then their depths, then the records loaded several at a time.
// Of more, the thread writes the indices down and a warp blends them later, all
// of the CTA's warps together those of more than kWarpDeep: 64 images of 256^2,
// 480 us (sorted by insertion, a thread a pixel, 1110 us; by the whole CTA one
// after the other, with one thread walking the list, 11 ms); one pixel of 5000
// records 2.9 ms (861 by insertion). n_out (may be NULL)
// receives the count, -1 when a record was outside the caller's range.
template <int ROWS, bool WIDE>
__global__ void __launch_bounds__(kSlotThreads, 4)
slot_emit_kernel(const Partial *__restrict__ in, const uint32_t *__restrict__ cnt,
                 const uint32_t *__restrict__ place, const uint32_t *__restrict__ head, uint32_t *next,
                 const uint2 *__restrict__ sums, int64_t r, Partial *__restrict__ out,
                 const uint32_t *__restrict__ totals, const unsigned *__restrict__ bad,
                 int64_t *__restrict__ n_out, uint2 *rows, uint32_t *__restrict__ used)
{
  constexpr int kTile = ROWS * kSlotThreads;   // pixels per CTA
  __shared__ uint2 part[ROWS][8];
  __shared__ int n_deep, n_deepest;       // pixels deeper than kLocalSort, and than kWarpDeep
  // of each: place in the tile, output, rows; the deepest from the end
  __shared__ int deep[kTile];
  __shared__ uint32_t deep_out[kTile], deep_row[kTile];
  if (threadIdx.x == 0) n_deep = n_deepest = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n_unique = totals[0];
  if (n_out && blockIdx.x == 0 && threadIdx.x == 0)
    *n_out = *bad ? -1 : (int64_t)n_unique + totals[1];
  // the counts and output slots of all of a thread's pixels first, so that
  // nothing is waited for between them
  __shared__ uint32_t counts[ROWS][kSlotThreads];
#pragma unroll
  for (int q = 0; q < ROWS; ++q) {
    const int64_t p = (int64_t)blockIdx.x * kTile + q * kSlotThreads + threadIdx.x;
    const uint32_t c = p < r ? __ldg(cnt + p) : 0u;
    const unsigned ones = __ballot_sync(0xffffffffu, c == 1), mores = __ballot_sync(0xffffffffu, c > 1);
    counts[q][threadIdx.x] = c;
    if (lane == 0) part[q][warp] = make_uint2(__popc(ones), __popc(mores));
  }
  __syncthreads();
  uint2 base = sums[blockIdx.x];
#pragma unroll 1
  for (int q = 0; q < ROWS; ++q) {
    const int64_t p = (int64_t)blockIdx.x * kTile + q * kSlotThreads + threadIdx.x;
    const uint32_t c = counts[q][threadIdx.x];
    uint32_t upos = base.x + __popc(__ballot_sync(0xffffffffu, c == 1) & ((1u << lane) - 1u));
    uint32_t mpos = base.y + __popc(__ballot_sync(0xffffffffu, c > 1) & ((1u << lane) - 1u));
    for (int w = 0; w < 8; ++w) {
      const uint2 v = part[q][w];
      if (w < warp) {
        upos += v.x;
        mpos += v.y;
      }
      base.x += v.x;
      base.y += v.y;
    }
    if (c == 0) continue;
    const uint32_t *seg = place + p;
    if (c == 1) {
      out[upos] = load_partial<WIDE>(in + seg[0]);
      continue;
    }
    Partial res;
    if (c <= kSlots) {
      uint32_t idx[8], key[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) idx[j] = (uint32_t)j < c ? __ldg(seg + j * r) : 0u;
      Partial rec[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if ((uint32_t)j < c) rec[j] = load_partial<WIDE>(in + idx[j]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if ((uint32_t)j < c) {
          key[j] = order_bits(rec[j].depth);
        } else {
          // sorts last, and blends as nothing
          key[j] = 0xffffffffu;
          idx[j] = 0xffffffffu;
          rec[j] = Partial{0, 0.f, {0.f, 0.f, 0.f}, 0.f};
        }
      }
      auto cx = [&](int a, int b) {
        const bool swap = before(key[b], idx[b], key[a], idx[a]);
        const uint32_t ka = key[a], ia = idx[a];
        const Partial ra = rec[a];
        key[a] = swap ? key[b] : ka;
        idx[a] = swap ? idx[b] : ia;
        key[b] = swap ? ka : key[b];
        idx[b] = swap ? ia : idx[b];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          rec[a].rgb[m] = swap ? rec[b].rgb[m] : ra.rgb[m];
          rec[b].rgb[m] = swap ? ra.rgb[m] : rec[b].rgb[m];
        }
        rec[a].alpha = swap ? rec[b].alpha : ra.alpha;
        rec[b].alpha = swap ? ra.alpha : rec[b].alpha;
      };
      cx(0, 1); cx(2, 3); cx(4, 5); cx(6, 7);
      cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7);
      cx(1, 2); cx(5, 6);
      cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7);
      cx(2, 4); cx(3, 5);
      cx(1, 2); cx(3, 4); cx(5, 6);
      res = rec[0];
      res.pixel_id = __ldg(&in[idx[0]].pixel_id);
      res.depth = __ldg(&in[idx[0]].depth);
#pragma unroll
      for (int j = 1; j < 8; ++j)
        if ((uint32_t)j < c) blend_into(res, rec[j]);
    } else if (c <= kLocalSort) {
      uint32_t key[kLocalSort], idx[kLocalSort];
      uint32_t held = kSlots;
#pragma unroll
      for (int m = 0; m < kSlots; ++m) idx[m] = __ldg(seg + m * r);
      for (uint32_t t = head[p]; t; t = next[t - 1]) idx[held++] = t - 1;
#pragma unroll 8
      for (uint32_t j = 0; j < c; ++j) key[j] = order_bits(__ldg(&in[idx[j]].depth));
      for (uint32_t j = 1; j < c; ++j) {
        const uint32_t k = key[j], i = idx[j];
        uint32_t to = j;
        while (to > 0 && before(k, i, key[to - 1], idx[to - 1])) {
          key[to] = key[to - 1];
          idx[to] = idx[to - 1];
          --to;
        }
        key[to] = k;
        idx[to] = i;
      }
      res = load_partial<WIDE>(in + idx[0]);
#pragma unroll 4
      for (uint32_t j = 1; j < c; ++j) blend_into(res, load_partial<WIDE>(in + idx[j]));
    } else {
      const uint32_t row = atomicAdd(used, c);
      uint32_t m = row;
      for (int j = 0; j < kSlots; ++j) rows[m++].y = seg[j * r];
      for (uint32_t t = head[p]; t; t = next[t - 1]) rows[m++].y = t - 1;
      const int d = c <= kWarpDeep ? atomicAdd(&n_deep, 1) : kTile - 1 - atomicAdd(&n_deepest, 1);
      deep[d] = q * kSlotThreads + (int)threadIdx.x;
      deep_out[d] = n_unique + mpos;
      deep_row[d] = row;
      continue;
    }
    out[n_unique + mpos] = res;
  }
  __syncthreads();
  for (int d = warp; d < n_deep; d += kSlotThreads / 32) {
    const Partial res = blend_deep<false, WIDE>(in, rows + deep_row[d], cnt[(int64_t)blockIdx.x * kTile + deep[d]], next);
    if (lane == 0) out[deep_out[d]] = res;
  }
  for (int d = kTile - 1; d > kTile - 1 - n_deepest; --d) {
    const Partial res = blend_deep<true, WIDE>(in, rows + deep_row[d], cnt[(int64_t)blockIdx.x * kTile + deep[d]], next);
    if (threadIdx.x == 0) out[deep_out[d]] = res;
  }
}

int grid_of(int64_t n)
{
  const int64_t b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 152 * 32 ? 152 * 32 : b));
}

// Scratch of one call, carved from a single stream-ordered allocation.
struct Arena {
  char *base = nullptr;
  size_t used = 0;
  template <typename T>
  T *take(size_t count)
  {
    T *p = reinterpret_cast<T *>(base + used);
    used += (sizeof(T) * std::max<size_t>(count, 1) + 255) & ~(size_t)255;
    return p;
  }
};

size_t dense_bytes(int64_t n, int64_t r)
{
  return 256 * 9 + (4 * (size_t)r + 3 * (size_t)n + std::max<size_t>(scan_scratch_words(r), 3 * 1024) + 3) *
                       sizeof(uint32_t);
}

size_t sorted_bytes(int64_t n)
{
  return 256 * 12 + (2 * sizeof(uint64_t) + 6 * sizeof(uint32_t)) * (size_t)n +
         (sort_scratch_words(n) + scan_scratch_words(n) + 2) * sizeof(uint32_t);
}

// Whether the slots serve: their places are read for every pixel, and take 32
// bytes of scratch each (40 a pixel and 12 a record in all, the histogram path
// 16 and 12: where the larger amount is not to be had, that path is taken).
bool use_slots(int64_t n, int64_t r) { return r <= 2 * n; }

size_t slot_bytes(int64_t n, int64_t r)
{
  return 256 * 9 + ((2 + kSlots) * (size_t)r + 3 * (size_t)n + 2 * (size_t)((r + kSlotThreads - 1) / kSlotThreads) + 8) *
                       sizeof(uint32_t);
}

// Four pixels per thread of the last two passes, whose loads overlap, where the
// records fit their places on average and the CTAs of 1024 pixels fill the SMs
// once, four each; otherwise one, as the few CTAs or a thread's deep pixels one
// after the other make the pass longer. 8 images of 1024^2 at 80%: 116 us with
// four, 135 with one; 12 images (9.6 records a pixel) 347 and 324; 8 of 256^2:
// 41 and 36.
constexpr int64_t kSlotWave = 152 * 4;
bool four_per_thread(int64_t n, int64_t r) { return n <= kSlots * r && r >= kSlotWave * 4 * kSlotThreads; }

template <int ROWS>
void launch_slot_passes(const Partial *in, int64_t r, Partial *out, const uint32_t *cnt, const uint32_t *place,
                        const uint32_t *head, uint32_t *next, uint2 *sums, uint32_t *totals, unsigned *bad,
                        unsigned *finished, uint32_t *used, int64_t *n_out, uint2 *rows, cudaStream_t st)
{
  const unsigned tiles = (unsigned)((r + ROWS * kSlotThreads - 1) / (ROWS * kSlotThreads));
  slot_sums_kernel<ROWS><<<tiles, kSlotThreads, 0, st>>>(cnt, r, sums, (int)tiles, finished, totals);
  const auto emit = ((uintptr_t)in & 7) == 0 ? slot_emit_kernel<ROWS, true> : slot_emit_kernel<ROWS, false>;
  emit<<<tiles, kSlotThreads, 0, st>>>(in, cnt, place, head, next, sums, r, out, totals, bad, n_out, rows, used);
}

// Dense pixel ids, no more than twice as many as records: slots, tile sums,
// per-pixel emit. n_out: see slot_emit_kernel.
cudaError_t composite_slots(const Partial *in, int64_t n, int lo, int64_t r, Partial *out, Arena &a,
                            uint32_t *totals, int64_t *n_out, cudaStream_t st)
{
  uint32_t *place = a.take<uint32_t>(kSlots * (size_t)r);
  uint32_t *next = a.take<uint32_t>(n);
  uint2 *rows = a.take<uint2>(n);   // deep pixels' records: key, index
  uint2 *sums = a.take<uint2>((r + kSlotThreads - 1) / kSlotThreads);
  // counts, list heads and the three words are cleared together
  uint32_t *cnt = a.take<uint32_t>(2 * (size_t)r + 3), *head = cnt + r;
  unsigned *bad = head + r, *finished = bad + 1, *used = bad + 2;
  cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * (2 * (size_t)r + 3), st);
  if (e != cudaSuccess) return e;
  slot_kernel<<<grid_of(n), 256, 0, st>>>(in, n, lo, r, cnt, place, head, next, bad);
  const auto passes = four_per_thread(n, r) ? launch_slot_passes<4> : launch_slot_passes<1>;
  passes(in, r, out, cnt, place, head, next, sums, totals, bad, finished, used, n_out, rows, st);
  count_launch(3);
  return cudaGetLastError();
}

// Dense pixel ids: histogram, bucket, per-pixel emit.
cudaError_t composite_dense(const Partial *in, int64_t n, int lo, int64_t r, Partial *out,
                            Arena &a, uint32_t *totals, unsigned *bad, cudaStream_t st)
{
  uint32_t *cnt = a.take<uint32_t>(r), *off = a.take<uint32_t>(r);
  uint32_t *upos = a.take<uint32_t>(r), *mpos = a.take<uint32_t>(r);
  uint2 *pr = a.take<uint2>(n);
  uint32_t *order = a.take<uint32_t>(n);
  uint32_t *scan_tmp = a.take<uint32_t>(std::max<size_t>(scan_scratch_words(r), 3 * (size_t)kTile3));
  cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * r, st);
  if (e != cudaSuccess) return e;
  count_kernel<<<grid_of(n), 256, 0, st>>>(in, n, lo, r, cnt, pr, bad);
  count_launch();
  const int64_t tiles = (r + kTile3 - 1) / kTile3;
  if (tiles <= kTile3) {
    uint3 *sums = reinterpret_cast<uint3 *>(scan_tmp);   // 3 words per tile, within scan_tmp
    scan3_tile_kernel<<<(unsigned)tiles, kTile3, 0, st>>>(cnt, r, off, upos, mpos, sums);
    count_launch();
    if (tiles > 1) {
      scan3_top_kernel<<<1, kTile3, 0, st>>>(sums, (int)tiles);
      scan3_add_kernel<<<(unsigned)tiles, kTile3, 0, st>>>(r, off, upos, mpos, sums);
      count_launch(2);
    }
  } else {
    if ((e = cudaMemcpyAsync(off, cnt, sizeof(uint32_t) * r, cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
      return e;
    if ((e = exclusive_scan(off, r, scan_tmp, st)) != cudaSuccess) return e;
    pixel_flag_kernel<<<grid_of(r), 256, 0, st>>>(cnt, r, upos, mpos);
    count_launch();
    if ((e = exclusive_scan(upos, r, scan_tmp, st)) != cudaSuccess) return e;
    if ((e = exclusive_scan(mpos, r, scan_tmp, st)) != cudaSuccess) return e;
  }
  bucket_kernel<<<grid_of(n), 256, 0, st>>>(pr, n, r, off, order);
  count_launch();
  pixel_emit_kernel<<<grid_of(r), 256, 0, st>>>(in, cnt, off, upos, mpos, order, r, out, totals);
  count_launch();
  return cudaGetLastError();
}

// Any pixel ids: stable radix sort by (pixel id, depth), segment scans.
cudaError_t composite_sorted(const Partial *in, int64_t n, Partial *out, Arena &a,
                             uint32_t *totals, cudaStream_t st)
{
  uint64_t *keys = a.take<uint64_t>(n), *keys_tmp = a.take<uint64_t>(n);
  uint32_t *idx = a.take<uint32_t>(n), *idx_tmp = a.take<uint32_t>(n);
  uint32_t *uniq = a.take<uint32_t>(n), *multi = a.take<uint32_t>(n);
  uint32_t *upos = a.take<uint32_t>(n), *mpos = a.take<uint32_t>(n);
  uint32_t *scratch = a.take<uint32_t>(sort_scratch_words(n));
  uint32_t *scan_tmp = a.take<uint32_t>(scan_scratch_words(n));
  key_kernel<<<grid_of(n), 256, 0, st>>>(in, n, keys, idx);
  count_launch();
  cudaError_t e = radix_sort_pairs<uint64_t>(keys, idx, keys_tmp, idx_tmp, n, 64, scratch, st);
  if (e != cudaSuccess) return e;
  flag_kernel<<<grid_of(n), 256, 0, st>>>(keys, n, uniq, multi);
  count_launch();
  if ((e = cudaMemcpyAsync(upos, uniq, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(mpos, multi, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
  if ((e = exclusive_scan(upos, n, scan_tmp, st)) != cudaSuccess) return e;
  if ((e = exclusive_scan(mpos, n, scan_tmp, st)) != cudaSuccess) return e;
  sorted_totals_kernel<<<1, 32, 0, st>>>(upos, uniq, mpos, multi, n, totals);
  count_launch();
  emit_kernel<<<grid_of(n), 256, 0, st>>>(in, keys, idx, n, upos, mpos, uniq, multi, totals, out);
  count_launch();
  return cudaGetLastError();
}

}  // namespace
}  // namespace gvr

using namespace gvr;

extern "C" int gvr_composite_partials(const gvr_partial *partials, int64_t n, gvr_partial *out,
                                      int64_t *n_out, int location, void *stream)
{
  if (!n_out || n < 0 || (n > 0 && (!partials || !out)))
    return set_error(GVR_ERR_INVALID_ARGUMENT, "bad partial arrays");
  if (location != GVR_MEM_HOST && location != GVR_MEM_DEVICE)
    return set_error(GVR_ERR_INVALID_ARGUMENT, "bad location");
  if (n >= ((int64_t)1 << 31)) return set_error(GVR_ERR_UNSUPPORTED, "at most 2^31 - 1 partials");
  *n_out = 0;
  if (n == 0) return GVR_OK;
  cudaStream_t st = (cudaStream_t)stream;
  Partial *d_in = nullptr, *d_out = nullptr;
  unsigned *mm = nullptr;
  Arena arena;
  unsigned hm[2] = {0u, 0u};
  uint32_t ht[2] = {0u, 0u};
  uint32_t *totals = nullptr;
  cudaError_t e = cudaSuccess;
  int rc = GVR_OK;
#define CP_TRY(expr, what)                                        \
  do {                                                            \
    e = (expr);                                                   \
    if (e != cudaSuccess) { rc = cuda_error(e, what); goto done; } \
  } while (0)
  if (location == GVR_MEM_HOST) {
    CP_TRY(scratch_alloc((void **)&d_in, sizeof(Partial) * n, st), "allocate partials");
    CP_TRY(scratch_alloc((void **)&d_out, sizeof(Partial) * n, st), "allocate output");
    CP_TRY(cudaMemcpyAsync(d_in, partials, sizeof(Partial) * n, cudaMemcpyHostToDevice, st), "copy partials");
  } else {
    d_in = const_cast<Partial *>(partials);
    d_out = out;
  }
  // pixel-id range (merge computes the same, PartialCompositor.cpp:279-306)
  CP_TRY(scratch_alloc((void **)&mm, 2 * sizeof(unsigned), st), "allocate range");
  CP_TRY(cudaMemsetAsync(mm, 0xff, sizeof(unsigned), st), "range");
  CP_TRY(cudaMemsetAsync(mm + 1, 0, sizeof(unsigned), st), "range");
  range_kernel<<<grid_of(n), 256, 0, st>>>(d_in, n, mm);
  count_launch();
  CP_TRY(cudaMemcpyAsync(hm, mm, sizeof(hm), cudaMemcpyDeviceToHost, st), "read range");
  CP_TRY(cudaStreamSynchronize(st), "composite");
  {
    const int lo = (int)(hm[0] ^ 0x80000000u), hi = (int)(hm[1] ^ 0x80000000u);
    const int64_t r = (int64_t)hi - lo + 1;
    const bool dense = r <= 2 * n + 65536 && r < ((int64_t)1 << 31);
    bool slots = dense && use_slots(n, r);
    CP_TRY(slots ? scratch_alloc((void **)&arena.base, slot_bytes(n, r), dense_bytes(n, r), &slots, st)
                 : scratch_alloc((void **)&arena.base, dense ? dense_bytes(n, r) : sorted_bytes(n), st),
           "allocate scratch");
    totals = arena.take<uint32_t>(2);
    // the range was measured, so no record is outside it: mm[0] serves as
    // the (unused) flag word
    CP_TRY(slots   ? composite_slots(d_in, n, lo, r, d_out, arena, totals, nullptr, st)
           : dense ? composite_dense(d_in, n, lo, r, d_out, arena, totals, mm, st)
                   : composite_sorted(d_in, n, d_out, arena, totals, st),
           "composite");
    CP_TRY(cudaMemcpyAsync(ht, totals, sizeof(ht), cudaMemcpyDeviceToHost, st), "read counts");
    CP_TRY(cudaStreamSynchronize(st), "composite");
    const int64_t total = (int64_t)ht[0] + ht[1];
    if (location == GVR_MEM_HOST) {
      CP_TRY(cudaMemcpyAsync(out, d_out, sizeof(Partial) * total, cudaMemcpyDeviceToHost, st), "copy output");
      CP_TRY(cudaStreamSynchronize(st), "composite");
    }
    *n_out = total;
  }
done:
#undef CP_TRY
  if (location == GVR_MEM_HOST) {
    if (d_in) cudaFreeAsync(d_in, st);
    if (d_out) cudaFreeAsync(d_out, st);
  }
  if (mm) cudaFreeAsync(mm, st);
  if (arena.base) cudaFreeAsync(arena.base, st);
  return rc;
}

extern "C" int gvr_composite_partials_async(const gvr_partial *partials, int64_t n, int32_t pixel_lo,
                                            int32_t pixel_hi, gvr_partial *out, int64_t *n_out,
                                            void *stream)
{
  if (!n_out || n < 0 || (n > 0 && (!partials || !out)))
    return set_error(GVR_ERR_INVALID_ARGUMENT, "bad partial arrays");
  if (pixel_hi < pixel_lo) return set_error(GVR_ERR_INVALID_ARGUMENT, "pixel_hi < pixel_lo");
  if (n >= ((int64_t)1 << 31)) return set_error(GVR_ERR_UNSUPPORTED, "at most 2^31 - 1 partials");
  const int64_t r = (int64_t)pixel_hi - pixel_lo + 1;
  if (r > ((int64_t)1 << 30)) return set_error(GVR_ERR_UNSUPPORTED, "pixel range above 2^30");
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e;
  if (n == 0) {
    e = cudaMemsetAsync(n_out, 0, sizeof(int64_t), st);
    return e == cudaSuccess ? GVR_OK : cuda_error(e, "composite");
  }
  Arena arena;
  bool slots = use_slots(n, r);
  e = slots ? scratch_alloc((void **)&arena.base, slot_bytes(n, r), dense_bytes(n, r), &slots, st)
            : scratch_alloc((void **)&arena.base, dense_bytes(n, r), st);
  if (e != cudaSuccess) return cuda_error(e, "allocate scratch");
  uint32_t *totals = arena.take<uint32_t>(2);
  if (slots) {
    e = composite_slots(reinterpret_cast<const Partial *>(partials), n, pixel_lo, r, reinterpret_cast<Partial *>(out),
                        arena, totals, n_out, st);
    cudaFreeAsync(arena.base, st);
    return e == cudaSuccess ? GVR_OK : cuda_error(e, "composite");
  }
  unsigned *bad = arena.take<unsigned>(1);
  e = cudaMemsetAsync(bad, 0, sizeof(unsigned), st);
  if (e == cudaSuccess)
    e = composite_dense(reinterpret_cast<const Partial *>(partials), n, pixel_lo, r,
                        reinterpret_cast<Partial *>(out), arena, totals, bad, st);
  if (e == cudaSuccess) {
    count_out_kernel<<<1, 32, 0, st>>>(totals, bad, n_out);
    count_launch();
    e = cudaGetLastError();
  }
  cudaFreeAsync(arena.base, st);
  if (e != cudaSuccess) return cuda_error(e, "composite");
  return GVR_OK;
}
