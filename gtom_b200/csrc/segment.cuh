// Row segments: the pixels of a slice whose sample position falls in a box,
// found analytically instead of by a per-pixel binning pass.
//
// A slice pixel (u, v) sits at u * c0 + v * c1 in the volume (c0, c1 the
// first two matrix columns; the third column meets z = 0 for 2D slices).
// For a box [lo, hi] each axis r bounds u in row v to the interval
//   lo_r <= u * c0_r + v * c1_r <= hi_r,
// and the rows that can hold such a pixel lie between the extremes over the
// box of the linear function v(p) that recovers v from a point of the plane.
// The plan (brick_plan.cu) stores one record per (slice, side, brick) with
// such rows; a warp takes a few records of its brick at a time and deals
// their rows out to its lanes, then the rows' pixels (seg_deal).  The boxes
// are widened by a margin well above the float error of both the positions
// and these bounds, so the candidates are a superset of the pixels the box
// holds; the caller applies the exact test with the kernels' own
// arithmetic (project_sample / backproject_sample), which decides alone.
#pragma once

#include "brick.cuh"

namespace gtomrln {

// Margin (voxels) by which callers widen a box: above the float error of a
// sample position (|pos| < 2^14 voxels: a few ulp, ~1e-3) and of the
// interval bounds below (relative 1e-6 of the same magnitudes).
constexpr float kSegMargin = 0.01f;

// A box and the pixel -> position map of one (slice, side): c0, c1 the
// matrix columns (negated for the mirror side).
struct SegBox {
  float c0[3], c1[3], lo[3], hi[3];
};

// The box of brick origin o, edge B, widened by `widen` (a bound on how far
// samples leave the flat map, e.g. by the Ewald curvature) and the margin.
__device__ __forceinline__ void seg_box_bounds(SegBox& b, int3 o, int B, float widen) {
  const float w = widen + kSegMargin;
  b.lo[0] = (float)o.x - w;
  b.lo[1] = (float)o.y - w;
  b.lo[2] = (float)o.z - w;
  const float e = (float)B + w;
  b.hi[0] = (float)o.x + e;
  b.hi[1] = (float)o.y + e;
  b.hi[2] = (float)o.z + e;
}

// Largest u with u^2 <= rem (0 <= rem < 2^24: radii below 4 096), exactly:
// the approximate square root is within a unit of the truth there, which the
// two integer corrections absorb.
__device__ __forceinline__ int seg_isqrt(int rem) {
  float f;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"((float)rem));
  int r = (int)f;
  r -= r * r > rem;
  r += (r + 1) * (r + 1) <= rem;
  return r;
}

// Approximate reciprocal (a few ulp), for bounds that a margin widens.
__device__ __forceinline__ float seg_rcp(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

// The linear functions of a slice that bound its rows in a box: on the plane
// v(p) = w . p and u(p) = w' . p, w = (g00 c1 - g01 c0) / det, w' =
// (g11 c0 - g01 c1) / det, whose extremes over the box bound the rows and
// reject a box that lies wholly at u < 0 (the other side's pixels).
// Near-parallel columns (det small against g00 g11) keep the full range;
// well-conditioned ones (det above a quarter of g00 g11: an error of a few
// 1e-6 of the magnitudes) need little padding.
struct SegRows {
  float wv[3], wu[3];  // w and w'
  float av, au;        // sums of their magnitudes
  float pad0, padr;    // padding: absolute, and relative to the magnitudes
  int vmin, vmax;      // the slice's rows within the pixel set's radius
  bool plane;          // whether w, w' exist
};
__device__ __forceinline__ SegRows seg_rows_setup(const float* m, const PixelSet& px) {
  SegRows s;
  const int rlim = seg_isqrt(px.strict ? px.rmax2 - 1 : px.rmax2);
  s.vmin = max(px.n / 2 + 1 - px.n, -rlim);  // rows idy > n/2 hold v = idy - n
  s.vmax = min(px.n / 2, rlim);
  const float g00 = m[0] * m[0] + m[1] * m[1] + m[2] * m[2];
  const float g11 = m[3] * m[3] + m[4] * m[4] + m[5] * m[5];
  const float g01 = m[0] * m[3] + m[1] * m[4] + m[2] * m[5];
  const float det = g00 * g11 - g01 * g01;
  s.plane = det > 1e-3f * g00 * g11 && g00 > 0.f;
  const bool well = det > 0.25f * g00 * g11;
  s.pad0 = well ? 0.02f : 0.5f;
  s.padr = well ? 1e-4f : 1e-3f;
  const float inv = 1.f / det;
  s.av = s.au = 0.f;
#pragma unroll
  for (int r = 0; r < 3; r++) {
    s.wv[r] = (g00 * m[3 + r] - g01 * m[r]) * inv;
    s.wu[r] = (g11 * m[r] - g01 * m[3 + r]) * inv;
    s.av += fabsf(s.wv[r]);
    s.au += fabsf(s.wu[r]);
  }
  return s;
}
// Row ranges of side 0 and side 1 (mirrored: the functions negated) in the
// cube of centre (cx, cy, cz) and half edge h; empty as vlo > vhi.
__device__ __forceinline__ void seg_rows(const SegRows& s, const PixelSet& px, float cx, float cy, float cz, float h,
                                         int vlo[2], int vhi[2]) {
  const float vc = s.wv[0] * cx + s.wv[1] * cy + s.wv[2] * cz, uc = s.wu[0] * cx + s.wu[1] * cy + s.wu[2] * cz;
  const float vh = s.av * h, uh = s.au * h;
  const float pu = uh + s.pad0 + s.padr * (fabsf(uc) + uh), pv = vh + s.pad0 + s.padr * (fabsf(vc) + vh);
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const float u = side ? -uc : uc, v = side ? -vc : vc;
    vlo[side] = s.vmin;
    vhi[side] = s.vmax;
    if (s.plane) {
      vlo[side] = max(s.vmin, (int)ceilf(fmaxf(v - pv, -1e6f)));
      vhi[side] = min(s.vmax, (int)floorf(fminf(v + pv, 1e6f)));
      if (u + pu < 0.f || u - pu > (float)(px.dimft - 1)) vhi[side] = vlo[side] - 1;
    }
  }
}

// Pixel interval [ua, ub] of row v holding the box, clipped to the pixel set
// (ub < ua when empty).  The bounds multiply by the approximate reciprocal of
// the column entry: a few more ulp, far inside the margin.
__device__ __forceinline__ void seg_row(const SegBox& b, const PixelSet& px, int v, int& ua, int& ub) {
  float umin = -1.f, umax = (float)px.dimft;
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const float a = b.c0[r], t = (float)v * b.c1[r];
    const float l = b.lo[r] - t, h = b.hi[r] - t;
    // |a| <= 1e-20 moves a * u by < 1e-16 over the row: a u-free test, which
    // the margin keeps conservative (and 1 / a stays finite otherwise)
    if (fabsf(a) > 1e-20f) {
      const float ra = seg_rcp(a);
      const float e0 = l * ra, e1 = h * ra;
      umin = fmaxf(umin, fminf(e0, e1));
      umax = fminf(umax, fmaxf(e0, e1));
    } else if (l > 0.f || h < 0.f) {
      umin = 1.f;
      umax = 0.f;
    }
  }
  const int rem = (px.strict ? px.rmax2 - 1 : px.rmax2) - v * v;
  if (rem < 0 || !(umin <= umax)) {
    ua = 1;
    ub = 0;
    return;
  }
  ua = max((int)ceilf(umin), (px.strict && v < 0) ? 1 : 0);
  ub = min((int)floorf(umax), min(seg_isqrt(rem), px.dimft - 1));
}

// One (slice, side, brick) of a segment plan, grouped by brick: the slice
// matrix's first two columns (negated on side 1 where the plan's geometry
// asks for it), the slice and side, and the row range.
struct __align__(32) SegRec {
  float c0[3], c1[3];
  int ss;    // 2 * slice + side
  int rows;  // first row in the low 16 bits (signed), row count above
};
static_assert(sizeof(SegRec) == 32, "SegRec is read as two 16-byte words");

// A record's two 16-byte words: {c0, c1.x} and {c1.y, c1.z, ss, rows}.
struct SegWords {
  float4 a, b;
  __device__ __forceinline__ int ss() const { return __float_as_int(b.z); }
};
__device__ __forceinline__ SegWords seg_load(const SegRec* rec) {  // from shared memory
  const float4* p = reinterpret_cast<const float4*>(rec);
  SegWords w;
  w.a = p[0];
  w.b = p[1];
  return w;
}

__device__ __forceinline__ int seg_pack_rows(int vlo, int vhi) {
  return (int)(((unsigned)vlo & 0xffffu) | ((unsigned)(vhi - vlo + 1) << 16));
}

// Records a warp takes at a time.  A record has ~13 rows of ~8 pixels at
// padding 2 (256^2 slices, 25..29-voxel bricks), so eight of them fill the
// lanes of three to four row passes and the pixels of a pass seven waves.
constexpr int kSegChunk = 8;

// Deals the pixels of np <= kSegChunk consecutive records out to the warp:
// their rows 32 at a time to the lanes, each lane bounding its row's pixel
// interval (bounds(p, v, ua, ub): record p, row v), then the pixels of those
// rows 32 per wave, f(p, u, v, valid) once per lane and wave (valid false on
// idle lanes of a last wave, whose p stays a record of the chunk).  rows:
// the record's packed rows on lane p, 0 on lanes >= np.  Taking one record
// at a time instead left most row lanes and every record's last wave
// part-filled and cost 380 instructions per 32 samples in the projector.
// Warp-synchronous.
template <class Bounds, class F>
__device__ __forceinline__ void seg_deal(int rows, Bounds&& bounds, F&& f) {
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nr = rows >> 16;
  int incl = nr;
#pragma unroll
  for (int o = 1; o < kSegChunk; o <<= 1) {
    const int t = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += t;
  }
  const int total = __shfl_sync(full, incl, kSegChunk - 1);
  const int vs = (int)(short)(rows & 0xffff) - (incl - nr);  // row k of the chunk is v = vs + k
  const unsigned le = full >> (31 - lane);
  for (int rb = 0; rb < total; rb += 32) {
    const int k = rb + lane;
    // record of row k: the number of records whose rows end at or before k
    int p = 0;
#pragma unroll
    for (int step = kSegChunk / 2; step > 0; step >>= 1) {
      const int t = __shfl_sync(full, incl, p + step - 1);
      if (t <= k) p += step;
    }
    const int v = __shfl_sync(full, vs, p) + k;
    int ua = 0, cnt = 0;
    if (k < total) {
      int ub;
      bounds(p, v, ua, ub);
      cnt = max(0, ub - ua + 1);
    }
    const unsigned nz = __ballot_sync(full, cnt > 0);
    if (!nz) continue;
    int inc2 = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(full, inc2, o);
      if (lane >= o) inc2 += t;
    }
    const int tot = __shfl_sync(full, inc2, 31);
    // the non-empty rows moved to the first lanes: lane i gets the row at
    // the (i+1)-th set bit of nz
    int r = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__popc(nz & ((1u << (r + step)) - 1u)) <= lane) r += step;
    const int key = __shfl_sync(full, (p << 16) | (v & 0xffff), r);
    const int st = __shfl_sync(full, inc2 - cnt, r);
    const int off = __shfl_sync(full, ua, r) - st;
    const int start = lane < __popc(nz) ? st : 0x7fffffff;
    // wave by wave: the rows that start in the wave mark their first lane,
    // and a lane's row is the last one started at or before it
    int row0 = -1;
    for (int base = 0; base < tot; base += 32) {
      const unsigned d = (unsigned)(start - base);
      const unsigned m = __reduce_or_sync(full, d < 32u ? 1u << d : 0u);
      const int row = row0 + __popc(m & le);
      row0 += __popc(m);
      const int kk = __shfl_sync(full, key, row), ko = __shfl_sync(full, off, row);
      const int q = base + lane;
      f(kk >> 16, ko + q, (int)(short)(kk & 0xffff), q < tot);
    }
  }
}

// The warps of a CTA take the records of a work item a few at a time:
// run(rec, rows) per chunk with the chunk's records in the warp's slots of
// shared memory (stage: kSegChunk per warp, 16-byte aligned), the next chunk
// fetched into registers before the current one is processed.  next_s: the
// item's shared cursor, 0 at the start.  Small items are dealt in smaller
// chunks, so that every warp gets several (an item's end waits for its last
// warp).
template <class Run>
__device__ __forceinline__ void seg_for_each_chunk(const SegRec* __restrict__ recs, int count, SegRec* stage,
                                                   int* next_s, Run&& run) {
  const int lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5;
  const int step = count >= nwarps * kSegChunk * 4 ? kSegChunk : (count >= nwarps * 8 ? 4 : 2);
  SegRec* slots = stage + (threadIdx.x >> 5) * kSegChunk;
  auto take = [&]() {
    int j = 0;
    if (lane == 0) j = atomicAdd(next_s, step);
    return __shfl_sync(0xffffffffu, j, 0);
  };
  // lane l holds word l of the chunk (two words a record)
  auto fetch = [&](int j) {
    return lane < 2 * step && j + (lane >> 1) < count ? __ldg(reinterpret_cast<const float4*>(recs + j) + lane)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  int j = take();
  float4 w = fetch(j);
  while (j < count) {
    const int jn = take();
    const float4 wn = fetch(jn);
    __syncwarp();  // the previous chunk is done with the slots
    if (lane < 2 * kSegChunk) reinterpret_cast<float4*>(slots)[lane] = w;
    const int rows = __shfl_sync(0xffffffffu, __float_as_int(w.w), 2 * lane + 1 < 32 ? 2 * lane + 1 : 0);
    __syncwarp();
    run(slots, lane < kSegChunk ? rows : 0);
    j = jn;
    w = wn;
  }
}

// Shared memory of the record slots.
inline size_t seg_stage_bytes(int threads) { return sizeof(SegRec) * kSegChunk * (size_t)(threads / 32); }

}  // namespace gtomrln
