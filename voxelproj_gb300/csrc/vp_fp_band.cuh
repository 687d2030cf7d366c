// Per-warp body of the z_order 0 forward projection in banded form.
//
// On one major line a run of 4 bins sees a window of neighbouring voxels of
// the minor axis, and bin b of the run (bins taken in the window's order)
// only a band of them that starts at a fixed place:
//   narrow angles, (2 b + 1) / |minor step| <= 2.9:  voxels b .. b + 3 of 7
//   the rest (to 45 degrees):  5 voxels of 9 from 0, 1, 3, 4
// where the window starts 1 (2) voxels before the one nearest to the first
// bin.  With s = 1 / |minor step|, hw = (b + 1/2) s the half-width of a bin's
// support in voxels and n0 the nearest voxel, bin k's voxels lie in
// n0 + (k s - hw - 1/2, k s + hw + 1/2); the bands hold these intervals for
// every angle, with 0.05 voxels to spare.  So a line is straight-line code:
// load the window, multiply 16 (20) weights, no branch per voxel and every
// register index static.  Weights outside a voxel's three bins are zero.
//
// G runs per warp: 32 / G lanes x 4 heights each, so that few heights still
// fill the warp.  The warp computes the weights of 32 (line, run) pairs at a
// time, one per lane, into a shared table.
//
// Per bin the voxels are added in the order of the candidate lists
// (vp_fp_z0.cuh) with the same weights, so the sums are equal bit for bit.
// A zero weight times an infinite voxel would spread it to bins that do not
// see it: a warp whose sums are not all finite repeats its runs with the
// candidate lists (without their zero weights where g.skip_zero).
#pragma once

#include "vp_common.cuh"
#include "vp_fp_z0.cuh"

namespace vp {
namespace detail {

constexpr int FPB_WARPS = 4;
constexpr float kBandNarrow = 2.9f;

struct BandEntry {
  float4 w[5];  // narrow: 4 bands of 4; wide: 4 bands of 5
  int4 meta;    // voxel index of the window's first voxel, its minor index, kind
};
enum : int { BAND_EMPTY = 0, BAND_INSIDE = 1, BAND_EDGE = 2 };

template <bool NARROW>
struct Band {
  static constexpr int T = NARROW ? 4 : 5;       // voxels per bin
  static constexpr int W = NARROW ? 7 : 9;       // voxels per window
  static constexpr int before = NARROW ? 1 : 2;  // window start before the nearest voxel
  static __host__ __device__ constexpr int start(int b) { return NARROW || b < 2 ? b : b + 1; }
};

// One warp's table, or its candidate list on the repeat.
union BandSmem {
  BandEntry tab[32];
  float4 cand[Fp0Cap<4>::list];
};

struct BandAngle {
  AngleConst k;
  bool minor_x;
  int maj_lo, maj_hi, min_lo, min_hi;  // the slab's lines and voxels (min_hi inclusive)
  float cent_major, cent_minor, sh_major, inv;
  bool up;  // bins ascend with the minor axis
};

// The table entry of line i and the run at bin p0.
template <bool NARROW>
__device__ __forceinline__ void band_entry(const BandAngle& A, const Geom& g, int i, int p0,
                                           BandEntry* e) {
  using B = Band<NARROW>;
  const int first_bin = A.up ? p0 : p0 + 3;
  const float u0 = ((float)first_bin - (((float)i - A.cent_major) * A.sh_major + g.pcent)) * A.inv +
                   A.cent_minor;
  const int m0 = __float2int_rn(u0) - B::before;
  float w[4][B::T];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int t = 0; t < B::T; ++t) w[b][t] = 0.0f;
#pragma unroll
  for (int u = 0; u < B::W; ++u) {
    const float rel_minor = (float)(m0 + u) - A.cent_minor;
    const float rel_major = (float)i - A.cent_major;
    const BinWeights bw = voxel_weights(A.minor_x ? rel_minor : rel_major,
                                        A.minor_x ? rel_major : rel_minor, A.k, g.pcent, g.trig);
    // bin b's distance from round(xp), in the window's order
    const int q = A.up ? bw.r - p0 : p0 + 3 - bw.r;
    const float wl = A.up ? bw.w0 : bw.w2, wr = A.up ? bw.w2 : bw.w0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int t = u - B::start(b);
      if (t >= 0 && t < B::T)
        w[b][t] = q == b ? bw.w1 : q == b + 1 ? wl : q == b - 1 ? wr : 0.0f;
    }
  }
  const float* ws = &w[0][0];
#pragma unroll
  for (int j = 0; j < B::T; ++j)
    e->w[j] = make_float4(ws[4 * j], ws[4 * j + 1], ws[4 * j + 2], ws[4 * j + 3]);
  const bool some = m0 <= A.min_hi && m0 + B::W - 1 >= A.min_lo;
  const bool inside = m0 >= A.min_lo && m0 + B::W - 1 <= A.min_hi;
  e->meta = make_int4(A.minor_x ? i * g.SX + m0 : m0 * g.SX + i, m0,
                      !some ? BAND_EMPTY : inside ? BAND_INSIDE : BAND_EDGE, 0);
}

// With G runs per warp a run has 32 / G lanes of 4 heights; lanes left over
// (G = 3) follow the last run and hold no heights.
template <int G>
__device__ __forceinline__ int band_run(int lane) {
  return G == 1 ? 0 : min(lane / (32 / G), G - 1);
}
template <int G>
__device__ __forceinline__ int band_height(int lane) {
  constexpr int LH = 32 / G;
  return lane < G * LH ? (lane % LH) * 4 : 1 << 29;
}

// The lines [lo, hi) of the slab for G runs from bin 4 * run0.
template <int G, bool NARROW>
__device__ __forceinline__ void band_lines(float4 (&acc)[4], const float* xs, const BandAngle& A,
                                           const Geom& g, int run0, int lo, int hi,
                                           BandEntry* tab) {
  using B = Band<NARROW>;
  constexpr int LB = 32 / G;  // lines per table
  const int lane = threadIdx.x & 31;
  const BandEntry* mine = tab + band_run<G>(lane);
  const ptrdiff_t sm = (ptrdiff_t)(A.minor_x ? 1 : g.SX) * g.Hx;  // one voxel along the minor axis
  for (int i0 = lo; i0 < hi; i0 += LB) {
    __syncwarp();
    if (lane < LB * G && i0 + lane / G < hi)
      band_entry<NARROW>(A, g, i0 + lane / G, 4 * (run0 + lane % G), &tab[lane]);
    __syncwarp();
    const int nl = min(LB, hi - i0);
    for (int l = 0; l < nl; ++l) {
      const BandEntry& e = mine[l * G];
      const int4 meta = e.meta;
      if (G == 1 && meta.z == BAND_EMPTY) continue;  // warp-uniform
      const float* p = xs + (ptrdiff_t)meta.x * g.Hx;
      float4 win[B::W];
      if (G == 1 ? meta.z == BAND_INSIDE : __all_sync(0xffffffffu, meta.z == BAND_INSIDE)) {
#pragma unroll
        for (int u = 0; u < B::W; ++u) win[u] = __ldg(reinterpret_cast<const float4*>(p + u * sm));
      } else {
#pragma unroll
        for (int u = 0; u < B::W; ++u) {
          const int m = meta.y + u;
          win[u] = ld_or_zero<float4>(p + u * sm, m >= A.min_lo && m <= A.min_hi);
        }
      }
      float ws[4 * B::T];
#pragma unroll
      for (int j = 0; j < B::T; ++j) {
        const float4 v = e.w[j];
        ws[4 * j] = v.x;
        ws[4 * j + 1] = v.y;
        ws[4 * j + 2] = v.z;
        ws[4 * j + 3] = v.w;
      }
#pragma unroll
      for (int u = 0; u < B::W; ++u)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int t = u - B::start(b);
          if (t >= 0 && t < B::T) acc[b] = f4_fma(ws[b * B::T + t], win[u], acc[b]);
        }
    }
  }
}

// True in a lane whose sums, those of its heights below n, are not all finite.
__device__ __forceinline__ bool not_finite(const float4 (&acc)[4], int n) {
  float4 s = vzero<float4>();
#pragma unroll
  for (int b = 0; b < 4; ++b) s = f4_fma(0.0f, acc[b], s);
  const float t = ((n > 0 ? s.x : 0.0f) + (n > 1 ? s.y : 0.0f)) +
                  ((n > 2 ? s.z : 0.0f) + (n > 3 ? s.w : 0.0f));
  return t != t;
}

__device__ __forceinline__ BandAngle band_angle(const AngleConst& k, const Geom& g,
                                                const Slab& s) {
  BandAngle A;
  A.k = k;
  A.minor_x = fabsf(k.c) >= fabsf(k.s);
  A.maj_lo = A.minor_x ? s.y_lo : s.x_lo;
  A.maj_hi = A.minor_x ? s.y_hi : s.x_hi;
  A.min_lo = A.minor_x ? 0 : s.yy_lo;
  A.min_hi = A.minor_x ? g.SX - 1 : s.yy_hi - 1;
  A.cent_major = A.minor_x ? g.ycent : g.xcent;
  A.cent_minor = A.minor_x ? g.xcent : g.ycent;
  A.sh_major = A.minor_x ? k.s : k.c;
  const float step = A.minor_x ? k.c : k.s;
  A.inv = 1.0f / step;
  A.up = step >= 0.0f;
  return A;
}

// Cuts [lo, hi) to the lines on which a window of the G runs from run0 can meet
// the slab's voxels; the others add nothing.  On line i bin q has its centre at
// minor coordinate c(q) - s (i - cent_major); 3 voxels are kept beyond the
// windows, far above the rounding of either side.
// Where the detector is wider than the volume, or the volume longer than broad,
// many runs see few lines: A (40, 300, 48) with 240 angles and 450 bins 460 us
// with all lines, candidate lists 287, 168 with this.
template <int G>
__device__ __forceinline__ void band_clip(const BandAngle& A, const Geom& g, int run0, int* lo,
                                          int* hi) {
  constexpr float kBelow = (float)Band<false>::W + 3.0f, kAbove = (float)Band<false>::before + 3.0f;
  const float s = A.sh_major * A.inv;
  if (!(fabsf(s) > 1e-6f)) return;  // no line differs from the next (or NaN)
  const float qa = (float)(4 * run0), qb = qa + (float)(4 * G - 1);
  const float ca = (qa - g.pcent) * A.inv + A.cent_minor, cb = (qb - g.pcent) * A.inv + A.cent_minor;
  const float u = (fmaxf(ca, cb) - ((float)A.min_lo - kBelow)) / s;
  const float v = (fminf(ca, cb) - ((float)A.min_hi + kAbove)) / s;
  const float first = floorf(fminf(u, v) + A.cent_major), last = ceilf(fmaxf(u, v) + A.cent_major);
  *lo = min(max(*lo, (int)fmaxf(first, -1.0f)), *hi);
  *hi = max(*lo, (int)fminf((float)*hi, last + 1.0f));
}

// The sums of G runs from run0 on the lines [lo, hi).
template <int G>
__device__ __forceinline__ void band_sums(float4 (&acc)[4], const float* xs, const BandAngle& A,
                                          const Geom& g, int run0, int lo, int hi,
                                          BandEntry* tab) {
#pragma unroll
  for (int b = 0; b < 4; ++b) acc[b] = vzero<float4>();
  if ((2.0f * A.k.b + 1.0f) * fabsf(A.inv) <= kBandNarrow)
    band_lines<G, true>(acc, xs, A, g, run0, lo, hi, tab);
  else
    band_lines<G, false>(acc, xs, A, g, run0, lo, hi, tab);
}

// Adds or stores the sums of G runs from run0 on (over the lines [lo, hi)), by the
// whole warp, after wait(); h: this lane's heights (several runs: of the one
// chunk).
template <int G, class Wait, bool VOUT>
__device__ __forceinline__ void band_write(const float4 (&acc)[4], const float* x, float* y,
                                           const float* angles, const Geom& g, const Slab& s,
                                           const BandAngle& A, int lo, int hi, int run0, int a,
                                           int h, int accumulate, float4* cand,
                                           const Wait& wait) {
  wait();
  if (lo >= hi && accumulate) return;
  const int lane = threadIdx.x & 31;
  if (__any_sync(0xffffffffu, not_finite(acc, g.H - h))) {
    Slab part = s;
    (A.minor_x ? part.y_lo : part.x_lo) = lo;
    (A.minor_x ? part.y_hi : part.x_hi) = hi;
    for (int r = 0; r < G; ++r) {
      __syncwarp();
      fp_z0_warp<4, 4, 2, Wait, false, VOUT, true>(x, y, angles, g, 4 * (run0 + r), a,
                                                   G > 1 ? 4 * lane : h, part, accumulate, cand,
                                                   wait);
    }
    return;
  }
  const LaneH<4> lh(h, g.H);
  const int p0 = 4 * (run0 + band_run<G>(lane));
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const int p = A.up ? p0 + b : p0 + 3 - b;
    if (p < g.PX) {
      float* row = y + ((size_t)a * g.PX + p) * g.Hy;
      if constexpr (VOUT) store_lane<4, Wait::coherent>(row, lh, acc[b], accumulate);
      else store_lane_heights<4, Wait::coherent>(row, lh, acc[b], accumulate, g.H);
    }
  }
}

// Block body.  A warp takes G runs of 4 bins (from run0) of angle a and its
// lanes' heights from h, on the slab's lines; with SP warps per run set, warp
// `part` takes every SP-th share of the lines and part 0 writes the sum of all
// (sums: FPB_WARPS x 32 x 4 vectors of shared memory, where partial sums of
// `lines` lines gather too; with one warp they are added into y).  has: this warp
// has work (all warps of a block must call, with SP = 4 with the same runs).
template <int G, int SP, class Wait, bool VOUT>
__device__ __forceinline__ void fp_band_block(const float* __restrict__ x, float* __restrict__ y,
                                              const float* __restrict__ angles, const Geom& g,
                                              int run0, int a, int h, const Slab& s, bool has,
                                              int part, int lines, int accumulate, BandSmem* sm,
                                              float4 (*sums)[32][4]) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const Wait wait;
  if (!has) {  // (with SP = 4: the whole block)
    wait();
    return;
  }
  const float* xs = x + (h < g.H ? h : 0);
  float4 acc[4];
  const BandAngle A = band_angle(angle_const(__ldg(angles + a), g.trig), g, s);
  int lo = A.maj_lo, hi = A.maj_hi;
  band_clip<G>(A, g, run0, &lo, &hi);
  if constexpr (SP == 1) {
    for (;;) {
      const int end = min(lo + lines, hi);
      band_sums<G>(acc, xs, A, g, run0, lo, end, sm->tab);
      band_write<G, Wait, VOUT>(acc, x, y, angles, g, s, A, lo, end, run0, a, h, accumulate,
                                sm->cand, wait);
      if (end >= hi) return;
      lo = end;
      accumulate = 1;
    }
  } else {
    const int all_lo = lo, all_hi = hi, share = (hi - lo + SP - 1) / SP;
    lo = min(lo + part * share, hi);
    hi = min(lo + share, hi);
    float4* mine = sums[warp][lane];
    for (bool first = true;; first = false) {
      const int end = min(lo + lines, hi);
      band_sums<G>(acc, xs, A, g, run0, lo, end, sm->tab);
      if (!first) {
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[b] = f4_add(mine[b], acc[b]);
      }
      if (end >= hi) break;
#pragma unroll
      for (int b = 0; b < 4; ++b) mine[b] = acc[b];
      lo = end;
    }
    if (part > 0)
#pragma unroll
      for (int b = 0; b < 4; ++b) mine[b] = acc[b];
    __syncthreads();
    if (part > 0) {
      wait();
      return;
    }
#pragma unroll
    for (int j = 1; j < SP; ++j)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[b] = f4_add(acc[b], sums[warp + j][lane][b]);
    band_write<G, Wait, VOUT>(acc, x, y, angles, g, s, A, all_lo, all_hi, run0, a, h, accumulate,
                              sm->cand, wait);
  }
}

// One warp of a batch: as fp_band_block without a split, in one sum (a batch's
// slabs are those of the candidate lists).
template <int G, class Wait>
__device__ __forceinline__ void fp_band_warp(const float* __restrict__ x, float* __restrict__ y,
                                             const float* __restrict__ angles, const Geom& g,
                                             int run0, int a, int h, const Slab& s,
                                             BandSmem* sm, const Wait& wait) {
  if (a >= g.n_ang || 4 * run0 >= g.PX) {  // warp-uniform
    wait();
    return;
  }
  float4 acc[4];
  const BandAngle A = band_angle(angle_const(__ldg(angles + a), g.trig), g, s);
  int lo = A.maj_lo, hi = A.maj_hi;
  band_clip<G>(A, g, run0, &lo, &hi);
  band_sums<G>(acc, x + (h < g.H ? h : 0), A, g, run0, lo, hi, sm->tab);
  __syncwarp();
  band_write<G, Wait, true>(acc, x, y, angles, g, s, A, lo, hi, run0, a, h, 1, sm->cand, wait);
}

}  // namespace detail
}  // namespace vp
