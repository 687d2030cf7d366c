// Projections of few heights: z_order 2 below 32 heights, z_order 0 up to 8.
//
// The other kernels put heights across the lanes of a warp and pay for each
// weight once per 128 or 256 heights.  With few heights the weights are the
// cost, so here a lane owns one bin (forward) or one voxel (adjoint) and RH
// heights, and the weights come from shortened forms of the trapezoid's CDF:
// with tail(m) the area beyond m >= 0 of the footprint, F(-m) = tail(m),
//   adjoint, r = round(xp), xv = r - xp:  w0 = tail(1/2 - xv),
//     w2 = tail(1/2 + xv), w1 = 1 - w0 - w2        (bins r - 1, r + 1, r)
//   forward: the tails of the voxels that an edge between bins cuts, from
//     which the weights of the bins on its two sides differ.
// They are the same piecewise quadratics as trap_cdf (vp_common.cuh), term by
// term on the side of the footprint where they are needed: about 30
// instructions for the adjoint's three weights.
//
// What bounds them: instruction issue (one slice moves a few MB).
#include <cuda_runtime.h>

#include <cstdint>

#include "vp_common.cuh"
#include "vp_launch.h"

namespace vp {

namespace {

constexpr int kMaxGridYZ = 65535;
constexpr int THIN_WARPS = 4;
constexpr int THIN_BINS = 31;  // bins per warp of the forward

// Element strides of the volume and the sinogram: (height, voxel) and
// (height, bin).
struct ThinStrides {
  long long xh, xv, yh, yb;
};

// Area of the footprint beyond m >= 0.  (b - m <= b < 1: the clamp at 0 is the
// add's saturation.)
__device__ __forceinline__ float tail_area(float m, const AngleConst& k) {
  const float e = __saturatef(k.b - m);
  return m < k.a ? fmaf(-2.0f * k.coeff, m, 0.5f) : (k.cd * e) * e;
}

// p - xp of a voxel for a bin at fp.  MX: x is the minor axis.
template <bool MX, int TRIG>
__device__ __forceinline__ float bin_distance(float fp, float rel_minor, float rel_major,
                                              const AngleConst& k, float pcent) {
  const float relx = MX ? rel_minor : rel_major, rely = MX ? rel_major : rel_minor;
  if (TRIG == TRIG_PRECISE) {
    float xv;
    const int r = compensated_offset(relx, rely, k, pcent, &xv);  // r - xp
    return (fp - (float)r) + xv;
  }
  return fp - det_coord(relx, rely, k.c, k.s, pcent);
}

// ---------------------------------------------------------------------------
// Forward.  A warp owns 31 neighbouring bins of one angle and a quarter of
// the major lines; the four warps of a block add up their sums in shared
// memory.  The lines come in chunks of LC: the piece of the volume that the
// warp's bins see on them (at most 31 sqrt(2) + LC + 7 voxels along the minor
// axis) is read row by row, whichever axis is the minor one, into a shared
// tile, line-major.  A lane evaluates one edge between bins, which cuts two
// voxels per line; its bin's other edge comes from the lane below, and with
// it the bin's four weights.
//
// 512 x 512, 360 angles: one slice 1838 -> 279 us, 4 slices 2239 -> 564 us
// (the kernel before took the voxels straight from global memory: 32 cache
// lines per load where y is the minor axis, one wave of warps that each waited
// for every line's loads in turn).  With both edges of the bin evaluated for
// each of its 3 or 4 voxels, on 32 bins per warp: 315 and 594 us.  One slice
// issues in 80% of the cycles.
// ---------------------------------------------------------------------------
template <int LC>
struct ThinTile {
  static constexpr int W = (45 + LC + 7) | 1;  // odd pitch: column writes hit all banks
};

// UT elements of the tile: lines l .. l + UT - 1 of voxel m (LINES), or voxels m,
// m + 32 / LC, .. of line l; every load is issued before the first store.
template <int RH, int LC, int UT, bool LINES>
__device__ __forceinline__ void tile_load(float (*tl)[LC][ThinTile<LC>::W], const float* corner,
                                          int l, int m, int bound, bool in, int nh,
                                          long long s_h, long long s_maj, long long s_min,
                                          int m0 = 0, int n_minor = 0) {
  float v[UT][RH];
#pragma unroll
  for (int u = 0; u < UT; ++u) {
    const int lu = LINES ? l + u : l;
    const int mu = LINES ? m : m + u * (32 / LC);
    const bool ok = in && (LINES ? lu : mu) < bound &&
                    (LINES || (unsigned)(m0 + mu) < (unsigned)n_minor);
    const float* q = corner + lu * s_maj + mu * s_min;
#pragma unroll
    for (int h = 0; h < RH; ++h) v[u][h] = ok && h < nh ? __ldg(q + h * s_h) : 0.0f;
  }
#pragma unroll
  for (int u = 0; u < UT; ++u) {
    const int lu = LINES ? l + u : l;
    const int mu = LINES ? m : m + u * (32 / LC);
    if ((LINES ? lu : mu) < bound) {
#pragma unroll
      for (int h = 0; h < RH; ++h) tl[h][lu][mu] = v[u][h];
    }
  }
}

// Minor coordinate of bin q's centre on major line i.
__device__ __forceinline__ float bin_centre(float q, int i, float cent_major, float sh_major,
                                            float inv, float cent_minor, float pcent) {
  return (q - (((float)i - cent_major) * sh_major + pcent)) * inv + cent_minor;
}

struct ThinChunk {
  int i0, nl, m0;  // lines [i0, i0 + nl), the tile's first voxel
  float cent_major, cent_minor, sh_major, inv;
};

// This lane's bin on the lines of one chunk.  fe: the bin's edge on the side of
// larger minor coordinates; the other edge is that of the lane below.  An edge
// at minor coordinate u cuts at most the voxels m = floor(u) and m + 1: t0 of
// the first lies beyond it and t1 of the second before it.  A bin is 1 to 1.42
// voxels wide, so with m the lower edge's voxel is m - n, n = 1, 2 (or 0 by
// rounding), and four weights are left.
template <int RH, int LC, int TRIG, bool MX>
__device__ __forceinline__ void gather_lines(float (&acc)[RH],
                                             const float (*tl)[LC][ThinTile<LC>::W],
                                             const ThinChunk& c, float fe, const AngleConst& k,
                                             float pcent) {
  const float sign = c.inv > 0.0f ? 1.0f : -1.0f;
  const float u0 = bin_centre(fe, c.i0, c.cent_major, c.sh_major, c.inv, c.cent_minor, pcent);
  const float du = -c.sh_major * c.inv;
  const float base = (float)(c.m0 + 2) - c.cent_minor;
  float fl = 0.0f;
  float rel_major = (float)c.i0 - c.cent_major;
#pragma unroll 1  // (2 and 4: one slice 283 and 288 us, 1: 279)
  for (int l = 0; l < c.nl; ++l, fl += 1.0f, rel_major += 1.0f) {
    // (inside the tile, one voxel of which on either side is for rounding; the
    // minimum only bounds the index)
    const int o = (int)min((unsigned)(__float2int_rd(fmaf(fl, du, u0)) - (c.m0 + 2)),
                           (unsigned)(ThinTile<LC>::W - 4));
    const float rel = base + (float)o;
    const float z0 = sign * bin_distance<MX, TRIG>(fe, rel, rel_major, k, pcent);
    const float z1 = sign * bin_distance<MX, TRIG>(fe, rel + 1.0f, rel_major, k, pcent);
    const float t0 = tail_area(z0, k), t1 = tail_area(-z1, k);
    const float s0 = __shfl_up_sync(0xffffffffu, t0, 1);
    const float s1 = __shfl_up_sync(0xffffffffu, t1, 1);
    const int n = o - __shfl_up_sync(0xffffffffu, o, 1);
    const float w[4] = {n >= 2 ? s0 : 0.0f,
                        n >= 2 ? 1.0f - s1 : n == 1 ? s0 : 0.0f,
                        (1.0f - t0) - (n >= 2 ? 0.0f : n == 1 ? s1 : 1.0f - s0),
                        t1 - (n >= 1 ? 0.0f : s1)};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (w[t] != 0.0f) {  // (a voxel that the bin does not see adds nothing, whatever it holds)
#pragma unroll
        for (int h = 0; h < RH; ++h) acc[h] = fmaf(w[t], tl[h][l][o + t], acc[h]);
      }
    }
  }
}

template <int RH, int LC, int TRIG>
__global__ void __launch_bounds__(32 * THIN_WARPS)
    fp_thin_kernel(const float* __restrict__ x, float* __restrict__ y,
                   const float* __restrict__ angles, Geom g, ThinStrides st, int a_base) {
  constexpr int W = ThinTile<LC>::W;
  __shared__ float tile[THIN_WARPS][RH][LC][W];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int a = a_base + blockIdx.y;
  const int h0 = blockIdx.z * RH;
  const int nh = min(RH, g.H - h0);

  const AngleConst k = angle_const(__ldg(angles + a), TRIG);
  const bool minor_x = fabsf(k.c) >= fabsf(k.s);
  const int n_major = minor_x ? g.SY : g.SX;
  const int n_minor = minor_x ? g.SX : g.SY;
  const float cent_major = minor_x ? g.ycent : g.xcent;
  const float cent_minor = minor_x ? g.xcent : g.ycent;
  const float sh_major = minor_x ? k.s : k.c;
  const float inv = 1.0f / (minor_x ? k.c : k.s);
  // lanes 1 .. 31 own bins, in the order of their minor coordinates
  const int p0 = blockIdx.x * THIN_BINS;
  const int p = inv > 0.0f ? p0 + lane - 1 : p0 + THIN_BINS - lane;
  const float fe = (float)p + (inv > 0.0f ? 0.5f : -0.5f);
  const long long s_maj = minor_x ? (long long)g.SX * st.xv : st.xv;
  const long long s_min = minor_x ? st.xv : (long long)g.SX * st.xv;
  const float* xs = x + h0 * st.xh;
  float(*tl)[LC][W] = tile[warp];

  // With 4 heights and more each chunk of lines has a sum of its own: an accumulator
  // that runs over a quarter of all lines had 1.2 times the error of the candidate
  // lists' slabs (A (500, 512, 4), 50 angles, precise).  Fewer heights replaced kernels
  // with one sum over all lines (one slice 278.4 us, 279.8 with a sum per chunk).
  constexpr bool kParts = RH >= 4;
  float acc[RH];
#pragma unroll
  for (int h = 0; h < RH; ++h) acc[h] = 0.0f;

  const auto centre = [&](float q, int i) {
    return bin_centre(q, i, cent_major, sh_major, inv, cent_minor, g.pcent);
  };

  for (int i0 = warp * LC; i0 < n_major; i0 += THIN_WARPS * LC) {
    // the chunk's voxels along the minor axis: [m0, m0 + nm)
    const float q0 = (float)p0 - 0.5f, q1 = q0 + (float)THIN_BINS;
    const int i1 = min(i0 + LC, n_major) - 1;
    const float ua = centre(q0, i0), ub = centre(q1, i0), uc = centre(q0, i1), ud = centre(q1, i1);
    const int m0 = (int)floorf(fminf(fminf(ua, ub), fminf(uc, ud))) - 3;
    const int m1 = min(m0 + W, (int)ceilf(fmaxf(fmaxf(ua, ub), fmaxf(uc, ud))) + 3);
    if (m1 <= 0 || m0 >= n_minor) continue;  // warp-uniform
    const int nl = i1 - i0 + 1;
    const int nm = m1 - m0;
    __syncwarp();  // the chunk before is done with
    // UT tile elements per lane in flight; a lane's elements are UT lines of one
    // voxel of the minor axis, or UT voxels of one line
    constexpr int UT = RH >= 8 ? 1 : LC / RH < 8 ? LC / RH : 8;
    const float* corner = xs + i0 * s_maj + m0 * s_min;
    if (minor_x) {
      for (int m = lane; m < nm; m += 32) {
        const bool in = (unsigned)(m0 + m) < (unsigned)n_minor;
        for (int l = 0; l < nl; l += UT) tile_load<RH, LC, UT, true>(tl, corner, l, m, nl, in, nh, st.xh, s_maj, s_min);
      }
    } else {
      const int l = lane % LC;
      for (int m = lane / LC; m < nm; m += UT * (32 / LC))
        tile_load<RH, LC, UT, false>(tl, corner, l, m, nm, l < nl, nh, st.xh, s_maj, s_min, m0, n_minor);
    }
    __syncwarp();
    const ThinChunk c{i0, nl, m0, cent_major, cent_minor, sh_major, inv};
    float sum[RH];
#pragma unroll
    for (int h = 0; h < RH; ++h) sum[h] = kParts ? 0.0f : acc[h];
    if (minor_x) gather_lines<RH, LC, TRIG, true>(sum, tl, c, fe, k, g.pcent);
    else gather_lines<RH, LC, TRIG, false>(sum, tl, c, fe, k, g.pcent);
#pragma unroll
    for (int h = 0; h < RH; ++h) acc[h] = kParts ? acc[h] + sum[h] : sum[h];
  }

  // the block's four sums
  __syncthreads();
  float* sums = &tile[0][0][0][0];
#pragma unroll
  for (int h = 0; h < RH; ++h) sums[(warp * RH + h) * 32 + lane] = acc[h];
  __syncthreads();
  if (lane == 0 || p >= g.PX) return;
  for (int h = warp; h < nh; h += THIN_WARPS) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < THIN_WARPS; ++w) v += sums[(w * RH + h) * 32 + lane];
    store_out(y + (h0 + h) * st.yh + ((long long)a * g.PX + p) * st.yb, v, g.accumulate);
  }
}

// ---------------------------------------------------------------------------
// Adjoint.  A lane owns VR voxels, neighbours along y, of 32 columns; the
// angles' constants come from a per-warp shared table, at most 32 angles at a
// time.  With SPLIT the four warps of a block take the same voxels and a quarter
// of the angles each and add up in shared memory (small volumes: enough warps to
// fill the GPU); else neighbouring rows.  Z2: bins are contiguous, else heights.
// 512 x 512, 360 angles: one slice 304 -> 137 us, 8 slices 932 -> 554 us.  One
// slice issues in 75% of the cycles.  With tables of 32 angles whatever their
// number, the first warp had all of up to 32 angles: 256 x 256 x 8 and 30 angles
// 83 us, 24 with equal shares; 24 x 24 x 16 58 and 14.
// ---------------------------------------------------------------------------
template <int RH, int VR, bool SPLIT, bool Z2, int TRIG>
__global__ void __launch_bounds__(32 * THIN_WARPS)
    bp_thin_kernel(const float* __restrict__ y, float* __restrict__ x,
                   const float* __restrict__ angles, Geom g, ThinStrides st) {
  struct Entry {
    float4 w;   // a, b, coeff, cd
    float2 cs;
  };
  __shared__ Entry tab[THIN_WARPS][32];
  __shared__ float sums[SPLIT ? THIN_WARPS : 1][VR][RH][32];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int xi = blockIdx.x * 32 + lane;
  const int yi = (SPLIT ? blockIdx.y : blockIdx.y * THIN_WARPS + warp) * VR;
  const int h0 = blockIdx.z * RH;
  const int nh = min(RH, g.H - h0);
  const long long yb = Z2 ? 1 : st.yb, yh = Z2 ? st.yh : 1;
  const float relx = (float)xi - g.xcent;

  float acc[VR][RH];
#pragma unroll
  for (int v = 0; v < VR; ++v)
#pragma unroll
    for (int h = 0; h < RH; ++h) acc[v][h] = 0.0f;

  // angles per table: with SPLIT as many as give the four warps equal shares
  constexpr int kMost = 32 * (SPLIT ? THIN_WARPS : 1);
  const int rounds = (g.n_ang + kMost - 1) / kMost;
  const int at = SPLIT ? (g.n_ang + rounds * THIN_WARPS - 1) / (rounds * THIN_WARPS) : 32;
  const int step = SPLIT ? at * THIN_WARPS : 32;
  for (int a0 = SPLIT ? at * warp : 0; a0 < g.n_ang; a0 += step) {
    __syncwarp();
    if (lane < at && a0 + lane < g.n_ang) {
      const AngleConst k = angle_const(__ldg(angles + a0 + lane), TRIG);
      tab[warp][lane] = Entry{make_float4(k.a, k.b, k.coeff, k.cd), make_float2(k.c, k.s)};
    }
    __syncwarp();
    const int na = min(at, g.n_ang - a0);
    const float* ya = y + h0 * yh + (long long)a0 * g.PX * yb;
    for (int j = 0; j < na; ++j, ya += g.PX * yb) {
      const Entry& e = tab[warp][j];
      const float4 w = e.w;
      const float2 cs = e.cs;
      AngleConst k;
      k.c = cs.x;
      k.s = cs.y;
      k.a = w.x;
      k.b = w.y;
      k.coeff = w.z;
      k.cd = w.w;
#pragma unroll
      for (int v = 0; v < VR; ++v) {
        const float rely = (float)(yi + v) - g.ycent;
        float xv;
        const int r = voxel_offset(relx, rely, k, g.pcent, TRIG, &xv);
        const float w0 = tail_area(0.5f - xv, k);
        const float w2 = tail_area(0.5f + xv, k);
        const float w1 = (1.0f - w0) - w2;
        const float* q = ya + r * yb;
        if (RH > 1 && __all_sync(0xffffffffu, r >= 1 && r + 1 < g.PX)) {
          // every lane's three bins on the detector: loads without the zeros and
          // selects of the guarded ones (8 heights 652 -> 554 us below; one
          // height 137 -> 148, so not there)
#pragma unroll
          for (int h = 0; h < RH; ++h) {
            if (h < nh) {
              acc[v][h] = fmaf(w0, __ldg(q - yb), acc[v][h]);
              acc[v][h] = fmaf(w1, __ldg(q), acc[v][h]);
              acc[v][h] = fmaf(w2, __ldg(q + yb), acc[v][h]);
              q += yh;
            }
          }
        } else {
          const bool ok0 = (unsigned)(r - 1) < (unsigned)g.PX;
          const bool ok1 = (unsigned)r < (unsigned)g.PX;
          const bool ok2 = (unsigned)(r + 1) < (unsigned)g.PX;
#pragma unroll
          for (int h = 0; h < RH; ++h) {
            if (h < nh) {
              const float v0 = ok0 ? __ldg(q - yb) : 0.0f;
              const float v1 = ok1 ? __ldg(q) : 0.0f;
              const float v2 = ok2 ? __ldg(q + yb) : 0.0f;
              acc[v][h] = fmaf(w0, v0, acc[v][h]);
              acc[v][h] = fmaf(w1, v1, acc[v][h]);
              acc[v][h] = fmaf(w2, v2, acc[v][h]);
              q += yh;
            }
          }
        }
      }
    }
  }

  float* out = x + h0 * st.xh + ((long long)yi * g.SX + xi) * st.xv;
  if constexpr (SPLIT) {
#pragma unroll
    for (int v = 0; v < VR; ++v)
#pragma unroll
      for (int h = 0; h < RH; ++h) sums[warp][v][h][lane] = acc[v][h];
    __syncthreads();
    if (xi >= g.SX) return;
    for (int i = warp; i < VR * nh; i += THIN_WARPS) {
      const int v = i / nh, h = i - v * nh;
      if (yi + v >= g.SY) continue;
      float t = 0.0f;
#pragma unroll
      for (int w = 0; w < THIN_WARPS; ++w) t += sums[w][v][h][lane];
      store_out(out + v * g.SX * st.xv + h * st.xh, t, g.accumulate);
    }
  } else {
    if (xi >= g.SX) return;
#pragma unroll
    for (int v = 0; v < VR; ++v) {
      if (yi + v >= g.SY) continue;
#pragma unroll
      for (int h = 0; h < RH; ++h)
        if (h < nh) store_out(out + v * g.SX * st.xv + h * st.xh, acc[v][h], g.accumulate);
    }
  }
}

inline unsigned ceil_div(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

ThinStrides thin_strides(const Geom& g, int z) {
  if (z == 2)
    return {(long long)g.SY * g.SX, 1, (long long)g.n_ang * g.PX, 1};
  return {1, g.Hx, 1, g.Hy};
}

template <int RH, int LC>
cudaError_t launch_fp(const float* x, float* y, const float* angles, const Geom& g, int z,
                      cudaStream_t stream) {
  for (int a = 0; a < g.n_ang; a += kMaxGridYZ) {
    const dim3 grid(ceil_div(g.PX, THIN_BINS), g.n_ang - a < kMaxGridYZ ? g.n_ang - a : kMaxGridYZ,
                    ceil_div(g.H, RH));
    if (g.trig == TRIG_PRECISE)
      fp_thin_kernel<RH, LC, TRIG_PRECISE><<<grid, 32 * THIN_WARPS, 0, stream>>>(
          x, y, angles, g, thin_strides(g, z), a);
    else
      fp_thin_kernel<RH, LC, TRIG_REF><<<grid, 32 * THIN_WARPS, 0, stream>>>(
          x, y, angles, g, thin_strides(g, z), a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Blocks of 4 warps below which the adjoint splits the angles over them
// (152 SMs, about 12 resident blocks each).  From 8 angles on: with fewer a
// quarter of them saves less than the sum over the warps costs.
constexpr long long kSplitRows = 4096;
constexpr long long kFourVoxels = 4096;  // rows of 32 voxels per slice

template <int RH, int VR, bool Z2>
cudaError_t launch_bp(const float* y, float* x, const float* angles, const Geom& g, int z,
                      cudaStream_t stream) {
  const long long rows = ceil_div(g.SY, VR);
  const long long warps = (long long)ceil_div(g.SX, 32) * rows * ceil_div(g.H, RH);
  const ThinStrides st = thin_strides(g, z);
  const bool split = warps < kSplitRows && rows <= kMaxGridYZ && g.n_ang >= 2 * THIN_WARPS;
  const dim3 grid(ceil_div(g.SX, 32), split ? (unsigned)rows : ceil_div(rows, THIN_WARPS),
                  ceil_div(g.H, RH));
  const auto kernel = g.trig == TRIG_PRECISE
                          ? (split ? bp_thin_kernel<RH, VR, true, Z2, TRIG_PRECISE>
                                   : bp_thin_kernel<RH, VR, false, Z2, TRIG_PRECISE>)
                          : (split ? bp_thin_kernel<RH, VR, true, Z2, TRIG_REF>
                                   : bp_thin_kernel<RH, VR, false, Z2, TRIG_REF>);
  kernel<<<grid, 32 * THIN_WARPS, 0, stream>>>(y, x, angles, g, st);
  return cudaGetLastError();
}

template <bool Z2>
cudaError_t launch_bp_z(const float* y, float* x, const float* angles, const Geom& g, int z,
                        cudaStream_t stream) {
  // four voxels per lane share an angle's constants where that leaves enough
  // warps; 512 x 512, 360 angles: one slice 209 us with one, 177 with two, 152
  // with four; 64 x 64, 60 angles: 12 us with one, 20 with four; 384 x 384 x 4 and
  // 2 angles 10.4 with one, 13.7 with four
  const bool four = (long long)ceil_div(g.SX, 32) * g.SY >= kFourVoxels && g.n_ang >= 8;
  if (g.H == 1)
    return four ? launch_bp<1, 4, Z2>(y, x, angles, g, z, stream)
                : launch_bp<1, 1, Z2>(y, x, angles, g, z, stream);
  if (g.H == 2)
    return four ? launch_bp<2, 4, Z2>(y, x, angles, g, z, stream)
                : launch_bp<2, 1, Z2>(y, x, angles, g, z, stream);
  if (g.H <= 4)
    return four ? launch_bp<4, 4, Z2>(y, x, angles, g, z, stream)
                : launch_bp<4, 1, Z2>(y, x, angles, g, z, stream);
  return launch_bp<8, 1, Z2>(y, x, angles, g, z, stream);
}

}  // namespace

// Heights per lane: the smallest of 1, 2, 4, 8 that holds them all, 8 per chunk
// beyond.
cudaError_t launch_forward_thin(const float* x, float* y, const float* angles, const Geom& g,
                                int z, cudaStream_t stream) {
  if (g.H == 1) return launch_fp<1, 16>(x, y, angles, g, z, stream);
  if (g.H == 2) return launch_fp<2, 16>(x, y, angles, g, z, stream);
  if (g.H <= 4) return launch_fp<4, 8>(x, y, angles, g, z, stream);
  return launch_fp<8, 4>(x, y, angles, g, z, stream);
}

cudaError_t launch_backward_thin(const float* y, float* x, const float* angles, const Geom& g,
                                 int z, cudaStream_t stream) {
  return z == 2 ? launch_bp_z<true>(y, x, angles, g, z, stream)
                : launch_bp_z<false>(y, x, angles, g, z, stream);
}

int launches_forward_thin(const Geom& g) { return (int)ceil_div(g.n_ang, kMaxGridYZ); }

}  // namespace vp
