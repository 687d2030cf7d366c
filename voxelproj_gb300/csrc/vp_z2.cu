// z_order 2 through the z_order 0 kernels.
//
// In z_order 2 the height axis is the slowest one: x (H, SY, SX) and
// y (H, n_ang, PX).  The projector's weights do not depend on the height,
// so the fast kernels put heights across the lanes of a warp; that needs
// heights contiguous.  For H >= 32, and for the forward from 5 heights on where
// it has the scratch, the z_order 2 operators therefore run as
//     transpose the input to height-fastest order  (HBM-bound tiled transpose)
//     z_order 0 kernel, storing (not accumulating) into scratch
//     transpose the result back, adding it to the caller's output
// which costs about 2 * (|x| + |y|) of extra HBM traffic, a fraction of a
// millisecond at 512^3 against several milliseconds of projector work, and
// keeps the reference's accumulate semantics.  Other small H run the kernels
// for few heights (vp_thin.cu: lanes across bins / voxels).
//
// Scratch: SY*SX*Hp + n_ang*PX*Hp floats (Hp = H rounded up to 4), supplied by
// the caller (vp_*_z2_ws) or taken from a library-private stream-ordered pool.
#include <cuda_runtime.h>

#include <cstdint>

#include "vp_common.cuh"
#include "vp_launch.h"

namespace vp {

namespace {

constexpr int TT = 64;        // tile edge
constexpr int TQ = TT / 4;    // float4 per tile row
constexpr int TTHREADS = 256;
constexpr int TROWS = TTHREADS / TQ;  // tile rows moved at a time
constexpr int TK = TT / TROWS;        // steps per tile

// 4 floats from p + i, of which those below n (counted from i) exist; VEC: by
// one float4 (p + i is 16-byte aligned and the row is padded to whole float4).
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* p, long long i, long long n) {
  if (i >= n) return make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (VEC) return __ldg(reinterpret_cast<const float4*>(p + i));
  return make_float4(__ldg(p + i), i + 1 < n ? __ldg(p + i + 1) : 0.f,
                     i + 2 < n ? __ldg(p + i + 2) : 0.f, i + 3 < n ? __ldg(p + i + 3) : 0.f);
}

// dst[c * dst_ld + r] (+)= src[r * src_ld + c] for r < rows, c < cols; the
// storing form writes zeros for rows <= r < rows_out (pad heights).
//
// One 64 x 64 tile per block: each thread brings 4 float4 of source rows into
// shared memory and takes 4 float4 of destination rows out, with the adding
// form's current values loaded before the barrier.  VS / VD: source / destination
// rows in float4 (else single floats; VS rows are padded to whole float4).
// Bound by HBM.  256^3 to height-fastest order (134 MB moved) 31.5 -> 20.5 us,
// a (360, 256, 256) sinogram back (189 MB) 60 -> 26 us, against 4-byte accesses
// of 32 x 32 tiles by one wave of blocks.
template <bool ADD, bool VS, bool VD>
__global__ void __launch_bounds__(TTHREADS)
    transpose_kernel(const float* __restrict__ src, float* __restrict__ dst, long long rows,
                     long long cols, long long src_ld, long long dst_ld, long long rows_out,
                     unsigned tiles_c) {
  __shared__ float tile[TT][TT + 1];  // [c][r]
  const long long r0 = (long long)(blockIdx.x / tiles_c) * TT;
  const long long c0 = (long long)(blockIdx.x % tiles_c) * TT;
  const int q = threadIdx.x % TQ, t = threadIdx.x / TQ;
  float4 v[TK], old[TK];
  (void)old;
#pragma unroll
  for (int k = 0; k < TK; ++k) {
    const long long r = r0 + t + k * TROWS;
    v[k] = r < rows ? load4<VS>(src + r * src_ld, c0 + 4 * q, cols)
                    : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if constexpr (ADD) {
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      const long long c = c0 + t + k * TROWS;
      if (c >= cols) continue;
      const float* d = dst + c * dst_ld;
      const long long r = r0 + 4 * q;
      if (VD && r + 3 < rows_out) {
        old[k] = *reinterpret_cast<const float4*>(d + r);
      } else {
        old[k] = make_float4(r < rows_out ? d[r] : 0.f, r + 1 < rows_out ? d[r + 1] : 0.f,
                             r + 2 < rows_out ? d[r + 2] : 0.f, r + 3 < rows_out ? d[r + 3] : 0.f);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < TK; ++k) {
    const int r = t + k * TROWS;
    tile[4 * q][r] = v[k].x;
    tile[4 * q + 1][r] = v[k].y;
    tile[4 * q + 2][r] = v[k].z;
    tile[4 * q + 3][r] = v[k].w;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < TK; ++k) {
    const int tc = t + k * TROWS;
    const long long c = c0 + tc;
    if (c >= cols) continue;
    const long long r = r0 + 4 * q;
    float4 o = make_float4(tile[tc][4 * q], tile[tc][4 * q + 1], tile[tc][4 * q + 2],
                           tile[tc][4 * q + 3]);
    if constexpr (ADD) o = f4_add(old[k], o);
    float* d = dst + c * dst_ld;
    if (VD && r + 3 < rows_out) {
      *reinterpret_cast<float4*>(d + r) = o;
    } else {
      if (r < rows_out) d[r] = o.x;
      if (r + 1 < rows_out) d[r + 1] = o.y;
      if (r + 2 < rows_out) d[r + 2] = o.z;
      if (r + 3 < rows_out) d[r + 3] = o.w;
    }
  }
}

// rows_out: as many rows of zeros as the storing form is to pad to.
cudaError_t transpose(const float* src, float* dst, long long rows, long long cols,
                      long long src_ld, long long dst_ld, int accumulate, cudaStream_t stream,
                      long long pad_to = 0) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  const long long rows_out = rows < pad_to ? pad_to : rows;
  const auto aligned = [](const float* p, long long ld) {
    return ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
  };
  // a float4 at the end of a source row reads up to 3 floats past cols: inside
  // the row where it is padded, into the next one where it is not
  const bool vs = aligned(src, src_ld) && (cols % 4 == 0 || (cols + 3) / 4 * 4 <= src_ld);
  const bool vd = aligned(dst, dst_ld);
  const long long tiles_c = (cols + TT - 1) / TT, tiles_r = (rows_out + TT - 1) / TT;
  // a grid holds 2^31 - 1 blocks: bands of tile rows
  const long long band = ((1ll << 31) - 1) / tiles_c;
  for (long long b = 0; b < tiles_r; b += band) {
    const long long nr = tiles_r - b < band ? tiles_r - b : band;
    const float* s = src + b * TT * src_ld;
    float* d = dst + b * TT;
    const auto kernel = accumulate ? (vs ? (vd ? transpose_kernel<true, true, true>
                                               : transpose_kernel<true, true, false>)
                                         : (vd ? transpose_kernel<true, false, true>
                                               : transpose_kernel<true, false, false>))
                                   : (vs ? (vd ? transpose_kernel<false, true, true>
                                               : transpose_kernel<false, true, false>)
                                         : (vd ? transpose_kernel<false, false, true>
                                               : transpose_kernel<false, false, false>));
    kernel<<<(unsigned)(nr * tiles_c), TTHREADS, 0, stream>>>(s, d, rows - b * TT, cols, src_ld,
                                                              dst_ld, rows_out - b * TT,
                                                              (unsigned)tiles_c);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

inline long long round4(long long v) { return (v + 3) / 4 * 4; }

// dst rows of Hd floats (16-byte aligned) from src rows of Hs: heights [0, H),
// then zeros.  blockDim.x lanes share a row, a float4 of it each per step.
__global__ void __launch_bounds__(256)
    pad_kernel(const float* __restrict__ src, float* __restrict__ dst, long long rows, int Hs,
               int Hd, int H) {
  const int nq = Hd / 4;
  for (long long r = (long long)blockIdx.x * blockDim.y + threadIdx.y; r < rows;
       r += (long long)gridDim.x * blockDim.y) {
    const float* s = src + r * Hs;
    float4* d = reinterpret_cast<float4*>(dst + r * Hd);
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = 4 * q + i < H ? __ldg(s + 4 * q + i) : 0.0f;
      d[q] = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
}

}  // namespace

cudaError_t pad_heights(const float* src, float* dst, long long rows, int Hs, int Hd, int H,
                        cudaStream_t stream) {
  int tx = 32;
  while (tx > 1 && tx / 2 >= Hd / 4) tx /= 2;
  const int ty = 256 / tx;
  const long long blocks = (rows + ty - 1) / ty;
  pad_kernel<<<(unsigned)(blocks < 8192 ? blocks : 8192), dim3(tx, ty), 0, stream>>>(
      src, dst, rows, Hs, Hd, H);
  return cudaGetLastError();
}

bool z2_uses_transpose(const Geom& g) { return g.H >= 32; }

bool z2_can_transpose(const Geom& g) { return g.H >= 5; }

bool z2_few_transposes(const Geom& g) {
  return z2_can_transpose(g) && kernel_variant(OP_FORWARD_Z0) == 0 && fp0_band_ok(g);
}

size_t z2_workspace_bytes(const Geom& g) {
  if (!z2_can_transpose(g)) return 0;
  const long long Hp = round4(g.H);
  return (size_t)(((long long)g.SY * g.SX + (long long)g.n_ang * g.PX) * Hp) * sizeof(float);
}

int launches_z2(const Geom& g, bool forward) {
  // the transposed path runs the z_order 0 kernels on 16-byte aligned scratch
  // with a height extent that is a multiple of 4
  Geom g0 = g;
  g0.H = g0.Hx = g0.Hy = (int)round4(g.H);
  static const float aligned[4] = {};
  return 2 + (forward ? launches_forward_z0(aligned, aligned, g0)
                      : launches_backward_z0(aligned, aligned, g0));
}

// The first steps of the transposed form, into ws: the input to
// height-fastest order, then its z_order 0 projection (stored).
//   forward:  x (Hx, SY, SX) -> xt (SY, SX, Hp); yt = A xt
//   adjoint:  y (Hy, n, PX) -> yt (n, PX, Hp); xt = A^T yt
cudaError_t z2_project(bool forward, const float* in, const float* angles, const Geom& g,
                       float* ws, cudaStream_t stream) {
  const long long Hp = round4(g.H);
  const long long nvox = (long long)g.SY * g.SX;
  const long long nbin = (long long)g.n_ang * g.PX;
  float* xt = ws;
  float* yt = ws + nvox * Hp;
  Geom g0 = g;
  g0.H = g0.Hx = g0.Hy = (int)Hp;
  g0.accumulate = 0;
  // as the kernel for few heights (vp_thin.cu) does
  g0.skip_zero = forward && !z2_uses_transpose(g);
  if (forward) {
    const cudaError_t e = transpose(in, xt, g.H, nvox, nvox, Hp, 0, stream, Hp);
    if (e != cudaSuccess) return e;
    return launch_forward_z0(xt, yt, angles, g0, stream);
  }
  const cudaError_t e = transpose(in, yt, g.H, nbin, nbin, Hp, 0, stream, Hp);
  if (e != cudaSuccess) return e;
  return launch_backward_z0(yt, xt, angles, g0, stream);
}

// The last step: out (+)= the projection in ws, back in heights-slowest
// order (add = 1 adds, 0 stores).
cudaError_t z2_transpose_out(bool forward, float* out, const Geom& g, const float* ws, int add,
                             cudaStream_t stream) {
  const long long Hp = round4(g.H);
  const long long nvox = (long long)g.SY * g.SX;
  const long long nbin = (long long)g.n_ang * g.PX;
  if (forward) return transpose(ws + nvox * Hp, out, nbin, g.H, Hp, nbin, add, stream);
  return transpose(ws, out, nvox, g.H, Hp, nvox, add, stream);
}

// Volume rows [lo, hi) of a heights-slowest volume chunk in (g.H, SY, SX)
// into the transposed form's xt (SY, SX, Hp), stored.
cudaError_t z2_transpose_in_rows(const float* x, const Geom& g, float* ws, int lo, int hi,
                                 cudaStream_t stream) {
  const long long Hp = round4(g.H);
  const long long nvox = (long long)g.SY * g.SX;
  return transpose(x + (long long)lo * g.SX, ws + (long long)lo * g.SX * Hp, g.H,
                   (long long)(hi - lo) * g.SX, nvox, Hp, 0, stream, Hp);
}

// Angles [a0, a1) of a heights-slowest sinogram in (g.H, n_ang, PX) into the
// transposed form's yt (n_ang, PX, Hp), stored.
cudaError_t z2_transpose_in_angles(const float* y, const Geom& g, float* ws, int a0, int a1,
                                   cudaStream_t stream) {
  const long long Hp = round4(g.H);
  const long long nvox = (long long)g.SY * g.SX;
  const long long nbin = (long long)g.n_ang * g.PX;
  return transpose(y + (long long)a0 * g.PX, ws + nvox * Hp + (long long)a0 * g.PX * Hp, g.H,
                   (long long)(a1 - a0) * g.PX, nbin, Hp, 0, stream, Hp);
}

// Angles [a0, a1) of the forward's yt (n_ang, PX, Hp) in ws into a
// heights-slowest sinogram y (g.H, n_ang, PX): added (add = 1) or stored (0).
cudaError_t z2_transpose_out_angles(float* y, const Geom& g, const float* ws, int a0, int a1,
                                    int add, cudaStream_t stream) {
  const long long Hp = round4(g.H);
  const long long nvox = (long long)g.SY * g.SX;
  const long long nbin = (long long)g.n_ang * g.PX;
  return transpose(ws + nvox * Hp + (long long)a0 * g.PX * Hp, y + (long long)a0 * g.PX,
                   (long long)(a1 - a0) * g.PX, g.H, Hp, nbin, add, stream);
}

// Volume rows [lo, hi) of the adjoint's xt (SY, SX, Hp) in ws into a
// heights-slowest chunk x (g.H, SY, SX): added (add = 1) or stored (0).
cudaError_t z2_transpose_out_rows(float* x, const Geom& g, const float* ws, int lo, int hi,
                                  int add, cudaStream_t stream) {
  const long long Hp = round4(g.H);
  const long long nvox = (long long)g.SY * g.SX;
  return transpose(ws + (long long)lo * g.SX * Hp, x + (long long)lo * g.SX,
                   (long long)(hi - lo) * g.SX, g.H, Hp, nvox, add, stream);
}

// x (Hx, SY, SX) -> xt (SY, SX, Hp); yt = A xt; y (Hy, n, PX) (+)= yt^T.
cudaError_t forward_z2_transposed(const float* x, float* y, const float* angles, const Geom& g,
                                  float* ws, cudaStream_t stream) {
  const cudaError_t e = z2_project(true, x, angles, g, ws, stream);
  if (e != cudaSuccess) return e;
  return z2_transpose_out(true, y, g, ws, g.accumulate, stream);
}

// y (Hy, n, PX) -> yt (n, PX, Hp); xt = A^T yt; x (Hx, SY, SX) (+)= xt^T.
cudaError_t backward_z2_transposed(const float* y, float* x, const float* angles, const Geom& g,
                                   float* ws, cudaStream_t stream) {
  const cudaError_t e = z2_project(false, y, angles, g, ws, stream);
  if (e != cudaSuccess) return e;
  return z2_transpose_out(false, x, g, ws, g.accumulate, stream);
}

}  // namespace vp
