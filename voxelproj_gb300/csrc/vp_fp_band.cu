// Launches of the banded z_order 0 forward (vp_fp_band.cuh).
#include <cuda_runtime.h>

#include <type_traits>

#include "vp_common.cuh"
#include "vp_fp_band.cuh"
#include "vp_launch.h"

namespace vp {

namespace {

using namespace detail;

constexpr int kMaxGridYZ = 65535;

// blockIdx.x: run sets of G runs (SP = 1: the block's 4 warps on neighbouring
// ones; SP = 4: all on one); blockIdx.y: angles from a_base; blockIdx.z: height
// chunks.  6 blocks per SM (80 registers) with one run per warp, 5 (96) with
// more, whose window loads are guarded per lane: 128^3 and 192 angles 147
// against 149 us, 384 x 384 x 16 and 180 (split) 252 against 243 us.
template <int G, int SP, bool PDL, bool VOUT>
__global__ void __launch_bounds__(32 * FPB_WARPS, G == 1 ? 6 : 5)
    fp_band_kernel(const float* __restrict__ x, float* __restrict__ y,
                   const float* __restrict__ angles, Geom g, int a_base, Slab slab,
                   int accumulate, int lines) {
  __shared__ BandSmem sm[FPB_WARPS];
  __shared__ float4 sums[SP > 1 ? FPB_WARPS : 1][32][4];
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int set = blockIdx.x * (FPB_WARPS / SP) + warp / SP;
  const int a = a_base + blockIdx.y;
  const int h = G > 1 ? band_height<G>(lane) : blockIdx.z * 128 + lane * 4;
  const bool has = a < g.n_ang && 4 * G * set < g.PX;
  using Wait = std::conditional_t<PDL, PdlWait, NoWait>;
  fp_band_block<G, SP, Wait, VOUT>(x, y, angles, g, set * G, a, h, slab, has,
                                   SP > 1 ? warp % SP : 0, lines, accumulate,
                                   &sm[warp], sums);
}

inline unsigned ceil_div(long long a, long long b) { return (unsigned)((a + b - 1) / b); }

template <int G, int SP, bool VOUT>
cudaError_t launch_band(const BandLaunch& L, cudaStream_t stream, int* launches) {
  Geom g = L.g;
  g.n_ang = L.a_hi;
  for (long long a = L.a_lo; a < L.a_hi; a += kMaxGridYZ) {
    const long long rows = L.a_hi - a < kMaxGridYZ ? L.a_hi - a : kMaxGridYZ;
    const dim3 grid(ceil_div(g.PX, 4 * G * (FPB_WARPS / SP)), (unsigned)rows,
                    G > 1 ? 1 : ceil_div(g.H, 128));
    const dim3 block(32 * FPB_WARPS);
    const bool p = L.programmatic || a > L.a_lo;
    cudaError_t e =
        p ? launch_ex(fp_band_kernel<G, SP, true, VOUT>, grid, block, 0, stream, true, L.x, L.y,
                      L.angles, g, (int)a, L.slab, L.accumulate, L.lines)
          : launch_ex(fp_band_kernel<G, SP, false, VOUT>, grid, block, 0, stream, false, L.x, L.y,
                      L.angles, g, (int)a, L.slab, L.accumulate, L.lines);
    if (launches) ++*launches;
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int G>
cudaError_t launch_band_g(const BandLaunch& L, bool split, cudaStream_t s, int* n) {
  if (split)
    return L.vec_out ? launch_band<G, 4, true>(L, s, n) : launch_band<G, 4, false>(L, s, n);
  return L.vec_out ? launch_band<G, 1, true>(L, s, n) : launch_band<G, 1, false>(L, s, n);
}

}  // namespace

cudaError_t launch_fp_band(const BandLaunch& L, int runs_per_warp, bool split,
                           cudaStream_t stream, int* launches) {
  switch (runs_per_warp) {
    case 8: return launch_band_g<8>(L, split, stream, launches);
    case 3: return launch_band_g<3>(L, split, stream, launches);
    case 4: return launch_band_g<4>(L, split, stream, launches);
    case 2: return launch_band_g<2>(L, split, stream, launches);
    default: return launch_band_g<1>(L, split, stream, launches);
  }
}

}  // namespace vp
