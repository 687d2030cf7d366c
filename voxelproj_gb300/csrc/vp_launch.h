// Internal launch interface between the C-ABI layer (vp_capi.cu) and the
// kernel translation units.  Every launcher enqueues on `stream`, never
// synchronises, and returns the launch status.
#pragma once

#include <cuda_runtime.h>

#include "vp_common.cuh"
#include "vp_fp_z0.cuh"

namespace vp {

// Launches kernel k; with programmatic set, with programmatic stream
// serialization, so that it may start while the kernel before it in the
// stream still runs (the kernel must run PdlWait, vp_common.cuh, before it
// reads back outputs that kernel writes).  Set only on a launch that directly
// follows one of this library's own kernels in the same call: the kernel
// before may then be running, but every operation before that one is done.
template <typename... KArgs, typename... Args>
cudaError_t launch_ex(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem,
                      cudaStream_t stream, bool programmatic, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  if (programmatic) {
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}

// y (z_order 0: (n_ang, PX, Hy), z_order 2: (Hy, n_ang, PX)) += A x.
cudaError_t launch_forward_z0(const float* x, float* y, const float* angles, const Geom& g,
                              cudaStream_t stream);
// x (z_order 0: (SY, SX, Hx), z_order 2: (Hx, SY, SX)) += A^T y.
cudaError_t launch_backward_z0(const float* y, float* x, const float* angles, const Geom& g,
                               cudaStream_t stream);
cudaError_t launch_backward_z2(const float* y, float* x, const float* angles, const Geom& g,
                               cudaStream_t stream);

// Status bookkeeping shared by the C entry points (vp_capi.cu): records a
// CUDA error for vp_last_cuda_error() and returns VP_ERR_CUDA; counts launches
// for vp_launch_count().
int record_cuda_error(cudaError_t e);
void count_launches(int n);

// Kernel variant selection (0 = automatic), set through vp_set_kernel_variant.
enum Op : int { OP_FORWARD_Z0 = 0, OP_BACKWARD_Z0 = 1, OP_FORWARD_Z2 = 2, OP_BACKWARD_Z2 = 3,
                OP_COUNT = 4 };
int kernel_variant(int op);

// The banded z_order 0 forward (vp_fp_band.cu): one slab launch on angles
// [a_lo, a_hi); runs_per_warp (1 to 4, 8) runs of 4 bins share a warp (more
// than one: H <= 4 * (32 / runs_per_warp)), split spreads their lines over the 4
// warps of a block.  x's rows are 16-byte aligned.
struct BandLaunch {
  const float* x;
  float* y;
  const float* angles;
  Geom g;
  detail::Slab slab;
  int accumulate;
  int a_lo, a_hi;
  bool programmatic;  // follows this call's previous slab launch
  bool vec_out;       // y's rows take float4 stores
  int lines;          // per partial sum
};
cudaError_t launch_fp_band(const BandLaunch& L, int runs_per_warp, bool split,
                           cudaStream_t stream, int* launches);

// The banded form's windows are placed with float coordinates, off by less
// than its 0.05 voxels of margin up to here.
inline bool fp0_band_ok(const Geom& g) {
  constexpr int kMax = 1 << 16;
  return g.SY <= kMax && g.SX <= kMax && g.PX <= kMax;
}
// Its runs per warp: as many as leave a run the lanes for the heights (at most
// 128).  A (213, 213, 40) and 492 angles 564 us with 2 runs, 444 with 3, (300, 300, 40)
// and 360 797 / 629; 5 runs at 17 to 24 heights gave nothing over 4 (256 x 256 x 20
// and 180 angles 170 us, 32 heights with 4 163).
inline int fp0_band_runs(int H) {
  return H <= 16 ? 8 : H <= 32 ? 4 : H <= 40 ? 3 : H <= 64 ? 2 : 1;
}

// Few heights (vp_thin.cu): the arrays in z_order z.
cudaError_t launch_forward_thin(const float* x, float* y, const float* angles, const Geom& g,
                                int z, cudaStream_t stream);
cudaError_t launch_backward_thin(const float* y, float* x, const float* angles, const Geom& g,
                                 int z, cudaStream_t stream);
int launches_forward_thin(const Geom& g);
// The defaults take them in z_order 0 up to 8 heights, the adjoint only for
// height counts that are not a multiple of 4 (it must equal the batched run
// adjoint bit for bit on the others).  256 x 256, 180 angles, against the
// scalar and 4-height kernels: A 455 -> 53 us (1 height), 573 -> 116 (4),
// 582 -> 200 (8), but 583 -> 545 (16) and 477 -> 529 (19); A^T 363 -> 39 (1),
// 367 -> 67 (3), 378 -> 107 (7), but 321 -> 644 (16).
inline bool z0_forward_thin(const Geom& g) { return g.H <= 4; }
// (Of 5 to 7 heights, small volumes with fewer than 8 angles stay on the scalar
// kernel: 24 x 24 x 7, 4 angles 8 us, 10 on this one.)
inline bool z0_backward_thin(const Geom& g) {
  if (g.n_ang < 8 && g.H > 4 && (long long)g.SY * g.SX < 32 * 32) return false;
  return g.H <= 7 && g.H % 4 != 0;
}

// dst rows of Hd floats from src rows of Hs: heights [0, H), then zeros; dst
// 16-byte aligned, Hd a multiple of 4 (vp_z2.cu).
cudaError_t pad_heights(const float* src, float* dst, long long rows, int Hs, int Hd, int H,
                        cudaStream_t stream);
// Whether a call whose input rows are not whole float4 takes a padded copy, so
// that the float4 kernels run (their epilogues write such outputs by single
// heights).  The copy costs one read and one write of the input; the scalar
// kernels it replaces held one height per lane: (301, 257, 203) and 181 angles,
// A 3.76 -> 1.16 ms, A^T 3.00 -> 0.81 ms.
// Few angles do not pay for it.  The adjoint then runs two class launches and
// the copy where the scalar kernel is one launch, and the 256-height forward
// has a block for 16 bins (or 4 angles x 4 bins) where the scalar one has 8 by
// 32-height chunks.  Times by scalar / padded rows, in us:
//   A^T 512 x 512 x 15: 1 angle 33 / 88, 8 angles 85 / 138, 30 angles 247 / 225;
//   A^T 128 x 128 x 131: 8 angles 31 / 44, 16 angles 51 / 51;
//   A^T 64 x 64 x 127: 30 angles 26 / 27, 60 angles 46 / 34;
//   A^T 24 x 24 x 203: 60 angles 34 / 37, 120 angles 63 / 52;
//   A 128 x 128 x 203: 16 angles 138 / 185, 30 angles 201 / 174;
//   A 64 x 64 x 203: 30 angles 67 / 84, 60 angles 110 / 96;
//   A 512 x 512 x 511, 1 angle: 0.65 / 1.07 ms between synchronisations (the
//   copy's memory, past what its pool keeps, is mapped anew).
// Up to 128 heights the banded forward takes 1.2 to 7 times less at any number of
// angles, the copy included; its 128 + rest parts up to 192 take no more from 4
// angles or 48 x 48 voxels on.
inline bool z0_pad_pays(int op, const Geom& g) {
  const long long vox = (long long)g.SY * g.SX;
  const int least = g.SY < g.SX ? g.SY : g.SX;  // side
  const int n = g.n_ang;
  if (op == OP_FORWARD_Z0) {
    if (g.H <= 192) return g.H <= 128 || n >= 4 || vox >= 48 * 48;
    if (vox >= 320 * 320) return n >= (g.H <= 256 ? 1 : 8);
    if (vox >= 128 * 128) return n >= (vox >= 192 * 192 ? 16 : 30);
    if (vox >= 64 * 64) return n >= (g.H > 256 && least >= 90 ? 30 : 60);
    return n >= (least >= 32 ? 120 : 240);
  }
  if (16ll * g.PX > vox) return false;  // (the sinogram is the copy)
  if (vox >= 128 * 128) return n >= (g.H > 32 ? 16 : vox >= 256 * 256 ? 30 : 60);
  if (vox >= 90 * 90 && g.H > 32) return n >= (g.H >= 200 ? 16 : 30);
  if (vox >= 64 * 64 || g.H <= 128) return n >= 60;
  return n >= (vox >= 45 * 45 && g.H >= 400 ? 60 : 120);
}
inline bool z0_pads(int op, const Geom& g) {
  return kernel_variant(op) == 0 &&
         !(op == OP_FORWARD_Z0 ? z0_forward_thin(g) : z0_backward_thin(g)) && z0_pad_pays(op, g);
}

// z_order 2 through the z_order 0 kernels (vp_z2.cu).
// From 32 heights on always; from 5 on the forward does where it has the
// workspace (z2_workspace_bytes, more than 0 then), else it runs the kernel
// for few heights, which needs none: 384 x 384 x 16, 180 angles 685 against
// 262 us with the transposes, 512 x 512 x 4 and 360 662 against 780 us.  It does so
// with the banded form only, which leaves out zero weights as that kernel does
// (z2_few_transposes).
bool z2_uses_transpose(const Geom& g);
bool z2_can_transpose(const Geom& g);
bool z2_few_transposes(const Geom& g);
size_t z2_workspace_bytes(const Geom& g);
int launches_z2(const Geom& g, bool forward);  // of the transposed form
cudaError_t forward_z2_transposed(const float* x, float* y, const float* angles, const Geom& g,
                                  float* ws, cudaStream_t stream);
cudaError_t backward_z2_transposed(const float* y, float* x, const float* angles, const Geom& g,
                                   float* ws, cudaStream_t stream);
// The two halves of the transposed form: z2_project puts the input in
// height-fastest order and stores its z_order 0 projection, both in ws;
// z2_transpose_out adds (add = 1) or stores (0) that projection into the
// caller's heights-slowest output.
cudaError_t z2_project(bool forward, const float* in, const float* angles, const Geom& g,
                       float* ws, cudaStream_t stream);
cudaError_t z2_transpose_out(bool forward, float* out, const Geom& g, const float* ws, int add,
                             cudaStream_t stream);
// Row ranges of the same: volume rows [lo, hi) of a (g.H, SY, SX) chunk into
// the forward's height-fastest workspace (stored), and of the adjoint's
// workspace result back into a (g.H, SY, SX) chunk (add = 1 adds, 0 stores).
// The workspace's z_order 0 views are xt = ws, yt = ws + SY*SX*Hp (Hp = g.H
// rounded up to 4).
cudaError_t z2_transpose_in_rows(const float* x, const Geom& g, float* ws, int lo, int hi,
                                 cudaStream_t stream);
cudaError_t z2_transpose_out_rows(float* x, const Geom& g, const float* ws, int lo, int hi,
                                  int add, cudaStream_t stream);
// Angle ranges likewise: angles [a0, a1) of a (g.H, n_ang, PX) sinogram into
// the adjoint's workspace (stored), and of the forward's workspace result
// back into a (g.H, n_ang, PX) sinogram (add = 1 adds, 0 stores).
cudaError_t z2_transpose_in_angles(const float* y, const Geom& g, float* ws, int a0, int a1,
                                   cudaStream_t stream);
cudaError_t z2_transpose_out_angles(float* y, const Geom& g, const float* ws, int a0, int a1,
                                    int add, cudaStream_t stream);

// Height split of the 8-heights-per-lane forms: heights [0, r8_heights(H))
// run with 8 per lane (chunks of 256); a last chunk of at most 128 heights
// runs with 4 per lane instead, since 8 would leave half of it idle.
inline int r8_heights(int H) {
  const int full = H / 256 * 256;
  return (H - full > 128 || full == 0) ? H : full;
}

// Forward launch plan of a kernel variant (0 = default) for a geometry:
// heights per lane R, bins per warp KW, candidates in flight un, block on
// neighbouring angles, class slabs, and nslabs slabs of wy rows (and wx
// columns for class slabs; slab k as detail::slab_of).  The batched kernel
// follows the same plan, so its results equal the single-problem kernel's.
struct Fp0Plan {
  int R, KW, un;
  bool agroup, cls, split, staged;
  int nslabs, wy, wx;
};
Fp0Plan forward_z0_plan(const Geom& g, bool vec4, int variant);

// Streamed forms for host buffers.
// Forward, on the main height part: launch_forward_z0_stream gathers angles
// [a_lo, a_hi) from volume rows [rows_lo, rows_hi) for angles whose minor
// axis is x and from columns [cols_lo, cols_hi) for the others (an empty
// range skips that class when adding).  Rows in pieces of up to
// forward_z0_stream_rows (columns empty) as they arrive, then columns in
// pieces of up to forward_z0_stream_cols (rows empty), the first launch in
// the caller's mode and the rest adding, then launch_forward_z0_rest (the
// 4-height remainder of a split heights range, whole), give the full result.
// Adjoint: voxel rows [row_lo, row_hi) alone, row_lo a multiple of
// backward_z0_row_step() (0: rows cannot be split, launch [0, SY) only).
// Pieces hold at most piece_mb MB of one height chunk (and no more than the
// forward plan's slabs).
int forward_z0_stream_rows(const float* x, const float* y, const Geom& g, int piece_mb);
int forward_z0_stream_cols(const float* x, const float* y, const Geom& g, int piece_mb);
cudaError_t launch_forward_z0_stream(const float* x, float* y, const float* angles,
                                     const Geom& g, int rows_lo, int rows_hi, int cols_lo,
                                     int cols_hi, int a_lo, int a_hi, int accumulate,
                                     cudaStream_t stream, int* launches);
cudaError_t launch_forward_z0_rest(const float* x, float* y, const float* angles,
                                   const Geom& g, cudaStream_t stream, int* launches);
int backward_z0_row_step(const float* y, const float* x, const Geom& g);
// Bounded waits in this library's kernels that ran out (synchronising read).
unsigned long long wait_timeouts();
// Limits of the bounded waits for launches enqueued from now on
// (vp_set_wait_limits): polls of a bulk copy's barrier in the staged adjoint
// (the default with use_default), and a batch stage's sleeps (0: default) and
// extra completions waited for (0 in operation).
void set_copy_wait_polls(unsigned polls, bool use_default);
void set_stage_wait_limits(unsigned spins, unsigned extra);
// The current limit of copy waits, and the device address (current device)
// of the counter vp_wait_timeouts reads, for kernels of other units.
unsigned copy_wait_polls();
cudaError_t wait_timeout_counter(unsigned long long** out);
cudaError_t launch_backward_z0_rows(const float* y, float* x, const float* angles,
                                    const Geom& g, int row_lo, int row_hi,
                                    cudaStream_t stream);
// As launch_backward_z0_rows, and then adds addend (same layout as x) into
// those rows: x = (x + A^T y) + addend in adding mode, A^T y + addend in
// store mode, in the same order as a separate add after the projection.
// Only for the run variants (backward_z0_rows_can_add).  addend_ready (may
// be null): an event recorded once addend is in; the launches that read it
// wait for it, the ones before them do not.
bool backward_z0_rows_can_add(const float* y, const float* x, const Geom& g);
cudaError_t launch_backward_z0_rows_add(const float* y, float* x, const float* angles,
                                        const Geom& g, int row_lo, int row_hi,
                                        const float* addend, cudaStream_t stream,
                                        cudaEvent_t addend_ready = nullptr);

// Host-buffer projections (vp_host.cu): g.accumulate selects out += result
// (1) or out = result (0); *launches is incremented by the kernels launched.
cudaError_t forward_z0_host(const float* x_host, float* y_host, const float* angles,
                            const Geom& g, cudaMemPool_t pool, cudaStream_t s, int* launches);
cudaError_t backward_z0_host(const float* y_host, float* x_host, const float* angles,
                             const Geom& g, cudaMemPool_t pool, cudaStream_t s, int* launches);
// z_order 2 (heights slowest): in is x for the forward, y for the adjoint.
cudaError_t z2_host(bool forward, const float* in_host, float* out_host, const float* angles,
                    const Geom& g, cudaMemPool_t pool, cudaStream_t s, int* launches);

// Kernel launches the forward launchers issue for a geometry (grids are
// split past 65535 angle blocks).
int launches_forward_z0(const float* x, const float* y, const Geom& g);
int launches_backward_z0(const float* y, const float* x, const Geom& g);

}  // namespace vp
