// Launchers of the tile step kernel; included once per build flavour with
// SEIS_NS set (exact / fast).
#pragma once
#include "fd_tile.cuh"

namespace seis {
namespace SEIS_NS {

// ptab of every shot: the coefficients of the one-way update (fd.cpp:1098-1104
// and its mirrors, :1146-1178) and the blend weights (InitInversion.cpp:20-37),
// each rounded as the build's per-cell formulas (absorb_geom) round it.  Formed once per run: in the step
// kernels these divisions cost more per pad cell than the stencil (the upper
// left corner's, in double, held its whole tile for 15,000 cycles).
__device__ float tab_recip(float d) {
  const float r = 1.0f / d;
  return r >= 0x1p-30f && r <= 1.0f ? r : 0.0f;
}
// (the contracted build's Born steps have always rounded the ramp once, its
// other steps twice)
__device__ float tab_weight(int d, const ShotDev &g, int born) {
#ifdef SEIS_FAST_MATH
  return born ? __fmaf_rn(-(float)d, g.inv_pml, 1.0f) : 1.0f - __fmul_rn((float)d, g.inv_pml);
#else
  return d == 0 ? 1.0f : 1.0f - (float)d * 1.0f / (float)g.pml;
#endif
}
__global__ void pad_tab_kernel(const ShotDev *__restrict__ shots, int born) {
  const ShotDev &g = shots[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int NX = g.NX, NZ = g.NZ, n = pad_tab_nz(NZ), m = pad_tab_nx(NX);
  float *T = const_cast<float *>(g.ptab);
  if (i < n) {  // left and right strip of a row
    const int iz = min(i, NZ - 1);
    for (int b = 0; b < 2; b++) {
      const float v = g.vel[(size_t)(b ? NX - 1 : 0) * g.LDZ + iz];
#ifdef SEIS_FAST_MATH
      const float a2 = g.hdt2 * (1.0f / v), a3 = v * g.q4dz2;
#else
      const float a2 = g.hdt2 / v, a3 = v / 4.0f / g.dz / g.dz;
#endif
      float *t = T + 3 * b * n + i;
      t[0] = a2;
      t[n] = a3;
#ifdef SEIS_FAST_MATH
      t[2 * n] = __fadd_rn(g.a1x, a2);
#else
      t[2 * n] = tab_recip(g.a1x + a2);
#endif
    }
    T[6 * n + i] = tab_weight(max(max(g.pml - iz, iz - (g.pml + g.nz - 1)), 0), g, born);
  } else if (i < n + m) {  // top and bottom strip of a column
    const int j = i - n, ix = min(j, NX - 1);
    float *C = T + pad_tab_x(NZ);
    for (int b = 0; b < 2; b++) {
      const float v = g.vel[(size_t)ix * g.LDZ + (b ? NZ - 1 : 0)];
#ifdef SEIS_FAST_MATH
      const float a2 = g.hdt2 * (1.0f / v), a3 = v * g.q4dx2;
#else
      const float a2 = g.hdt2 / v, a3 = v / 4.0f / g.dx / g.dx;
#endif
      float *t = C + 3 * b * m + j;
      t[0] = a2;
      t[m] = a3;
#ifdef SEIS_FAST_MATH
      t[2 * m] = __fadd_rn(g.a1z, a2);
#else
      t[2 * m] = tab_recip(g.a1z + a2);
#endif
    }
    C[6 * m + j] = tab_weight(max(max(g.pml - ix, ix - (g.pml + g.nx - 1)), 0), g, born);
  } else if (i < n + m + 4) {
    const int c = i - n - m;
    const float v = g.vel[(size_t)(c & 2 ? NX - 1 : 0) * g.LDZ + (c & 1 ? NZ - 1 : 0)];
    // upper left: sqrt(2)/v/dt formed in double (:1176)
    const float a3 = c == 0 ? __double2float_rn(g.sqrt2d / (double)v / (double)g.dt)
                            : g.sqrt2f / v / g.dt;
    const float d = g.ax1 + g.ax2 + a3;
    float *t = T + pad_tab_c(NX, NZ) + 3 * c;
    t[0] = a3;
    t[1] = d;
    t[2] = tab_recip(d);
  }
}

namespace {
// CTAs of the persistent interior kernel: as many as are resident at once
template <int S, int MODE>
struct LoopGrid {
  static int ctas;
};
template <int S, int MODE>
int LoopGrid<S, MODE>::ctas = 0;

template <int S, int MODE>
cudaError_t setup() {
  cudaError_t e = cudaFuncSetAttribute(step_tile_kernel<S, MODE>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)UCfg<S, MODE>::bytes);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(interior_loop_kernel<S, MODE>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)LCfg<S, MODE>::bytes);
  int dev = 0, nsm = 0, per = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, interior_loop_kernel<S, MODE>,
                                                      Geo<S>::NT, LCfg<S, MODE>::bytes);
  if (e == cudaSuccess) LoopGrid<S, MODE>::ctas = (per > 0 ? per : 1) * nsm;
  return e;
}

template <int S>
cudaError_t setup_shape() {
  cudaError_t e = setup<S, MODE_MODEL>();
  if (e == cudaSuccess) e = setup<S, MODE_RCV>();
  if (e == cudaSuccess) e = setup<S, MODE_BORN>();
#ifdef SEIS_FAST_MATH
  if (e == cudaSuccess) e = setup<S, MODE_ADJ>();
#endif
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(step_pair_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)UCfg<S, MODE_MODEL>::bytes);
  return e;
}

// A launch that may start before the last one on the stream has finished
// (programmatic) when `pdl`.
template <class K, class... A>
cudaError_t launch_pdl(K kernel, int grid, int block, size_t smem, cudaStream_t s, int pdl, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, args...);
}

// Every tile in one launch on s_int, or the interior tiles by the persistent
// kernel on s_int and the pad tiles on s_pad: as `loop` says; by default the
// latter when each persistent CTA gets at least LOOP_MIN_TILES tiles (its
// double buffering pays, and the last round of tiles is a small part of the
// launch).
constexpr int LOOP_MIN_TILES = 4;
template <int S, int MODE>
bool splits(int n_int, int loop) {
  return n_int > 0 && (loop > 0 || (loop < 0 && n_int >= LOOP_MIN_TILES * LoopGrid<S, MODE>::ctas));
}
template <int S, int MODE>
cudaError_t launch_t(const ShotDev *d_shots, const Tile *d_tiles, int n_int, int n_pad,
                     const StepArgs &a, int *d_err, cudaStream_t s_int, cudaStream_t s_pad) {
  constexpr int NT = Geo<S>::NT;
  const bool split = splits<S, MODE>(n_int, a.loop);
  if (split) {
    int G = LoopGrid<S, MODE>::ctas;
    // Born's persistent CTAs (two of 112 KB per SM in the 256-thread shapes)
    // leave no shared memory for a pad tile's CTA: beside pad tiles one per SM,
    // which the memory-bound interior tiles hardly miss, so that the pad tiles,
    // bound by latency and instructions, run beside them instead of after them
    // (eight shots of 4000 x 1000: 151 -> 136 us a step, three: 54 -> 49).  The
    // other modes' CTAs are smaller (one field: 1-2% either way; adjoint:
    // slower), as are Born's in 32 x 32 tiles (slower).
    if (MODE == MODE_BORN && LCfg<S, MODE>::MIN_CTAS == 2 && n_pad > 0 && s_int != s_pad) G /= 2;
    interior_loop_kernel<S, MODE><<<G < n_int ? G : n_int, NT, LCfg<S, MODE>::bytes, s_int>>>(
        d_shots, d_tiles, n_int, a, d_err);
    d_tiles += n_int;
    n_int = 0;
  }
  if (n_int + n_pad > 0) {
    cudaError_t e = launch_pdl(step_tile_kernel<S, MODE>, n_int + n_pad, NT, UCfg<S, MODE>::bytes,
                               n_int > 0 ? s_int : s_pad, a.pdl, d_shots, d_tiles, n_int, n_pad, a,
                               d_err);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

template <int S>
cudaError_t launch_mode(int mode, const ShotDev *d_shots, const Tile *d_tiles, int n_int,
                        int n_pad, const StepArgs &a, int *d_err, cudaStream_t s_int,
                        cudaStream_t s_pad) {
  switch (mode) {
    case MODE_MODEL:
      return launch_t<S, MODE_MODEL>(d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    case MODE_RCV:
      return launch_t<S, MODE_RCV>(d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    case MODE_BORN:
      return launch_t<S, MODE_BORN>(d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
#ifdef SEIS_FAST_MATH
    case MODE_ADJ:
      return launch_t<S, MODE_ADJ>(d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
#endif
    default:
      return cudaErrorInvalidValue;
  }
}
template <int S>
bool splits_mode(int mode, int n_int, int loop) {
#ifdef SEIS_FAST_MATH
  if (mode == MODE_ADJ) return splits<S, MODE_ADJ>(n_int, loop);
#endif
  return mode == MODE_MODEL  ? splits<S, MODE_MODEL>(n_int, loop)
         : mode == MODE_RCV ? splits<S, MODE_RCV>(n_int, loop)
                            : splits<S, MODE_BORN>(n_int, loop);
}
}  // namespace

bool step_splits(int mode, int n_int, int shape, int loop) {
  switch (shape) {
    case SHAPE_32x64: return splits_mode<SHAPE_32x64>(mode, n_int, loop);
    case SHAPE_64x32: return splits_mode<SHAPE_64x32>(mode, n_int, loop);
    case SHAPE_16x128: return splits_mode<SHAPE_16x128>(mode, n_int, loop);
    case SHAPE_64x64: return splits_mode<SHAPE_64x64>(mode, n_int, loop);
    case SHAPE_32x32: return splits_mode<SHAPE_32x32>(mode, n_int, loop);
    default: return false;
  }
}

cudaError_t launch_pad_tab(const ShotDev *d_shots, int nshots, int max_len, int born,
                           cudaStream_t s) {
  pad_tab_kernel<<<dim3((max_len + 127) / 128, nshots), 128, 0, s>>>(d_shots, born);
  return cudaGetLastError();
}

cudaError_t configure() {
  cudaError_t e = setup_shape<SHAPE_32x64>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_64x32>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_16x128>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_64x64>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_32x32>();
  return e;
}

template <int S>
static cudaError_t launch_pair_s(const ShotDev *d_shots, const Tile *d_tiles, int n_int, int n_pad,
                                 const StepArgs &a, int *d_err, cudaStream_t s) {
  return launch_pdl(step_pair_kernel<S>, 2 * (n_int + n_pad), Geo<S>::NT,
                    UCfg<S, MODE_MODEL>::bytes, s, a.pdl, d_shots, d_tiles, n_int, n_pad, a, d_err);
}
cudaError_t launch_pair(const ShotDev *d_shots, const Tile *d_tiles, int n_int, int n_pad,
                        int shape, const StepArgs &a, int *d_err, cudaStream_t s) {
  switch (shape) {
    case SHAPE_32x64: return launch_pair_s<SHAPE_32x64>(d_shots, d_tiles, n_int, n_pad, a, d_err, s);
    case SHAPE_64x32: return launch_pair_s<SHAPE_64x32>(d_shots, d_tiles, n_int, n_pad, a, d_err, s);
    case SHAPE_16x128: return launch_pair_s<SHAPE_16x128>(d_shots, d_tiles, n_int, n_pad, a, d_err, s);
    case SHAPE_64x64: return launch_pair_s<SHAPE_64x64>(d_shots, d_tiles, n_int, n_pad, a, d_err, s);
    case SHAPE_32x32: return launch_pair_s<SHAPE_32x32>(d_shots, d_tiles, n_int, n_pad, a, d_err, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_step(int mode, const ShotDev *d_shots, const Tile *d_tiles, int n_int,
                        int n_pad, int shape, const StepArgs &a, int *d_err, cudaStream_t s_int,
                        cudaStream_t s_pad) {
  switch (shape) {
    case SHAPE_32x64:
      return launch_mode<SHAPE_32x64>(mode, d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    case SHAPE_64x32:
      return launch_mode<SHAPE_64x32>(mode, d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    case SHAPE_16x128:
      return launch_mode<SHAPE_16x128>(mode, d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    case SHAPE_64x64:
      return launch_mode<SHAPE_64x64>(mode, d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    case SHAPE_32x32:
      return launch_mode<SHAPE_32x32>(mode, d_shots, d_tiles, n_int, n_pad, a, d_err, s_int, s_pad);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace SEIS_NS
}  // namespace seis
