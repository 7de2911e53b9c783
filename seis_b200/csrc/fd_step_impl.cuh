// Launchers of the tile step kernel; included once per build flavour with
// SEIS_NS set (exact / fast).
#pragma once
#include "fd_tile.cuh"

namespace seis {
namespace SEIS_NS {

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
  return e;
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
    const int G = LoopGrid<S, MODE>::ctas;
    interior_loop_kernel<S, MODE><<<G < n_int ? G : n_int, NT, LCfg<S, MODE>::bytes, s_int>>>(
        d_shots, d_tiles, n_int, a, d_err);
    d_tiles += n_int;
    n_int = 0;
  }
  if (n_int + n_pad > 0) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(n_int + n_pad);
    c.blockDim = dim3(NT);
    c.dynamicSmemBytes = UCfg<S, MODE>::bytes;
    c.stream = n_int > 0 ? s_int : s_pad;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = a.pdl ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&c, step_tile_kernel<S, MODE>, d_shots, d_tiles, n_int,
                                       n_pad, a, d_err);
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
    default:
      return cudaErrorInvalidValue;
  }
}
template <int S>
bool splits_mode(int mode, int n_int, int loop) {
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

cudaError_t configure() {
  cudaError_t e = setup_shape<SHAPE_32x64>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_64x32>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_16x128>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_64x64>();
  if (e == cudaSuccess) e = setup_shape<SHAPE_32x32>();
  return e;
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
