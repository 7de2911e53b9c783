// Auxiliary kernels of the FD engine (sm_100a): model padding, gather
// transposes, and the reverse-pass helpers of the reference RTM.  The time
// step itself is the tile kernel (fd_tile.cuh).
//
// Compiled with --fmad=false and IEEE division: the RTM imaging arithmetic
// rounds as the reference's does.
#include <algorithm>

#define SEIS_NS exact
#include "fd_cell.cuh"

namespace seis {
namespace {

using exact::coef;

// Pad a [nx][nz] model into a shot's field layout (cell (0,0) at dst):
// clamp-to-edge (setVel, InitInversion.cpp:92-113) or zero (setDv, :116-126).
// Only cells of the padded grid are written; the margins stay zero.
__global__ void pad_kernel(const float *__restrict__ src, int nx, int nz, int pml, int LDZ,
                           int clamp, float *__restrict__ dst) {
  const int NX = nx + 2 * pml, NZ = nz + 2 * pml;
  size_t n = (size_t)NX * NZ;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    int ix = (int)(i / NZ), iz = (int)(i - (size_t)ix * NZ);
    int jx = ix - pml, jz = iz - pml;
    float v = 0.0f;
    if (clamp) {
      jx = jx < 0 ? 0 : (jx >= nx ? nx - 1 : jx);
      jz = jz < 0 ? 0 : (jz >= nz ? nz - 1 : jz);
      v = src[(size_t)jx * nz + jz];
    } else if (jx >= 0 && jx < nx && jz >= 0 && jz < nz) {
      v = src[(size_t)jx * nz + jz];
    }
    dst[(size_t)ix * LDZ + iz] = v;
  }
}

__global__ void transpose_kernel(const float *__restrict__ src, int rows, int cols,
                                 float *__restrict__ dst) {
  __shared__ float tile[32][33];
  int c = blockIdx.x * 32 + threadIdx.x, r0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int r = r0 + k;
    if (r < rows && c < cols) tile[k][threadIdx.x] = src[(size_t)r * cols + c];
  }
  __syncthreads();
  int r = r0 + threadIdx.x;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    int cc = blockIdx.x * 32 + k;
    if (r < rows && cc < cols) dst[(size_t)cc * rows + r] = tile[threadIdx.x][k];
  }
}

// Reverse pass of the reference RTM, before each step (fd.cpp:659-663):
// subtract the source from the older field and write the saved boundary
// strips of sample it-ndel into the current field.
__global__ void rtm_restore_kernel(const ShotDev *__restrict__ shots, int nshots, int rot,
                                   int it) {
  const int s = blockIdx.y;
  if (s >= nshots) return;
  const ShotDev &g = shots[s];
  if (it >= g.NT || it < g.ndel) return;
  float *prev = g.fa[rot % 3];
  float *cur = g.fa[(rot + 1) % 3];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && it - 1 > 0) {
    size_t off = (size_t)g.sxp * g.LDZ + g.szp;
    float vt2 = coef(g.vel[off], g).vt2;
    prev[off] = prev[off] - vt2 * g.wav[it - 1];
  }
  if (i >= g.strip_len) return;
  const float *src = g.strips + (size_t)(it - g.ndel) * g.strip_len;
  int rowcells = 2 * LAYERS * g.nx;
  int ix, iz;
  if (i < rowcells) {
    int l = i / g.nx, x = i - l * g.nx;
    ix = x + g.pml;
    iz = l < LAYERS ? g.pml + l : g.nz + g.pml - 1 - (l - LAYERS);
  } else {
    int j = i - rowcells;
    int l = j / g.nz, z = j - l * g.nz;
    iz = z + g.pml;
    ix = l < LAYERS ? g.pml + l : g.nx + g.pml - 1 - (l - LAYERS);
  }
  cur[(size_t)ix * g.LDZ + iz] = src[i];
}

// Before a re-propagation step of the plane-wave receiver field
// (adjointPlane, fd.cpp:870-893): the boundary layers kept for sample strip_k
// restored into the current field, and the receiver samples rec_k (times vt2)
// taken off the previous field at the receiver rows.  Either part is skipped
// when its index is negative.
__global__ void plane_rcv_prep_kernel(const ShotDev *__restrict__ shots, int nshots, int rot_b,
                                      int strip_k, int rec_k) {
  const int s = blockIdx.y;
  if (s >= nshots) return;
  const ShotDev &g = shots[s];
  float *prev = g.fb[rot_b % 3];
  float *cur = g.fb[(rot_b + 1) % 3];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (rec_k >= 0 && i < g.nx) {  // fd.cpp:870-874
    const size_t off = (size_t)(i + g.pml) * g.LDZ + (g.gz[i] + g.pml);
    const float vt2 = coef(g.vel[off], g).vt2;
    prev[off] = prev[off] - g.rec[(size_t)rec_k * g.nx + i] * vt2;
  }
  if (strip_k < 0 || i >= g.strip_len) return;
  const float *src = g.strips + (size_t)strip_k * g.strip_len;
  const int rowcells = 2 * LAYERS * g.nx;
  int ix, iz;
  if (i < rowcells) {
    int l = i / g.nx, x = i - l * g.nx;
    ix = x + g.pml;
    iz = l < LAYERS ? g.pml + l : g.nz + g.pml - 1 - (l - LAYERS);
  } else {
    int j = i - rowcells;
    int l = j / g.nz, z = j - l * g.nz;
    iz = z + g.pml;
    ix = l < LAYERS ? g.pml + l : g.nx + g.pml - 1 - (l - LAYERS);
  }
  cur[(size_t)ix * g.LDZ + iz] = src[i];  // SaveAtBoundary restore, fd.cpp:1206-1223
}

// Packed pairs (see V4 of the step kernels): a product rounded by itself is
// x y + (-0), the zero read from constant memory.
__constant__ float IMG_NEG_ZERO = -0.0f;
__device__ __forceinline__ uint64_t bits2(const float2 &x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x.x), "f"(x.y));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t x, uint64_t y, uint64_t nz) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(nz));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t x, uint64_t y) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ float2 pair2(uint64_t r) {
  float2 x;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x.x), "=f"(x.y) : "l"(r));
  return x;
}

// Imaging of the reference RTM, one CTA per interior column (fd.cpp:668-669,
// :681-684, FaQi :1272-1298):
//   U = ((u2 + u0 - 2 u1)/dt^2) vel3,  img += U R,  img += 0.5 (U R - H[U] H[R])
// with H the 61-tap Hilbert FIR along z over the whole padded column, whose
// taps at even offsets are exactly zero (hilbert.h:67).  Bound by the filter's
// arithmetic (30 products and sums of two fields, each rounded, per cell): U
// and R lie interleaved in shared memory with HILB_HALF zeros on either side,
// a thread forms IMG_K outputs two rows apart, so that each pair it reads
// serves all of them and both fields share one packed operation; every third
// pair of rows puts the 16 lanes of a half warp on different banks.  A column
// of 320 rows: 210 -> 75 instructions a cell.
// Then, when restore_it >= 0, the column's part of rtm_restore_kernel for the
// next reverse step: nothing else reads these cells before it.
// ZEROS = false: the column alone in shared memory, rows outside it by a test;
// for columns that fit there without the zeros only (the last 66 rows up to
// IMG_SMEM).
constexpr int HILB_HALF = 30;
constexpr int IMG_K = 3, IMG_THREADS = 128;
constexpr size_t IMG_SMEM = 227 * 1024;  // the most a CTA can have
// imaging of adjoint (lap vel3 R + FaQi), adjointPlane (FaQi of lap vel3),
// rtm_true (FaQi of the source field times vel3)
enum ImageMode { IMG_RTM = 0, IMG_PLANE = 1, IMG_TRUE = 2 };
template <bool ZEROS>
__global__ void __launch_bounds__(IMG_THREADS) rtm_image_kernel(
    const ShotDev *__restrict__ shots, const int2 *__restrict__ cols, int rot, int rot_b,
    const __grid_constant__ HilbertTaps taps, int mode, int restore_it) {
  extern __shared__ float2 sUR[];  // HILB_HALF zeros, the column, zeros
  constexpr int H = ZEROS ? HILB_HALF : 0;  // the column's first row
  const int2 c = cols[blockIdx.x];
  const ShotDev &g = shots[c.x];
  const int ix = c.y + g.pml, NZ = g.NZ;
  // reverse-pass naming: u2 = older (prev), u1 = current, u0 = newest
  const size_t col = (size_t)ix * g.LDZ;
  const float *u2 = g.fa[rot % 3] + col, *r0 = g.fb[(rot_b + 2) % 3] + col;
  float *u1 = g.fa[(rot + 1) % 3] + col, *u0 = g.fa[(rot + 2) % 3] + col;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (ZEROS) {
    for (int i = threadIdx.x; i < HILB_HALF; i += IMG_THREADS)
      sUR[i] = make_float2(0.0f, 0.0f);
    // up to a whole group of outputs past the last row
    for (int i = H + NZ + threadIdx.x; i < NZ + 2 * HILB_HALF + 2 * IMG_K; i += IMG_THREADS)
      sUR[i] = make_float2(0.0f, 0.0f);
  }
  // before the wait what no step of the pass writes: vel3 into the field's
  // place, the layers to be restored towards L2.  With one shot the kernel is a
  // chain of memory latencies: with these loads and the image's taken off it, a
  // reverse step of one 817 x 320 shot (two fields and imaging) takes 16.6 us
  // instead of 18.2.
  for (int iz = threadIdx.x; iz < NZ; iz += IMG_THREADS) {
    const float v = g.vel[col + iz];
    sUR[H + iz].x = 2.0f / (v * v * v);
  }
  const bool restore = restore_it >= 0 && restore_it < g.NT && restore_it >= g.ndel;
  const int edge = c.y < LAYERS ? c.y : c.y >= g.nx - LAYERS ? LAYERS + (g.nx - 1 - c.y) : -1;
  // the saved boundary layers of the sample; this thread's first cell of them
  const float *src = g.strips + (size_t)(restore ? restore_it - g.ndel : 0) * g.strip_len;
  const float *layer = edge >= 0 ? src + 2 * LAYERS * g.nx + edge * g.nz + threadIdx.x
                                 : src + threadIdx.x * g.nx + c.y;
  if (restore && threadIdx.x < (edge >= 0 ? g.nz : 2 * LAYERS))
    asm volatile("prefetch.global.L2 [%0];" ::"l"(layer));
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // this thread's first outputs, loaded beside the fields
  float *img0 = g.img + (size_t)c.y * g.nz;
  const int zq = 2 * IMG_K * (threadIdx.x >> 1) + (threadIdx.x & 1);
  float old[IMG_K];
#pragma unroll
  for (int k = 0; k < IMG_K; k++) old[k] = zq + 2 * k < g.nz ? img0[zq + 2 * k] : 0.0f;
  for (int iz = threadIdx.x; iz < NZ; iz += IMG_THREADS) {
    const float vel3 = sUR[H + iz].x;
    float u;
    if (mode == IMG_TRUE) {  // rtm_true images the source field itself, fd.cpp:1014
      u = u0[iz] * vel3;
    } else {
      const float lap = (u2[iz] + u0[iz] - 2.0f * u1[iz]) * g.idt2;
      u = lap * vel3;
    }
    sUR[H + iz] = make_float2(u, r0[iz]);
  }
  __syncthreads();
  const uint64_t nz = bits2(make_float2(IMG_NEG_ZERO, IMG_NEG_ZERO));
  for (int q = threadIdx.x; 2 * IMG_K * (q >> 1) + (q & 1) < g.nz; q += IMG_THREADS) {
    const int z0 = 2 * IMG_K * (q >> 1) + (q & 1);  // outputs z0, z0 + 2, ... (model rows)
    const int in0 = z0 + g.pml - 29;                 // their first input
    uint64_t acc[IMG_K];
#pragma unroll
    for (int k = 0; k < IMG_K; k++) acc[k] = 0;
    // input m (row z0 + pml - 29 + 2 m) meets output k at offset 2 (m - k) - 29,
    // tap h[30 - offset]; each output sums by increasing row
#pragma unroll
    for (int m = 0; m < HILB_HALF + IMG_K - 1; m++) {
      const int row = in0 + 2 * m;
      const uint64_t x = ZEROS || (row >= 0 && row < NZ) ? bits2(sUR[H + row]) : 0;
#pragma unroll
      for (int k = 0; k < IMG_K; k++) {
        const int n = m - k;
        if (n < 0 || n >= HILB_HALF) continue;
        const float h = taps.h[HILB_HALF - (2 * n - 29)];
        acc[k] = add2(acc[k], mul2(x, bits2(make_float2(h, h)), nz));
      }
    }
#pragma unroll
    for (int k = 0; k < IMG_K; k++) {
      const int z = z0 + 2 * k;
      if (z >= g.nz) break;
      const float2 ur = sUR[H + g.pml + z], f = pair2(acc[k]);
      const float was = q == threadIdx.x ? old[k] : img0[z];
      float a = mode == IMG_RTM ? was + ur.x * ur.y : was;  // the others image with FaQi alone
      a = a + 0.5f * (ur.x * ur.y - f.x * f.y);
      img0[z] = a;
    }
  }
  if (!restore) return;
  __syncthreads();  // the column's fields have been read
  // the source off the field that is the older one of the next step (a source
  // outside the model's columns: the first column's CTA, as no other reads it)
  const bool mine = ix == g.sxp || (c.y == 0 && (g.sxp < g.pml || g.sxp >= g.pml + g.nx));
  if (threadIdx.x == 0 && restore_it - 1 > 0 && mine) {
    const size_t off = (size_t)g.sxp * g.LDZ + g.szp;
    float *prev = g.fa[(rot + 1) % 3];
    prev[off] = prev[off] - coef(g.vel[off], g).vt2 * g.wav[restore_it - 1];
  }
  // the saved layers into the newest field
  if (edge >= 0) {
    for (int z = threadIdx.x; z < g.nz; z += IMG_THREADS)
      u0[g.pml + z] = layer[z - (int)threadIdx.x];
  } else if (threadIdx.x < 2 * LAYERS) {
    const int l = threadIdx.x;
    u0[l < LAYERS ? g.pml + l : g.nz + g.pml - 1 - (l - LAYERS)] = *layer;
  }
}

// adjointUpDown imaging (fd.cpp:501-521), one CTA per interior column: with
// S the source field of the wavelet, St that of its Hilbert transform (the
// shadow shot table) and R the receiver field, each with its 61-tap z-Hilbert
// transform over the padded column,
//   comp0 += S R, comp1 += H[S] H[R], comp2 += St H[R], comp3 += H[St] R.
__global__ void updown_image_kernel(const ShotDev *__restrict__ shots,
                                    const ShotDev *__restrict__ shots_h,
                                    const int2 *__restrict__ cols, int rot, int rot_b,
                                    const float *__restrict__ taps) {
  extern __shared__ float sh[];
  const int2 c = cols[blockIdx.x];
  const ShotDev &g = shots[c.x];
  const ShotDev &gh = shots_h[c.x];
  const int ix = c.y + g.pml, NZ = g.NZ;
  float *sS = sh, *sR = sh + NZ, *sT = sh + 2 * NZ;
  __shared__ float h[2 * HILB_HALF + 1];
  if (threadIdx.x < 2 * HILB_HALF + 1) h[threadIdx.x] = taps[threadIdx.x];
  const size_t col = (size_t)ix * g.LDZ;
  const float *S = g.fa[(rot + 2) % 3] + col, *T = gh.fa[(rot + 2) % 3] + col;
  const float *R = g.fb[(rot_b + 2) % 3] + col;
  for (int iz = threadIdx.x; iz < NZ; iz += blockDim.x) {
    sS[iz] = S[iz];
    sR[iz] = R[iz];
    sT[iz] = T[iz];
  }
  __syncthreads();
  const size_t plane = (size_t)g.nx * g.nz;
  for (int iz = g.pml + threadIdx.x; iz < NZ - g.pml; iz += blockDim.x) {
    const int i0 = max(iz - HILB_HALF, 0), i1 = min(iz + HILB_HALF, NZ - 1);
    float hs = 0.0f, hr = 0.0f, ht = 0.0f;
    const int start = i0 + (((iz - i0) & 1) ? 0 : 1);  // odd offsets: even taps are zero
    for (int i = start; i <= i1; i += 2) {
      const float hk = h[iz - i + HILB_HALF];
      hs = hs + sS[i] * hk;
      hr = hr + sR[i] * hk;
      ht = ht + sT[i] * hk;
    }
    float *cp = g.comp + (size_t)c.y * g.nz + (iz - g.pml);
    cp[0] = cp[0] + sS[iz] * sR[iz];
    cp[plane] = cp[plane] + hs * hr;
    cp[2 * plane] = cp[2 * plane] + sT[iz] * hr;
    cp[3 * plane] = cp[3 * plane] + ht * sR[iz];
  }
}

// img = comp0 - comp1 + comp3 + comp2 (fd.cpp:538-547)
__global__ void updown_finalize_kernel(const ShotDev *__restrict__ shots) {
  const ShotDev &g = shots[blockIdx.y];
  const size_t n = (size_t)g.nx * g.nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    g.img[i] = g.comp[i] - g.comp[n + i] + g.comp[3 * n + i] + g.comp[2 * n + i];
}

// Exact adjoint, last step: img = vt2 vel3 grad on the model interior (the
// scattering source is vt2 lap vel3 dv, fd.cpp:138-139; dv is zero-padded).
__global__ void finalize_image_kernel(const ShotDev *__restrict__ shots) {
  const ShotDev &g = shots[blockIdx.y];
  const int n = g.nx * g.nz;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int x = i / g.nz, z = i - x * g.nz;
    float v = g.vel[(size_t)(x + g.pml) * g.LDZ + (z + g.pml)];
    float vt2 = coef(v, g).vt2;
    float vel3 = 2.0f / (v * v * v);
    g.img[i] = (float)((double)(vt2 * vel3) * g.grad[image_index(g.nz, g.pml, x, z + g.pml)]);
  }
}

}  // namespace

cudaError_t launch_finalize_image(const ShotDev *d_shots, int nshots, cudaStream_t s) {
  dim3 grid(64, nshots);
  finalize_image_kernel<<<grid, 256, 0, s>>>(d_shots);
  return cudaGetLastError();
}

cudaError_t configure_kernels() {
  cudaError_t e = exact::configure();
  return e == cudaSuccess ? fast::configure() : e;
}

cudaError_t launch_step(int mode, bool use_exact, const ShotDev *d_shots, const Tile *d_tiles,
                        int n_int, int n_pad, int shape, const StepArgs &a, int *d_err,
                        cudaStream_t s_int, cudaStream_t s_pad) {
  return use_exact ? exact::launch_step(mode, d_shots, d_tiles, n_int, n_pad, shape, a, d_err,
                                        s_int, s_pad)
                   : fast::launch_step(mode, d_shots, d_tiles, n_int, n_pad, shape, a, d_err,
                                       s_int, s_pad);
}

cudaError_t launch_pair(bool use_exact, const ShotDev *d_shots, const Tile *d_tiles, int n_int,
                        int n_pad, int shape, const StepArgs &a, int *d_err, cudaStream_t s) {
  return use_exact ? exact::launch_pair(d_shots, d_tiles, n_int, n_pad, shape, a, d_err, s)
                   : fast::launch_pair(d_shots, d_tiles, n_int, n_pad, shape, a, d_err, s);
}

bool step_splits(int mode, bool use_exact, int n_int, int shape, int loop) {
  return use_exact ? exact::step_splits(mode, n_int, shape, loop)
                   : fast::step_splits(mode, n_int, shape, loop);
}

cudaError_t launch_pad_tab(bool use_exact, const ShotDev *d_shots, int nshots, int max_len,
                           int born, cudaStream_t s) {
  return use_exact ? exact::launch_pad_tab(d_shots, nshots, max_len, born, s)
                   : fast::launch_pad_tab(d_shots, nshots, max_len, born, s);
}

cudaError_t launch_pad(const float *d_src, int nx, int nz, int pml, int LDZ, int clamp,
                       float *d_dst, cudaStream_t s) {
  size_t n = (size_t)(nx + 2 * pml) * (nz + 2 * pml);
  int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
  pad_kernel<<<blocks, 256, 0, s>>>(d_src, nx, nz, pml, LDZ, clamp, d_dst);
  return cudaGetLastError();
}

cudaError_t launch_transpose(const float *d_src, int rows, int cols, float *d_dst,
                             cudaStream_t s) {
  dim3 grid((cols + 31) / 32, (rows + 31) / 32), block(32, 8);
  transpose_kernel<<<grid, block, 0, s>>>(d_src, rows, cols, d_dst);
  return cudaGetLastError();
}

cudaError_t launch_rtm_restore(const ShotDev *d_shots, int nshots, int max_strip, int rot,
                               int it, cudaStream_t s) {
  dim3 grid((max_strip + 255) / 256, nshots);
  rtm_restore_kernel<<<grid, 256, 0, s>>>(d_shots, nshots, rot, it);
  return cudaGetLastError();
}

template <bool ZEROS>
static cudaError_t launch_rtm_image_z(const ShotDev *d_shots, const int2 *d_cols, int ncols,
                                      int rot, int rot_b, size_t smem, const HilbertTaps &taps,
                                      cudaStream_t s, int mode, int restore_it, int pdl) {
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(rtm_image_kernel<ZEROS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)std::max(smem, IMG_SMEM));
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(ncols);
  c.blockDim = dim3(IMG_THREADS);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&c, rtm_image_kernel<ZEROS>, d_shots, d_cols, rot, rot_b, taps, mode,
                            restore_it);
}
cudaError_t launch_rtm_image(const ShotDev *d_shots, const int2 *d_cols, int ncols, int rot,
                             int rot_b, int max_nz, const HilbertTaps &taps, cudaStream_t s,
                             int mode, int restore_it, int pdl) {
  const size_t column = (size_t)max_nz * sizeof(float2);
  const size_t zeros = (2 * HILB_HALF + 2 * IMG_K) * sizeof(float2);
  return column + zeros <= IMG_SMEM
             ? launch_rtm_image_z<true>(d_shots, d_cols, ncols, rot, rot_b, column + zeros, taps, s,
                                        mode, restore_it, pdl)
             : launch_rtm_image_z<false>(d_shots, d_cols, ncols, rot, rot_b, column, taps, s, mode,
                                         restore_it, pdl);
}

cudaError_t launch_updown_image(const ShotDev *d_shots, const ShotDev *d_shots_h,
                                const int2 *d_cols, int ncols, int rot, int rot_b, int max_nz,
                                const float *d_taps, cudaStream_t s) {
  size_t smem = 3 * (size_t)max_nz * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(updown_image_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  updown_image_kernel<<<ncols, 256, smem, s>>>(d_shots, d_shots_h, d_cols, rot, rot_b, d_taps);
  return cudaGetLastError();
}

cudaError_t launch_updown_finalize(const ShotDev *d_shots, int nshots, cudaStream_t s) {
  dim3 grid(64, nshots);
  updown_finalize_kernel<<<grid, 256, 0, s>>>(d_shots);
  return cudaGetLastError();
}

cudaError_t launch_plane_rcv_prep(const ShotDev *d_shots, int nshots, int max_strip, int rot_b,
                                  int strip_k, int rec_k, cudaStream_t s) {
  dim3 grid((max_strip + 255) / 256, nshots);
  plane_rcv_prep_kernel<<<grid, 256, 0, s>>>(d_shots, nshots, rot_b, strip_k, rec_k);
  return cudaGetLastError();
}

}  // namespace seis
