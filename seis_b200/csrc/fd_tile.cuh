// Time-step kernels of the 2-D acoustic FD engine (sm_100a).
//
// The tile list of a batch holds two kinds of tiles: interior tiles, whose every
// cell is a model cell in the 8th-order region, where the absorbing blend is
// the identity (w = 1, u31 = 0; src/util/fd.cpp:55-56), and pad tiles, every
// other.  A pad tile is one pass: the two-way update, injection, the two-way
// values of the tile and a one-cell halo kept in shared memory, then the
// one-way update and blend of the pad cells (processBoundary,
// fd.cpp:1092-1179).  One step is one launch of
//  * step_tile_kernel<S, MODE>, one tile per CTA,
// or, with many interior tiles, that kernel over the pad tiles beside
//  * interior_loop_kernel<S, MODE>: persistent CTAs, each taking every G-th
//    interior tile through two shared-memory stages (the tensor copies of the
//    next tile in flight while the current one is computed).
// Tiles are TX x TZ cells (shape S); arrays are staged by 2-D TMA tensor
// copies into shared memory (mbarriers, bounded waits, no multicast); each
// thread owns a 4-row x 2-column micro-tile.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "fd_cell.cuh"

namespace seis {
namespace SEIS_NS {

// Geometry of tile shape S (TileShapeId).
template <int S>
struct Geo {
  static constexpr int TX = shape_tx(S), TZ = shape_tz(S);
  static constexpr int NT = TX * TZ / 8;       // threads per CTA
  static constexpr int QZ = TZ / 4;            // row quads per column
  static constexpr int SR = TZ + 2 * ZM;       // staged rows per column
  static constexpr int CW_C = TX + 2 * HXC;    // staged columns of the current fields
  static constexpr int CW_P = TX + 2;          // staged columns of the other arrays
  static constexpr int U3C = TX + 2;           // pad tiles: two-way values of tile + halo
  static constexpr int U3R = TZ + 8;
  static constexpr int U3N = U3C * U3R;
  static constexpr int NHALO = 2 * (TX + 2) + 2 * TZ;  // halo ring cells of a tile
  static_assert(NT % 32 == 0 && NT <= 1024, "whole warps");
  static_assert(NT * sizeof(int) >= sizeof(ShotDev), "one thread per word of the shot table");
};
// Local names for the geometry of shape S inside a kernel or device function.
#define SEIS_GEO(S)                                                                   \
  using G_ = Geo<S>;                                                                  \
  constexpr int TX = G_::TX, TZ = G_::TZ, NT_T = G_::NT, QZ = G_::QZ, SR = G_::SR;    \
  constexpr int CW_C = G_::CW_C, CW_P = G_::CW_P;                                     \
  (void)TX; (void)TZ; (void)NT_T; (void)QZ; (void)SR; (void)CW_C; (void)CW_P

// CTAs per SM that a kernel's shared memory allows (227 KB per SM, 1 KB
// reserved per CTA), at most `cap`.
constexpr int ctas_fit(size_t bytes, int cap) {
  return (int)((227 * 1024) / (bytes + 1024)) < cap ? (int)((227 * 1024) / (bytes + 1024)) : cap;
}

// ---- PTX helpers: mbarrier + bulk asynchronous copy global -> shared
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int c0, int c1,
                                            uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}
// untiled copy: both addresses 16-byte aligned, a multiple of 16 bytes
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void prefetch_map(const CUtensorMap *m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, "
      "0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after WAIT_LIMIT polls (each poll may suspend the
// thread for a short hardware-defined time).
constexpr int WAIT_LIMIT = 1 << 21;
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  for (int i = 0; i < WAIT_LIMIT; i++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ float comp(const float4 &v, int r) {
  return r == 0 ? v.x : (r == 1 ? v.y : (r == 2 ? v.z : v.w));
}
__device__ __forceinline__ void set_comp(float4 &v, int r, float x) {
  if (r == 0) v.x = x; else if (r == 1) v.y = x; else if (r == 2) v.z = x; else v.w = x;
}

// Accessor of one staged array by padded-grid coordinates (SR staged rows
// per column).
template <int SR>
struct SAT {
  const float *s;  // staged column x0h, row z0m
  int x0h, z0m;    // first staged column and row (the tile's origin less the halo)
  __device__ __forceinline__ float operator()(int ix, int iz) const {
    return s[(ix - x0h) * SR + (iz - z0m)];
  }
  __device__ __forceinline__ float4 quad(int ix, int iz) const {
    return *reinterpret_cast<const float4 *>(s + (ix - x0h) * SR + (iz - z0m));
  }
};

// Injection into the two-way value before the absorbing step: point source
// into field A (fd.cpp:49-51), or receiver data rec*vt2 in receiver mode
// (fd.cpp:673-677).  `gzc` = padded receiver row of the column (-1: none).
template <int MODE>
__device__ __forceinline__ float inject(const ShotDev &g, const StepArgs &a, int ix, int iz,
                                        int gzc, float u3, float vt2) {
  if (MODE != MODE_RCV) {
    if (a.src_k >= 0) {
      if (g.sou) {  // areal source of forwordPlane, fd.cpp:221-225
        if (iz == g.szp && ix >= g.pml && ix < g.pml + g.nx)
          u3 = u3 + vt2 * g.sou[(size_t)a.src_k * g.nx + (ix - g.pml)];
      } else if (ix == g.sxp && iz == g.szp) {
        u3 = u3 + vt2 * g.wav[a.src_k];
      }
    }
  } else if (a.rec_k >= 0 && gzc >= 0) {
    const float r = g.rec[(size_t)a.rec_k * g.nx + (ix - g.pml)];
    if (!g.rcv_dipole) {
      if (iz == gzc) u3 = u3 + r * vt2;
    } else if (iz == gzc) {  // rtm_true, fd.cpp:1003-1008
      u3 = u3 - r * vt2 / g.dz;
    } else if (iz == gzc + 1) {
      u3 = u3 + r * vt2 / g.dz;
    }
  }
  return u3;
}

// Boundary strips per sample: [top 4 x nx][bottom 4 x nx][left 4 x nz]
// [right 4 x nz] (SaveAtBoundary, fd.cpp:1183-1203); a cell can sit in several
// strips when the model is thin.
__device__ __forceinline__ void save_strips(const ShotDev &g, int strip_k, int ix, int iz,
                                            float out) {
  const int x = ix - g.pml, z = iz - g.pml;
  float *dst = g.strips + (size_t)strip_k * g.strip_len;
  if (x >= 0 && x < g.nx) {
    int lt = z, lb = g.nz - 1 - z;
    if (lt >= 0 && lt < LAYERS) dst[lt * g.nx + x] = out;
    if (lb >= 0 && lb < LAYERS) dst[(LAYERS + lb) * g.nx + x] = out;
  }
  if (z >= 0 && z < g.nz) {
    const int base = 2 * LAYERS * g.nx;
    int ll = x, lr = g.nx - 1 - x;
    if (ll >= 0 && ll < LAYERS) dst[base + ll * g.nz + z] = out;
    if (lr >= 0 && lr < LAYERS) dst[base + (LAYERS + lr) * g.nz + z] = out;
  }
}

// ---- Four rows of a column as two packed pairs (rows 0, 1 and 2, 3): the
// add, multiply and fused multiply-add of a pair are one instruction each and
// round every element as the scalar operation does, so the issue slots of the
// stencil's arithmetic halve and its results stay the same bits.
//
// The assembler contracts a packed multiply that feeds a packed add into one
// fused operation, whatever the rounding qualifiers and switches say.  It
// cannot do that to a fused multiply-add of an unknown addend: a product that
// is rounded by itself (*) is x y + (-0), the zero read from constant memory;
// what the contracted build fuses is written fused (madd, msub).
struct V4 {
  float2 a, b;
};
__device__ __forceinline__ V4 v4(const float4 &q) {
  return V4{make_float2(q.x, q.y), make_float2(q.z, q.w)};
}
__device__ __forceinline__ V4 v4(float x) { return V4{make_float2(x, x), make_float2(x, x)}; }
__device__ __forceinline__ float4 f4(const V4 &v) {
  return make_float4(v.a.x, v.a.y, v.b.x, v.b.y);
}
__device__ __forceinline__ uint64_t bits2(const float2 &x) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x.x), "f"(x.y));
  return r;
}
__device__ __forceinline__ float2 pair2(uint64_t r) {
  float2 x;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x.x), "=f"(x.y) : "l"(r));
  return x;
}
__device__ __forceinline__ float2 add2(const float2 &x, const float2 &y) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits2(x)), "l"(bits2(y)));
  return pair2(r);
}
__device__ __forceinline__ float2 fma2(const float2 &x, const float2 &y, const float2 &z) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(bits2(x)), "l"(bits2(y)), "l"(bits2(z)));
  return pair2(r);
}
__constant__ float NEG_ZERO = -0.0f;
__device__ __forceinline__ V4 operator+(const V4 &x, const V4 &y) {
  return V4{add2(x.a, y.a), add2(x.b, y.b)};
}
__device__ __forceinline__ V4 operator*(const V4 &x, const V4 &y) {
  const float2 z = make_float2(NEG_ZERO, NEG_ZERO);
  return V4{fma2(x.a, y.a, z), fma2(x.b, y.b, z)};
}
__device__ __forceinline__ V4 operator*(const V4 &x, float y) { return x * v4(y); }
__device__ __forceinline__ V4 fma4(const V4 &x, const V4 &y, const V4 &z) {
  return V4{fma2(x.a, y.a, z.a), fma2(x.b, y.b, z.b)};
}
// x - y, -x: the product with -1 is exact
__device__ __forceinline__ V4 operator-(const V4 &x, const V4 &y) { return fma4(y, v4(-1.0f), x); }
__device__ __forceinline__ V4 operator-(const V4 &x) { return x * v4(-1.0f); }
__device__ __forceinline__ V4 operator/(const V4 &x, const V4 &y) {
  return V4{make_float2(x.a.x / y.a.x, x.a.y / y.a.y), make_float2(x.b.x / y.b.x, x.b.y / y.b.y)};
}
// z + 2 x, z - 2 x.  The doubling is exact, so the fused form rounds once as
// the separate one does; only where 2 x overflows by itself do they part: the
// exact build doubles first, as the reference does.
__device__ __forceinline__ V4 add_twice(const V4 &z, const V4 &x) {
#ifdef SEIS_FAST_MATH
  return fma4(x, v4(2.0f), z);
#else
  return z + (x + x);
#endif
}
__device__ __forceinline__ V4 sub_twice(const V4 &z, const V4 &x) {
#ifdef SEIS_FAST_MATH
  return fma4(x, v4(-2.0f), z);
#else
  return z - (x + x);
#endif
}
// z + x y and z - x y as the build rounds them
__device__ __forceinline__ V4 madd(const V4 &x, const V4 &y, const V4 &z) {
#ifdef SEIS_FAST_MATH
  return fma4(x, y, z);
#else
  return z + x * y;
#endif
}
__device__ __forceinline__ V4 madd(const V4 &x, float y, const V4 &z) { return madd(x, v4(y), z); }
__device__ __forceinline__ V4 msub(const V4 &x, const V4 &y, const V4 &z) {
#ifdef SEIS_FAST_MATH
  return fma4(-x, y, z);
#else
  return z - x * y;
#endif
}
// rows one below / above a quad (e: the row after its last / before its first)
__device__ __forceinline__ float4 shift_dn(const float4 &q, float e) {
  return make_float4(q.y, q.z, q.w, e);
}
__device__ __forceinline__ float4 shift_up(const float4 &q, float e) {
  return make_float4(e, q.x, q.y, q.z);
}

// lap8 of a quad from its nine taps, in the order of lap8
__device__ __forceinline__ V4 lap8_quad(const V4 &m4, const V4 &m3, const V4 &m2, const V4 &m1,
                                        const V4 &c, const V4 &p1, const V4 &p2, const V4 &p3,
                                        const V4 &p4) {
  V4 s = m4 * SEIS_C0;
  s = madd(m3, SEIS_C1, s);
  s = madd(m2, SEIS_C2, s);
  s = madd(m1, SEIS_C3, s);
  s = madd(c, SEIS_C4, s);
  s = madd(p1, SEIS_C3, s);
  s = madd(p2, SEIS_C2, s);
  s = madd(p3, SEIS_C1, s);
  return madd(p4, SEIS_C0, s);
}
// the same along z: taps of rows iz0 .. iz0+3 from the quads above, at and
// below
__device__ __forceinline__ V4 lap8_along(const float4 &za, const float4 &zb, const float4 &zc) {
  const float z[12] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w, zc.x, zc.y, zc.z, zc.w};
  V4 t[9];
#pragma unroll
  for (int k = 0; k < 9; k++)
    t[k] = V4{make_float2(z[k], z[k + 1]), make_float2(z[k + 2], z[k + 3])};
  return lap8_quad(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8]);
}
struct Coef4 {
  V4 vt2, vz, vx;
};
__device__ __forceinline__ Coef4 coef4(const float4 &v, const ShotDev &g) {
  const V4 t = v4(v) * g.dt;
  Coef4 c;
  c.vt2 = t * t;
  c.vz = c.vt2 * g.invdz2;
  c.vx = c.vt2 * g.invdx2;
  return c;
}

// The second differences of two columns x 4 rows, 8th order (fd.cpp:1259-1268):
// along z of the field CZ and along x of the field CX (the same one, except in
// the adjoint), from shared memory: 14 quads for 8 cells.  `cen`: CX's quads.
template <class SC>
__device__ __forceinline__ void pair_sums(const SC &CZ, const SC &CX, int ix, int iz0, V4 (&uzz)[2],
                                          V4 (&uxx)[2], float4 (&cen)[2]) {
  // both columns' sums along x as the window's ten columns go by: one quad of
  // it live at a time
  constexpr float W[9] = {SEIS_C0, SEIS_C1, SEIS_C2, SEIS_C3, SEIS_C4,
                          SEIS_C3, SEIS_C2, SEIS_C1, SEIS_C0};
#pragma unroll
  for (int m = 0; m < 10; m++) {
    const float4 q = CX.quad(ix - 4 + m, iz0);
    const V4 x = v4(q);
    if (m == 0) uxx[0] = x * W[0];
    if (m == 1) uxx[1] = x * W[0];
    if (m >= 1 && m <= 8) uxx[0] = madd(x, W[m], uxx[0]);
    if (m >= 2) uxx[1] = madd(x, W[m - 1], uxx[1]);
    if (m == 4 || m == 5) cen[m - 4] = q;
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const float4 zc = &CZ == &CX ? cen[j] : CZ.quad(ix + j, iz0);
    uzz[j] = lap8_along(CZ.quad(ix + j, iz0 - 4), zc, CZ.quad(ix + j, iz0 + 4));
  }
}

// Two-way update of two columns x 4 rows: u3 = vvzz uzz + vvxx uxx + 2 cur -
// prev, 8th order (fd.cpp:1259-1270) and, for the rows of `low`, 2nd order
// (:1226-1241); the previous field and the velocity in registers.
template <class SC>
__device__ __forceinline__ void pair_twoway(const SC &C, const ShotDev &g, int ix, int iz0,
                                            const float4 (&prv)[2], const float4 (&vel)[2],
                                            float4 (&out)[2], float4 (&cen)[2],
                                            unsigned low0 = 0u, unsigned low1 = 0u) {
  V4 uzz[2], uxx[2];
  pair_sums(C, C, ix, iz0, uzz, uxx, cen);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const Coef4 k = coef4(vel[j], g);
    out[j] = f4(add_twice(madd(k.vz, uzz[j], k.vx * uxx[j]), v4(cen[j])) - v4(prv[j]));
    const unsigned low = j ? low1 : low0;
    if (low) {
      const V4 c = v4(cen[j]);
      const V4 lzz = sub_twice(v4(shift_up(cen[j], C(ix + j, iz0 - 1))) +
                                   v4(shift_dn(cen[j], C(ix + j, iz0 + 4))), c);
      const V4 lxx = sub_twice(v4(C.quad(ix + j + 1, iz0)) + v4(C.quad(ix + j - 1, iz0)), c);
      const float4 l = f4(add_twice(madd(k.vz, lzz, k.vx * lxx), c) - v4(prv[j]));
#pragma unroll
      for (int r = 0; r < 4; r++)
        if ((low >> r) & 1u) set_comp(out[j], r, comp(l, r));
    }
  }
}

#ifndef SEIS_FAST_MATH
// x in [2^LO, 2^60] in magnitude
template <int LO>
__device__ __forceinline__ bool in_range(float x) {
  const uint32_t lo = (uint32_t)(127 + LO) << 23, hi = (127u + 60u) << 23;
  return (__float_as_uint(x) & 0x7fffffffu) - lo <= hi - lo;
}
// n / d given rd = 1 / d rounded to nearest (1 <= d <= 2^30), for quotients
// that the correction below cannot reach: a numerator below 2^-60 is divided
// scaled by 2^90, where nothing underflows, and the quotient scaled back.
// Below 2^-126 that rounds a second time; where the first rounding ended
// half way between two results, the remainder's sign tells which side the
// quotient lies on.
__device__ __forceinline__ float quot_small(float n, float d, float rd, bool &ok) {
  const bool t = fabsf(n) < 0x1p-60f;
  const float N = n * (t ? 0x1p90f : 1.0f);
  float q = N * rd;
  ok = ok && (in_range<-100>(q) || n == 0.0f);
  q = fmaf(fmaf(q, -d, N), rd, q);
  q = fmaf(fmaf(q, -d, N), rd, q);
  float o = q * (t ? 0x1p-90f : 1.0f);
  const float e = fmaf(o, 0x1p90f, -q), rem = fmaf(q, -d, N);
  if (t && fabsf(q) < 0x1p-36f && fabsf(e) == 0x1p-60f && rem != 0.0f)
    o = (q + copysignf(0x1p-60f, rem)) * 0x1p-90f;
  return n == 0.0f ? n : o;  // the sign of zero
}
// n / d of four rows given rd = 1 / d rounded to nearest: Markstein's
// correction of an approximate quotient by its fused remainder (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990), which rounds correctly where nothing underflows or
// overflows (1 <= d <= 2^30: from quotients of 2^-100 up), quads with smaller
// quotients by quot_small; others (and zero reciprocals, see ptab) divide.
// Four quotients without a branch each: the plain division tests every operand
// and takes its slow path for a zero or tiny numerator, which is every pad
// cell that the wave has not reached, and those just ahead of it: the pad
// tiles that the front was crossing took 12,000 cycles for this phase instead
// of 4,000, and a step waits for its slowest tile.
__device__ __forceinline__ float4 quot_quad(const V4 &n, const V4 &d, const V4 &rd) {
  const V4 q0 = n * rd;
  const float4 q = f4(q0), N = f4(n);
  if ((in_range<-100>(q.x) || N.x == 0.0f) && (in_range<-100>(q.y) || N.y == 0.0f) &&
      (in_range<-100>(q.z) || N.z == 0.0f) && (in_range<-100>(q.w) || N.w == 0.0f)) {
    const V4 m = d * -1.0f;
    const V4 q1 = fma4(fma4(q0, m, n), rd, q0);
    float4 r = f4(fma4(fma4(q1, m, n), rd, q1));
    if (N.x == 0.0f) r.x = N.x;  // the sign of zero
    if (N.y == 0.0f) r.y = N.y;
    if (N.z == 0.0f) r.z = N.z;
    if (N.w == 0.0f) r.w = N.w;
    return r;
  }
  const float4 D = f4(d), R = f4(rd);
  bool ok = true;
  float4 r;
#pragma unroll
  for (int k = 0; k < 4; k++) set_comp(r, k, quot_small(comp(N, k), comp(D, k), comp(R, k), ok));
  return ok ? r : f4(n / d);
}
#endif
// 2 / x of four rows: the hardware's approximate reciprocal and two Newton
// steps with fused residuals (Markstein, as above: correctly rounded; equal to
// the division for every mantissa), doubled exactly.
#ifndef SEIS_FAST_MATH
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#endif
__device__ __forceinline__ V4 two_over(const V4 &x_) {
#ifndef SEIS_FAST_MATH
  const float4 x = f4(x_);
  if (in_range<-60>(x.x) && in_range<-60>(x.y) && in_range<-60>(x.z) && in_range<-60>(x.w)) {
    const V4 m = x_ * -1.0f, one = v4(1.0f);
    V4 y = v4(make_float4(rcp_approx(x.x), rcp_approx(x.y), rcp_approx(x.z), rcp_approx(x.w)));
    y = fma4(fma4(m, y, one), y, y);
    y = fma4(fma4(m, y, one), y, y);
    return y + y;
  }
#endif
  return v4(2.0f) / x_;
}

// Second time difference of the background field over dt^2 (fd.cpp:134-139)
// and the scattering source vt2 lap vel3 dv of a quad
__device__ __forceinline__ float4 second_diff(const float4 &out, const float4 &prv,
                                              const float4 &cen, const ShotDev &g) {
  return f4(sub_twice(v4(out) + v4(prv), v4(cen)) * g.idt2);
}
__device__ __forceinline__ float4 scatter_source(const float4 &vel, const float4 &lap,
                                                 const float4 &dv, const ShotDev &g) {
  const V4 v = v4(vel), t = v * g.dt;
  return f4(t * t * v4(lap) * two_over(v * v * v) * v4(dv));
}
__device__ __forceinline__ float4 add4(const float4 &x, const float4 &y) { return f4(v4(x) + v4(y)); }

// Write this thread's source-term values (lap of the background field) of
// snapshot `k`: two column quads (columns ix, ix + 1 from row iz0), the rows of
// mask[j], zero in a quad's other rows.  BF16 / FP16 snapshots carry one
// power-of-two scale per (snapshot, tile), taken from the tile's largest
// magnitude so that the scaled values lie in [0.5, 1).  Every thread of the CTA
// calls this (it holds block barriers).
template <int NTH, int TX, int TZ>
__device__ __forceinline__ void snap_write(const ShotDev &g, int k, int x0, int z0, int ix, int iz0,
                                           float4 (&v)[2], const unsigned (&mask)[2], float *red) {
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int r = 0; r < 4; r++)
      if (!((mask[j] >> r) & 1u)) set_comp(v[j], r, 0.0f);
  float scale = 1.0f;
  if (g.snap_dtype != SNAP_F32) {
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int r = 0; r < 4; r++) m = fmaxf(m, fabsf(comp(v[j], r)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = m;
    __syncthreads();
    m = 0.0f;
#pragma unroll
    for (int w = 0; w < NTH / 32; w++) m = fmaxf(m, red[w]);
    int e = 0;
    frexpf(m, &e);
    // tiny (denormal) maxima would overflow the scale: clamp to 2^126
    scale = m > 0.0f ? ldexpf(1.0f, min(-e, 126)) : 1.0f;
    if (threadIdx.x == 0) {
      const int ntx = (g.NX + TX - 1) / TX;
      g.snap_scale[(size_t)k * ntx * g.ntz + (x0 / TX) * g.ntz + z0 / TZ] = scale;
    }
    __syncthreads();
  }
  const size_t base = (size_t)k * g.nx * image_ld(g.nz, g.pml);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    if (!mask[j]) continue;
    const size_t i = base + image_index(g.nz, g.pml, ix + j - g.pml, iz0);
    const float4 q = make_float4(v[j].x * scale, v[j].y * scale, v[j].z * scale, v[j].w * scale);
    if (g.snap_dtype == SNAP_F32) {
      *reinterpret_cast<float4 *>(reinterpret_cast<float *>(g.snap) + i) = q;
    } else {
      uint2 h;
      if (g.snap_dtype == SNAP_BF16) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(q.x, q.y), hi = __floats2bfloat162_rn(q.z, q.w);
        h.x = *reinterpret_cast<const uint32_t *>(&lo);
        h.y = *reinterpret_cast<const uint32_t *>(&hi);
      } else {
        const __half2 lo = __floats2half2_rn(q.x, q.y), hi = __floats2half2_rn(q.z, q.w);
        h.x = *reinterpret_cast<const uint32_t *>(&lo);
        h.y = *reinterpret_cast<const uint32_t *>(&hi);
      }
      *reinterpret_cast<uint2 *>(reinterpret_cast<unsigned short *>(g.snap) + i) = h;
    }
  }
}

// Global-memory accessor of one field by padded-grid coordinates.
struct GA {
  const float *p;  // cell (0, 0)
  int ldz;
  __device__ __forceinline__ float operator()(int ix, int iz) const {
    return __ldg(p + (size_t)ix * ldz + iz);
  }
};

// i / len given r = 1 / len as the build divides (within two units in the last
// place), for i < 2^13: (i + 0.5) / len lies at least 0.5 / len from an integer,
// the rounded product within 2^13 / len * 2^-21 = 2^-8 / len of it.
__device__ __forceinline__ int quot(int i, float r) { return (int)(((float)i + 0.5f) * r); }

// Two-way values of a pad tile and its one-cell halo in shared memory:
// columns x0-1 .. x0+TX, rows z0-4 .. z0+TZ+3 (U3R = TZ + 8 rows per column;
// the tile's row quads stay 16-byte aligned; only rows z0-1 .. z0+TZ are
// used).
template <int U3R>
struct UAT {
  float *s;
  int x0, z0;
  __device__ __forceinline__ float &ref(int ix, int iz) const {
    return s[(ix - x0 + 1) * U3R + (iz - z0 + 4)];
  }
  __device__ __forceinline__ float operator()(int ix, int iz) const { return ref(ix, iz); }
  __device__ __forceinline__ float4 quad(int ix, int iz) const {
    return *reinterpret_cast<const float4 *>(&ref(ix, iz));
  }
};
// Halo cell i of the tile at (x0, z0): the rows above and below the tile
// (TX + 2 cells each, corners included), then the columns left and right.
template <int TX, int TZ>
__device__ __forceinline__ void halo_cell(int i, int x0, int z0, int &hx, int &hz) {
  if (i < 2 * (TX + 2)) {
    hx = x0 - 1 + i % (TX + 2);
    hz = i < TX + 2 ? z0 - 1 : z0 + TZ;
  } else {
    const int j = i - 2 * (TX + 2);
    hx = j < TZ ? x0 - 1 : x0 + TX;
    hz = z0 + j % TZ;
  }
}

// Row quads [4q, 4q + 3] of a tile's columns that hold at least one grid cell
// outside a rectangle [rx0, rx1) x [rz0, rz1) (the model, or the model less its
// edge cells), enumerated column by column, rows fastest, so that the threads
// of a CTA can share them evenly (indices by quot).
struct QuadList {
  int x0, xe;      // tile columns inside the grid
  int ma, mb;      // tile columns crossing the model: [ma, mb)
  int top, bot;    // quads of such a column from the top / from the bottom
  int cp, cm, n;   // quads per other column, per crossing column, in all
  float rcp, rcm;
  __device__ __forceinline__ QuadList(int x0_, int z0, int xe_, int ze, int rx0, int rx1, int rz0,
                                      int rz1)
      : x0(x0_), xe(xe_) {
    ma = min(max(rx0, x0), xe);
    mb = min(max(rx1, ma), xe);
    cp = (ze - z0 + 3) / 4;
    top = min(max(0, (min(ze, rz0) - z0 + 3) / 4), cp);
    bot = rz1 < ze ? cp - max(0, rz1 - z0) / 4 : 0;
    if (top + bot > cp) top = cp, bot = 0;
    cm = top + bot;
    n = (xe - x0 - (mb - ma)) * cp + (mb - ma) * cm;
    rcp = cp > 0 ? 1.0f / (float)cp : 0.0f;
    rcm = cm > 0 ? 1.0f / (float)cm : 0.0f;
  }
  // quad i: its column and its first row's offset from the tile
  __device__ __forceinline__ void quad(int i, int &cx, int &dz) const {
    const int na = (ma - x0) * cp;
    int base = x0, q;
    if (i >= na) {
      i -= na;
      const int nm = (mb - ma) * cm;
      if (i < nm) {
        q = quot(i, rcm);
        cx = ma + q;
        const int r = i - q * cm;
        dz = 4 * (r < top ? r : cp - bot + (r - top));
        return;
      }
      i -= nm;
      base = mb;
    }
    q = quot(i, rcp);
    cx = base + q;
    dz = 4 * (i - q * cp);
  }
};

// One-way update of a quad (fd.cpp:1098-1104 and its mirrors), in the order
// of oneway
__device__ __forceinline__ float4 oneway_quad(float a1, const V4 &a2, const V4 &a3, const V4 &rd,
                                              const float4 &u3i_, const float4 &u3tp,
                                              const float4 &u3tm, const float4 &cK,
                                              const float4 &ci, const float4 &pK_,
                                              const float4 &pi_, const float4 &ptp,
                                              const float4 &ptm) {
  const V4 u3i = v4(u3i_), pK = v4(pK_), pi = v4(pi_), A1 = v4(a1);
  V4 t = madd(u3i, v4(-a1), (pK - pi) * (-a1));
  t = madd(a2, sub_twice(sub_twice(pK, v4(cK)) + u3i + pi, v4(ci)), t);
  t = msub(a3, sub_twice(sub_twice(v4(u3tp) + v4(u3tm), u3i) + v4(ptp) + v4(ptm), pK), t);
#ifdef SEIS_FAST_MATH
  return f4(-t / rd);  // rd: the table's a1 + a2
#else
  return quot_quad(-t, A1 + a2, rd);
#endif
}

// A tile's part of ptab in shared memory.
template <int TX, int TZ>
struct alignas(16) TileTab {
  float x[2][3][TZ];  // left, right strip by row
  float wz[TZ];
  float z[2][3][TX];  // top, bottom strip by column
  float wx[TX];
  float c[4][3];
  static constexpr int BYTES = (7 * TZ + 7 * TX + 12) * (int)sizeof(float);
  // one thread: its copies, completing on `bar` (BYTES in all)
  __device__ __forceinline__ void issue(const ShotDev &g, int x0, int z0, uint64_t *bar) {
    const float *T = g.ptab, *C = T + pad_tab_x(g.NZ);
    const int n = pad_tab_nz(g.NZ), m = pad_tab_nx(g.NX);
#pragma unroll 1
    for (int k = 0; k < 7; k++) {
      bulk_load(&x[0][0][0] + k * TZ, T + k * n + z0, TZ * sizeof(float), bar);
      bulk_load(&z[0][0][0] + k * TX, C + k * m + x0, TX * sizeof(float), bar);
    }
    bulk_load(&c[0][0], T + pad_tab_c(g.NX, g.NZ), 12 * sizeof(float), bar);
  }
};

// Where one pad quad (column cx, rows iz0 .. iz0+3) sits.  `z` rows take the
// one-way update along z (top or bottom strip), `x` rows that along x, `c`
// rows the diagonal corner; the other rows are model cells.
struct PadQuad {
  unsigned z, x, c, in;  // row masks; `in`: pad rows inside the grid
  int sz, sx;            // toward the interior
  bool both;             // rows of the top and of the bottom pad (a model of 1 or 2 rows)
  bool xw;               // the x ramp's weight (it wins in the corners, InitInversion.cpp:20-37)
  __device__ __forceinline__ PadQuad(const ShotDev &g, int cx, int iz0) {
    const int dl = g.pml - cx, dr = cx - (g.pml + g.nx - 1);
    const int distx = max(max(dl, dr), 0);
    sx = dl > 0 ? 1 : -1;
    const bool upper = iz0 < g.pml, lower = iz0 + 3 >= g.pml + g.nz;
    both = upper && lower;
    sz = upper ? 1 : -1;
    xw = distx > 0;
    // the row whose distance to the model along z is distx (from the top pad's
    // quads the distance falls with the row, from the bottom pad's it grows)
    const int e = upper ? g.pml - iz0 - distx : distx - (iz0 - (g.pml + g.nz - 1));
    const unsigned lt = (1u << min(max(e, 0), 4)) - 1u;           // rows < e
    const unsigned le = (1u << min(max(e + 1, 0), 4)) - 1u;       // rows <= e
    const unsigned gt = 0xFu & ~le;
    const bool padz = upper || lower;
    z = !padz ? 0u : upper ? lt : gt;
    x = distx == 0 ? 0u : !padz ? 0xFu : upper ? gt : lt;
    c = distx > 0 && padz ? le & ~lt : 0u;
    const int left = g.NZ - iz0;
    in = z | x | c;
    if (both) {  // the masks above know one pad only
      const unsigned model = ((1u << (g.pml + g.nz - iz0)) - 1u) & ~((1u << (g.pml - iz0)) - 1u);
      in = distx > 0 ? 0xFu : 0xFu & ~model;
    }
    in &= left >= 4 ? 0xFu : (1u << left) - 1u;
  }
};

// New values of a pad quad's rows from the two-way values U (tile + halo), the
// current field C and the previous field P (the absorbing part of
// processBoundary, fd.cpp:1092-1179, and the blend, :55-56)
template <int TX, int TZ, class UA_, class SC, class SP>
__device__ __forceinline__ float4 absorb_quad(const PadQuad &q, const TileTab<TX, TZ> &T,
                                              const UA_ &U, const SC &C, const SP &P,
                                              const ShotDev &g, int cx, int iz0, int col, int row) {
  const float4 u = U.quad(cx, iz0), c = C.quad(cx, iz0), p = P.quad(cx, iz0);
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (q.z) {
    const float4 ul = U.quad(cx - 1, iz0), ur = U.quad(cx + 1, iz0);
    const float4 pl = P.quad(cx - 1, iz0), pr = P.quad(cx + 1, iz0);
    const float(*t)[TX] = T.z[q.sz < 0];
    const V4 a2 = v4(t[0][col]), a3 = v4(t[1][col]), rd = v4(t[2][col]);
    if (q.sz > 0)
      o = oneway_quad(g.a1z, a2, a3, rd, shift_dn(u, U(cx, iz0 + 4)),
                      shift_dn(ur, U(cx + 1, iz0 + 4)), shift_dn(ul, U(cx - 1, iz0 + 4)), c,
                      shift_dn(c, C(cx, iz0 + 4)), p, shift_dn(p, P(cx, iz0 + 4)), pr, pl);
    else
      o = oneway_quad(g.a1z, a2, a3, rd, shift_up(u, U(cx, iz0 - 1)),
                      shift_up(ur, U(cx + 1, iz0 - 1)), shift_up(ul, U(cx - 1, iz0 - 1)), c,
                      shift_up(c, C(cx, iz0 - 1)), p, shift_up(p, P(cx, iz0 - 1)), pr, pl);
  }
  if (q.x) {
    const int I = cx + q.sx;
    const float4 ui = U.quad(I, iz0), ci = C.quad(I, iz0), pi = P.quad(I, iz0);
    const float(*t)[TZ] = T.x[q.sx < 0];
    const float4 a2 = *reinterpret_cast<const float4 *>(&t[0][row]);
    const float4 a3 = *reinterpret_cast<const float4 *>(&t[1][row]);
    const float4 rd = *reinterpret_cast<const float4 *>(&t[2][row]);
    const float4 w = oneway_quad(g.a1x, v4(a2), v4(a3), v4(rd), ui, shift_dn(ui, U(I, iz0 + 4)),
                                 shift_up(ui, U(I, iz0 - 1)), c, ci, p, pi,
                                 shift_dn(p, P(cx, iz0 + 4)), shift_up(p, P(cx, iz0 - 1)));
#pragma unroll
    for (int r = 0; r < 4; r++)
      if ((q.x >> r) & 1u) set_comp(o, r, comp(w, r));
  }
  if (q.c) {  // one diagonal row per quad (fd.cpp:1146-1178)
    const int r = __ffs(q.c) - 1, iz = iz0 + r;
    const float *t = T.c[2 * (q.sx < 0) + (q.sz < 0)];
    const float n = -(-g.ax1 * U(cx, iz + q.sz) - g.ax2 * U(cx + q.sx, iz) + t[0] * (-C(cx, iz)));
#ifdef SEIS_FAST_MATH
    const float s = n / t[1];
#else
    const float s = quot_quad(v4(n), v4(t[1]), v4(t[2])).x;
#endif
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k == r) set_comp(o, k, s);
  }
  const V4 w = q.xw ? v4(T.wx[col]) : v4(*reinterpret_cast<const float4 *>(&T.wz[row]));
  return f4(madd(v4(u), w, v4(o) * (v4(1.0f) - w)));
}

// The adjoint's quads of a corner tile by kind.  Around the diagonal a quad
// needs the general gather; in the order of the list nearly every warp held
// such quads, and the corner tiles, a few per shot, took four times the mean
// tile's time (51,000 cycles of a step's 65,000 on four 1280 x 480 shots).
// Sorted before the wait for the last step, by what no step changes.  The
// forward step's quads measured 10% slower sorted.
template <int N>
struct QuadSort {
  unsigned short pure[N];   // strips along z from the front, along x from the back
  unsigned short mixed[N];
  int nz, nx, nm;
  __device__ __forceinline__ void put(int i, int kind) {
    if (kind == 0) pure[atomicAdd(&nz, 1)] = (unsigned short)i;
    else if (kind == 1) pure[N - 1 - atomicAdd(&nx, 1)] = (unsigned short)i;
    else mixed[atomicAdd(&nm, 1)] = (unsigned short)i;
  }
  // the e-th of the pure quads
  __device__ __forceinline__ int get(int e) const { return e < nz ? pure[e] : pure[N - 1 - (e - nz)]; }
};
// both a strip along x and one along z cross the tile
template <int TX, int TZ>
__device__ __forceinline__ bool corner_tile(const ShotDev &g, int x0, int z0) {
  return (x0 <= g.pml || x0 + TX >= g.pml + g.nx) && (z0 <= g.pml || z0 + TZ >= g.pml + g.nz);
}

template <int S, int MODE>
struct UCfg;
}  // namespace SEIS_NS
}  // namespace seis
#include "fd_adjoint.cuh"
namespace seis {
namespace SEIS_NS {

// Staged arrays of one tile of the one-tile-per-CTA kernel.  Pad tiles: the
// current fields with the wide halo, the previous fields and the velocity with
// one column and four rows around the tile, the tile's coefficient table, and
// the two-way values of the tile and its halo; interior tiles: the current
// fields with the stencil's halo and the rest as the tile alone, in the same
// memory.  Everything comes by tensor copies that need nothing but the tile's
// entry of the list: loads into registers and a table built by the threads
// held every tile for 4,000 cycles before its first copy was issued.
constexpr int align32(int floats) { return (floats + 31) / 32 * 32; }  // 128-byte tensor-copy targets
template <int S, int MODE>
struct UCfg {
  using G = Geo<S>;
  static constexpr bool BORN = MODE == MODE_BORN;
  static constexpr int NF = BORN ? 2 : 1;
  static constexpr int PR = G::TZ + 8;              // staged rows of the previous fields
  static constexpr int CUR = align32(G::CW_C * G::SR);
  static constexpr int PRV = align32(G::CW_P * PR);
  static constexpr int U3 = align32(G::U3N);
  static constexpr bool ADJ = MODE == MODE_ADJ;
  // the velocity (adjoint: with the current field's halo) and, in the
  // adjoint, the second weighted field; Born: the perturbation; adjoint: the
  // ring terms (pad tiles)
  static constexpr int VEL = ADJ ? CUR : PRV, WGT = ADJ ? CUR : 0;
  static constexpr int DV = BORN ? G::TX * G::TZ : ADJ ? PRV : 0;
  static constexpr int TAB_BYTES = ADJ ? AdjTab<G::TX, G::TZ>::BYTES : TileTab<G::TX, G::TZ>::BYTES;
  static constexpr int TAB = align32(TAB_BYTES / 4);
  // interior tiles
  static constexpr int CW = G::TX + 2 * HI, RW = G::TZ + 2 * HI;
  static constexpr int CUR_I = align32(CW * RW), PRV_I = G::TX * G::TZ;
  // offsets: current fields, previous fields, velocity, perturbation, table,
  // two-way values
  static constexpr int O_P = NF * CUR, O_V = O_P + NF * PRV, O_W = O_V + VEL;
  static constexpr int O_D = O_W + WGT, O_T = O_D + DV;
  static constexpr int O_U = O_T + TAB, FLOATS = O_U + NF * U3;
  static_assert(CUR_I <= CUR && PRV_I <= PRV, "an interior tile fits a pad tile's memory");
  static constexpr size_t bytes = sizeof(float) * (size_t)FLOATS + 2 * sizeof(uint64_t);
  static constexpr int TX_PAD = ((NF + ADJ) * G::CW_C * G::SR + (NF + 1) * G::CW_P * PR +
                                 (BORN ? DV : 0)) * 4;
  static constexpr int TX_INT = ((NF + ADJ) * CW * RW + (NF + !ADJ) * PRV_I + (BORN ? DV : 0)) * 4;
  // at most 768 threads per SM (85 registers a thread; at 64 they spill and
  // one field measured 5% slower, at 128 up to 20% slower)
  static constexpr int CAP = 768 / G::NT;
  static constexpr int MIN_CTAS = ctas_fit(bytes, CAP) > 0 ? ctas_fit(bytes, CAP) : 1;
};

// Programmatic dependent launch: a step's kernel may start while the last
// step's is finishing; what the last step wrote is read only after the wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Per-cell side effects of a finished model quad (rows of `cm`): recording,
// boundary strips, illumination.
template <int MODE>
__device__ __forceinline__ void model_quad_out(const ShotDev &g, const StepArgs &aa, int cx,
                                               int iz0, unsigned cm, int gzr, const float4 &o) {
  if (MODE == MODE_RCV || MODE == MODE_BORN) return;
  if (aa.rec_k >= 0 && gzr >= iz0 && gzr <= iz0 + 3 && ((cm >> (gzr - iz0)) & 1u))
    g.rec[(size_t)aa.rec_k * g.nx + (cx - g.pml)] = comp(o, gzr - iz0);
  if (aa.illum_on) {  // illum, fd.cpp:317-319
    float *ss = g.illum + (size_t)(cx - g.pml) * g.nz + (iz0 - g.pml);
#pragma unroll
    for (int r = 0; r < 4; r++)
      if ((cm >> r) & 1u) ss[r] = ss[r] + comp(o, r) * comp(o, r);
  }
}
template <int MODE>
__device__ __forceinline__ void strips_quad(const ShotDev &g, const StepArgs &aa, int cx, int iz0,
                                            unsigned cm, const float4 &o) {
  if (MODE == MODE_BORN || aa.strip_k < 0) return;
  // columns and rows away from the model's edge lie in no strip
  const int x = cx - g.pml, z = iz0 - g.pml;
  if (x >= LAYERS && x < g.nx - LAYERS && z >= LAYERS && z + 3 < g.nz - LAYERS) return;
#pragma unroll
  for (int r = 0; r < 4; r++)
    if ((cm >> r) & 1u) save_strips(g, aa.strip_k, cx, iz0 + r, comp(o, r));
}

// The cells of one interior tile (every cell a model cell in the 8th-order
// region, where the absorbing blend is the identity: w = 1, u31 = 0;
// src/util/fd.cpp:55-56): the current fields CA, CB staged with the stencil's
// halo, the previous fields, velocity and perturbation through PA, PB, V, D; one 4-row x 2-column micro-tile per thread, gzq the padded
// receiver rows of its two columns.  Every thread of the CTA calls this (the
// snapshot holds block barriers).
template <int S, int MODE, class SC, class SO>
__device__ __forceinline__ void interior_cells(const ShotDev &g, const StepArgs &a, int x0, int z0,
                                               const SC &CA, const SC &CB, const SO &PA,
                                               const SO &PB, const SO &V, const SO &D,
                                               const int (&gzq)[2], float *red) {
  SEIS_GEO(S);
  constexpr bool BORN = MODE == MODE_BORN;
  StepArgs aa = a;
  if (MODE != MODE_RCV && aa.rec_k >= g.nt) aa.rec_k = -1;
  float *na = g.fa[(a.rot + 2) % 3];
  float *nb_ = g.fb[(a.rot_b + 2) % 3];
  float *out_a = MODE == MODE_RCV ? nb_ : na;
  const int tid = threadIdx.x;
  const int qz = tid % QZ, cx = tid / QZ;  // micro-tile: rows 4qz.., columns 2cx, 2cx+1
  const int ix = x0 + 2 * cx, iz0 = z0 + 4 * qz;
  const bool snap = MODE == MODE_MODEL && aa.snap_k >= 0 && g.snap != nullptr;

  float4 o[2], cen[2], lap[2], qs[2];
  const float4 prv[2] = {PA.quad(ix, iz0), PA.quad(ix + 1, iz0)};
  const float4 vel[2] = {V.quad(ix, iz0), V.quad(ix + 1, iz0)};
  pair_twoway(CA, g, ix, iz0, prv, vel, o, cen);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int cxj = ix + j;
    bool inj;
    if (MODE != MODE_RCV)
      inj = aa.src_k >= 0 && g.szp >= iz0 && g.szp <= iz0 + 3 && (g.sou || cxj == g.sxp);
    else
      inj = aa.rec_k >= 0 && gzq[j] >= iz0 - 1 && gzq[j] <= iz0 + 3;
    if (inj)
#pragma unroll
      for (int r = 0; r < 4; r++)
        set_comp(o[j], r, inject<MODE>(g, aa, cxj, iz0 + r, gzq[j], comp(o[j], r),
                                       coef(comp(vel[j], r), g).vt2));
    o[j] = f4(v4(o[j]) + v4(0.0f));
    model_quad_out<MODE>(g, aa, cxj, iz0, 0xFu, gzq[j], o[j]);
    strips_quad<MODE>(g, aa, cxj, iz0, 0xFu, o[j]);
    if (BORN || snap) lap[j] = second_diff(o[j], prv[j], cen[j], g);
    if (BORN) qs[j] = scatter_source(vel[j], lap[j], D.quad(cxj, iz0), g);
    *reinterpret_cast<float4 *>(out_a + (size_t)cxj * g.LDZ + iz0) = o[j];
  }
  if (BORN) {
    const float4 pb[2] = {PB.quad(ix, iz0), PB.quad(ix + 1, iz0)};
    pair_twoway(CB, g, ix, iz0, pb, vel, o, cen);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int cxj = ix + j;
      o[j] = f4(v4(o[j]) + v4(qs[j]) + v4(0.0f));
      if (aa.rec_k >= 0 && gzq[j] >= iz0 && gzq[j] <= iz0 + 3)
        g.rec[(size_t)aa.rec_k * g.nx + (cxj - g.pml)] = comp(o[j], gzq[j] - iz0);
      *reinterpret_cast<float4 *>(nb_ + (size_t)cxj * g.LDZ + iz0) = o[j];
    }
  }
  if (snap) {
    const unsigned all[2] = {0xFu, 0xFu};
    snap_write<NT_T, TX, TZ>(g, aa.snap_k, x0, z0, ix, iz0, lap, all, red);
  }
}

// Pad tiles: tiles with a pad cell, a cell within 3 of the grid edge (frame,
// src/util/fd.cpp:1057-1091; low-order rings, :1226-1241) or a model cell the
// interior tiles do not take.  One pass per step:
//  1. the two-way values (before injection) of the tile's and its halo's
//     frame cells, by the per-cell formula, into shared memory;
//  2. the tile's cells: the 8th- or 2nd-order two-way value (or the value of
//     step 1), injection (fd.cpp:49-51) and, for Born, the
//     scattering source; model cells are final (w = 1) and stored, every
//     two-way value is kept in shared memory;
//  3. the same for the halo ring (one cell around the tile), which the
//     one-way update of the tile's edge cells reads;
//  4. every pad quad: the one-way update from the two-way values and the
//     blend (processBoundary fd.cpp:1092-1179, :55-56), stored.
// A halo cell's two-way value is formed by the same per-cell arithmetic as
// in the tile that owns it.
// The tile's arrays at (x0, z0) are staged at `sm` (UCfg; the table's copies
// complete on tab_bar; the result is whether they did).  Every thread of the
// CTA calls this (it holds block barriers).
// What bounds it: instruction issue and latency, not memory.  The pad cells
// are taken a quad of rows at a time (the strip's kind, weights and
// coefficients once per quad and from tables, neighbours by 16-byte loads)
// instead of a cell at a time with its own classification, six divisions and
// a dozen 4-byte loads.
template <int S, int MODE>
__device__ __forceinline__ bool pad_cells(const ShotDev &g, const StepArgs &a, int x0, int z0,
                                          float *sm, uint64_t *tab_bar, const int (&gzq)[2],
                                          float *red) {
  SEIS_GEO(S);
  using SA = SAT<SR>;
  using K = UCfg<S, MODE>;
  using SP = SAT<K::PR>;
  using UA = UAT<G_::U3R>;
  constexpr int NHALO = G_::NHALO, NF = K::NF;
  constexpr bool BORN = K::BORN;
  const int tid = threadIdx.x;
  const int NX = g.NX, NZ = g.NZ;
  StepArgs aa = a;
  if (MODE != MODE_RCV && aa.rec_k >= g.nt) aa.rec_k = -1;
  float *na = g.fa[(a.rot + 2) % 3];
  float *nb_ = g.fb[(a.rot_b + 2) % 3];
  float *out_a = MODE == MODE_RCV ? nb_ : na;
  const int zm = z0 - ZM;
  float *sp = sm + K::O_P, *su = sm + K::O_U;
  const SA CA{sm, x0 - HXC, zm}, CB{sm + (NF - 1) * K::CUR, x0 - HXC, zm};
  const SP PA{sp, x0 - 1, z0 - 4}, PB{sp + (NF - 1) * K::PRV, x0 - 1, z0 - 4};
  const UA UA_{su, x0, z0}, UB_{su + (NF - 1) * K::U3, x0, z0};
  const SP V{sm + K::O_V, x0 - 1, z0 - 4};
  const SAT<TZ> D{sm + K::O_D, x0, z0};
  const TileTab<TX, TZ> &tab = *reinterpret_cast<const TileTab<TX, TZ> *>(sm + K::O_T);
  const GA DG{g.dv, g.LDZ};
  const bool snap = MODE == MODE_MODEL && aa.snap_k >= 0 && g.snap != nullptr;
  auto model = [&](int cx, int cz) {
    return cx >= g.pml && cx < g.pml + g.nx && cz >= g.pml && cz < g.pml + g.nz;
  };
  auto rcv_row = [&](int cx) {
    const int x = cx - g.pml;
    return (x >= 0 && x < g.nx) ? g.gz[x] + g.pml : -1;
  };

  // 1. the frame cells of the tile and its halo: the tile's edge rows, then
  // its edge columns (a corner is formed twice, to the same value)
  const int xa = max(x0 - 1, 0), xb = min(x0 + TX + 1, NX);
  const int za = max(z0 - 1, 0), zb = min(z0 + TZ + 1, NZ);
  const bool edge = xa <= 3 || za <= 3 || xb - 1 >= NX - 4 || zb - 1 >= NZ - 4;
  const int fzn = (za == 0) + (zb == NZ), fxn = (xa == 0) + (xb == NX);
  if (fzn + fxn > 0) {
    const int nc = xb - xa, nr = zb - za;
    auto frame = [&](const auto &Vf) {
      for (int i = tid; i < fzn * nc + fxn * nr; i += NT_T) {
        int cx, cz;
        if (i < fzn * nc) {
          const int second = i >= nc;
          cx = xa + i - second * nc;
          cz = za == 0 && !second ? 0 : NZ - 1;
        } else {
          const int j = i - fzn * nc, second = j >= nr;
          cz = za + j - second * nr;
          cx = xa == 0 && !second ? 0 : NX - 1;
        }
        UA_.ref(cx, cz) = frame_cell(CA, PA, Vf, g, cx, cz);
        if (BORN) UB_.ref(cx, cz) = frame_cell(CB, PB, Vf, g, cx, cz);
      }
    };
    // every read lies in the staged windows, except the normal extrapolation's
    // of the velocity two columns inside in a tile of one grid column
    if (x0 <= NX - 2) frame(V);
    else frame(GA{g.vel, g.LDZ});
    __syncthreads();
  }

  // 2. the tile's cells, one 4-row x 2-column micro-tile per thread
  const int qz = tid % QZ, cxp = tid / QZ;
  const int ix = x0 + 2 * cxp, iz0 = z0 + 4 * qz;
  float4 lap[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
  // per column the quad's rows inside the grid (cin) and its model cells (cm)
  unsigned cin[2] = {0u, 0u}, cm[2] = {0u, 0u};
  if (ix < NX && iz0 < NZ) {
    unsigned rin = 0u, rmod = 0u;
    // rows of the 2nd-order rings and of the frame
    unsigned low[2] = {0u, 0u}, frame[2] = {0u, 0u};
    if (edge)
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int r = 0; r < 4; r++) {
          const int d = min(min(ix + j, iz0 + r), min(NX - 1 - ix - j, NZ - 1 - iz0 - r));
          if (d <= 3) low[j] |= 1u << r;
          if (d == 0) frame[j] |= 1u << r;
        }
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int iz = iz0 + r;
      if (iz < NZ) rin |= 1u << r;
      if (iz < NZ && iz >= g.pml && iz < g.pml + g.nz) rmod |= 1u << r;
    }
    bool inj[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int cxj = ix + j;
      const bool colm = cxj < NX && cxj >= g.pml && cxj < g.pml + g.nx;
      cin[j] = cxj < NX ? rin : 0u;
      cm[j] = colm ? rmod : 0u;
      if (MODE != MODE_RCV)
        inj[j] = aa.src_k >= 0 && g.szp >= iz0 && g.szp <= iz0 + 3 &&
                 (g.sou ? colm : cxj == g.sxp);
      else
        inj[j] = aa.rec_k >= 0 && gzq[j] >= iz0 - 1 && gzq[j] <= iz0 + 3;
    }
    // the two-way values kept, the model cells stored
    auto keep = [&](const UA &U, float *out, int j, const float4 &u4, const float4 &o4) {
      const int cxj = ix + j;
      // rows below the grid hold finite values that nothing but masked rows read
      if (cin[j]) *reinterpret_cast<float4 *>(&U.ref(cxj, iz0)) = u4;
      if (cm[j] == 0xFu)
        *reinterpret_cast<float4 *>(out + (size_t)cxj * g.LDZ + iz0) = o4;
      else if (cm[j])
#pragma unroll
        for (int r = 0; r < 4; r++)
          if ((cm[j] >> r) & 1u) out[(size_t)cxj * g.LDZ + iz0 + r] = comp(o4, r);
    };
    auto from_frame = [&](const UA &U, float4 (&o)[2]) {
#pragma unroll
      for (int j = 0; j < 2; j++)
        if (frame[j])
#pragma unroll
          for (int r = 0; r < 4; r++)
            if ((frame[j] >> r) & 1u) set_comp(o[j], r, U(ix + j, iz0 + r));
    };
    float4 o[2], cen[2], qs[2];
    const float4 vel[2] = {V.quad(ix, iz0), V.quad(ix + 1, iz0)};
    {
      const float4 prv[2] = {PA.quad(ix, iz0), PA.quad(ix + 1, iz0)};
      pair_twoway(CA, g, ix, iz0, prv, vel, o, cen, low[0], low[1]);
      from_frame(UA_, o);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int cxj = ix + j;
        if (inj[j])
#pragma unroll
          for (int r = 0; r < 4; r++)
            if ((cin[j] >> r) & 1u)
              set_comp(o[j], r, inject<MODE>(g, aa, cxj, iz0 + r, gzq[j], comp(o[j], r),
                                             coef(comp(vel[j], r), g).vt2));
        const float4 out = f4(v4(o[j]) + v4(0.0f));
        keep(UA_, out_a, j, o[j], out);
        if (cm[j]) {
          model_quad_out<MODE>(g, aa, cxj, iz0, cm[j], gzq[j], out);
          strips_quad<MODE>(g, aa, cxj, iz0, cm[j], out);
        }
        qs[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if ((BORN || snap) && cm[j]) {
          lap[j] = second_diff(out, prv[j], cen[j], g);
          if (BORN) {
            const float4 t = scatter_source(vel[j], lap[j], D.quad(cxj, iz0), g);
#pragma unroll
            for (int r = 0; r < 4; r++)
              if ((cm[j] >> r) & 1u) set_comp(qs[j], r, comp(t, r));
          }
        }
      }
    }
    if (BORN) {
      const float4 pb[2] = {PB.quad(ix, iz0), PB.quad(ix + 1, iz0)};
      pair_twoway(CB, g, ix, iz0, pb, vel, o, cen, low[0], low[1]);
      from_frame(UB_, o);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int cxj = ix + j;
        const float4 u4 = add4(o[j], qs[j]);
        const float4 out = f4(v4(u4) + v4(0.0f));
        keep(UB_, nb_, j, u4, out);
        if (aa.rec_k >= 0 && gzq[j] >= iz0 && gzq[j] <= iz0 + 3 &&
            ((cm[j] >> (gzq[j] - iz0)) & 1u))
          g.rec[(size_t)aa.rec_k * g.nx + (cxj - g.pml)] = comp(out, gzq[j] - iz0);
      }
    }
  }

  // snapshot of the model cells' source terms (holds block barriers)
  if (snap) snap_write<NT_T, TX, TZ>(g, aa.snap_k, x0, z0, ix, iz0, lap, cm, red);

  // 3. the halo ring: the same two-way values, injection and scattering
  // source, for the halo cells next to a pad cell of the tile (the one-way
  // update reads its neighbours within one cell; zero elsewhere, where
  // nothing reads them)
  const int xe = min(x0 + TX, NX), ze = min(z0 + TZ, NZ);
  auto tile_pad = [&](int cx, int cz) {
    return cx >= x0 && cx < xe && cz >= z0 && cz < ze && !model(cx, cz);
  };
  for (int i = tid; i < NHALO; i += NT_T) {
    int hx, hz;
    halo_cell<TX, TZ>(i, x0, z0, hx, hz);
    bool read = false;
    if (i < 2 * (TX + 2)) {  // row above / below: the tile row next to it
      const int zz = hz < z0 ? z0 : ze - 1;
      read = tile_pad(hx - 1, zz) || tile_pad(hx, zz) || tile_pad(hx + 1, zz);
    } else {  // column left / right
      const int xx = hx < x0 ? x0 : xe - 1;
      read = tile_pad(xx, hz - 1) || tile_pad(xx, hz) || tile_pad(xx, hz + 1);
    }
    if (!read || hx < 0 || hz < 0 || hx >= NX || hz >= NZ) {
      UA_.ref(hx, hz) = 0.0f;
      if (BORN) UB_.ref(hx, hz) = 0.0f;
      continue;
    }
    const int d = min(min(hx, hz), min(NX - 1 - hx, NZ - 1 - hz));
    const float va = V(hx, hz);
    auto twoway = [&](const UA &U, const SA &C, const SP &P) {
      return d > 3 ? twoway_high(C, P, va, g, hx, hz)
             : d > 0 ? twoway_low(C, P, va, g, hx, hz) : U(hx, hz);
    };
    float ua = twoway(UA_, CA, PA);
    const Coef kk = coef(va, g);
    ua = inject<MODE>(g, aa, hx, hz, MODE == MODE_RCV ? rcv_row(hx) : -1, ua, kk.vt2);
    UA_.ref(hx, hz) = ua;
    if (BORN) {
      float ub = twoway(UB_, CB, PB);
      float q = 0.0f;
      if (model(hx, hz)) {
        const float out = ua + 0.0f;
        const float lap_ = (out + PA(hx, hz) - 2.0f * CA(hx, hz)) * g.idt2;
        const float vel3 = 2.0f / (va * va * va);
        q = kk.vt2 * lap_ * vel3 * DG(hx, hz);
      }
      UB_.ref(hx, hz) = ub + q;
    }
  }
  // every two-way value of the tile and halo is in shared memory, and the table
  const bool landed = mbar_wait(tab_bar, 0);
  __syncthreads();

  // 4. pad quads: one-way update and blend, shared evenly by all threads
  const QuadList pads(x0, z0, xe, ze, g.pml, g.pml + g.nx, g.pml, g.pml + g.nz);
  for (int i = tid; i < pads.n; i += NT_T) {
    int cx, dz;
    pads.quad(i, cx, dz);
    const int iz = z0 + dz;
    const size_t at = (size_t)cx * g.LDZ + iz;
    const PadQuad q(g, cx, iz);
    auto put = [&](float *out, const float4 &v) {
      if (q.in == 0xFu) {
        *reinterpret_cast<float4 *>(out + at) = v;
      } else {
#pragma unroll
        for (int r = 0; r < 4; r++)
          if ((q.in >> r) & 1u) out[at + r] = comp(v, r);
      }
    };
    if (!q.both) {
      put(out_a, absorb_quad(q, tab, UA_, CA, PA, g, cx, iz, cx - x0, dz));
      if (BORN) put(nb_, absorb_quad(q, tab, UB_, CB, PB, g, cx, iz, cx - x0, dz));
    } else {  // rows of both pads in one quad: a cell at a time
#pragma unroll 1
      for (int r = 0; r < 4; r++) {
        if (!((q.in >> r) & 1u)) continue;
        const Absorb b = absorb_geom(V, g, cx, iz + r);
        out_a[at + r] = absorb_apply(b, UA_(cx, iz + r), UA_, CA, PA, g, cx, iz + r);
        if (BORN) nb_[at + r] = absorb_apply(b, UB_(cx, iz + r), UB_, CB, PB, g, cx, iz + r);
      }
    }
  }
  return landed;
}

// One tile per CTA: the pad tiles (the list's n_pad tiles after its first
// n_int) start first, since they take longest, then the interior tiles.  The
// copies of what no step changes (velocity, perturbation, coefficient table)
// are issued before the wait for the last step, those of the fields after it.
// Measured per step (before: interior and pad kernels on two streams): one
// 281 x 281 shot 18.6 -> 6.7 us, Born 817 x 320 27 -> 11.6 us, eight 1280 x 480
// shots in the exact build 57 -> 25.5 us (16 B per cell at the copy rate: 12 us);
// the pad tiles of eight Born shots of 4000 x 1000: 84 -> 68 us.
template <int S, int MODE>
__device__ __forceinline__ void tile_step(const ShotDev *__restrict__ shots, const Tile &t,
                                          const StepArgs &a, int *__restrict__ err) {
  SEIS_GEO(S);
  using K = UCfg<S, MODE>;
  constexpr bool BORN = K::BORN;
  constexpr int NF = K::NF;
  extern __shared__ __align__(128) unsigned char smraw[];
  float *sm = reinterpret_cast<float *>(smraw);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + K::FLOATS);
  __shared__ ShotDev sg;
  __shared__ float red[33];
  __shared__ QuadSort<K::ADJ ? TX * QZ : 1> sort;
  const int tid = threadIdx.x;
  const bool pad = t.kind == TILE_PAD;
  if (K::ADJ && tid == 0) sort.nz = sort.nx = sort.nm = 0;
  pdl_trigger();
  if (tid == NT_T - 32) {  // the last warp's first lane, while the others fetch the shot table
    const int ra = a.rot % 3, rca = (a.rot + 1) % 3, rb = a.rot_b % 3, rcb = (a.rot_b + 1) % 3;
    const CUtensorMap *m = a.maps + (size_t)t.shot * NMAPS;
    constexpr bool B0 = MODE == MODE_RCV;  // the first field is field B
    const int c0 = B0 ? rcb : rca, p0 = B0 ? rb : ra;
    // rows count from the allocation start, ZM rows above row 0, columns from
    // XM to the left of column 0: no coordinate is negative and every row
    // coordinate is a multiple of 4 (16-byte aligned)
    const int xt = t.x0 + XM, zt = t.z0 + ZM;
    const CUtensorMap *mc = m + (pad ? (B0 ? MAP_FB_WIDE : MAP_FA_WIDE)
                                     : (B0 ? MAP_FB_HALO : MAP_FA_HALO)) + c0;
    const CUtensorMap *mp = m + (pad ? (B0 ? MAP_FB_PREV : MAP_FA_PREV)
                                     : (B0 ? MAP_FB_TILE : MAP_FA_TILE)) + p0;
    const CUtensorMap *mcb = m + (pad ? MAP_FB_WIDE : MAP_FB_HALO) + rcb;
    const CUtensorMap *mpb = m + (pad ? MAP_FB_PREV : MAP_FB_TILE) + rb;
    prefetch_map(mc);
    prefetch_map(mp);
    if (BORN) {
      prefetch_map(mcb);
      prefetch_map(mpb);
    }
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
    fence_barrier_init();
    mbar_expect_tx(bar, (uint32_t)(pad ? K::TX_PAD : K::TX_INT));
    const int xc = pad ? xt - HXC : xt - HI, zc = pad ? t.z0 : zt - HI;
    const int xp = pad ? xt - 1 : xt, zp = pad ? zt - 4 : zt;
    if (K::ADJ)
      tma_load_2d(sm + K::O_V, m + (pad ? MAP_VEL_WIDE : MAP_VEL_HALO), zc, xc, bar);
    else
      tma_load_2d(sm + K::O_V, m + (pad ? MAP_VEL_PREV : MAP_VEL_TILE), zp, xp, bar);
    if (BORN) tma_load_2d(sm + K::O_D, m + MAP_DV_TILE, zt, xt, bar);
    if (K::ADJ && pad) prefetch_map(m + MAP_E_PREV + (a.rot & 1));
    pdl_wait();
    tma_load_2d(sm, mc, zc, xc, bar);
    tma_load_2d(sm + K::O_P, mp, zp, xp, bar);
    if (BORN) {
      tma_load_2d(sm + K::CUR, mcb, zc, xc, bar);
      tma_load_2d(sm + K::O_P + K::PRV, mpb, zp, xp, bar);
    }
    if (K::ADJ && pad) tma_load_2d(sm + K::O_D, m + MAP_E_PREV + (a.rot & 1), zp, xp, bar);
    if (pad) {  // needed last, and its address takes one more read
      mbar_expect_tx(bar + 1, (uint32_t)K::TAB_BYTES);
      if (K::ADJ)
        reinterpret_cast<AdjTab<TX, TZ> *>(sm + K::O_T)->issue(shots[t.shot], t.x0, t.z0, bar + 1);
      else
        reinterpret_cast<TileTab<TX, TZ> *>(sm + K::O_T)->issue(shots[t.shot], t.x0, t.z0, bar + 1);
    }
  } else {
    for (int i = tid; i < (int)(sizeof(ShotDev) / sizeof(int)); i += NT_T - 32)
      if (tid < NT_T - 32)
        reinterpret_cast<int *>(&sg)[i] = reinterpret_cast<const int *>(shots + t.shot)[i];
  }
  __syncthreads();
  const ShotDev &g = sg;
  const int ix = t.x0 + 2 * (tid / QZ), iz0 = t.z0 + 4 * (tid % QZ);
  int gzq[2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int x = ix + j - g.pml;
    gzq[j] = x >= 0 && x < g.nx ? g.gz[x] + g.pml : -1;
  }
  bool corner = false;
  if constexpr (K::ADJ) {
    corner = pad && corner_tile<TX, TZ>(g, t.x0, t.z0);
    if (corner) {
      const QuadList l(t.x0, t.z0, min(t.x0 + TX, g.NX), min(t.z0 + TZ, g.NZ), g.pml + 1,
                       g.pml + g.nx - 1, g.pml + 1, g.pml + g.nz - 1);
      for (int i = tid; i < l.n; i += NT_T) {
        int cx, dz;
        l.quad(i, cx, dz);
        sort.put(i, RingQuad(g, cx, t.z0 + dz).kind);
      }
    }
  }
  pdl_wait();
  Imager im;
  if (K::ADJ) im.template load<TX, TZ>(g, a, t.x0, t.z0, ix, iz0);
  // the copies of a CTA that gives up land before its shared memory is freed
  // (waited for with a limit again)
  auto give_up = [&]() {
    if (tid != 0) return;
    atomicExch(err, 1);
    mbar_wait(bar, 0);
    if (pad) mbar_wait(bar + 1, 0);
  };
  if (!mbar_wait(bar, 0)) {
    give_up();
    return;
  }
  if (pad) {
    bool ok;
    if constexpr (K::ADJ)
      ok = adj_pad_cells<S>(g, a, t.x0, t.z0, sm, bar + 1, gzq, sort, corner, im);
    else
      ok = pad_cells<S, MODE>(g, a, t.x0, t.z0, sm, bar + 1, gzq, red);
    if (!ok) give_up();
  } else {
    using SW = SAT<K::RW>;
    using ST = SAT<TZ>;
    const SW CA{sm, t.x0 - HI, t.z0 - HI}, CB{sm + (NF - 1) * K::CUR, t.x0 - HI, t.z0 - HI};
    const ST PA{sm + K::O_P, t.x0, t.z0}, PB{sm + K::O_P + (NF - 1) * K::PRV, t.x0, t.z0};
    if constexpr (K::ADJ) {
      adj_interior_cells<S>(g, a, t.x0, t.z0, sm, sm + K::O_V, sm + K::O_W, PA, gzq, im);
    } else {
      const ST V{sm + K::O_V, t.x0, t.z0}, D{sm + K::O_D, t.x0, t.z0};
      interior_cells<S, MODE>(g, a, t.x0, t.z0, CA, CB, PA, PB, V, D, gzq, red);
    }
  }
}

template <int S, int MODE>
__global__ void __launch_bounds__(Geo<S>::NT, UCfg<S, MODE>::MIN_CTAS) step_tile_kernel(
    const ShotDev *__restrict__ shots, const Tile *__restrict__ tiles, int n_int, int n_pad,
    StepArgs a, int *__restrict__ err) {
  const int b = blockIdx.x;
  tile_step<S, MODE>(shots, tiles[b < n_pad ? n_int + b : b - n_pad], a, err);
}

// One reverse step of the reference RTM: the source field (A) reconstructed
// and the receiver field (B) propagated, which do not depend on one another,
// in one launch over the tile list twice (the pad tiles of both first).  As
// two launches on single shots each waited for the other's last tile.
template <int S>
__global__ void __launch_bounds__(Geo<S>::NT, UCfg<S, MODE_MODEL>::MIN_CTAS) step_pair_kernel(
    const ShotDev *__restrict__ shots, const Tile *__restrict__ tiles, int n_int, int n_pad,
    StepArgs a, int *__restrict__ err) {
  static_assert(UCfg<S, MODE_MODEL>::bytes == UCfg<S, MODE_RCV>::bytes, "one launch for both");
  int b = blockIdx.x;
  const bool rcv = b & 1;
  b >>= 1;
  const Tile t = tiles[b < n_pad ? n_int + b : b - n_pad];
  if (rcv) {
    tile_step<S, MODE_RCV>(shots, t, a, err);
  } else {
    a.rec_k = -1;
    tile_step<S, MODE_MODEL>(shots, t, a, err);
  }
}

// Persistent interior kernel: CTA b of G takes the interior tiles b, b + G,
// b + 2G, ... through two shared-memory stages, so that the tensor copies of
// its next tile are in flight while the current one is computed.  The
// current fields are staged with an HI-cell halo on every side, the other
// arrays as the tile alone (interior cells read them at the cell only).
template <int S, int MODE>
struct LCfg {
  using G = Geo<S>;
  static constexpr bool BORN = MODE == MODE_BORN;
  static constexpr bool ADJ = MODE == MODE_ADJ;
  static constexpr int NCUR = BORN || ADJ ? 2 : 1;  // current fields; adjoint: field, velocity
  static constexpr int NOTH = BORN ? 4 : ADJ ? 1 : 2;  // prev, vel [, prev B, dv]; adjoint: prev
  static constexpr int CW = G::TX + 2 * HI, RW = G::TZ + 2 * HI;
  static constexpr int TILE = G::TX * G::TZ;
  static constexpr int STAGE = NCUR * CW * RW + NOTH * TILE;  // floats
  static constexpr int WGT = ADJ ? CW * RW : 0;  // the second weighted field
  static constexpr size_t bytes =
      sizeof(float) * (2 * (size_t)STAGE + WGT) + 2 * sizeof(uint64_t);
  // static shared memory: two shot tables and the snapshot reduction
  static constexpr size_t static_bytes = 2 * sizeof(ShotDev) + 33 * sizeof(float);
  // at most 512 threads per SM for Born's two fields and for the adjoint's
  // imaging (128 registers a thread), 1024 for one field
  static constexpr int CAP = (BORN || MODE == MODE_ADJ ? 512 : 1024) / G::NT;
  static constexpr int MIN_CTAS =
      ctas_fit(bytes + static_bytes, CAP) > 0 ? ctas_fit(bytes + static_bytes, CAP) : 1;
  static_assert((NCUR * CW * RW * sizeof(float)) % 128 == 0 && (TILE * sizeof(float)) % 128 == 0 &&
                    (STAGE * sizeof(float)) % 128 == 0,
                "tensor-copy destinations stay 128-byte aligned");
};

template <int S, int MODE>
__global__ void __launch_bounds__(Geo<S>::NT, LCfg<S, MODE>::MIN_CTAS) interior_loop_kernel(
    const ShotDev *__restrict__ shots, const Tile *__restrict__ tiles, int n, StepArgs a,
    int *__restrict__ err) {
  SEIS_GEO(S);
  using L = LCfg<S, MODE>;
  constexpr bool BORN = L::BORN;
  constexpr int CW = L::CW, RW = L::RW, TILE = L::TILE;
  using SW = SAT<RW>;  // current fields, HI-cell halo
  using ST = SAT<TZ>;  // the other arrays, the tile alone
  extern __shared__ __align__(128) unsigned char smraw[];
  float *stage0 = reinterpret_cast<float *>(smraw);
  uint64_t *bar = reinterpret_cast<uint64_t *>(stage0 + 2 * L::STAGE + L::WGT);
  __shared__ ShotDev sg[2];
  __shared__ int2 sxz[2];  // tile origin of each stage
  __shared__ float red[33];
  __shared__ int s_fail;
  const int tid = threadIdx.x;
  int i = blockIdx.x;
  if (i >= n) return;
  auto load_shot = [&](int st, int ti) {
    const int shot = tiles[ti].shot;
    if (tid < (int)(sizeof(ShotDev) / sizeof(int)))
      reinterpret_cast<int *>(&sg[st])[tid] = reinterpret_cast<const int *>(shots + shot)[tid];
  };
  // thread 0: the tensor copies of tile ti into stage st (row coordinates
  // count from the allocation start, ZM rows above row 0; columns XM to the
  // left of column 0)
  auto issue = [&](int st, int ti) {
    const Tile t = tiles[ti];
    sxz[st] = make_int2(t.x0, t.z0);
    const CUtensorMap *maps = shots[t.shot].maps;
    float *bb = stage0 + st * L::STAGE;
    fence_proxy_async();
    mbar_expect_tx(bar + st, (uint32_t)(L::STAGE * sizeof(float)));
    const int ra = a.rot % 3, rca = (a.rot + 1) % 3, rb = a.rot_b % 3, rcb = (a.rot_b + 1) % 3;
    int cur[2], oth[4];
    if (MODE == MODE_RCV) {
      cur[0] = MAP_FB_HALO + rcb; oth[0] = MAP_FB_TILE + rb; oth[1] = MAP_VEL_TILE;
    } else if (L::ADJ) {
      cur[0] = MAP_FA_HALO + rca; cur[1] = MAP_VEL_HALO; oth[0] = MAP_FA_TILE + ra;
    } else if (!BORN) {
      cur[0] = MAP_FA_HALO + rca; oth[0] = MAP_FA_TILE + ra; oth[1] = MAP_VEL_TILE;
    } else {
      cur[0] = MAP_FA_HALO + rca; cur[1] = MAP_FB_HALO + rcb;
      oth[0] = MAP_FA_TILE + ra; oth[1] = MAP_VEL_TILE; oth[2] = MAP_FB_TILE + rb; oth[3] = MAP_DV_TILE;
    }
#pragma unroll
    for (int c = 0; c < L::NCUR; c++)
      tma_load_2d(bb + c * CW * RW, maps + cur[c], t.z0 + ZM - HI, t.x0 + XM - HI, bar + st);
#pragma unroll
    for (int o = 0; o < L::NOTH; o++)
      tma_load_2d(bb + L::NCUR * CW * RW + o * TILE, maps + oth[o], t.z0 + ZM, t.x0 + XM, bar + st);
  };
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
    fence_barrier_init();
    s_fail = 0;
  }
  load_shot(0, i);
  __syncthreads();
  if (tid == 0) issue(0, i);
  __syncthreads();  // the first tile's origin
  uint32_t par = 0;  // bit st: parity of the next completion of stage st
  int st = 0;
  const int cxq = 2 * (tid / QZ);
  for (;;) {
    const int next = i + (int)gridDim.x;
    const bool more = next < n;
    if (more) {  // the other stage was released at the end of the last tile
      load_shot(st ^ 1, next);
      if (tid == 0) issue(st ^ 1, next);
    }
    // this tile's receiver rows, loaded while its copies land
    const ShotDev &g = sg[st];
    const int x0 = sxz[st].x, z0 = sxz[st].y;
    const int gzq[2] = {g.gz[x0 + cxq - g.pml] + g.pml, g.gz[x0 + cxq + 1 - g.pml] + g.pml};
    Imager im;
    if (L::ADJ) im.template load<TX, TZ>(g, a, x0, z0, x0 + cxq, z0 + 4 * (tid % QZ));
    // a wait that gives up leaves garbage in the stage (indices stay in
    // range); the CTA then ends after this tile
    if (!mbar_wait(bar + st, (par >> st) & 1u)) s_fail = 1;
    par ^= 1u << st;
    float *bb = stage0 + st * L::STAGE, *ob = bb + L::NCUR * CW * RW;
    const ST PA{ob, x0, z0};
    if constexpr (L::ADJ) {
      adj_interior_cells<S>(g, a, x0, z0, bb, bb + CW * RW, stage0 + 2 * L::STAGE, PA, gzq, im);
    } else {
      const SW CA{bb, x0 - HI, z0 - HI};
      const SW CB{bb + (BORN ? CW * RW : 0), x0 - HI, z0 - HI};
      const ST VV{ob + TILE, x0, z0};
      const ST PB{ob + (BORN ? 2 : 0) * TILE, x0, z0};
      const ST DV{ob + (BORN ? 3 : 1) * TILE, x0, z0};
      interior_cells<S, MODE>(g, a, x0, z0, CA, CB, PA, PB, VV, DV, gzq, red);
    }
    __syncthreads();  // stage st, its origin and shot table are free for the tile after next
    if (s_fail) {
      // the copies in flight into the other stage land before the CTA ends
      if (tid == 0) {
        atomicExch(err, 1);
        if (more) mbar_wait(bar + (st ^ 1), (par >> (st ^ 1)) & 1u);
      }
      return;
    }
    if (!more) break;
    i = next;
    st ^= 1;
  }
}

}  // namespace SEIS_NS
}  // namespace seis
