// Exact adjoint of the Born operator (sm_100a).  No counterpart in the
// reference: its adjoint() (src/util/fd.cpp:592-719) is a different imaging
// operator and fails the dot-product test.  Contracted build only; included by
// fd_tile.cuh, whose kernels run it as MODE_ADJ.
//
// One forward step maps (cur, prev) to next through
//   u3  = S(cur, prev)                 two-way update + frame  fd.cpp:1057-1091, :1226-1271
//   u31 = P(u3, cur, prev)             one-way update on the pad rings  :1092-1179
//   nxt = w u3 + (1 - w) u31           blend  :55-56
// and the scattering source enters u3.  With Lk the complete adjoint of the
// field of step k, one reverse step computes
//   mu(L)  = w L + P_u3^T ((1-w) L)          (adjoint of u3: where sources enter)
//   L_k    = S_cur^T mu(L_{k+1}) + P_cur^T((1-w) L_{k+1})
//          - mu(L_{k+2}) + P_prev^T((1-w) L_{k+2}) + R^T d_{k-1-ndel}
// and images grad += w_img * lap_k * mu(L_{k+1}) on the model interior
// (lap_k = source-field second time derivative from the snapshots).
//
// The field kept between steps is M_k = mu(L_k), not L_k; with the ring
// values rho_k = (1 - w) L_k on the pad rings, one reverse step is
//   L_k = S_cur^T M_{k+1} - M_{k+2} + E_k + R^T d,
//   E_k = P_cur^T rho_{k+1} + P_prev^T rho_{k+2},
// and every term is a gather over a fixed neighbourhood summed in a fixed
// order, so the adjoint is bit-for-bit repeatable without atomics.  E
// alternates between two buffers by step (a tile reads this step's E on its
// halo while its neighbour writes the next step's); the P_prev^T part is kept
// one step in adj_b.
#pragma once

namespace seis {
namespace SEIS_NS {

// [t == s + 1] + [t == s - 1] - 2 [t == s]
__device__ __forceinline__ float lap3(int t, int s) {
  return t == s ? -2.0f : (t == s + 1 || t == s - 1) ? 1.0f : 0.0f;
}

// Coefficient of cur(tx, tz) in the two-way value of a consumer cell (cx, cz)
// in the frame or the low-order rings: the transpose of frame_cell (fd.cpp:
// 1057-1091) and twoway_low (:1226-1241) without the 2 cur term that every
// branch has.
template <class VA>
__device__ float dcur(const ShotDev &g, const VA &V, int cx, int cz, int tx, int tz) {
  const int NX = g.NX, NZ = g.NZ;
  const int ox = tx - cx, oz = tz - cz;
  float k = 0.0f;
  const bool fx = (cx == 0 || cx == NX - 1), fz = (cz == 0 || cz == NZ - 1);
  if (fx || fz) {
    if (!(fx && fz)) {  // second difference along the edge
      const float v = V(cx, cz);
      if (fz) {
        const float e = v * v * g.kx;
        if (oz == 0) k += e * lap3(tx, cx);
      } else {
        const float e = v * v * (cx == 0 ? g.kz : g.kx);
        if (ox == 0) k += e * lap3(tz, cz);
      }
    }
    if (fz && ox == 0) {  // normal extrapolation along z: + 2 y1 - y2
      const int s1 = cz == 0 ? 1 : NZ - 2, s2 = cz == 0 ? 2 : NZ - 3;
      if (tz >= min(s1, s2) - 1 && tz <= max(s1, s2) + 1) {
        const float v1 = V(cx, s1), v2 = V(cx, s2);
        k += 2.0f * (v1 * v1 * g.kz) * lap3(tz, s1) - (v2 * v2 * g.kz) * lap3(tz, s2);
      }
    }
    if (fx && oz == 0) {  // along x
      const int s1 = cx == 0 ? 1 : NX - 2, s2 = cx == 0 ? 2 : NX - 3;
      if (tx >= min(s1, s2) - 1 && tx <= max(s1, s2) + 1) {
        const float v1 = V(s1, cz), v2 = V(s2, cz);
        k += 2.0f * (v1 * v1 * g.kx) * lap3(tx, s1) - (v2 * v2 * g.kx) * lap3(tx, s2);
      }
    }
    return k;
  }
  const Coef c = coef(V(cx, cz), g);
  if (ox == 0) k += c.vz * lap3(tz, cz);
  if (oz == 0) k += c.vx * lap3(tx, cx);
  return k;
}

// The part of the transposed two-way update at cell (tx, tz) that comes from
// frame and low-order consumers (cells within 3 of the grid edge) on its cross
// is nonzero only within 4 of the edge.  A 2nd-order consumer reads its
// neighbours within one cell, a frame consumer (edge row or column) those
// within one cell along the edge and three cells along its normal
// extrapolation, so the part is
//   sum over m = -3..3 of c_z[m] M(tx, tz + m) + sum over m != 0 of c_x[m] M(tx + m, tz)
// with c = dcur of the consumer (zero for the other offsets and for consumers
// in the 8th-order region).  The coefficients depend on the
// velocity only: this kernel forms them for every cell of the four edge
// bands of every shot (band cell i of band b, see edge_index).
#ifdef SEIS_ADJOINT_TABLES
__global__ void edge_coef_kernel(const ShotDev *__restrict__ shots, int nshots) {
  const ShotDev &g = shots[blockIdx.y];
  const int NX = g.NX, NZ = g.NZ, n = edge_cells(NX, NZ);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int cx, cz;
  if (i < 5 * NX) {
    cx = i / 5; cz = i % 5;
  } else if (i < 10 * NX) {
    cx = (i - 5 * NX) / 5; cz = NZ - 5 + (i - 5 * NX) % 5;
  } else if (i < 10 * NX + 5 * NZ) {
    cx = (i - 10 * NX) / NZ; cz = (i - 10 * NX) % NZ;
  } else {
    cx = NX - 5 + (i - 10 * NX - 5 * NZ) / NZ; cz = (i - 10 * NX - 5 * NZ) % NZ;
  }
  const GA V{g.vel, g.LDZ};
  auto low = [&](int x, int z) {
    return x >= 0 && x < NX && z >= 0 && z < NZ && !(x >= 4 && x <= NX - 5 && z >= 4 && z <= NZ - 5);
  };
  float *c = g.edge_coef + i;
  const bool in = cx >= 0 && cx < NX && cz >= 0 && cz < NZ;
  int k = 0;
  for (int m = -3; m <= 3; m++, k++) {
    const int z = cz + m;
    float v = 0.0f;
    if (in && ((m >= -1 && m <= 1) || z == 0 || z == NZ - 1) && low(cx, z))
      v = dcur(g, V, cx, z, cx, cz);
    c[(size_t)k * n] = v;
  }
  for (int m = -3; m <= 3; m++) {
    if (m == 0) continue;
    const int x = cx + m;
    float v = 0.0f;
    if (in && ((m >= -1 && m <= 1) || x == 0 || x == NX - 1) && low(x, cz))
      v = dcur(g, V, x, cz, cx, cz);
    c[(size_t)k * n] = v;
    k++;
  }
}

// The one-way update of a strip cell (fd.cpp:1098-1104) is
//   u31 = al (u3_i + p) + be (u3_i+t + u3_i-t + p_+t + p_-t) + ga (c + c_i) - p_i
// with al = (a1 - a2 - 2 a3)/d, be = a3/d, ga = 2 a2/d, d = a1 + a2 (c, p =
// cur, prev at the cell; _i at the inner neighbour, +-t along the strip), and
// of a corner cell (fd.cpp:1146-1178) u31 = cz u3_z + cx u3_x + bK c.  atab
// (ShotDev): per row of the left and right strip and per column of the top and
// bottom strip al, be, ga; per corner cz, cx and bK.  Without a pad there is no
// strip cell and all are zero: the quads along the grid's edge take them times
// a weight of zero, which a zero velocity's infinite ones would make NaN.
__global__ void adj_tab_kernel(const ShotDev *__restrict__ shots) {
  const ShotDev &g = shots[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int NX = g.NX, NZ = g.NZ, n = adj_tab_nz(NZ), m = adj_tab_nx(NX);
  auto strip = [&](float *t, int stride, float v, float a1, float invh2) {
    if (g.pml == 0) {
      t[0] = t[stride] = t[2 * stride] = 0.0f;
      return;
    }
    const float rv = 1.0f / v, a2 = __fmul_rn(g.hdt2, rv), a3 = __fmul_rn(v * 0.25f, invh2);
    const float rd = 1.0f / __fadd_rn(a1, a2);
    t[0] = __fmul_rn(__fmaf_rn(-2.0f, a3, __fsub_rn(a1, a2)), rd);
    t[stride] = __fmul_rn(a3, rd);
    t[2 * stride] = __fmul_rn(2.0f * a2, rd);
  };
  if (i < n) {
    const int iz = min(max(i - ADJ_TAB_M, 0), NZ - 1);
    for (int b = 0; b < 2; b++)
      strip(g.atab + 3 * b * n + i, n, g.vel[(size_t)(b ? NX - 1 : 0) * g.LDZ + iz], g.a1x,
            g.invdz2);
  } else if (i < n + m) {
    const int j = i - n, ix = min(max(j - ADJ_TAB_M, 0), NX - 1);
    for (int b = 0; b < 2; b++)
      strip(g.atab + 6 * n + 3 * b * m + j, m, g.vel[(size_t)ix * g.LDZ + (b ? NZ - 1 : 0)],
            g.a1z, g.invdx2);
  } else if (i < n + m + 4) {
    const int c = i - n - m;
    const float v = g.vel[(size_t)(c & 2 ? NX - 1 : 0) * g.LDZ + (c & 1 ? NZ - 1 : 0)];
    const float ax3 = g.sqrt2f / v / g.dt;
    const float re = 1.0f / (g.ax1 + g.ax2 + ax3);
    float *t = g.atab + 6 * (n + m) + 4 * c;
    t[0] = g.pml == 0 ? 0.0f : g.ax1 * re;
    t[1] = g.pml == 0 ? 0.0f : g.ax2 * re;
    t[2] = g.pml == 0 ? 0.0f : ax3 * re;
    t[3] = 0.0f;
  }
}
#endif

// A tile's part of atab in shared memory: its rows and columns and
// ADJ_TAB_M on either side.
template <int TX, int TZ>
struct alignas(16) AdjTab {
  static constexpr int NR = TZ + 2 * ADJ_TAB_M, NC = TX + 2 * ADJ_TAB_M;
  float x[2][3][NR];  // left, right strip by row
  float z[2][3][NC];  // top, bottom strip by column
  float c[4][4];
  static constexpr int BYTES = (6 * (NR + NC) + 16) * (int)sizeof(float);
  __device__ __forceinline__ void issue(const ShotDev &g, int x0, int z0, uint64_t *bar) {
    const float *T = g.atab;
    const int n = adj_tab_nz(g.NZ), m = adj_tab_nx(g.NX);
#pragma unroll 1
    for (int k = 0; k < 6; k++) {
      bulk_load(&x[0][0][0] + k * NR, T + k * n + z0, NR * sizeof(float), bar);
      bulk_load(&z[0][0][0] + k * NC, T + 6 * n + k * m + x0, NC * sizeof(float), bar);
    }
    bulk_load(&c[0][0], T + 6 * (n + m), 16 * sizeof(float), bar);
  }
};

// Imaging of a thread's two column quads: the snapshot and the accumulator are
// read before the step's inputs are waited for, so that their latencies
// overlap the copies', and written after.
struct Imager {
  float4 lap[2];
  double2 acc[2][2];
  unsigned on;  // bit j: column j's quad holds model cells
  float scale;  // weight of the step over the tile's snapshot scale
  template <int TX, int TZ>
  __device__ __forceinline__ void load(const ShotDev &g, const StepArgs &a, int x0, int z0, int ix,
                                       int iz0) {
    on = 0u;
    if (a.snap_k < 0 || g.snap == nullptr || iz0 + 3 < g.pml || iz0 >= g.pml + g.nz) return;
    float s = 1.0f;
    if (g.snap_dtype != SNAP_F32) {
      const int ntx = (g.NX + TX - 1) / TX;
      s = 1.0f / g.snap_scale[(size_t)a.snap_k * ntx * g.ntz + (x0 / TX) * g.ntz + z0 / TZ];
    }
    scale = s;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int x = ix + j - g.pml;
      if (x < 0 || x >= g.nx) continue;
      on |= 1u << j;
      const size_t i = image_index(g.nz, g.pml, x, iz0);
      const size_t k = (size_t)a.snap_k * g.nx * image_ld(g.nz, g.pml) + i;
      if (g.snap_dtype == SNAP_F32) {
        lap[j] = *reinterpret_cast<const float4 *>(reinterpret_cast<const float *>(g.snap) + k);
      } else {
        const uint2 q = *reinterpret_cast<const uint2 *>(
            reinterpret_cast<const unsigned short *>(g.snap) + k);
        float2 lo, hi;
        if (g.snap_dtype == SNAP_BF16) {
          lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&q.x));
          hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&q.y));
        } else {
          lo = __half22float2(*reinterpret_cast<const __half2 *>(&q.x));
          hi = __half22float2(*reinterpret_cast<const __half2 *>(&q.y));
        }
        lap[j] = make_float4(lo.x, lo.y, hi.x, hi.y);
      }
      const double2 *d = reinterpret_cast<const double2 *>(g.grad + i);
      acc[j][0] = d[0];
      acc[j][1] = d[1];
    }
  }
  // grad += w lap M1 of column j (the product rounded to float, then
  // accumulated in double); rows outside the model accumulate nothing that is
  // read (their snapshots are zero)
  __device__ __forceinline__ void store(const ShotDev &g, const StepArgs &a, int j, int ix, int iz0,
                                        const float4 &n) const {
    if (!((on >> j) & 1u)) return;
    double2 *d = reinterpret_cast<double2 *>(
        g.grad + image_index(g.nz, g.pml, ix + j - g.pml, iz0));
    const float4 p = f4(v4(lap[j]) * scale * a.img_w * v4(n));
    d[0] = make_double2(acc[j][0].x + (double)p.x, acc[j][0].y + (double)p.y);
    d[1] = make_double2(acc[j][1].x + (double)p.z, acc[j][1].y + (double)p.w);
  }
};

// Gathers of one target quad: m = P_u3^T rho, e = P_cur^T rho, b = P_prev^T
// rho, and its blend weights w, from L of the tile and halo.
struct RingTerms {
  V4 m, e, b, w;
};
// distance to the model along x of a column, along z of a row (0 inside)
__device__ __forceinline__ int dist_x(const ShotDev &g, int cx) {
  return max(max(g.pml - cx, cx - (g.pml + g.nx - 1)), 0);
}
__device__ __forceinline__ int dist_z(const ShotDev &g, int cz) {
  return max(max(g.pml - cz, cz - (g.pml + g.nz - 1)), 0);
}
__device__ __forceinline__ V4 dist_quad(const ShotDev &g, int iz) {
  return v4(make_float4((float)dist_z(g, iz), (float)dist_z(g, iz + 1), (float)dist_z(g, iz + 2),
                        (float)dist_z(g, iz + 3)));
}

// The general gather of one cell: its 3 x 3 neighbourhood's ring cells, each
// by its own kind, column by column.
template <int TX, int TZ, class UA_>
__device__ __noinline__ float4 ring_cell(const ShotDev &g, const AdjTab<TX, TZ> &T, const UA_ &U,
                                         int x0, int z0, int cx, int cz) {
  float m = 0.0f, e = 0.0f, b = 0.0f;
  for (int dx = -1; dx <= 1; dx++)
    for (int dz = -1; dz <= 1; dz++) {
      const int qx = cx + dx, qz = cz + dz;
      if (qx < 0 || qz < 0 || qx >= g.NX || qz >= g.NZ) continue;
      const int D = dist_x(g, qx), Z = dist_z(g, qz);
      if ((D | Z) == 0) continue;
      const int sx = qx < g.pml ? 1 : -1, sz = qz < g.pml ? 1 : -1;  // toward the interior
      const float w = __fmaf_rn(-(float)(D > 0 ? D : Z), g.inv_pml, 1.0f);
      const float r = __fmul_rn(1.0f - w, U(qx, qz));  // rho
      const int ox = -dx, oz = -dz;  // this cell as seen from the ring cell
      if (D == Z) {
        const float *t = T.c[2 * (sx < 0) + (sz < 0)];
        if (ox == 0 && oz == sz) m = __fadd_rn(m, __fmul_rn(t[0], r));
        else if (ox == sx && oz == 0) m = __fadd_rn(m, __fmul_rn(t[1], r));
        else if (ox == 0 && oz == 0) e = __fadd_rn(e, __fmul_rn(t[2], r));
        continue;
      }
      const bool vert = Z > D;
      const int in = vert ? oz * sz : ox * sx, along = vert ? ox : oz;
      float al, be, ga;
      if (vert) {
        const int i = qx - x0 + ADJ_TAB_M;
        const float(*t)[AdjTab<TX, TZ>::NC] = T.z[sz < 0];
        al = t[0][i]; be = t[1][i]; ga = t[2][i];
      } else {
        const int i = qz - z0 + ADJ_TAB_M;
        const float(*t)[AdjTab<TX, TZ>::NR] = T.x[sx < 0];
        al = t[0][i]; be = t[1][i]; ga = t[2][i];
      }
      al = __fmul_rn(al, r); be = __fmul_rn(be, r); ga = __fmul_rn(ga, r);
      if (along == 0) {
        if (in == 0) { e = __fadd_rn(e, ga); b = __fadd_rn(b, al); }
        else if (in == 1) { m = __fadd_rn(m, al); e = __fadd_rn(e, ga); b = __fsub_rn(b, r); }
      } else {
        if (in == 0) b = __fadd_rn(b, be);
        else if (in == 1) m = __fadd_rn(m, be);
      }
    }
  return make_float4(m, e, b, 0.0f);
}

// Where one target quad (column cx, rows iz0 .. iz0+3) sits: kind 0, every
// ring cell around it lies in one top or bottom strip; 1, in one left or right
// strip; 2, anything else.
struct RingQuad {
  int Dl, Dc, Dr, kind;
  bool upper, left;
  __device__ __forceinline__ RingQuad(const ShotDev &g, int cx, int iz0) {
    Dl = dist_x(g, cx - 1), Dc = dist_x(g, cx), Dr = dist_x(g, cx + 1);
    const int Za = dist_z(g, iz0 - 1), Zb = dist_z(g, iz0 + 4);
    const int Dmax = max(max(Dl, Dr), Dc), Dmin = min(min(Dl, Dr), Dc);
    const bool lower = iz0 + 4 >= g.pml + g.nz, right = cx + 1 >= g.pml + g.nx;
    upper = iz0 - 1 < g.pml;
    left = cx - 1 < g.pml;
    // largest and smallest distance along z over the rows iz0 - 1 .. iz0 + 4
    const bool twice = upper && lower;
    const int Zmax = max(Za, Zb), Zmin = twice ? 0 : min(Za, Zb);
    kind = !twice && (Dmax == 0 || Zmin > Dmax) ? 0
           : !(left && right) && (Zmax == 0 || (Dmin > Zmax && !twice)) ? 1 : 2;
  }
};

// The terms of a quad of kind 0 or 1, summed in ring_cell's order: by column,
// rows fastest.
template <int TX, int TZ, class UA_>
__device__ __forceinline__ RingTerms ring_quad(const ShotDev &g, const RingQuad &k,
                                               const AdjTab<TX, TZ> &T, const UA_ &U, int x0,
                                               int z0, int cx, int iz0) {
  RingTerms o;
  const int Dl = k.Dl, Dc = k.Dc, Dr = k.Dr;
  const bool upper = k.upper, left = k.left;
  const V4 one = v4(1.0f);
  auto weight = [&](const V4 &d) { return fma4(d, v4(-g.inv_pml), one); };
  const V4 Zq = dist_quad(g, iz0);
  const float4 q = U.quad(cx, iz0);
  o.w = weight(Dc > 0 ? v4((float)Dc) : Zq);
  // every ring cell around the quad in one top or bottom strip
  if (k.kind == 0) {
    const float(*t)[AdjTab<TX, TZ>::NC] = T.z[!upper];
    const int c = cx - x0 + ADJ_TAB_M;
    const float al = t[0][c], bl = t[1][c - 1], br = t[1][c + 1], ga = t[2][c];
    const float4 ql = U.quad(cx - 1, iz0), qr = U.quad(cx + 1, iz0);
    // the rows one further out, whose inner neighbours these are
    V4 Zs, qs, qls, qrs;
    if (upper) {
      Zs = dist_quad(g, iz0 - 1);
      qs = v4(shift_up(q, U(cx, iz0 - 1)));
      qls = v4(shift_up(ql, U(cx - 1, iz0 - 1)));
      qrs = v4(shift_up(qr, U(cx + 1, iz0 - 1)));
    } else {
      Zs = dist_quad(g, iz0 + 1);
      qs = v4(shift_dn(q, U(cx, iz0 + 4)));
      qls = v4(shift_dn(ql, U(cx - 1, iz0 + 4)));
      qrs = v4(shift_dn(qr, U(cx + 1, iz0 + 4)));
    }
    // 1 - w of the rows and of those one further out; the x ramp wins in the
    // corners
    const V4 vq = one - weight(Zq), vs = one - weight(Zs);
    auto w1 = [&](int D, const V4 &vz) { return D > 0 ? one - weight(v4((float)D)) : vz; };
    const V4 rc = w1(Dc, vq) * v4(q), rs = w1(Dc, vs) * qs;
    const V4 pl = w1(Dl, vq) * v4(ql) * bl, pr = w1(Dr, vq) * v4(qr) * br;
    o.m = w1(Dl, vs) * qls * bl + rs * al + w1(Dr, vs) * qrs * br;
    if (upper) {
      o.e = rs * ga + rc * ga;
      o.b = pl - rs + rc * al + pr;
    } else {
      o.e = rc * ga + rs * ga;
      o.b = pl + rc * al - rs + pr;
    }
    return o;
  }
  // in one left or right strip
  {
    const float(*t)[AdjTab<TX, TZ>::NR] = T.x[!left];
    const int r = iz0 - z0 + ADJ_TAB_M, xn = left ? cx - 1 : cx + 1;
    const V4 wn = one - weight(v4((float)(left ? Dl : Dr))), wc = one - weight(v4((float)Dc));
    const V4 al = v4(*reinterpret_cast<const float4 *>(&t[0][r]));
    const float4 be = *reinterpret_cast<const float4 *>(&t[1][r]);
    const V4 bu = v4(shift_up(be, t[1][r - 1])), bd = v4(shift_dn(be, t[1][r + 4]));
    const V4 ga = v4(*reinterpret_cast<const float4 *>(&t[2][r]));
    const float4 n = U.quad(xn, iz0);
    const V4 nu = v4(shift_up(n, U(xn, iz0 - 1))), nd = v4(shift_dn(n, U(xn, iz0 + 4)));
    const V4 qu = v4(shift_up(q, U(cx, iz0 - 1))), qd = v4(shift_dn(q, U(cx, iz0 + 4)));
    const V4 rc = wc * v4(q), rn = wn * v4(n);
    const V4 pu = wc * qu * bu, pd = wc * qd * bd;
    o.m = wn * nu * bu + rn * al + wn * nd * bd;
    if (left) {
      o.e = rn * ga + rc * ga;
      o.b = pu - rn + rc * al + pd;
    } else {
      o.e = rc * ga + rn * ga;
      o.b = pu + rc * al + pd - rn;
    }
    return o;
  }
}

// vx M1 over the staged velocity `v` and vz M1 into `wz` of a quad
__device__ __forceinline__ void weigh_quad(const ShotDev &g, const float *m1, float *v, float *wz) {
  const V4 m = v4(*reinterpret_cast<const float4 *>(m1));
  const Coef4 k = coef4(*reinterpret_cast<const float4 *>(v), g);
  *reinterpret_cast<float4 *>(wz) = f4(k.vz * m);
  *reinterpret_cast<float4 *>(v) = f4(k.vx * m);
}

// The cells of one interior tile (no pad cell, no model-edge cell, every
// consumer 8th order): L_k = Lz(vz M1) + Lx(vx M1) + 2 M1 - M2 + R^T d = M_k;
// grad += w lap M1.  m1 and v: M1 and the velocity staged with the stencil's
// halo (v is overwritten), wz: as much again; M2 through P.  Every thread of
// the CTA calls this (it holds a block barrier).
template <int S, class SO>
__device__ __forceinline__ void adj_interior_cells(const ShotDev &g, const StepArgs &a, int x0,
                                                   int z0, const float *m1, float *v, float *wz,
                                                   const SO &P, const int (&gzq)[2],
                                                   const Imager &im) {
  SEIS_GEO(S);
  constexpr int RW = TZ + 2 * HI, HALO = (TX + 2 * HI) * RW;
  using SW = SAT<RW>;
  const int tid = threadIdx.x;
  for (int k = 4 * tid; k < HALO; k += 4 * NT_T) weigh_quad(g, m1 + k, v + k, wz + k);
  __syncthreads();
  const int ix = x0 + 2 * (tid / QZ), iz0 = z0 + 4 * (tid % QZ);
  const SW M1{m1, x0 - HI, z0 - HI}, WZ{wz, x0 - HI, z0 - HI}, WX{v, x0 - HI, z0 - HI};
  float *out = g.fa[(a.rot + 2) % 3];
  V4 sz[2], sx[2];
  float4 cw[2];
  pair_sums(WZ, WX, ix, iz0, sz, sx, cw);
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const float4 c = M1.quad(ix + j, iz0);
    float4 o = f4(add_twice(sz[j] + sx[j], v4(c)) - v4(P.quad(ix + j, iz0)));
    if (a.rec_k >= 0 && gzq[j] >= iz0 && gzq[j] <= iz0 + 3)
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (iz0 + r == gzq[j])
          set_comp(o, r, comp(o, r) + g.rec[(size_t)a.rec_k * g.nx + (ix + j - g.pml)]);
    im.store(g, a, j, ix, iz0, c);
    *reinterpret_cast<float4 *>(out + (size_t)(ix + j) * g.LDZ + iz0) = o;
  }
}

// One pad tile of a reverse step at (x0, z0), its arrays staged at `sm` (UCfg;
// the coefficient table's copies complete on tab_bar; the result is whether
// they did):
//  1. the weighted fields vz M1, vx M1 of the 8th-order consumers; tiles within
//     4 of the grid edge: the frame and low-order consumers' terms of tile and
//     halo, by their precomputed coefficients, into U;
//  2. U = L of the tile's cells, imaging on its model cells; cells with no ring
//     cell around them are final (M = L) and stored;
//  3. L of the halo's pad cells;
//  4. every quad with a pad or model-edge cell: M = w L + P_u3^T rho, E of the
//     next step and the kept prev terms.
// Bound by instruction issue and latency like the forward pad tiles.  A quad
// gathers from L by its strip's fixed directions with coefficients from
// tables; the earlier form kept four products and a mask of roles per ring
// cell in shared memory and gathered a cell at a time, at 390 thread
// instructions a cell.
// Measured: four 1280 x 480 shots 45 -> 38 us alone and 57 -> 34 us for the
// whole reverse step (64 x 32 tiles), the pad tiles of six 4000 x 1000 shots
// 73 -> 59 us.
template <int S>
__device__ __forceinline__ bool adj_pad_cells(const ShotDev &g, const StepArgs &a, int x0, int z0,
                                              float *sm, uint64_t *tab_bar, const int (&gzq)[2],
                                              const QuadSort<Geo<S>::TX * Geo<S>::QZ> &sort,
                                              bool corner, const Imager &im) {
  SEIS_GEO(S);
  using SA = SAT<SR>;
  using K = UCfg<S, MODE_ADJ>;
  using SP = SAT<K::PR>;
  using UA = UAT<G_::U3R>;
  constexpr int NHALO = G_::NHALO;
  const int tid = threadIdx.x;
  const int NX = g.NX, NZ = g.NZ;
  float *out = g.fa[(a.rot + 2) % 3];
  float *Enext = g.adj_e[(a.rot + 1) & 1];
  float *sV = sm + K::O_V, *sWZ = sm + K::O_W;
  const SA M1{sm, x0 - HXC, z0 - ZM}, WX{sV, x0 - HXC, z0 - ZM}, WZ{sWZ, x0 - HXC, z0 - ZM};
  const SP P{sm + K::O_P, x0 - 1, z0 - 4}, E{sm + K::O_D, x0 - 1, z0 - 4};
  const AdjTab<TX, TZ> &tab = *reinterpret_cast<const AdjTab<TX, TZ> *>(sm + K::O_T);
  const UA U{sm + K::O_U, x0, z0};
  const int qz = tid % QZ, cxp = tid / QZ;
  const int ix = x0 + 2 * cxp, iz0 = z0 + 4 * qz;

  // 1. weighted fields, zero at consumers outside the 8th-order region
  for (int i = 4 * tid; i < CW_C * SR; i += 4 * NT_T) {
    const int cx = x0 - HXC + i / SR, cz = z0 - ZM + i % SR;
    if (cx < 4 || cx > NX - 5 || cz + 3 < 4 || cz > NZ - 5) {
      *reinterpret_cast<float4 *>(sV + i) = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4 *>(sWZ + i) = make_float4(0.f, 0.f, 0.f, 0.f);
      continue;
    }
    weigh_quad(g, sm + i, sV + i, sWZ + i);
    if (cz < 4 || cz + 3 > NZ - 5)
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (cz + r < 4 || cz + r > NZ - 5) sV[i + r] = sWZ[i + r] = 0.0f;
  }
  // the grid edge's terms
  const int xa = max(x0 - 1, 0), xb = min(x0 + TX + 1, NX);
  const int za = max(z0 - 1, 0), zb = min(z0 + TZ + 1, NZ);
  const bool edge = xa <= 4 || za <= 4 || xb - 1 >= NX - 5 || zb - 1 >= NZ - 5;
  auto near4 = [&](int cx, int cz) {
    return cx >= 0 && cz >= 0 && cx < NX && cz < NZ &&
           min(min(cx, cz), min(NX - 1 - cx, NZ - 1 - cz)) <= 4;
  };
  if (edge) {
    const int n = edge_cells(NX, NZ);
#pragma unroll 1
    for (int b = 0; b < 4; b++) {  // top, bottom, left, right band
      const int bxa = b == 3 ? max(xa, NX - 5) : xa, bxb = b == 2 ? min(xb, 5) : xb;
      const int bza = b == 1 ? max(za, NZ - 5) : za, bzb = b == 0 ? min(zb, 5) : zb;
      const int nr = bzb - bza, nc = bxb - bxa;
      if (nr <= 0 || nc <= 0) continue;
      const float rn = 1.0f / (float)nr;  // see quot
      for (int i = tid; i < nr * nc; i += NT_T) {
        const int q = quot(i, rn);
        const int cx = bxa + q, cz = bza + (i - q * nr);
        const float *c = g.edge_coef + edge_index(b, NX, NZ, cx, cz);
        float s = 0.0f;
#pragma unroll
        for (int m = -3; m <= 3; m++) s = __fmaf_rn(__ldg(c + (size_t)(m + 3) * n), M1(cx, cz + m), s);
#pragma unroll
        for (int m = -3, k = 7; m <= 3; m++) {
          if (m == 0) continue;
          s = __fmaf_rn(__ldg(c + (size_t)k * n), M1(cx + m, cz), s);
          k++;
        }
        U.ref(cx, cz) = s;  // a cell in two bands is formed twice, to the same value
      }
    }
  }
  __syncthreads();

  // 2. the tile's cells
  {
    V4 sz[2], sx[2];
    float4 cw[2];
    pair_sums(WZ, WX, ix, iz0, sz, sx, cw);
#pragma unroll
    for (int j = 0; j < 2; j++) {
      const int cx = ix + j;
      const float4 c = M1.quad(cx, iz0);
      float4 o = f4(add_twice(sz[j] + sx[j], v4(c)));
      if (edge && (near4(cx, iz0) || near4(cx, iz0 + 3)))
#pragma unroll
        for (int r = 0; r < 4; r++)
          if (near4(cx, iz0 + r)) set_comp(o, r, comp(o, r) + U(cx, iz0 + r));
      o = f4(v4(o) - v4(P.quad(cx, iz0)) + v4(E.quad(cx, iz0)));
      if (a.rec_k >= 0 && gzq[j] >= iz0 && gzq[j] <= iz0 + 3)
#pragma unroll
        for (int r = 0; r < 4; r++)
          if (iz0 + r == gzq[j])
            set_comp(o, r, comp(o, r) + g.rec[(size_t)a.rec_k * g.nx + (cx - g.pml)]);
      im.store(g, a, j, ix, iz0, c);
      // zero outside the grid, where the gathers below may look
      *reinterpret_cast<float4 *>(&U.ref(cx, iz0)) = o;
      if (cx > g.pml && cx < g.pml + g.nx - 1 && iz0 > g.pml && iz0 + 3 < g.pml + g.nz - 1)
        *reinterpret_cast<float4 *>(out + (size_t)cx * g.LDZ + iz0) = o;
    }
  }
  // 3. the halo's pad cells; the other halo cells are no ring cells
  for (int i = tid; i < NHALO; i += NT_T) {
    int hx, hz;
    halo_cell<TX, TZ>(i, x0, z0, hx, hz);
    float u = 0.0f;
    if (hx >= 0 && hz >= 0 && hx < NX && hz < NZ && (dist_x(g, hx) | dist_z(g, hz)) != 0) {
      const float s1 = lap8(WZ(hx, hz - 4), WZ(hx, hz - 3), WZ(hx, hz - 2), WZ(hx, hz - 1),
                            WZ(hx, hz), WZ(hx, hz + 1), WZ(hx, hz + 2), WZ(hx, hz + 3),
                            WZ(hx, hz + 4));
      const float s2 = lap8(WX(hx - 4, hz), WX(hx - 3, hz), WX(hx - 2, hz), WX(hx - 1, hz),
                            WX(hx, hz), WX(hx + 1, hz), WX(hx + 2, hz), WX(hx + 3, hz),
                            WX(hx + 4, hz));
      u = __fmaf_rn(2.0f, M1(hx, hz), s1 + s2);
      if (edge && near4(hx, hz)) u = u + U(hx, hz);
      u = u - P(hx, hz) + E(hx, hz);
      const int x = hx - g.pml;
      if (a.rec_k >= 0 && x >= 0 && x < g.nx && hz == g.gz[x] + g.pml)
        u += g.rec[(size_t)a.rec_k * g.nx + x];
    }
    U.ref(hx, hz) = u;
  }
  // 4. the quads outside the model less its edge cells; their kept prev terms
  // are read ahead of the barrier
  const int xe = min(x0 + TX, NX), ze = min(z0 + TZ, NZ);
  const QuadList aff(x0, z0, xe, ze, g.pml + 1, g.pml + g.nx - 1, g.pml + 1, g.pml + g.nz - 1);
  constexpr int KMAX = (TX * QZ + NT_T - 1) / NT_T;
  float4 bold[KMAX];
  const int npure = corner ? sort.nz + sort.nx : aff.n;
  auto quad_of = [&](int e, int &cx, int &dz) { aff.quad(corner ? sort.get(e) : e, cx, dz); };
#pragma unroll
  for (int k = 0; k < KMAX; k++) {
    const int e = tid + k * NT_T;
    if (e < npure) {
      int cx, dz;
      quad_of(e, cx, dz);
      bold[k] = *reinterpret_cast<const float4 *>(g.adj_b + (size_t)cx * g.LDZ + z0 + dz);
    }
  }
  const bool landed = mbar_wait(tab_bar, 0);
  __syncthreads();
  // one cell by the general gather
  auto general = [&](int cx, int iz) {
    const float4 t = ring_cell<TX, TZ>(g, tab, U, x0, z0, cx, iz);
    const int D = dist_x(g, cx), Z = dist_z(g, iz);
    const float w = __fmaf_rn(-(float)(D > 0 ? D : Z), g.inv_pml, 1.0f);
    const size_t at = (size_t)cx * g.LDZ + iz;
    out[at] = __fmaf_rn(w, U(cx, iz), t.x);
    Enext[at] = t.y + g.adj_b[at];
    g.adj_b[at] = t.z;
  };
#pragma unroll
  for (int k = 0; k < KMAX; k++) {
    const int i = tid + k * NT_T;
    if (i >= npure) continue;
    int cx, dz;
    quad_of(i, cx, dz);
    const int iz = z0 + dz;
    const RingQuad rq(g, cx, iz);
    if (rq.kind == 2) {  // not in a corner tile: a model of a few cells
#pragma unroll 1
      for (int r = 0; r < 4 && iz + r < NZ; r++) general(cx, iz + r);
      continue;
    }
    const RingTerms t = ring_quad<TX, TZ>(g, rq, tab, U, x0, z0, cx, iz);
    const size_t at = (size_t)cx * g.LDZ + iz;
    const float4 n = f4(fma4(t.w, v4(U.quad(cx, iz)), t.m));
    const float4 e = f4(t.e + v4(bold[k])), b = f4(t.b);
    if (iz + 3 < NZ) {
      *reinterpret_cast<float4 *>(out + at) = n;
      *reinterpret_cast<float4 *>(Enext + at) = e;
      *reinterpret_cast<float4 *>(g.adj_b + at) = b;
    } else {
#pragma unroll
      for (int r = 0; r < 4; r++)
        if (iz + r < NZ) {
          out[at + r] = comp(n, r);
          Enext[at + r] = comp(e, r);
          g.adj_b[at + r] = comp(b, r);
        }
    }
  }
  // the corner tile's other quads, a cell per thread
  for (int j = tid; corner && j < 4 * sort.nm; j += NT_T) {
    int cx, dz;
    aff.quad(sort.mixed[j >> 2], cx, dz);
    const int iz = z0 + dz + (j & 3);
    if (iz < NZ) general(cx, iz);
  }
  return landed;
}

}  // namespace SEIS_NS
}  // namespace seis
