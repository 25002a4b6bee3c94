// agpu_tile32.cu — tiled gather + push + deposit of the FP32 split form with
// the reference's quadratic shapes, on the tile step of agpu_tile32.cuh.
// Bound: instruction latency at 16 warps per SM (43 % of the issue slots,
// DRAM traffic the algorithmic 76 B a particle).  The earlier kernel, one node
// per thread throughout, ran its warps with 25 of 32 lanes in a driven plasma
// (384x96x96 cells, 2.8e7 electrons): a pass of 10 steps 39.6 ms against 34.4
// now; with an ionization-born population 46.5 against 39.1; 2D 1024x256 1.64
// against 1.54.
#include "agpu_tile32.cuh"

namespace agpu {

namespace {

// S = 160: a row of 32 nodes at 8 particles per cell (256, a few more where
// the plasma is driven) is two groups, and two CTAs fit an SM's shared
// memory; with 128 a row of 257 was three groups.
template <int NDIM>
using CQ = C32<NDIM, 1, 1, 2, 2, 160>;

__device__ __forceinline__ void wq(float s, float a[3]) {
  float s2 = s * s;
  a[1] = 0.75f - s2;
  a[2] = 0.5f * (0.25f + s2 + s);
  a[0] = 1.f - a[1] - a[2];
}

// The qlh gather of one particle from the staged field pairs {E1, B1},
// {E2, B3}, {E3, B2} (q = the stencil's first node of the first pair): the
// components of a pair share rows or taps, so one 8-byte load serves two and
// the products run two at a time in packed FP32 (58 loads and about 100
// multiply-adds instead of 90 and 150).  A tap that belongs to one component
// only is added to that component alone.
__device__ __forceinline__ void gather3(const float2* __restrict__ q, float sx, float sy, float sz, float ap[6]) {
  using C = CQ<3>;
  constexpr int FX = C::FX, FXY = C::FX * C::FY, FV = C::FV;
  float ax[3], ay[3], az[3];
  wq(sx, ax);
  wq(sy, ay);
  wq(sz, az);
  const float xh[2] = {0.5f - sx, sx + 0.5f}, yh[2] = {0.5f - sy, sy + 0.5f}, zh[2] = {0.5f - sz, sz + 0.5f};
  float2 v1 = make_float2(0.f, 0.f), v2 = v1, v3 = v1;  // (E1, B1), (E2, B3), (E3, B2)
  const float2 w0 = make_float2(ax[0], xh[0]), w1 = make_float2(ax[1], xh[1]);
  const float2 u0 = make_float2(xh[0], ax[0]), u1 = make_float2(xh[1], ax[1]);
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const float2* r = q + FX * j + FXY * k;
      if (j < 2 && k < 2) {
        float2 t = __ffma2_rn(u1, r[1], __fmul2_rn(u0, r[0]));
        t.y = fmaf(ax[2], r[2].y, t.y);
        v1 = __ffma2_rn(__fmul2_rn(make_float2(ay[j], yh[j]), make_float2(az[k], zh[k])), t, v1);
      } else {
        v1.x = fmaf(ay[j] * az[k], fmaf(xh[1], r[1].x, xh[0] * r[0].x), v1.x);
      }
      if (j < 2) {
        const float2* p = r + FV;
        float2 t = __ffma2_rn(w1, p[1], __fmul2_rn(w0, p[0]));
        t.x = fmaf(ax[2], p[2].x, t.x);
        const float d = yh[j] * az[k];
        v2 = __ffma2_rn(make_float2(d, d), t, v2);
      }
      if (k < 2) {
        const float2* p = r + 2 * FV;
        float2 t = __ffma2_rn(w1, p[1], __fmul2_rn(w0, p[0]));
        t.x = fmaf(ax[2], p[2].x, t.x);
        const float d = ay[j] * zh[k];
        v3 = __ffma2_rn(make_float2(d, d), t, v3);
      }
    }
  ap[0] = v1.x;
  ap[1] = v2.x;
  ap[2] = v3.x;
  ap[3] = v1.y;
  ap[4] = v3.y;
  ap[5] = v2.y;
}

// Esirkepov terms of a particle that keeps its nearest node, added to the
// node's register sums.  With the quadratic shapes as polynomials of the
// offset s, S = (1/8 - s/2 + s^2/2, 3/4 - s^2, 1/8 + s/2 + s^2/2), the sums
// run over monomials,
//   J(d, a, b) = sum w D(d) (U0(a) v0^b + U1(a) v1^b),
// D = (s1 - s0, s1^2 - s0^2) along the component's axis, U0(a) = u0^a + u1^a/2
// and U1(a) = u1^a + u0^a/2 along the first, v0, v1 the offsets along the
// second transverse axis, and become window slots once per node
// (flush_stay): fewer operations per particle than the shapes themselves and
// no difference of nearly equal shapes in D.  The factors 3 and 3/2 of
// a, b = 0 are applied there.
// 3D: Jx (u = y) and Jy (u = x) are summed as packed pairs (Jy, Jx), v = z in
// both; Jz (u = x, v = y) by itself.  2D: Jx with y, Jy with x.
struct Stay3 {
  float2 xy[2][9];
  float z[2][9];
};
struct Stay2 {
  float2 xy[2][3];  // (Jy, Jx)
};
template <int NDIM>
struct StayOf {
  using T = Stay3;
};
template <>
struct StayOf<2> {
  using T = Stay2;
};
__device__ __forceinline__ void clear_stay(Stay3& m) {
#pragma unroll
  for (int q = 0; q < 18; ++q) {
    m.xy[q / 9][q % 9] = make_float2(0.f, 0.f);
    m.z[q / 9][q % 9] = 0.f;
  }
}
__device__ __forceinline__ void clear_stay(Stay2& m) {
#pragma unroll
  for (int q = 0; q < 6; ++q) m.xy[q / 3][q % 3] = make_float2(0.f, 0.f);
}
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

__device__ __forceinline__ void accumulate_stay(Stay3& m, const Moved& o) {
  const float2 h = dup(0.5f);
  const float2 s0 = make_float2(o.sx, o.sy), s1 = make_float2(o.nsx, o.nsy);
  const float2 sum = __fadd2_rn(s1, s0);
  const float2 e0 = __fmul2_rn(dup(o.wght), __ffma2_rn(dup(-1.f), s0, s1)), e1 = __fmul2_rn(e0, sum);
  const float2 D[2] = {make_float2(e0.y, e0.x), make_float2(e1.y, e1.x)};
  const float2 q0 = __fmul2_rn(s0, s0), q1 = __fmul2_rn(s1, s1);
  const float2 U0 = __ffma2_rn(h, s1, s0), U1 = __ffma2_rn(h, s0, s1);
  const float2 V0 = __ffma2_rn(h, q1, q0), V1 = __ffma2_rn(h, q0, q1);
  {
    const float2 b0 = dup(o.sz), b1 = dup(o.nsz), r0 = __fmul2_rn(b0, b0), r1 = __fmul2_rn(b1, b1);
    float2 p[9];
    p[1] = __fadd2_rn(b0, b1);
    p[2] = __fadd2_rn(r0, r1);
    p[3] = sum;
    p[4] = __ffma2_rn(U0, b0, __fmul2_rn(U1, b1));
    p[5] = __ffma2_rn(U0, r0, __fmul2_rn(U1, r1));
    p[6] = __fadd2_rn(q0, q1);
    p[7] = __ffma2_rn(V0, b0, __fmul2_rn(V1, b1));
    p[8] = __ffma2_rn(V0, r0, __fmul2_rn(V1, r1));
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      m.xy[d][0] = __fadd2_rn(m.xy[d][0], D[d]);
#pragma unroll
      for (int q = 1; q < 9; ++q) m.xy[d][q] = __ffma2_rn(D[d], p[q], m.xy[d][q]);
    }
  }
  {
    float Dz[2];
    Dz[0] = o.wght * (o.nsz - o.sz);
    Dz[1] = Dz[0] * (o.nsz + o.sz);
    float p[9];
    p[1] = sum.y;
    p[2] = q0.y + q1.y;
    p[3] = sum.x;
    p[4] = fmaf(U0.x, s0.y, U1.x * s1.y);
    p[5] = fmaf(U0.x, q0.y, U1.x * q1.y);
    p[6] = q0.x + q1.x;
    p[7] = fmaf(V0.x, s0.y, V1.x * s1.y);
    p[8] = fmaf(V0.x, q0.y, V1.x * q1.y);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      m.z[d][0] += Dz[d];
#pragma unroll
      for (int q = 1; q < 9; ++q) m.z[d][q] = fmaf(Dz[d], p[q], m.z[d][q]);
    }
  }
}
__device__ __forceinline__ void accumulate_stay(Stay2& m, const Moved& o) {
  const float2 s0 = make_float2(o.sx, o.sy), s1 = make_float2(o.nsx, o.nsy);
  const float2 sum = __fadd2_rn(s1, s0);
  const float2 e0 = __fmul2_rn(dup(o.wght), __ffma2_rn(dup(-1.f), s0, s1)), e1 = __fmul2_rn(e0, sum);
  const float2 D[2] = {make_float2(e0.y, e0.x), make_float2(e1.y, e1.x)};
  const float2 q = __ffma2_rn(s1, s1, __fmul2_rn(s0, s0));
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    m.xy[d][0] = __fadd2_rn(m.xy[d][0], D[d]);
    m.xy[d][1] = __ffma2_rn(D[d], sum, m.xy[d][1]);
    m.xy[d][2] = __ffma2_rn(D[d], q, m.xy[d][2]);
  }
}

// Arithmetic of the moment sums, on one component or on the packed pair.
__device__ __forceinline__ float2 operator*(float f, float2 v) { return __fmul2_rn(dup(f), v); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return __ffma2_rn(dup(-1.f), b, a); }
__device__ __forceinline__ float sub(float a, float b) { return a - b; }
__device__ __forceinline__ float2 fma_(float f, float2 a, float2 b) { return __ffma2_rn(dup(f), a, b); }
__device__ __forceinline__ float fma_(float f, float a, float b) { return fmaf(f, a, b); }

// Sums of 1, s, s^2 into sums of the three shapes.
template <class T>
__device__ __forceinline__ void slots3(T& m0, T& m1, T& m2) {
  const T e = fma_(0.125f, m0, 0.5f * m2), o = 0.5f * m1;
  m1 = sub(0.75f * m0, m2);
  m0 = sub(e, o);
  m2 = add(e, o);
}
// Moments m[d][a * 3 + b] into window slots [d][u * 3 + v].
template <class T>
__device__ __forceinline__ void slots_all(T m[2][9]) {
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    // the window slots along d are (D1 - D2)/2 and (D1 + D2)/2; the factors
    // 3 and 3/2 of a, b = 0
    const float f = q == 0 ? 1.5f : (q < 3 || q % 3 == 0) ? 0.75f : 0.5f;
    const T x = f * m[0][q], y = f * m[1][q];
    m[0][q] = sub(x, y);
    m[1][q] = add(x, y);
  }
#pragma unroll
  for (int d = 0; d < 2; ++d) {
#pragma unroll
    for (int a = 0; a < 3; ++a) slots3(m[d][3 * a], m[d][3 * a + 1], m[d][3 * a + 2]);
#pragma unroll
    for (int v = 0; v < 3; ++v) slots3(m[d][v], m[d][3 + v], m[d][6 + v]);
  }
}

// The node's register sums into the shared current tile ((lx, ly, lz) =
// local current coordinates of slot 0, node - 2).
template <int NDIM>
__device__ __forceinline__ void flush_stay(float* sJ, int lx, int ly, int lz, typename StayOf<NDIM>::T& s) {
  using C = CQ<NDIM>;
  constexpr int JX = C::JX, JXY = C::JX * C::JY, JV = C::JV;
  if constexpr (NDIM == 3) {
    float* c = sJ + lx + 1 + JX * (ly + 1) + JXY * (lz + 1);
    slots_all(s.xy);
    slots_all(s.z);
#pragma unroll
    for (int d = 0; d < 2; ++d)
#pragma unroll
      for (int u = 0; u < 3; ++u)
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const int q = 3 * u + v;
          atomicAdd(c + d + JX * u + JXY * v, s.xy[d][q].y);       // Jx: d = x, u = y, v = z
          atomicAdd(c + JV + u + JX * d + JXY * v, s.xy[d][q].x);  // Jy: d = y, u = x, v = z
          atomicAdd(c + 2 * JV + u + JX * v + JXY * d, s.z[d][q]);  // Jz: d = z, u = x, v = y
        }
  } else {
    float* c = sJ + lx + 1 + JX * (ly + 1);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float f = q ? 0.5f : 1.f;  // 1/2 of D, 2 of the constant's two shapes
      const float2 x = f * s.xy[0][q], y = f * s.xy[1][q];
      s.xy[0][q] = sub(x, y);
      s.xy[1][q] = add(x, y);
    }
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      slots3(s.xy[d][0], s.xy[d][1], s.xy[d][2]);
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        atomicAdd(c + d + JX * u, s.xy[d][u].y);
        atomicAdd(c + JV + u + JX * d, s.xy[d][u].x);
      }
    }
  }
}

template <int NDIM>
struct Quad {
  using C = CQ<NDIM>;
  static constexpr bool NODES = NDIM == 3;  // regular tiles take nodes()

  // Gather (qlh shapes from the staged fields; (lx, ly, lz) = local field
  // coordinates of node i0-1, j0-1, k0-1), push, the new position and record
  // of particle p, and its new binning key.
  static __device__ __forceinline__ Moved push(const TileArgs32& a, const float* __restrict__ sF, int p,
                                               const Rec& rec, int i0, int j0, int k0, int fx, int fy, int fz,
                                               bool interior, int nodekey) {
    constexpr int FX = C::FX, FY = C::FY, FV = C::FV;
    const Geo& g = a.g;
    const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
    Moved o;
    const float sx = rec.ox, sy = rec.oy, sz = rec.oz;
    float ap[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (NDIM == 3) {
      gather3(reinterpret_cast<const float2*>(sF) + fx + FX * (fy + FY * fz), sx, sy, sz, ap);
    } else {
      float ax1[3], ay1[3];
      wq(sx, ax1);
      wq(sy, ay1);
      const float axh[2] = {0.5f - sx, sx + 0.5f};
      const float ayh[2] = {0.5f - sy, sy + 0.5f};
      const float* e1 = sF;
      const float* e2 = sF + FV;
      const float* b3 = sF + 2 * FV;
#pragma unroll
      for (int j1 = 0; j1 < 3; ++j1) {
        int q = fx + FX * (fy + j1);
        ap[0] += ay1[j1] * (axh[0] * e1[q] + axh[1] * e1[q + 1]);
      }
#pragma unroll
      for (int j1 = 0; j1 < 2; ++j1) {
        int q = fx + FX * (fy + j1);
        ap[1] += ayh[j1] * (ax1[0] * e2[q] + ax1[1] * e2[q + 1] + ax1[2] * e2[q + 2]);
        ap[5] += ayh[j1] * (axh[0] * b3[q] + axh[1] * b3[q + 1]);
      }
    }
    float pn[3];
    const float dtg = boris32<NDIM>(a, ap, rec, pn);
    float nsx = sx + a.dtx * dtg * pn[0];
    float nsy = sy + a.dty * dtg * pn[1];
    float nsz = (NDIM == 3) ? sz + a.dtz * dtg * pn[2] : 0.f;
    const int mi = renorm(nsx), mj = renorm(nsy), mk = (NDIM == 3) ? renorm(nsz) : 0;
    const int i1n = i0 + mi, j1n = j0 + mj, k1n = k0 + mk;
    a.p.ox[p] = nsx;
    a.p.oy[p] = nsy;
    a.p.px[p] = pn[0];
    a.p.py[p] = pn[1];
    if (NDIM == 3) {
      a.p.oz[p] = nsz;
      a.p.pz[p] = pn[2];
    }
    if (!(pn[0] == pn[0] && pn[1] == pn[1] && pn[2] == pn[2])) raise_err(a.err, AGPU_EBIT_NONFINITE);
    bool keep = true;
    if ((mi | mj | mk) == 0 && interior) {
      // kept its node, away from the box edges: same cell, same tile row
      o.key = nodekey + offset_octant(nsx, nsy, nsz, NDIM);
    } else {
      a.p.cell[p] = (int)goff(g, i1n, j1n, k1n);
      keep = inside(i1n, nsx, nx) && inside(j1n, nsy, ny);
      if (NDIM == 3) keep = keep && inside(k1n, nsz, nz);
      o.key = keep ? tile_key_c<C::TX, C::TY, C::TZ, C::NQ>(a.t, i1n, j1n, (NDIM == 3) ? k1n : 3,
                                                            offset_octant(nsx, nsy, nsz, NDIM))
                   : a.t.nkeys;
    }
    o.sx = sx;
    o.sy = sy;
    o.sz = sz;
    o.nsx = nsx;
    o.nsy = nsy;
    o.nsz = nsz;
    o.mi = mi;
    o.mj = mj;
    o.mk = mk;
    o.wght = (float)slot_charge(rec.slot) * slot_wgh(rec.slot);
    o.keep = keep;
    return o;
  }

  static __device__ __forceinline__ void window(float* sJ, int lx, int ly, int lz, const Moved& m) {
    float s0[3][3], s1[3][3];
    wq(m.sx, s0[0]);
    wq(m.sy, s0[1]);
    wq(m.nsx, s1[0]);
    wq(m.nsy, s1[1]);
    if (NDIM == 3) {
      wq(m.sz, s0[2]);
      wq(m.nsz, s1[2]);
    }
    const int sh[3] = {m.mi + 1, m.mj + 1, m.mk + 1};
    deposit_window<NDIM, 3, C::JX, C::JY, C::JV>(sJ + lx + C::JX * (ly + C::JY * (NDIM == 3 ? lz : 0)), m.wght, s0, s1, sh);
  }

  static __device__ __forceinline__ void stays(float* sJ, int lane, int ly, int lz, const Dep32<C::S>& view,
                                               const unsigned char* idx, int nk) {
    typename StayOf<NDIM>::T acc;
    clear_stay(acc);
#pragma unroll 1
    for (int k = 0; k < nk; ++k) accumulate_stay(acc, view.at(idx[k * 32]));
    if (nk > 0) flush_stay<NDIM>(sJ, lane, ly, lz, acc);
  }

  // ---- regular tiles (3D): one node per thread -----------------------------
  // Where every binning key of a tile holds about the same number of records
  // (plasma that still sits on its lattice), a warp takes one x-row, a thread
  // pushes its node's particles in turn and keeps the node's sums in
  // registers throughout: no group data to write and read back, one flush per
  // node instead of one per node and group, but a warp runs as long as its
  // fullest node.  1024x256x256 cells, 5.4e8 electrons, mostly undisturbed, a
  // pass of 20 steps: 797 ms with groups alone, 730 with this path for the
  // regular tiles, 732 with it for all; on a driven 384x96x96 plasma the last
  // took 1.14 times as long.  The line: no key above 9/8 of the mean (a key
  // of plasma on its lattice holds 32 of 32, of a randomised one 32 +- 6), at
  // most LIST particles.
  static constexpr int LIST = (NDIM == 3) ? 5632 : 0;  // node-sorted record indices
  static constexpr int QCAP = 48;                      // mover queue entries per warp
  static constexpr int QDRAIN = 16;                    // drain the queue from this fill on
  static constexpr int QW = 8;                         // words per queue entry
  static constexpr int NCELL = C::TX * C::TY * C::TZ;
  // the groups' shared memory, laid out for this path: 2 x NT packed slots and
  // records (two staging buffers), node starts and cursors, list, queues
  static constexpr int W_REC = 4 * NT, W_START = W_REC + 12 * NT, W_CUR = W_START + NCELL + 1, W_LIST = W_CUR + NCELL;
  static constexpr int W_Q = W_LIST + LIST;
  static_assert(NDIM == 2 || W_Q + C::NW * QW * QCAP <= C::NW * C::G_WORDS, "fits the groups' shared memory");
  static_assert(QCAP >= QDRAIN - 1 + 32, "a warp adds at most 32 entries per iteration");

  // Mover queue: entry e, word j at q[j * QCAP + e]; word 0 packs the
  // tile-local node (bits 0-9) and the node changes + 1 (bits 10-15).
  static __device__ __forceinline__ void put(float* q, int e, int lc, const Moved& m) {
    q[0 * QCAP + e] = __int_as_float(lc | ((m.mi + 1) << 10) | ((m.mj + 1) << 12) | ((m.mk + 1) << 14));
    q[1 * QCAP + e] = m.sx;
    q[2 * QCAP + e] = m.sy;
    q[3 * QCAP + e] = m.sz;
    q[4 * QCAP + e] = m.nsx;
    q[5 * QCAP + e] = m.nsy;
    q[6 * QCAP + e] = m.nsz;
    q[7 * QCAP + e] = m.wght;
  }
  static __device__ __forceinline__ void drain(float* sJ, const float* q, int e) {
    const int w0 = __float_as_int(q[e]), lc = w0 & 1023;
    Moved m;
    m.mi = ((w0 >> 10) & 3) - 1;
    m.mj = ((w0 >> 12) & 3) - 1;
    m.mk = ((w0 >> 14) & 3) - 1;
    m.sx = q[1 * QCAP + e];
    m.sy = q[2 * QCAP + e];
    m.sz = q[3 * QCAP + e];
    m.nsx = q[4 * QCAP + e];
    m.nsy = q[5 * QCAP + e];
    m.nsz = q[6 * QCAP + e];
    m.wght = q[7 * QCAP + e];
    window(sJ, lc % C::TX, (lc / C::TX) % C::TY, lc / (C::TX * C::TY), m);
  }
  static __device__ __forceinline__ void nodes(const TileArgs32& a, const float* __restrict__ sF, float* sJ, int* sHist,
                                               float* area, int kbase, int beg, int end, int i0t, int j0t, int k0t) {
    constexpr int TX = C::TX, TY = C::TY, TZ = C::TZ, NPASS = NCELL / NT;
    const Geo& g = a.g;
    const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* sStart = reinterpret_cast<int*>(area + W_START);
    int* sCur = reinterpret_cast<int*>(area + W_CUR);
    int* sList = reinterpret_cast<int*>(area + W_LIST);
    __shared__ int sWarp[NT / 32];
    for (int e = threadIdx.x; e < NCELL; e += NT) sCur[e] = 0;
    __syncthreads();
    // 2: counting sort of the tile's particles by node; each thread holds
    // its (at most U) record indices and nodes in registers, all
    // loads of a thread in flight together
    // (the slots past the chunk's particles are skipped: nu is the same
    // for the whole CTA)
    constexpr int U = LIST / NT;
    const int nu = (end - beg + NT - 1) / NT;
    int pv[U], lv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      pv[u] = -1;
      lv[u] = 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      const int q = beg + threadIdx.x + u * NT;
      pv[u] = (q < end) ? __ldg(&a.perm[q]) : -1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      lv[u] = (pv[u] >= 0) ? a.p.cell[pv[u]] : 0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      if (pv[u] < 0) continue;
      int i0, j0, k0;
      cell_split(g, lv[u], i0, j0, k0);
      const unsigned lx = (unsigned)(i0 - i0t), ly = (unsigned)(j0 - j0t), lz = (unsigned)(k0 - k0t);
      if (lx < (unsigned)TX && ly < (unsigned)TY && lz < (unsigned)TZ) {
        lv[u] = lx + TX * (ly + TY * lz);
        atomicAdd(&sCur[lv[u]], 1);
      } else {
        raise_err(a.err, AGPU_EBIT_INDEX);  // not binned in this tile: drop it
        a.key[pv[u]] = a.t.nkeys;
        hist_add(a.hist, a.t.nkeys);
        pv[u] = -1;
      }
    }
    __syncthreads();
    {
      // exclusive scan of the NCELL counts, NPASS consecutive per thread
      int c[NPASS], s = 0;
#pragma unroll
      for (int u = 0; u < NPASS; ++u) {
        c[u] = sCur[threadIdx.x * NPASS + u];
        s += c[u];
      }
      int incl = s;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane == 31) sWarp[warp] = incl;
      __syncthreads();
      int wbase = 0;
#pragma unroll
      for (int w = 0; w < NT / 32; ++w) wbase += (w < warp) ? sWarp[w] : 0;
      int st = wbase + incl - s;
#pragma unroll
      for (int u = 0; u < NPASS; ++u) {
        sStart[threadIdx.x * NPASS + u] = st;
        sCur[threadIdx.x * NPASS + u] = st;
        st += c[u];
      }
      if (threadIdx.x == NT - 1) sStart[NCELL] = st;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= nu) break;
      if (pv[u] >= 0) sList[atomicAdd(&sCur[lv[u]], 1)] = pv[u];
    }
    __syncthreads();

    // 3: one node per thread, pass by pass (a warp = one x-row of 32 nodes);
    // the next record of the node is copied into the thread's staging slot
    // while the current one is pushed
    float* qw = area + W_Q + warp * (QW * QCAP);
    float* stg0 = area + W_REC + threadIdx.x;
    uint64_t* stg_slot0 = reinterpret_cast<uint64_t*>(area) + threadIdx.x;
    auto fetch = [&](int p, int b) {
      float* stg = stg0 + b * (6 * NT);
      cpa4(stg + 0 * NT, a.p.ox + p);
      cpa4(stg + 1 * NT, a.p.oy + p);
      cpa4(stg + 2 * NT, a.p.oz + p);
      cpa4(stg + 3 * NT, a.p.px + p);
      cpa4(stg + 4 * NT, a.p.py + p);
      cpa4(stg + 5 * NT, a.p.pz + p);
      cpa8(stg_slot0 + b * NT, a.p.slot + p);
    };
    int qn = 0;  // entries in this warp's mover queue (warp-uniform)
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll 1
    for (int pass = 0; pass < NPASS; ++pass) {
      const int lc = pass * NT + threadIdx.x;
      const int lx = lc % TX, ly = (lc / TX) % TY, lz = lc / (TX * TY);
      const int i0 = i0t + lx, j0 = j0t + ly, k0 = k0t + lz;
      const int cs = sStart[lc], nk = sStart[lc + 1] - cs;
      const int nmax = __reduce_max_sync(FULL, nk);
      // a node strictly inside the box keeps every particle that stays on it
      const bool interior = (unsigned)(i0 - 4) < (unsigned)(nx - 1) && (unsigned)(j0 - 4) < (unsigned)(ny - 1) &&
                            (unsigned)(k0 - 4) < (unsigned)(nz - 1);
      const int nodekey = kbase + (ly + TY * lz) * C::NQ;
      Stay3 acc;
      clear_stay(acc);
      int pnext = (nk > 0) ? sList[cs] : 0;
      if (nk > 0) fetch(pnext, 0);
      cpa_commit();
#pragma unroll 1
      for (int k = 0; k < nmax; ++k) {
        bool mover = false;
        Moved m;
        cpa_wait_all();
        const int p = pnext;
        const float* stg = stg0 + (k & 1) * (6 * NT);
        Rec rec;
        rec.ox = stg[0];
        rec.oy = stg[NT];
        rec.oz = stg[2 * NT];
        rec.px = stg[3 * NT];
        rec.py = stg[4 * NT];
        rec.pz = stg[5 * NT];
        rec.slot = stg_slot0[(k & 1) * NT];
        if (k + 1 < nk) {
          pnext = sList[cs + k + 1];
          fetch(pnext, (k + 1) & 1);
        }
        cpa_commit();
        if (k < nk) {
          m = push(a, sF, p, rec, i0, j0, k0, lx, ly, lz, interior, nodekey);
          a.key[p] = m.key;
          if ((unsigned)(m.key - kbase) < (unsigned)C::NSUB) atomicAdd(&sHist[m.key - kbase], 1);
          else hist_add(a.hist, m.key);
          if (m.keep) {
            if (m.mi == 0 && m.mj == 0 && m.mk == 0)
              accumulate_stay(acc, m);
            else
              mover = true;
          }
        }
        const unsigned mm = __ballot_sync(FULL, mover);
        if (mover) put(qw, qn + __popc(mm & lt), lc, m);
        qn += __popc(mm);
        if (qn >= QDRAIN) {
          // rare: hand the node sums over first so that no register sum is
          // live across the full-window deposits
          if (nk > 0) flush_stay<3>(sJ, lx, ly, lz, acc);
          clear_stay(acc);
          const int d = qn < 32 ? qn : 32;
          __syncwarp();
          if (lane < d) drain(sJ, qw, qn - d + lane);
          qn -= d;
          __syncwarp();
        }
      }
      if (nk > 0) flush_stay<3>(sJ, lx, ly, lz, acc);
    }
    __syncwarp();
    if (lane < qn) drain(sJ, qw, lane);
  }
};

}  // namespace

template <int NDIM>
__global__ void __launch_bounds__(NT, (NDIM == 3) ? 2 : 3) k32_tile(TileArgs32 a) {
  tile32_first<NDIM, Quad<NDIM>>(a, blockIdx.x);
}

template <int NDIM>
__global__ void __launch_bounds__(NT, (NDIM == 3) ? 2 : 3) k32_tile_more(TileArgs32 a) {
  tile32_more<NDIM, Quad<NDIM>>(a);
}

// One block per tile of any instance: instance i owns the global tiles
// [tile_off[i], tile_off[i+1]).
template <int NDIM>
__global__ void __launch_bounds__(NT, (NDIM == 3) ? 2 : 3) km32_tile(const MultiInst* __restrict__ d,
                                                                      const int* __restrict__ tile_off, int n) {
  const int b = blockIdx.x;
  int lo = 0, hi = n;  // tile_off[lo] <= b < tile_off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(&tile_off[mid]) <= b) lo = mid; else hi = mid;
  }
  // the instance's arguments in shared memory: read from the global
  // descriptor they would be reloaded after every global store (which the
  // compiler cannot prove does not alias them)
  __shared__ TileArgs32 sa;
  if (threadIdx.x == 0) sa = d[lo].ta;
  __syncthreads();
  tile32_all<NDIM, Quad<NDIM>>(sa, b - __ldg(&tile_off[lo]));
}

static size_t tile32_smem(int ndim) { return ndim == 3 ? CQ<3>::BYTES : CQ<2>::BYTES; }

int tile32_list_cap(int ndim) { return (ndim == 3) ? CQ<3>::CHUNK : CQ<2>::CHUNK; }

// Returns the kernels launched (hist_reset has cleared the work-list counters).
int tile_push32(const TileArgs32& a, cudaStream_t st, int sms) {
  if (a.t.ntiles <= 0) return 0;
  const size_t sm = tile32_smem(a.g.ndim);
  if (a.g.ndim == 3) {
    auto k = k32_tile<3>;
    auto k2 = k32_tile_more<3>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<a.t.ntiles, NT, sm, st>>>(a);
    if (a.work) k2<<<2 * sms, NT, sm, st>>>(a);
  } else {
    auto k = k32_tile<2>;
    auto k2 = k32_tile_more<2>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<a.t.ntiles, NT, sm, st>>>(a);
    if (a.work) k2<<<3 * sms, NT, sm, st>>>(a);
  }
  return a.work ? 2 : 1;
}

void multi_tile32(const MultiInst* d, const int* tile_off, const MultiPlan& pl, cudaStream_t st, int* launches) {
  if (pl.total_tiles <= 0) return;
  const size_t sm = tile32_smem(pl.ndim);
  if (pl.ndim == 3) {
    auto k = km32_tile<3>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<pl.total_tiles, NT, sm, st>>>(d, tile_off, pl.n);
  } else {
    auto k = km32_tile<2>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    k<<<pl.total_tiles, NT, sm, st>>>(d, tile_off, pl.n);
  }
  *launches += 1;
}

}  // namespace agpu
