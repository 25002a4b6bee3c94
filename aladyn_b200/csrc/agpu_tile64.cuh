// agpu_tile64.cuh — the FP64 tile step shared by the standard cycle
// (agpu_tile64.cu) and the envelope cycle's position step (agpu_env_tile.cu):
// one CTA per tile of TX x TY x TZ nodes (3D 32x4x2, 2D 32x8), one warp per
// x-row of 32 nodes.  The tile's fields plus a guard are staged in shared
// memory; each warp then takes its row's records (contiguous in the binning
// permutation) in groups of S:
//   1. particle per lane: the cycle's gather and push (P::push) in the
//      reference's statement order on the staged values, so positions and
//      momenta stay bit-identical to the oracle.  The offsets before and
//      after the move and the weight go to shared memory; a particle that
//      keeps its node is entered in that node's list, one that changes node
//      in the warp's mover list;
//   2. movers, one per lane: the full Esirkepov window with global FP64
//      atomics;
//   3. node per lane: the terms of the particles that keep this node are
//      summed in registers, one current component at a time (18 sums), the
//      three x slots of neighbouring lanes are added by shuffles, and one
//      atomic per window row and node reaches global memory.
// A row's records beyond its cap (RowList) are shared out over the warps of
// further CTAs of the same launch.
// Include only from units compiled with -fmad=false: only the current sums
// use fma(), their order is free.
#pragma once
#include "agpu_bin.cuh"
#include "agpu_common.cuh"
#include "agpu_tile.h"

namespace agpu {

// qden's nearest node of a local position and the offset from it.
__device__ __forceinline__ int node_d(double xp, double& s) {
  const double xx = 3.0 + xp;
  const int i = (int)(xx + 0.5);
  s = xx - (double)i;
  return i;
}
// Quadratic shape of an offset s from the nearest node, qden's expressions.
__device__ __forceinline__ void wq_d(double s, double a[3]) {
  const double s2 = s * s;
  a[1] = 0.75 - s2;
  a[2] = 0.5 * (0.25 + s2 + s);
  a[0] = 1. - a[1] - a[2];
}

// Tile constants, NF staged components with LO guard nodes below the tile
// and one above.  S = 128: a row of 32 nodes at 8 particles per cell holds
// two groups, so the register sums of a node cover about four particles per
// flush, and two CTAs (16 warps at 128 registers) fit an SM's shared memory.
template <int NDIM, int NF_, int LO_>
struct C64 {
  static constexpr int NF = NF_, LO = LO_;
  static constexpr int TX = (NDIM == 3) ? TILE3_X : TILE2_X;
  static constexpr int TY = (NDIM == 3) ? TILE64_Y : TILE2_Y;
  static constexpr int TZ = (NDIM == 3) ? TILE64_Z : 1;
  static constexpr int NROW = TY * TZ, NT = 32 * NROW;
  static constexpr int NQ = (NDIM == 3) ? 8 : 4, NSUB = NROW * NQ;
  static constexpr int FX = TX + LO + 1, FY = TY + LO + 1, FZ = (NDIM == 3) ? TZ + LO + 1 : 1, FV = FX * FY * FZ;
  static constexpr int S = 128;            // particles of a group
  static constexpr int RMAX = 16;          // list entries of a node; the rest go to the movers
  static constexpr int ND = 2 * NDIM + 1;  // offsets before, offsets after, weight
  static constexpr int W_DEP = NF * FV;    // doubles
  static constexpr int DOUBLES = W_DEP + NROW * ND * S;
  // node counts; the group's record indices, then its movers; next histogram
  static constexpr int INTS = NROW * (32 + S) + NSUB;
  static constexpr size_t BYTES = sizeof(double) * DOUBLES + sizeof(int) * INTS + NROW * (RMAX + 1) * 32;
  static_assert(TX == 32 && S <= 256, "one x-row of 32 nodes per warp, list entries in one byte");
};

__device__ __forceinline__ void cpa8z(void* sdst, const void* gsrc, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  const int n = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(gsrc), "r"(n) : "memory");
}

__device__ __forceinline__ void cpa8(void* sdst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gsrc) : "memory");
}

// Source lane of each lane when the lanes with `low` set come first, both
// parts in lane order; ord: 32 bytes of the warp's shared memory.
__device__ __forceinline__ int partition_lanes(bool low, unsigned char* ord) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, low), lt = (1u << lane) - 1u;
  ord[low ? __popc(m & lt) : __popc(m) + __popc(~m & lt)] = (unsigned char)lane;
  __syncwarp();
  const int src = ord[lane];
  __syncwarp();
  return src;
}

__device__ __forceinline__ void red64(double* p, double v) {
  if (v != 0.) atomicAdd(p, v);
}
// One window row of 32 neighbouring nodes: v0, v1, v2 are this lane's sums for
// the nodes one below, at and one above its own (c points at its own node).
template <bool THREE>
__device__ __forceinline__ void flush_row(double* c, int lane, double v0, double v1, double v2) {
  const double up = __shfl_down_sync(0xffffffffu, v0, 1);
  double v = (lane < 31) ? v1 + up : v1;
  if (THREE) {
    const double dn = __shfl_up_sync(0xffffffffu, v2, 1);
    if (lane > 0) v = v + dn;
  }
  red64(c, v);
  if (lane == 0) red64(c - 1, v0);
  if (THREE && lane == 31) red64(c + 1, v2);
}

// Sums of 1, s, s^2 into sums of the three shapes.
__device__ __forceinline__ void slots3(double& m0, double& m1, double& m2) {
  const double e = fma(0.125, m0, 0.5 * m2), o = 0.5 * m1;
  m1 = fma(0.75, m0, -m2);
  m0 = e - o;
  m2 = e + o;
}

// Sums of one current component over the particles that keep a node,
//   J(d, u, v) = sum w D(d) (W0(u) S0(v) + W1(u) S1(v)),
// D the running sum of (old - new) shapes along the component's axis (its
// third slot is zero), W0 = S1/2 + S0 and W1 = S1 + S0/2 along u.  The shapes
// are fixed quadratic polynomials of the offset s,
//   S = (1/8 - s/2 + s^2/2, 3/4 - s^2, 1/8 + s/2 + s^2/2),
// so the sums run over the monomials 1, s, s^2 (and s1 - s0, s1^2 - s0^2 along
// the component's axis) and are turned into window slots once per group:
// about 45 operations a particle instead of 80, and no cancellation of nearly
// equal shapes in D.  od, ou, ov: the axes' columns in the group's shared
// data (old offsets; the new ones three columns later).
template <int S>
__device__ __forceinline__ void stay_sum3(const double* __restrict__ dep, const unsigned char* __restrict__ idx, int n,
                                          int od, int ou, int ov, double acc[18]) {
  double m[2][3][3];
#pragma unroll
  for (int q = 0; q < 18; ++q) m[q / 9][(q / 3) % 3][q % 3] = 0.;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    const double* e = dep + idx[k * 32];
    const double s0 = e[od * S], s1 = e[(od + 3) * S];
    const double a0 = e[ou * S], a1 = e[(ou + 3) * S], b0 = e[ov * S], b1 = e[(ov + 3) * S];
    double D[2];
    D[0] = e[6 * S] * (s1 - s0);
    D[1] = D[0] * (s1 + s0);
    const double q0 = a0 * a0, q1 = a1 * a1, r0 = b0 * b0, r1 = b1 * b1;
    const double U0 = fma(0.5, a1, a0), U1 = fma(0.5, a0, a1), V0 = fma(0.5, q1, q0), V1 = fma(0.5, q0, q1);
    // p(a, b) of the monomials u^a v^b; the factors 3 and 3/2 of p(0, .) and
    // p(., 0) are applied after the sum
    double p[3][3];
    p[0][1] = b0 + b1;
    p[0][2] = r0 + r1;
    p[1][0] = a0 + a1;
    p[2][0] = q0 + q1;
    p[1][1] = fma(U0, b0, U1 * b1);
    p[1][2] = fma(U0, r0, U1 * r1);
    p[2][1] = fma(V0, b0, V1 * b1);
    p[2][2] = fma(V0, r0, V1 * r1);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      m[d][0][0] = m[d][0][0] + D[d];
#pragma unroll
      for (int q = 1; q < 9; ++q) m[d][q / 3][q % 3] = fma(D[d], p[q / 3][q % 3], m[d][q / 3][q % 3]);
    }
  }
  // D(0) = (D1 - D2)/2, D(1) = (D1 + D2)/2, then the slots along v and u
  // (the halves and the factors above folded into the constants)
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double f0 = a ? 0.75 : 1.5, f1 = a ? 0.5 : 0.75;  // of b = 0 and of b = 1, 2
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double f = b ? f1 : f0;
      const double x = f * m[0][a][b], y = f * m[1][a][b];
      m[0][a][b] = x - y;
      m[1][a][b] = x + y;
    }
  }
#pragma unroll
  for (int d = 0; d < 2; ++d) {
#pragma unroll
    for (int a = 0; a < 3; ++a) slots3(m[d][a][0], m[d][a][1], m[d][a][2]);
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      slots3(m[d][0][v], m[d][1][v], m[d][2][v]);
#pragma unroll
      for (int u = 0; u < 3; ++u) acc[d * 9 + u * 3 + v] = m[d][u][v];
    }
  }
}

// Element m of a three-point shape, zero outside it.
__device__ __forceinline__ double at3(const double a[3], int m) {
  return (m == 0) ? a[0] : (m == 1) ? a[1] : (m == 2) ? a[2] : 0.;
}

// Full-window Esirkepov deposit of one move (grid_part_connect.f90:979-1059,
// 1168-1334) with global FP64 atomics: e = its column of the group's shared
// data, o = offset of window slot (0, 0, 0) (old node - 2 along each axis),
// ih, jh, kh = node change + 1.  Old-plane and new-plane terms that land on
// one node are summed first; the last slot of a component along its own axis
// is zero and left out.  Only the x windows are held in registers (four slots
// from x0); y and z are walked with running sums.
template <int NDIM, int S>
__device__ __forceinline__ void deposit_full(const Geo& g, double* jc, long long o, const double* e, int ih, int jh,
                                             int kh) {
  const long long sy = g.n1p, sz = (long long)g.n1p * g.n2p;
  const double w = e[2 * NDIM * S];
  double ax0[3], axn[3], ay0[3], ayn[3], az0[3], azn[3];
  wq_d(e[0], ax0);
  wq_d(e[S], ay0);
  wq_d(e[NDIM * S], axn);
  wq_d(e[(NDIM + 1) * S], ayn);
  if (NDIM == 3) {
    wq_d(e[2 * S], az0);
    wq_d(e[5 * S], azn);
  }
  const int x0 = ih < 1 ? ih : 1, nx = (ih == 1) ? 2 : 3;  // slots x0 .. x0+nx
  const int y0 = jh < 1 ? jh : 1, y1 = (jh + 2) > 3 ? jh + 2 : 3;
  double cx[4], X0[4], X1[4], run = 0.;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const double p = at3(ax0, x0 + s - 1), q = at3(axn, x0 + s - ih);
    run = run + p - q;
    cx[s] = w * run;
    X0[s] = (NDIM == 3) ? fma(0.5, q, p) : q + p;
    X1[s] = (NDIM == 3) ? fma(0.5, p, q) : 0.;
  }
  jc += o + x0;
  if (NDIM == 2) {
    double cy = 0.;
#pragma unroll 1
    for (int v = y0; v <= y1; ++v) {
      const double p = at3(ay0, v - 1), q = at3(ayn, v - jh);
      cy = cy + p - q;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        if (s > nx) continue;
        double* c = jc + s + sy * v;
        if (s < nx) atomicAdd(c, cx[s] * (p + q));
        if (v < y1) atomicAdd(c + g.ncell, (w * cy) * X0[s]);
      }
    }
    return;
  }
  const int z0 = kh < 1 ? kh : 1, z1 = (kh + 2) > 3 ? kh + 2 : 3;
  double cz = 0.;
#pragma unroll 1
  for (int t = z0; t <= z1; ++t) {
    const double A0 = at3(az0, t - 1), A1 = at3(azn, t - kh);
    cz = cz + A0 - A1;
    double cy = 0.;
#pragma unroll 1
    for (int v = y0; v <= y1; ++v) {
      const double p = at3(ay0, v - 1), q = at3(ayn, v - jh);
      cy = cy + p - q;
      const double wyv = fma(fma(0.5, q, p), A0, fma(0.5, p, q) * A1);
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        if (s > nx) continue;
        double* c = jc + s + sy * v + sz * t;
        if (s < nx) atomicAdd(c, cx[s] * wyv);
        if (v < y1) atomicAdd(c + g.ncell, (w * cy) * fma(X0[s], A0, X1[s] * A1));
        if (t < z1) atomicAdd(c + 2 * g.ncell, (w * cz) * fma(X0[s], p, X1[s] * q));
      }
    }
  }
}

// Stages NF components of the nodes from (i0, j0, k0) on, FX x FY x FZ of them
// each, one x-row per warp and pass, as asynchronous copies (nodes outside
// the array are zero-filled); comp(c) points at component c.
template <int NF, int FX, int FY, int FZ, int NWARP, class Comp>
__device__ __forceinline__ void stage64(double* sF, const Geo& g, int i0, int j0, int k0, Comp comp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gi0 = i0 + lane, gi1 = gi0 + 32;
  const bool in0 = gi0 >= 1 && gi0 <= g.n1p, in1 = (lane < FX - 32) && gi1 <= g.n1p;
  for (int row = warp; row < NF * FY * FZ; row += NWARP) {
    const int c = row / (FY * FZ), r = row - c * (FY * FZ);
    const int gj = j0 + r % FY, gk = (FZ > 1) ? k0 + r / FY : 1;
    const bool rin = gj >= 1 && gj <= g.n2p && gk >= 1 && gk <= g.n3p;
    const double* base = comp(c);
    const double* src = base + goff(g, gi0, gj, gk);
    cpa8z(&sF[row * FX + lane], (rin && in0) ? src : base, rin && in0);
    if (lane < FX - 32) cpa8z(&sF[row * FX + 32 + lane], (rin && in1) ? src + 32 : base, rin && in1);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The next item of the dense rows for the whole CTA, or -1 (the first barrier
// also ends the CTA's item before).
__device__ __forceinline__ int next_item(const RowList& rows) {
  __shared__ int s_item;
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned i = atomicAdd(&rows.n[1], 1u);
    s_item = i < min(rows.n[0], (unsigned)rows.size) ? (int)i : -1;
  }
  __syncthreads();
  return s_item;
}
// Records [c0, end) of item q for one of nwarps warps, evenly in batches of 32.
__device__ __forceinline__ void item_records(const RowList& rows, const int* tstart, int nq, int q, int warp, int nwarps,
                                             int& c0, int& end) {
  const int row = rows.item[2 * q], first = tstart[row * nq] + (int)rows.n[3] + rows.item[2 * q + 1];
  const int n = min(ROW_ITEM, tstart[(row + 1) * nq] - first), seg = (n + 32 * nwarps - 1) / (32 * nwarps) * 32;
  c0 = first + min(n, warp * seg);
  end = min(first + n, c0 + seg);
}
// After a CTA's last item: the last of the launch's `extra` CTAs, none of
// which reads the list any more, rewinds it, or empties it for the next scan.
__device__ __forceinline__ void items_done(const RowList& rows, int extra, bool empty) {
  if (threadIdx.x == 0 && atomicInc(&rows.n[2], (unsigned)extra - 1u) == (unsigned)extra - 1u) {
    rows.n[1] = 0u;
    if (empty) rows.n[0] = 0u;
  }
}

// The body of a tile kernel: the records [c0, qend) of row `row` of tile t for
// the warp.  P: NF and LO of the staged fields, comp(a, c)
// their arrays, and push(a, sF, fx, fy, fz, xo, rec, p, xn): gather at the
// local position xo of the particle whose nearest node is (fx, fy, fz) of
// the tile, advance it and store its new position (also in xn) and momenta.
// rec points at its copied record (column stride S): x, y[, z], px, py[, pz],
// slot.
template <int NDIM, class P>
__device__ __forceinline__ void tile64_rows(const typename P::Args& a, const int t, const int row, int c0, const int qend) {
  using C = C64<NDIM, P::NF, P::LO>;
  constexpr int TX = C::TX, TY = C::TY, TZ = C::TZ;
  constexpr int S = C::S, ND = C::ND, NT = C::NT, RMAX = C::RMAX;
  extern __shared__ double smd[];
  double* sF = smd;
  int* sInt = reinterpret_cast<int*>(smd + C::DOUBLES);
  int* sHist = sInt + C::NROW * (32 + S);

  const Geo g = a.g;
  const int kbase = t * C::NSUB;
  const int tx = t % a.t.ntx, ty = (t / a.t.ntx) % a.t.nty, tz = t / (a.t.ntx * a.t.nty);
  const int i0t = 3 + tx * TX, j0t = 3 + ty * TY, k0t = (NDIM == 3) ? 3 + tz * TZ : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  double* dep = smd + C::W_DEP + warp * ND * S;
  int* cnt = sInt + warp * (32 + S);
  int* mov = cnt + 32;
  unsigned char* idx = reinterpret_cast<unsigned char*>(sHist + C::NSUB) + warp * (RMAX + 1) * 32;
  unsigned char* ord = idx + RMAX * 32;

  stage64<C::NF, C::FX, C::FY, C::FZ, C::NROW>(sF, g, i0t - C::LO, j0t - C::LO, (NDIM == 3) ? k0t - C::LO : 1,
                                               [&](int c) { return P::comp(a, c); });
  for (int e = threadIdx.x; e < C::NSUB; e += NT) sHist[e] = 0;
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();

  const int wy = row % TY, wz = row / TY;
  int pv[S / 32];  // record indices of the next group
#pragma unroll
  for (int u = 0; u < S / 32; ++u) pv[u] = (c0 + u * 32 + lane < qend) ? a.perm[c0 + u * 32 + lane] : 0;
  for (; c0 < qend; c0 += S) {
    cnt[lane] = 0;
    // the group's records are copied into the columns that their offsets take
    // after the push, all in flight together (one batch of 32 a copy group)
#pragma unroll
    for (int u = 0; u < S / 32; ++u) {
      const int e = u * 32 + lane, p = pv[u];
      if (c0 + e < qend) {
        mov[e] = p;
        cpa8(dep + e, a.x + p);
        cpa8(dep + S + e, a.y + p);
        if (NDIM == 3) cpa8(dep + 2 * S + e, a.z + p);
        cpa8(dep + NDIM * S + e, a.px + p);
        cpa8(dep + (NDIM + 1) * S + e, a.py + p);
        if (NDIM == 3) cpa8(dep + (NDIM + 2) * S + e, a.pz + p);
        cpa8(dep + 2 * NDIM * S + e, a.slot + p);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    __syncwarp();
    int nmov = 0;  // warp-uniform
    // ---- 1: gather and push, one particle per lane
#pragma unroll 1
    for (int b = 0; b < S; b += 32) {
      if (c0 + b >= qend) break;
      if (b == 0) asm volatile("cp.async.wait_group %0;\n" ::"n"(S / 32 - 1) : "memory");
      else if (b == 32) asm volatile("cp.async.wait_group %0;\n" ::"n"(S / 32 - 2) : "memory");
      else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncwarp();  // the batch's records, copied by its other lanes too
      // lanes of the row's lower 16 nodes first: an 8-byte shared load serves
      // 16 lanes at a time, and nodes i and i + 16 share banks (the records of
      // a batch stay the same, so global accesses stay coalesced)
      const int nact = min(32, qend - c0 - b);
      double s_;
      const bool low = lane < nact && node_d(a.dx_inv * (dep[b + lane] - a.xmn), s_) < i0t + 16;
      const int src = partition_lanes(low, ord);
      int meta = -1;  // mover list entry
      if (src < nact) {
        const int e = b + src;
        const int p = mov[e];  // this batch's entries are read before its movers are listed
        // (the record is read again after the gather instead of held through it)
        const double xo[3] = {a.dx_inv * (dep[e] - a.xmn), a.dy_inv * (dep[S + e] - a.ymn),
                              (NDIM == 3) ? a.dz_inv * (dep[2 * S + e] - a.zmn) : 0.};
        const int fx = node_d(xo[0], s_) - i0t, fy = node_d(xo[1], s_) - j0t, fz = (NDIM == 3) ? node_d(xo[2], s_) - k0t : 0;
        if ((unsigned)fx >= (unsigned)TX || fy != wy || (NDIM == 3 && fz != wz)) {
          raise_err(a.err, AGPU_EBIT_INDEX);  // not binned in this row: drop it
          a.key[p] = a.t.nkeys;
          hist_add(a.hist, a.t.nkeys);
        } else {
          double xn[3] = {0., 0., 0.};
          P::push(a, sF, fx, fy, fz, xo, dep + e, p, xn);
          bool keep = (xn[0] > a.gxmin && xn[0] <= a.gxmax) && (xn[1] > a.gymin && xn[1] <= a.gymax);
          if (NDIM == 3) keep = keep && (xn[2] > a.gzmin && xn[2] <= a.gzmax);
          // qden's nodes and offsets before and after the move
          double so[3] = {0., 0., 0.}, sn[3] = {0., 0., 0.};
          node_d(a.dx_inv * (dep[e] - a.xmn), so[0]);
          node_d(a.dy_inv * (dep[S + e] - a.ymn), so[1]);
          if (NDIM == 3) node_d(a.dz_inv * (dep[2 * S + e] - a.zmn), so[2]);
          const int in = node_d(a.dx_inv * (xn[0] - a.xmn), sn[0]), jn = node_d(a.dy_inv * (xn[1] - a.ymn), sn[1]);
          const int kn = (NDIM == 3) ? node_d(a.dz_inv * (xn[2] - a.zmn), sn[2]) : 0;
          const int ih = in - (i0t + fx) + 1, jh = jn - (j0t + fy) + 1, kh = (NDIM == 3) ? kn - (k0t + fz) + 1 : 1;
          // a move of more than one cell has no window slot: no current, the
          // record stays (the comoving frame can move one by almost two)
          const bool slots = (unsigned)ih <= 2u && (unsigned)jh <= 2u && (unsigned)kh <= 2u;
          if (keep && !slots) raise_err(a.err, AGPU_EBIT_INDEX);
          const int oct = offset_octant((float)sn[0], (float)sn[1], (float)sn[2], NDIM);
          const int nkey = keep ? tile_key_c<TX, TY, TZ, C::NQ>(a.t, in, jn, (NDIM == 3) ? kn : 3, oct) : a.t.nkeys;
          a.key[p] = nkey;
          // keys of this tile counted in shared memory, added to the global
          // histogram once per tile
          if ((unsigned)(nkey - kbase) < (unsigned)C::NSUB) atomicAdd(&sHist[nkey - kbase], 1);
          else hist_add(a.hist, nkey);
          if (keep && slots) {
            dep[e] = so[0];
            dep[S + e] = so[1];
            if (NDIM == 3) dep[2 * S + e] = so[2];
            dep[NDIM * S + e] = sn[0];
            dep[(NDIM + 1) * S + e] = sn[1];
            if (NDIM == 3) dep[(NDIM + 2) * S + e] = sn[2];
            const uint64_t sl = dbits(dep[2 * NDIM * S + e]);
            dep[2 * NDIM * S + e] = (double)((float)slot_charge(sl) * slot_wgh(sl));
            bool mover = ih != 1 || jh != 1 || kh != 1;
            if (!mover) {
              const int rank = atomicAdd(&cnt[fx], 1);
              if (rank < RMAX) idx[rank * 32 + fx] = (unsigned char)e;
              else mover = true;  // the node's list is full: the general path serves it too
            }
            if (mover) meta = e | (fx << 8) | (ih << 13) | (jh << 15) | (kh << 17);
          }
        }
      }
      const unsigned mm = __ballot_sync(0xffffffffu, meta >= 0);
      __syncwarp();
      if (meta >= 0) mov[nmov + __popc(mm & lt)] = meta;
      nmov += __popc(mm);
    }
    // the next group's record indices, on their way during the deposit
#pragma unroll
    for (int u = 0; u < S / 32; ++u) {
      const int q = c0 + S + u * 32 + lane;
      pv[u] = (q < qend) ? a.perm[q] : 0;
    }
    __syncwarp();
    // ---- 2: movers, the full window each (grid_part_connect.f90:979-1059, 1168-1334)
    for (int m = lane; m < nmov; m += 32) {
      const int meta = mov[m], e = meta & 255;
      const int ih = (meta >> 13) & 3, jh = (meta >> 15) & 3, kh = (meta >> 17) & 3;
      const long long o = goff(g, i0t + ((meta >> 8) & 31) - 2, j0t + wy - 2, (NDIM == 3) ? k0t + wz - 2 : 1);
      deposit_full<NDIM, S>(g, a.jc, o, dep + e, ih, jh, kh);
    }
    // ---- 3: the particles that kept their node, one node per lane
    const int n = min(cnt[lane], RMAX);
    if (__any_sync(0xffffffffu, n > 0)) {
      const long long sy = g.n1p, sz = (long long)g.n1p * g.n2p;
      double* J = a.jc + goff(g, i0t + lane, j0t + wy, (NDIM == 3) ? k0t + wz : 1);
      const unsigned char* my = idx + lane;
      if (NDIM == 3) {
        double acc[18];
        stay_sum3<S>(dep, my, n, 0, 1, 2, acc);  // Jx: d = x, u = y, v = z
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
          for (int v = 0; v < 3; ++v)
            flush_row<false>(J + (u - 1) * sy + (v - 1) * sz, lane, acc[u * 3 + v], acc[9 + u * 3 + v], 0.);
        stay_sum3<S>(dep, my, n, 1, 0, 2, acc);  // Jy: d = y, u = x, v = z
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int v = 0; v < 3; ++v)
            flush_row<true>(J + g.ncell + (d - 1) * sy + (v - 1) * sz, lane, acc[d * 9 + v], acc[d * 9 + 3 + v],
                            acc[d * 9 + 6 + v]);
        stay_sum3<S>(dep, my, n, 2, 0, 1, acc);  // Jz: d = z, u = x, v = y
#pragma unroll
        for (int d = 0; d < 2; ++d)
#pragma unroll
          for (int v = 0; v < 3; ++v)
            flush_row<true>(J + 2 * g.ncell + (v - 1) * sy + (d - 1) * sz, lane, acc[d * 9 + v], acc[d * 9 + 3 + v],
                            acc[d * 9 + 6 + v]);
      } else {
        // Jx(s, t) = sum w Dx(s) (S0y + S1y)(t), Jy(s, t) = sum w (S0x + S1x)(s) Dy(t), by moments as above
        double jx[6] = {0., 0., 0., 0., 0., 0.}, jy[6] = {0., 0., 0., 0., 0., 0.};  // jx[s*3+t], jy[s*2+t]
#pragma unroll 1
        for (int k = 0; k < n; ++k) {
          const double* e = dep + my[k * 32];
          const double x0 = e[0], y0 = e[S], x1 = e[2 * S], y1 = e[3 * S], w = e[4 * S];
          const double dx = x1 - x0, dy = y1 - y0, sx = x1 + x0, sy_ = y1 + y0;
          const double qx = fma(x1, x1, x0 * x0), qy = fma(y1, y1, y0 * y0);
          double X[2], Y[2];
          X[0] = w * dx;
          X[1] = X[0] * sx;
          Y[0] = w * dy;
          Y[1] = Y[0] * sy_;
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            jx[d * 3] = jx[d * 3] + X[d];
            jx[d * 3 + 1] = fma(X[d], sy_, jx[d * 3 + 1]);
            jx[d * 3 + 2] = fma(X[d], qy, jx[d * 3 + 2]);
            jy[d] = jy[d] + Y[d];
            jy[2 + d] = fma(Y[d], sx, jy[2 + d]);
            jy[4 + d] = fma(Y[d], qx, jy[4 + d]);
          }
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const double f = q ? 0.5 : 1.;  // 1/2 of D, 2 of the constant's two shapes
          const double x = f * jx[q], y = f * jx[3 + q];
          jx[q] = x - y;
          jx[3 + q] = x + y;
          const double u = f * jy[q * 2], v = f * jy[q * 2 + 1];
          jy[q * 2] = u - v;
          jy[q * 2 + 1] = u + v;
        }
#pragma unroll
        for (int d = 0; d < 2; ++d) {
          slots3(jx[d * 3], jx[d * 3 + 1], jx[d * 3 + 2]);
          slots3(jy[d], jy[2 + d], jy[4 + d]);
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) flush_row<false>(J + (q - 1) * sy, lane, jx[q], jx[3 + q], 0.);
#pragma unroll
        for (int d = 0; d < 2; ++d)
          flush_row<true>(J + g.ncell + (d - 1) * sy, lane, jy[d], jy[2 + d], jy[4 + d]);
      }
    }
    __syncwarp();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < C::NSUB; e += NT)
    if (sHist[e]) atomicAdd(&a.hist[kbase + e], sHist[e]);
}

// A tile's CTA, or one of the `extra` CTAs for the dense rows' items.  The
// body is inlined for each: shared by both kinds of CTA it took 1 % longer (a
// pass of 10 steps on 256x96x96 cells 30.9 ms against 30.5).
template <int NDIM, class P>
__device__ __forceinline__ void tile64_step(const typename P::Args& a) {
  using C = C64<NDIM, P::NF, P::LO>;
  const int warp = threadIdx.x >> 5;
  const int cap = a.extra ? (int)a.rows.n[3] : 0x7fffffff;
  if ((int)blockIdx.x < a.t.ntiles) {
    const int* start = a.tstart + blockIdx.x * C::NSUB;
    if (start[0] >= start[C::NSUB]) return;
    const int c0 = start[warp * C::NQ], end = start[(warp + 1) * C::NQ];
    tile64_rows<NDIM, P>(a, blockIdx.x, warp, c0, end - c0 > cap ? c0 + cap : end);
    return;
  }
  if (a.rows.n[0] == 0u) return;  // nothing to take or to rewind
  for (int q, c0, end; (q = next_item(a.rows)) >= 0;) {
    const int row = a.rows.item[2 * q];
    item_records(a.rows, a.tstart, C::NQ, q, warp, C::NROW, c0, end);
    tile64_rows<NDIM, P>(a, row / C::NROW, row % C::NROW, c0, end);
  }
  items_done(a.rows, a.extra, true);
}

}  // namespace agpu
