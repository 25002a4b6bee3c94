// agpu_tile32.cuh — the split-form tile step (kernels in agpu_tile32.cu).
//
// One CTA of eight warps per spatial tile of TX x TY x TZ nodes (3D 32x4x4,
// 2D 32x8).  The tile's particles are the permutation range
// perm[tstart[t] .. tstart[t+1]) of the binning pass, x-row by x-row.  The CTA
//   1. stages the tile's field components plus a guard into shared memory
//      and zeroes a shared FP32 current tile with a guard;
//   2. shares the rows' groups of at most S particles out to its warps.  A
//      warp pushes its group one particle per lane (P::push: gather,
//      exact-gamma Boris, new record, next binning key); the offsets before
//      and after the move and the weight stay in shared memory, and a
//      particle that keeps its node is entered in the node's list;
//   3. the warp then deposits the particles that changed node on their full
//      windows with FP32 shared atomics, one per lane (P::window), and sums
//      the terms of the others in registers, one node per lane (P::stays),
//      before one shared atomic per window slot and node;
//   4. at the end the CTA flushes the shared currents once to the global
//      (hi, lo) pair with the TwoSum error of each global add accumulated
//      into lo (compensated accumulation), and its next histogram.
// Every current contribution is an FP32 product summed in FP32: no fixed
// point, so the discrete continuity of the Esirkepov currents holds to FP32
// round-off.
#pragma once
#include "agpu_bin.cuh"
#include "agpu_common.cuh"
#include "agpu_multi.h"
#include "agpu_tile.h"

namespace agpu {

constexpr int NT = 256;  // threads per CTA
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ int renorm(float& s) {
  int m = (s >= 0.5f) ? 1 : ((s < -0.5f) ? -1 : 0);
  s = s - (float)m;
  return m;
}
__device__ __forceinline__ bool inside(int node, float o, int n) {
  int m = node - 3;
  return ((m > 0) || (m == 0 && o > 0.f)) && ((m < n) || (m == n && o <= 0.f));
}

// Tile constants: LO (HI) field guard nodes below (above) the tile, JLO (JHI)
// current guard nodes, groups of S particles.
template <int NDIM, int LO_, int HI_, int JLO_, int JHI_, int S_>
struct C32 {
  static constexpr int LO = LO_, JLO = JLO_, S = S_;
  static constexpr int TX = (NDIM == 3) ? TILE3_X : TILE2_X;
  static constexpr int TY = (NDIM == 3) ? TILE3_Y : TILE2_Y;
  static constexpr int TZ = (NDIM == 3) ? TILE3_Z : 1;
  static constexpr int FX = TX + LO_ + HI_, FY = TY + LO_ + HI_, FZ = (NDIM == 3) ? TZ + LO_ + HI_ : 1;
  static constexpr int JX = TX + JLO_ + JHI_, JY = TY + JLO_ + JHI_, JZ = (NDIM == 3) ? TZ + JLO_ + JHI_ : 1;
  static constexpr int FV = FX * FY * FZ, JV = JX * JY * JZ;
  static constexpr int NF = (NDIM == 3) ? 6 : 3, NC = (NDIM == 3) ? 3 : 2;
  static constexpr int NQ = (NDIM == 3) ? 8 : 4, NROW = TY * TZ, NSUB = NROW * NQ;
  static constexpr int CHUNK = (NDIM == 3) ? 6144 : 4096;  // particles of a work item (a dense tile has several)
  static constexpr int NW = NT / 32;
  static constexpr int RMAX = 16;  // list entries of a node; the rest go to the movers
  // a warp's group data, in 4-byte words: the packed slots (then the weights),
  // offsets and momenta (then the new offsets), cells, record indices (then
  // the movers), node counts and lists
  static constexpr int G_COL = 2 * S, G_CELL = G_COL + 6 * S, G_MOV = G_CELL + S, G_CNT = G_MOV + S, G_IDX = G_CNT + 32;
  static constexpr int G_WORDS = G_IDX + RMAX * 32 / 4;
  // dynamic shared memory, in 4-byte words
  static constexpr int W_F = 0;
  static constexpr int W_GRP = W_F + NF * FV + (NF * FV) % 2;
  static constexpr int W_J = W_GRP + NW * G_WORDS;
  static constexpr size_t BYTES = sizeof(float) * (W_J + NC * JV);
  static_assert(W_GRP % 2 == 0 && G_WORDS % 2 == 0, "field pairs and packed slots are 8-byte aligned");
  static_assert(TX == 32 && NROW <= 32 && S <= 256 && S % 32 == 0, "a row is one node per lane; list entries in one byte");
};

// One particle record as the push reads it.
struct Rec {
  float ox, oy, oz, px, py, pz;
  uint64_t slot;
};

// Asynchronous 4- and 8-byte copies global -> shared (cp.async, sm_80+):
// a group's records are fetched together, without holding registers for the
// loads.
__device__ __forceinline__ void cpa4(void* sdst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpa8(void* sdst, const void* gsrc) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gsrc) : "memory");
}
// 4-byte copy, or a zero fill (no read) when !valid
__device__ __forceinline__ void cpa4z(void* sdst, const void* gsrc, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(sdst);
  const int n = valid ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(gsrc), "r"(n) : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cpa_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// What a push leaves for the deposit: offsets from the node whose window is
// deposited on.
struct Moved {
  float sx, sy, sz;     // before the push
  float nsx, nsy, nsz;  // after it, from the new node
  int mi, mj, mk;       // node change (-1, 0, 1)
  float wght;           // charge * weight (real(charge * wgh, sp))
  bool keep;            // still inside the box
  int key;              // new binning key
};
// A group's entries as the deposits read them.
template <int S>
struct Dep32 {
  const float* w;  // weight of entry e at w[2 e]
  const float* d;  // offset columns
  __device__ __forceinline__ Moved at(int e) const {
    Moved m;
    m.sx = d[e];
    m.sy = d[S + e];
    m.sz = d[2 * S + e];
    m.nsx = d[3 * S + e];
    m.nsy = d[4 * S + e];
    m.nsz = d[5 * S + e];
    m.mi = m.mj = m.mk = 0;
    m.wght = w[2 * e];
    m.keep = true;
    return m;
  }
};

// Element m of an N-point shape, zero outside it.
template <int N>
__device__ __forceinline__ float atn(const float* a, int m) {
  float v = 0.f;
#pragma unroll
  for (int q = 0; q < N; ++q) v = (m == q) ? a[q] : v;
  return v;
}

// Esirkepov deposit of one move on its full window (grid_part_connect.f90:
// 956-1334) into the shared current tile, N-point shapes s0 (old, on slots
// 1 .. N of each axis) and s1 (new, from slot sh on).  c: window slot
// (0, 0, 0) of the first component; components JV apart.  Old-plane and
// new-plane terms are regrouped onto the slots; a component's last slot
// along its own axis, where its running sum is zero, is left out.  Only the
// x windows are held in registers; y and z are walked with running sums, so
// the code stays small beside the push.
template <int NDIM, int N, int JX, int JY, int JV>
__device__ __forceinline__ void deposit_window(float* c, float w, const float s0[3][N], const float s1[3][N],
                                               const int sh[3]) {
  const int x0 = sh[0] < 1 ? sh[0] : 1, nx = (sh[0] == 1) ? N - 1 : N;  // slots x0 .. x0+nx
  const int y0 = sh[1] < 1 ? sh[1] : 1, y1 = (sh[1] == 2) ? N + 1 : N;
  float cx[N + 1], X0[N + 1], X1[N + 1], run = 0.f;
#pragma unroll
  for (int s = 0; s <= N; ++s) {
    const float p = atn<N>(s0[0], x0 + s - 1), q = atn<N>(s1[0], x0 + s - sh[0]);
    run += p - q;
    cx[s] = w * run;
    X0[s] = (NDIM == 3) ? fmaf(0.5f, q, p) : q + p;
    X1[s] = (NDIM == 3) ? fmaf(0.5f, p, q) : 0.f;
  }
  c += x0;
  if (NDIM == 2) {
    float cy = 0.f;
#pragma unroll 1
    for (int v = y0; v <= y1; ++v) {
      const float p = atn<N>(s0[1], v - 1), q = atn<N>(s1[1], v - sh[1]);
      cy += p - q;
#pragma unroll
      for (int s = 0; s <= N; ++s) {
        if (s > nx) continue;
        float* o = c + s + JX * v;
        if (s < nx) atomicAdd(o, cx[s] * (p + q));
        if (v < y1) atomicAdd(o + JV, (w * cy) * X0[s]);
      }
    }
    return;
  }
  const int z0 = sh[2] < 1 ? sh[2] : 1, z1 = (sh[2] == 2) ? N + 1 : N;
  float cz = 0.f;
#pragma unroll 1
  for (int t = z0; t <= z1; ++t) {
    const float A0 = atn<N>(s0[2], t - 1), A1 = atn<N>(s1[2], t - sh[2]);
    cz += A0 - A1;
    float cy = 0.f;
#pragma unroll 1
    for (int v = y0; v <= y1; ++v) {
      const float p = atn<N>(s0[1], v - 1), q = atn<N>(s1[1], v - sh[1]);
      cy += p - q;
      const float wyv = fmaf(fmaf(0.5f, q, p), A0, fmaf(0.5f, p, q) * A1), wcy = w * cy, wcz = w * cz;
#pragma unroll
      for (int s = 0; s <= N; ++s) {
        if (s > nx) continue;
        float* o = c + s + JX * (v + JY * t);
        if (s < nx) atomicAdd(o, cx[s] * wyv);
        if (v < y1) atomicAdd(o + JV, wcy * fmaf(X0[s], A0, X1[s] * A1));
        if (t < z1) atomicAdd(o + 2 * JV, wcz * fmaf(X0[s], p, X1[s] * q));
      }
    }
  }
}

// init_lpf_momenta on the first step (boris_push.f90:34-73), then the
// exact-gamma Boris push (75-168) from the gathered fields ap: the new
// momenta in pn, returns 1/gamma.
template <int NDIM>
__device__ __forceinline__ float boris32(const TileArgs32& a, const float ap[6], const Rec& rec, float pn[3]) {
  float pp[3] = {rec.px, rec.py, rec.pz};
  const uint64_t sl = rec.slot;
  const float qc = (float)slot_charge(sl);
  if (a.initial) {
    // init_lpf_momenta (boris_push.f90:34-73): p^0 -> p^{-1/2}
    float alp0 = a.dth * a.lfact * qc;
    float gi = rsqrtf(1.f + pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2]);
    float v0 = gi * pp[0], v1 = gi * pp[1], v2 = gi * pp[2];
    float e[6];
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) e[cc] = -alp0 * ap[cc];
    pp[0] = pp[0] + e[0] + v1 * e[5] - v2 * e[4];
    pp[1] = pp[1] + e[1] + v2 * e[3] - v0 * e[5];
    pp[2] = pp[2] + e[2] + v0 * e[4] - v1 * e[3];
  }
  // exact-gamma Boris (boris_push.f90:75-168)
  const float alp = a.dth * a.lfact * qc;
  const float vp[3] = {pp[0] + alp * ap[0], pp[1] + alp * ap[1], pp[2] + alp * ap[2]};
  const float bb[3] = {alp * ap[3], alp * ap[4], alp * ap[5]};
  const float b2v = bb[0] * bb[0] + bb[1] * bb[1] + bb[2] * bb[2];
  const float bv = bb[0] * vp[0] + bb[1] * vp[1] + bb[2] * vp[2];
  const float gam02 = 1.f + vp[0] * vp[0] + vp[1] * vp[1] + vp[2] * vp[2] - b2v;
  const float gam2 = 0.5f * (gam02 + sqrtf(gam02 * gam02 + 4.f * (b2v + bv * bv)));
  const float gam = sqrtf(gam2);
  const float inv = 1.f / (b2v + gam2);
  pn[0] = 2.f * (gam2 * vp[0] + bb[0] * bv + gam * (vp[1] * bb[2] - vp[2] * bb[1])) * inv - pp[0];
  pn[1] = 2.f * (gam2 * vp[1] + bb[1] * bv + gam * (vp[2] * bb[0] - vp[0] * bb[2])) * inv - pp[1];
  pn[2] = (NDIM == 3) ? 2.f * (gam2 * vp[2] + bb[2] * bv + gam * (vp[0] * bb[1] - vp[1] * bb[0])) * inv - pp[2] : 0.f;
  const float dtg = rsqrtf(1.f + pn[0] * pn[0] + pn[1] * pn[1] + pn[2] * pn[2]);
  return dtg;
}

// Particles [beg, end) of tile t's permutation range.
template <int NDIM, class P>
__device__ __forceinline__ void tile32_chunk(const TileArgs32& a, const int t, const int beg, const int end) {
  using C = typename P::C;
  constexpr int TX = C::TX, TY = C::TY, TZ = C::TZ, S = C::S;
  constexpr int FX = C::FX, FY = C::FY, JX = C::JX, JY = C::JY, JV = C::JV;
  constexpr int NF = C::NF, NC = C::NC;
  extern __shared__ __align__(16) float smem[];
  float* sF = smem + C::W_F;
  float* sJ = smem + C::W_J;
  __shared__ int sHist[C::NSUB];

  const Geo g = a.g;
  const int tx = t % a.t.ntx, ty = (t / a.t.ntx) % a.t.nty, tz = t / (a.t.ntx * a.t.nty);
  const int i0t = 3 + tx * TX, j0t = 3 + ty * TY, k0t = (NDIM == 3) ? 3 + tz * TZ : 1;
  const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kbase = t * C::NSUB;

  // 1: stage fields (nodes i0t-LO .. ), one x-row of FX nodes per
  // warp and pass (lane = node, the first FX - 32 lanes take the rest), as
  // asynchronous copies that complete while the CTA zeroes its currents
  // (nodes outside the array are zero-filled)
  __syncthreads();  // a previous chunk of this CTA has finished with shared memory
  {
    constexpr int NROW = NF * FY * C::FZ;
    const int gi0 = i0t - C::LO + lane, gi1 = gi0 + 32;
    const bool in0 = gi0 >= 1 && gi0 <= g.n1p, in1 = (lane < FX - 32) && gi1 <= g.n1p;
    for (int row = warp; row < NROW; row += NT / 32) {
      const int c = row / (FY * C::FZ), r = row - c * (FY * C::FZ);
      const int gj = j0t - C::LO + r % FY, gk = (NDIM == 3) ? k0t - C::LO + r / FY : 1;
      const bool rin = gj >= 1 && gj <= g.n2p && gk >= 1 && gk <= g.n3p;
      const float* src = a.ebf + g.ncell * c + goff(g, gi0, gj, gk);
      // 3D: component c is half c >= 3 of its pair (E1 B1, E2 B3, E3 B2)
      float* dst = (NDIM == 3) ? sF + 2 * ((c == 0 || c == 3 ? 0 : c == 1 || c == 5 ? 1 : 2) * C::FV + r * FX) + (c >= 3)
                               : sF + row * FX;
      constexpr int DS = (NDIM == 3) ? 2 : 1;
      cpa4z(dst + DS * lane, (rin && in0) ? src : a.ebf, rin && in0);
      if (lane < FX - 32) cpa4z(dst + DS * (32 + lane), (rin && in1) ? src + 32 : a.ebf, rin && in1);
    }
    cpa_commit();
  }
  for (int e = threadIdx.x; e < NC * JV; e += NT) sJ[e] = 0.f;
  for (int e = threadIdx.x; e < C::NSUB; e += NT) sHist[e] = 0;
  cpa_wait_all();  // this thread's field copies; the barrier makes all of them visible
  __syncthreads();

  bool regular = false;
  if constexpr (P::NODES) {
    const int kfirst = a.tstart[kbase], np = a.tstart[kbase + C::NSUB] - kfirst;
    const int q = threadIdx.x < C::NSUB ? a.tstart[kbase + threadIdx.x + 1] - a.tstart[kbase + threadIdx.x] : 0;
    const bool uneven = (long long)q * (8 * C::NSUB) > 9ll * np;
    regular = !__syncthreads_or(uneven) && np <= P::LIST && beg == kfirst && end - beg == np;
    if (regular) P::nodes(a, sF, sJ, sHist, smem + C::W_GRP, kbase, beg, end, i0t, j0t, k0t);
  }
  if (!regular) {
    // lane r: the chunk's part of row r and its groups
    int rb = 0, re = 0;
    if (lane < C::NROW) {
      rb = max(beg, a.tstart[kbase + lane * C::NQ]);
      re = min(end, a.tstart[kbase + (lane + 1) * C::NQ]);
    }
    // a row's groups of about equal size, whole batches of 32 but for the last
    const int ng = re > rb ? (re - rb + S - 1) / S : 0;
    const int gsz = ng ? ((re - rb + ng - 1) / ng + 31) / 32 * 32 : 0;
    int incl = ng;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    // 2, 3: the warp's groups
    float* gw = smem + C::W_GRP + warp * C::G_WORDS;
    uint64_t* dslot = reinterpret_cast<uint64_t*>(gw);
    float* dep = gw + C::G_COL;
    int* cell = reinterpret_cast<int*>(gw + C::G_CELL);
    int* mov = reinterpret_cast<int*>(gw + C::G_MOV);
    int* cnt = reinterpret_cast<int*>(gw + C::G_CNT);
    unsigned char* idx = reinterpret_cast<unsigned char*>(gw + C::G_IDX);
    const unsigned lt = (1u << lane) - 1u;
    const Dep32<S> view{gw, dep};
    int row = 0, n = 0;  // the warp's group: row, particles, record indices
    int pv[S / 32];
    auto group = [&](int gr) {
      row = __popc(__ballot_sync(FULL, incl <= gr));
      const int c0 = __shfl_sync(FULL, rb, row) + (gr - __shfl_sync(FULL, incl - ng, row)) * __shfl_sync(FULL, gsz, row);
      n = min(__shfl_sync(FULL, gsz, row), __shfl_sync(FULL, re, row) - c0);
#pragma unroll
      for (int u = 0; u < S / 32; ++u) pv[u] = (u * 32 + lane < n) ? __ldg(&a.perm[c0 + u * 32 + lane]) : 0;
    };
    if (warp < total) group(warp);
#pragma unroll 1
    for (int gr = warp; gr < total; gr += C::NW) {
      const int ly = row % TY, lz = row / TY, nn = n, nodekey = kbase + row * C::NQ;
      const int j0 = j0t + ly, k0 = (NDIM == 3) ? k0t + lz : 1;
      const int rowcell = (int)goff(g, i0t, j0, k0);
      cnt[lane] = 0;
#pragma unroll
      for (int u = 0; u < S / 32; ++u) {
        const int e = u * 32 + lane;
        if (e < nn) {
          const int p = pv[u];
          mov[e] = p;
          cpa4(cell + e, a.p.cell + p);
          cpa4(dep + e, a.p.ox + p);
          cpa4(dep + S + e, a.p.oy + p);
          if (NDIM == 3) cpa4(dep + 2 * S + e, a.p.oz + p);
          cpa4(dep + 3 * S + e, a.p.px + p);
          cpa4(dep + 4 * S + e, a.p.py + p);
          if (NDIM == 3) cpa4(dep + 5 * S + e, a.p.pz + p);
          cpa8(dslot + e, a.p.slot + p);
        }
        cpa_commit();
      }
      __syncwarp();
      int nmov = 0;  // warp-uniform
      int nhist = 0;  // lane q < NQ: records of the group whose new key is the row's q-th
#pragma unroll 1
      for (int b = 0; b < nn; b += 32) {
        // the batch's copies (each lane reads what it copied itself)
        if (b == 0) asm volatile("cp.async.wait_group %0;\n" ::"n"(S / 32 - 1) : "memory");
        else if (b == 32) asm volatile("cp.async.wait_group %0;\n" ::"n"(S / 32 - 2) : "memory");
        else cpa_wait_all();
        const int e = b + lane;
        int meta = -1;  // mover list entry
        int key = -1;   // new key, from the row's first
        if (e < nn) {
          Rec rec;
          rec.ox = dep[e];
          rec.oy = dep[S + e];
          rec.oz = (NDIM == 3) ? dep[2 * S + e] : 0.f;
          rec.px = dep[3 * S + e];
          rec.py = dep[4 * S + e];
          rec.pz = (NDIM == 3) ? dep[5 * S + e] : 0.f;
          rec.slot = dslot[e];
          const int p = mov[e], lx = cell[e] - rowcell;
          if ((unsigned)lx >= (unsigned)TX || i0t + lx > g.n1p) {
            raise_err(a.err, AGPU_EBIT_INDEX);  // not binned in this row: drop it
            a.key[p] = a.t.nkeys;
            hist_add(a.hist, a.t.nkeys);
          } else {
            const int i0 = i0t + lx;
            // a node strictly inside the box keeps every particle that stays on it
            const bool interior = (unsigned)(i0 - 4) < (unsigned)(nx - 1) && (unsigned)(j0 - 4) < (unsigned)(ny - 1) &&
                                  (NDIM == 2 || (unsigned)(k0 - 4) < (unsigned)(nz - 1));
            const Moved m = P::push(a, sF, p, rec, i0, j0, k0, lx, ly, lz, interior, nodekey);
            a.key[p] = m.key;
            key = m.key - nodekey;
            // the next histogram: keys of this row are counted by ballots below,
            // the tile's others in shared memory
            if ((unsigned)key >= (unsigned)C::NQ) {
              if ((unsigned)(m.key - kbase) < (unsigned)C::NSUB) atomicAdd(&sHist[m.key - kbase], 1);
              else hist_add(a.hist, m.key);
            }
            if (m.keep) {
              dep[3 * S + e] = m.nsx;
              dep[4 * S + e] = m.nsy;
              if (NDIM == 3) dep[5 * S + e] = m.nsz;
              gw[2 * e] = m.wght;
              bool mover = (m.mi | m.mj | m.mk) != 0;
              if (!mover) {
                const int rank = atomicAdd(&cnt[lx], 1);
                if (rank < C::RMAX) idx[rank * 32 + lx] = (unsigned char)e;
                else mover = true;  // the node's list is full: the general path serves it too
              }
              if (mover) meta = e | (lx << 8) | ((m.mi + 1) << 13) | ((m.mj + 1) << 15) | ((m.mk + 1) << 17);
            }
          }
        }
        {
          const bool in = (unsigned)key < (unsigned)C::NQ;
          unsigned h = __ballot_sync(FULL, in);
#pragma unroll
          for (int q = 1; q < C::NQ; q <<= 1) {
            const unsigned bq = __ballot_sync(FULL, in && (key & q));
            h &= (lane & q) ? bq : ~bq;
          }
          nhist += __popc(h);
        }
        const unsigned mm = __ballot_sync(FULL, meta >= 0);
        __syncwarp();
        if (meta >= 0) mov[nmov + __popc(mm & lt)] = meta;  // slots of this batch or earlier ones
        nmov += __popc(mm);
      }
      if (lane < C::NQ && nhist) atomicAdd(&sHist[nodekey - kbase + lane], nhist);
      // the next group's record indices, on their way during the deposits
      if (gr + C::NW < total) group(gr + C::NW);
      __syncwarp();
      for (int q = lane; q < nmov; q += 32) {
        const int meta = mov[q], e = meta & 255;
        Moved m = view.at(e);
        m.mi = ((meta >> 13) & 3) - 1;
        m.mj = ((meta >> 15) & 3) - 1;
        m.mk = ((meta >> 17) & 3) - 1;
        P::window(sJ, (meta >> 8) & 31, ly, lz, m);
      }
      const int nk = min(cnt[lane], C::RMAX);
      if (__any_sync(FULL, nk > 0)) P::stays(sJ, lane, ly, lz, view, idx + lane, nk);
      __syncwarp();
    }
  }
  __syncthreads();
  // 4: the tile's histogram counts, then one compensated flush of its
  // currents (nodes i0t-JLO ..)
  for (int e = threadIdx.x; e < C::NSUB; e += NT)
    if (sHist[e]) atomicAdd(&a.hist[kbase + e], sHist[e]);
  // x-rows of JX nodes, R per warp and pass (lane = node, the first
  // JX - 32 lanes take the rest): the rows' global adds in flight together,
  // then their TwoSum errors into lo
  {
    constexpr int NROW = NC * JY * C::JZ;
    const int gi0 = i0t - C::JLO + lane;
    const bool xin0 = gi0 >= 1 && gi0 <= g.n1p, xin1 = (lane < JX - 32) && gi0 + 32 <= g.n1p;
    constexpr int R = 8;  // rows of a warp in flight
    for (int row0 = warp; row0 < NROW; row0 += R * (NT / 32)) {
      float v[2 * R], old[2 * R];
      long long o[R];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int row = row0 + u * (NT / 32);
        v[2 * u] = v[2 * u + 1] = 0.f;
        o[u] = 0;
        if (row < NROW) {
          const int c = row / (JY * C::JZ), r = row - c * (JY * C::JZ);
          const int gj = j0t - C::JLO + r % JY, gk = (NDIM == 3) ? k0t - C::JLO + r / JY : 1;
          const bool rin = gj >= 1 && gj <= g.n2p && gk >= 1 && gk <= g.n3p;
          v[2 * u] = sJ[row * JX + lane];
          v[2 * u + 1] = (lane < JX - 32) ? sJ[row * JX + 32 + lane] : 0.f;
          const bool in0 = rin && xin0, in1 = rin && xin1;
          if ((v[2 * u] != 0.f && !in0) || (v[2 * u + 1] != 0.f && !in1)) {
            raise_err(a.err, AGPU_EBIT_INDEX);
            if (!in0) v[2 * u] = 0.f;
            if (!in1) v[2 * u + 1] = 0.f;
          }
          o[u] = g.ncell * c + goff(g, gi0, gj, gk);
        }
      }
#pragma unroll
      for (int e = 0; e < 2 * R; ++e)
        old[e] = (v[e] != 0.f) ? atomicAdd(&a.jhi[o[e >> 1] + 32 * (e & 1)], v[e]) : 0.f;
#pragma unroll
      for (int e = 0; e < 2 * R; ++e) {
        if (v[e] == 0.f) continue;
        const float sm = __fadd_rn(old[e], v[e]);
        const float bp = __fsub_rn(sm, old[e]);
        const float err = __fadd_rn(__fsub_rn(old[e], __fsub_rn(sm, bp)), __fsub_rn(v[e], bp));
        if (err != 0.f) atomicAdd(&a.jlo[o[e >> 1] + 32 * (e & 1)], err);
      }
    }
  }
}

// Tile t, first chunk of at most CHUNK particles; the CTA lists the
// tile's further chunks (a dense tile) as (tile, chunk) pairs for the
// second launch (tile32_more).
template <int NDIM, class P>
__device__ __forceinline__ void tile32_first(const TileArgs32& a, const int t) {
  constexpr int CAP = P::C::CHUNK;
  const int beg = a.tstart[t * a.t.nsub], end = a.tstart[(t + 1) * a.t.nsub];
  if (beg >= end) return;
  const int nch = (end - beg + CAP - 1) / CAP;
  if (nch > 1 && threadIdx.x == 0) {
    const unsigned base = atomicAdd(&a.work_n[0], (unsigned)(nch - 1));
    for (int c = 1; c < nch; ++c) {
      const unsigned e = base + (unsigned)(c - 1);
      if (e < (unsigned)a.work_cap) {
        a.work[2 * e] = t;
        a.work[2 * e + 1] = c;
      } else {
        raise_err(a.err, AGPU_EBIT_CAPACITY);  // cannot happen: the list holds capacity / CHUNK chunks
      }
    }
  }
  tile32_chunk<NDIM, P>(a, t, beg, min(end, beg + CAP));
}

// Tile t, all its chunks in turn (the multi-instance kernel, no work list).
template <int NDIM, class P>
__device__ __forceinline__ void tile32_all(const TileArgs32& a, const int t) {
  constexpr int CAP = P::C::CHUNK;
  const int beg = a.tstart[t * a.t.nsub], end = a.tstart[(t + 1) * a.t.nsub];
  for (int c = beg; c < end; c += CAP) tile32_chunk<NDIM, P>(a, t, c, min(end, c + CAP));
}

// The listed further chunks of dense tiles, pulled by a fixed grid of CTAs
// from a shared counter (the list is complete: the first launch has finished).
template <int NDIM, class P>
__device__ __forceinline__ void tile32_more(const TileArgs32& a) {
  constexpr int CAP = P::C::CHUNK;
  __shared__ unsigned s_item;
  const unsigned total = min(a.work_n[0], (unsigned)a.work_cap);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(&a.work_n[1], 1u);
    __syncthreads();
    const unsigned item = s_item;
    if (item >= total) return;
    const int t = a.work[2 * item], c = a.work[2 * item + 1];
    const int beg = a.tstart[t * a.t.nsub], end = a.tstart[(t + 1) * a.t.nsub];
    tile32_chunk<NDIM, P>(a, t, beg + c * CAP, min(end, beg + (c + 1) * CAP));
  }
}

}  // namespace agpu
