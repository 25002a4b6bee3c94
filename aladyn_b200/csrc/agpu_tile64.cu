// agpu_tile64.cu — tiled gather + push + deposit of the plain FP64 form, on
// the tile step of agpu_tile64.cuh.  Bound: FP64 latency and shared-memory
// bandwidth at 16 warps per SM (FP64 pipe 41 % busy, LSU 56 %), no longer L2
// atomics: the earlier deposit, one particle per lane with 81 global FP64
// atomics each (4.2e11 atomics/s), took 4.5 ms a step for 1.88e7 electrons
// in a laser-driven plasma (256x96x96 cells) against 2.4 ms now; 2D
// (1024x256, 1.05e6 electrons) 0.11 against 0.045 ms.
// Compiled with -fmad=false.
#include "agpu_tile64.cuh"

namespace agpu {

namespace {

__device__ __forceinline__ int qlh_d(double xp, double ax[3], double axh[2]) {
  double xx = 3.0 + xp;
  int i = (int)(xx + 0.5);
  double sx = xx - (double)i;
  double sx2 = sx * sx;
  ax[1] = 0.75 - sx2;
  ax[2] = 0.5 * (0.25 + sx2 + sx);
  ax[0] = 1. - ax[1] - ax[2];
  axh[1] = sx + 0.5;
  axh[0] = 1. - axh[1];
  return i - 1;
}

template <int NDIM>
struct Push64 {
  using Args = TileArgs64;
  static constexpr int NF = (NDIM == 3) ? 6 : 3, LO = 1;
  static __device__ __forceinline__ const double* comp(const Args& a, int c) { return a.ebf + a.g.ncell * c; }
  // The qlh gather (fx, fy, fz are the local coordinates of the stencil's
  // first node too, the guard being one node), the exact-gamma push of
  // boris_push.f90:34-168.
  static __device__ __forceinline__ void push(const Args& a, const double* __restrict__ sF, int fx, int fy, int fz,
                                              const double xo[3], const double* rec, int p, double xn[3]) {
    using C = C64<NDIM, NF, LO>;
    constexpr int FX = C::FX, FY = C::FY, FV = C::FV, S = C::S;
    double ax1[3], axh[2], ay1[3], ayh[2], az1[3], azh[2];
    qlh_d(xo[0], ax1, axh);
    qlh_d(xo[1], ay1, ayh);
    if (NDIM == 3) qlh_d(xo[2], az1, azh);
    double ap[6] = {0, 0, 0, 0, 0, 0};
    if (NDIM == 3) {
      const double* e1 = sF;
      const double* e2 = sF + FV;
      const double* e3 = sF + 2 * FV;
      const double* b1 = sF + 3 * FV;
      const double* b2 = sF + 4 * FV;
      const double* b3 = sF + 5 * FV;
      // set_part3d_hcell_acc loop order (grid_part_connect.f90:222-281)
#pragma unroll
      for (int k1 = 0; k1 <= 2; ++k1) {
#pragma unroll
        for (int j1 = 0; j1 <= 2; ++j1) {
          double dvol = ay1[j1] * az1[k1];
          int o = fx + FX * (fy + j1 + FY * (fz + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 1; ++i1) ap[0] = ap[0] + axh[i1] * dvol * e1[o + i1];
        }
#pragma unroll
        for (int j1 = 0; j1 <= 1; ++j1) {
          double dvol = ayh[j1] * az1[k1];
          int o = fx + FX * (fy + j1 + FY * (fz + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 2; ++i1) ap[1] = ap[1] + ax1[i1] * dvol * e2[o + i1];
#pragma unroll
          for (int i1 = 0; i1 <= 1; ++i1) ap[5] = ap[5] + axh[i1] * dvol * b3[o + i1];
        }
      }
#pragma unroll
      for (int k1 = 0; k1 <= 1; ++k1) {
#pragma unroll
        for (int j1 = 0; j1 <= 1; ++j1) {
          double dvol = ayh[j1] * azh[k1];
          int o = fx + FX * (fy + j1 + FY * (fz + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 2; ++i1) ap[3] = ap[3] + ax1[i1] * dvol * b1[o + i1];
        }
#pragma unroll
        for (int j1 = 0; j1 <= 2; ++j1) {
          double dvol = ay1[j1] * azh[k1];
          int o = fx + FX * (fy + j1 + FY * (fz + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 1; ++i1) ap[4] = ap[4] + axh[i1] * dvol * b2[o + i1];
#pragma unroll
          for (int i1 = 0; i1 <= 2; ++i1) ap[2] = ap[2] + ax1[i1] * dvol * e3[o + i1];
        }
      }
    } else {
      const double* e1 = sF;
      const double* e2 = sF + FV;
      const double* b3 = sF + 2 * FV;
      // set_part2d_hcell_acc (grid_part_connect.f90:110-138)
#pragma unroll
      for (int j1 = 0; j1 <= 2; ++j1) {
        double dvol = ay1[j1];
        int o = fx + FX * (fy + j1);
#pragma unroll
        for (int i1 = 0; i1 <= 1; ++i1) {
          double dvol1 = axh[i1] * dvol;
          ap[0] = ap[0] + dvol1 * e1[o + i1];
        }
      }
#pragma unroll
      for (int j1 = 0; j1 <= 1; ++j1) {
        double dvol = ayh[j1];
        int o = fx + FX * (fy + j1);
#pragma unroll
        for (int i1 = 0; i1 <= 2; ++i1) {
          double dvol1 = ax1[i1] * dvol;
          ap[1] = ap[1] + dvol1 * e2[o + i1];
        }
#pragma unroll
        for (int i1 = 0; i1 <= 1; ++i1) {
          double dvol1 = axh[i1] * dvol;
          ap[2] = ap[2] + dvol1 * b3[o + i1];
        }
      }
    }
    double pp[3] = {rec[NDIM * S], rec[(NDIM + 1) * S], (NDIM == 3) ? rec[(NDIM + 2) * S] : 0.};
    const uint64_t sl = dbits(rec[2 * NDIM * S]);
    const double x = rec[0], y = rec[S], z = (NDIM == 3) ? rec[2 * S] : 0.;
    const double qc = (double)slot_charge(sl);
    double xnew, ynew, znew = 0.;
    if (NDIM == 3) {
#pragma unroll
      for (int c = 0; c < 6; ++c) ap[c] = qc * ap[c];
      if (a.initial) {
        double alp0 = a.dth * a.lfact;
        double efp[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) efp[c] = -alp0 * ap[c];
        double gam2 = 1. + (pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2]);
        double gam_inv = 1. / sqrt(gam2);
        double vp[3] = {gam_inv * pp[0], gam_inv * pp[1], gam_inv * pp[2]};
        pp[0] = pp[0] + efp[0] + vp[1] * efp[5] - vp[2] * efp[4];
        pp[1] = pp[1] + efp[1] + vp[2] * efp[3] - vp[0] * efp[5];
        pp[2] = pp[2] + efp[2] + vp[0] * efp[4] - vp[1] * efp[3];
      }
      double alp = a.dth * a.lfact;
      double efp[6];
#pragma unroll
      for (int c = 0; c < 6; ++c) efp[c] = alp * ap[c];
      double vp[3] = {pp[0] + efp[0], pp[1] + efp[1], pp[2] + efp[2]};
      double bb[3] = {efp[3], efp[4], efp[5]};
      double gam02 = 1. + (vp[0] * vp[0] + vp[1] * vp[1] + vp[2] * vp[2]);
      double b2v = bb[0] * bb[0] + bb[1] * bb[1] + bb[2] * bb[2];
      double bv = bb[0] * vp[0] + bb[1] * vp[1] + bb[2] * vp[2];
      gam02 = gam02 - b2v;
      double gam2 = 0.5 * (gam02 + sqrt(gam02 * gam02 + 4. * (b2v + bv * bv)));
      double gam = sqrt(gam2);
      double vph[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) vph[c] = gam2 * vp[c] + bb[c] * bv;
      vph[0] = vph[0] + gam * (vp[1] * bb[2] - vp[2] * bb[1]);
      vph[1] = vph[1] + gam * (vp[2] * bb[0] - vp[0] * bb[2]);
      vph[2] = vph[2] + gam * (vp[0] * bb[1] - vp[1] * bb[0]);
#pragma unroll
      for (int c = 0; c < 3; ++c) vph[c] = vph[c] / (b2v + gam2);
#pragma unroll
      for (int c = 0; c < 3; ++c) pp[c] = 2. * vph[c] - pp[c];
      gam2 = 1. + (pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2]);
      double dtg = a.dt / sqrt(gam2);
      xnew = x + dtg * pp[0];
      ynew = y + dtg * pp[1];
      znew = z + dtg * pp[2];
      a.pz[p] = pp[2];
      a.z[p] = znew;
    } else {
      ap[0] = qc * ap[0];
      ap[1] = qc * ap[1];
      ap[2] = qc * ap[2];
      if (a.initial) {
        double alp0 = a.dth * a.lfact;
        double efp1 = -alp0 * ap[0], efp2 = -alp0 * ap[1], efp3 = -alp0 * ap[2];
        double gam2 = 1. + (pp[0] * pp[0] + pp[1] * pp[1]);
        double gam_inv = 1. / sqrt(gam2);
        double vp1 = pp[0] * gam_inv, vp2 = pp[1] * gam_inv;
        pp[0] = pp[0] + efp1 + vp2 * efp3;
        pp[1] = pp[1] + efp2 - vp1 * efp3;
      }
      double alp = a.dth * a.lfact;
      double efp1 = alp * ap[0], efp2 = alp * ap[1], efp3 = alp * ap[2];
      double vp1 = pp[0] + efp1, vp2 = pp[1] + efp2, vp3 = efp3;
      double gam02 = 1. + (vp1 * vp1 + vp2 * vp2);
      double b2 = vp3 * vp3;
      gam02 = gam02 - b2;
      double gam2 = 0.5 * (gam02 + sqrt(gam02 * gam02 + 4. * b2));
      double gam = sqrt(gam2);
      double vph1 = gam2 * vp1 + gam * vp2 * vp3;
      double vph2 = gam2 * vp2 - gam * vp1 * vp3;
      vph1 = vph1 / (gam2 + b2);
      vph2 = vph2 / (gam2 + b2);
      double pn1 = 2. * vph1 - pp[0];
      double pn2 = 2. * vph2 - pp[1];
      pp[0] = pn1;
      pp[1] = pn2;
      gam2 = 1. + (pn1 * pn1 + pn2 * pn2);
      double dtg = a.dt / sqrt(gam2);
      xnew = x + dtg * pn1;
      ynew = y + dtg * pn2;
    }
    // comoving frame (boris_push.f90:161-166)
    if (a.vdt > 0.) xnew = xnew - a.vdt;
    a.px[p] = pp[0];
    a.py[p] = pp[1];
    a.x[p] = xnew;
    a.y[p] = ynew;
    if (!(pp[0] == pp[0] && pp[1] == pp[1] && pp[2] == pp[2])) raise_err(a.err, AGPU_EBIT_NONFINITE);
    xn[0] = xnew;
    xn[1] = ynew;
    xn[2] = znew;
  }
};

template <int NDIM>
__global__ void __launch_bounds__(C64<NDIM, 1, 1>::NT, (NDIM == 3) ? 2 : 3) k64_tile(TileArgs64 a) {
  tile64_step<NDIM, Push64<NDIM>>(a);
}

template <int NDIM>
void tile_push64_t(const TileArgs64& a, cudaStream_t st) {
  using C = C64<NDIM, Push64<NDIM>::NF, Push64<NDIM>::LO>;
  auto k = k64_tile<NDIM>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::BYTES);
  k<<<a.t.ntiles + a.extra, C::NT, C::BYTES, st>>>(a);
}

}  // namespace

void tile_push64(const TileArgs64& a, cudaStream_t st) {
  if (a.t.ntiles <= 0) return;
  if (a.g.ndim == 3) tile_push64_t<3>(a, st);
  else tile_push64_t<2>(a, st);
}

__global__ void k_hist_reset(HistReset h) { hist_reset_bin(h, blockIdx.x * blockDim.x + threadIdx.x); }
void hist_reset(const HistReset& h, cudaStream_t st) { k_hist_reset<<<(h.nkeys + 256) / 256, 256, 0, st>>>(h); }

TileGeo make_tiles(const Geo& g, int nx, int ny, int nz, bool fp32) {
  TileGeo t;
  if (g.ndim == 3) {
    t.tx = TILE3_X;
    t.ty = fp32 ? TILE3_Y : TILE64_Y;
    t.tz = fp32 ? TILE3_Z : TILE64_Z;
  } else {
    t.tx = TILE2_X;
    t.ty = TILE2_Y;
    t.tz = 1;
  }
  // alive nodes 3 .. n+3 (n+1 nodes per axis)
  t.ntx = (nx + 1 + t.tx - 1) / t.tx;
  t.nty = (ny + 1 + t.ty - 1) / t.ty;
  t.ntz = (g.ndim == 3) ? (nz + 1 + t.tz - 1) / t.tz : 1;
  t.ntiles = t.ntx * t.nty * t.ntz;
  t.nq = (g.ndim == 3) ? 8 : 4;
  t.nsub = t.ty * t.tz * t.nq;
  t.nkeys = t.ntiles * t.nsub;
  return t;
}

}  // namespace agpu
