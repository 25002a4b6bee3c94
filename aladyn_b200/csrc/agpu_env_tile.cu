// agpu_env_tile.cu — the envelope cycle's particle steps on spatial tiles
// (FP64 form): fields staged in shared memory, one warp per x-row of 32
// nodes, deposits summed per node before they reach global memory.
//
//   k_env_acc_tile   set_env_acc + lpf_env_momenta + set_env_density
//   k_env_pos_tile   set_env_grad_interp + lpf_env_positions + box test +
//                    Esirkepov deposit + the next binning keys, on the tile
//                    step of agpu_tile64.cuh
//
// Bound: FP64 arithmetic (270 + 108 gather taps a particle) once the stencils
// come from shared memory and the atomics are per node.  The earlier
// per-particle kernels (stencils from global memory, 27 and 81 atomics a
// particle) took 1.88 and 2.15 ms for 7.1e6 particles (192x96x96 cells, 4 per
// cell) against 1.27 and 1.03 ms now.  Compiled with -fmad=false; the
// arithmetic up to the deposits keeps the reference's statement order.
#include "agpu_env.h"
#include "agpu_fp64_dep.cuh"
#include "agpu_tile64.cuh"

namespace agpu {
namespace {

template <int NDIM>
struct PushEnv {
  using Args = EnvTileArgs;
  static constexpr int NF = NDIM + 1, LO = 2;
  static __device__ __forceinline__ const double* comp(const Args& a, int c) { return a.av + a.g.ncell * c; }
  // set_env_grad_interp (grid_part_connect.f90:760-882), lpf_env_positions
  // (boris_push.f90:225-295)
  static __device__ __forceinline__ void push(const Args& a, const double* __restrict__ sF, int fx, int fy, int fz,
                                              const double xo[3], const double* rec, int p, double xn[3]) {
    using C = C64<NDIM, NF, LO>;
    constexpr int FX = C::FX, FY = C::FY, FV = C::FV, S = C::S;
    double ax1[3], axh1[3], ay1[3], ayh1[3], az1[3], azh1[3];
    int i, ih, j, jh, k = 0, kh = 0;
    qqh64(xo[0], ax1, axh1, &i, &ih);
    qqh64(xo[1], ay1, ayh1, &j, &jh);
    if (NDIM == 3) qqh64(xo[2], az1, azh1, &k, &kh);
    // local coordinates of the first stencil nodes
    const int li = fx + 1, lj = fy + 1, lk = (NDIM == 3) ? fz + 1 : 0;
    const int hi = li + ih - i, hj = lj + jh - j, hk = (NDIM == 3) ? lk + kh - k : 0;
    const double dt_lp = a.dt;
    if (NDIM == 2) {
      double ap[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j1 = 0; j1 <= 2; ++j1) {
        const double dvol = ay1[j1];
        const int o = FX * (lj + j1);
#pragma unroll
        for (int i1 = 0; i1 <= 2; ++i1) {
          const double dvol1 = dvol * axh1[i1];
          ap[1] = ap[1] + dvol1 * sF[FV + o + hi + i1];
          ap[3] = ap[3] + ax1[i1] * dvol * sF[o + li + i1];
        }
      }
#pragma unroll
      for (int j1 = 0; j1 <= 2; ++j1) {
        const double dvol = ayh1[j1];
        const int o = FX * (hj + j1);
#pragma unroll
        for (int i1 = 0; i1 <= 2; ++i1) {
          const double dvol1 = dvol * ax1[i1];
          ap[2] = ap[2] + dvol1 * sF[2 * FV + o + li + i1];
        }
      }
      const double pp1 = rec[2 * S], pp2 = rec[3 * S];
      const double gam2 = 1. + (pp1 * pp1 + pp2 * pp2) + ap[3];
      const double gam = sqrt(gam2);
      const double gam3 = gam2 * gam;
      const double b2 = 0.25 * (pp1 * ap[1] + pp2 * ap[2]);
      double gam_inv = 1. / gam;
      gam_inv = gam_inv * (1. - dt_lp * b2 / gam3);
      const double vp1 = dt_lp * gam_inv * pp1, vp2 = dt_lp * gam_inv * pp2;
      xn[0] = rec[0] + vp1;
      xn[1] = rec[S] + vp2;
    } else {
      double ap[5] = {0, 0, 0, 0, 0};
#pragma unroll
      for (int k1 = 0; k1 <= 2; ++k1) {
#pragma unroll
        for (int j1 = 0; j1 <= 2; ++j1) {
          const double dvol = ay1[j1] * az1[k1];
          const int o = FX * (lj + j1 + FY * (lk + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 2; ++i1) {
            const double dvol1 = dvol * axh1[i1];
            ap[1] = ap[1] + dvol1 * sF[FV + o + hi + i1];
            ap[4] = ap[4] + ax1[i1] * dvol * sF[o + li + i1];
          }
        }
#pragma unroll
        for (int j1 = 0; j1 <= 2; ++j1) {
          const double dvol = ayh1[j1] * az1[k1];
          const int o = FX * (hj + j1 + FY * (lk + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 2; ++i1) {
            const double dvol1 = dvol * ax1[i1];
            ap[2] = ap[2] + dvol1 * sF[2 * FV + o + li + i1];
          }
        }
#pragma unroll
        for (int j1 = 0; j1 <= 2; ++j1) {
          const double dvol = ay1[j1] * azh1[k1];
          const int o = FX * (lj + j1 + FY * (hk + k1));
#pragma unroll
          for (int i1 = 0; i1 <= 2; ++i1) {
            const double dvol1 = dvol * ax1[i1];
            ap[3] = ap[3] + dvol1 * sF[3 * FV + o + li + i1];
          }
        }
      }
      const double pp[3] = {rec[3 * S], rec[4 * S], rec[5 * S]};
      const double gam2 = 1. + (pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2]) + ap[4];
      const double gam = sqrt(gam2);
      const double gam3 = gam2 * gam;
      const double b2 = 0.25 * (pp[0] * ap[1] + pp[1] * ap[2] + pp[2] * ap[3]);
      double gam_inv = 1. / sqrt(gam2);
      gam_inv = gam_inv * (1. - dt_lp * b2 / gam3);
      double vp[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) vp[c] = dt_lp * gam_inv * pp[c];
      xn[0] = rec[0] + vp[0];
      xn[1] = rec[S] + vp[1];
      xn[2] = rec[2 * S] + vp[2];
      a.z[p] = xn[2];
    }
    if (a.vdt > 0.) xn[0] = xn[0] - a.vdt;  // comoving frame (boris_push.f90:288-294)
    a.x[p] = xn[0];
    a.y[p] = xn[1];
  }
};

template <int NDIM>
__global__ void __launch_bounds__(C64<NDIM, 1, 1>::NT, (NDIM == 3) ? 2 : 3) k_env_pos_tile(EnvTileArgs a) {
  tile64_step<NDIM, PushEnv<NDIM>>(a);
}

// Tile constants of the momentum step: in 3D a CTA takes two tiles that are
// neighbours along z (32x4x4 nodes, 16 warps): the ten staged components of
// one 32x4x2 tile would leave room for one CTA of eight warps per SM.
template <int NDIM>
struct CAcc {
  using T = C64<NDIM, 1, 2>;
  static constexpr int NZT = (NDIM == 3) ? 2 : 1;  // tiles of a CTA
  static constexpr int TX = T::TX, TY = T::TY, TZ = T::TZ * NZT;
  static constexpr int NROW = TY * TZ, NT = 32 * NROW;
  static constexpr int FX = TX + 3, FY = TY + 3, FZ = (NDIM == 3) ? TZ + 3 : 1, FV = FX * FY * FZ;
  static constexpr int NE = (NDIM == 3) ? 6 : 3, NF = NE + NDIM + 1;  // E, B; then F and grad F
  static constexpr int S = 128, RMAX = 16, ND = NDIM + 1;             // offsets and weight / gamma
  static constexpr int W_DEP = NF * FV, DOUBLES = W_DEP + NROW * ND * S;
  static constexpr int INTS = NROW * 32;
  static constexpr size_t BYTES = sizeof(double) * DOUBLES + sizeof(int) * INTS + NROW * (RMAX + 1) * 32;
};

// Density of one particle on its 3^NDIM nodes (set_env_density), for those
// beyond a node's list.
template <int NDIM, int S>
__device__ __forceinline__ void density_full(const Geo& g, double* d, const double* e) {
  double ax[3], ay[3], az[3] = {1., 0., 0.};
  wq_d(e[0], ax);
  wq_d(e[S], ay);
  if (NDIM == 3) wq_d(e[2 * S], az);
  const double w = e[NDIM * S];
  for (int k1 = 0; k1 < (NDIM == 3 ? 3 : 1); ++k1)
#pragma unroll
    for (int j1 = 0; j1 < 3; ++j1) {
      const double dv = ay[j1] * (NDIM == 3 ? at3(az, k1) : 1.) * w;
      double* r = d + (long long)g.n1p * (j1 - 1) + (NDIM == 3 ? (long long)g.n1p * g.n2p * (k1 - 1) : 0);
#pragma unroll
      for (int i1 = 0; i1 < 3; ++i1) atomicAdd(r + i1 - 1, dv * ax[i1]);
    }
}

// The records [c0, qend) of row `row` of the tiles (tx, ty, NZT zp ..) for the
// warp.
template <int NDIM>
__device__ __forceinline__ void acc_rows(const EnvTileArgs& a, const int tx, const int ty, const int zp, const int row,
                                         int c0, const int qend) {
  using C = CAcc<NDIM>;
  constexpr int FX = C::FX, FY = C::FY, FV = C::FV, NE = C::NE, S = C::S, ND = C::ND, RMAX = C::RMAX;
  extern __shared__ double smd[];
  double* sF = smd;
  const Geo g = a.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* dep = smd + C::W_DEP + warp * ND * S;
  int* cnt = reinterpret_cast<int*>(smd + C::DOUBLES) + warp * 32;
  unsigned char* idx = reinterpret_cast<unsigned char*>(smd + C::DOUBLES) + sizeof(int) * C::INTS + warp * (RMAX + 1) * 32;
  unsigned char* ord = idx + RMAX * 32;

  const int i0t = 3 + tx * C::TX, j0t = 3 + ty * C::TY, k0t = (NDIM == 3) ? 3 + zp * C::TZ : 1;
  const int wy = row % C::TY, wz = row / C::TY;

  stage64<C::NF, FX, FY, C::FZ, C::NROW>(sF, g, i0t - 2, j0t - 2, (NDIM == 3) ? k0t - 2 : 1, [&](int c) {
    return c < NE ? a.ebf + g.ncell * c : a.av + g.ncell * (c - NE);
  });
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  const double* ef = sF;
  const double* av = sF + NE * FV;
  const double dth = a.dth;
  const double alp = 0.5 * a.dt * a.lfact;
  for (; c0 < qend; c0 += S) {
    cnt[lane] = 0;
    __syncwarp();
#pragma unroll 1
    for (int bq = 0; bq < S; bq += 32) {
      if (c0 + bq >= qend) break;
      // lanes of the row's lower 16 nodes first (see tile64_step)
      const int nact = min(32, qend - c0 - bq), e = bq + lane;
      const int n0 = lane < nact ? a.perm[c0 + e] : 0;
      double s;
      const bool low = lane < nact && node_d(a.dx_inv * (a.x[n0] - a.xmn), s) < i0t + 16;
      const int src = partition_lanes(low, ord);
      const int n = __shfl_sync(0xffffffffu, n0, src);
      if (src < nact) {
        const uint64_t sl = dbits(a.slot[n]);
        const double charge = (double)slot_charge(sl);
        const double wgh = (double)slot_wgh(sl);
        double ax1[3], axh1[3], ay1[3], ayh1[3], az1[3], azh1[3];
        int i, ih, j, jh, k = 0, kh = 0;
        const double xl = a.dx_inv * (a.x[n] - a.xmn);
        const double yl = a.dy_inv * (a.y[n] - a.ymn);
        const double zl = (NDIM == 3) ? a.dz_inv * (a.z[n] - a.zmn) : 0.;
        qqh64(xl, ax1, axh1, &i, &ih);
        qqh64(yl, ay1, ayh1, &j, &jh);
        if (NDIM == 3) qqh64(zl, az1, azh1, &k, &kh);
        const int fx = i + 1 - i0t;
        if ((unsigned)fx >= (unsigned)C::TX || j + 1 - j0t != wy || (NDIM == 3 && k + 1 - k0t != wz)) {
          raise_err(a.err, AGPU_EBIT_INDEX);  // not binned in this row
        } else if (!in_stencil(i, g.n1p) || !in_stencil(ih, g.n1p) || !in_stencil(j, g.n2p) || !in_stencil(jh, g.n2p) ||
                   (NDIM == 3 && (!in_stencil(k, g.n3p) || !in_stencil(kh, g.n3p)))) {
          // the last tiles reach beyond the array: a record out there (only
          // the host can put one) is not gathered or deposited; the position
          // step drops it
          raise_err(a.err, AGPU_EBIT_INDEX);
        } else {
          const int li = fx + 1, lj = wy + 1, lk = (NDIM == 3) ? wz + 1 : 0;
          const int hi = li + ih - i, hj = lj + jh - j, hk = (NDIM == 3) ? lk + kh - k : 0;
          double wghp;
          if (NDIM == 2) {
            double ap[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int j1 = 0; j1 <= 2; ++j1) {
              const double dvol = ay1[j1];
              const int o = FX * (lj + j1);
#pragma unroll
              for (int i1 = 0; i1 <= 2; ++i1) ap[6] = ap[6] + ax1[i1] * dvol * av[o + li + i1];
#pragma unroll
              for (int i1 = 0; i1 <= 2; ++i1) {
                const double dvol1 = dvol * axh1[i1];
                ap[1] = ap[1] + dvol1 * ef[o + hi + i1];
                ap[4] = ap[4] + dvol1 * av[FV + o + hi + i1];
              }
            }
#pragma unroll
            for (int j1 = 0; j1 <= 2; ++j1) {
              const double dvol = ayh1[j1];
              const int o = FX * (hj + j1);
#pragma unroll
              for (int i1 = 0; i1 <= 2; ++i1) {
                const double dvol1 = dvol * ax1[i1];
                ap[2] = ap[2] + dvol1 * ef[FV + o + li + i1];
                ap[5] = ap[5] + dvol1 * av[2 * FV + o + li + i1];
              }
#pragma unroll
              for (int i1 = 0; i1 <= 2; ++i1) ap[3] = ap[3] + axh1[i1] * dvol * ef[2 * FV + o + hi + i1];
            }
            const double u1 = a.px[n], u2 = a.py[n];
            const double gam2 = 1. + u1 * u1 + u2 * u2 + ap[6];
#pragma unroll
            for (int c = 1; c <= 3; ++c) ap[c] = charge * ap[c];
#pragma unroll
            for (int c = 4; c <= 5; ++c) ap[c] = 0.5 * charge * charge * ap[c];
            const double aa1 = dth * (ap[1] * u1 + ap[2] * u2);
            const double b1 = dth * (ap[4] * u1 + ap[5] * u2);
            const double gam = sqrt(gam2);
            const double dgam = (aa1 * gam - b1) / gam2;
            const double gam_inv = (gam - dgam) / gam2;
#pragma unroll
            for (int c = 3; c <= 5; ++c) ap[c] = ap[c] * gam_inv;
            const double f1 = ap[1] - ap[4], f2 = ap[2] - ap[5], f3 = ap[3];
            wghp = wgh * gam_inv;
            // lpf_env_momenta, curr_ndim = 2
            const double efp1 = alp * f1, efp2 = alp * f2, efp3 = alp * f3;
            const double vp1 = u1 + efp1, vp2 = u2 + efp2;
            const double bb1 = efp3;
            const double b2 = 1. + bb1 * bb1;
            double vph1 = vp1 + vp2 * bb1;
            double vph2 = vp2 - vp1 * bb1;
            vph1 = vph1 / b2;
            vph2 = vph2 / b2;
            const double pn1 = 2. * vph1 - u1, pn2 = 2. * vph2 - u2;
            a.px[n] = pn1;
            a.py[n] = pn2;
            if (!(pn1 == pn1 && pn2 == pn2)) raise_err(a.err, AGPU_EBIT_NONFINITE);
          } else {
            double ap[11] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int k1 = 0; k1 <= 2; ++k1) {
#pragma unroll
              for (int j1 = 0; j1 <= 2; ++j1) {
                const double dvol = ay1[j1] * az1[k1];
                const int o = FX * (lj + j1 + FY * (lk + k1));
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) ap[10] = ap[10] + ax1[i1] * dvol * av[o + li + i1];
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) {
                  const double dvol1 = dvol * axh1[i1];
                  ap[1] = ap[1] + dvol1 * ef[o + hi + i1];
                  ap[7] = ap[7] + dvol1 * av[FV + o + hi + i1];
                }
              }
#pragma unroll
              for (int j1 = 0; j1 <= 2; ++j1) {
                const double dvol = ayh1[j1] * az1[k1];
                const int o = FX * (hj + j1 + FY * (lk + k1));
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) {
                  const double dvol1 = dvol * ax1[i1];
                  ap[2] = ap[2] + dvol1 * ef[FV + o + li + i1];
                  ap[8] = ap[8] + dvol1 * av[2 * FV + o + li + i1];
                }
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) ap[6] = ap[6] + axh1[i1] * dvol * ef[5 * FV + o + hi + i1];
              }
            }
#pragma unroll
            for (int k1 = 0; k1 <= 2; ++k1) {
#pragma unroll
              for (int j1 = 0; j1 <= 2; ++j1) {
                const double dvol = ayh1[j1] * azh1[k1];
                const int o = FX * (hj + j1 + FY * (hk + k1));
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) ap[4] = ap[4] + ax1[i1] * dvol * ef[3 * FV + o + li + i1];
              }
#pragma unroll
              for (int j1 = 0; j1 <= 2; ++j1) {
                const double dvol = ay1[j1] * azh1[k1];
                const int o = FX * (lj + j1 + FY * (hk + k1));
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) ap[5] = ap[5] + axh1[i1] * dvol * ef[4 * FV + o + hi + i1];
#pragma unroll
                for (int i1 = 0; i1 <= 2; ++i1) {
                  const double dvol1 = dvol * ax1[i1];
                  ap[3] = ap[3] + dvol1 * ef[2 * FV + o + li + i1];
                  ap[9] = ap[9] + dvol1 * av[3 * FV + o + li + i1];
                }
              }
            }
            const double pp[3] = {a.px[n], a.py[n], a.pz[n]};
            const double gam2 = 1. + pp[0] * pp[0] + pp[1] * pp[1] + pp[2] * pp[2] + ap[10];
#pragma unroll
            for (int c = 1; c <= 6; ++c) ap[c] = charge * ap[c];
#pragma unroll
            for (int c = 7; c <= 9; ++c) ap[c] = 0.5 * charge * charge * ap[c];
            const double aa1 = dth * (ap[1] * pp[0] + ap[2] * pp[1] + ap[3] * pp[2]);
            const double b1 = dth * (ap[7] * pp[0] + ap[8] * pp[1] + ap[9] * pp[2]);
            const double gam = sqrt(gam2);
            const double dgam = (aa1 * gam - b1) / gam2;
            const double gam_inv = (gam - dgam) / gam2;
#pragma unroll
            for (int c = 4; c <= 9; ++c) ap[c] = ap[c] * gam_inv;
            double fp[6];
#pragma unroll
            for (int c = 0; c < 3; ++c) fp[c] = ap[c + 1] - ap[c + 7];
#pragma unroll
            for (int c = 3; c < 6; ++c) fp[c] = ap[c + 1];
            wghp = wgh * gam_inv;
            // lpf_env_momenta, curr_ndim = 3
            double efp[6], vp[3], bb[3], vph[3];
#pragma unroll
            for (int c = 0; c < 6; ++c) efp[c] = alp * fp[c];
#pragma unroll
            for (int c = 0; c < 3; ++c) vp[c] = efp[c] + pp[c];
#pragma unroll
            for (int c = 0; c < 3; ++c) bb[c] = efp[3 + c];
            const double b2 = 1. + (bb[0] * bb[0] + bb[1] * bb[1] + bb[2] * bb[2]);
            const double bv = bb[0] * vp[0] + bb[1] * vp[1] + bb[2] * vp[2];
            vph[0] = vp[0] + vp[1] * bb[2] - vp[2] * bb[1] + bb[0] * bv;
            vph[1] = vp[1] + vp[2] * bb[0] - vp[0] * bb[2] + bb[1] * bv;
            vph[2] = vp[2] + vp[0] * bb[1] - vp[1] * bb[0] + bb[2] * bv;
#pragma unroll
            for (int c = 0; c < 3; ++c) vph[c] = vph[c] / b2;
            double pn[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) pn[c] = 2. * vph[c] - pp[c];
            a.px[n] = pn[0];
            a.py[n] = pn[1];
            a.pz[n] = pn[2];
            if (!(pn[0] == pn[0] && pn[1] == pn[1] && pn[2] == pn[2])) raise_err(a.err, AGPU_EBIT_NONFINITE);
          }
          node_d(xl, s);
          dep[e] = s;
          node_d(yl, s);
          dep[S + e] = s;
          if (NDIM == 3) {
            node_d(zl, s);
            dep[2 * S + e] = s;
          }
          dep[NDIM * S + e] = wghp;
          const int rank = atomicAdd(&cnt[fx], 1);
          if (rank < RMAX) {
            idx[rank * 32 + fx] = (unsigned char)e;
          } else {
            // beyond the node's list: its nodes now, one particle per lane
            density_full<NDIM, S>(g, a.den + goff(g, i0t + fx, j0t + wy, (NDIM == 3) ? k0t + wz : 1), dep + e);
          }
        }
      }
    }
    __syncwarp();
    // node per lane: moments of w over 1, s, s^2 along each axis, then the
    // shapes' slots (agpu_tile64.cuh), one atomic per window row and node
    const int n = min(cnt[lane], RMAX);
    if (__any_sync(0xffffffffu, n > 0)) {
      constexpr int NM = (NDIM == 3) ? 3 : 1;
      double m[NM][3][3];  // [z][y][x]
#pragma unroll
      for (int q = 0; q < NM * 9; ++q) m[q / 9][(q / 3) % 3][q % 3] = 0.;
#pragma unroll 1
      for (int k = 0; k < n; ++k) {
        const double* e = dep + idx[k * 32 + lane];
        const double sx = e[0], sy = e[S], sz = (NDIM == 3) ? e[2 * S] : 0.;
        const double qx = sx * sx;
        double wz_ = e[NDIM * S];
#pragma unroll
        for (int c = 0; c < NM; ++c) {
          double wyz = wz_;
#pragma unroll
          for (int r = 0; r < 3; ++r) {
            m[c][r][0] = m[c][r][0] + wyz;
            m[c][r][1] = fma(wyz, sx, m[c][r][1]);
            m[c][r][2] = fma(wyz, qx, m[c][r][2]);
            if (r < 2) wyz = wyz * sy;
          }
          if (c < NM - 1) wz_ = wz_ * sz;
        }
      }
#pragma unroll
      for (int c = 0; c < NM; ++c) {
#pragma unroll
        for (int r = 0; r < 3; ++r) slots3(m[c][r][0], m[c][r][1], m[c][r][2]);
#pragma unroll
        for (int q = 0; q < 3; ++q) slots3(m[c][0][q], m[c][1][q], m[c][2][q]);
      }
      if (NDIM == 3) {
#pragma unroll
        for (int q = 0; q < 9; ++q) slots3(m[0][q / 3][q % 3], m[NM / 2][q / 3][q % 3], m[NM - 1][q / 3][q % 3]);
      }
      const long long sy = g.n1p, sz = (long long)g.n1p * g.n2p;
      double* d = a.den + goff(g, i0t + lane, j0t + wy, (NDIM == 3) ? k0t + wz : 1);
#pragma unroll
      for (int c = 0; c < NM; ++c)
#pragma unroll
        for (int r = 0; r < 3; ++r)
          flush_row<true>(d + (r - 1) * sy + ((NDIM == 3) ? (c - 1) * sz : 0), lane, m[c][r][0], m[c][r][1], m[c][r][2]);
    }
    __syncwarp();
  }
}

// A CTA of NZT tiles, or one of the `extra` CTAs for the dense rows' items.
template <int NDIM>
__global__ void __launch_bounds__(CAcc<NDIM>::NT, (NDIM == 3) ? 1 : 2) k_env_acc_tile(EnvTileArgs a) {
  using C = CAcc<NDIM>;
  using T = typename C::T;
  const int warp = threadIdx.x >> 5, b = blockIdx.x, plane = a.t.ntx * a.t.nty;
  const int cap = a.extra ? (int)a.rows.n[3] : 0x7fffffff;
  if (b < (int)gridDim.x - a.extra) {
    const int zp = b / plane, tile = zp * C::NZT * plane + b % plane + warp / T::NROW * plane;
    int c0 = 0, end = 0;
    if (tile < a.t.ntiles) {  // the last CTA along z may have fewer tiles
      const int* start = a.tstart + (tile * T::NROW + warp % T::NROW) * T::NQ;
      c0 = start[0];
      end = start[T::NQ];
    }
    if (!__syncthreads_or(c0 < end)) return;
    acc_rows<NDIM>(a, b % a.t.ntx, (b / a.t.ntx) % a.t.nty, zp, warp, c0, end - c0 > cap ? c0 + cap : end);
    return;
  }
  if (a.rows.n[0] == 0u) return;
  for (int q, c0, end; (q = next_item(a.rows)) >= 0;) {
    const int row = a.rows.item[2 * q], t = row / T::NROW, tz = t / plane;
    item_records(a.rows, a.tstart, T::NQ, q, warp, C::NROW, c0, end);
    acc_rows<NDIM>(a, t % a.t.ntx, (t / a.t.ntx) % a.t.nty, tz / C::NZT, tz % C::NZT * T::NROW + row % T::NROW, c0, end);
  }
  items_done(a.rows, a.extra, false);  // the position step takes the same items
}

template <int NDIM>
void acc_t(const EnvTileArgs& a, cudaStream_t st) {
  using C = CAcc<NDIM>;
  auto k = k_env_acc_tile<NDIM>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::BYTES);
  const int nzp = (NDIM == 3) ? (a.t.ntz + C::NZT - 1) / C::NZT : 1;
  k<<<a.t.ntx * a.t.nty * nzp + a.extra, C::NT, C::BYTES, st>>>(a);
}
template <int NDIM>
void pos_t(const EnvTileArgs& a, cudaStream_t st) {
  using C = C64<NDIM, PushEnv<NDIM>::NF, PushEnv<NDIM>::LO>;
  auto k = k_env_pos_tile<NDIM>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::BYTES);
  k<<<a.t.ntiles + a.extra, C::NT, C::BYTES, st>>>(a);
}

}  // namespace

void env_acc_tile(const EnvTileArgs& a, cudaStream_t st) {
  if (a.t.ntiles <= 0) return;
  if (a.g.ndim == 3) acc_t<3>(a, st);
  else acc_t<2>(a, st);
}
void env_pos_tile(const EnvTileArgs& a, cudaStream_t st) {
  if (a.t.ntiles <= 0) return;
  if (a.g.ndim == 3) pos_t<3>(a, st);
  else pos_t<2>(a, st);
}

}  // namespace agpu
