// agpu_yee.cuh — field kernels templated on the storage type: boundary
// extrapolation (A1), current fold (A13) and the leapfrog Yee update with
// Mur-type open boundaries (A14).  Included by agpu_fp64.cu (T = double,
// compiled without FMA contraction so the statement order of the reference
// is kept bit for bit) and agpu_fp32.cu (T = float).
#pragma once
#include <type_traits>

#include "agpu_common.cuh"
#include "agpu_bin.cuh"
#include "agpu_kernels.h"

namespace agpu {

// Every kernel body is a device function over "its" blocks bid_ of nb_, so
// that the same body runs as a single-instance kernel (bid_ = blockIdx.x) or
// inside a kernel that serves many instances at once (one row of blocks per
// instance).
#define GRID_STRIDE(t, total) \
  for (long long t = bid_ * (long long)blockDim.x + threadIdx.x; t < (total); t += nb_ * (long long)blockDim.x)

// ---- A1: field_xyzbd (src/parallel/mpi_field_interface.f90:53-198) --------
// One ghost layer by linear extrapolation along x, then y over the widened x
// range, then z over the widened x and y ranges.  A ghost of a later axis is
// formed from the earlier axes' extrapolations of the interior (the same
// operations on the same values), so one sweep reads interior nodes only
// and writes every ghost: one launch instead of a dependent one per axis
// (4 us each on the small grids, where a launch costs more than its work).
template <typename T>
__device__ __forceinline__ T bd_x(const T* f, const Geo& g, int i, int j, int k) {
  if (i < g.ix1) return (T)2. * f[goff(g, g.ix1, j, k)] - f[goff(g, g.ix1 + 1, j, k)];
  if (i > g.ix2) return (T)2. * f[goff(g, g.ix2, j, k)] - f[goff(g, g.ix2 - 1, j, k)];
  return f[goff(g, i, j, k)];
}
template <typename T>
__device__ __forceinline__ T bd_y(const T* f, const Geo& g, int i, int j, int k) {
  if (j < g.jy1) return (T)2. * bd_x(f, g, i, g.jy1, k) - bd_x(f, g, i, g.jy1 + 1, k);
  if (j > g.jy2) return (T)2. * bd_x(f, g, i, g.jy2, k) - bd_x(f, g, i, g.jy2 - 1, k);
  return bd_x(f, g, i, j, k);
}
template <typename T>
__device__ __forceinline__ T bd_z(const T* f, const Geo& g, int i, int j, int k) {
  if (k < g.kz1) return (T)2. * bd_y(f, g, i, j, g.kz1) - bd_y(f, g, i, j, g.kz1 + 1);
  return (T)2. * bd_y(f, g, i, j, g.kz2) - bd_y(f, g, i, j, g.kz2 - 1);
}
// ghost nodes of one component: two x faces, two y faces, two z faces (3D)
AGPU_HD int bd_nodes(const Geo& g) {
  const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  return 2 * (ny * nz + (nx + 2) * nz + (g.ndim == 3 ? (nx + 2) * (ny + 2) : 0));
}
// ghost node r of component f
template <typename T>
__device__ __forceinline__ void field_bd_node(T* f, const Geo& g, int r) {
  const int nxe = g.ix2 - g.ix1 + 3, nye = g.jy2 - g.jy1 + 3, ny = nye - 2, nz = g.kz2 - g.kz1 + 1;
  const int fx = 2 * ny * nz, fy = 2 * nxe * nz;
  {
    int i, j, k;
    T v;
    if (r < fx) {
      const int hi = r >= fx / 2;
      r -= hi * (fx / 2);
      i = hi ? g.ix2 + 1 : g.ix1 - 1;
      j = g.jy1 + r % ny;
      k = g.kz1 + r / ny;
      v = bd_x(f, g, i, j, k);
    } else if (r < fx + fy) {
      r -= fx;
      const int hi = r >= fy / 2;
      r -= hi * (fy / 2);
      i = g.ix1 - 1 + r % nxe;
      j = hi ? g.jy2 + 1 : g.jy1 - 1;
      k = g.kz1 + r / nxe;
      v = bd_y(f, g, i, j, k);
    } else {
      r -= fx + fy;
      const int hi = r >= nxe * nye;
      r -= hi * (nxe * nye);
      i = g.ix1 - 1 + r % nxe;
      j = g.jy1 - 1 + r / nxe;
      k = hi ? g.kz2 + 1 : g.kz1 - 1;
      v = bd_z(f, g, i, j, k);
    }
    f[goff(g, i, j, k)] = v;
  }
}
// one thread per node, one grid row per component
template <typename T>
__global__ void k_field_bd(T* ebf, Geo g) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < bd_nodes(g)) field_bd_node(ebf + g.ncell * blockIdx.y, g, r);
}
template <typename T>
void field_bd_t(T* ebf, const Geo& g, cudaStream_t st) {
  k_field_bd<T><<<dim3((bd_nodes(g) + 255) / 256, g.nf), 256, 0, st>>>(ebf, g);
}

// What a step clears before its push, in one launch with the field
// extrapolation: the currents (both parts) and the next histogram
// (hist_reset).  On small grids each of the four launches it replaces cost
// about 3 us.  Block ranges: ghost nodes, histogram, currents (nzero blocks).
template <typename T>
__global__ void k_step_pre(T* ebf, Geo g, T* j0, T* j1, HistReset h, int bbd, int bhist, int nzero) {
  int b = blockIdx.x;
  if (b < bbd * g.nf) {
    const int c = b / bbd, r = (b - c * bbd) * blockDim.x + threadIdx.x;
    if (r < bd_nodes(g)) field_bd_node(ebf + g.ncell * c, g, r);
    return;
  }
  b -= bbd * g.nf;
  if (b < bhist) {
    hist_reset_bin(h, b * blockDim.x + threadIdx.x);
    return;
  }
  b -= bhist;
  const long long n = g.ncell * g.nc;
  for (long long q = b * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)nzero * blockDim.x) {
    j0[q] = (T)0;
    if (j1) j1[q] = (T)0;
  }
}
template <typename T>
void step_pre_t(T* ebf, T* j0, T* j1, const Geo& g, const HistReset& h, cudaStream_t st, int sms) {
  const int bbd = (bd_nodes(g) + 255) / 256, bhist = (h.nkeys + 256) / 256;
  const int nzero = grid_for(g.ncell * g.nc, 256, sms, 16);
  k_step_pre<T><<<bbd * g.nf + bhist + nzero, 256, 0, st>>>(ebf, g, j0, j1, h, bbd, bhist, nzero);
}

// ---- A13: jc_xyzbd (src/parallel/mpi_curr_interface.f90:551-643) ----------
// The ghost currents added to the faces' nodes and cleared, x, then y, then
// z.  A node's ghosts along one axis lie on interior nodes of the others, so
// no fold touches what another reads: one sweep over the boundary nodes adds
// them in that order, for both parts of a two-float current.
// boundary nodes of one component: the x faces, then what the y and z faces
// have beyond them
AGPU_HD int fold_nodes(const Geo& g) {
  const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  return 2 * (ny * nz + (nx - 2) * nz + (g.ndim == 3 ? (nx - 2) * (ny - 2) : 0));
}
// boundary node r of component q (j0's components, then j1's)
template <typename T>
__device__ __forceinline__ void jfold_node(T* j0, T* j1, const Geo& g, int q, int r) {
  const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  const int fx = 2 * ny * nz, fy = 2 * (nx - 2) * nz;
  const long long sy = g.n1p, sz = (long long)g.n1p * g.n2p;
  {
    int i, j, k;
    if (r < fx) {
      const int hi = r >= fx / 2;
      r -= hi * (fx / 2);
      i = hi ? g.ix2 : g.ix1;
      j = g.jy1 + r % ny;
      k = g.kz1 + r / ny;
    } else if (r < fx + fy) {
      r -= fx;
      const int hi = r >= fy / 2;
      r -= hi * (fy / 2);
      i = g.ix1 + 1 + r % (nx - 2);
      j = hi ? g.jy2 : g.jy1;
      k = g.kz1 + r / (nx - 2);
    } else {
      r -= fx + fy;
      const int m = (nx - 2) * (ny - 2), hi = r >= m;
      r -= hi * m;
      i = g.ix1 + 1 + r % (nx - 2);
      j = g.jy1 + 1 + r / (nx - 2);
      k = hi ? g.kz2 : g.kz1;
    }
    T* c = (q < g.nc ? j0 + g.ncell * q : j1 + g.ncell * (q - g.nc)) + goff(g, i, j, k);
    // All loads before the first store: a load behind a store to a line near
    // it waits for that store (a 24-run 2D scan of 10 steps 11.7 ms with the
    // loads in between, 11.2 so).
    const bool xl = i == g.ix1, xh = i == g.ix2, yl = j == g.jy1, yh = j == g.jy2;
    const bool zl = g.ndim == 3 && k == g.kz1, zh = g.ndim == 3 && k == g.kz2;
    const T o = (T)0;
    T v = *c;
    const T xl1 = xl ? c[-1] : o, xh1 = xh ? c[1] : o, xh2 = xh ? c[2] : o;
    const T yl1 = yl ? c[-sy] : o, yl2 = yl ? c[-2 * sy] : o, yh1 = yh ? c[sy] : o, yh2 = yh ? c[2 * sy] : o;
    const T zl1 = zl ? c[-sz] : o, zh1 = zh ? c[sz] : o, zh2 = zh ? c[2 * sz] : o;
    // the nearer, then the farther ghost node along one direction
    if (xl) {
      v = v + xl1;
      c[-1] = o;
    }
    if (xh) {
      v = v + xh1 + xh2;
      c[1] = c[2] = o;
    }
    if (yl) {
      v = v + yl1 + yl2;
      c[-sy] = c[-2 * sy] = o;
    }
    if (yh) {
      v = v + yh1 + yh2;
      c[sy] = c[2 * sy] = o;
    }
    if (zl) {
      v = v + zl1;
      c[-sz] = o;
    }
    if (zh) {
      v = v + zh1 + zh2;
      c[sz] = c[2 * sz] = o;
    }
    *c = v;
  }
}
template <typename T>
__global__ void k_jfold(T* j0, T* j1, Geo g) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < fold_nodes(g)) jfold_node(j0, j1, g, blockIdx.y, r);
}
// One axis of the fold: both of its faces, all interior nodes of the other
// two axes.  Bound by memory latency; the loads come before the stores: with
// the farther ghost loaded behind a store the three launches took 43 us on
// 384x96x96 cells (both parts of a two-float current, in L2; 65 from DRAM),
// against 19 (24).
template <typename T, int AX>
__global__ void k_jfold_axis(T* j0, T* j1, Geo g) {
  const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  const int m = (AX == 0) ? ny : nx, n = m * ((AX == 2) ? ny : nz);
  int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= 2 * n) return;
  const int hi = r >= n;
  r -= hi * n;
  const int u = r % m, v = r / m;
  const int i = (AX == 0) ? (hi ? g.ix2 : g.ix1) : g.ix1 + u;
  const int j = (AX == 1) ? (hi ? g.jy2 : g.jy1) : g.jy1 + (AX == 0 ? u : v);
  const int k = (AX == 2) ? (hi ? g.kz2 : g.kz1) : g.kz1 + v;
  const int q = blockIdx.y;
  T* c = (q < g.nc ? j0 + g.ncell * q : j1 + g.ncell * (q - g.nc)) + goff(g, i, j, k);
  const long long s = (AX == 0) ? 1 : (AX == 1) ? g.n1p : (long long)g.n1p * g.n2p, d = hi ? s : -s;
  const bool two = hi || AX == 1;
  const T a = c[0], b = c[d], e = two ? c[2 * d] : (T)0;
  c[0] = two ? a + b + e : a + b;
  c[d] = (T)0;
  if (two) c[2 * d] = (T)0;
}
// j1: the compensation part of a two-float current, or null.  2D in one sweep
// (4 us against 8: launches are what counts), 3D in one launch per axis (on
// 384x96x96 cells the 19 us above, 24 from DRAM; the one sweep 23 and 36).
template <typename T>
void jfold_t(T* j0, T* j1, const Geo& g, cudaStream_t st) {
  const int nq = g.nc * (j1 ? 2 : 1);
  if (g.ndim == 2) {
    k_jfold<T><<<dim3((fold_nodes(g) + 255) / 256, nq), 256, 0, st>>>(j0, j1, g);
    return;
  }
  const int nx = g.ix2 - g.ix1 + 1, ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  auto blocks = [&](int n) { return dim3((2 * n + 255) / 256, nq); };
  k_jfold_axis<T, 0><<<blocks(ny * nz), 256, 0, st>>>(j0, j1, g);
  k_jfold_axis<T, 1><<<blocks(nx * nz), 256, 0, st>>>(j0, j1, g);
  k_jfold_axis<T, 2><<<blocks(nx * ny), 256, 0, st>>>(j0, j1, g);
}

// ---- A14: Yee (advance_lpf_fields, curr_and_fields_util.f90:176-260) ------

// ef_bds (src/fields/grid_fields.f90:1204-1354): right-face Mur boundary of E.
template <typename T>
__device__ __forceinline__ void d_ef_bds(T* ebf, Geo g, YeeC c, double dtl, long long bid_, long long nb_) {
  int ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1, nx = g.ix2 - g.ix1 + 1;
  long long nfx = (long long)ny * nz, nfy = (long long)nx * nz, nfz = (g.ndim == 3) ? (long long)nx * ny : 0;
  int nf = g.nf;
  T* E1 = ebf;
  T* E2 = ebf + g.ncell;
  T* E3 = ebf + 2 * g.ncell;
  T* B1 = ebf + 3 * g.ncell;
  T* B2 = ebf + 4 * g.ncell;
  T* Bn = ebf + (nf - 1) * g.ncell;
  const T one = (T)1., two = (T)2.;
  GRID_STRIDE(t, nfx + nfy + nfz) {
    if (t < nfx) {
      int j = g.jy1 + (int)(t % ny), k = g.kz1 + (int)(t / ny);
      T aphx = (T)(1.0 * c.dx_inv * dtl);
      long long o = goff(g, g.ix2, j, k);
      E2[o + 1] = (two * Bn[o] - (one - aphx) * E2[o]) / (one + aphx);
      if (nf > 3) E3[o + 1] = -(two * B2[o] + (one - aphx) * E3[o]) / (one + aphx);
    } else if (t < nfx + nfy) {
      long long u = t - nfx;
      int i = g.ix1 + (int)(u % nx), k = g.kz1 + (int)(u / nx);
      T aphy = (T)(c.ty4 * c.dy_inv * dtl);  // loc_yg(ny, 4) dy_inv dt
      long long o = goff(g, i, g.jy2, k), o1 = o + g.n1p;
      E1[o1] = -(two * Bn[o] + (one - aphy) * E1[o]) / (one + aphy);
      if (nf > 3) E3[o1] = (two * B1[o] - (one - aphy) * E3[o]) / (one + aphy);
    } else {
      long long u = t - nfx - nfy;
      int i = g.ix1 + (int)(u % nx), j = g.jy1 + (int)(u / nx);
      T aphz = (T)(c.tz4 * c.dz_inv * dtl);  // loc_zg(nz, 4) dz_inv dt
      long long o = goff(g, i, j, g.kz2), o1 = o + (long long)g.n1p * g.n2p;
      E1[o1] = (two * B2[o] - (one - aphz) * E1[o]) / (one + aphz);
      E2[o1] = -(two * B1[o] + (one - aphz) * E2[o]) / (one + aphz);
    }
  }
}
template <typename T>
__global__ void k_ef_bds(T* ebf, Geo g, YeeC c, double dtl) {
  d_ef_bds<T>(ebf, g, c, dtl, blockIdx.x, gridDim.x);
}
// bf_bds (src/fields/grid_fields.f90:1069-1202): left-face Mur boundary of B.
template <typename T>
__device__ __forceinline__ void d_bf_bds(T* ebf, Geo g, YeeC c, double dtl, long long bid_, long long nb_) {
  int ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1, nx = g.ix2 - g.ix1 + 1;
  long long nfx = (long long)ny * nz, nfy = (long long)nx * nz, nfz = (g.ndim == 3) ? (long long)nx * ny : 0;
  int nf = g.nf;
  T* E1 = ebf;
  T* E2 = ebf + g.ncell;
  T* E3 = ebf + 2 * g.ncell;
  T* B1 = ebf + 3 * g.ncell;
  T* B2 = ebf + 4 * g.ncell;
  T* Bn = ebf + (nf - 1) * g.ncell;
  const T one = (T)1., two = (T)2.;
  GRID_STRIDE(t, nfx + nfy + nfz) {
    if (t < nfx) {
      int j = g.jy1 + (int)(t % ny), k = g.kz1 + (int)(t / ny);
      T aphx = (T)(1.0 * c.dx_inv * dtl);
      long long o = goff(g, g.ix1, j, k);
      Bn[o - 1] = -(two * E2[o] + (one - aphx) * Bn[o]) / (one + aphx);
      if (nf > 3) B2[o - 1] = (two * E3[o] - (one - aphx) * B2[o]) / (one + aphx);
    } else if (t < nfx + nfy) {
      long long u = t - nfx;
      int i = g.ix1 + (int)(u % nx), k = g.kz1 + (int)(u / nx);
      T aphy = (T)(c.by3 * c.dy_inv * dtl);  // loc_yg(1, 3) dy_inv dt
      long long o = goff(g, i, g.jy1, k), o1 = o - g.n1p;
      T v = two * E1[o] - (one - aphy) * Bn[o];
      Bn[o1] = v / (one + aphy);
      if (nf > 3) {
        T w = -two * E3[o] - (one - aphy) * B1[o];
        B1[o1] = w / (one + aphy);
      }
    } else {
      long long u = t - nfx - nfy;
      int i = g.ix1 + (int)(u % nx), j = g.jy1 + (int)(u / nx);
      T aphz = (T)(c.bz3 * c.dz_inv * dtl);  // loc_zg(1, 3) dz_inv dt
      long long o = goff(g, i, j, g.kz1), o1 = o - (long long)g.n1p * g.n2p;
      T v = two * E2[o] - (one - aphz) * B1[o];
      B1[o1] = v / (one + aphz);
      T w = -two * E1[o] - (one - aphz) * B2[o];
      B2[o1] = w / (one + aphz);
    }
  }
}
template <typename T>
__global__ void k_bf_bds(T* ebf, Geo g, YeeC c, double dtl) {
  d_bf_bds<T>(ebf, g, c, dtl, blockIdx.x, gridDim.x);
}

// rote (grid_fields.f90:1405-1478): B -= dtf curl E at node o = (i, j, k).
// BDS: the right-face Mur ghosts of E (ef_bds with dtl), which this node's
// differences read, depend on this node's fields alone, so the node forms and
// stores them itself and no boundary sweep runs before this one.  Only with
// the compact x difference (SE2 false: se2 = 0), whose stencil has no node
// further out.
template <typename T, int NDIM, bool BDS, bool SE2>
__device__ __forceinline__ void rote_node(T* ebf, const Geo& g, const YeeC& c, long long o, int i, int j, int k, T aph1,
                                          T aph2, T sdhy, T sdhz, double dtl) {
  const long long sy = g.n1p, sz = (long long)g.n1p * g.n2p;
  T* E1 = ebf;
  T* E2 = ebf + g.ncell;
  T* E3 = ebf + 2 * g.ncell;
  T* Bx = ebf + 3 * g.ncell;
  T* By = ebf + 4 * g.ncell;
  T* Bz = ebf + (NDIM == 3 ? 5 : 2) * g.ncell;
  // the sweep writes no E that another node reads: read-only loads
  const T e1 = __ldg(E1 + o), e2 = __ldg(E2 + o), e3 = (NDIM == 3) ? __ldg(E3 + o) : (T)0;
  const T bz = Bz[o], bx = (NDIM == 3) ? Bx[o] : (T)0, by = (NDIM == 3) ? By[o] : (T)0;
  T e2x, e3x = (T)0, e1y, e3y = (T)0, e1z = (T)0, e2z = (T)0;  // E one node up along x, y, z
  const T one = (T)1., two = (T)2.;
  if (BDS && i == g.ix2) {
    const T aphx = (T)(1.0 * c.dx_inv * dtl);
    E2[o + 1] = e2x = (two * bz - (one - aphx) * e2) / (one + aphx);
    if (NDIM == 3) E3[o + 1] = e3x = -(two * by + (one - aphx) * e3) / (one + aphx);
  } else {
    e2x = __ldg(E2 + o + 1);
    if (NDIM == 3) e3x = __ldg(E3 + o + 1);
  }
  if (BDS && j == g.jy2) {
    const T aphy = (T)(c.ty4 * c.dy_inv * dtl);  // loc_yg(ny, 4) dy_inv dt
    E1[o + sy] = e1y = -(two * bz + (one - aphy) * e1) / (one + aphy);
    if (NDIM == 3) E3[o + sy] = e3y = (two * bx - (one - aphy) * e3) / (one + aphy);
  } else {
    e1y = __ldg(E1 + o + sy);
    if (NDIM == 3) e3y = __ldg(E3 + o + sy);
  }
  if (NDIM == 3) {
    if (BDS && k == g.kz2) {
      const T aphz = (T)(c.tz4 * c.dz_inv * dtl);  // loc_zg(nz, 4) dz_inv dt
      E1[o + sz] = e1z = (two * by - (one - aphz) * e1) / (one + aphz);
      E2[o + sz] = e2z = -(two * bx + (one - aphz) * e2) / (one + aphz);
    } else {
      e1z = __ldg(E1 + o + sz);
      e2z = __ldg(E2 + o + sz);
    }
  }
  const T nz = bz - aph1 * (e2x - e2) + sdhy * (e1y - e1);
  Bz[o] = SE2 ? nz - aph2 * (E2[o + 2] - E2[o - 1]) : nz;
  if (NDIM == 3) {
    Bx[o] = bx - sdhy * (e3y - e3) + sdhz * (e2z - e2);
    const T ny = by + aph1 * (e3x - e3) - sdhz * (e1z - e1);
    By[o] = SE2 ? ny + aph2 * (E3[o + 2] - E3[o - 1]) : ny;
  }
}

// rotb (grid_fields.f90:1480-1552) + E -= ompe * (djc * J)
// (curr_and_fields_util.f90:111-115, 227-231) at node o.  jlo (optional)
// holds the compensation term of a two-float current.  BDS: the left-face
// Mur ghosts of B (bf_bds with dt) formed by the nodes that read them, as in
// rote_node.
template <typename T, int NDIM, bool BDS, bool SE2>
__device__ __forceinline__ void rotb_node(T* ebf, const T* jc, const T* jlo, const Geo& g, const YeeC& c, long long o,
                                          int i, int j, int k, T aph1, T aph2, T sdy, T sdz, double dtl) {
  const long long sy = g.n1p, sz = (long long)g.n1p * g.n2p;
  T* E1 = ebf;
  T* E2 = ebf + g.ncell;
  T* E3 = ebf + 2 * g.ncell;
  T* Bx = ebf + 3 * g.ncell;
  T* By = ebf + 4 * g.ncell;
  T* Bz = ebf + (NDIM == 3 ? 5 : 2) * g.ncell;
  const T ompe = (T)c.ompe, djc1 = (T)c.djc1, djc2 = (T)c.djc2, djc3 = (T)c.djc3;
  T j1 = __ldg(jc + o), j2 = __ldg(jc + o + g.ncell), j3 = (NDIM == 3) ? __ldg(jc + o + 2 * g.ncell) : (T)0;
  if (jlo) {
    j1 = j1 + __ldg(jlo + o);
    j2 = j2 + __ldg(jlo + o + g.ncell);
    if (NDIM == 3) j3 = j3 + __ldg(jlo + o + 2 * g.ncell);
  }
  const T e1 = E1[o], e2 = E2[o], e3 = (NDIM == 3) ? E3[o] : (T)0;
  // the sweep writes no B that another node reads
  const T bz = __ldg(Bz + o), bx = (NDIM == 3) ? __ldg(Bx + o) : (T)0, by = (NDIM == 3) ? __ldg(By + o) : (T)0;
  T bzx, byx = (T)0, bzy, bxy = (T)0, bxz = (T)0, byz = (T)0;  // B one node down along x, y, z
  const T one = (T)1., two = (T)2.;
  if (BDS && i == g.ix1) {
    const T aphx = (T)(1.0 * c.dx_inv * dtl);
    Bz[o - 1] = bzx = -(two * e2 + (one - aphx) * bz) / (one + aphx);
    if (NDIM == 3) By[o - 1] = byx = (two * e3 - (one - aphx) * by) / (one + aphx);
  } else {
    bzx = __ldg(Bz + o - 1);
    if (NDIM == 3) byx = __ldg(By + o - 1);
  }
  if (BDS && j == g.jy1) {
    const T aphy = (T)(c.by3 * c.dy_inv * dtl);  // loc_yg(1, 3) dy_inv dt
    const T v = two * e1 - (one - aphy) * bz;
    Bz[o - sy] = bzy = v / (one + aphy);
    if (NDIM == 3) {
      const T w = -two * e3 - (one - aphy) * bx;
      Bx[o - sy] = bxy = w / (one + aphy);
    }
  } else {
    bzy = __ldg(Bz + o - sy);
    if (NDIM == 3) bxy = __ldg(Bx + o - sy);
  }
  if (NDIM == 3) {
    if (BDS && k == g.kz1) {
      const T aphz = (T)(c.bz3 * c.dz_inv * dtl);  // loc_zg(1, 3) dz_inv dt
      const T v = two * e2 - (one - aphz) * bx;
      Bx[o - sz] = bxz = v / (one + aphz);
      const T w = -two * e1 - (one - aphz) * by;
      By[o - sz] = byz = w / (one + aphz);
    } else {
      bxz = __ldg(Bx + o - sz);
      byz = __ldg(By + o - sz);
    }
  }
  T ex = e1 + sdy * (bz - bzy);
  T ey = e2 - aph1 * (bz - bzx);
  if (SE2) ey = ey - aph2 * (Bz[o + 1] - Bz[o - 2]);
  T ez = (T)0;
  if (NDIM == 3) {
    ex = ex - sdz * (by - byz);
    ey = ey + sdz * (bx - bxz);
    ez = e3 + aph1 * (by - byx) - sdy * (bx - bxy);
    if (SE2) ez = ez + aph2 * (By[o + 1] - By[o - 2]);
  }
  if (c.my3) {
    // curr_mpi_collect on stretched axes: 2D dery, derhy; 3D dery derz,
    // derhy derz, dery derhz
    const T dery = (T)c.my3[j - 2], derhy = (T)c.my4[j - 2];
    if (NDIM == 2) {
      E1[o] = ex - ompe * (dery * (djc1 * j1));
      E2[o] = ey - ompe * (derhy * (djc2 * j2));
    } else {
      const T derz = (T)c.mz3[k - 2], derhz = (T)c.mz4[k - 2];
      E1[o] = ex - ompe * ((dery * derz) * (djc1 * j1));
      E2[o] = ey - ompe * ((derhy * derz) * (djc2 * j2));
      E3[o] = ez - ompe * ((dery * derhz) * (djc3 * j3));
    }
    return;
  }
  E1[o] = ex - ompe * (djc1 * j1);
  E2[o] = ey - ompe * (djc2 * j2);
  if (NDIM == 3) E3[o] = ez - ompe * (djc3 * j3);
}

// The two sweeps: one thread per node, blocks of 128 x 2 nodes over (i, j)
// and one z plane per grid layer, so the node indices come without 64-bit
// divisions.  Measured on the 1024x256x256 grid: the FP32 phase 2.42 -> 2.06
// ms; marching each thread over several z planes (carrying the z-neighbour
// loads) was slower.
constexpr int YEE_BX = 128, YEE_BY = 2;

template <typename T, int NDIM, bool BDS, bool SE2>
__device__ __forceinline__ void rote_at(T* ebf, const Geo& g, const YeeC& c, double dtf, double dtl, int i, int j, int k) {
  const double aphxd = dtf * c.dx_inv, aphyd = dtf * c.dy_inv, aphzd = dtf * c.dz_inv;
  // loc_yg(jj, 4) * aphy, loc_zg(kk, 4) * aphz (1 on a uniform axis)
  rote_node<T, NDIM, BDS, SE2>(ebf, g, c, goff(g, i, j, k), i, j, k, (T)(aphxd * c.se1), (T)(aphxd * c.se2),
                               (T)((c.my4 ? c.my4[j - 2] : 1.0) * aphyd),
                               (T)((c.mz4 && NDIM == 3 ? c.mz4[k - 2] : 1.0) * aphzd), dtl);
}
template <typename T, int NDIM, bool BDS, bool SE2>
__device__ __forceinline__ void rotb_at(T* ebf, const T* jc, const T* jlo, const Geo& g, const YeeC& c, double dtf,
                                        int i, int j, int k) {
  const double aphxd = dtf * c.dx_inv, aphyd = dtf * c.dy_inv, aphzd = dtf * c.dz_inv;
  // loc_yg(jj, 3) * aphy, aphz * loc_zg(kk, 3) (1 on a uniform axis)
  rotb_node<T, NDIM, BDS, SE2>(ebf, jc, jlo, g, c, goff(g, i, j, k), i, j, k, (T)(aphxd * c.se1), (T)(aphxd * c.se2),
                               (T)((c.my3 ? c.my3[j - 2] : 1.0) * aphyd),
                               (T)(aphzd * (c.mz3 && NDIM == 3 ? c.mz3[k - 2] : 1.0)), dtf);
}
template <typename T, int NDIM, bool BDS, bool SE2>
__global__ void __launch_bounds__(YEE_BX* YEE_BY) k_rote(T* ebf, Geo g, YeeC c, double dtf, double dtl) {
  const int i = g.ix1 + blockIdx.x * YEE_BX + threadIdx.x;
  const int j = g.jy1 + blockIdx.y * YEE_BY + threadIdx.y;
  if (i > g.ix2 || j > g.jy2) return;
  rote_at<T, NDIM, BDS, SE2>(ebf, g, c, dtf, dtl, i, j, (NDIM == 3) ? g.kz1 + (int)blockIdx.z : 1);
}
template <typename T, int NDIM, bool BDS, bool SE2>
__global__ void __launch_bounds__(YEE_BX* YEE_BY) k_rotb_j(T* ebf, const T* jc, const T* jlo, Geo g, YeeC c, double dtf) {
  const int i = g.ix1 + blockIdx.x * YEE_BX + threadIdx.x;
  const int j = g.jy1 + blockIdx.y * YEE_BY + threadIdx.y;
  if (i > g.ix2 || j > g.jy2) return;
  rotb_at<T, NDIM, BDS, SE2>(ebf, jc, jlo, g, c, dtf, i, j, (NDIM == 3) ? g.kz1 + (int)blockIdx.z : 1);
}

// ---- comoving frame: field_xadvect (src/fields/grid_fields.f90:210-324) ----

// x ghosts: f(ix1-1) = f(ix1+1), f(ix2+1) = f(ix2), components ic1..ic2
template <typename T>
__global__ void k_xadv_ghost(T* ebf, Geo g, int ic1, int ic2) {
  const int ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  const long long rows = (long long)ny * nz;
  const long long total = rows * (ic2 - ic1 + 1);
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int ic = ic1 + (int)(t / rows);
    const long long r = t - (long long)(ic - ic1) * rows;
    const int j = g.jy1 + (int)(r % ny), k = g.kz1 + (int)(r / ny);
    T* row = ebf + g.ncell * (ic - 1) + goff(g, 1, j, k) - 1;  // row[i] = f(i)
    row[g.ix1 - 1] = row[g.ix1 + 1];
    row[g.ix2 + 1] = row[g.ix2];
  }
}
// explicit step of one component into the row buffer, then back
template <typename T>
__global__ void k_xadv_explicit(const T* f, double* tmp, Geo g, double aphx_exp) {
  const int i = g.ix1 + blockIdx.x * YEE_BX + threadIdx.x;
  const int j = g.jy1 + blockIdx.y * YEE_BY + threadIdx.y;
  if (i > g.ix2 || j > g.jy2) return;
  const long long o = goff(g, i, j, g.ndim == 3 ? g.kz1 + (int)blockIdx.z : 1);
  tmp[o] = f[o] - aphx_exp * (f[o + 1] - f[o - 1]);
}
template <typename T>
__global__ void k_xadv_copy(T* f, const double* tmp, Geo g) {
  const int i = g.ix1 + blockIdx.x * YEE_BX + threadIdx.x;
  const int j = g.jy1 + blockIdx.y * YEE_BY + threadIdx.y;
  if (i > g.ix2 || j > g.jy2) return;
  const long long o = goff(g, i, j, g.ndim == 3 ? g.kz1 + (int)blockIdx.z : 1);
  f[o] = tmp[o];
}
// implicit step: one thread per row (component ic1..ic2), the Thomas sweeps
// in place in trid_der1's order
template <typename T>
__global__ void k_xadv_implicit(T* ebf, Geo g, int ic1, int ic2, XAdv x) {
  const int ny = g.jy2 - g.jy1 + 1, nz = g.kz2 - g.kz1 + 1;
  const long long rows = (long long)ny * nz;
  const long long total = rows * (ic2 - ic1 + 1);
  const int n = g.ix2 - g.ix1 + 1;
  const double a = x.a, an = 0.0;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const int ic = ic1 + (int)(t / rows);
    const long long r = t - (long long)(ic - ic1) * rows;
    const int j = g.jy1 + (int)(r % ny), k = g.kz1 + (int)(r / ny);
    T* u = ebf + g.ncell * (ic - 1) + goff(g, g.ix1, j, k) - 1;  // u[kk] = f(ix1 + kk - 1), kk = 1..n
    u[1] = u[1] / x.bet[1];
    for (int kk = 2; kk <= n - 1; ++kk) u[kk] = (u[kk] - a * u[kk - 1]) / x.bet[kk];
    u[n] = (u[n] - an * u[n - 1]) / x.bet[n];
    for (int kk = n - 1; kk >= 1; --kk) u[kk] = u[kk] - x.w1[kk + 1] * u[kk + 1];
  }
}
template <typename T>
void xadvect_t(T* ebf, const Geo& g, int ic1, int ic2, int isch, const XAdv& x, cudaStream_t st, int sms) {
  const long long rows = (long long)(g.jy2 - g.jy1 + 1) * (g.kz2 - g.kz1 + 1) * (ic2 - ic1 + 1);
  k_xadv_ghost<T><<<grid_for(rows, 256, sms), 256, 0, st>>>(ebf, g, ic1, ic2);
  if (isch == 0) {
    const dim3 blk(YEE_BX, YEE_BY, 1);
    const dim3 grd((g.ix2 - g.ix1 + YEE_BX) / YEE_BX, (g.jy2 - g.jy1 + YEE_BY) / YEE_BY, g.ndim == 3 ? g.kz2 - g.kz1 + 1 : 1);
    for (int ic = ic1; ic <= ic2; ++ic) {
      k_xadv_explicit<T><<<grd, blk, 0, st>>>(ebf + g.ncell * (ic - 1), x.tmp, g, x.aphx_exp);
      k_xadv_copy<T><<<grd, blk, 0, st>>>(ebf + g.ncell * (ic - 1), x.tmp, g);
    }
  } else {
    k_xadv_implicit<T><<<(int)((rows + 127) / 128), 128, 0, st>>>(ebf, g, ic1, ic2, x);
  }
}

// xa: the comoving frame's advection scratch (c.vbeam > 0), else null;
// hk: a y slab's halo exchange after each boundary sweep, else null
template <typename T>
void yee_t(T* ebf, const T* jc, const T* jlo, const Geo& g, const YeeC& c, cudaStream_t st, int sms,
           const XAdv* xa = nullptr, YeeHook* hk = nullptr) {
  long long faces = (long long)(g.jy2 - g.jy1 + 1) * (g.kz2 - g.kz1 + 1) + (long long)(g.ix2 - g.ix1 + 1) * (g.kz2 - g.kz1 + 1) +
                    (g.ndim == 3 ? (long long)(g.ix2 - g.ix1 + 1) * (g.jy2 - g.jy1 + 1) : 0);
  int gf = grid_for(faces, 256, sms);
  const dim3 blk(YEE_BX, YEE_BY, 1);
  const dim3 grd((g.ix2 - g.ix1 + YEE_BX) / YEE_BX, (g.jy2 - g.jy1 + YEE_BY) / YEE_BY,
                 g.ndim == 3 ? g.kz2 - g.kz1 + 1 : 1);
  double dt = c.dt, dth = 0.5 * dt;
  // the comoving frame's advection substeps (curr_and_fields_util.f90:200-258)
  const bool adv = xa && c.vbeam > 0.0;
  const int nb1 = g.nc + 1, nb2 = g.nf, ne1 = 1, ne2 = g.nc;
  auto halo = [&](int point) {
    if (hk && !hk->rc) hk->rc = hk->fn(hk->ctx, point);
    return hk && hk->rc;
  };
  // the boundary ghosts ride in the sweeps unless something runs between the
  // two (a halo exchange, an advection substep) or the wide x difference
  // reads further out: three launches instead of six (the boundary sweeps
  // took 4 to 5 us each on every grid)
  if (!hk && !adv && c.se2 == 0.0) {
    auto sweeps = [&](auto nd) {
      constexpr int N = decltype(nd)::value;
      k_rote<T, N, true, false><<<grd, blk, 0, st>>>(ebf, g, c, dth, 0.0);
      k_rotb_j<T, N, true, false><<<grd, blk, 0, st>>>(ebf, jc, jlo, g, c, dt);
      k_rote<T, N, true, false><<<grd, blk, 0, st>>>(ebf, g, c, dth, dt);
    };
    if (g.ndim == 3) sweeps(std::integral_constant<int, 3>());
    else sweeps(std::integral_constant<int, 2>());
    return;
  }
  auto rote = [&]() {
    if (g.ndim == 3) k_rote<T, 3, false, true><<<grd, blk, 0, st>>>(ebf, g, c, dth, 0.0);
    else k_rote<T, 2, false, true><<<grd, blk, 0, st>>>(ebf, g, c, dth, 0.0);
  };
  k_ef_bds<T><<<gf, 256, 0, st>>>(ebf, g, c, 0.0);
  if (halo(AGPU_HALO_E)) return;
  if (adv) xadvect_t<T>(ebf, g, nb1, nb2, 0, *xa, st, sms);
  rote();
  k_bf_bds<T><<<gf, 256, 0, st>>>(ebf, g, c, dt);
  if (halo(AGPU_HALO_B)) return;
  if (adv) xadvect_t<T>(ebf, g, ne1, ne2, 0, *xa, st, sms);
  if (g.ndim == 3) k_rotb_j<T, 3, false, true><<<grd, blk, 0, st>>>(ebf, jc, jlo, g, c, dt);
  else k_rotb_j<T, 2, false, true><<<grd, blk, 0, st>>>(ebf, jc, jlo, g, c, dt);
  if (adv) xadvect_t<T>(ebf, g, ne1, ne2, 2, *xa, st, sms);
  k_ef_bds<T><<<gf, 256, 0, st>>>(ebf, g, c, dt);
  if (halo(AGPU_HALO_E)) return;
  rote();
  if (adv) xadvect_t<T>(ebf, g, nb1, nb2, 2, *xa, st, sms);
}

}  // namespace agpu
