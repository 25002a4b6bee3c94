// agpu_bin.cu — per-step binning of particles by spatial tile: a key per
// particle (its tile and row inside the tile, or the removed bin), a
// histogram, an exclusive scan and a scatter of particle indices into the
// permutation perm, so that tile t's particles are
// perm[tstart[t * nsub] .. tstart[(t + 1) * nsub]), row by row.  The particle records stay
// where they are; the permutation is rebuilt every step from the keys that
// the push kernel writes, and the records are physically reordered along it
// whenever the window compaction copies them.
#include "agpu_bin.cuh"
#include "agpu_multi.h"
#include "agpu_util.h"
#include "agpu_select.cuh"

namespace agpu {

// keys from the split form's node index and offsets
__global__ void k_keys_split(const int* cell, const float* ox, const float* oy, const float* oz, long long np, Geo g,
                             TileGeo t, int* key, int* hist, unsigned int* err) {
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < np; n += (long long)gridDim.x * blockDim.x) {
    int c = cell[n];
    int i, j, k;
    cell_split(g, c, i, j, k);
    if (g.ndim != 3) k = 3;
    int kk = tile_key(t, i, j, k, offset_octant(ox[n], oy[n], (g.ndim == 3) ? oz[n] : 0.f, g.ndim));
    key[n] = kk;
    if (kk == t.nkeys) raise_err(err, AGPU_EBIT_INDEX);  // a record outside the node range
    hist_add(hist, kk);
  }
}

// keys from FP64 absolute positions: node = int(3 + x_loc + 0.5) (qden)
__global__ void k_keys_abs(const double* x, const double* y, const double* z, long long np, Geo g, TileGeo t,
                           double xmn, double ymn, double zmn, double dxi, double dyi, double dzi, int* key, int* hist,
                           unsigned int* err) {
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < np; n += (long long)gridDim.x * blockDim.x) {
    double xx = 3.0 + dxi * (x[n] - xmn);
    double yy = 3.0 + dyi * (y[n] - ymn);
    int i = (xx > -1e9 && xx < 2e9) ? (int)(xx + 0.5) : -1;
    int j = (yy > -1e9 && yy < 2e9) ? (int)(yy + 0.5) : -1;
    int k = 3;
    float sz = 0.f;
    if (g.ndim == 3) {
      double zz = 3.0 + dzi * (z[n] - zmn);
      k = (zz > -1e9 && zz < 2e9) ? (int)(zz + 0.5) : -1;
      sz = (float)(zz - (double)k);
    }
    int kk = tile_key(t, i, j, k, offset_octant((float)(xx - (double)i), (float)(yy - (double)j), sz, g.ndim));
    key[n] = kk;
    if (kk == t.nkeys) raise_err(err, AGPU_EBIT_INDEX);  // a record outside the node range
    hist_add(hist, kk);
  }
}

// perm[cursor[key]++] = n with warp-aggregated cursors (which start at the
// keys' first slots).  Each warp
// takes SC_U consecutive runs of 32 records per pass, so that SC_U cursor
// atomics (one round trip to L2 each) are in flight together; the lanes of
// a run with one key get consecutive slots in lane order.  Warp-uniform loop
// (blockDim a multiple of 32).
constexpr int SC_U = 4;
__device__ void d_perm_scatter(const int* key, long long np, int* cursor, int* perm, long long bid_, long long nb_) {
  const int lane = threadIdx.x & 31;
  const long long warp = (bid_ * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (nb_ * (long long)blockDim.x) >> 5;
  for (long long base = warp * 32 * SC_U; base < np; base += nwarps * 32 * SC_U) {
    int kk[SC_U], b[SC_U], rank[SC_U], lead[SC_U];
#pragma unroll
    for (int u = 0; u < SC_U; ++u) {
      const long long n = base + u * 32 + lane;
      kk[u] = (n < np) ? key[n] : -1;
    }
#pragma unroll
    for (int u = 0; u < SC_U; ++u) {
      const unsigned peers = __match_any_sync(0xffffffffu, kk[u]);
      lead[u] = __ffs(peers) - 1;
      rank[u] = __popc(peers & ((1u << lane) - 1u));
      b[u] = 0;
      if (lane == lead[u] && kk[u] >= 0) b[u] = atomicAdd(&cursor[kk[u]], __popc(peers));
    }
#pragma unroll
    for (int u = 0; u < SC_U; ++u) {
      const int bb = __shfl_sync(0xffffffffu, b[u], lead[u]);
      if (kk[u] >= 0) perm[bb + rank[u]] = (int)(base + u * 32 + lane);
    }
  }
}
__global__ void k_perm_scatter(const int* key, long long np, int* cursor, int* perm) {
  d_perm_scatter(key, np, cursor, perm, blockIdx.x, gridDim.x);
}

void bin_keys_split(const int* cell, const float* ox, const float* oy, const float* oz, long long np, const Geo& g,
                    const TileGeo& t, int* key, int* hist, unsigned int* err, cudaStream_t st, int sms) {
  if (np <= 0) return;
  k_keys_split<<<grid_for(np, 256, sms, 16), 256, 0, st>>>(cell, ox, oy, oz, np, g, t, key, hist, err);
}
void bin_keys_abs(const double* x, const double* y, const double* z, long long np, const Geo& g, const TileGeo& t,
                  double xmn, double ymn, double zmn, double dxi, double dyi, double dzi, int* key, int* hist,
                  unsigned int* err, cudaStream_t st, int sms) {
  if (np <= 0) return;
  k_keys_abs<<<grid_for(np, 256, sms, 16), 256, 0, st>>>(x, y, z, np, g, t, xmn, ymn, zmn, dxi, dyi, dzi, key, hist, err);
}
// ---- exclusive scan of the histogram ------------------------------------
// start[i] = cursor[i] = sum of hist[0..i), start[n] = total.  A block scans
// SCAN_BLOCK bins and finds its first value itself, by adding what precedes
// it: up to SCAN_ONE bins straight from the histogram (one launch, whose
// last block reads 256 KB from L2: 6.2 us at 2.6e3 keys, 12.5 at 3.5e4),
// beyond that from the blocks' sums (two launches: 10.3 + 15.0 us at 1.04e6).
// The earlier scan of the block sums by one serial block was a launch of its
// own of 9 us on every grid beside two of that size.
constexpr int SCAN_ITEMS = 16, SCAN_THREADS = 256, SCAN_BLOCK = SCAN_ITEMS * SCAN_THREADS;
constexpr int SCAN_ONE = 16 * SCAN_BLOCK;

// Sum over the block of v and this thread's exclusive prefix.
__device__ __forceinline__ int block_exclusive_sum(int v, int* total) {
  __shared__ int s_warp[SCAN_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  __syncthreads();  // s_warp may still be read for an earlier sum
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  int base = 0, all = 0;
#pragma unroll
  for (int w = 0; w < SCAN_THREADS / 32; ++w) {
    base += (w < warp) ? s_warp[w] : 0;
    all += s_warp[w];
  }
  *total = all;
  return base + inc - v;
}

// Sum of block blk's bins.
__device__ __forceinline__ void d_scan_sums(const int* hist, int n, int blk, int* bsum) {
  const int base = blk * SCAN_BLOCK;
  int v = 0, total;
  for (int e = threadIdx.x; e < SCAN_BLOCK; e += SCAN_THREADS)
    if (base + e < n) v += hist[base + e];
  block_exclusive_sum(v, &total);
  if (threadIdx.x == 0) bsum[blk] = total;
}
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_sums(const int* hist, int n, int* bsum) {
  d_scan_sums(hist, n, blockIdx.x, bsum);
}

// The thread's rows with more than cap records, listed (SCAN_ITEMS keys from
// `base` on are whole rows; key n - 1 marks removed records).
__device__ __forceinline__ void list_rows(const int h[SCAN_ITEMS], int base, int n, int nq, const RowList& rows, int cap) {
  int c[4], nrow = 4;  // four rows of quadrants or two of octants
#pragma unroll
  for (int r = 0; r < 4; ++r) c[r] = h[4 * r] + h[4 * r + 1] + h[4 * r + 2] + h[4 * r + 3];
  if (nq == 8) {
    c[0] += c[1];
    c[1] = c[2] + c[3];
    nrow = 2;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int row = base / nq + r;
    if (r >= nrow || (row + 1) * nq > n - 1 || c[r] <= cap) continue;
    const int items = (c[r] - cap + ROW_ITEM - 1) / ROW_ITEM;
    const unsigned e = atomicAdd(&rows.n[0], (unsigned)items);
    for (int q = 0; q < items && e + q < (unsigned)rows.size; ++q) {
      rows.item[2 * (e + q)] = row;
      rows.item[2 * (e + q) + 1] = q * ROW_ITEM;
    }
  }
}

// Block blk of the scan; before[0..nbefore) adds up to its first value.
__device__ __forceinline__ void d_scan(const int* hist, int n, const int* before, int nbefore, int blk, int* start,
                                       int* cursor, int nq = 0, const RowList* rows = nullptr, int cap = 0) {
  int v = 0, first, total;
  for (int e = threadIdx.x; e < nbefore; e += SCAN_THREADS) v += before[e];
  block_exclusive_sum(v, &first);
  const int base = blk * SCAN_BLOCK + threadIdx.x * SCAN_ITEMS;
  int h[SCAN_ITEMS], sum = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    h[k] = (base + k < n) ? hist[base + k] : 0;
    sum += h[k];
  }
  int run = first + block_exclusive_sum(sum, &total);
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    if (base + k < n) {
      start[base + k] = run;
      cursor[base + k] = run;
    }
    run += h[k];
    if (base + k == n - 1) start[n] = run;
  }
  if (rows) {
    if (blk == 0 && threadIdx.x == 0) rows->n[3] = (unsigned)cap;
    list_rows(h, base, n, nq, *rows, cap);
  }
}
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(const int* hist, int n, const int* bsum, int* start, int* cursor,
                                                       int nq, RowList rows, int cap) {
  const int blk = blockIdx.x;
  d_scan(hist, n, bsum ? bsum : hist, bsum ? blk : blk * SCAN_BLOCK, blk, start, cursor, nq, rows.n ? &rows : nullptr, cap);
}

// hist has nkeys+1 bins (the last one: removed particles).  scan_tmp holds
// bin_scan_tmp_ints(t) ints.  Returns the kernels launched.
int bin_finish(const int* key, long long np, const TileGeo& t, const int* hist, int* start, int* cursor, int* perm,
               int* scan_tmp, const RowList& rows, cudaStream_t st, int sms) {
  const int n = t.nkeys + 1;
  const int nb = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
  const bool one = n <= SCAN_ONE;
  if (!one) k_scan_sums<<<nb, SCAN_THREADS, 0, st>>>(hist, n, scan_tmp);
  k_scan<<<nb, SCAN_THREADS, 0, st>>>(hist, n, one ? nullptr : scan_tmp, start, cursor, t.nq, rows, row_cap(np, t));
  if (np > 0) k_perm_scatter<<<grid_for(np, 256, sms, 16), 256, 0, st>>>(key, np, cursor, perm);
  return (one ? 1 : 2) + (np > 0 ? 1 : 0);
}
int bin_scan_tmp_ints(const TileGeo& t) { return (t.nkeys + 1) / SCAN_BLOCK + 1; }

// ---- compaction along the permutation (physical reorder by tile) --------
struct PermAlive {
  const int* perm;
  long long nalive;
  __device__ bool operator()(long long q) const { return q < nalive; }
};
struct PermAliveInBox64 {
  const int* perm;
  long long nalive;
  const double* x;
  double x0, x1;
  __device__ bool operator()(long long q) const {
    if (q >= nalive) return false;
    double a = x[perm[q]];
    return a > x0 && a <= x1;
  }
};
struct PermMove64 {
  const int* perm;
  const double* src;
  double* dst;
  long long ld;
  int ndv;
  __device__ void operator()(long long q, long long o) const {
    long long p = perm[q];
    for (int c = 0; c < ndv; ++c) dst[(long long)c * ld + o] = src[(long long)c * ld + p];
  }
};
long long perm_compact64(const int* perm, long long nalive, double* part, double* tmp, long long cap, int ndv, bool xbox,
                         double x0, double x1, Scratch& s, cudaStream_t st) {
  PermMove64 mv{perm, part, tmp, cap, ndv};
  if (xbox) {
    PermAliveInBox64 pr{perm, nalive, part, x0, x1};
    return select_run(pr, mv, nalive, s, st);
  }
  PermAlive pr{perm, nalive};
  return select_run(pr, mv, nalive, s, st);
}

struct PermAliveInBox32 {
  const int* perm;
  long long nalive;
  const int* cell;
  const float* ox;
  int n1p, nx;
  __device__ bool operator()(long long q) const {
    if (q >= nalive) return false;
    int p = perm[q];
    int i = cell[p] % n1p + 1;
    int m = i - 3;
    float o = ox[p];
    return ((m > 0) || (m == 0 && o > 0.f)) && ((m < nx) || (m == nx && o <= 0.f));
  }
};
struct PermMove32 {
  const int* perm;
  Part32View src, dst;
  __device__ void operator()(long long q, long long o) const {
    int p = perm[q];
    dst.cell[o] = src.cell[p];
    dst.ox[o] = src.ox[p];
    dst.oy[o] = src.oy[p];
    dst.px[o] = src.px[p];
    dst.py[o] = src.py[p];
    dst.slot[o] = src.slot[p];
    if (src.oz) {
      dst.oz[o] = src.oz[p];
      dst.pz[o] = src.pz[p];
    }
  }
};
long long perm_compact32(const int* perm, long long nalive, const Part32View& src, const Part32View& dst, bool xbox, int n1p,
                         int nx, Scratch& s, cudaStream_t st) {
  PermMove32 mv{perm, src, dst};
  if (xbox) {
    PermAliveInBox32 pr{perm, nalive, src.cell, src.ox, n1p, nx};
    return select_run(pr, mv, nalive, s, st);
  }
  PermAlive pr{perm, nalive};
  return select_run(pr, mv, nalive, s, st);
}


// ---- multi-instance binning: scan, scatter (a row of blocks per instance) --
// The scan's routes and their line are bin_finish's, instance by instance: with
// the one-launch form at every size two instances of 256x128x128 cells (1.25e6
// keys each) took 181 us a step against 11 + 31 us, and a step of two of
// 512x256x256 cells 27.8 ms against 24.0.
namespace {
__global__ void __launch_bounds__(SCAN_THREADS) km_scan_sums(const MultiInst* __restrict__ d) {
  const MultiInst& m = d[blockIdx.y];
  const int n = m.ta.t.nkeys + 1;
  if (n <= SCAN_ONE || (int)blockIdx.x * SCAN_BLOCK >= n) return;
  d_scan_sums(m.ta.hist, n, blockIdx.x, m.scan_tmp);
}
__global__ void __launch_bounds__(SCAN_THREADS) km_scan(const MultiInst* __restrict__ d) {
  const MultiInst& m = d[blockIdx.y];
  const int n = m.ta.t.nkeys + 1, blk = blockIdx.x;
  if (blk * SCAN_BLOCK >= n) return;
  int* start = const_cast<int*>(m.ta.tstart);
  if (n > SCAN_ONE) d_scan(m.ta.hist, n, m.scan_tmp, blk, blk, start, m.cursor);
  else d_scan(m.ta.hist, n, m.ta.hist, blk * SCAN_BLOCK, blk, start, m.cursor);
}
__global__ void km_scatter(const MultiInst* __restrict__ d) {
  const MultiInst& m = d[blockIdx.y];
  d_perm_scatter(m.ta.key, m.np, m.cursor, const_cast<int*>(m.ta.perm), blockIdx.x, gridDim.x);
}
}  // namespace

void multi_bin32(const MultiInst* d, const MultiPlan& pl, cudaStream_t st, int* launches) {
  const dim3 grd((pl.max_keys + SCAN_BLOCK) / SCAN_BLOCK, pl.n);
  if (pl.max_keys + 1 > SCAN_ONE) {  // some instance is beyond the one-launch limit
    km_scan_sums<<<grd, SCAN_THREADS, 0, st>>>(d);
    *launches += 1;
  }
  km_scan<<<grd, SCAN_THREADS, 0, st>>>(d);
  km_scatter<<<dim3(pl.gx_parts, pl.n), 256, 0, st>>>(d);
  *launches += 2;
}

}  // namespace agpu
