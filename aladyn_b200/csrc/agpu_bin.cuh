// agpu_bin.cuh — spatial tiles of the particle binning (tile geometry and
// node -> tile key), shared by the tiled push kernels and the binning pass.
#pragma once
#include "agpu_common.cuh"

namespace agpu {

// A tile is TX x TY x TZ integer nodes; node i (Fortran) of an alive particle
// lies in [3, nx+3], so tiles cover nodes 3.. in steps of TX.  The binning
// key of a particle is its tile, its row (y, z) inside the tile and the
// octant of its offset from its node (quadrant in 2D):
//   key = tile * nsub + (ly + ty * lz) * nq + octant,  nsub = ty * tz * nq,
// so tile t's particles are perm[tstart[t * nsub] .. tstart[(t + 1) * nsub]),
// row by row and, inside a row, octant by octant.  A row's octant bucket
// holds about one particle per cell of the row (the lattice points of a cell
// start in different octants and a cell's particles spread over them), so
// a warp of the tile kernel covers one or two buckets: consecutive cells of
// one row, about two lanes per cell, whatever order the window compactions
// and tile changes left the records in.  Its shared-memory reads then hit
// distinct banks and its atomics few lanes per address.  Key nkeys =
// ntiles * nsub marks a removed particle.
struct TileGeo {
  int tx, ty, tz;     // tile extent in nodes
  int ntx, nty, ntz;  // tiles per axis
  int ntiles;         // ntx*nty*ntz
  int nq;             // offset octants (3D: 8) or quadrants (2D: 4)
  int nsub;           // keys per tile, ty*tz*nq
  int nkeys;          // ntiles*nsub; key nkeys = removed particle
};

// octant (quadrant) of a particle's offsets from its node
AGPU_HD int offset_octant(float ox, float oy, float oz, int ndim) {
  return (ox >= 0.f ? 1 : 0) + (oy >= 0.f ? 2 : 0) + ((ndim == 3 && oz >= 0.f) ? 4 : 0);
}

AGPU_HD int tile_key(const TileGeo& t, int i, int j, int k, int oct) {
  const int a = (i - 3), b = (j - 3), c = (k - 3);
  if (a < 0 || b < 0 || c < 0) return t.nkeys;
  const int ta = a / t.tx, tb = b / t.ty, tc = c / t.tz;
  if (ta >= t.ntx || tb >= t.nty || tc >= t.ntz) return t.nkeys;
  const int tile = ta + t.ntx * (tb + t.nty * tc);
  return tile * t.nsub + ((b - tb * t.ty) + t.ty * (c - tc * t.tz)) * t.nq + oct;
}

// tile_key for a kernel compiled for the tile extent (TX, TY, TZ) == (t.tx,
// t.ty, t.tz) and NQ == t.nq.
template <int TX, int TY, int TZ, int NQ>
AGPU_HD int tile_key_c(const TileGeo& t, int i, int j, int k, int oct) {
  const unsigned a = (unsigned)(i - 3), b = (unsigned)(j - 3), c = (unsigned)(k - 3);
  const unsigned ta = a / TX, tb = b / TY, tc = c / TZ;
  if (ta >= (unsigned)t.ntx || tb >= (unsigned)t.nty || tc >= (unsigned)t.ntz) return t.nkeys;
  const int tile = (int)ta + t.ntx * ((int)tb + t.nty * (int)tc);
  return tile * (TY * TZ * NQ) + ((int)(b - tb * TY) + TY * (int)(c - tc * TZ)) * NQ + oct;
}

// Warp-aggregated histogram increment of key (all active lanes call it).
__device__ __forceinline__ void hist_add(int* hist, int key) {
  unsigned int act = __activemask();
  unsigned int peers = __match_any_sync(act, key);
  int leader = __ffs(peers) - 1;
  if ((threadIdx.x & 31) == leader) atomicAdd(&hist[key], __popc(peers));
}

// Dense rows of the FP64 tile kernels, which give a row of 32 nodes to one
// warp.  A row's own warp takes its first `cap` records; the scan lists the
// rest in items of ROW_ITEM records, which further CTAs of the tile kernels'
// launches share out over all their warps.  A bunch a few cells wide lies in a
// handful of rows, and with one warp a row a launch ran at the pace of the
// fullest: 4e6 electrons of sigma (8, 1, 1) cells in a 192x96x96 box took
// 171 ms an envelope step against 6.3 so (FP64 standard cycle 115 against
// 5.4); sigma (25, 6, 6): 4.9 against 3.2 (5.0 against 2.8).
struct RowList {
  unsigned int* n;  // items listed, items taken, CTAs that found no more, cap; null: no list (split form)
  int* item;        // (row, first record past the cap) pairs
  int size;         // items the list holds
};
constexpr int ROW_ITEM = 4096;
// Records of a row that stay with its warp: four times the mean of all rows
// (evenly dense plasma needs no sharing out, and an item stages its tile's
// fields again), and what a warp gets through while the launch takes an eighth
// of its time (0.3 us a record against 0.13 ns of the whole chip: np / 16384),
// at least four groups.  Without the second, smooth bunches and ionized regions
// of large runs were cut up for nothing: 512x256x256 cells with a bunch of
// sigma (25, 6, 6) took 52.4 ms an envelope step against 49.9, 768x192x192 cells
// with ionization 30.4 against 27.8 (49.6 and 27.6 with no sharing out at all).
AGPU_HD int row_cap(long long np, const TileGeo& t) {
  const long long nrows = (long long)t.nkeys / t.nq, mean4 = 4 * np / nrows, c = mean4 > np / 16384 ? mean4 : np / 16384;
  return c < 512 ? 512 : c > (1 << 30) ? (1 << 30) : (int)((c + 127) / 128 * 128);
}
// Items of rows with np records in all: a row beyond its cap (>= 512) lists
// at most one item more than its records fill.
AGPU_HD int row_list_size(long long np) { return (int)(np / ROW_ITEM + np / 512 + 1); }
// The list behind a binning's key starts: ints for both.
AGPU_HD size_t tstart_ints(long long np, const TileGeo& t) { return (size_t)t.nkeys + 2 + 4 + 2 * (size_t)row_list_size(np); }
inline RowList row_list(int* tstart, long long np, const TileGeo& t) {
  int* n = tstart + t.nkeys + 2;
  return RowList{(unsigned int*)n, n + 4, row_list_size(np)};
}

// The next histogram's reset: bins zero, the dead bin seeded with the records
// already dead (no tile visits them); with `pushed` set, the alive count of
// this push (tstart[nkeys]) is added to it (the deferred-count mode keeps the
// push count on the device); the split form's work-list counters cleared.
struct HistReset {
  int* hist;
  const int* tstart;
  int nkeys, np;
  unsigned long long* pushed;
  unsigned int* work_n;
};
__device__ __forceinline__ void hist_reset_bin(const HistReset& h, int b) {
  if (h.work_n && b < 2) h.work_n[b] = 0u;
  if (b > h.nkeys) return;
  const int alive = (b == h.nkeys) ? h.tstart[b] : 0;
  h.hist[b] = (b == h.nkeys) ? h.np - alive : 0;
  if (b == h.nkeys && h.pushed) *h.pushed += (unsigned long long)alive;
}

struct Scratch;
struct Part32View;
void bin_keys_split(const int* cell, const float* ox, const float* oy, const float* oz, long long np, const Geo& g,
                    const TileGeo& t, int* key, int* hist, unsigned int* err, cudaStream_t st, int sms);
void bin_keys_abs(const double* x, const double* y, const double* z, long long np, const Geo& g, const TileGeo& t,
                  double xmn, double ymn, double zmn, double dxi, double dyi, double dzi, int* key, int* hist,
                  unsigned int* err, cudaStream_t st, int sms);
// Returns the number of kernels it launched.
int bin_finish(const int* key, long long np, const TileGeo& t, const int* hist, int* start, int* cursor, int* perm,
               int* scan_tmp, const RowList& rows, cudaStream_t st, int sms);
// ints of bin_finish's scan_tmp
int bin_scan_tmp_ints(const TileGeo& t);
long long perm_compact64(const int* perm, long long nalive, double* part, double* tmp, long long cap, int ndv, bool xbox,
                         double x0, double x1, Scratch& s, cudaStream_t st);
long long perm_compact32(const int* perm, long long nalive, const Part32View& src, const Part32View& dst, bool xbox, int n1p,
                         int nx, Scratch& s, cudaStream_t st);

}  // namespace agpu
