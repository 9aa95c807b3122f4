// Plan construction: bit-exact cell assignment of every visibility (K1),
// counting sort into grid tiles or kernel groups (K2), and the work list of
// the persistent gridding kernels.
//
// Replaces the per-visibility coordinate work of convgrid/convdegrid
// (crocodile/synthesis.py:476-479, 497-499 via frac_coords :438-449) and the
// w ordering of sort_vis_w (:506-515).
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <new>

#include "cg_internal.cuh"

namespace cg {

static inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// ---------------------------------------------------------------- scan
// Exclusive scan of int32 counts (bucket histograms).  Three phases:
// per-block scan + block totals, scan of the totals, add-back.
static constexpr int SCAN_THREADS = 1024;
static constexpr int SCAN_PER_THREAD = 4;
static constexpr int SCAN_TILE = SCAN_THREADS * SCAN_PER_THREAD;

__device__ __forceinline__ int block_exclusive_scan(int v, int *s_warp,
                                                    int &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int nw = blockDim.x >> 5;
    int w = lane < nw ? s_warp[lane] : 0;
    int winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    if (lane < nw) s_warp[lane] = winc - w;
    if (lane == 31) s_warp[32] = winc;
  }
  __syncthreads();
  total = s_warp[32];
  int r = s_warp[warp] + inc - v;
  __syncthreads();
  return r;
}

__global__ void k_scan_tiles(const int32_t *__restrict__ in,
                             int32_t *__restrict__ out, int n,
                             int32_t *__restrict__ block_sums) {
  __shared__ int s_warp[33];
  const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  int v[SCAN_PER_THREAD];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    sum += v[k];
  }
  int total;
  int run = block_exclusive_scan(sum, s_warp, total);
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0 && block_sums) block_sums[blockIdx.x] = total;
}

__global__ void k_scan_add(int32_t *__restrict__ out, int n,
                           const int32_t *__restrict__ block_offsets) {
  const int i = blockIdx.x * SCAN_TILE + threadIdx.x;
  const int add = block_offsets[blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    int j = i + k * SCAN_THREADS;
    if (j < n && j < (blockIdx.x + 1) * SCAN_TILE) out[j] += add;
  }
}

// Scratch of the recursive scan: per level the block totals and their scan.
size_t scan_scratch_words(int n) {
  const int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nb <= 1) return 0;
  return 2 * (size_t)(nb + 1) + scan_scratch_words(nb);
}

int launch_scan(const int32_t *in, int32_t *out, int n, int32_t *scratch,
                cudaStream_t s) {
  if (n <= 0) return CG_OK;
  const int nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nb == 1) {
    k_scan_tiles<<<1, SCAN_THREADS, 0, s>>>(in, out, n, nullptr);
    CG_LAUNCH("scan");
    return CG_OK;
  }
  int32_t *sums = scratch, *sums_off = scratch + nb + 1;
  k_scan_tiles<<<nb, SCAN_THREADS, 0, s>>>(in, out, n, sums);
  CG_LAUNCH("scan");
  const int rc = launch_scan(sums, sums_off, nb, scratch + 2 * (nb + 1), s);
  if (rc) return rc;
  k_scan_add<<<nb, SCAN_THREADS, 0, s>>>(out, n, sums_off);
  CG_LAUNCH("scan");
  return CG_OK;
}

// ---------------------------------------------------------------- K1 coordinates
struct CoordParams {
  const double *uvw;
  int64_t stride;
  double lam;
  int64_t n;
  int H, W, Q, S, G, sep;
  const int32_t *kidx;
  int mode, T, tblog, nbx, nbuckets, sublog, subshift;
  const int32_t *layer;  // per-visibility layer (grid of the stack), or NULL
  int layers, tpl;
  const int32_t *group;  // groups mode: per-visibility launch group, or NULL (= kernel group)
  int ngroups;
  AxisConst ax, ay;    // filtered-exact constants for x (width W) and y (height H)
  double wstep, inv_wstep;  // wstep != 0: the kernel group is the w bin - kmin
  int kmin, nk;
  VisRec *rec;
  int32_t *key;
  int32_t *rank;
  int32_t *hist;
  int32_t *status;
};

// Warp-aggregated increment of hist[key]; returns this lane's slot.  All 32
// lanes of the warp must call it (invalid lanes pass valid = false).
__device__ __forceinline__ int aggregated_slot(int32_t *hist, int key,
                                               bool valid) {
  const int lane = threadIdx.x & 31;
  unsigned peers = __match_any_sync(0xffffffffu, valid ? key : -1);
  int leader = __ffs(peers) - 1;
  int base = 0;
  if (valid && lane == leader) base = atomicAdd(&hist[key], __popc(peers));
  base = __shfl_sync(peers, base, leader);
  return base + __popc(peers & ((1u << lane) - 1u));
}

// Interleave the low 8 bits of x and y (Morton / Z order).
__device__ __forceinline__ int morton2(int x, int y) {
  return (int)(spread_bits((unsigned)x) | (spread_bits((unsigned)y) << 1));
}

// Tiled-mode bucket: tile (numbered along the blocked Morton curve), then the
// 4x4-cell sub-tile of the footprint origin along a Morton curve, so that
// consecutive visibilities of a work item are spatial neighbours.
__device__ __forceinline__ int tile_bucket(const CoordParams &P, int lyr, int x0, int y0) {
  const int ty = y0 / P.T, tx = x0 / P.T;
  const int ly = y0 - ty * P.T, lx = x0 - tx * P.T;
  return ((lyr * P.tpl + tile_index(tx, ty, P.tblog, P.nbx)) << (2 * P.sublog)) |
         morton2(lx >> P.subshift, ly >> P.subshift);
}

__global__ void k_plan_coords(CoordParams P) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool live = i < P.n;
  bool ok = live;
  int key = -1;
  VisRec r = {0, 0, 0, 0};
  if (live) {
    const double u = P.uvw[i * P.stride], v = P.uvw[i * P.stride + 1];
    int x, xf, y, yf;
    const bool inx = coord_fast(u, P.lam, P.ax, P.W, P.Q, x, xf);
    const bool iny = coord_fast(v, P.lam, P.ay, P.H, P.Q, y, yf);
    if (!(inx && iny)) {
      atomicAdd(&P.status[ST_RANGE], 1);
      ok = false;
    } else {
      int x0 = x - P.S / 2, y0 = y - P.S / 2;
      if (x0 < 0 || y0 < 0 || x0 + P.S > P.W || y0 + P.S > P.H) {
        atomicAdd(&P.status[ST_BOUNDS], 1);
        ok = false;
      }
      int g = 0;
      if (P.wstep != 0.0) {
        const long long j = w_bin_fast(P.uvw[i * P.stride + 2], P.wstep, P.inv_wstep) - P.kmin;
        g = (j >= 0 && j < P.nk) ? (int)j : -1;
      } else if (P.kidx) {
        g = P.kidx[i];
      }
      if (g < 0 || g >= P.G) {
        atomicAdd(&P.status[ST_INDEX], 1);
        ok = false;
      }
      const int lyr = P.layer ? P.layer[i] : 0;
      if (lyr < 0 || lyr >= P.layers) {
        atomicAdd(&P.status[ST_INDEX], 1);
        ok = false;
      }
      r.x0 = x0;
      r.y0 = y0;
      if (P.sep) {
        r.k0 = g * P.Q + yf;
        r.k1 = g * P.Q + xf;
      } else {
        r.k0 = g;
        r.k1 = yf * P.Q + xf;
      }
      int grp = g, gper = P.G;
      if (P.mode == CG_PLAN_GROUPS && P.group) {
        grp = P.group[i];
        gper = P.ngroups;
        if (grp < 0 || grp >= gper) {
          atomicAdd(&P.status[ST_INDEX], 1);
          ok = false;
        }
      }
      if (ok) key = (P.mode == CG_PLAN_TILED) ? tile_bucket(P, lyr, x0, y0) : lyr * gper + grp;
      if (ok && (unsigned)key >= (unsigned)P.nbuckets) {  // never: a bucket outside the histogram
        atomicAdd(&P.status[ST_INDEX], 1);
        ok = false;
        key = -1;
      }
    }
  }
  int slot = aggregated_slot(P.hist, key, ok);
  if (live) {
    P.rec[i] = r;
    P.key[i] = ok ? key : -1;
    P.rank[i] = slot;
  }
}

__global__ void k_plan_scatter(int64_t n, const VisRec *__restrict__ rec,
                               const int32_t *__restrict__ key,
                               const int32_t *__restrict__ rank,
                               const int32_t *__restrict__ offsets,
                               VisRec *__restrict__ out, int32_t *__restrict__ perm) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int k = key[i];
  if (k < 0) return;
  int pos = offsets[k] + rank[i];
  out[pos] = rec[i];
  perm[pos] = (int32_t)i;
}

// Work items: each tile's sorted range (its 4^sublog sub-tile buckets are
// contiguous) cut into pieces of at most `chunk` visibilities.  First the
// number of pieces per tile, then (after an exclusive scan of those numbers)
// the items at their scanned positions, so that the work list follows the
// tile numbering exactly and the persistent kernels, which take items in list
// order, visit the tiles in that order.
__global__ void k_plan_item_counts(int ntiles, int sublog, const int32_t *__restrict__ counts,
                                   const int32_t *__restrict__ offsets, int chunk,
                                   int32_t *__restrict__ nch) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  const int b0 = t << (2 * sublog), b1 = b0 + (1 << (2 * sublog)) - 1;
  const int c = offsets[b1] + counts[b1] - offsets[b0];
  nch[t] = (c + chunk - 1) / chunk;
}

__global__ void k_plan_items(int ntiles, int sublog, const int32_t *__restrict__ counts,
                             const int32_t *__restrict__ offsets, int chunk,
                             const int32_t *__restrict__ nch, const int32_t *__restrict__ ioff,
                             WorkItem *__restrict__ items, int32_t *__restrict__ nitems) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ntiles) return;
  if (t == ntiles - 1) *nitems = ioff[t] + nch[t];
  const int m = nch[t];
  if (m == 0) return;
  const int b0 = t << (2 * sublog), b1 = b0 + (1 << (2 * sublog)) - 1;
  const int off = offsets[b0];
  const int c = offsets[b1] + counts[b1] - off;
  const int base = ioff[t];
  for (int j = 0; j < m; ++j) {
    WorkItem w;
    w.tile = t;
    w.start = off + j * chunk;
    w.count = min(chunk, c - j * chunk);
    w.pad = 0;
    items[base + j] = w;
  }
}

// The whole of the above (bucket scan, item counts, their scan, items) in one
// block for small grids, where launches are most of a plan's time: up to 16384
// buckets in the place of five launches (27 us against 12 and their gaps), up to
// 4096 where two can do it (16384 tiles: 27 us against 10).
static constexpr int PLAN_SMALL_BUCKETS = 16384, PLAN_SMALL_TILES = 4096;

// Visibilities per item, by the tile's count.  An item's window reaches the grid by
// one addition per cell, so a crowded tile cut short (32 or 64, where n is small)
// adds up thousands of windows in 32 bits: 204,800 equal visibilities in one cell, off
// by 2.4e-5 in items of 64, by 5.3e-6 in items of 512.  So a tile makes at most 128
// items until they are that long (and its list, which one thread writes, is as much
// shorter).  (The longest for all of a crowded tile: S 16, 200k on 512^2, density 1 / r,
// 7,800 in the central tile: 146 us, 71 so, 69 in items of 64.)
struct ItemSize {
  int usual, crowded;
  __device__ __forceinline__ int of(int count) const {
    return max(usual, min(crowded, (count / 128 + 31) & ~31));
  }
};

__device__ __forceinline__ void write_items(int tile, int off, int count, int chunk, int base,
                                            WorkItem *items) {
  for (int j = 0; j * chunk < count; ++j) {
    WorkItem w;
    w.tile = tile;
    w.start = off + j * chunk;
    w.count = min(chunk, count - j * chunk);
    w.pad = 0;
    items[base + j] = w;
  }
}

// Whether a cell could get more than DIRECT_CELL_TAPS taps.  Taps reach it from the
// visibilities of `reach` tiles to an axis, so no cell does unless the tiles of
// some reach x reach block hold that many, and then one of them holds `few`
// (INT32_MAX: a plan that is not for the direct gridder, or for that alone).
struct Crowd {
  int few, reach, tblog, nbx, ntx, nty, tpl;
  template <int R>
  __device__ __forceinline__ bool blocks(const int32_t *c, int tx, int ty) const {
    constexpr int M = 2 * R - 1;
    int v[M][M];
#pragma unroll
    for (int y = 0; y < M; ++y)
#pragma unroll
      for (int x = 0; x < M; ++x) {  // loads in flight together
        const int px = tx - R + 1 + x, py = ty - R + 1 + y;
        v[y][x] = (unsigned)px < (unsigned)ntx && (unsigned)py < (unsigned)nty
                      ? __ldg(&c[tile_index(px, py, tblog, nbx)])
                      : 0;
      }
    bool over = false;
#pragma unroll
    for (int y = 0; y < R; ++y)
#pragma unroll
      for (int x = 0; x < R; ++x) {
        int sum = 0;
#pragma unroll
        for (int k = 0; k < R * R; ++k) sum += v[y + k / R][x + k % R];
        over = over || sum > DIRECT_CELL_TAPS;
      }
    return over;
  }
  // a tile of `few` or more
  __device__ bool around(const int32_t *counts, int tile) const {
    const int lyr = tile / tpl;
    int tx, ty;
    tile_xy(tile - lyr * tpl, tblog, nbx, tx, ty);
    const int32_t *c = counts + (int64_t)lyr * tpl;
    return reach == 1   ? blocks<1>(c, tx, ty)
           : reach == 2 ? blocks<2>(c, tx, ty)
           : reach == 3 ? blocks<3>(c, tx, ty)
                        : true;  // (requested tiles of 4 and 8 cells)
  }
};

// Where the direct gridder could run, the work list goes to it or, when a cell is
// crowded, to the windowed one that is launched beside it; the other finds none.
__device__ __forceinline__ void split_items(int nitems, bool crowded, int32_t *split) {
  split[0] = crowded ? 0 : nitems;
  split[1] = crowded ? nitems : 0;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_plan_small(
    int nbuckets, int ntiles, int sublog, const int32_t *__restrict__ counts, ItemSize size,
    Crowd crowd, int32_t *__restrict__ offsets, WorkItem *__restrict__ items,
    int32_t *__restrict__ nitems, int32_t *__restrict__ split) {
  __shared__ int s_warp[33];
  int carry = 0;
  bool over = false;
  for (int b0 = 0; b0 < nbuckets; b0 += SCAN_TILE) {
    const int base = b0 + threadIdx.x * SCAN_PER_THREAD;
    int v[SCAN_PER_THREAD], sum = 0, total;
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; ++k) {
      v[k] = base + k < nbuckets ? counts[base + k] : 0;
      sum += v[k];
    }
    int run = carry + block_exclusive_scan(sum, s_warp, total);
#pragma unroll
    for (int k = 0; k < SCAN_PER_THREAD; ++k) {
      if (base + k < nbuckets) offsets[base + k] = run;
      run += v[k];
    }
    carry += total;
  }
  const int n = carry;
  carry = 0;
  __syncthreads();  // the offsets of every bucket
  for (int t0 = 0; t0 < ntiles; t0 += SCAN_THREADS) {
    const int t = t0 + threadIdx.x;
    int off = 0, c = 0, total;
    if (t < ntiles) {
      const int next = (t + 1) << (2 * sublog);
      off = offsets[t << (2 * sublog)];
      c = (next < nbuckets ? offsets[next] : n) - off;
    }
    if (c >= crowd.few) over = over || crowd.around(counts, t);
    const int chunk = size.of(c), m = (c + chunk - 1) / chunk;
    const int at = carry + block_exclusive_scan(m, s_warp, total);
    write_items(t, off, c, chunk, at, items);
    carry += total;
  }
  const bool crowded = __syncthreads_or(over);
  if (threadIdx.x == 0) {
    *nitems = carry;
    split_items(carry, crowded, split);
  }
}

// Larger grids whose buckets are tiles: both scans as one (counts in the lower
// half of a 64-bit value, items in the upper), each block its SCAN_TILE buckets,
// the last block to finish the blocks' totals; then the items.
__device__ __forceinline__ unsigned long long block_exclusive_scan64(unsigned long long v,
                                                                     unsigned long long *s_warp,
                                                                     unsigned long long &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long w = lane < nw ? s_warp[lane] : 0;
    unsigned long long winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    if (lane < nw) s_warp[lane] = winc - w;
    if (lane == 31) s_warp[32] = winc;
  }
  __syncthreads();
  total = s_warp[32];
  const unsigned long long r = s_warp[warp] + inc - v;
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_plan_scan(
    int nbuckets, const int32_t *__restrict__ counts, ItemSize size, Crowd crowd,
    int32_t *__restrict__ offsets, int32_t *__restrict__ ioff, unsigned long long *sums,
    int32_t *done, int32_t *crowded, int32_t *__restrict__ nitems, int32_t *__restrict__ split) {
  __shared__ unsigned long long s_warp[33];
  __shared__ bool s_last;
  const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER_THREAD;
  unsigned long long v[SCAN_PER_THREAD], sum = 0, total;
  bool over = false;
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    const int c = base + k < nbuckets ? counts[base + k] : 0;
    if (c >= crowd.few) over = over || crowd.around(counts, base + k);
    const int chunk = size.of(c);
    v[k] = (unsigned long long)c | (unsigned long long)((c + chunk - 1) / chunk) << 32;
    sum += v[k];
  }
  unsigned long long run = block_exclusive_scan64(sum, s_warp, total);
#pragma unroll
  for (int k = 0; k < SCAN_PER_THREAD; ++k) {
    if (base + k < nbuckets) {
      offsets[base + k] = (int32_t)run;
      ioff[base + k] = (int32_t)(run >> 32);
    }
    run += v[k];
  }
  over = __syncthreads_or(over);
  if (threadIdx.x == 0) {
    sums[blockIdx.x] = total;
    if (over) atomicOr(crowded, 1);
    __threadfence();
    s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  unsigned long long carry = 0;
  for (int b0 = 0; b0 < (int)gridDim.x; b0 += SCAN_THREADS) {
    const int b = b0 + threadIdx.x;
    const unsigned long long x = b < (int)gridDim.x ? __ldcg(&sums[b]) : 0;
    const unsigned long long e = carry + block_exclusive_scan64(x, s_warp, total);
    if (b < (int)gridDim.x) sums[b] = e;
    carry += total;
  }
  if (threadIdx.x == 0) {
    *nitems = (int32_t)(carry >> 32);
    split_items((int32_t)(carry >> 32), __ldcg(crowded) != 0, split);
  }
}

__global__ void k_plan_finish(int nbuckets, const int32_t *__restrict__ counts, ItemSize size,
                              int32_t *__restrict__ offsets, const int32_t *__restrict__ ioff,
                              const unsigned long long *__restrict__ sums,
                              WorkItem *__restrict__ items) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nbuckets) return;
  const unsigned long long s = sums[t / SCAN_TILE];
  const int off = offsets[t] + (int32_t)s;
  offsets[t] = off;
  write_items(t, off, counts[t], size.of(counts[t]), ioff[t] + (int32_t)(s >> 32), items);
}

__global__ void k_frac_coords(const double *uvw, int64_t stride, double lam,
                              int64_t n, int H, int W, int Q, AxisConst ax, AxisConst ay,
                              int32_t *x, int32_t *xf, int32_t *y, int32_t *yf,
                              int32_t *status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double u = uvw[i * stride], v = uvw[i * stride + 1];
  int a = 0, b = 0, c = 0, d = 0;
  const bool inx = coord_fast(u, lam, ax, W, Q, a, b);
  const bool iny = coord_fast(v, lam, ay, H, Q, c, d);
  if (!(inx && iny)) atomicAdd(&status[ST_RANGE], 1);
  x[i] = a;
  xf[i] = b;
  y[i] = c;
  yf[i] = d;
}

// ---------------------------------------------------------------- w bins
// w_cache_imaging's bin (synthesis.py:793): wbin = wstep * round(w / wstep),
// half-to-even.  k = rint(w / wstep) is the bin number.
__global__ void k_w_bins(const double *uvw, int64_t stride, int64_t n, double wstep,
                         double inv_wstep, int32_t *kidx, int32_t *minmax, int32_t *status) {
  int lo = INT32_MAX, hi = INT32_MIN, bad = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const long long k = w_bin_fast(uvw[i * stride + 2], wstep, inv_wstep);
    if (!(k > -1000000000 && k < 1000000000)) {
      ++bad;
      kidx[i] = 0;
    } else {
      const int ki = (int)k;
      kidx[i] = ki;
      lo = min(lo, ki);
      hi = max(hi, ki);
    }
  }
  if (bad) atomicAdd(&status[ST_RANGE], bad);
  block_atomic_min_max(&minmax[0], &minmax[1], lo, hi);
}

__global__ void k_w_bins_rebase(int32_t *kidx, int64_t n, const int32_t *minmax) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) kidx[i] -= minmax[0];
}

// Bins against a known table range [kmin, kmin + nk): no host round trip.
__global__ void k_w_bins_fixed(const double *uvw, int64_t stride, int64_t n, double wstep,
                               double inv_wstep, int kmin, int nk, int32_t *kidx,
                               int32_t *status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long j = w_bin_fast(uvw[i * stride + 2], wstep, inv_wstep) - kmin;
  if (!(j >= 0 && j < nk)) {
    atomicAdd(&status[ST_INDEX], 1);
    kidx[i] = 0;
    return;
  }
  kidx[i] = (int32_t)j;
}

__global__ void k_minmax_init(int32_t *mm) {
  mm[0] = INT32_MAX;
  mm[1] = INT32_MIN;
}

// ---------------------------------------------------------------- ranges
// What an imaging call has to know on the host before it can lay out its kernel
// table: the extremes of u and v, and of the w bins, in one pass over uvw and
// one copy back.  Values travel as unsigned integers in the values' order, so
// that one atomicMax (of the value, or of its complement for a minimum) per
// block and extreme works from zeroed memory.  A NaN among u, v makes the
// minimum -inf.  2M visibilities: the strided minimum and maximum of two
// columns, the bins' own pass and their rebase took 97 us and three
// synchronisations per call; with this pass, the bins found in the plan's
// coordinate pass, and the table padded by one kernel, w_cache_imaging and
// w_cache_predict together went from 2.03 to 1.63 ms.
struct UvwRanges {
  unsigned long long uv_max, uv_min;  // order_bits of the maximum; ~ of the minimum
  uint32_t w_max, w_min;
};

__device__ __forceinline__ unsigned long long order_bits(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : b | (1ull << 63);
}

__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, v, o);
    v = t > v ? t : v;
  }
  return v;
}

__global__ void k_uvw_ranges(const double *__restrict__ uvw, int64_t stride, int64_t n,
                             double wstep, double inv_wstep, UvwRanges *out, int32_t *status) {
  unsigned long long hi = 0, lo = 0;
  uint32_t whi = 0, wlo = 0;
  int bad = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double *p = uvw + i * stride;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const double x = p[c];
      const unsigned long long b = order_bits(x);
      const bool nan = (unsigned long long)__double_as_longlong(x) << 1 > 0x7FFull << 53;
      const unsigned long long m = nan ? ~order_bits(-INFINITY) : ~b;
      hi = b > hi ? b : hi;
      lo = m > lo ? m : lo;
    }
    if (wstep != 0.0) {
      const long long k = w_bin_fast(p[2], wstep, inv_wstep);
      if (k > -1000000000 && k < 1000000000) {
        const uint32_t b = (uint32_t)(int)k ^ 0x80000000u;
        whi = max(whi, b);
        wlo = max(wlo, ~b);
      } else {
        ++bad;
      }
    }
  }
  if (bad) atomicAdd(&status[ST_RANGE], bad);
  __shared__ unsigned long long s_uv[2][32];
  __shared__ uint32_t s_w[2][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  hi = warp_max(hi);
  lo = warp_max(lo);
  whi = __reduce_max_sync(0xffffffffu, whi);
  wlo = __reduce_max_sync(0xffffffffu, wlo);
  if (lane == 0) {
    s_uv[0][warp] = hi;
    s_uv[1][warp] = lo;
    s_w[0][warp] = whi;
    s_w[1][warp] = wlo;
  }
  __syncthreads();
  if (warp != 0) return;
  const bool in = lane < (int)(blockDim.x >> 5);
  hi = warp_max(in ? s_uv[0][lane] : 0);
  lo = warp_max(in ? s_uv[1][lane] : 0);
  whi = __reduce_max_sync(0xffffffffu, in ? s_w[0][lane] : 0);
  wlo = __reduce_max_sync(0xffffffffu, in ? s_w[1][lane] : 0);
  if (lane != 0) return;
  atomicMax(&out->uv_max, hi);
  atomicMax(&out->uv_min, lo);
  if (wstep != 0.0) {
    atomicMax(&out->w_max, whi);
    atomicMax(&out->w_min, wlo);
  }
}

static double from_order_bits(unsigned long long b) {
  b = (b >> 63) ? b & ~(1ull << 63) : ~b;
  double x;
  memcpy(&x, &b, 8);
  return x;
}

// The S x S slices of a 4-D table with a zero first row and column.
__global__ void k_pad_even(const float2 *__restrict__ src, int64_t nslices, int S,
                           float2 *__restrict__ dst) {
  const int P = S + 1, PP = P * P;
  for (int64_t s = (int64_t)blockIdx.x * (blockDim.x / 256) + threadIdx.x / 256; s < nslices;
       s += (int64_t)gridDim.x * (blockDim.x / 256))
    for (int t = threadIdx.x % 256; t < PP; t += 256) {
      const int y = t / P, x = t - y * P;
      dst[s * PP + t] = y && x ? src[s * S * S + (y - 1) * S + x - 1] : make_float2(0.f, 0.f);
    }
}

// ---------------------------------------------------------------- key compaction
// The keys in use as a bitmap (one bit per possible key), the rank of a key
// = the prefix of the words' popcounts + the bits below it in its word: the
// key space of the tower schemes (chunks x planes x antenna pairs) runs to
// hundreds of millions of keys for a few hundred thousand visibilities, and
// a bit per key keeps the passes over it 32 times smaller than a flag word.
// Bits of the keys in use.  Small key spaces (at most KEY_SMEM_WORDS words:
// the w-towers' chunk x plane keys) collect in a shared-memory copy of the
// bitmap that each block ORs into the global one at the end, one atomic per
// non-zero word per block: the keys of a few thousand words take atomics
// from every warp of the grid otherwise, and atomics on one address
// serialise.  Larger key spaces set their bits directly, the lanes of a warp
// that set bits of one word merging them first.
constexpr int KEY_SMEM_WORDS = 8192;

__global__ void k_key_bits(const int32_t *__restrict__ key, int64_t n, int nkeys,
                           uint32_t *__restrict__ bits, int32_t *status) {
  extern __shared__ uint32_t s_bits[];
  const int nw = (nkeys + 31) >> 5;
  const bool local = nw <= KEY_SMEM_WORDS;
  if (local) {
    for (int w = threadIdx.x; w < nw; w += blockDim.x) s_bits[w] = 0u;
    __syncthreads();
  }
  int bad = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // whole warps walk the range together (the merge below needs all 32 lanes)
  const int64_t nround = (n + 31) & ~(int64_t)31;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nround; i += stride) {
    const int k = i < n ? key[i] : -1;
    const bool ok = k >= 0 && k < nkeys;
    if (i < n && !ok) ++bad;
    if (local) {
      if (ok) atomicOr(&s_bits[k >> 5], 1u << (k & 31));
      continue;
    }
    const int word = ok ? k >> 5 : -1;
    const uint32_t bit = ok ? 1u << (k & 31) : 0u;
    const uint32_t same = __match_any_sync(0xffffffffu, word);
    uint32_t acc = 0;
#pragma unroll
    for (int l = 0; l < 32; ++l) {
      const uint32_t b = __shfl_sync(0xffffffffu, bit, l);
      if (same & (1u << l)) acc |= b;
    }
    if (ok && (threadIdx.x & 31) == __ffs(same) - 1) atomicOr(&bits[word], acc);
  }
  if (bad) atomicAdd(&status[ST_INDEX], bad);
  if (local) {
    __syncthreads();
    for (int w = threadIdx.x; w < nw; w += blockDim.x)
      if (s_bits[w]) atomicOr(&bits[w], s_bits[w]);
  }
}

__global__ void k_key_popc(const uint32_t *__restrict__ bits, int nw, int32_t *__restrict__ cnt) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w < nw) cnt[w] = __popc(bits[w]);
}

__global__ void k_key_rows(const int32_t *__restrict__ key, int64_t n, int nkeys,
                           const uint32_t *__restrict__ bits, const int32_t *__restrict__ wpre,
                           int32_t *__restrict__ row) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = key[i];
  if (k < 0 || k >= nkeys) {
    row[i] = 0;
    return;
  }
  const uint32_t below = (1u << (k & 31)) - 1u;
  row[i] = wpre[k >> 5] + __popc(bits[k >> 5] & below);
}

__global__ void k_key_of_row(int nw, const uint32_t *__restrict__ bits,
                             const int32_t *__restrict__ wpre, int32_t *__restrict__ key_of_row) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nw) return;
  uint32_t b = bits[w];
  int r = wpre[w];
  while (b) {
    const int t = __ffs(b) - 1;
    key_of_row[r++] = (w << 5) + t;
    b &= b - 1u;
  }
}

// Kernel-cache key of every visibility for w_cache_imaging with src columns
// (synthesis.py:793-794: kernel_cache(theta, wbin, *src[i])): the w bin and
// the integer src columns of the row packed in mixed radix,
//   key = ((wbin - kmin) * r0 + (c0 - m0)) * r1 + (c1 - m1) ...
// A column value outside [m, m + r) is an index error (key 0).
struct RowKeyCols {
  int ncols;
  int32_t mins[8], ranges[8];
};

__global__ void k_row_keys(const double *__restrict__ uvw, int64_t stride, int64_t n,
                           double wstep, double inv_wstep, int kmin, int nbins,
                           const int32_t *__restrict__ cols, RowKeyCols C,
                           int32_t *__restrict__ key, int32_t *status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long j = w_bin_fast(uvw[i * stride + 2], wstep, inv_wstep) - kmin;
  bool ok = j >= 0 && j < nbins;
  int64_t k = ok ? (int64_t)j : 0;
  for (int c = 0; c < C.ncols; ++c) {
    const int v = cols[i * C.ncols + c] - C.mins[c];
    ok = ok && v >= 0 && v < C.ranges[c];
    k = k * C.ranges[c] + (ok ? v : 0);
  }
  if (!ok) {
    atomicAdd(&status[ST_INDEX], 1);
    k = 0;
  }
  key[i] = (int32_t)k;
}

// AW kernel key of every visibility: (a1 * nant + a2) * nbins + w bin - kmin, the
// (wbin, a1, a2) key of the AW kernel cache (scripts/image_dataset.py:153-171,
// synthesis.py:793).
__global__ void k_aw_keys(const double *__restrict__ uvw, int64_t stride,
                          const int32_t *__restrict__ a1, const int32_t *__restrict__ a2,
                          int64_t n, int nant, double wstep, double inv_wstep, int kmin,
                          int nbins, int32_t *__restrict__ key, int32_t *status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long j = w_bin_fast(uvw[i * stride + 2], wstep, inv_wstep) - kmin;
  const int p = a1[i], q = a2[i];
  if (!(j >= 0 && j < nbins) || p < 0 || p >= nant || q < 0 || q >= nant) {
    atomicAdd(&status[ST_INDEX], 1);
    key[i] = 0;
    return;
  }
  key[i] = (p * nant + q) * nbins + (int)j;
}

// ---------------------------------------------------------------- sizing
struct Layout {
  size_t rec_tmp, key, rank, recs, perm, counts, offsets, scan, items, tnch, tioff, ctr, kpad,
      total;
};

static int tile_edge(const cg_kernel_desc &kd, int req) {
  const cg_tuning t = tuning();
  const int S = kd.S;
  if (req > 0) return std::max(4, std::min(64, req & ~3));
  if (t.tile > 0) return std::max(4, std::min(64, t.tile & ~3));
  if (layout_for(kd) == CG_LAYOUT_LANE) return 16;  // per-warp windows stay small
  if (S <= 8) return 32;
  if (S <= 16) return 48;
  return 64;
}

// Most buckets of a plan, which are zeroed and scanned on each call
static constexpr int64_t MAX_BUCKETS = 1 << 24;
static int64_t tiles_of(const cg_plan &p, int T) {
  return (int64_t)((p.W + T - 1) / T) * ((p.H + T - 1) / T) * p.layers;
}

// Window edge of the register-window gridder for separable tables
// (grid_outer.cu) and its tile edge T (window >= T + S - 1), or 0 where another
// gridder runs: the one with shared-memory tiles for supports to 4 (its time goes with
// S, the window's flush does not; plan and grid, warp gridder / this one, us: S 3, 1M on
// 2048^2: 153 / 181, S 5: 174 / 179, on 4096^2: 200 / 183, S 6: 210 / 172, S 8: 239 / 170, on
// 4096^2: 259 / 218; 8 visibilities a cell of 512^2, S 1: 284 / 389, S 4: 311 / 384, S 5: 372 /
// 384, S 6: 433 / 387), but for dense visibilities of small calls, where its launches
// are the shorter (8 a cell of 48^2, 18,432, S 1: 39 / 33, S 4: 41 / 33; 98,304 on 256^2,
// S 1: 46 / 49, S 4: 48 / 50).  Stacks of grids, requested or tuned tiles and tuned
// layouts keep the other gridders.
static int outer_edge(const cg_plan &p, int &T) {
  const cg_tuning t = tuning();
  const int S = p.kd.S;
  if (p.lean || !p.kd.sep || S > 16 || p.layers != 1 || p.tile_req > 0 || t.tile > 0 ||
      t.layout > 0 || (int64_t)p.kd.G * p.kd.Q * S >= INT32_MAX)
    return 0;
  const double rho = (double)p.n / ((double)p.H * (double)p.W);
  const bool few = direct_fits(p);
  if (!few && S <= 4 && (rho < 1.5 || p.n >= 65536)) return 0;
  // few visibilities: small tiles, whose counts bound a cell's taps more closely;
  // larger tiles where they fit the window and are not full: fewer flushes, but
  // more visibilities to a counter of the plan (S 5, 1M on 1024^2: plan 117 us with
  // tiles of 12, 74 with 8, gridder 99 with either)
  T = rho < 0.25 && ((S <= 5 && !few) || (S >= 10 && S <= 13)) ? 12 : 8;
  // as many tiles as plans may have buckets: beyond (a side of 32768 with tiles of 8)
  // the lists would be gigabytes.  Within, this gridder leads however sparse (plan and
  // grid, us, warp / this one: S 8 on 32768^2, 0.9M 2494 / 774, 9M 6157 / 4329; S 16,
  // 0.45M, one visibility to ten tiles, 2813 / 768)
  if (tiles_of(p, T) > MAX_BUCKETS) return 0;
  return S <= 9 ? 16 : 24;
}

// 4-D tables of odd support, which layout_for gives to the warp layout, get the
// lane layout's 16-cell tiles under no tuning and no requested tile, for the lane
// kernel with taps by loads: not for the narrowest, nor where tiles are nearly
// empty (plan and grid, warp gridder / lane kernel, us: S 9, 123k on 1531^2: 94 / 81,
// 2M on 4096^2: 541 / 467, 400k: 172 / 168; S 7, 2M: 422 / 419, 545 / 578 fused).  On one
// grid's few visibilities any, beside the direct gridder.  Not for stacks of so many
// tiles that their numbers would run out.
static bool lane_odd(const cg_plan &p) {
  const cg_tuning t = tuning();
  const int S = p.kd.S;
  const double cells = (double)p.H * (double)p.W * (double)p.layers;
  const bool few = p.layers == 1 && direct_fits(p);  // beside the direct gridder: any
  return !p.lean && !p.kd.sep && S <= 16 && S % 2 == 1 && p.tile_req == 0 && t.tile == 0 &&
         t.layout == 0 && tiles_of(p, 16) <= MAX_BUCKETS && (few || (S >= 9 && (double)p.n >= 0.04 * cells)) &&
         (int64_t)p.kd.G * p.kd.Q * p.kd.Q < INT32_MAX;
}

static void plan_geometry(cg_plan &p) {
  if (p.mode == CG_PLAN_TILED) {
    int outer_T = 0;
    p.outer = outer_edge(p, outer_T);
    p.lane_odd = lane_odd(p);
    const bool lane = p.lane_odd || layout_for(p.kd) == CG_LAYOUT_LANE;
    const cg_tuning t = tuning();
    // few visibilities: one grid's small tiles are the register-window gridder's or
    // the lane kernel's, which take the call where a cell is crowded
    p.direct = !p.lean && t.layout == 0 && t.tile == 0 && direct_fits(p) &&
               (p.layers > 1 || p.tile_req > 0 || p.outer || lane);
    p.beside = p.direct && p.n > DIRECT_CELL_TAPS;
    // no order inside a tile (for few visibilities it is not worth its buckets)
    const bool flat = p.outer || lane || p.direct;
    p.T = p.outer ? outer_T : p.lane_odd ? 16 : tile_edge(p.kd, p.tile_req);
    // few visibilities, 4-D: tiles as small as lets a cell see two to an axis
    if (p.direct && !p.outer && p.layers == 1 && p.tile_req == 0) {
      const int T = p.kd.S <= 9 ? 8 : p.kd.S <= 13 ? 12 : 16;
      if (tiles_of(p, T) <= MAX_BUCKETS) p.T = T;
    }
    p.ntx = (p.W + p.T - 1) / p.T;
    p.nty = (p.H + p.T - 1) / p.T;
    // Morton blocks of up to 32 x 32 tiles (no larger than the grid needs)
    p.tblog = tile_block_log(p.ntx, p.nty);
    p.nbx = (p.ntx + (1 << p.tblog) - 1) >> p.tblog;
    const int nby = (p.nty + (1 << p.tblog) - 1) >> p.tblog;
    p.tpl = (p.nbx * nby) << (2 * p.tblog);
    p.ntiles = p.tpl * p.layers;
    // 4x4-cell sub-tiles, 2^sublog per tile edge (4 << full >= T), except for the
    // lane layout and the separable gridder, whose private windows need no order
    // inside a tile (tile buckets only), and few visibilities.  The sub-tile edge is 1 <<
    // subshift cells, so that an in-tile coordinate shifted by subshift is always below 2^sublog.
    int full = 0;
    while ((4 << full) < p.T) ++full;
    p.sublog = flat ? 0 : full;
    p.subshift = 2 + full - p.sublog;
    // keep the histogram (4 B per bucket) within 2^24 buckets: coarser sub-tiles
    // for very large grid stacks
    while (p.sublog > 0 && ((int64_t)p.ntiles << (2 * p.sublog)) > MAX_BUCKETS) {
      --p.sublog;
      ++p.subshift;
    }
    p.nbuckets = p.ntiles << (2 * p.sublog);
    p.win = p.T + p.kd.S - 1;
    // pitch = S (mod 16): the taps t = dy*S + dx of consecutive lanes fall on
    // consecutive 8-byte bank pairs of the window (no bank conflicts)
    p.pitch = p.win;
    while ((p.pitch - p.kd.S) % 16 != 0) ++p.pitch;
    // Visibilities per work item.  The tiled kernels take an item per CTA.  The
    // lane gridder and the separable gridder take one per warp, so that an item
    // is a chain of its visibilities' updates: short enough for a few items per
    // warp (14 lane, 24 separable warps per SM), long enough to be worth a
    // window's flush (S 16 lane gridder, 500k visibilities, 2048^2: 276 us with
    // 512, 172 with 128, 179 with 64; 50k on 1024^2: 185 against 55 with 64; 2M
    // on 4096^2: 606 with 512, 614 with 128).
    const int64_t per_warp = p.n / (int64_t)(num_sms() * (p.outer ? 64 : 28));
    auto clamp = [](int64_t v, int64_t lo, int64_t hi) {
      return (int)(std::min(hi, std::max(lo, v)) & ~(int64_t)31);
    };
    // (a lane item with taps for less than half its window's cells adds them to the grid
    // one by one, which full items of narrow supports on wide tiles must not)
    const int64_t lane_least =
        std::max<int64_t>(64, (int64_t)p.win * p.win / (2 * p.kd.S * p.kd.S) + 32);
    const int per_cta = (int)std::min<int64_t>(
        2048, std::max<int64_t>(256, p.n / (int64_t)(num_sms() * 16) + 1));
    p.chunk = t.chunk > 0 ? t.chunk
              : p.outer   ? clamp(per_warp, 32, 256)
              : lane      ? (p.lean ? 512 : clamp(per_warp, lane_least, 512))
                          : per_cta;
    p.chunk_crowded = t.chunk > 0 ? t.chunk : lane && !p.lane_odd ? 512 : per_cta;
    p.max_items = (p.n + p.chunk - 1) / p.chunk + p.ntiles;
    // The lane gridder streams each visibility's S x S slice with one bulk copy,
    // which needs a multiple of 16 bytes: for odd S * S it reads a copy of the
    // table whose slices are padded by one element (made in the workspace by
    // every gridding call).
    const int SS = p.kd.S * p.kd.S;
    p.slice_stride = SS;
    p.kpad_slices = 0;
    if (layout_for(p.kd) == CG_LAYOUT_LANE && !p.kd.sep && (SS & 1)) {
      p.slice_stride = SS + 1;
      p.kpad_slices = (int64_t)p.kd.G * p.kd.Q * p.kd.Q;
    }
  } else {
    p.T = 0;
    p.ntx = p.nty = 0;
    p.tblog = 0;
    p.nbx = 1;
    p.tpl = 1;
    p.nbuckets = p.gper * p.layers;
    p.win = p.pitch = 0;
    p.chunk = p.chunk_crowded = 0;
    p.max_items = 0;
    p.slice_stride = p.kd.sep ? p.kd.S : p.kd.S * p.kd.S;
    p.kpad_slices = 0;
  }
}

static Layout layout_of(const cg_plan &p) {
  Layout L;
  size_t o = 0;
  size_t n = (size_t)std::max<int64_t>(p.n, 1);
  L.rec_tmp = o; o = align256(o + n * sizeof(VisRec));
  L.key = o;     o = align256(o + n * 4);
  L.rank = o;    o = align256(o + n * 4);
  L.recs = o;    o = align256(o + n * sizeof(VisRec));
  L.perm = o;    o = align256(o + n * 4);
  L.ctr = o;     o = align256(o + 8 * 4);  // before the counts: zeroed with them
  L.counts = o;  o = align256(o + (size_t)p.nbuckets * 4);
  L.offsets = o; o = align256(o + (size_t)p.nbuckets * 4);
  L.scan = o;    o = align256(o + scan_scratch_words(p.nbuckets) * 4);
  L.items = o;   o = align256(o + (size_t)std::max<int64_t>(p.max_items, 1) * sizeof(WorkItem));
  const size_t nt = p.mode == CG_PLAN_TILED ? (size_t)p.ntiles : 0;  // items per tile, scanned
  L.tnch = o;    o = align256(o + nt * 4);
  L.tioff = o;   o = align256(o + nt * 4);
  L.kpad = o;    o = align256(o + (size_t)p.kpad_slices * p.slice_stride * sizeof(float2));
  L.total = o;
  return L;
}

static int check_desc(const cg_kernel_desc *kd, int H, int W) {
  CG_REQUIRE(kd, "kernel descriptor is NULL");
  CG_REQUIRE(kd->Q >= 1 && kd->S >= 1 && kd->G >= 1,
             "bad kernel descriptor Q=%d S=%d G=%d", kd->Q, kd->S, kd->G);
  CG_REQUIRE(kd->S <= 32, "support %d exceeds the supported maximum 32", kd->S);
  CG_REQUIRE(H >= 1 && W >= 1 && H <= 65536 && W <= 65536, "bad grid %dx%d", H, W);
  return CG_OK;
}

// Plan built into a caller-provided struct (no host or device allocation):
// geometry, workspace layout, coordinates + histogram, scan, scatter and (tiled
// mode) the work list.  wstep != 0 derives each visibility's kernel group
// from its w bin (round(w / wstep) - kmin, synthesis.py:793) in the same pass.
int plan_build_into(cg_plan *p, int mode, const cg_kernel_desc *kd, int H, int W,
                    const double *uvw, int64_t stride, double lam, const int32_t *kidx,
                    double wstep, int kmin, int layers, const int32_t *layer,
                    const int32_t *group, int ngroups, int64_t n, void *workspace,
                    size_t workspace_bytes, int32_t *d_status, cudaStream_t s, int tile_req = 0) {
  int rc = check_desc(kd, H, W);
  CG_REQUIRE(!group || (mode == CG_PLAN_GROUPS && ngroups >= 1),
             "launch groups need a CG_PLAN_GROUPS plan and ngroups >= 1");
  if (rc) return rc;
  CG_REQUIRE(layers >= 1 && (layers == 1 || layer || n == 0), "bad layer arguments");
  CG_REQUIRE((int64_t)layers * H * W < ((int64_t)1 << 40), "grid stack too large");
  CG_REQUIRE(mode == CG_PLAN_TILED || mode == CG_PLAN_GROUPS, "bad plan mode %d", mode);
  CG_REQUIRE(n >= 0 && n < (int64_t)INT32_MAX, "visibility count %lld unsupported",
             (long long)n);
  CG_REQUIRE(n == 0 || (uvw && stride >= (wstep != 0.0 ? 3 : 2)), "uvw is NULL or stride too small");
  CG_REQUIRE(d_status, "status block is NULL");
  CG_REQUIRE(kd->G == 1 || kidx || wstep != 0.0 || n == 0,
             "G > 1 needs per-visibility kernel indices");
  memset(p, 0, sizeof(*p));
  p->mode = mode;
  p->kd = *kd;
  p->H = H;
  p->W = W;
  p->n = n;
  p->layers = layers;
  p->gper = group ? ngroups : kd->G;
  p->tile_req = tile_req;
  plan_geometry(*p);
  CG_REQUIRE((int64_t)p->nbuckets < (int64_t)INT32_MAX / 2, "too many tiles");
  Layout L = layout_of(*p);
  if (p->mode == CG_PLAN_TILED && workspace_bytes < L.total) {  // short items and small tiles take more
    p->lean = 1;
    plan_geometry(*p);
    L = layout_of(*p);
  }
  if (!workspace || workspace_bytes < L.total)
    return set_error(CG_ERR_WORKSPACE, "plan needs %zu workspace bytes, got %zu", L.total,
                     workspace_bytes);
  char *ws = (char *)workspace;
  VisRec *rec_tmp = (VisRec *)(ws + L.rec_tmp);
  int32_t *key = (int32_t *)(ws + L.key);
  int32_t *rank = (int32_t *)(ws + L.rank);
  p->recs = (VisRec *)(ws + L.recs);
  p->perm = (int32_t *)(ws + L.perm);
  p->counts = (int32_t *)(ws + L.counts);
  p->offsets = (int32_t *)(ws + L.offsets);
  p->items = (WorkItem *)(ws + L.items);
  p->kpad = p->kpad_slices ? (float2 *)(ws + L.kpad) : nullptr;
  int32_t *ctr = (int32_t *)(ws + L.ctr);
  p->nitems = ctr;
  p->ticket = ctr + 1;
  p->split = ctr + 4;
  p->status = d_status;
  // everything later kernels accumulate into starts at zero on every call
  CG_CUDA(cudaMemsetAsync(ctr, 0, (char *)(p->counts + p->nbuckets) - (char *)ctr, s));
  if (n == 0) return CG_OK;
  CoordParams P;
  P.uvw = uvw;
  P.stride = stride;
  P.lam = lam;
  P.n = n;
  P.H = H;
  P.W = W;
  P.Q = kd->Q;
  P.S = kd->S;
  P.G = kd->G;
  P.sep = kd->sep;
  P.kidx = kidx;
  P.mode = mode;
  P.T = p->T;
  P.tblog = p->tblog;
  P.nbx = p->nbx;
  P.nbuckets = p->nbuckets;
  P.sublog = p->sublog;
  P.subshift = p->subshift;
  P.layer = layer;
  P.layers = layers;
  P.group = group;
  P.ngroups = ngroups;
  P.tpl = p->tpl;
  P.ax = axis_const(W, kd->Q, lam);
  P.ay = axis_const(H, kd->Q, lam);
  P.wstep = wstep;
  P.inv_wstep = wstep != 0.0 ? 1.0 / wstep : 0.0;
  P.kmin = kmin;
  P.nk = kd->G;
  P.rec = rec_tmp;
  P.key = key;
  P.rank = rank;
  P.hist = p->counts;
  P.status = d_status;
  const int blocks = (int)((n + 255) / 256);
  k_plan_coords<<<blocks, 256, 0, s>>>(P);
  CG_LAUNCH("coords");
  // Buckets' offsets and, tiled, the work list: one block for small grids, two
  // launches where the buckets are tiles, else the separate passes.  A plan of
  // 1000 visibilities on 256^2 took eight launches, one on 1531^2 eleven; now four
  // and five (conv_imaging + conv_predict there: 286 -> 266 us, 370 -> 340 us).
  const bool tiled = mode == CG_PLAN_TILED;
  const ItemSize size = {p->chunk, p->chunk_crowded};
  const int reach = kd->S > 1 && p->T > 0 ? (kd->S - 2) / p->T + 2 : 1;
  const Crowd crowd = {p->beside ? std::max(1, DIRECT_CELL_TAPS / (reach * reach)) : INT32_MAX,
                       reach, p->tblog, p->nbx, p->ntx, p->nty, p->tpl};
  const int scan_blocks = (p->nbuckets + SCAN_TILE - 1) / SCAN_TILE;
  if (tiled && p->nbuckets <= (p->sublog ? PLAN_SMALL_BUCKETS : PLAN_SMALL_TILES)) {
    k_plan_small<<<1, SCAN_THREADS, 0, s>>>(p->nbuckets, p->ntiles, p->sublog, p->counts, size,
                                            crowd, p->offsets, p->items, p->nitems, p->split);
    CG_LAUNCH("plan offsets and items");
  } else if (tiled && p->sublog == 0) {
    unsigned long long *sums = (unsigned long long *)(ws + L.scan);
    int32_t *tioff = (int32_t *)(ws + L.tioff);
    k_plan_scan<<<scan_blocks, SCAN_THREADS, 0, s>>>(p->nbuckets, p->counts, size, crowd,
                                                     p->offsets, tioff, sums, ctr + 3, ctr + 6,
                                                     p->nitems, p->split);
    CG_LAUNCH("plan scan");
    k_plan_finish<<<(p->nbuckets + 255) / 256, 256, 0, s>>>(p->nbuckets, p->counts, size,
                                                            p->offsets, tioff, sums, p->items);
    CG_LAUNCH("plan items");
  } else {
    rc = launch_scan(p->counts, p->offsets, p->nbuckets, (int32_t *)(ws + L.scan), s);
    if (rc) return rc;
    if (tiled) {
      int32_t *tnch = (int32_t *)(ws + L.tnch), *tioff = (int32_t *)(ws + L.tioff);
      const unsigned tb = (unsigned)((p->ntiles + 255) / 256);
      k_plan_item_counts<<<tb, 256, 0, s>>>(p->ntiles, p->sublog, p->counts, p->offsets, p->chunk,
                                            tnch);
      CG_LAUNCH("plan item counts");
      // the bucket scan's scratch is free again (ntiles <= nbuckets)
      rc = launch_scan(tnch, tioff, p->ntiles, (int32_t *)(ws + L.scan), s);
      if (rc) return rc;
      k_plan_items<<<tb, 256, 0, s>>>(p->ntiles, p->sublog, p->counts, p->offsets, p->chunk, tnch,
                                      tioff, p->items, p->nitems);
      CG_LAUNCH("plan items");
    }
  }
  k_plan_scatter<<<blocks, 256, 0, s>>>(n, rec_tmp, key, rank, p->offsets, p->recs, p->perm);
  CG_LAUNCH("plan sort");
  return CG_OK;
}

int plan_build_tiled_into(cg_plan *p, const cg_kernel_desc *kd, int H, int W,
                          const double *uvw, int64_t stride, double lam,
                          const int32_t *kidx, int64_t n, void *workspace,
                          size_t workspace_bytes, int32_t *d_status, cudaStream_t s) {
  return plan_build_into(p, CG_PLAN_TILED, kd, H, W, uvw, stride, lam, kidx, 0.0, 0, 1, nullptr,
                         nullptr, 0, n, workspace, workspace_bytes, d_status, s);
}

// The least workspace a tiled plan can be built in (cg_plan_workspace_bytes is
// what it would take of a larger one).
size_t plan_workspace_least(const cg_kernel_desc *kd, int H, int W, int64_t n) {
  if (check_desc(kd, H, W) != CG_OK) return 0;
  cg_plan p;
  memset(&p, 0, sizeof(p));
  p.mode = CG_PLAN_TILED;
  p.kd = *kd;
  p.H = H;
  p.W = W;
  p.n = n;
  p.layers = 1;
  p.gper = kd->G;
  plan_geometry(p);
  const size_t need = layout_of(p).total;
  p.lean = 1;
  plan_geometry(p);
  return std::min(need, layout_of(p).total);
}

// Heap plan; the groups form of a stack of grids also copies the group ranges to
// the host.
static int plan_create_heap(cg_plan **out, int mode, const cg_kernel_desc *kd, int H, int W,
                            const double *uvw, int64_t stride, double lam, const int32_t *kidx,
                            double wstep, int kmin, int layers, const int32_t *layer,
                            const int32_t *group, int ngroups, int64_t n, void *workspace,
                            size_t workspace_bytes, int32_t *d_status, cudaStream_t s, int tile_req = 0) {
  CG_REQUIRE(out, "plan output pointer is NULL");
  *out = nullptr;
  cg_plan *p = new (std::nothrow) cg_plan;
  CG_REQUIRE(p, "out of host memory");
  int rc = plan_build_into(p, mode, kd, H, W, uvw, stride, lam, kidx, wstep, kmin, layers, layer,
                           group, ngroups, n, workspace, workspace_bytes, d_status, s, tile_req);
  if (rc) {
    delete p;
    return rc;
  }
  if (mode == CG_PLAN_GROUPS && layers > 1) {
    p->h_counts = (int32_t *)malloc((size_t)p->nbuckets * 4);
    p->h_offsets = (int32_t *)malloc((size_t)p->nbuckets * 4);
    cudaError_t e = cudaSuccess;
    if (!p->h_counts || !p->h_offsets) {
      rc = set_error(CG_ERR_ARG, "out of host memory");
    } else if (n == 0) {
      memset(p->h_counts, 0, (size_t)p->nbuckets * 4);
      memset(p->h_offsets, 0, (size_t)p->nbuckets * 4);
    } else if ((e = cudaMemcpyAsync(p->h_counts, p->counts, (size_t)p->nbuckets * 4,
                                    cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
               (e = cudaMemcpyAsync(p->h_offsets, p->offsets, (size_t)p->nbuckets * 4,
                                    cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
               (e = cudaStreamSynchronize(s)) != cudaSuccess) {
      rc = cuda_error(e, "plan group readback");
    }
    if (rc) {
      free(p->h_counts);
      free(p->h_offsets);
      delete p;
      return rc;
    }
  }
  *out = p;
  return CG_OK;
}

}  // namespace cg

using namespace cg;

extern "C" {

size_t cg_plan_workspace_bytes(int mode, int64_t n, int H, int W,
                               const cg_kernel_desc *kd) {
  if (check_desc(kd, H, W) != CG_OK) return 0;
  cg_plan p;
  memset(&p, 0, sizeof(p));
  p.mode = mode;
  p.kd = *kd;
  p.H = H;
  p.W = W;
  p.n = n;
  p.layers = 1;
  p.gper = kd->G;
  plan_geometry(p);
  return layout_of(p).total;
}

int cg_plan_create(cg_plan **out, int mode, const cg_kernel_desc *kd, int H,
                   int W, const double *uvw, int64_t stride, double lam,
                   const int32_t *kidx, int64_t n, void *workspace,
                   size_t workspace_bytes, int32_t *d_status,
                   cg_stream_t stream) {
  return plan_create_heap(out, mode, kd, H, W, uvw, stride, lam, kidx, 0.0, 0, 1, nullptr, nullptr,
                          0, n, workspace, workspace_bytes, d_status, (cudaStream_t)stream);
}

static void opts_or_default(const cg_plan_opts *o, cg_plan_opts &r) {
  r.layers = 1;
  r.layer = nullptr;
  r.wstep = 0.0;
  r.kmin = 0;
  r.group = nullptr;
  r.ngroups = 0;
  r.tile = 0;
  if (o) r = *o;
  if (r.layers < 1) r.layers = 1;
}

size_t cg_plan_workspace_bytes_ex(int mode, int64_t n, int H, int W, const cg_kernel_desc *kd,
                                  const cg_plan_opts *opts) {
  if (check_desc(kd, H, W) != CG_OK) return 0;
  cg_plan_opts o;
  opts_or_default(opts, o);
  cg_plan p;
  memset(&p, 0, sizeof(p));
  p.mode = mode;
  p.kd = *kd;
  p.H = H;
  p.W = W;
  p.n = n;
  p.layers = o.layers;
  p.gper = o.group ? o.ngroups : kd->G;
  p.tile_req = o.tile;
  plan_geometry(p);
  return layout_of(p).total;
}

int cg_plan_create_ex(cg_plan **out, int mode, const cg_kernel_desc *kd, int H, int W,
                      const double *uvw, int64_t stride, double lam, const int32_t *kidx,
                      int64_t n, const cg_plan_opts *opts, void *workspace,
                      size_t workspace_bytes, int32_t *d_status, cg_stream_t stream) {
  cg_plan_opts o;
  opts_or_default(opts, o);
  return plan_create_heap(out, mode, kd, H, W, uvw, stride, lam, kidx, o.wstep, o.kmin, o.layers,
                          o.layer, o.group, o.ngroups, n, workspace, workspace_bytes, d_status,
                          (cudaStream_t)stream, o.tile);
}

int cg_plan_create_wbins(cg_plan **out, int mode, const cg_kernel_desc *kd, int H, int W,
                         const double *uvw, int64_t stride, double lam, double wstep, int kmin,
                         int64_t n, void *workspace, size_t workspace_bytes,
                         int32_t *d_status, cg_stream_t stream) {
  CG_REQUIRE(wstep != 0.0, "wstep must be non-zero");
  return plan_create_heap(out, mode, kd, H, W, uvw, stride, lam, nullptr, wstep, kmin, 1, nullptr,
                          nullptr, 0, n, workspace, workspace_bytes, d_status,
                          (cudaStream_t)stream);
}

int cg_plan_destroy(cg_plan *p) {
  if (p) {
    free(p->h_counts);
    free(p->h_offsets);
    delete p;
  }
  return CG_OK;
}

int cg_plan_info(const cg_plan *p, int64_t *info) {
  CG_REQUIRE(p && info, "NULL argument");
  info[0] = p->T;
  info[1] = p->max_items;
  info[2] = p->chunk;
  info[3] = p->nbuckets;
  return CG_OK;
}

int cg_plan_export(const cg_plan *p, int32_t *recs, int32_t *perm, int32_t *counts,
                   cg_stream_t stream) {
  CG_REQUIRE(p, "NULL plan");
  cudaStream_t s = (cudaStream_t)stream;
  if (recs && p->n > 0)
    CG_CUDA(cudaMemcpyAsync(recs, p->recs, (size_t)p->n * sizeof(VisRec),
                            cudaMemcpyDeviceToDevice, s));
  if (perm && p->n > 0)
    CG_CUDA(cudaMemcpyAsync(perm, p->perm, (size_t)p->n * 4, cudaMemcpyDeviceToDevice, s));
  if (counts)
    CG_CUDA(cudaMemcpyAsync(counts, p->counts, (size_t)p->nbuckets * 4, cudaMemcpyDeviceToDevice,
                            s));
  return CG_OK;
}

int cg_w_bins(const double *uvw, int64_t stride, int64_t n, double wstep, int32_t *kidx,
              int32_t *d_minmax, int32_t *h_minmax, int32_t *d_status, cg_stream_t stream) {
  CG_REQUIRE(n >= 1 && uvw && stride >= 3 && kidx && d_minmax && h_minmax && d_status,
             "bad w_bins arguments");
  CG_REQUIRE(wstep != 0.0, "wstep must be non-zero");
  cudaStream_t s = (cudaStream_t)stream;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  k_minmax_init<<<1, 1, 0, s>>>(d_minmax);
  k_w_bins<<<stride_blocks(n, 256), 256, 0, s>>>(uvw, stride, n, wstep, 1.0 / wstep, kidx,
                                                 d_minmax, d_status);
  k_w_bins_rebase<<<blocks, 256, 0, s>>>(kidx, n, d_minmax);
  CG_LAUNCH("w_bins");
  CG_CUDA(cudaMemcpyAsync(h_minmax, d_minmax, 8, cudaMemcpyDeviceToHost, s));
  CG_CUDA(cudaStreamSynchronize(s));
  return CG_OK;
}

int cg_w_bins_fixed(const double *uvw, int64_t stride, int64_t n, double wstep, int kmin,
                    int nk, int32_t *kidx, int32_t *d_status, cg_stream_t stream) {
  CG_REQUIRE(n >= 0 && (n == 0 || (uvw && stride >= 3 && kidx && d_status)) && nk >= 1,
             "bad w_bins_fixed arguments");
  CG_REQUIRE(wstep != 0.0, "wstep must be non-zero");
  if (n == 0) return CG_OK;
  k_w_bins_fixed<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      uvw, stride, n, wstep, 1.0 / wstep, kmin, nk, kidx, d_status);
  CG_LAUNCH("w_bins_fixed");
  return CG_OK;
}

int cg_uvw_ranges(const double *uvw, int64_t stride, int64_t n, double wstep, void *d_work,
                  double *h_uv, int32_t *h_w, int32_t *d_status, cg_stream_t stream) {
  CG_REQUIRE(n >= 1 && uvw && stride >= (wstep != 0.0 ? 3 : 2) && d_work && h_uv && d_status &&
                 (h_w || wstep == 0.0),
             "bad uvw_ranges arguments");
  cudaStream_t s = (cudaStream_t)stream;
  UvwRanges *d = (UvwRanges *)d_work, h;
  CG_CUDA(cudaMemsetAsync(d, 0, sizeof(h), s));
  k_uvw_ranges<<<stride_blocks(n, 256), 256, 0, s>>>(
      uvw, stride, n, wstep, wstep != 0.0 ? 1.0 / wstep : 0.0, d, d_status);
  CG_LAUNCH("uvw_ranges");
  CG_CUDA(cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, s));
  CG_CUDA(cudaStreamSynchronize(s));
  h_uv[0] = from_order_bits(~h.uv_min);
  h_uv[1] = from_order_bits(h.uv_max);
  if (wstep != 0.0) {
    h_w[0] = (int32_t)(~h.w_min ^ 0x80000000u);
    h_w[1] = (int32_t)(h.w_max ^ 0x80000000u);
  }
  return CG_OK;
}

int cg_pad_even(const void *table, int64_t nslices, int S, void *out, cg_stream_t stream) {
  CG_REQUIRE(nslices >= 0 && S >= 1 && (nslices == 0 || (table && out)), "bad pad_even arguments");
  if (nslices == 0) return CG_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>(nslices, (int64_t)num_sms() * 32);
  k_pad_even<<<blocks, 256, 0, (cudaStream_t)stream>>>((const float2 *)table, nslices, S,
                                                       (float2 *)out);
  CG_LAUNCH("pad_even");
  return CG_OK;
}

size_t cg_compact_keys_workspace_bytes(int nkeys) {
  const int nw = (std::max(nkeys, 1) + 31) / 32;
  return (3 * (size_t)nw + scan_scratch_words(nw) + 64) * 4;
}

int cg_compact_keys(const int32_t *key, int64_t n, int nkeys, int32_t *row, int32_t *key_of_row,
                    int32_t *h_nrows, void *ws, size_t ws_bytes, int32_t *d_status,
                    cg_stream_t stream) {
  CG_REQUIRE(nkeys >= 1 && h_nrows && d_status && (n == 0 || (key && row && key_of_row)),
             "bad compact_keys arguments");
  if (!ws || ws_bytes < cg_compact_keys_workspace_bytes(nkeys))
    return set_error(CG_ERR_WORKSPACE, "compact_keys needs %zu workspace bytes",
                     cg_compact_keys_workspace_bytes(nkeys));
  cudaStream_t s = (cudaStream_t)stream;
  const int nw = (nkeys + 31) / 32;
  uint32_t *bits = (uint32_t *)ws;
  int32_t *cnt = (int32_t *)(bits + nw), *wpre = cnt + nw, *scratch = wpre + nw;
  CG_CUDA(cudaMemsetAsync(bits, 0, (size_t)nw * 4, s));
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (n > 0)
    k_key_bits<<<stride_blocks(n, 256), 256, nw <= KEY_SMEM_WORDS ? (size_t)nw * 4 : 0, s>>>(
        key, n, nkeys, bits, d_status);
  k_key_popc<<<(nw + 255) / 256, 256, 0, s>>>(bits, nw, cnt);
  CG_LAUNCH("key bits");
  int rc = launch_scan(cnt, wpre, nw, scratch, s);
  if (rc) return rc;
  if (n > 0) k_key_rows<<<blocks, 256, 0, s>>>(key, n, nkeys, bits, wpre, row);
  k_key_of_row<<<(nw + 255) / 256, 256, 0, s>>>(nw, bits, wpre, key_of_row);
  CG_LAUNCH("key rows");
  int32_t last[2];
  CG_CUDA(cudaMemcpyAsync(&last[0], wpre + nw - 1, 4, cudaMemcpyDeviceToHost, s));
  CG_CUDA(cudaMemcpyAsync(&last[1], cnt + nw - 1, 4, cudaMemcpyDeviceToHost, s));
  CG_CUDA(cudaStreamSynchronize(s));
  *h_nrows = last[0] + last[1];
  return CG_OK;
}

int cg_aw_keys(const double *uvw, int64_t stride, const int32_t *a1, const int32_t *a2, int64_t n,
               int nant, double wstep, int kmin, int nbins, int32_t *key, int32_t *d_status,
               cg_stream_t stream) {
  CG_REQUIRE(nant >= 1 && nbins >= 1 && wstep != 0.0 && d_status &&
                 (n == 0 || (uvw && stride >= 3 && a1 && a2 && key)),
             "bad aw_keys arguments");
  CG_REQUIRE((int64_t)nant * nant * nbins < (int64_t)INT32_MAX, "too many AW keys");
  if (n == 0) return CG_OK;
  k_aw_keys<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      uvw, stride, a1, a2, n, nant, wstep, 1.0 / wstep, kmin, nbins, key, d_status);
  CG_LAUNCH("aw keys");
  return CG_OK;
}

int cg_row_keys(const double *uvw, int64_t stride, int64_t n, double wstep, int kmin, int nbins,
                const int32_t *cols, int ncols, const int32_t *col_min, const int32_t *col_range,
                int32_t *key, int32_t *d_status, cg_stream_t stream) {
  CG_REQUIRE(nbins >= 1 && wstep != 0.0 && d_status && ncols >= 0 && ncols <= 8 &&
                 (ncols == 0 || (col_min && col_range)) &&
                 (n == 0 || (uvw && stride >= 3 && key && (ncols == 0 || cols))),
             "bad row_keys arguments");
  RowKeyCols C;
  C.ncols = ncols;
  int64_t space = nbins;
  for (int c = 0; c < ncols; ++c) {
    CG_REQUIRE(col_range[c] >= 1, "column %d has an empty range", c);
    C.mins[c] = col_min[c];
    C.ranges[c] = col_range[c];
    space *= col_range[c];
    CG_REQUIRE(space < (int64_t)INT32_MAX, "key space of %lld keys or more is too large",
               (long long)space);
  }
  if (n == 0) return CG_OK;
  k_row_keys<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      uvw, stride, n, wstep, 1.0 / wstep, kmin, nbins, cols, C, key, d_status);
  CG_LAUNCH("row keys");
  return CG_OK;
}

int cg_frac_coords(const double *uvw, int64_t stride, double lam, int64_t n,
                   int H, int W, int Q, int32_t *x, int32_t *xf, int32_t *y,
                   int32_t *yf, int32_t *d_status, cg_stream_t stream) {
  CG_REQUIRE(Q >= 1 && H >= 1 && W >= 1, "bad frac_coords arguments");
  CG_REQUIRE(n == 0 || (uvw && x && xf && y && yf && d_status && stride >= 2),
             "NULL argument");
  if (n == 0) return CG_OK;
  k_frac_coords<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      uvw, stride, lam, n, H, W, Q, axis_const(W, Q, lam), axis_const(H, Q, lam), x, xf, y,
      yf, d_status);
  CG_LAUNCH("frac_coords");
  return CG_OK;
}

}  // extern "C"
