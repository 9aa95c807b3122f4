// FP32 gridder of separable tables on one grid (convgrid, crocodile/synthesis.py:
// 464-481): rank-1 updates of a window held in registers.
//
// A visibility adds v ky kx^T to the grid.  One warp takes a work item
// (visibilities of one T x T tile) and owns the E x E window (E >= T + S - 1,
// 16 or 24) that their footprints can reach, a few cells per lane.  Per
// visibility it needs the two factors over the window's edge, zero outside the
// footprint: a batch of them is laid out in shared memory (one table load per
// entry, the column factor times v), then every lane multiplies its rows'
// entries by its columns' into its accumulators.  No read-modify-write of a
// window, no atomics but the flush, no order between visibilities: what bounds
// it is instruction issue, E^2 / 32 complex multiply-adds per lane and
// visibility beside the layout of the factors, whatever the support (81 warp
// instructions per visibility at E 16, 2.65 a clock).  The products with zeros
// are the price (S 8: 64 of 256 cells used), and still cheaper than a
// shared-memory float atomic or a dependent read-modify-write per tap.
//
// 1M visibilities, 2048^2: S 8 175 -> 124 us (window with shared-memory atomics
// before), S 13 468 -> 216, S 16 551 -> 231; 200k on 1024^2, S 8: 54 -> 36.
// Measured slower: packed FP32 multiply-adds on duplicated factors (148 us at S
// 8: half the FMA instructions, but four-word broadcasts filled the shared-memory
// pipe), and places and values broadcast by shuffles instead of from shared
// memory (136).
//
// The records, then the values, of the next batch are loaded while this one is
// worked on, and items are taken in turn (item w, w + warps, ...), so the next
// one is known ahead.
#include <algorithm>

#include "tiled.cuh"

namespace cg {

static constexpr int OUTER_THREADS = 256;

template <int E>
struct OuterShape;
template <>
struct OuterShape<16> {
  static constexpr int LX = 16, CX = 1, RY = 8;  // lanes along x, columns and rows per lane
  static constexpr int BATCH = 16;               // visibilities laid out at a time
};
template <>
struct OuterShape<24> {
  static constexpr int LX = 8, CX = 3, RY = 6;
  static constexpr int BATCH = 16;
};

// mode 0: vis, 1: vis * weight, 2: weight, 3: vis - sub (the residual of a
// fused pass).
struct OuterArgs {
  const float2 *ktab, *vis, *sub;
  const float *weight;
  float2 *grid;
  int mode;
};

// A warp's shared memory: the factors of a batch (rows, then columns), and 32
// visibilities' places, table rows and values.
template <int E>
struct __align__(16) OuterWarp {
  float2 fac[OuterShape<E>::BATCH][2 * E];
  int4 place[32];  // window offset y, x, row of the row factor, of the column factor
  float2 value[32];
};

template <int E>
__global__ void __launch_bounds__(OUTER_THREADS) k_grid_outer(TiledArgs A, OuterArgs O) {
  using Sh = OuterShape<E>;
  constexpr int LX = Sh::LX, CX = Sh::CX, RY = Sh::RY, BATCH = Sh::BATCH;
  static_assert(CX * LX == E && RY * (32 / LX) == E, "the lanes cover the window");
  extern __shared__ __align__(16) unsigned char smem[];
  if (status_failed(A.status)) return;
  const int lane = threadIdx.x & 31, S = A.S;
  OuterWarp<E> &sw = ((OuterWarp<E> *)smem)[threadIdx.x >> 5];
  const int lx = lane % LX, ly = lane / LX * RY;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int nitems = *A.nitems;
  if (gw >= nitems) return;
  const WorkItem none = {0, 0, 0, 0};
  auto item = [&](int64_t it) { return it < nitems ? A.items[it] : none; };
  auto value = [&](int src) {
    if (O.mode == 2) return make_float2(O.weight[src], 0.f);
    float2 v = O.vis[src];
    if (O.mode == 1) {
      const float wt = O.weight[src];
      v.x *= wt;
      v.y *= wt;
    }
    if (O.mode == 3) {
      const float2 s = O.sub[src];
      v.x -= s.x;
      v.y -= s.y;
    }
    return v;
  };
  float2 acc[RY][CX];
#pragma unroll
  for (int r = 0; r < RY; ++r)
#pragma unroll
    for (int c = 0; c < CX; ++c) acc[r][c] = make_float2(0.f, 0.f);

  int64_t it = gw;
  WorkItem w = item(it), wn = item(it + nw);
  VisRec rec = {0, 0, 0, 0};
  float2 v = make_float2(0.f, 0.f);
  if (lane < w.count) {
    rec = A.recs[w.start + lane];
    v = value(A.perm[w.start + lane]);
  }
  for (int b = 0;;) {
    const TileOrigin org = tile_origin(A, w.tile);
    const int nb = min(32, w.count - b);
    // the next batch's records
    const bool same = b + 32 < w.count;
    const int nstart = same ? w.start + b + 32 : wn.start;
    const bool nlive = lane < (same ? w.count - b - 32 : wn.count);
    VisRec nrec = {0, 0, 0, 0};
    int nsrc = 0;
    if (nlive) {
      nrec = A.recs[nstart + lane];
      nsrc = A.perm[nstart + lane];
    }
    sw.place[lane] = make_int4(rec.y0 - org.wy0, rec.x0 - org.wx0, rec.k0 * S, rec.k1 * S);
    sw.value[lane] = v;
    __syncwarp();
    for (int h = 0; h < nb; h += BATCH) {
      const int m = min(BATCH, nb - h);
#pragma unroll 4
      for (int j = 0; j < m; ++j) {
        const int4 pl = sw.place[h + j];
        const float2 u = sw.value[h + j];
#pragma unroll
        for (int e = lane; e < 2 * E; e += 32) {
          const bool column = e >= E;
          const int t = column ? e - E - pl.y : e - pl.x;
          float2 f = make_float2(0.f, 0.f);
          if ((unsigned)t < (unsigned)S) f = __ldg(&O.ktab[(column ? pl.w : pl.z) + t]);
          sw.fac[j][e] = column ? cmul(f, u) : f;
        }
      }
      __syncwarp();
#pragma unroll 4
      for (int j = 0; j < m; ++j) {
        float2 x[CX];
#pragma unroll
        for (int c = 0; c < CX; ++c) x[c] = sw.fac[j][E + lx + LX * c];
#pragma unroll
        for (int r = 0; r < RY; r += 2) {
          const float4 y = *(const float4 *)&sw.fac[j][ly + r];
#pragma unroll
          for (int c = 0; c < CX; ++c) {
            cfma(acc[r][c], make_float2(y.x, y.y), x[c]);
            cfma(acc[r + 1][c], make_float2(y.z, y.w), x[c]);
          }
        }
      }
      __syncwarp();
    }
    rec = nrec;
    if (nlive) v = value(nsrc);
    if (same) {
      b += 32;
      continue;
    }
    bool finite = true;
#pragma unroll
    for (int r = 0; r < RY; ++r)
#pragma unroll
      for (int c = 0; c < CX; ++c)
        finite = finite && fabsf(acc[r][c].x) < INFINITY && fabsf(acc[r][c].y) < INFINITY;
    if (__all_sync(0xffffffffu, finite)) {
#pragma unroll
      for (int r = 0; r < RY; ++r)
#pragma unroll
        for (int c = 0; c < CX; ++c) {
          const float2 a = acc[r][c];
          const int gy = org.wy0 + ly + r, gx = org.wx0 + lx + LX * c;
          if ((a.x != 0.f || a.y != 0.f) && gy < A.H && gx < A.W)
            atomicAdd(&O.grid[org.layer_off + (size_t)gy * A.W + gx], a);
        }
    } else {
      // a NaN or infinity, which the zeros around a footprint would spread over
      // the window: this item's taps one by one
      for (int j = 0; j < w.count; ++j) {
        const VisRec q = A.recs[w.start + j];
        const float2 u = value(A.perm[w.start + j]);
        for (int t = lane; t < S * S; t += 32) {
          const int dy = t / S, dx = t - dy * S;
          const float2 f = cmul(O.ktab[q.k0 * S + dy], O.ktab[q.k1 * S + dx]);
          atomicAdd(&O.grid[org.layer_off + (size_t)(q.y0 + dy) * A.W + q.x0 + dx], cmul(f, u));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RY; ++r)
#pragma unroll
      for (int c = 0; c < CX; ++c) acc[r][c] = make_float2(0.f, 0.f);
    it += nw;
    if (it >= nitems) return;
    w = wn;
    wn = item(it + nw);
    b = 0;
  }
}

int outer_launch(const cg_plan *p, const float2 *ktab, const float2 *vis, const float2 *sub,
                 const float *weight, int mode, float2 *grid, cudaStream_t s) {
  void (*fn)(TiledArgs, OuterArgs) = p->outer == 16 ? k_grid_outer<16> : k_grid_outer<24>;
  const int warps = OUTER_THREADS / 32;
  const size_t smem = warps * (p->outer == 16 ? sizeof(OuterWarp<16>) : sizeof(OuterWarp<24>));
  CG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  CG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, OUTER_THREADS, smem));
  CG_REQUIRE(per_sm > 0, "separable gridder does not fit on an SM");
  const int64_t blocks = std::max<int64_t>(
      1, std::min<int64_t>((int64_t)per_sm * num_sms(), (p->max_items + warps - 1) / warps));
  const OuterArgs O = {ktab, vis, sub, weight, grid, mode};
  fn<<<(unsigned)blocks, OUTER_THREADS, smem, s>>>(tiled_args(p), O);
  CG_LAUNCH("separable grid");
  return CG_OK;
}

}  // namespace cg
