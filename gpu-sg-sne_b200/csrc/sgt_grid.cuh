// sgt_grid.cuh -- repulsive-term kernels: grid decision, point binning,
// scatter-to-grid (S2G), gather-from-grid (G2S) with the Z reduction.
//
// Reference semantics (CU = code/cuda/SG-tSNE-CUDA/src):
//   min shift (thrust init 100.0)          CU/Frep.cu:96-102
//   max, h-driven grid size, table lookup  CU/gradient_descend_varGrid.cu:88-92
//   scale into [0, N-3), clamp 1-FLT_EPS   CU/nuconv.cu:9-36
//   cubic Lagrange S2G / G2S               CU/gridding.cu:90-338
//   Z = sum((1+2|y|^2)Phi0 - 2 y.Phi) - n,
//   F = (y Phi0 - Phi)/Z                   CU/Frep.cu:42-80, HYB/qq.cpp:75-106
//
// B200 structure: two modes, picked per iteration by the grid decision.
//   scatter mode (T = 0): no sort.  A group of lanes per point adds the
//     point's weighted charges to one of several copies of the grid with
//     vector reductions in L2 (k_scatter), k_spec_rows sums the copies into V,
//     and k_gather gathers with the same lane groups.
//   cell mode (T = 1; large jobs on grids with many points per cell): the
//     points are counting-sorted by cell, and S2G sums each cell's points in
//     registers (k_s2g_cell).
// Every kernel reads the grid decision from SgtState, so the chain is
// graph-capturable with fixed launch shapes.
#pragma once
#include "sgt_common.cuh"
#include "sgt_grid_rules.h"

// Scatter mode: lanes that share a point.  The 4 nodes of a stencil row are
// 64 contiguous bytes (32 in 1-D), so 4 lanes per point make one row one
// request; 3-D spreads its 16 rows over 16 lanes.  100k points on 64^2 nodes:
// 22.8 us with 4 lanes per point, 37.1 us with one.
#define SGT_LPP(D) ((D) == 3 ? 16 : 4)
// Lanes per point of the gather: 4 in 3-D too.  Loads of 16 rows fly in one
// lane as well as in 16, and the stencil is worked out 4 times instead of 16.
#define SGT_GLPP 4
// Points a thread loads before it uses the first of them in the point loops
// of the binning, S2G (cell mode) and G2S kernels: these kernels are bound by
// load latency, not bandwidth, at a few warps per SM.
#define SGT_PTS_U 4

// Smallest FFT length >= need among 32, 64, 96, 128, 192, ..., 768, 1024
// (2^k and 3 * 2^k): the 3 * 2^k lengths cut the padding of grids just above
// a power of two (N = 33..48 takes 96 points per axis instead of 128).
__device__ __forceinline__ int sgt_fft_length(int need) {
  int m = 32;
  while (m < 1024) {
    if (m >= need) return m;
    if (m >= 64 && (m / 2) * 3 >= need) return (m / 2) * 3;
    m <<= 1;
  }
  return 1024;
}

// ---------------------------------------------------------------------------
// Grid decision from the stats of the coordinates that the next kernels bin.
// minv/maxv are per-dim min/max of Ynext, sums its per-dim sums; the
// coordinates actually binned are Y = Ynext - mean (mean = 0 if !centre).
// Rounding is monotone, so min/max of the rounded differences equal the
// rounded differences of min/max: the decision is the one the reference
// takes on the centred array.
// ---------------------------------------------------------------------------
template <int D>
__device__ void sgt_finalize_grid(SgtState *st, const SgtJobParams &jp,
                                  const float *minv, const float *maxv,
                                  const double *sums, bool centre) {
  float maxy = 0.0f;
  for (int k = 0; k < D; k++) {
    const float mean = centre ? (float)(sums[k] / (double)jp.n) : 0.0f;
    const float lo = __fsub_rn(minv[k], mean);
    const float hi = __fsub_rn(maxv[k], mean);
    const float mn = fminf(100.0f, lo);
    st->mean[k] = mean;
    st->miny[k] = mn;
    maxy = fmaxf(maxy, __fsub_rn(hi, mn));
  }
  if (!(maxy > 0.0f) || !isfinite(maxy)) {
    if (!isfinite(maxy)) st->error |= SGT_EFLAG_NONFINITE;
    maxy = 1.0f;  // all points coincide: any positive extent gives zero force
  }
  int n1;
  if (jp.grid_mode == 1) {
    n1 = jp.n1_fixed;
  } else {
    int ng = (int)ceilf(__fdiv_rn(maxy, jp.h));
    ng = ng < 14 ? 14 : ng;
    n1 = sgt_best_grid_size_dev(ng);
  }
  int N = n1 + 2;
  int M = sgt_fft_length(2 * N - 1);
  if (M > jp.mmax) {  // keep the grid inside the allocated FFT workspace
    st->error |= SGT_EFLAG_GRID_CLAMP;
    st->grid_clamped = 1;
    int i = 136;
    while (i > 0 && 2 * c_grid_sizes[i] - 1 > jp.mmax) i--;
    N = c_grid_sizes[i];
    n1 = N - 2;
    M = sgt_fft_length(2 * N - 1);
  }
  st->maxy = maxy;
  st->N = N;
  st->M = M;
  st->scale = (float)(unsigned)(N - 3);
  const double inv = (double)(N - 3) / (double)maxy;
  st->inv_hi = (float)inv;
  st->inv_lo = (float)(inv - (double)st->inv_hi);
  st->direct = sgt_plain_conv(D, N, M, jp.conv_max, jp.conv_work) ? 1 : 0;
  st->h_eff = __fdiv_rn(maxy, (float)(n1 - 1) - 1.1920928955078125e-7f);
  const int cells = n1 - 1;  // floor bins lie in [0, n1-2]
  long ncell = cells;
  if (D >= 2) ncell *= cells;
  if (D >= 3) ncell *= cells;
  const bool cell_mode = jp.cell_blocks > 0 && sgt_cell_mode(jp.n, ncell, jp.cell_dense);
  st->T = cell_mode ? 1 : 0;
  st->tiles_dim = cell_mode ? cells : 0;
  st->ntiles = cell_mode ? (int)ncell : 0;
  long nodes = N;
  if (D >= 2) nodes *= N;
  if (D >= 3) nodes *= N;
  st->copies =
      sgt_copies(((long)jp.n << (2 * D)) / nodes, nodes, jp.vc_nodes, jp.copy_adds, jp.copies_max);
}

// Scaled coordinate exactly as CU/nuconv.cu:9-36: (y - miny)/maxy, clamp to
// 1-FLT_EPSILON, times (N-3).  The cells are the floors of these values.
__device__ __forceinline__ float sgt_scale(float y, float miny, float maxy, float scale) {
  float v = __fdiv_rn(__fsub_rn(y, miny), maxy);
  if (v >= 1.0f) v = 1.0f - 1.1920928955078125e-7f;
  return __fmul_rn(v, scale);
}

// Grid geometry of the current iteration, read once per thread.
template <int D>
struct GridGeom {
  float miny[D], maxy, scale, inv_hi, inv_lo;
  int N, cells;
  __device__ __forceinline__ explicit GridGeom(const SgtState *st) {
#pragma unroll
    for (int k = 0; k < D; k++) miny[k] = st->miny[k];
    maxy = st->maxy;
    scale = st->scale;
    inv_hi = st->inv_hi;
    inv_lo = st->inv_lo;
    N = st->N;
    cells = N - 3;
  }
  // Cell f of coordinate y along axis k, and the point's place dd in it, in
  // cells.  The cell is the floor of the reference's rounded coordinate; the
  // place is taken from y itself with a two-term (N-3)/maxy and the rounding
  // error of the shift, so it is good to a few 2^-24 of a cell however far
  // the cell is from the origin (the rounded coordinate's error grows with
  // the cell number, 3e-6 of a cell at cell 25).
  __device__ __forceinline__ float place(float y, int k, int &f) const {
    const float fl = floorf(sgt_scale(y, miny[k], maxy, scale));
    f = (int)fl;
    const float sh = __fsub_rn(y, miny[k]);
    const float bb = __fsub_rn(sh, y);
    const float err = __fsub_rn(__fsub_rn(y, __fsub_rn(sh, bb)), __fadd_rn(miny[k], bb));
    return __fmaf_rn(sh, inv_hi, -fl) + __fmaf_rn(sh, inv_lo, __fmul_rn(err, inv_hi));
  }
};

template <int D>
__device__ __forceinline__ int sgt_cell_of(const int *f, int td) {
  int t = f[0];
  if (D >= 2) t += td * f[1];
  if (D >= 3) t += td * td * f[2];
  return t;
}

// Per-block min/max/sum of the coordinates -> partials; the last block to
// finish reduces all partials and turns them into the grid decision.  Returns
// true in thread 0 of that block.  Both reductions are trees of shuffles, in
// a fixed order: walked by one thread, 592 partials took 80 of the 84 us that
// the statistics of 100,000 points cost.
template <int D>
__device__ __forceinline__ bool block_finish_stats(int vb_, int vg_, SgtState *st,
                                                   const SgtJobParams &jp, unsigned *done,
                                                   bool centre, float *mn, float *mx, double *sm,
                                                   float4 *part_min, float4 *part_max,
                                                   double *part_sum) {
  constexpr int W = SGT_THREADS / 32;
  __shared__ float smin[W][4], smax[W][4];
  __shared__ double ssum[W][4];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  // the block's values in warp 0's lanes, lane l holding warp l's
  auto reduce = [&](float *lo, float *hi, double *s) {
#pragma unroll
    for (int k = 0; k < D; k++) {
      lo[k] = warp_min_f(lo[k]);
      hi[k] = warp_max_f(hi[k]);
      s[k] = warp_sum_d(s[k]);
      if (l == 0) { smin[w][k] = lo[k]; smax[w][k] = hi[k]; ssum[w][k] = s[k]; }
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
      for (int k = 0; k < D; k++) {
        lo[k] = l < W ? smin[l][k] : INFINITY;
        hi[k] = l < W ? smax[l][k] : -INFINITY;
        s[k] = l < W ? ssum[l][k] : 0.0;
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) {
          lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
          hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
          s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        }
      }
    }
  };
  reduce(mn, mx, sm);
  if (threadIdx.x == 0) {
    part_min[vb_] = make_float4(mn[0], D > 1 ? mn[1] : 0.f, D > 2 ? mn[2] : 0.f, 0.f);
    part_max[vb_] = make_float4(mx[0], D > 1 ? mx[1] : 0.f, D > 2 ? mx[2] : 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < D; k++) part_sum[vb_ * 4 + k] = sm[k];
    __threadfence();
    last = (atomicAdd(done, 1u) == (unsigned)vg_ - 1u);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  double s[3] = {0, 0, 0};
  for (int b = threadIdx.x; b < vg_; b += blockDim.x) {
    const float4 a = __ldcg(&part_min[b]), c = __ldcg(&part_max[b]);
    lo[0] = fminf(lo[0], a.x); hi[0] = fmaxf(hi[0], c.x);
    if (D > 1) { lo[1] = fminf(lo[1], a.y); hi[1] = fmaxf(hi[1], c.y); }
    if (D > 2) { lo[2] = fminf(lo[2], a.z); hi[2] = fmaxf(hi[2], c.z); }
#pragma unroll
    for (int k = 0; k < D; k++) s[k] += __ldcg(&part_sum[b * 4 + k]);
  }
  reduce(lo, hi, s);
  if (threadIdx.x != 0) return false;
#pragma unroll
  for (int k = 0; k < D; k++) {
    st->minv[k] = lo[k];
    st->maxv[k] = hi[k];
    st->sum[k] = s[k];
  }
  sgt_finalize_grid<D>(st, jp, lo, hi, s, centre);
  *done = 0;
  return true;
}

// ---------------------------------------------------------------------------
// init: stats of a given coordinate array (first iteration / operator mode)
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_init_stats(const typename Vec<D>::T *__restrict__ Y, int n, SgtState *st,
             SgtJobParams jp, float4 *part_min, float4 *part_max,
             double *part_sum, int centre) {
  float mn[3] = {INFINITY, INFINITY, INFINITY};
  float mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  double sm[3] = {0, 0, 0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += gridDim.x * blockDim.x) {
    const typename Vec<D>::T y = Y[i];
#pragma unroll
    for (int k = 0; k < D; k++) {
      const float v = comp<D>(y, k);
      mn[k] = fminf(mn[k], v);
      mx[k] = fmaxf(mx[k], v);
      sm[k] += (double)v;
    }
  }
  block_finish_stats<D>(blockIdx.x, gridDim.x, st, jp, &st->done_init, centre != 0, mn, mx, sm,
                        part_min, part_max, part_sum);
}

// The grid decision again, from the same statistics, by other parameters: a job
// that leaves a batch may stand in a mode that its own launches do not run.
template <int D>
__global__ void k_regrid(SgtState *st, SgtJobParams jp) {
  sgt_finalize_grid<D>(st, jp, st->minv, st->maxv, st->sum, true);
}

// ---------------------------------------------------------------------------
// bin scan (run by the last block of bin_count): cell offsets and the chunk
// work list
// ---------------------------------------------------------------------------
// exclusive scan over the threads of a block (blockDim a multiple of 32)
__device__ __forceinline__ int block_exclusive_scan(int v, int *total) {
  __shared__ int wsum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    int s = lane < nw ? wsum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    wsum[lane] = s;
  }
  __syncthreads();
  const int excl = x - v + (w > 0 ? wsum[w - 1] : 0);
  *total = wsum[nw - 1];
  __syncthreads();
  return excl;
}

// Thread t owns the cells [t per, t per + per); the counts (written by other
// blocks' atomics) are read from L2.
__device__ __forceinline__ void bin_scan_block(SgtState *st, const SgtJobParams &jp,
                                               int *__restrict__ tile_count,
                                               int *__restrict__ cursor,
                                               int4 *__restrict__ chunks, int nblk) {
  const int ntiles = st->ntiles;
  // chunk length: about two chunks per persistent S2G CTA, at least 1024
  // points (256 in 3-D, where a point costs 64 nodes)
  int chunk = (jp.n + 2 * nblk - 1) / (2 * nblk);
  chunk = ((chunk + 255) / 256) * 256;
  const int cmin = jp.chunk_min > 0 ? jp.chunk_min : (jp.d == 3 ? 256 : 1024);
  if (chunk < cmin) chunk = cmin;
  const int per = (ntiles + blockDim.x - 1) / blockDim.x;
  const int t0 = threadIdx.x * per, t1 = min(t0 + per, ntiles);
  int mysum = 0, mych = 0;
  for (int t = t0; t < t1; t++) {
    const int c = __ldcg(&tile_count[t]);
    mysum += c;
    mych += (c + chunk - 1) / chunk;
  }
  int tot_pts, tot_ch;
  int base = block_exclusive_scan(mysum, &tot_pts);
  int cbase = block_exclusive_scan(mych, &tot_ch);
  for (int t = t0; t < t1; t++) {
    const int cnt = __ldcg(&tile_count[t]);
    const int cpt = (cnt + chunk - 1) / chunk;
    cursor[t] = base;
    for (int c = 0; c < cpt; c++) {
      const int idx = cbase + c;
      if (idx < jp.chunk_cap) {
        const int len = min(chunk, cnt - c * chunk);
        chunks[idx] = make_int4(t, base + c * chunk, len, 0);
      }
    }
    base += cnt;
    cbase += cpt;
    tile_count[t] = 0;  // ready for the next iteration
  }
  if (threadIdx.x == 0) {
    st->chunk = chunk;
    if (tot_ch > jp.chunk_cap) {
      st->error |= SGT_EFLAG_CHUNK_OVERFLOW;
      tot_ch = jp.chunk_cap;
    }
    st->nchunks = tot_ch;
  }
}

// ---------------------------------------------------------------------------
// Scatter mode: centre the points and add their weighted charges to the grid
// copy vb_ mod copies.  The charges at a node are [1, y - y_node], the
// distance in cells: F and Z do not depend on the origin that y is measured
// from, and with the node's own place as origin no sum cancels (k_gather,
// k_spec_cols; the FFT passes move the origin to the grid's middle).  SGT_LPP(D) lanes share a point; lane q of
// a group owns the stencil nodes with x offset q & 3 (3-D: and y offset
// q >> 2), and every lane works out the point's weights for itself.
// Bound by the reductions L2 takes: 100k points on 64^2 nodes 10.5 us (1.6M
// 16-byte node updates), on 117^2 10.3 us, 400k on 512^2 31 us.  In the
// sorted form it took over from, a tile of the grid in shared memory took 200 to
// 420 us where clustered points met on few nodes: shared-memory float adds
// are compare-and-swap loops there.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void red_node(float2 *p, float a, float b) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void red_node(float4 *p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}
// w[q] without a dynamically indexed (local memory) array
__device__ __forceinline__ float pick4(const float *w, int q) {
  return q == 0 ? w[0] : (q == 1 ? w[1] : (q == 2 ? w[2] : w[3]));
}

template <int D>
__device__ __forceinline__ void k_scatter_body(int vb_, int vg_,
                                               const typename Vec<D>::T *__restrict__ Ynext,
                                               typename Vec<D>::T *__restrict__ Y, int n,
                                               SgtState *st, typename Node<D>::T *Vc) {
  sgt_pdl_wait();
  if (st->T != 0) return;  // cell mode
  constexpr int L = SGT_LPP(D);
  const GridGeom<D> g(st);
  const int N = g.N;
  float mean[D];
#pragma unroll
  for (int k = 0; k < D; k++) mean[k] = st->mean[k];
  long nodes = N;
  if (D >= 2) nodes *= N;
  if (D >= 3) nodes *= N;
  Vc += (long)(vb_ & (st->copies - 1)) * nodes;
  const int q = threadIdx.x % L, qx = q & 3;
  const int step = vg_ * (SGT_THREADS / L);
  for (int i = vb_ * (SGT_THREADS / L) + threadIdx.x / L; i < n; i += step) {
    typename Vec<D>::T y = Ynext[i];
    int f[3];
    float w[3][4], u[3];  // u: distance from node 0 of the stencil, in cells
    bool ok = true;
#pragma unroll
    for (int k = 0; k < D; k++) {
      const float yc = __fsub_rn(comp<D>(y, k), mean[k]);
      setcomp<D>(y, k, yc);
      const float dd = g.place(yc, k, f[k]);
      sgt_weights(dd, w[k]);
      u[k] = dd + 1.0f;
      ok = ok && (unsigned)f[k] < (unsigned)g.cells;
    }
    if (q == 0) Y[i] = y;
    if (!ok) {  // outside the grid: skip the point
      if (q == 0) atomicOr(&st->error, SGT_EFLAG_CHUNK_OVERFLOW);
      continue;
    }
    const float wx = pick4(w[0], qx), ux = u[0] - (float)qx;
    if constexpr (D == 1) {
      red_node(&Vc[f[0] + qx], wx, wx * ux);
    } else if constexpr (D == 2) {
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const float wt = w[1][b] * wx;
        red_node(&Vc[f[0] + qx + N * (f[1] + b)], wt, wt * ux, wt * (u[1] - (float)b), 0.f);
      }
    } else {
      const int qy = q >> 2;
      const float wy = pick4(w[1], qy) * wx, uy = u[1] - (float)qy;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float wt = wy * w[2][c];
        red_node(&Vc[f[0] + qx + (long)N * (f[1] + qy + (long)N * (f[2] + c))], wt, wt * ux,
                 wt * uy, wt * (u[2] - (float)c));
      }
    }
  }
}

template <int D>
__global__ void __launch_bounds__(SGT_THREADS, 8)
k_scatter(const typename Vec<D>::T *__restrict__ Ynext, typename Vec<D>::T *__restrict__ Y, int n,
          SgtState *st, typename Node<D>::T *Vc) {
  k_scatter_body<D>(blockIdx.x, gridDim.x, Ynext, Y, n, st, Vc);
}

// ---------------------------------------------------------------------------
// bin_count (cell mode): centre (Y = Ynext - mean), zero the grid V, count
// points per cell
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k_bin_count_body(int vb_, int vg_, const typename Vec<D>::T *__restrict__ Ynext,
            typename Vec<D>::T *__restrict__ Y, int n, SgtState *st,
            int *__restrict__ tile_count, typename Node<D>::T *__restrict__ V,
            const SgtJobParams &jp, int *__restrict__ cursor,
            int4 *__restrict__ chunks, int nblk) {
  sgt_pdl_wait();
  if (st->T == 0) return;  // scatter mode
  __shared__ int hist[SGT_HIST_MAX];
  const int ntiles = st->ntiles, td = st->tiles_dim, N = st->N;
  const float maxy = st->maxy, scale = st->scale;
  float mean[3], miny[3];
#pragma unroll
  for (int k = 0; k < D; k++) { mean[k] = st->mean[k]; miny[k] = st->miny[k]; }
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x) hist[t] = 0;
  // zero the grid for this iteration's S2G
  long nodes = N;
  if (D >= 2) nodes *= N;
  if (D >= 3) nodes *= N;
  typename Node<D>::T z;
  if constexpr (D == 1) z = make_float2(0.f, 0.f); else z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long g = vb_ * (long)blockDim.x + threadIdx.x; g < nodes;
       g += (long)vg_ * blockDim.x)
    V[g] = z;
  __syncthreads();
  // warp-uniform trip count: lanes with the same cell are merged with
  // match_any and add their count in one shared-memory atomic (points of an
  // embedding cluster in few cells).  A warp takes SGT_PTS_U runs of 32
  // points per round and issues all their loads before the first use.
  const int lane = threadIdx.x & 31;
  constexpr int U = SGT_PTS_U;
  const long stride = (long)vg_ * blockDim.x * U;
  for (long i0 = ((long)vb_ * blockDim.x + (threadIdx.x & ~31)) * U; i0 < n; i0 += stride) {
    typename Vec<D>::T yv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long i = i0 + 32 * u + lane;
      if (i < n) yv[u] = Ynext[i];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const long i = i0 + 32 * u + lane;
      int key = -1;
      if (i < n) {
        typename Vec<D>::T y = yv[u];
        int f[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < D; k++) {
          const float yc = __fsub_rn(comp<D>(y, k), mean[k]);
          setcomp<D>(y, k, yc);
          f[k] = (int)floorf(sgt_scale(yc, miny[k], maxy, scale));
        }
        Y[i] = y;
        key = sgt_cell_of<D>(f, td);
      }
      const unsigned grp = __match_any_sync(0xffffffffu, key);
      if (key >= 0 && lane == __ffs(grp) - 1) atomicAdd(&hist[key], __popc(grp));
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
    if (hist[t]) atomicAdd(&tile_count[t], hist[t]);
  // the last block to finish turns the cell counts into cell offsets and
  // the chunk list (no separate launch between the count and the sort)
  // (the barrier orders the block's count atomics before thread 0's
  // device-scope fence, which is cumulative over them)
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&st->done_bin, 1u) == (unsigned)vg_ - 1u;
    __threadfence();
  }
  __syncthreads();
  if (last) {
    bin_scan_block(st, jp, tile_count, cursor, chunks, nblk);
    if (threadIdx.x == 0) st->done_bin = 0;
  }
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_bin_count(const typename Vec<D>::T *__restrict__ Ynext,
            typename Vec<D>::T *__restrict__ Y, int n, SgtState *st,
            int *__restrict__ tile_count, typename Node<D>::T *__restrict__ V,
            SgtJobParams jp, int *__restrict__ cursor, int4 *__restrict__ chunks, int nblk) {
  k_bin_count_body<D>(blockIdx.x, gridDim.x, Ynext, Y, n, st, tile_count, V, jp, cursor, chunks,
                      nblk);
}

// ---------------------------------------------------------------------------
// bin_scatter: counting-sort points into cell order (cell mode).  Each CTA owns a
// contiguous range; it counts per cell, reserves its slots with one global
// atomic per touched cell, then places its points.
// sorted[p] = the point's places in its cell per axis, and its index in the .w
// bits: S2G and G2S know the cell from the chunk and need not work it out again
// (s2g and g2s of 1.3M points 29.5 + 38 us with coordinates).
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k_bin_scatter_body(int vb_, int vg_, const typename Vec<D>::T *__restrict__ Y, int n, SgtState *st,
              int *__restrict__ cursor, float4 *__restrict__ sorted) {
  sgt_pdl_wait();
  __shared__ int lc[SGT_HIST_MAX];
  if (st->T == 0) return;  // scatter mode: no sort
  const int ntiles = st->ntiles, td = st->tiles_dim;
  const GridGeom<D> gg(st);
  const float maxy = st->maxy, scale = st->scale;
  float miny[3];
#pragma unroll
  for (int k = 0; k < D; k++) miny[k] = st->miny[k];
  const int per = (n + vg_ - 1) / vg_;
  const int lo = vb_ * per, hi = min(n, lo + per);
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x) lc[t] = 0;
  __syncthreads();
  // warp-uniform trip counts; lanes of one cell are merged with match_any,
  // the group leader does the shared-memory atomic and the lanes take
  // consecutive slots in lane order.  A warp takes SGT_PTS_U runs of 32
  // points per round and issues all their loads before the first use.
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  constexpr int U = SGT_PTS_U;
  const int wstart = lo + (threadIdx.x & ~31) * U, wstep = blockDim.x * U;
  for (int i0 = wstart; i0 < hi; i0 += wstep) {
    typename Vec<D>::T yv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + 32 * u + lane;
      if (i < hi) yv[u] = Y[i];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + 32 * u + lane;
      int key = -1;
      if (i < hi) {
        int f[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < D; k++) {
          f[k] = (int)floorf(sgt_scale(comp<D>(yv[u], k), miny[k], maxy, scale));
        }
        key = sgt_cell_of<D>(f, td);
      }
      const unsigned grp = __match_any_sync(0xffffffffu, key);
      if (key >= 0 && lane == __ffs(grp) - 1) atomicAdd(&lc[key], __popc(grp));
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < ntiles; t += blockDim.x)
    if (lc[t]) lc[t] = atomicAdd(&cursor[t], lc[t]);
  __syncthreads();
  for (int i0 = wstart; i0 < hi; i0 += wstep) {
    typename Vec<D>::T yv[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + 32 * u + lane;
      if (i < hi) yv[u] = Y[i];
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int i = i0 + 32 * u + lane;
      int key = -1;
      float4 rec = make_float4(0.f, 0.f, 0.f, __int_as_float(i));
      if (i < hi) {
        int f[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < D; k++) {
          const float dd = gg.place(comp<D>(yv[u], k), k, f[k]);
          if (k == 0) rec.x = dd; else if (k == 1) rec.y = dd; else rec.z = dd;
        }
        key = sgt_cell_of<D>(f, td);
      }
      const unsigned grp = __match_any_sync(0xffffffffu, key);
      const int leader = __ffs(grp) - 1;
      int base = 0;
      if (key >= 0 && lane == leader) base = atomicAdd(&lc[key], __popc(grp));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (key >= 0) sorted[base + __popc(grp & below)] = rec;
    }
  }
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_bin_scatter(const typename Vec<D>::T *__restrict__ Y, int n, SgtState *st,
              int *__restrict__ cursor, float4 *__restrict__ sorted) {
  k_bin_scatter_body<D>(blockIdx.x, gridDim.x, Y, n, st, cursor, sorted);
}

// weights and distances from stencil node 0 (in cells) of a sorted point
template <int D>
__device__ __forceinline__ void sgt_point_stencil(const float4 &rec, float (*w)[4], float *u) {
#pragma unroll
  for (int k = 0; k < D; k++) {
    const float dd = k == 0 ? rec.x : (k == 1 ? rec.y : rec.z);
    sgt_weights(dd, w[k]);
    u[k] = dd + 1.0f;
  }
}

// ---------------------------------------------------------------------------
// S2G in cell mode (T = 1): every point of a chunk lies in the chunk's cell,
// so all of them touch the same 4^d nodes.  Each thread sums its points'
// weighted charges in registers (no shared-memory atomics), the block reduces
// once per chunk, and one global atomic per node and channel goes to V.
// d = 3 runs in four passes over the z offset of the stencil (64 sums each).
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k_s2g_cell_body(int vb_, int vg_, const float4 *__restrict__ sorted, SgtState *st,
           const int4 *__restrict__ chunks, typename Node<D>::T *__restrict__ V) {
  sgt_pdl_wait();
  if (st->T != 1) return;  // scatter mode: k_scatter did the S2G
  constexpr int NN = D == 1 ? 4 : 16;  // stencil nodes per pass
  constexpr int C = D + 1;             // charge channels
  constexpr int K = NN * C;
  constexpr int CS = D == 1 ? 2 : 4;   // floats per node of V
  constexpr int PASSES = D == 3 ? 4 : 1;
  __shared__ float red[SGT_THREADS / 32][K];
  const int td = st->tiles_dim, N = st->N, nch = st->nchunks;
  float *Vf = reinterpret_cast<float *>(V);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int c = vb_; c < nch; c += vg_) {
    const int4 ch = chunks[c];
    int cf[3] = {0, 0, 0};
    cf[0] = ch.x % td;
    if (D >= 2) cf[1] = (ch.x / td) % td;
    if (D >= 3) cf[2] = ch.x / (td * td);
#pragma unroll
    for (int pass = 0; pass < PASSES; pass++) {
      float acc[K];
#pragma unroll
      for (int q = 0; q < K; q++) acc[q] = 0.f;
      constexpr int U = SGT_PTS_U;
      const int end = ch.y + ch.z;
      for (int j0 = ch.y + threadIdx.x; j0 < end; j0 += U * blockDim.x) {
        float4 rv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int j = j0 + u * blockDim.x;
          if (j < end) rv[u] = sorted[j];
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (j0 + u * blockDim.x >= end) break;
          float w[3][4], du[3];
          sgt_point_stencil<D>(rv[u], w, du);
          // weights times distances, per axis: every sum below is one
          // multiply-add of two of them
          float wu[4];
#pragma unroll
          for (int a0 = 0; a0 < 4; a0++) wu[a0] = w[0][a0] * (du[0] - (float)a0);
          const float wz = D == 3 ? w[2][pass] : 1.f;
#pragma unroll
          for (int a1 = 0; a1 < (D >= 2 ? 4 : 1); a1++) {
            const float wy = (D >= 2 ? w[1][a1] : 1.f) * wz;
            const float wv = D >= 2 ? wy * (du[1] - (float)a1) : 0.f;
            const float ww = D >= 3 ? wy * (du[2] - (float)pass) : 0.f;
#pragma unroll
            for (int a0 = 0; a0 < 4; a0++) {
              const int nd = a1 * 4 + a0;
              acc[nd * C] += wy * w[0][a0];
              acc[nd * C + 1] += wy * wu[a0];
              if constexpr (D >= 2) acc[nd * C + 2] += wv * w[0][a0];
              if constexpr (D >= 3) acc[nd * C + 3] += ww * w[0][a0];
            }
          }
        }
      }
      {
        int base = 0;
        warp_multi_sum<K, 16>(acc, lane, base);
        constexpr int KF = wsum_count(K, 16);
        if ((lane & wsum_full_mask(K, 16)) == 0) {
#pragma unroll
          for (int q = 0; q < KF; q++) red[wid][base + q] = acc[q];
        }
      }
      __syncthreads();
      for (int q = threadIdx.x; q < K; q += blockDim.x) {
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < SGT_THREADS / 32; j++) sum += red[j][q];
        const int nd = q / C, chn = q % C;
        long g = cf[0] + (nd & 3);
        if (D >= 2) g += (long)N * (cf[1] + (nd >> 2));
        if (D >= 3) g += (long)N * N * (cf[2] + pass);
        if (sum != 0.f) atomicAdd(&Vf[g * CS + chn], sum);
      }
      __syncthreads();
    }
  }
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_s2g_cell(const float4 *__restrict__ sorted, SgtState *st,
           const int4 *__restrict__ chunks, typename Node<D>::T *__restrict__ V) {
  k_s2g_cell_body<D>(blockIdx.x, gridDim.x, sorted, st, chunks, V);
}

// Interpolated p[0] = Phi0 and p[1 + k] = y_k Phi0 - Phi_k (the repulsive
// force numerator in cells) at a point with stencil weights w, from the
// block's copy cn of the 4^d nodes of the point's cell, node a0 + 4 a1 +
// 16 a2.  o: the point's distance per axis from the origin that Phi_k is
// taken about.
template <int D>
__device__ __forceinline__ void g2s_potentials(const float (*w)[4], const float *o,
                                               const typename Node<D>::T *cn, float *p) {
#pragma unroll
  for (int a2 = 0; a2 < (D >= 3 ? 4 : 1); a2++)
#pragma unroll
    for (int a1 = 0; a1 < (D >= 2 ? 4 : 1); a1++) {
      float wy = 1.f;
      if (D >= 2) wy *= w[1][a1];
      if (D >= 3) wy *= w[2][a2];
#pragma unroll
      for (int a0 = 0; a0 < 4; a0++) {
        const float wt = wy * w[0][a0];
        const typename Node<D>::T v = cn[a0 + 4 * (a1 + 4 * a2)];
        p[0] += wt * v.x;
        p[1] += wt * v.y;
        if constexpr (D >= 2) p[2] += wt * v.z;
        if constexpr (D >= 3) p[3] += wt * v.w;
      }
    }
#pragma unroll
  for (int k = 0; k < D; k++) p[k + 1] = o[k] * p[0] - p[k + 1];
}

// Force numerator and z of a point from its p (g2s_potentials) and its
// distance m from the grid's middle in cells: z_i = Phi0 + 2 (y_i - c).F_i,
// which is (1 + 2|y|^2) Phi0 - 2 y.Phi without its cancellation.
template <int D>
__device__ __forceinline__ double point_force(const float *p, const float *m, float h,
                                              typename Vec<D>::T &fr) {
  double dot = 0.0;
  if constexpr (D == 3) fr.w = 0.f;
#pragma unroll
  for (int k = 0; k < D; k++) {
    setcomp<D>(fr, k, h * p[k + 1]);
    dot += (double)m[k] * (double)p[k + 1];
  }
  return (double)p[0] + 2.0 * (double)h * (double)h * dot;
}

// Which convolution's potentials a G2S launch gathers; the other launch of the
// iteration returns at once.
#define SGT_G2S_BOTH 0
#define SGT_G2S_SMALL 1
#define SGT_G2S_FFT 2
__device__ __forceinline__ bool g2s_skips(const SgtState *st, int after) {
  return after != SGT_G2S_BOTH && (after == SGT_G2S_SMALL) != (st->direct != 0);
}

// Z of a G2S launch: the block's FP64 partial, then the last block to finish
// sums the partials in block order and writes Z = sum - n.
__device__ __forceinline__ void g2s_finish(int vb_, int vg_, SgtState *st, double *part_z, int n,
                                           double zacc, double *wz, bool &last) {
  zacc = warp_sum_d(zacc);
  if ((threadIdx.x & 31) == 0) wz[threadIdx.x >> 5] = zacc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int k = 0; k < SGT_THREADS / 32; k++) s += wz[k];
    part_z[vb_] = s;
    __threadfence();
    last = (atomicAdd(&st->done_g2s, 1u) == vg_ - 1);
  }
  __syncthreads();
  if (last) {
    __threadfence();
    double s = 0;
    for (int b = threadIdx.x; b < (int)vg_; b += blockDim.x) s += __ldcg(&part_z[b]);
    s = warp_sum_d(s);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) wz[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0;
      for (int k = 0; k < SGT_THREADS / 32; k++) t += wz[k];
      st->Z = t - (double)n;
      st->done_g2s = 0;
    }
  }
}

// ---------------------------------------------------------------------------
// G2S + repulsive force numerator + Z (FP64, fixed-order finish).
// Frep_un[i] = y_i*Phi0 - Phi_{1..d}; Z = sum_i z_i - n.
// Scatter mode: the points in their own order, SGT_GLPP lanes per point.
// Lane q reads the nodes with x offset q (a stencil row is one 64-byte
// request) and the group sums the potentials by shuffles; its first lane
// forms F and the point's Z.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k_gather_body(int vb_, int vg_, SgtState *st,
                                              const typename Node<D>::T *__restrict__ Phi,
                                              typename Vec<D>::T *__restrict__ Frep_un,
                                              double *part_z, int n,
                                              const typename Vec<D>::T *__restrict__ Y, int after) {
  sgt_pdl_wait();
  if (st->T != 0 || g2s_skips(st, after)) return;  // cell mode: k_g2s
  __shared__ double wz[SGT_THREADS / 32];
  __shared__ bool last;
  constexpr int L = SGT_GLPP, R = D == 1 ? 1 : (D == 2 ? 4 : 16);  // stencil rows
  const GridGeom<D> g(st);
  const int N = g.N;
  const float h = st->h_eff, half = 0.5f * g.scale;
  const bool direct = st->direct != 0;
  const float loc = direct ? 1.0f : 0.0f;
  double zacc = 0.0;
  const int qx = threadIdx.x % L;
  const int step = vg_ * (SGT_THREADS / L);
  const int rounds = (n + step - 1) / step;  // uniform, so that the shuffles converge
  int i = vb_ * (SGT_THREADS / L) + threadIdx.x / L;
  for (int r = 0; r < rounds; r++, i += step) {
    float p[4] = {0.f, 0.f, 0.f, 0.f}, m[3] = {0.f, 0.f, 0.f};
    if (i < n) {
      const typename Vec<D>::T y = Y[i];
      int f[3] = {0, 0, 0};
      float w[3][4], o[3];
      bool ok = true;
#pragma unroll
      for (int k = 0; k < D; k++) {
        const float dd = g.place(comp<D>(y, k), k, f[k]);
        sgt_weights(dd, w[k]);
        m[k] = ((float)f[k] - half) + dd;
        o[k] = direct ? dd + 1.0f : m[k];
        ok = ok && (unsigned)f[k] < (unsigned)g.cells;
      }
      if (!ok) {  // outside the grid (S2G skipped it too): no force, no Z
        if (qx == 0) atomicOr(&st->error, SGT_EFLAG_CHUNK_OVERFLOW);
      } else {
        typename Node<D>::T v[R];
        const typename Node<D>::T *ph = Phi + f[0] + qx + (D >= 2 ? N * f[1] : 0) +
                                        (D >= 3 ? (long)N * N * f[2] : 0);
#pragma unroll
        for (int b = 0; b < R; b++)
          v[b] = ph[(D >= 2 ? N * (b & 3) : 0) + (D >= 3 ? N * N * (b >> 2) : 0)];
        const float wx = pick4(w[0], qx), ox = o[0] - loc * (float)qx;
#pragma unroll
        for (int b = 0; b < R; b++) {
          float wt = wx;
          if (D >= 2) wt *= w[1][b & 3];
          if (D >= 3) wt *= w[2][b >> 2];
          p[0] += wt * v[b].x;
          p[1] += wt * (ox * v[b].x - v[b].y);
          if constexpr (D >= 2) p[2] += wt * ((o[1] - loc * (float)(b & 3)) * v[b].x - v[b].z);
          if constexpr (D >= 3) p[3] += wt * ((o[2] - loc * (float)(b >> 2)) * v[b].x - v[b].w);
        }
      }
    }
#pragma unroll
    for (int e = 1; e < L; e *= 2)
#pragma unroll
      for (int k = 0; k <= D; k++) p[k] += __shfl_xor_sync(0xffffffffu, p[k], e);
    if (i < n && qx == 0) {
      typename Vec<D>::T fr;
      zacc += point_force<D>(p, m, h, fr);
      Frep_un[i] = fr;
    }
  }
  g2s_finish(vb_, vg_, st, part_z, n, zacc, wz, last);
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS, D == 3 ? 3 : 6)
k_gather(SgtState *st, const typename Node<D>::T *__restrict__ Phi,
         typename Vec<D>::T *__restrict__ Frep_un, double *part_z, int n,
         const typename Vec<D>::T *__restrict__ Y, int after) {
  k_gather_body<D>(blockIdx.x, gridDim.x, st, Phi, Frep_un, part_z, n, Y, after);
}

// Cell mode: the same over the chunks of sorted points.
template <int D>
__device__ __forceinline__ void k_g2s_body(int vb_, int vg_, const float4 *__restrict__ sorted, SgtState *st,
      const int4 *__restrict__ chunks,
      const typename Node<D>::T *__restrict__ Phi,
      typename Vec<D>::T *__restrict__ Frep_un, double *part_z, int n, int after) {
  sgt_pdl_wait();
  if (st->T == 0 || g2s_skips(st, after)) return;  // scatter mode: k_gather
  __shared__ double wz[SGT_THREADS / 32];
  __shared__ bool last;
  const int N = st->N, nch = st->nchunks;
  const float h = st->h_eff, half = 0.5f * st->scale;
  const bool direct = st->direct != 0;
  const float loc = direct ? 1.0f : 0.0f;
  double zacc = 0.0;
  // every point of a chunk reads the same 4^d nodes, which the
  // block stages once per chunk in shared memory
  constexpr int NNODES = D == 1 ? 4 : (D == 2 ? 16 : 64);
  __shared__ typename Node<D>::T cn[NNODES];
  const int td = st->tiles_dim;
  for (int c = vb_; c < nch; c += vg_) {
    const int4 ch = chunks[c];
    int cf[3] = {0, 0, 0};
    cf[0] = ch.x % td;
    if (D >= 2) cf[1] = (ch.x / td) % td;
    if (D >= 3) cf[2] = ch.x / (td * td);
    __syncthreads();  // the previous chunk's points are done with cn
    for (int e = threadIdx.x; e < NNODES; e += blockDim.x) {
      long g = cf[0] + (e & 3);
      if (D >= 2) g += (long)N * (cf[1] + ((e >> 2) & 3));
      if (D >= 3) g += (long)N * N * (cf[2] + (e >> 4));
      // the potentials about the cell's stencil node 0 (k_spec_cols leaves
      // them about each node)
      typename Node<D>::T v = Phi[g];
      v.y += loc * (float)(e & 3) * v.x;
      if constexpr (D >= 2) v.z += loc * (float)((e >> 2) & 3) * v.x;
      if constexpr (D >= 3) v.w += loc * (float)(e >> 4) * v.x;
      cn[e] = v;
    }
    __syncthreads();
    constexpr int U = SGT_PTS_U;
    const int end = ch.y + ch.z;
    for (int j0 = ch.y + threadIdx.x; j0 < end; j0 += U * blockDim.x) {
      float4 rv[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int j = j0 + u * blockDim.x;
        if (j < end) rv[u] = sorted[j];
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (j0 + u * blockDim.x >= end) break;
        const float4 rec = rv[u];
        float w[3][4], o[3], m[3];
        sgt_point_stencil<D>(rec, w, o);
#pragma unroll
        for (int k = 0; k < D; k++) {
          m[k] = ((float)cf[k] - half) + (o[k] - 1.0f);
          if (!direct) o[k] = m[k];
        }
        float p[4] = {0.f, 0.f, 0.f, 0.f};
        g2s_potentials<D>(w, o, cn, p);
        typename Vec<D>::T fr;
        zacc += point_force<D>(p, m, h, fr);
        Frep_un[__float_as_int(rec.w)] = fr;
      }
    }
  }
  g2s_finish(vb_, vg_, st, part_z, n, zacc, wz, last);
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_g2s(const float4 *__restrict__ sorted, SgtState *st,
      const int4 *__restrict__ chunks,
      const typename Node<D>::T *__restrict__ Phi,
      typename Vec<D>::T *__restrict__ Frep_un, double *part_z, int n, int after) {
  k_g2s_body<D>(blockIdx.x, gridDim.x, sorted, st, chunks, Phi, Frep_un, part_z, n, after);
}

// ---------------------------------------------------------------------------
// Exact O(n^2) repulsion, for the -f error probe (CU/compute_error.cu:8-57):
// num_i = sum_{j != i} (y_i - y_j)/(1 + |y_i - y_j|^2)^2 and
// z_i = sum_{j != i} 1/(1 + |y_i - y_j|^2).  One point per thread; the other
// points stream through shared memory in tiles of SGT_THREADS, summed in
// FP32 within a tile and in FP64 across tiles.
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_frep_exact(const typename Vec<D>::T *__restrict__ Y, int n, double *__restrict__ num,
             double *__restrict__ z) {
  __shared__ float ts[SGT_THREADS][D];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  float yi[3] = {0.f, 0.f, 0.f};
  if (i < n) {
    const typename Vec<D>::T v = Y[i];
#pragma unroll
    for (int k = 0; k < D; k++) yi[k] = comp<D>(v, k);
  }
  double an[3] = {0, 0, 0}, az = 0;
  for (int j0 = 0; j0 < n; j0 += SGT_THREADS) {
    const int j = j0 + threadIdx.x;
    if (j < n) {
      const typename Vec<D>::T v = Y[j];
#pragma unroll
      for (int k = 0; k < D; k++) ts[threadIdx.x][k] = comp<D>(v, k);
    }
    __syncthreads();
    const int m = min(SGT_THREADS, n - j0);
    float fn[3] = {0.f, 0.f, 0.f}, fz = 0.f;
    for (int t = 0; t < m; t++) {
      if (j0 + t == i) continue;
      float df[3], d2 = 0.f;
#pragma unroll
      for (int k = 0; k < D; k++) {
        df[k] = yi[k] - ts[t][k];
        d2 += df[k] * df[k];
      }
      const float q = 1.0f / (1.0f + d2);
      fz += q;
#pragma unroll
      for (int k = 0; k < D; k++) fn[k] += q * q * df[k];
    }
    az += fz;
#pragma unroll
    for (int k = 0; k < D; k++) an[k] += fn[k];
    __syncthreads();
  }
  if (i < n) {
    z[i] = az;
#pragma unroll
    for (int k = 0; k < D; k++) num[(long)i * D + k] = an[k];
  }
}
