// sgt_common.cuh -- shared device types and helpers of the SG-t-SNE engine.
//
// Data layout in HBM (per embedding):
//   Y, Ynext, uY, gains, Frep  : point-major, padded stride S = 1,2,4 for
//                                d = 1,2,3 (one 4/8/16-byte load per point)
//   P (CSR)                    : rowptr int32[n+1], pairs int2[nnz]
//                                (.x = column, .y = float bits of p_ij)
//   grids V / PhiGrid          : node-major, channels packed in one float2
//                                (d=1) or float4 (d=2,3) per node, x fastest
//   FFT workspace              : NCH complex planes of M^d float2, x fastest
// All scalars that change per iteration (grid size, h, Z, means, alpha,
// momentum) live in one device-resident SgtState so a captured CUDA graph
// replays the whole iteration without host round trips.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define SGT_MAX_GRID 512        // largest grid (points per axis) of the size table
#define SGT_FFT_LINES 8         // lines per CTA in the FFT axis passes
#define SGT_THREADS 256

// Lagrange cubic weights on 4 nodes (CU/gridding.cuh:13-22,
// HYB/gridding.cpp:29-39).  The point at place dd of cell f lies between
// nodes f+1 and f+2; node f+a gets w[a].
__device__ __forceinline__ float sgt_l1(float x) {
  return 0.5f * x * x * x - 1.0f * x * x - 0.5f * x + 1.0f;
}
__device__ __forceinline__ float sgt_l2(float x) {
  const float cc = 1.0f / 6.0f;
  return -cc * x * x * x + 1.0f * x * x - 11.0f * cc * x + 1.0f;
}
__device__ __forceinline__ void sgt_weights(float dd, float w[4]) {
  w[0] = sgt_l2(1.0f + dd);
  w[1] = sgt_l1(dd);
  w[2] = sgt_l1(1.0f - dd);
  w[3] = sgt_l2(2.0f - dd);
}

// Per-embedding device state.  Written by the last CTA of the kernel that
// produces a value, read by the kernels that follow.
struct SgtState {
  // grid of the current iteration
  float miny[4];     // per-dim min of the centred coordinates (init 100.0)
  float mean[4];     // mean subtracted from Ynext when forming Y
  float maxy;        // max shifted coordinate over all dims
  float scale;       // float(N - 3): scaled coords lie in [0, N-3)
  float inv_hi, inv_lo;  // scale / maxy in two terms
  int direct;        // 1: k_spec_* convolve this grid, 0: the FFT passes do
  float h_eff;       // grid spacing in embedding units
  int N;             // grid points per axis (n1 + 2)
  int M;             // FFT length per axis (2^k or 3 * 2^k, >= 2N-1)
  int T;             // 0: scatter mode, 1: cell mode
  int tiles_dim;     // cell mode: cells per axis and in all
  int ntiles;
  int copies;        // scatter mode: copies of the grid (a power of two)
  int nchunks;
  int chunk;         // points per chunk
  int grid_clamped;  // 1 if N was clamped to the allocated FFT size
  // reductions
  double Z;
  double sum[4];
  float minv[4], maxv[4];
  // schedule
  int iter;
  float alpha;
  float momentum;
  // counters for last-block reductions (reset by the block that finishes)
  unsigned int done_g2s;
  unsigned int done_row;
  unsigned int done_kl;
  unsigned int done_init;
  unsigned int done_bin;
  double kl;
  int error;
};

// Parameters fixed for a job (passed by value to kernels).
struct SgtJobParams {
  int n;
  int d;
  int grid_mode;      // 0: h-driven + per-iteration centring, 1: fixed grid
  int n1_fixed;       // inner grid size in fixed mode
  float h;            // target grid spacing (h mode)
  float alpha0;       // early exaggeration
  int early_iter;     // last iteration (inclusive) using alpha0
  int mom_switch;     // last iteration (inclusive) using momentum 0.5
  float eta;
  int mmax;           // largest FFT length per axis allocated
  long vc_nodes;      // nodes held by the grid copies of the scatter mode
  int cell_dense;     // points per cell from which a grid is sorted by cell
  int copy_adds;      // scatter mode: adds of an average node per copy
  int copies_max;     // scatter mode: most copies
  int chunk_cap;      // max chunks held by the chunk array
  int chunk_min;      // cell mode: fewest points per chunk (0: 1024, 256 in 3-D)
  int conv_max;       // largest N that k_spec_* convolve
  int conv_work;      // 3-D: they convolve grids of 4 N^4 / M^3 below this
  int cell_blocks;    // blocks that work in cell mode (0: no cell mode)
};

template <int D> struct Vec;
template <> struct Vec<1> { typedef float T; };
template <> struct Vec<2> { typedef float2 T; };
template <> struct Vec<3> { typedef float4 T; };

template <int D>
__device__ __forceinline__ float comp(const typename Vec<D>::T &v, int k);
template <> __device__ __forceinline__ float comp<1>(const float &v, int) { return v; }
template <> __device__ __forceinline__ float comp<2>(const float2 &v, int k) {
  return k == 0 ? v.x : v.y;
}
template <> __device__ __forceinline__ float comp<3>(const float4 &v, int k) {
  return k == 0 ? v.x : (k == 1 ? v.y : v.z);
}
template <int D>
__device__ __forceinline__ void setcomp(typename Vec<D>::T &v, int k, float x);
template <> __device__ __forceinline__ void setcomp<1>(float &v, int, float x) { v = x; }
template <> __device__ __forceinline__ void setcomp<2>(float2 &v, int k, float x) {
  if (k == 0) v.x = x; else v.y = x;
}
template <> __device__ __forceinline__ void setcomp<3>(float4 &v, int k, float x) {
  if (k == 0) v.x = x; else if (k == 1) v.y = x; else v.z = x;
}

// Grid node type: D+1 channels packed.
template <int D> struct Node { typedef float4 T; };
template <> struct Node<1> { typedef float2 T; };

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Programmatic dependent launch.  The kernels of the repulsion chain after
// the first are launched with programmatic stream serialisation, so the
// hardware stages a kernel's launch while its predecessor on the stream
// drains; every such kernel begins here, which waits until the predecessor
// has completed and its writes are visible.  Launched without the attribute
// (batches, the operator entry points, stage timing) the wait returns at once.
__device__ __forceinline__ void sgt_pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_min_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sums K per-lane values over the lanes of a warp that differ in the bits up
// to O (16: the whole warp) in K/2 + K/4 + ... shuffles instead of K per bit: at each step with offset O a lane keeps one half of
// its values, sends the other half to lane ^ O and adds what it receives; once
// the count no longer halves, the remaining offsets add whole vectors.  On
// return acc[q], q < wsum_count(K, O), of lane L holds the warp total of the
// entry values acc[base + q], with base (zero on entry) advanced by the call;
// lanes that share a base hold the same totals, and the lanes with
// (L & wsum_full_mask(K, O)) == 0 are one of each.
__host__ __device__ constexpr int wsum_count(int k, int o) {
  return o == 0 ? k : ((k % 2 == 0) ? wsum_count(k / 2, o / 2) : wsum_count(k, o / 2));
}
__host__ __device__ constexpr int wsum_full_mask(int k, int o) {
  return o == 0 ? 0 : ((k % 2 == 0) ? wsum_full_mask(k / 2, o / 2) : (o | wsum_full_mask(k, o / 2)));
}
template <int K, int O>
__device__ __forceinline__ void warp_multi_sum(float *acc, int lane, int &base) {
  if constexpr (O > 0) {
    if constexpr (K % 2 == 0) {
      constexpr int H = K / 2;
      const bool up = (lane & O) != 0;
#pragma unroll
      for (int q = 0; q < H; q++) {
        const float send = up ? acc[q] : acc[q + H];
        const float keep = up ? acc[q + H] : acc[q];
        acc[q] = keep + __shfl_xor_sync(0xffffffffu, send, O);
      }
      if (up) base += H;
      warp_multi_sum<H, O / 2>(acc, lane, base);
    } else {
#pragma unroll
      for (int q = 0; q < K; q++) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], O);
      warp_multi_sum<K, O / 2>(acc, lane, base);
    }
  }
}

// The 137-entry size table shared with the reference (CU/utils.cu:197-207).
__device__ __constant__ int c_grid_sizes[137] = {
    8,   9,   10,  11,  12,  13,  14,  15,  16,  20,  25,  26,  28,  32,  33,
    35,  36,  39,  40,  42,  44,  45,  48,  49,  50,  52,  54,  55,  56,  60,
    63,  64,  65,  66,  70,  72,  75,  77,  78,  80,  84,  88,  90,  91,  96,
    98,  99,  100, 104, 105, 108, 110, 112, 117, 120, 125, 126, 130, 132, 135,
    140, 144, 147, 150, 154, 156, 160, 165, 168, 175, 176, 180, 182, 189, 192,
    195, 196, 198, 200, 208, 210, 216, 220, 224, 225, 231, 234, 240, 245, 250,
    252, 260, 264, 270, 273, 275, 280, 288, 294, 297, 300, 308, 312, 315, 320,
    325, 330, 336, 343, 350, 351, 352, 360, 364, 375, 378, 385, 390, 392, 396,
    400, 416, 420, 432, 440, 441, 448, 450, 455, 462, 468, 480, 490, 495, 500,
    504, 512};

__device__ __forceinline__ int sgt_best_grid_size_dev(int ng) {
  int lo = 0, hi = 136;  // the first entry >= ng + 2, or the last
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (ng + 2 <= c_grid_sizes[mid]) hi = mid;
    else lo = mid + 1;
  }
  return c_grid_sizes[lo] - 2;
}

// Error bits in SgtState::error
#define SGT_EFLAG_NONFINITE 1
#define SGT_EFLAG_GRID_CLAMP 2
#define SGT_EFLAG_CHUNK_OVERFLOW 4
