// sgt_grid_rules.h -- which form of the repulsion a grid takes, by sizes alone.
// Plain C++: the device decides with it (sgt_finalize_grid), the host sizes
// buffers and launches with it, and a test can hold it against measurements.
#pragma once

#ifndef SGT_RULE
#ifdef __CUDACC__
#define SGT_RULE __host__ __device__ __forceinline__
#else
#define SGT_RULE inline
#endif
#endif

#define SGT_HIST_MAX 4096  // cells held in shared memory by the binning kernels

// Points from which a job can sort dense grids by cell, and the points per cell
// that make a grid dense. us per iteration, sorted / scattered, at points per
// axis: 1-D 100k 16: 43 / 49, 64: 43 / 41, 150k 16: 54 / 66, 290k 16: 84 / 111,
// 250: 85 / 82 (89 scattered by a job that can sort); 2-D 200k 16: 79 / 95, 40: 81 / 93, 56: 90 / 90, 66: 95 /
// 89, 290k 16: 105 / 126, 56: 104 / 122; 3-D 200k 16: 137 / 163, 290k 16: 167 /
// 217. A job that can sort launches four kernels more, 2 to 5 us where its grid
// is not dense, which fewer points (2-D 150k 16: 62 / 72, 40: 73 / 70) do not
// repay over a run.
SGT_RULE constexpr long sgt_cell_min_n(int d) { return d == 1 ? 100000 : 200000; }
constexpr int SGT_CELL_DENSE = 64;

// Whether n points on ncell cells are sorted, for a job that can (its cells fit
// the cell arrays, and one block reduction per chunk of a cell is cheaper than
// a reduction in L2 per point and node).
SGT_RULE bool sgt_cell_mode(long n, long ncell, int dense) {
  return ncell <= SGT_HIST_MAX && n >= (long)dense * ncell;
}

// Copies of the grid in scatter mode: one per copy_adds adds that an average
// node receives, a power of two up to copies_max that fits vc_nodes. L2
// serialises the reductions that meet on one node, so copies pay while a job has
// the GPU to itself; k_spec_rows reads and clears them all. Of a job alone: with
// 32 copies 60k points on 16^2 nodes scatter in 10.5 us instead of 76, 100k on
// 117^2 in 10.3 instead of 20.7. 3-D grids have the larger fold: us per iteration
// with 16 / 32 / 64 / 128 adds per copy, 100k points 25 points per axis: 131 / 122 /
// 121 / 129, 299k 40: 328 / 287 / 294 / 305, 48: 321 / 294 / 287 / 302, 64: 425 / 384 /
// 386 / 414; 2-D 100k 40: 56 / 55 / 60 / 62, 299k 200: 137 / 136 / 148 / 148, 20
// iterations of 100k points in COO 1255 / 1272.
constexpr int SGT_COPIES = 32;
SGT_RULE constexpr int sgt_copy_adds(int d) { return d == 3 ? 32 : 16; }
SGT_RULE int sgt_copies(long adds, long nodes, long vc_nodes, int copy_adds, int copies_max) {
  int copies = 1;
  while (copies < copies_max && (long)copy_adds * copies < adds && 2L * copies * nodes <= vc_nodes)
    copies *= 2;
  return copies;
}

// A fused launch whose jobs hold SGT_BATCH_FULL points together fills the GPU:
// what counts is the work of all jobs, not the length of one job's chain. There
// fewer copies pay (their fold is memory traffic) and large jobs sort from fewer
// points on. 64 jobs of 2,000 to 200,000 points, half 3-D, 1000 iterations: 20.4
// embeddings/s by the rules above, 22.6 with SGT_BATCH_COPY_ADDS, 21.6 with the
// sort, 25.8 with both; sorting from 10,000 to 100,000 points on, or dense from
// 16, within 1 %. us per iteration by the rules above / by these: 24 jobs of 2,000
// to 40,000 points 346 / 322 (16 points per axis), 661 / 628 (32 in 3-D); 16 of
// 100,000 to 200,000 1410 / 1078, 1857 / 1609. Below SGT_BATCH_FULL they lose: 2
// jobs of 20,000 and 50,000 99 / 118, 170 / 198.
constexpr long SGT_BATCH_FULL = 150000;
constexpr int SGT_BATCH_COPY_ADDS = 64, SGT_BATCH_COPIES = 8;
constexpr long SGT_BATCH_CELL_MIN_N = 75000;
constexpr int SGT_BATCH_CELL_DENSE = 32;

// Largest grids, in points per axis, that the plain transforms (k_spec_*) hold;
// beyond, and for 3-D grids that sgt_plain_conv leaves to them, the FFT passes.
#define SGT_SPEC_MAX(D) ((D) == 1 ? 512 : ((D) == 2 ? 128 : 80))

// 3-D: the plain transforms cost N^4, the FFT passes M^3 with M = 64, 96, 128,
// 192 for N up to 32, 48, 64, 96. The plain ones have the shorter chain, which
// counts while the chain is alone; beside a long SpMV their work counts too. us
// per iteration, plain / FFT, at N points per axis: 2,000 points 25: 46 / 54, 39:
// 86 / 104, 48: 152 / 113, 54: 180 / 165, 63: 282 / 184, 72: 489 / 640; 30,000
// points (1.5M nonzeros) 40: 123 / 130, 48: 173 / 135, 64: 348 / 201, 72: 561 /
// 640; 100,000 (5M) 25: 122 / 121, 32: 146 / 123, 40: 181 / 176, 48: 248 / 180, 56:
// 309 / 235, 66: 517 / 644, 72: 694 / 679, 78: 755 / 715; 299,000 (15M) 40: 287 /
// 300, 48: 358 / 294, 64: 593 / 384.
// In a full batch (64 jobs, grids of 20 to 48 points at the end) limits of 24,
// 32, 40, 48 and 80 points take 3220, 3191, 3097, 3090, 3076 ms.
constexpr int SGT_CONV_WORK = 16, SGT_CONV_WORK_LONG = 11, SGT_CONV_WORK_BATCH = 24;  // of 4 N^4 / M^3
SGT_RULE bool sgt_plain_conv(int d, int N, int M, int conv_max, int conv_work) {
  if (N > conv_max) return false;
  return d < 3 || 4L * N * N * N * N < (long)conv_work * M * M * M;
}
// whether some grid of up to nmax points per axis takes the FFT passes
SGT_RULE bool sgt_needs_fft(int d, int nmax, int conv_max) {
  return nmax > conv_max || (d == 3 && nmax > 28);
}
