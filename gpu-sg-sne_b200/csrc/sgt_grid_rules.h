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
SGT_RULE bool sgt_cell_mode(long n, long ncell) {
  return ncell <= SGT_HIST_MAX && n >= (long)SGT_CELL_DENSE * ncell;
}
