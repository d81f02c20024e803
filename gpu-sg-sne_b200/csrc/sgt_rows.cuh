// sgt_rows.cuh -- attractive term, fused combine/update, KL cost.
//
// Reference semantics (CU = code/cuda/SG-tSNE-CUDA/src):
//   F_attr,i = sum_j p_ij (y_i - y_j) / (1 + |y_i - y_j|^2)
//        CU/pq.cuh:77-118 (COO), CU/hybridpq.cu:4-159 (ELL + COO),
//        HYB/pq.cpp:15-58 (CPU)
//   dY = alpha F_attr - F_rep                       CU/gradient_descend.cu:12-21
//   gains +0.2 / x0.8 (floor 0.01), uY = mu uY - eta g dY, Y += uY
//                                                   CU/gradient_descend.cu:29-44
//   per-iteration mean centring             CU/gradient_descend_varGrid.cu:41-65
//   alpha -> 1 after iteration early_iter, mu 0.5 -> 0.8 after iteration 250
//                                                   CU/gradient_descend.cu:226-233
//   KL = sum alpha p log((alpha p + FLT_MIN)/(q + FLT_MIN)), q = 1/(Z(1+d^2))
//                                                   CU/pq.cu:61-125
//
// B200 structure: the attractive SpMV streams P once per iteration (8 bytes
// per nonzero: column and value packed in an int2), a group of G lanes per
// row, neighbours' coordinates gathered as one 8/16-byte load.  It depends
// only on Y, so it runs concurrently with the latency-bound repulsion chain;
// one combine kernel (k_row_update) then applies the force combine, the
// gains/momentum update and the reductions that decide the next iteration's
// grid.  Y is double-buffered (the combine reads Y while writing Ynext).
#pragma once
#include "sgt_common.cuh"
#include "sgt_grid.cuh"

template <int D>
__device__ __forceinline__ void attr_term(const typename Vec<D>::T &yi,
                                          const typename Vec<D>::T &yj, float p,
                                          float *acc) {
  float df[3], dist = 0.f;
#pragma unroll
  for (int k = 0; k < D; k++) {
    df[k] = comp<D>(yi, k) - comp<D>(yj, k);
    dist += df[k] * df[k];
  }
  const float pq = __fdividef(p, 1.0f + dist);  // <= 2 ulp; p/(1+d^2) of the reference
#pragma unroll
  for (int k = 0; k < D; k++) acc[k] += pq * df[k];
}

template <int D, int G>
__device__ __forceinline__ void csr_row_sum(const int *__restrict__ rowptr,
                                            const int2 *__restrict__ pairs,
                                            const typename Vec<D>::T *__restrict__ Y,
                                            int i, int lane,
                                            const typename Vec<D>::T &yi,
                                            float *acc) {
  // P is streamed once per iteration: evict-first loads keep the gathered
  // coordinates resident in L2.  Four independent (column, value) loads and
  // four independent gathers per lane are in flight per step; a lane past
  // the row end gathers its own point with weight 0.
  const int s = __ldcs(&rowptr[i]), e = __ldcs(&rowptr[i + 1]);
  constexpr int U = 4;
  for (int t0 = s + lane; t0 < e; t0 += U * G) {
    int2 pr[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int t = t0 + u * G;
      pr[u] = t < e ? __ldcs(&pairs[t]) : make_int2(i, 0);
    }
    typename Vec<D>::T yj[U];
#pragma unroll
    for (int u = 0; u < U; u++) yj[u] = __ldg(&Y[pr[u].x]);
#pragma unroll
    for (int u = 0; u < U; u++) attr_term<D>(yi, yj[u], __int_as_float(pr[u].y), acc);
  }
}

// sum the partial row sums of a G-lane group (all 32 lanes must call it)
template <int D, int G>
__device__ __forceinline__ void group_reduce(float *acc) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < D; k++) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o, G);
}

__device__ __forceinline__ float sgn_f(float x) {
  return x == 0.f ? 0.f : (x < 0.f ? -1.f : 1.f);
}

// ---------------------------------------------------------------------------
// Forces and update, a point per thread: dY, gains, momentum, Ynext; the last
// block turns the per-block min/max/sum of Ynext into the next grid decision.
// Bound by memory at large n (64 n S bytes: 1.3M points in 20 us), by the
// chain of the finish at small (7 us).
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k_row_update_body(int vb_, int vg_,
             const typename Vec<D>::T *__restrict__ Fattr,
             const typename Vec<D>::T *__restrict__ Y,
             const typename Vec<D>::T *__restrict__ Frep_un,
             typename Vec<D>::T *__restrict__ uY,
             typename Vec<D>::T *__restrict__ gains,
             typename Vec<D>::T *__restrict__ Ynext, SgtState *st,
             const SgtJobParams &jp, float4 *part_min, float4 *part_max,
             double *part_sum) {
  const int n = jp.n;
  const int iter = st->iter;
  const float alpha = iter <= jp.early_iter ? jp.alpha0 : 1.0f;
  const float mom = iter <= jp.mom_switch ? 0.5f : 0.8f;
  const float eta = jp.eta;
  const float Zf = (float)st->Z;
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  double sm[3] = {0, 0, 0};
  for (int i = vb_ * blockDim.x + threadIdx.x; i < n; i += vg_ * blockDim.x) {
    const typename Vec<D>::T yi = Y[i], fa = Fattr[i], fr = __ldcs(&Frep_un[i]);
    typename Vec<D>::T u = __ldcs(&uY[i]), g = __ldcs(&gains[i]), yn = yi;
#pragma unroll
    for (int k = 0; k < D; k++) {
      const float frep = comp<D>(fr, k) / Zf;
      const float dy = alpha * comp<D>(fa, k) - frep;
      float gk = comp<D>(g, k), uk = comp<D>(u, k);
      gk = (sgn_f(dy) != sgn_f(uk)) ? (float)((double)gk + 0.2) : (float)((double)gk * 0.8);
      if ((double)gk < 0.01) gk = (float)0.01;
      uk = mom * uk - eta * gk * dy;
      const float y = comp<D>(yi, k) + uk;
      setcomp<D>(g, k, gk);
      setcomp<D>(u, k, uk);
      setcomp<D>(yn, k, y);
      mn[k] = fminf(mn[k], y);
      mx[k] = fmaxf(mx[k], y);
      sm[k] += (double)y;
    }
    if constexpr (D == 3) { u.w = 0.f; g.w = 0.f; yn.w = 0.f; }
    __stcs(&uY[i], u);
    __stcs(&gains[i], g);
    Ynext[i] = yn;
  }
  if (block_finish_stats<D>(vb_, vg_, st, jp, &st->done_row, true, mn, mx, sm, part_min, part_max,
                            part_sum)) {
#pragma unroll
    for (int k = 0; k < D; k++)
      if (!isfinite(st->minv[k]) || !isfinite(st->maxv[k])) st->error |= SGT_EFLAG_NONFINITE;
    st->alpha = alpha;
    st->momentum = mom;
    st->iter = iter + 1;
  }
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_row_update(const typename Vec<D>::T *__restrict__ Fattr,
             const typename Vec<D>::T *__restrict__ Y,
             const typename Vec<D>::T *__restrict__ Frep_un,
             typename Vec<D>::T *__restrict__ uY,
             typename Vec<D>::T *__restrict__ gains,
             typename Vec<D>::T *__restrict__ Ynext, SgtState *st,
             SgtJobParams jp, float4 *part_min, float4 *part_max,
             double *part_sum) {
  k_row_update_body<D>(blockIdx.x, gridDim.x, Fattr, Y, Frep_un, uY, gains, Ynext, st, jp,
                       part_min, part_max, part_sum);
}


// ---------------------------------------------------------------------------
// Attractive term of the CSR path: one row per G-lane group, launched over
// all rows (ceil(n G / 256) blocks; the hardware refills SMs as blocks
// retire, so a long row delays one group, not a persistent warp).  Kept lean
// (no loop state across rows) so 48+ warps stay resident per SM.  It reads
// only Y and P, so the iteration runs it as a graph branch beside the
// repulsion chain; k_row_update combines the two forces.  Row i is point
// row0 + i of Y (a shard of a row-split embedding holds rows row0.. of P
// with global column indices and gathers from the whole Y).
// ---------------------------------------------------------------------------
template <int D, int G>
__device__ __forceinline__ void k_attr_rows_body(int vb_, int vg_, const int *__restrict__ rowptr, const int2 *__restrict__ pairs,
            const typename Vec<D>::T *__restrict__ Y, typename Vec<D>::T *__restrict__ Fattr,
            int n, int row0) {
  const int lane = threadIdx.x % G;
  const int i = (vb_ * blockDim.x + threadIdx.x) / G;
  const bool valid = i < n;
  float acc[3] = {0.f, 0.f, 0.f};
  if (valid) {
    const typename Vec<D>::T yi = Y[row0 + i];
    csr_row_sum<D, G>(rowptr, pairs, Y, i, lane, yi, acc);
  }
  group_reduce<D, G>(acc);
  if (valid && lane == 0) {
    typename Vec<D>::T f;
    if constexpr (D == 3) f.w = 0.f;
#pragma unroll
    for (int k = 0; k < D; k++) setcomp<D>(f, k, acc[k]);
    Fattr[i] = f;
  }
}
template <int D, int G>
__global__ void __launch_bounds__(SGT_THREADS, (D == 3 ? 6 : 8))
k_attr_rows(const int *__restrict__ rowptr, const int2 *__restrict__ pairs,
            const typename Vec<D>::T *__restrict__ Y, typename Vec<D>::T *__restrict__ Fattr,
            int n, int row0) {
  k_attr_rows_body<D, G>(blockIdx.x, gridDim.x, rowptr, pairs, Y, Fattr, n, row0);
}

// ---------------------------------------------------------------------------
// Attractive term only (operator entry points and the COO/ELL formats).
// ---------------------------------------------------------------------------
template <int D, int G>
__global__ void __launch_bounds__(SGT_THREADS)
k_attr_csr(const int *__restrict__ rowptr, const int2 *__restrict__ pairs,
           const typename Vec<D>::T *__restrict__ Y, typename Vec<D>::T *__restrict__ F,
           int n) {
  const int lane = threadIdx.x % G;
  const int ngrp = gridDim.x * blockDim.x / G;
  const int grp0 = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  // uniform trip count per warp so the group shuffles stay converged
  const int rounds = (n + ngrp - 1) / ngrp;
  for (int r = 0; r < rounds; r++) {
    const int i = grp0 + r * ngrp;
    float acc[3] = {0.f, 0.f, 0.f};
    if (i < n) {
      const typename Vec<D>::T yi = Y[i];
      csr_row_sum<D, G>(rowptr, pairs, Y, i, lane, yi, acc);
    }
    group_reduce<D, G>(acc);
    if (i < n && lane == 0) {
      typename Vec<D>::T f;
      if constexpr (D == 3) f.w = 0.f;
#pragma unroll
      for (int k = 0; k < D; k++) setcomp<D>(f, k, acc[k]);
      F[i] = f;
    }
  }
}

// ELL part, column-major slots (CU/hybridpq.cu:4-70): one thread per row,
// overwrites F.
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_attr_ell(int n, int W, const unsigned *__restrict__ cols,
           const float *__restrict__ vals, const typename Vec<D>::T *__restrict__ Y,
           typename Vec<D>::T *__restrict__ F) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const typename Vec<D>::T yi = Y[i];
    float acc[3] = {0.f, 0.f, 0.f};
    // 4 slots of the row in flight at a time
    int k = 0;
    for (; k + 4 <= W; k += 4) {
      unsigned c[4];
      float v[4];
      typename Vec<D>::T yj[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        c[q] = __ldcs(&cols[(long)(k + q) * n + i]);
        v[q] = __ldcs(&vals[(long)(k + q) * n + i]);
      }
#pragma unroll
      for (int q = 0; q < 4; q++) yj[q] = __ldg(&Y[c[q]]);
#pragma unroll
      for (int q = 0; q < 4; q++) attr_term<D>(yi, yj[q], v[q], acc);
    }
    for (; k < W; k++) {
      const long s = (long)k * n + i;
      attr_term<D>(yi, __ldg(&Y[__ldg(&cols[s])]), __ldg(&vals[s]), acc);
    }
    typename Vec<D>::T f;
    if constexpr (D == 3) f.w = 0.f;
#pragma unroll
    for (int k = 0; k < D; k++) setcomp<D>(f, k, acc[k]);
    F[i] = f;
  }
}

// COO (rows sorted, CU/pq.cuh:77-118 and the hybrid tail CU/hybridpq.cu:71-113):
// 4 consecutive elements per lane (16-byte loads where the arrays allow them),
// summed while their row lasts; runs that end inside a lane go to F at once,
// the lanes' last runs through a warp segmented sum by row, one atomic per
// segment.  Bound by the gathers of Y: an element per lane spent 25 shuffles
// on each, 45 us for the 5M elements of 100,000 rows.
// F must hold the ELL result or zero.
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_attr_coo(long nnz, const unsigned *__restrict__ rows, const unsigned *__restrict__ cols,
           const float *__restrict__ vals, const typename Vec<D>::T *__restrict__ Y,
           float *__restrict__ F /* Vec<D> viewed as floats */) {
  constexpr int S = D == 3 ? 4 : D;
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * blockDim.x / 32;
  const bool wide = ((reinterpret_cast<size_t>(rows) | reinterpret_cast<size_t>(cols) |
                      reinterpret_cast<size_t>(vals)) & 15) == 0;
  for (long base = ((long)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 128; base < nnz;
       base += warps * 128) {
    const long e = base + 4 * lane;
    unsigned r[4], c[4];
    float v[4];
    if (wide && e + 4 <= nnz) {
      const uint4 r4 = __ldcs(reinterpret_cast<const uint4 *>(rows + e));
      const uint4 c4 = __ldcs(reinterpret_cast<const uint4 *>(cols + e));
      const float4 v4 = __ldcs(reinterpret_cast<const float4 *>(vals + e));
      r[0] = r4.x; r[1] = r4.y; r[2] = r4.z; r[3] = r4.w;
      c[0] = c4.x; c[1] = c4.y; c[2] = c4.z; c[3] = c4.w;
      v[0] = v4.x; v[1] = v4.y; v[2] = v4.z; v[3] = v4.w;
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const bool ok = e + q < nnz;
        r[q] = ok ? __ldg(&rows[e + q]) : 0xffffffffu;
        c[q] = ok ? __ldg(&cols[e + q]) : 0u;
        v[q] = ok ? __ldg(&vals[e + q]) : 0.f;
      }
    }
    typename Vec<D>::T yj[4];
#pragma unroll
    for (int q = 0; q < 4; q++) yj[q] = __ldg(&Y[c[q]]);
    unsigned cur = r[0];
    float acc[3] = {0.f, 0.f, 0.f};
    typename Vec<D>::T yi = __ldg(&Y[cur == 0xffffffffu ? 0u : cur]);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (r[q] != cur) {
#pragma unroll
        for (int k = 0; k < D; k++) atomicAdd(&F[(long)cur * S + k], acc[k]);
#pragma unroll
        for (int k = 0; k < 3; k++) acc[k] = 0.f;
        cur = r[q];
        if (cur != 0xffffffffu) yi = __ldg(&Y[cur]);
      }
      if (cur != 0xffffffffu) attr_term<D>(yi, yj[q], v[q], acc);
    }
    // segmented inclusive scan of the last runs (rows do not decrease along
    // the warp, so a lane whose last run continues its predecessor's holds
    // nothing else)
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned ro = __shfl_up_sync(0xffffffffu, cur, o);
#pragma unroll
      for (int k = 0; k < D; k++) {
        const float a = __shfl_up_sync(0xffffffffu, acc[k], o);
        if (lane >= o && ro == cur) acc[k] += a;
      }
    }
    const unsigned rn = __shfl_down_sync(0xffffffffu, cur, 1);
    // the next lane may begin with this row and end with another: its first
    // run has gone to F by itself
    if (cur != 0xffffffffu && (lane == 31 || rn != cur)) {
#pragma unroll
      for (int k = 0; k < D; k++) atomicAdd(&F[(long)cur * S + k], acc[k]);
    }
  }
}

// ---------------------------------------------------------------------------
// KL divergence (FP64 terms and sum; fixed-order finish in the last CTA)
// ---------------------------------------------------------------------------
template <int D, int G>
__global__ void __launch_bounds__(SGT_THREADS)
k_kl(const int *__restrict__ rowptr, const int2 *__restrict__ pairs,
     const typename Vec<D>::T *__restrict__ Y, SgtState *st, double alpha,
     double *part, int n) {
  __shared__ double ws[SGT_THREADS / 32];
  __shared__ bool last;
  const double Z = st->Z;
  const int lane = threadIdx.x % G;
  const int ngrp = gridDim.x * blockDim.x / G;
  double acc = 0.0;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) / G; i < n; i += ngrp) {
    const typename Vec<D>::T yi = Y[i];
    for (int t = rowptr[i] + lane; t < rowptr[i + 1]; t += G) {
      const int2 pr = pairs[t];
      const typename Vec<D>::T yj = Y[pr.x];
      double dist = 0;
#pragma unroll
      for (int k = 0; k < D; k++) {
        const double df = (double)comp<D>(yi, k) - (double)comp<D>(yj, k);
        dist += df * df;
      }
      const double p = alpha * (double)__int_as_float(pr.y);
      const double q = (1.0 / (1.0 + dist)) / Z;
      const double fmin = 1.17549435082228750797e-38;
      acc += p * log((p + fmin) / (q + fmin));
    }
  }
  acc = warp_sum_d(acc);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int k = 0; k < SGT_THREADS / 32; k++) s += ws[k];
    part[blockIdx.x] = s;
    __threadfence();
    last = (atomicAdd(&st->done_kl, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    double s = 0;
    for (int b = 0; b < (int)gridDim.x; b++) s += __ldcg(&part[b]);
    st->kl = s;
    st->done_kl = 0;
  }
}

// ---------------------------------------------------------------------------
// layout conversion between the caller's arrays and the padded point-major
// layout.  dim_major: src[i + k*n]; otherwise src[i*d + k].
// ---------------------------------------------------------------------------
template <int D>
__global__ void k_pack(const float *__restrict__ src, int n, int dim_major,
                       typename Vec<D>::T *__restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    typename Vec<D>::T v;
    if constexpr (D == 3) v.w = 0.f;
#pragma unroll
    for (int k = 0; k < D; k++)
      setcomp<D>(v, k, dim_major ? src[i + (long)k * n] : src[(long)i * D + k]);
    dst[i] = v;
  }
}
template <int D>
__global__ void k_unpack(const typename Vec<D>::T *__restrict__ src, int n,
                         int dim_major, float scale, const float *__restrict__ shift,
                         float *__restrict__ dst) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const typename Vec<D>::T v = src[i];
#pragma unroll
    for (int k = 0; k < D; k++) {
      float x = comp<D>(v, k);
      if (shift) x = x - shift[k];
      x = x * scale;
      if (dim_major) dst[i + (long)k * n] = x; else dst[(long)i * D + k] = x;
    }
  }
}

// dst[r] = src[perm[r]] (user order -> engine order), Vec<D> arrays
template <int D>
__global__ void k_permute_vec(const typename Vec<D>::T *__restrict__ src,
                              const int *__restrict__ perm, int n,
                              typename Vec<D>::T *__restrict__ dst) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
    dst[r] = src[perm[r]];
}

