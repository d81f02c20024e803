// sgt_fft.cuh -- grid-to-grid (G2G) step: aperiodic convolution of the
// charge grids with K(r) = (1 + h^2 |r|^2)^-2.
//
// The reference computes it as 2^d half-shifted size-N cyclic convolutions
// with cuFFT (CU/non_periodic_convF.cu:14-517, HYB/non_periodic_conv.cpp);
// the sum of those terms is exactly the aperiodic convolution.  Here the
// same convolution is one cyclic convolution of length M >= 2N-1 per axis
// (the smallest M = 2^k or 3 * 2^k): output nodes x < N only meet kernel
// offsets |x - x'| <= N-1 <= M/2, so K_c[r] = K(min(r, M-r)) reproduces it.
// Two real charge channels ride in one complex plane (K_c is real and even,
// so its transform is real and the channels separate after the inverse).
// Grids that sgt_plain_conv picks take plain transforms of length 2N instead (the
// k_spec kernels further down).
//
// FFTs are register-resident: one warp owns one line of M <= 1024 points, a
// lane holds the E = M/32 points lane + 32 e; butterflies whose span holds
// whole lanes (and the radix-3 stage of M = 3 * 2^k) stay inside a lane,
// shorter spans use warp shuffles.  Forward transforms are decimation in
// frequency (natural order in, digit-reversed out) and inverse transforms
// decimation in time (digit-reversed in, natural out), so spectra stay in
// that order in memory and no permutation pass exists.  Rows
// are read and written directly (coalesced); columns go through a shared
// memory transpose of 8 adjacent columns so every global access is a 64-byte
// segment.  Planes of zero charge (index >= N) are never stored or read.
// Kernels are persistent and size their work from the device-side grid
// decision, so the chain replays inside a CUDA graph as N changes.
#pragma once
#include "sgt_common.cuh"
#include "sgt_grid_rules.h"

#define SGT_FFT_COLS 8  // columns per CTA in column passes (one per warp)
#define SGT_FFT_PAD 1   // float2 padding per staged column
#define SGT_FFT_MAXM 1024  // longest FFT: twiddle tables hold M entries

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 shfl_x2(float2 v, int m) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// tw[j] = exp(-2 pi i j / M), j < M (accurate sincospi)
__device__ __forceinline__ void fft_twiddles(float2 *tw, int M) {
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    float s, c;
    sincospif(2.0f * (float)j / (float)M, &s, &c);
    tw[j] = make_float2(c, -s);
  }
}

// FFT lengths: 2^k or 3 * 2^k, 32 <= M <= 1024.  A lane holds E = M/32
// points, lane + 32 e.  Forward (DIF): radix-2 stages whose span holds whole
// lanes (span >= 32, or >= 96 when M has the factor 3) run inside the lane;
// for M = 3 * 2^k a radix-3 stage at span 32 follows, also inside the lane
// (elements e, e+1, e+2 of a 96-point block, then twiddles W_96^(lane k));
// the last five radix-2 stages (spans 16 .. 1) exchange between lanes by
// shuffles.  The output order is the digit reversal these stages imply; the
// inverse (DIT, conjugate twiddles, unscaled) applies the same stages in
// reverse order and takes that order back to natural order, so spectra are
// only ever multiplied pointwise in the permuted order.
template <int M>
struct FftLen {
  static constexpr bool R3 = (M % 3) == 0;
  static constexpr int E = M / 32;
  static constexpr int LANE_MIN = R3 ? 96 : 32;  // smallest in-lane radix-2 span
};

template <int M>
__device__ __forceinline__ void wfft_dif(float2 *v, const float2 *__restrict__ tw) {
  constexpr int E = FftLen<M>::E;
  const int lane = threadIdx.x & 31;
  // in-lane radix-2 stages
#pragma unroll
  for (int hs = M / 2; hs >= FftLen<M>::LANE_MIN; hs /= 2) {
    if ((hs & 31) != 0) continue;
    const int he = hs / 32, stride = M / (2 * hs);
#pragma unroll
    for (int e = 0; e < E; e++) {
      if ((e / he) % 2 == 0) {
        const float2 w = tw[((lane + 32 * e) % hs) * stride];
        const float2 u = v[e], t = v[e + he];
        v[e] = cadd(u, t);
        v[e + he] = cmul(csub(u, t), w);
      }
    }
  }
  if constexpr (FftLen<M>::R3) {
    // radix 3 over elements e, e+1, e+2 (positions i, i+32, i+64 of a
    // 96-point block), then twiddles W_96^(lane k)
    const float s3 = 0.8660254037844386f;  // sqrt(3)/2
    const float2 w1 = tw[lane * (M / 96)], w2 = tw[2 * lane * (M / 96)];
#pragma unroll
    for (int e = 0; e < E; e += 3) {
      const float2 a = v[e], b = v[e + 1], c = v[e + 2];
      const float2 sm = cadd(b, c), df = csub(b, c);
      const float2 t = make_float2(a.x - 0.5f * sm.x, a.y - 0.5f * sm.y);
      const float2 u = make_float2(s3 * df.y, -s3 * df.x);  // -i sqrt(3)/2 (b - c)
      v[e] = cadd(a, sm);
      v[e + 1] = cmul(cadd(t, u), w1);
      v[e + 2] = cmul(csub(t, u), w2);
    }
  }
  // shuffle radix-2 stages, spans 16 .. 1
#pragma unroll
  for (int hs = 16; hs >= 1; hs /= 2) {
    const bool upper = (lane & hs) != 0;
    const float2 w = tw[(lane & (hs - 1)) * (M / (2 * hs))];
#pragma unroll
    for (int e = 0; e < E; e++) {
      const float2 x = v[e], y = shfl_x2(x, hs);
      v[e] = upper ? cmul(csub(y, x), w) : cadd(x, y);
    }
  }
}

template <int M>
__device__ __forceinline__ void wfft_dit_inv(float2 *v, const float2 *__restrict__ tw) {
  constexpr int E = FftLen<M>::E;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int hs = 1; hs <= 16; hs *= 2) {
    const bool upper = (lane & hs) != 0;
    float2 w = tw[(lane & (hs - 1)) * (M / (2 * hs))];
    w.y = -w.y;
#pragma unroll
    for (int e = 0; e < E; e++) {
      const float2 x = v[e], y = shfl_x2(x, hs);
      v[e] = upper ? csub(y, cmul(x, w)) : cadd(x, cmul(y, w));
    }
  }
  if constexpr (FftLen<M>::R3) {
    const float s3 = 0.8660254037844386f;
    float2 w1 = tw[lane * (M / 96)], w2 = tw[2 * lane * (M / 96)];
    w1.y = -w1.y;
    w2.y = -w2.y;
#pragma unroll
    for (int e = 0; e < E; e += 3) {
      const float2 a = v[e], b = cmul(v[e + 1], w1), c = cmul(v[e + 2], w2);
      const float2 sm = cadd(b, c), df = csub(b, c);
      const float2 t = make_float2(a.x - 0.5f * sm.x, a.y - 0.5f * sm.y);
      const float2 u = make_float2(-s3 * df.y, s3 * df.x);  // +i sqrt(3)/2 (b - c)
      v[e] = cadd(a, sm);
      v[e + 1] = cadd(t, u);
      v[e + 2] = csub(t, u);
    }
  }
#pragma unroll
  for (int hs = FftLen<M>::LANE_MIN; hs <= M / 2; hs *= 2) {
    if ((hs & 31) != 0) continue;
    const int he = hs / 32, stride = M / (2 * hs);
#pragma unroll
    for (int e = 0; e < E; e++) {
      if ((e / he) % 2 == 0) {
        float2 w = tw[((lane + 32 * e) % hs) * stride];
        w.y = -w.y;
        const float2 u = v[e], t = cmul(v[e + he], w);
        v[e] = cadd(u, t);
        v[e + he] = csub(u, t);
      }
    }
  }
}

__device__ __forceinline__ float kern_val(float hsq, int M, int x, int y, int z) {
  const int dx = min(x, M - x), dy = min(y, M - y), dz = min(z, M - z);
  const float r2 = (float)(dx * dx + dy * dy + dz * dz);
  const float b = 1.0f + hsq * r2;
  return 1.0f / (b * b);
}

// Plane p of a node's charges for the FFT: the charges [1, y - y_node] with
// the origin moved to the grid's middle (x, y, z: the node's place from it).
template <int D>
__device__ __forceinline__ float2 node_plane(const typename Node<D>::T &v, int p, float x, float y,
                                             float z) {
  if (p == 0) return make_float2(v.x, v.y + x * v.x);
  return make_float2(v.z + y * v.x, D == 3 ? v.w + z * v.x : 0.f);
}

// the FFT lengths the grid decision picks (sgt_fft_length)
#define SGT_FFT_DISPATCH(M_EXPR, CALL)            \
  switch (M_EXPR) {                               \
    case 32: CALL(32); break;                     \
    case 64: CALL(64); break;                     \
    case 96: CALL(96); break;                     \
    case 128: CALL(128); break;                   \
    case 192: CALL(192); break;                   \
    case 256: CALL(256); break;                   \
    case 384: CALL(384); break;                   \
    case 512: CALL(512); break;                   \
    case 768: CALL(768); break;                   \
    default: CALL(1024); break;                   \
  }

// ---------------------------------------------------------------------------
// Convolution of small and middle grids: plain discrete Fourier transforms
// (M = 2N, any N) along all axes but the last, a direct sum along that one.
//
//   k_spec_rows  per row of charges: fold the grid copies, transform along x
//                (frequencies 0..N of the real rows); per row offset the
//                transforms of K and of x K.
//   k_spec_y     3-D, per plane and frequency: transform along y; likewise the
//                kernel's planes, with the transform of y K.
//   k_spec_z     3-D, per pair of frequencies: sum over the input planes.
//   k_spec_cols  per output row: 2-D, sum over the input rows; 3-D, transform
//                back along y; then back along x.
//
// The result is Phi0 = sum K V0 and, per axis, Psi_k(g) = sum_s K(g - s)
// (U_k(s) + (s_k - g_k) V0(s)): the potential of the charges about the output
// node itself, in cells, so that the force sum_g w_g ((y - y_g) Phi0 - Psi)
// cancels nothing.  Along a transformed axis that is K^ U^ + i S V0^ with S
// the sine transform of x K; along the summed one the distance is a number.
//
// Why: FFT passes of these grids (16 to 128 points per axis, where nearly all
// iterations run) are three to five kernels bound by latency, pad N to a
// power of two or three times one, and their column pass needs 100 KB of
// shared memory in 2-D, for which a block waits until a whole SM has drained
// of the concurrent SpMV.  The plain transforms cost more operations than FFTs
// and still only a few microseconds, with 256 threads and 13 to 22 KB a block.
// In 3-D the plain transforms grow with N^4; sgt_plain_conv draws the line.
// ---------------------------------------------------------------------------
// k_spec_rows in one go, or its halves (the charge grid of a row-split
// embedding is summed over the ranks between them)
#define SGT_SPEC_BOTH 0
#define SGT_SPEC_FOLD 1
#define SGT_SPEC_TRANSFORM 2
#define SGT_SPEC_TY(D) ((D) == 3 ? 4 : 1)  // output rows a block takes together
#define SGT_SPEC_FS 8  // 3-D: x frequencies a block of k_spec_y takes together
#define SGT_SPEC_TZ 4  // 3-D: output planes a warp of k_spec_z sums together

// floor(a / b) for 0 <= a < 2^16, inv = 1 / b: half a unit away from every
// integer quotient
__device__ __forceinline__ int small_div(int a, float inv) { return (int)(((float)a + 0.5f) * inv); }

// second half of a row's spectrum: Uy (and Uz)
template <int D> struct SpecB { typedef float4 T; };
template <> struct SpecB<2> { typedef float2 T; };

// The spectra live in the FFT workspace.  Rows: (V0, Ux) of every row and
// frequency, then (Uy, Uz), then (K^, S) per row offset.  3-D: before them the
// plane spectra g (plane, y frequency, x frequency; 8 floats) and the kernel's
// k2 ((K^, Sx, Sy) per plane offset and pair of frequencies up to N); the
// summed spectra h take the rows' place once k_spec_y has read those.
template <int D>
struct SpecBuf {
  float4 *g, *k2, *h;
  float4 *h0;
  typename SpecB<D>::T *h1;
  float2 *k;
  __device__ __forceinline__ SpecBuf(float2 *W, int N) {
    const long F = N + 1, rows = D == 2 ? N : (long)N * N;
    float4 *p = reinterpret_cast<float4 *>(W);
    g = p;
    k2 = p + (D == 3 ? 4 * rows * F : 0);
    h = k2 + (D == 3 ? (long)N * F * F : 0);
    h0 = h;
    h1 = reinterpret_cast<typename SpecB<D>::T *>(h0 + rows * F);
    k = reinterpret_cast<float2 *>(h1 + rows * F);
  }
};

// tw[j] = exp(-2 pi i j / M)
__device__ __forceinline__ void spec_twiddles(float2 *tw, int M) {
  for (int j = threadIdx.x; j < M; j += SGT_THREADS) {
    float sn, cs;
    sincospif(__fdiv_rn(2.0f * (float)j, (float)M), &sn, &cs);
    tw[j] = make_float2(cs, -sn);
  }
}

// ---------------------------------------------------------------------------
// fold: V = sum of the grid copies, which are left zero for the next
// iteration's scatter (they start zero at job creation).  Cell mode: V only
// (k_bin_count cleared it and k_s2g_cell has added to it), nothing to do.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k_fold_body(int vb_, int vg_, const SgtState *st,
                                            typename Node<D>::T *__restrict__ Vc,
                                            typename Node<D>::T *__restrict__ V) {
  if (st->T != 0) return;
  const int N = st->N, copies = st->copies;
  long nodes = N;
  if (D >= 2) nodes *= N;
  if (D >= 3) nodes *= N;
  typename Node<D>::T z;
  if constexpr (D == 1) z = make_float2(0.f, 0.f); else z = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long g = vb_ * (long)blockDim.x + threadIdx.x; g < nodes; g += (long)vg_ * blockDim.x) {
    typename Node<D>::T a = z;
    for (int c0 = 0; c0 < copies; c0 += 4) {
      typename Node<D>::T t[4];
#pragma unroll
      for (int c = 0; c < 4; c++) t[c] = c0 + c < copies ? Vc[(c0 + c) * nodes + g] : z;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        a.x += t[c].x;
        a.y += t[c].y;
        if constexpr (D >= 2) {
          a.z += t[c].z;
          if constexpr (D >= 3) a.w += t[c].w;
        }
        if (c0 + c < copies) Vc[(c0 + c) * nodes + g] = z;
      }
    }
    V[g] = a;
  }
}
template <int D>
__device__ __forceinline__ void k_spec_rows_body(int vb_, int vg_, const SgtState *st,
                                                 typename Node<D>::T *__restrict__ Vc,
                                                 typename Node<D>::T *__restrict__ V,
                                                 float2 *__restrict__ W, int phase) {
  const int N = st->N;
  if (D == 1 || !st->direct || phase == SGT_SPEC_FOLD) {
    // the fold alone: 1-D, grids of the FFT passes, the shards' scatter phase
    sgt_pdl_wait();
    if (phase != SGT_SPEC_TRANSFORM) k_fold_body<D>(vb_, vg_, st, Vc, V);
    return;
  }
  if constexpr (D >= 2) {
    __shared__ float2 tw[2 * 128];
    __shared__ float4 row[128];
    __shared__ float red[SGT_THREADS * 9];
    const int M = 2 * N, F = N + 1, rows = D == 2 ? N : N * N;
    if (vb_ >= rows) {
      sgt_pdl_wait();
      return;
    }
    const float inv_f = 1.0f / (float)F, inv_m = 1.0f / (float)M;
    const SpecBuf<D> B(W, N);
    spec_twiddles(tw, M);
    // thread: frequency f and segment sg of the row
    const int S = SGT_THREADS / F, t = threadIdx.x;  // F <= 129: S >= 1
    const int sg = small_div(t, inv_f), f = t - sg * F;
    const int len = (N + S - 1) / S, x0 = min(sg * len, N), x1 = min(N, x0 + len);
    const int w0 = f * x0 - M * small_div(f * x0, inv_m);
    float *K = reinterpret_cast<float *>(row);
    const float hsq = st->h_eff * st->h_eff;
    // kernel rows: fixed before the chain began, done while the previous
    // kernel drains
    for (int r = vb_; r < rows; r += vg_) {
      const int dz = D == 2 ? 0 : small_div(r, 1.0f / (float)N), dy = r - dz * N;
      __syncthreads();
      for (int x = t; x < N; x += SGT_THREADS) {
        const float b = 1.0f + hsq * (float)(x * x + dy * dy + dz * dz);
        K[x] = (x == 0 ? 1.0f : 2.0f) / (b * b);
      }
      __syncthreads();
      if (sg < S) {
        float kc = 0.f, ks = 0.f;
        int w = w0;
        for (int x = x0; x < x1; x++) {
          const float2 e = tw[w];
          const float k = K[x];
          kc += k * e.x;
          ks -= (float)x * k * e.y;
          w += f;
          if (w >= M) w -= M;
        }
        red[2 * t] = kc;
        red[2 * t + 1] = ks;
      }
      __syncthreads();
      if (t < F) {
        float kc = 0.f, ks = 0.f;
        for (int g = 0; g < S; g++) {
          kc += red[2 * (g * F + t)];
          ks += red[2 * (g * F + t) + 1];
        }
        B.k[(long)r * F + t] = make_float2(kc, ks);
      }
    }
    sgt_pdl_wait();
    const int copies = st->copies;
    const bool cell = st->T != 0 || phase == SGT_SPEC_TRANSFORM;  // V is complete
    const long nodes = (long)rows * N;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int r = vb_; r < rows; r += vg_) {
      __syncthreads();
      // the row's charges: 4 lanes a node, the copies dealt over them
      for (int e = t; e < ((4 * N + 31) & ~31); e += SGT_THREADS) {
        const int x = e >> 2, p = e & 3;
        float4 a = z4;
        if (x < N) {
          const long g = (long)r * N + x;
          if (cell) {
            if (p == 0) a = V[g];
          } else {
            for (int c0 = p; c0 < copies; c0 += 16) {
              float4 q[4];
#pragma unroll
              for (int u = 0; u < 4; u++)
                q[u] = c0 + 4 * u < copies ? Vc[(c0 + 4 * u) * nodes + g] : z4;
#pragma unroll
              for (int u = 0; u < 4; u++) {
                a.x += q[u].x; a.y += q[u].y; a.z += q[u].z; a.w += q[u].w;
                if (c0 + 4 * u < copies) Vc[(c0 + 4 * u) * nodes + g] = z4;
              }
            }
          }
        }
#pragma unroll
        for (int o = 1; o < 4; o *= 2) {
          a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
          a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
          a.z += __shfl_xor_sync(0xffffffffu, a.z, o);
          if (D == 3) a.w += __shfl_xor_sync(0xffffffffu, a.w, o);
        }
        if (p == 0 && x < N) {
          row[x] = a;
          if (!cell) V[(long)r * N + x] = a;
        }
      }
      __syncthreads();
      if (sg < S) {
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        int w = w0;
        for (int x = x0; x < x1; x++) {
          const float2 e = tw[w];
          const float4 v = row[x];
          a[0] += v.x * e.x; a[1] += v.x * e.y;
          a[2] += v.y * e.x; a[3] += v.y * e.y;
          a[4] += v.z * e.x; a[5] += v.z * e.y;
          if constexpr (D == 3) { a[6] += v.w * e.x; a[7] += v.w * e.y; }
          w += f;
          if (w >= M) w -= M;
        }
#pragma unroll
        for (int c = 0; c < (D == 3 ? 8 : 6); c++) red[t * 9 + c] = a[c];
      }
      __syncthreads();
      if (t < F) {
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int g = 0; g < S; g++)
#pragma unroll
          for (int c = 0; c < (D == 3 ? 8 : 6); c++) a[c] += red[(g * F + t) * 9 + c];
        const long at = (long)r * F + t;
        B.h0[at] = make_float4(a[0], a[1], a[2], a[3]);
        if constexpr (D == 3) B.h1[at] = make_float4(a[4], a[5], a[6], a[7]);
        else B.h1[at] = make_float2(a[4], a[5]);
      }
    }
  }
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS, 4)
k_spec_rows(const SgtState *st, typename Node<D>::T *__restrict__ Vc,
            typename Node<D>::T *__restrict__ V, float2 *__restrict__ W, int phase) {
  k_spec_rows_body<D>(blockIdx.x, gridDim.x, st, Vc, V, W, phase);
}

// 3-D: transform along y.  A block takes a plane (or a plane offset of the
// kernel) and SGT_SPEC_FS x frequencies, the inputs in shared memory; a thread
// sums an output frequency pair over the N rows, 16 multiply-adds per row.
__device__ __forceinline__ void k_spec_y_body(int vb_, int vg_, const SgtState *st,
                                              float2 *__restrict__ W) {
  if (!st->direct) {
    sgt_pdl_wait();
    return;
  }
  constexpr int FS = SGT_SPEC_FS;
  const int N = st->N, M = 2 * N, F = N + 1, fb = (F + FS - 1) / FS, items = N * fb;
  if (vb_ >= 2 * items) {
    sgt_pdl_wait();
    return;
  }
  __shared__ float2 tw[2 * SGT_SPEC_MAX(3)];
  __shared__ float4 in[SGT_SPEC_MAX(3) * FS * 2];
  const SpecBuf<3> B(W, N);
  spec_twiddles(tw, M);
  const int t = threadIdx.x;
  const float inv_fb = 1.0f / (float)fb;
  sgt_pdl_wait();
  for (int it = vb_; it < 2 * items; it += vg_) {
    const bool kernel = it >= items;
    const int e = kernel ? it - items : it;
    const int z = small_div(e, inv_fb), f0 = (e - z * fb) * FS, nf = min(FS, F - f0);
    __syncthreads();
    if (!kernel) {
      for (int q = t; q < N * FS; q += SGT_THREADS) {
        const int y = q / FS, f = min(q % FS, nf - 1);
        const long at = ((long)z * N + y) * F + f0 + f;
        in[2 * q] = B.h0[at];
        in[2 * q + 1] = B.h1[at];
      }
      __syncthreads();
      for (int q = t; q < M * FS; q += SGT_THREADS) {
        const int ky = q / FS, f = q % FS;
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        int w = 0;
        for (int y = 0; y < N; y++) {
          const float2 c = tw[w];
          const float4 u = in[2 * (y * FS + f)], v = in[2 * (y * FS + f) + 1];
          a[0] += u.x * c.x - u.y * c.y; a[1] += u.x * c.y + u.y * c.x;
          a[2] += u.z * c.x - u.w * c.y; a[3] += u.z * c.y + u.w * c.x;
          a[4] += v.x * c.x - v.y * c.y; a[5] += v.x * c.y + v.y * c.x;
          a[6] += v.z * c.x - v.w * c.y; a[7] += v.z * c.y + v.w * c.x;
          w += ky;
          if (w >= M) w -= M;
        }
        if (f < nf) {
          float4 *g = B.g + 2 * (((long)z * M + ky) * F + f0 + f);
          g[0] = make_float4(a[0], a[1], a[2], a[3]);
          g[1] = make_float4(a[4], a[5], a[6], a[7]);
        }
      }
    } else {
      float2 *kin = reinterpret_cast<float2 *>(in);
      for (int q = t; q < N * FS; q += SGT_THREADS) {
        const int y = q / FS, f = min(q % FS, nf - 1);
        float2 k = B.k[((long)z * N + y) * F + f0 + f];
        if (y > 0) { k.x *= 2.0f; k.y *= 2.0f; }
        kin[q] = k;
      }
      __syncthreads();
      for (int q = t; q < F * FS; q += SGT_THREADS) {
        const int ky = q / FS, f = q % FS;
        float kk = 0.f, sx = 0.f, sy = 0.f;
        int w = 0;
        for (int y = 0; y < N; y++) {
          const float2 c = tw[w], k = kin[y * FS + f];
          kk += k.x * c.x;
          sx += k.y * c.x;
          sy -= (float)y * k.x * c.y;
          w += ky;
          if (w >= M) w -= M;
        }
        if (f < nf) B.k2[((long)z * F + ky) * F + f0 + f] = make_float4(kk, sx, sy, 0.f);
      }
    }
  }
}
__global__ void __launch_bounds__(SGT_THREADS, 4)
k_spec_y(const SgtState *st, float2 *__restrict__ W) {
  k_spec_y_body(blockIdx.x, gridDim.x, st, W);
}

// 3-D: sum over the input planes, frequency by frequency.  A lane holds a
// frequency pair, a warp SGT_SPEC_TZ output planes (52 multiply-adds per input
// plane; the kernel's values slide through registers), a block 32 pairs and
// 8 warps of planes.
__device__ __forceinline__ void k_spec_z_body(int vb_, int vg_, const SgtState *st,
                                              float2 *__restrict__ W) {
  sgt_pdl_wait();
  if (!st->direct) return;
  constexpr int TZ = SGT_SPEC_TZ, WPB = SGT_THREADS / 32;
  const int N = st->N, M = 2 * N, F = N + 1, pairs = M * F;
  const int pb = (pairs + 31) / 32, zb = (N + TZ * WPB - 1) / (TZ * WPB), items = pb * zb;
  const SpecBuf<3> B(W, N);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int it = vb_; it < items; it += vg_) {
    const int zt = it / pb, pr = (it - zt * pb) * 32 + lane;
    const int z0 = (zt * WPB + warp) * TZ;
    if (z0 >= N || pr >= pairs) continue;
    const int ky = pr / F, f = pr - ky * F;
    const bool up = ky > N;  // K^ and Sx are even in ky, Sy odd
    const float4 *k2 = B.k2 + (long)(up ? M - ky : ky) * F + f;
    const float sgn = up ? -1.0f : 1.0f;
    const long ks = (long)F * F, gs = (long)M * F;
    const float4 *g = B.g + 2 * (long)pr;
    float a[TZ][8];
#pragma unroll
    for (int j = 0; j < TZ; j++)
#pragma unroll
      for (int c = 0; c < 8; c++) a[j][c] = 0.f;
    float4 k[TZ];  // k[j]: offset z0 + j - z
#pragma unroll
    for (int j = 1; j < TZ; j++) k[j] = k2[min(z0 + j, N - 1) * ks];
#pragma unroll 2
    for (int z = 0; z < N; z++) {
      k[0] = k2[abs(z0 - z) * ks];
      const float4 u = g[2 * z * gs], v = g[2 * z * gs + 1];
#pragma unroll
      for (int j = 0; j < TZ; j++) {
        const float dz = (float)(z - z0 - j), sy = sgn * k[j].z;
        a[j][0] += k[j].x * u.x;
        a[j][1] += k[j].x * u.y;
        a[j][2] += k[j].x * u.z - k[j].y * u.y;
        a[j][3] += k[j].x * u.w + k[j].y * u.x;
        a[j][4] += k[j].x * v.x - sy * u.y;
        a[j][5] += k[j].x * v.y + sy * u.x;
        a[j][6] += k[j].x * (v.z + dz * u.x);
        a[j][7] += k[j].x * (v.w + dz * u.y);
      }
#pragma unroll
      for (int j = TZ - 1; j > 0; j--) k[j] = k[j - 1];
    }
#pragma unroll
    for (int j = 0; j < TZ; j++)
      if (z0 + j < N) {
        float4 *h = B.h + 2 * ((z0 + j) * gs + pr);
        h[0] = make_float4(a[j][0], a[j][1], a[j][2], a[j][3]);
        h[1] = make_float4(a[j][4], a[j][5], a[j][6], a[j][7]);
      }
  }
}
__global__ void __launch_bounds__(SGT_THREADS, 2)
k_spec_z(const SgtState *st, float2 *__restrict__ W) {
  k_spec_z_body(blockIdx.x, gridDim.x, st, W);
}

template <int D>
__device__ __forceinline__ void k_spec_cols_body(int vb_, int vg_, const SgtState *st,
                                                 const typename Node<D>::T *__restrict__ V,
                                                 const float2 *__restrict__ W,
                                                 typename Node<D>::T *__restrict__ Phi) {
  if constexpr (D == 1) {
    // 1-D: a warp per output sums over the grid
    sgt_pdl_wait();
    const int N = st->N, lane = threadIdx.x & 31;
    const float hsq = st->h_eff * st->h_eff;
    constexpr int WPB = SGT_THREADS / 32;
    for (int x = vb_ * WPB + (threadIdx.x >> 5); x < N; x += vg_ * WPB) {
      float p0 = 0.f, p1 = 0.f;
      for (int s = lane; s < N; s += 32) {
        const float2 v = V[s];
        const float r = (float)(s - x), b = 1.0f + hsq * (r * r), k = 1.0f / (b * b);
        p0 += k * v.x;
        p1 += k * (v.y + r * v.x);
      }
      p0 = warp_sum_f(p0);
      p1 = warp_sum_f(p1);
      if (lane == 0) Phi[x] = make_float2(p0, p1);
    }
  } else {
    constexpr int TY = SGT_SPEC_TY(D), C = 2 * (D + 1);  // reals per output and frequency
    if (!st->direct) {
      sgt_pdl_wait();
      return;
    }
    const int N = st->N, M = 2 * N, F = N + 1;
    const int ty = (N + TY - 1) / TY, items = (D == 2 ? 1 : N) * ty;
    if (vb_ >= items) {
      sgt_pdl_wait();
      return;
    }
    __shared__ float2 tw[2 * 128];
    __shared__ float red[SGT_THREADS * 9];
    __shared__ float What[129 * (C + 1)];  // [frequency][C + 1]
    spec_twiddles(tw, M);
    const float inv_f = 1.0f / (float)F, inv_m = 1.0f / (float)M;
    const SpecBuf<D> B(const_cast<float2 *>(W), N);
    const int t = threadIdx.x, S = SGT_THREADS / F;
    const int sg = small_div(t, inv_f), f = t - sg * F;
    // the segments share the input rows (2-D) or y frequencies (3-D)
    const int nin = D == 2 ? N : M, len = (nin + S - 1) / S;
    const int r0 = min(sg * len, nin), r1 = min(nin, r0 + len);
    sgt_pdl_wait();
    __syncthreads();  // the twiddles
    for (int it = vb_; it < items; it += vg_) {
      const int oz = D == 2 ? 0 : small_div(it, 1.0f / (float)ty), y0 = (it - oz * ty) * TY;
      float a[TY][C];
#pragma unroll
      for (int j = 0; j < TY; j++)
#pragma unroll
        for (int c = 0; c < C; c++) a[j][c] = 0.f;
      if (sg < S) {
        if constexpr (D == 2) {
          const float2 *kp = B.k + f;
          const float4 *h0 = B.h0 + f;
          const typename SpecB<D>::T *h1 = B.h1 + f;
#pragma unroll 4
          for (int r = r0; r < r1; r++) {
            const float2 k = kp[abs(y0 - r) * F];
            const float4 v = h0[r * F];
            const typename SpecB<D>::T u = h1[r * F];
            const float dy = (float)(r - y0);
            a[0][0] += k.x * v.x;
            a[0][1] += k.x * v.y;
            a[0][2] += k.x * v.z - k.y * v.y;
            a[0][3] += k.x * v.w + k.y * v.x;
            a[0][4] += k.x * (u.x + dy * v.x);
            a[0][5] += k.x * (u.y + dy * v.y);
          }
        } else {
          const float4 *h = B.h + 2 * ((long)oz * M * F + f);
          int w[TY];
#pragma unroll
          for (int j = 0; j < TY; j++) w[j] = (y0 + j) * r0 - M * small_div((y0 + j) * r0, inv_m);
#pragma unroll 2
          for (int r = r0; r < r1; r++) {
            const float4 u = h[2 * (long)r * F], v = h[2 * (long)r * F + 1];
#pragma unroll
            for (int j = 0; j < TY; j++) {
              const float2 c = tw[w[j]];  // (cos, -sin): times (cos + i sin)
              a[j][0] += u.x * c.x + u.y * c.y; a[j][1] += u.y * c.x - u.x * c.y;
              a[j][2] += u.z * c.x + u.w * c.y; a[j][3] += u.w * c.x - u.z * c.y;
              a[j][4] += v.x * c.x + v.y * c.y; a[j][5] += v.y * c.x - v.x * c.y;
              a[j][6] += v.z * c.x + v.w * c.y; a[j][7] += v.w * c.x - v.z * c.y;
              w[j] += y0 + j;
              if (w[j] >= M) w[j] -= M;
            }
          }
        }
      }
      // back along x: P lanes (a power of two) per output
      int lp = 0;
      while ((N << (lp + 1)) <= SGT_THREADS && lp < 3) lp++;
      const int P = 1 << lp, p = t & (P - 1);
      const float scale = D == 2 ? 1.0f / (float)M : 1.0f / ((float)M * (float)M);
#pragma unroll
      for (int j = 0; j < TY; j++) {
        // the segments' sums, in order
        __syncthreads();
        if (sg < S) {
#pragma unroll
          for (int c = 0; c < C; c++) red[t * 9 + c] = a[j][c];
        }
        __syncthreads();
        for (int e = t; e < F * (C / 2); e += SGT_THREADS) {
          const int c2 = small_div(e, inv_f), ff = e - c2 * F;
          float re = 0.f, im = 0.f;
          for (int g = 0; g < S; g++) {
            re += red[(g * F + ff) * 9 + 2 * c2];
            im += red[(g * F + ff) * 9 + 2 * c2 + 1];
          }
          const float wt = (ff == 0 || ff == N) ? 1.0f : 2.0f;
          What[ff * (C + 1) + 2 * c2] = wt * re;
          What[ff * (C + 1) + 2 * c2 + 1] = wt * im;
        }
        __syncthreads();
        const int y = y0 + j;
        for (int o0 = 0; o0 < N; o0 += SGT_THREADS >> lp) {  // uniform
          const int o = o0 + (t >> lp), x = min(o, N - 1);
          float q[D + 1];
#pragma unroll
          for (int c = 0; c <= D; c++) q[c] = 0.f;
          const int step = x * P - M * small_div(x * P, inv_m);
          int w = x * p - M * small_div(x * p, inv_m);
          for (int ff = p; ff < F; ff += P) {
            const float2 e = tw[w];  // (cos, -sin): Re(W exp(+i)) = re cos + im (-sin)
            const float *wh = &What[ff * (C + 1)];
#pragma unroll
            for (int c = 0; c <= D; c++) q[c] += wh[2 * c] * e.x + wh[2 * c + 1] * e.y;
            w += step;
            if (w >= M) w -= M;
          }
#pragma unroll
          for (int e = 1; e < 8; e *= 2)
            if (e < P) {
#pragma unroll
              for (int c = 0; c <= D; c++) q[c] += __shfl_xor_sync(0xffffffffu, q[c], e);
            }
          if (p == 0 && o < N && y < N)
            Phi[((long)(D == 2 ? 0 : oz) * N + y) * N + x] = make_float4(
                q[0] * scale, q[1] * scale, q[2] * scale, D == 3 ? q[D] * scale : 0.f);
        }
      }
    }
  }
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS, 3)
k_spec_cols(const SgtState *st, const typename Node<D>::T *__restrict__ V,
            const float2 *__restrict__ W, typename Node<D>::T *__restrict__ Phi) {
  k_spec_cols_body<D>(blockIdx.x, gridDim.x, st, V, W, Phi);
}

// ---------------------------------------------------------------------------
// d >= 2, pass 1: build rows (x lines) of the data planes (rows y, z < N) and
// of the kernel plane (all rows), forward FFT along x.
// W plane p at W + p * M^d; the kernel plane is p = 2.
// ---------------------------------------------------------------------------
template <int D, int M>
__device__ void build_rows_body(int vb_, int vg_, const SgtState *st, const typename Node<D>::T *__restrict__ V,
                                float2 *__restrict__ W, const float2 *tw) {
  constexpr int E = M / 32;
  const int N = st->N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float hsq = st->h_eff * st->h_eff;
  const long plane = D == 2 ? (long)M * M : (long)M * M * M;
  const int nz_d = D == 3 ? N : 1, nz_k = D == 3 ? M : 1;
  const long lines_d = 2L * N * nz_d, lines = lines_d + (long)M * nz_k;
  const int wpb = blockDim.x >> 5;
  const float mid = 0.5f * (float)(N - 1);  // place of the grid's middle, in nodes
  for (long ln = (long)vb_ * wpb + warp; ln < lines; ln += (long)vg_ * wpb) {
    float2 v[E];
    int p, y, z;
    if (ln < lines_d) {
      p = (int)(ln / ((long)N * nz_d));
      const long r = ln % ((long)N * nz_d);
      z = (int)(r / N);
      y = (int)(r % N);
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int x = lane + 32 * e;
        v[e] = x < N ? node_plane<D>(V[x + (long)N * y + (D == 3 ? (long)N * N * z : 0)], p,
                                     (float)x - mid, (float)y - mid, (float)z - mid)
                     : make_float2(0.f, 0.f);
      }
    } else {
      p = 2;
      const long r = ln - lines_d;
      z = (int)(r / M);
      y = (int)(r % M);
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = make_float2(kern_val(hsq, M, lane + 32 * e, y, z), 0.f);
    }
    wfft_dif<M>(v, tw);
    float2 *row = W + p * plane + (long)M * y + (D == 3 ? (long)M * M * z : 0);
#pragma unroll
    for (int e = 0; e < E; e++) row[lane + 32 * e] = v[e];
  }
}

template <int D>
__device__ __forceinline__ void k_fft_build_x_body(int vb_, int vg_, const SgtState *st, const typename Node<D>::T *__restrict__ V, float2 *__restrict__ W) {
  sgt_pdl_wait();
  __shared__ float2 tw[SGT_FFT_MAXM];
  if (st->direct) return;  // k_spec_cols did it
  fft_twiddles(tw, st->M);
  __syncthreads();
#define CB(L) build_rows_body<D, L>(vb_, vg_, st, V, W, tw)
  SGT_FFT_DISPATCH(st->M, CB)
#undef CB
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_fft_build_x(const SgtState *st, const typename Node<D>::T *__restrict__ V, float2 *__restrict__ W) {
  k_fft_build_x_body<D>(blockIdx.x, gridDim.x, st, V, W);
}

// ---------------------------------------------------------------------------
// column passes: 8 adjacent columns per CTA staged through shared memory.
// MODE_LAST: last axis (y for d = 2, z for d = 3): kernel spectrum, data
//            forward, product with Re(K^), inverse, keep positions < N.
// MODE_MID_FWD / MODE_MID_INV: d = 3, axis y of the data planes z < N (and of
//            the kernel plane on the forward pass).
// ---------------------------------------------------------------------------
#define MODE_LAST 0
#define MODE_MID_FWD 1
#define MODE_MID_INV 2

template <int M>
__device__ __forceinline__ void stage_load(float2 *stg, const float2 *__restrict__ src, long stride,
                                           int lim) {
  constexpr int LS = M + SGT_FFT_PAD;
  for (int idx = threadIdx.x; idx < SGT_FFT_COLS * M; idx += blockDim.x) {
    const int t = idx / SGT_FFT_COLS, c = idx % SGT_FFT_COLS;
    stg[c * LS + t] = t < lim ? src[(long)t * stride + c] : make_float2(0.f, 0.f);
  }
}
template <int M>
__device__ __forceinline__ void stage_store(const float2 *stg, float2 *__restrict__ dst, long stride,
                                            int lim) {
  constexpr int LS = M + SGT_FFT_PAD;
  for (int idx = threadIdx.x; idx < SGT_FFT_COLS * lim; idx += blockDim.x) {
    const int t = idx / SGT_FFT_COLS, c = idx % SGT_FFT_COLS;
    dst[(long)t * stride + c] = stg[c * LS + t];
  }
}

template <int D, int MODE, int M>
__device__ void cols_body(int vb_, int vg_, const SgtState *st, float2 *__restrict__ W, const float2 *tw,
                          float2 *stg, float *kre) {
  constexpr int E = M / 32, LS = M + SGT_FFT_PAD;
  const int N = st->N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long plane = D == 2 ? (long)M * M : (long)M * M * M;
  const int ncb = M / SGT_FFT_COLS;
  // last pass: lines along y (d = 2, stride M) or z (d = 3, stride M^2)
  const long stride = (MODE == MODE_LAST && D == 3) ? (long)M * M : (long)M;
  long items;
  if (MODE == MODE_LAST) items = D == 2 ? ncb : (long)ncb * M;  // d = 3: every y
  else if (MODE == MODE_MID_FWD) items = (long)ncb * (2L * N + M);  // data z < N, kernel all z
  else items = (long)ncb * 2L * N;
  float2 v[E];
  for (long it = vb_; it < items; it += vg_) {
    const int cb = (int)(it % ncb);
    const long rest = it / ncb;
    __syncthreads();
    if (MODE == MODE_LAST) {
      const long off = (long)cb * SGT_FFT_COLS + (D == 3 ? (long)M * rest : 0);
      // kernel spectrum of the 8 columns, real part kept
      stage_load<M>(stg, W + 2 * plane + off, stride, M);
      __syncthreads();
#pragma unroll
      for (int e = 0; e < E; e++) v[e] = stg[warp * LS + lane + 32 * e];
      wfft_dif<M>(v, tw);
#pragma unroll
      for (int e = 0; e < E; e++) kre[warp * M + lane + 32 * e] = v[e].x;
      for (int p = 0; p < 2; p++) {
        float2 *base = W + p * plane + off;
        __syncthreads();
        stage_load<M>(stg, base, stride, N);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = stg[warp * LS + lane + 32 * e];
        wfft_dif<M>(v, tw);
#pragma unroll
        for (int e = 0; e < E; e++) {
          const float kr = kre[warp * M + lane + 32 * e];
          v[e] = make_float2(v[e].x * kr, v[e].y * kr);
        }
        wfft_dit_inv<M>(v, tw);
#pragma unroll
        for (int e = 0; e < E; e++) stg[warp * LS + lane + 32 * e] = v[e];
        __syncthreads();
        stage_store<M>(stg, base, stride, N);
      }
    } else {
      int p, z;
      if (rest < 2L * N) {
        p = (int)(rest / N);
        z = (int)(rest % N);
      } else {
        p = 2;
        z = (int)(rest - 2L * N);
      }
      float2 *base = W + p * plane + (long)M * M * z + (long)cb * SGT_FFT_COLS;
      if (MODE == MODE_MID_FWD) {
        stage_load<M>(stg, base, M, p == 2 ? M : N);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = stg[warp * LS + lane + 32 * e];
        wfft_dif<M>(v, tw);
#pragma unroll
        for (int e = 0; e < E; e++) stg[warp * LS + lane + 32 * e] = v[e];
        __syncthreads();
        stage_store<M>(stg, base, M, M);
      } else {
        stage_load<M>(stg, base, M, M);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = stg[warp * LS + lane + 32 * e];
        wfft_dit_inv<M>(v, tw);
#pragma unroll
        for (int e = 0; e < E; e++) stg[warp * LS + lane + 32 * e] = v[e];
        __syncthreads();
        stage_store<M>(stg, base, M, N);
      }
    }
  }
}

template <int D, int MODE>
__device__ __forceinline__ void k_fft_cols_body(int vb_, int vg_, const SgtState *st,
                                                float2 *__restrict__ W) {
  sgt_pdl_wait();
  extern __shared__ float2 sm[];
  if (st->direct) return;
  float2 *tw = sm;
  float2 *stg = sm + SGT_FFT_MAXM;
  float *kre = reinterpret_cast<float *>(stg + SGT_FFT_COLS * (st->M + SGT_FFT_PAD));
  fft_twiddles(tw, st->M);
  __syncthreads();
#define CC(L) cols_body<D, MODE, L>(vb_, vg_, st, W, tw, stg, kre)
  SGT_FFT_DISPATCH(st->M, CC)
#undef CC
}
template <int D, int MODE>
__global__ void __launch_bounds__(SGT_THREADS)
k_fft_cols(const SgtState *st, float2 *__restrict__ W) {
  k_fft_cols_body<D, MODE>(blockIdx.x, gridDim.x, st, W);
}

// ---------------------------------------------------------------------------
// final pass: inverse FFT along x of rows y (, z) < N, scale by 1/M^d, write
// the potential grid (channels packed per node: plane 0 -> .xy, 1 -> .zw).
// ---------------------------------------------------------------------------
template <int D, int M>
__device__ void final_rows_body(int vb_, int vg_, const SgtState *st, const float2 *__restrict__ W,
                                float2 *__restrict__ Phi2, const float2 *tw) {
  constexpr int E = M / 32;
  const int N = st->N, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long plane = D == 2 ? (long)M * M : (long)M * M * M;
  const long lines = 2L * N * (D == 3 ? N : 1);
  const int wpb = blockDim.x >> 5;
  float inv = 1.0f / (float)M;
  inv = inv / (float)M;
  if (D == 3) inv = inv / (float)M;
  for (long ln = (long)vb_ * wpb + warp; ln < lines; ln += (long)vg_ * wpb) {
    const int p = (int)(ln % 2);
    const long r = ln / 2;
    const int y = (int)(r % N), z = D == 3 ? (int)(r / N) : 0;
    const float2 *row = W + p * plane + (long)M * y + (D == 3 ? (long)M * M * z : 0);
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; e++) v[e] = row[lane + 32 * e];
    wfft_dit_inv<M>(v, tw);
    const long g0 = (long)N * y + (D == 3 ? (long)N * N * z : 0);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int x = lane + 32 * e;
      if (x < N) Phi2[2 * (g0 + x) + p] = make_float2(v[e].x * inv, v[e].y * inv);
    }
  }
}

template <int D>
__device__ __forceinline__ void k_fft_final_x_body(int vb_, int vg_, const SgtState *st, const float2 *__restrict__ W, typename Node<D>::T *__restrict__ Phi) {
  sgt_pdl_wait();
  __shared__ float2 tw[SGT_FFT_MAXM];
  if (st->direct) return;
  fft_twiddles(tw, st->M);
  __syncthreads();
#define CF(L) final_rows_body<D, L>(vb_, vg_, st, W, reinterpret_cast<float2 *>(Phi), tw)
  SGT_FFT_DISPATCH(st->M, CF)
#undef CF
}
template <int D>
__global__ void __launch_bounds__(SGT_THREADS)
k_fft_final_x(const SgtState *st, const float2 *__restrict__ W, typename Node<D>::T *__restrict__ Phi) {
  k_fft_final_x_body<D>(blockIdx.x, gridDim.x, st, W, Phi);
}

// shared memory of a column pass for FFT length Mmax
__host__ __device__ inline size_t fft_cols_smem(int Mmax) {
  return sizeof(float2) * (SGT_FFT_MAXM + (size_t)SGT_FFT_COLS * (Mmax + SGT_FFT_PAD)) +
         sizeof(float) * (size_t)SGT_FFT_COLS * Mmax;
}
