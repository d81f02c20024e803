// sgt_knn.cu -- exact k nearest neighbours on the device: the kNN stage in
// front of the perplexity equalisation (the reference's command line tool
// calls FLANN, an approximate search, at
// CU/testing_modules/demo_perplexity.cu:131; this search is exact).
// Two methods return the same bits: the SIMT search (k_knn) and a tensor-core
// filter (k_knn_tc, further down) whose candidates are re-ranked with the SIMT
// search's arithmetic.
//
// SIMT search: one query per thread, 128 queries per CTA.  Candidates stream through
// shared memory in tiles of 64 points x 64 dimensions, queries in tiles of
// 128 x 64; rows are padded to 68 floats so each thread's float4 loads of
// its query and the (broadcast) float4 loads of a candidate are free of bank
// conflicts.  Each thread accumulates the 64 squared distances of a tile in
// registers as sums of squared differences (not |x|^2 + |y|^2 - 2 x.y, whose
// cancellation would reorder near neighbours), then offers them to its
// sorted top-k list (local memory) behind a threshold test: after the list
// fills, only candidates closer than its current k-th neighbour are
// inserted, so insertions are rare.  The self match is skipped.  Output rows
// are sorted by distance, ties by index.
#include "../../include/sgtsne_b200.h"
#include "sgt_internal.h"
#include "sgt_async.cuh"
#include "sgt_knn_rules.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <string>

namespace {

constexpr int KNN_Q = 128;   // queries per CTA
constexpr int KNN_C = 64;    // candidates per tile
constexpr int KNN_DC = 64;   // dimensions per chunk
constexpr int KNN_LD = KNN_DC + 4;
constexpr int KNN_MAXK = 128;

__device__ __forceinline__ bool knn_less(float da, int ia, float db, int ib) {
  return da < db || (da == db && ia < ib);
}

// query of slot s: the s-th point, or the s-th entry of a query list
__device__ __forceinline__ int knn_query(const int *qlist, int nq, int s) {
  return s < nq ? (qlist ? qlist[s] : s) : -1;
}

// qlist == nullptr: every point is a query (nq == n); otherwise the nq
// points listed are.
__global__ void __launch_bounds__(KNN_Q)
k_knn(const float *__restrict__ X, int n, int dim, int k, const int *__restrict__ qlist, int nq,
      int *__restrict__ idx, float *__restrict__ d2) {
  extern __shared__ float sm[];
  float *sQ = sm;                   // [KNN_Q][KNN_LD]
  float *sC = sm + KNN_Q * KNN_LD;  // [KNN_C][KNN_LD]
  const int t = threadIdx.x;
  const int q0 = blockIdx.x * KNN_Q, q = knn_query(qlist, nq, q0 + t);
  float bd[KNN_MAXK];
  int bi[KNN_MAXK];
  int cnt = 0;
  float thr = INFINITY;
  int thi = 0x7fffffff;
  for (int c0 = 0; c0 < n; c0 += KNN_C) {
    float acc[KNN_C];
#pragma unroll
    for (int c = 0; c < KNN_C; c++) acc[c] = 0.f;
    for (int k0 = 0; k0 < dim; k0 += KNN_DC) {
      __syncthreads();
      for (int e = t; e < KNN_Q * KNN_DC; e += KNN_Q) {
        const int r = e / KNN_DC, cc = e % KNN_DC;
        const int gq = knn_query(qlist, nq, q0 + r), gk = k0 + cc;
        sQ[r * KNN_LD + cc] = (gq >= 0 && gk < dim) ? X[(long)gq * dim + gk] : 0.f;
      }
      for (int e = t; e < KNN_C * KNN_DC; e += KNN_Q) {
        const int r = e / KNN_DC, cc = e % KNN_DC;
        const int gc = c0 + r, gk = k0 + cc;
        sC[r * KNN_LD + cc] = (gc < n && gk < dim) ? X[(long)gc * dim + gk] : 0.f;
      }
      __syncthreads();
      const int kmax = min(KNN_DC, dim - k0);  // zero padding adds nothing
      for (int kk = 0; kk < kmax; kk += 4) {
        const float4 qv = *reinterpret_cast<const float4 *>(&sQ[t * KNN_LD + kk]);
#pragma unroll
        for (int c = 0; c < KNN_C; c++) {
          const float4 cv = *reinterpret_cast<const float4 *>(&sC[c * KNN_LD + kk]);
          float df = qv.x - cv.x;
          acc[c] = fmaf(df, df, acc[c]);
          df = qv.y - cv.y;
          acc[c] = fmaf(df, df, acc[c]);
          df = qv.z - cv.z;
          acc[c] = fmaf(df, df, acc[c]);
          df = qv.w - cv.w;
          acc[c] = fmaf(df, df, acc[c]);
        }
      }
    }
    if (q >= 0) {
#pragma unroll
      for (int c = 0; c < KNN_C; c++) {
        const int j = c0 + c;
        const float dd = acc[c];
        if (j >= n || j == q) continue;
        if (cnt == k && !knn_less(dd, j, thr, thi)) continue;
        // insert into the sorted list (drop the last when full)
        int p = cnt < k ? cnt : k - 1;
        while (p > 0 && knn_less(dd, j, bd[p - 1], bi[p - 1])) {
          bd[p] = bd[p - 1];
          bi[p] = bi[p - 1];
          p--;
        }
        bd[p] = dd;
        bi[p] = j;
        if (cnt < k) cnt++;
        if (cnt == k) {
          thr = bd[k - 1];
          thi = bi[k - 1];
        }
      }
    }
  }
  if (q >= 0) {
    for (int s = 0; s < k; s++) {
      idx[(long)q * k + s] = s < cnt ? bi[s] : -1;
      d2[(long)q * k + s] = s < cnt ? bd[s] : INFINITY;
    }
  }
}


// ---------------------------------------------------------------------------
// Tensor-core filter.
//
// q.c - |c|^2/2 = (|q|^2 - d^2)/2 ranks the candidates c of a query q: one dot
// product of (q, 1, 1, 1) and (c, the three BF16 terms of -|c|^2/2).  The
// products run on the tensor cores as BF16 MMAs (kind::f16) in three terms,
// hi.hi + hi.lo + lo.hi with x = hi + lo + e, hi = bf16(x), lo = bf16(x - hi),
// |e| <= 2^-18 |x|, FP32 accumulation in tensor memory; points that are BF16
// numbers themselves (8-bit images) have zero low parts and take the first
// term alone.  The list of nearest candidates under these keys is re-ranked
// with the exact arithmetic of k_knn (sums of squared differences in dimension
// order), so returned distances are bit-identical to it.  A query whose list
// could miss a true neighbour is redone by k_knn: the nearest candidate ever
// dropped, less the bound EPS (|q|^2 + max |c|^2) on a key's error and the
// rounding of a returned distance (both in sgt_knn_rules.h), has to lie beyond
// the k-th distance.
//
// Lists: a query's candidates are scanned by two threads (one per half of
// each tile's columns), each with an unordered buffer of CAP entries in L2.
// A key above the thread's threshold is appended; when a buffer is nearly
// full its warp selects the L best by a bitwise search for the L-th key
// (E = CAP / 32 entries a lane, one warp-wide count per bit) and that key
// becomes the threshold.  CAP / L = 3 to 4 times as many candidates are seen
// between selections each time, so a query needs a handful of them, and the
// scan of a tile is a load, an add and a compare per candidate.  (Lists kept
// sorted or with their maximum at hand in registers cost a serial pass per
// candidate admitted, with the whole block waiting: 12 ms per wave of query
// blocks, 62 ms of 62 at 100,000 points.)
//
// Operands: blocks of 128 query rows and 256 candidate rows are stored once
// as images of their shared-memory tiles: K-major, no swizzle, core matrices
// of 8 rows x 16 bytes (8 dimensions), unit u of all rows contiguous, hi and
// lo parts one after the other.  Points of up to 64 dimensions keep the query
// image resident and stream candidate tiles; wider points stream both in
// chunks of 64 dimensions.  One thread issues the copies, one the MMAs; each
// 128 x 256 tile accumulates into one of two halves of tensor memory while
// eight warps scan the other.
//
// Descriptor fields follow the PTX ISA's tcgen05 shared-memory and
// instruction descriptors (the same bit layout as CUTLASS's
// cute::UMMA::SmemDescriptor and UMMA::InstrDescriptor): start address,
// leading and stride byte offsets in 16-byte units, version 1 at bit 46,
// no swizzle; D format F32 at bit 4, A and B formats BF16 (1) at bits 7 and
// 10, both K-major, N/8 at bit 17 and M/16 at bit 24.
constexpr int KNN_TC_M = 128;      // queries per block
constexpr int KNN_TC_N = 256;      // candidates per tile
constexpr int KNN_TC_RES = 8;      // units (of 8 dimensions) up to which a query image is resident
constexpr int KNN_TC_MAXK = 32;    // limits of SGT_KNN_TENSOR
constexpr int KNN_TC_MAXDIM = 64;
constexpr int KNN_TC_SCAN = 256;   // scanning threads; two more warps issue MMAs and copies
constexpr int KNN_TC_THREADS = KNN_TC_SCAN + 64;
constexpr unsigned KNN_TC_SMEM = 192 * 1024;

// shared-memory matrix descriptor: K-major, no swizzle
__device__ __forceinline__ unsigned long long umma_desc(unsigned addr, unsigned lbo,
                                                        unsigned sbo) {
  return (unsigned long long)((addr >> 4) & 0x3FFFu) |
         ((unsigned long long)((lbo >> 4) & 0x3FFFu) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
__device__ __forceinline__ void umma_bf16(unsigned dtmem, unsigned long long a,
                                          unsigned long long b, unsigned idesc, unsigned acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(dtmem), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// bounded wait that also ends when another thread of the block gave up
__device__ __forceinline__ bool mbar_wait_or(unsigned bar, unsigned parity, volatile int *gave_up) {
  const long long t0 = clock64();
  while (true) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (*gave_up) return false;
    if (clock64() - t0 > SGT_SPIN_CYCLES) {
      *gave_up = 1;
      return false;
    }
  }
}
// starts a load of 32 columns; tmem_wait before the values are used
__device__ __forceinline__ void tmem_ld32(unsigned taddr, float *v) {
  unsigned r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, "
      "%28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
#pragma unroll
  for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
}
// waits for the loads in flight; v (their destination) is not read before
__device__ __forceinline__ void tmem_wait(float *v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; j++) asm volatile("" : "+f"(v[j]));
}

// BF16 (round to nearest even) of a float, as its upper 16 bits; inf and NaN
// keep their meaning
__device__ __forceinline__ unsigned bf16_bits(float x) {
  return (unsigned)__bfloat16_as_ushort(__float2bfloat16_rn(x));
}
__device__ __forceinline__ float bf16_value(unsigned b) { return __uint_as_float(b << 16); }

// squared norms (FP64 sums, rounded to FP32: an FP32 sum's error grows with the
// width, past a distance that is small against the norms), their maximum, and
// whether some coordinate is no BF16 number
__global__ void k_knn_norms(const float *__restrict__ X, int n, int dim, float *__restrict__ nrm,
                            unsigned *__restrict__ nmax, int *__restrict__ inexact) {
  __shared__ float tile[8][32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // a warp takes 32 points; 32 x 32 tiles turn coalesced loads into a
  // point per lane
  for (int i0 = (blockIdx.x * 8 + w) * 32; i0 < n; i0 += gridDim.x * 256) {
    double sum = 0.0;
    bool low = false;
    for (int k0 = 0; k0 < dim; k0 += 32) {
      __syncwarp();
      for (int r = 0; r < 32; r++)
        tile[w][r][lane] = i0 + r < n && k0 + lane < dim ? X[(long)(i0 + r) * dim + k0 + lane] : 0.f;
      __syncwarp();
      for (int kk = 0; kk < min(32, dim - k0); kk++) {
        const float x = tile[w][lane][kk];
        sum = fma((double)x, (double)x, sum);
        low |= bf16_value(bf16_bits(x)) != x;
      }
    }
    const int i = i0 + lane;
    const float s = (float)sum;
    if (i < n) nrm[i] = s;
    // non-negative floats order as integers (a NaN norm as the largest)
    const unsigned m = __reduce_max_sync(0xffffffffu, i < n ? __float_as_uint(s) : 0u);
    if (lane == 0) atomicMax(nmax, m);
    if (__any_sync(0xffffffffu, low) && lane == 0) *inexact = 1;
  }
}

// hi/lo images of the points in blocks of `rows` ([block][part][unit][row],
// 8 dimensions of 2 bytes), as queries (ones in columns dim .. dim + 2 of the
// hi part) or candidates (-|c|^2/2 in three BF16 terms there).  Unused columns
// and rows past n are zero, but candidate rows past n have -inf in column dim of
// the hi part: their key is -inf in one term, and NaN in three (the lo part of a
// query is 0 there). No threshold admits either: keys are taken by v > threshold.
__global__ void k_knn_split(const float *__restrict__ X, const float *__restrict__ nrm, int n,
                            int dim, int U, int rows, int nblk, int candidates,
                            uint4 *__restrict__ img) {
  const long total = (long)nblk * rows * U;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total;
       e += (long)gridDim.x * blockDim.x) {
    const int row = (int)(e % rows);
    const int u = (int)((e / rows) % U);
    const int b = (int)(e / ((long)rows * U));
    const int i = b * rows + row;
    unsigned h[8], l[8];
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const int kk = 8 * u + c;
      const float x = i < n && kk < dim ? X[(long)i * dim + kk] : 0.f;
      h[c] = bf16_bits(x);
      l[c] = bf16_bits(x - bf16_value(h[c]));
      if (kk >= dim && kk < dim + 3) {
        if (!candidates) {
          h[c] = i < n ? 0x3f80u : 0u;  // 1
        } else if (i >= n) {
          h[c] = kk == dim ? 0xff80u : 0u;  // -inf
        } else {
          const float a = -0.5f * nrm[i];
          const float h1 = bf16_value(bf16_bits(a)), r1 = a - h1;
          const float h2 = bf16_value(bf16_bits(r1));
          h[c] = kk == dim ? bf16_bits(a) : (kk == dim + 1 ? bf16_bits(r1) : bf16_bits(r1 - h2));
        }
        l[c] = 0u;
      }
    }
    uint4 vh, vl;
    vh = make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
    vl = make_uint4(l[0] | l[1] << 16, l[2] | l[3] << 16, l[4] | l[5] << 16, l[6] | l[7] << 16);
    const long base = (long)b * 2 * U * rows + (long)u * rows + row;
    img[base] = vh;
    img[base + (long)U * rows] = vl;
  }
}

// floats as unsigned integers in the same order
__device__ __forceinline__ unsigned knn_ordered(float x) {
  const unsigned b = __float_as_uint(x);
  return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float knn_unordered(unsigned u) {
  return __uint_as_float((u >> 31) ? u ^ 0x80000000u : ~u);
}

// The largest T with at least `want` of the warp's entries u >= T (entries of
// value 0 are empty; more than `want` are not), stopping early when exactly
// `want` reach it.
template <int E>
__device__ __forceinline__ unsigned knn_kth(const unsigned *u, int want) {
  // the bits that all entries share need no search
  unsigned hi = 0, lo = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < E; i++) {
    hi = max(hi, u[i]);
    lo = min(lo, u[i] - 1u);  // an empty entry becomes the largest number
  }
  hi = __reduce_max_sync(0xffffffffu, hi);
  lo = __reduce_min_sync(0xffffffffu, lo) + 1u;
  const int top = 31 - __clz((int)(hi ^ lo));  // -1: all equal
  unsigned T = top < 0 ? hi : hi & ~((2u << top) - 1u);
  for (int bit = top; bit >= 0; bit--) {
    const unsigned trial = T | (1u << bit);
    unsigned c = 0;
#pragma unroll
    for (int i = 0; i < E; i++) c += u[i] >= trial;
    c = __reduce_add_sync(0xffffffffu, c);
    if ((int)c >= want) T = trial;
    if ((int)c == want) break;
  }
  return T;
}

// One warp keeps the L best of a buffer's cnt > L entries, in place; returns
// the threshold: no dropped key is above it.
template <int L, int CAP>
__device__ __forceinline__ float knn_select(float2 *buf, int cnt) {
  constexpr int E = CAP / 32;
  const int lane = threadIdx.x & 31;
  float2 v[E];
  unsigned u[E];
#pragma unroll
  for (int i = 0; i < E; i++) {
    const int e = lane + 32 * i;
    v[i] = e < cnt ? buf[e] : make_float2(-INFINITY, 0.f);
    u[i] = e < cnt ? knn_ordered(v[i].x) : 0u;
  }
  const unsigned T = knn_kth<E>(u, L);
  __syncwarp();
  // all above T, then as many of those equal to it as fit
  int at = 0;
#pragma unroll
  for (int pass = 0; pass < 2; pass++)
#pragma unroll
    for (int i = 0; i < E; i++) {
      const bool keep = pass == 0 ? u[i] > T : u[i] == T;
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      const int slot = at + __popc(m & ((1u << lane) - 1u));
      if (keep && slot < L) buf[slot] = v[i];
      at += __popc(m);
    }
  __syncwarp();
  return knn_unordered(T);
}

// Exact distances of m candidates to query q by one warp: d[e] is candidate
// e's sum of squared differences in dimension order, as k_knn forms it.  A
// lane's sum is a serial chain over its candidate's row; read by the lanes
// themselves, 32 rows make 32 cache lines per request, and the L1 tag rate
// bound the filter's tail (1.3 ms per wave of query blocks of 784 dimensions
// and k = 90, 0.65 now: 60,000 points 20.4 -> 12.6 ms; 100,000 points of 50
// dimensions 12.9 -> 11.4 ms).  So runs of KNN_RR_W dimensions of 32 candidates and the query are
// copied to shared memory by lanes side by side, KNN_RR_ST - 1 runs ahead.
constexpr int KNN_RR_W = 32;              // dimensions per run
constexpr int KNN_RR_LD = KNN_RR_W + 4;   // row pitch in floats: float4 reads without conflicts
constexpr int KNN_RR_ST = 5;              // runs in flight
constexpr unsigned KNN_RR_BYTES = 24 * 1024;  // a warp's share of the operand memory
static_assert(KNN_RR_ST * 33 * KNN_RR_LD * 4 <= KNN_RR_BYTES && 8 * KNN_RR_BYTES <= KNN_TC_SMEM,
              "re-rank staging");

// global -> shared copy of B bytes; zeros when !in
template <int B>
__device__ __forceinline__ void cp_async(unsigned dst, const float *src, bool in) {
  if constexpr (B == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                 "r"(in ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(B),
                 "r"(in ? B : 0) : "memory");
}
// rows 0..31: candidates list[0..31], row 32: the query; dimensions k0 ..
// k0 + KNN_RR_W - 1, zeros from dim
template <int F>
__device__ __forceinline__ void knn_stage(const float *__restrict__ X, int dim, int q,
                                          const int *list, int k0, unsigned dst) {
  constexpr int PER = KNN_RR_W / F, ROWS = 32 / PER;  // lanes per row, rows per request
  const int lane = threadIdx.x & 31, r0 = lane / PER, kk = k0 + (lane % PER) * F;
  const bool in = kk < dim;
  const float *src = X + (in ? kk : 0);
  dst += (r0 * KNN_RR_LD + (lane % PER) * F) * 4u;
#pragma unroll 8
  for (int r = 0; r < 32; r += ROWS)
    cp_async<4 * F>(dst + r * (KNN_RR_LD * 4u), src + (long)list[r + r0] * dim, in);
  if (r0 == 0) cp_async<4 * F>(dst + 32 * (KNN_RR_LD * 4u), src + (long)q * dim, in);
}
// (list has entries to the next multiple of 32 from m)
__device__ __forceinline__ void knn_rerank(const float *__restrict__ X, int dim, int q, int m,
                                           const int *list, float *d, float *stage) {
  const int lane = threadIdx.x & 31;
  const int nrun = (dim + KNN_RR_W - 1) / KNN_RR_W, total = nrun * ((m + 31) / 32);
  const size_t xa = reinterpret_cast<size_t>(X);
  // floats per copy: rows start on multiples of it
  const int f = (dim & 3) == 0 && (xa & 15) == 0 ? 4 : ((dim & 1) == 0 && (xa & 7) == 0 ? 2 : 1);
  int ic = 0, ik = 0, is = 0;  // next run to issue: first candidate, first dimension, stage
  auto issue = [&](int s) {
    if (s < total) {
      const unsigned dst = smem_u32(stage + is * 33 * KNN_RR_LD);
      if (f == 4) knn_stage<4>(X, dim, q, list + ic, ik, dst);
      else if (f == 2) knn_stage<2>(X, dim, q, list + ic, ik, dst);
      else knn_stage<1>(X, dim, q, list + ic, ik, dst);
      ik += KNN_RR_W;
      if (ik >= dim) { ik = 0; ic += 32; }
      if (++is == KNN_RR_ST) is = 0;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int s = 0; s < KNN_RR_ST - 1; s++) issue(s);
  int cc = 0, ck = 0, cs = 0;
  float acc = 0.f;
  for (int s = 0; s < total; s++) {
    issue(s + KNN_RR_ST - 1);  // into the stage read last
    asm volatile("cp.async.wait_group %0;" ::"n"(KNN_RR_ST - 1) : "memory");
    __syncwarp();
    const float *b = stage + cs * 33 * KNN_RR_LD, *mine = b + lane * KNN_RR_LD,
                *qr = b + 32 * KNN_RR_LD;
    const int w = min(KNN_RR_W, dim - ck);  // zero padding adds nothing
#pragma unroll 8
    for (int kk = 0; kk < w; kk += 4) {
      const float4 a = *reinterpret_cast<const float4 *>(qr + kk);
      const float4 c = *reinterpret_cast<const float4 *>(mine + kk);
      float df = a.x - c.x;
      acc = fmaf(df, df, acc);
      df = a.y - c.y;
      acc = fmaf(df, df, acc);
      df = a.z - c.z;
      acc = fmaf(df, df, acc);
      df = a.w - c.w;
      acc = fmaf(df, df, acc);
    }
    ck += KNN_RR_W;
    if (++cs == KNN_RR_ST) cs = 0;
    if (ck >= dim) {
      if (cc + lane < m) d[cc + lane] = acc;
      acc = 0.f;
      ck = 0;
      cc += 32;
    }
    __syncwarp();
  }
}

// A block walks over query blocks; warps 0-7 scan (warp w: rows 32 (w & 3)..,
// columns 128 (w >> 2)..), lane 0 of warp 8 issues the MMAs, lane 0 of warp 9
// the copies.
template <int L, int CAP>
__global__ void __launch_bounds__(KNN_TC_THREADS, 1)
k_knn_tc(const unsigned char *__restrict__ imgA, const unsigned char *__restrict__ imgB,
         const float *__restrict__ nrm,
         const unsigned *__restrict__ nmax, const int *__restrict__ inexact,
         const float *__restrict__ X, int n, int dim, int U, int k, float2 *__restrict__ bufs,
         int *__restrict__ idx, float *__restrict__ d2, int *__restrict__ redo,
         int *__restrict__ nredo, int *__restrict__ err) {
  extern __shared__ __align__(1024) unsigned char smem[];
  // full x8, empty x8, accumulator full x2, empty x2, resident A
  __shared__ __align__(8) unsigned long long bars[21];
  __shared__ unsigned tslot;
  __shared__ volatile int gave_up;
  __shared__ int s_cnt[KNN_TC_SCAN];
  __shared__ float s_thr[KNN_TC_SCAN];
  __shared__ volatile float s_live[KNN_TC_SCAN];
  __shared__ int s_idx[8][L];
  __shared__ float s_d[8][L];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int nq = (n + KNN_TC_M - 1) / KNN_TC_M, ntile = (n + KNN_TC_N - 1) / KNN_TC_N;
  const int ku = U <= KNN_TC_RES ? 4 : 8, nch = (U + ku - 1) / ku;  // units and number of chunks
  const unsigned apart = ku * KNN_TC_M * 16u, bpart = ku * KNN_TC_N * 16u;
  const bool three = *inexact != 0, resident = U <= KNN_TC_RES;
  const int parts = three ? 2 : 1;
  const unsigned sm0 = smem_u32(smem);
  const unsigned a_bytes = resident ? 0u : parts * apart;
  const unsigned st_bytes = a_bytes + parts * bpart;
  const unsigned res_part = (unsigned)U * KNN_TC_M * 16u;  // a part of a resident query image
  const unsigned st0 = sm0 + (resident ? parts * res_part : 0u);
  const int nst = min(8, (int)((sm0 + KNN_TC_SMEM - st0) / st_bytes));
  auto bar_full = [&](int st) { return smem_u32(&bars[st]); };
  auto bar_free = [&](int st) { return smem_u32(&bars[8 + st]); };
  auto bar_acc = [&](int b) { return smem_u32(&bars[16 + b]); };
  auto bar_scan = [&](int b) { return smem_u32(&bars[18 + b]); };
  const unsigned bar_a = smem_u32(&bars[20]);
  if (t == 0) {
    gave_up = 0;
    for (int b = 0; b < 21; b++) mbar_init(smem_u32(&bars[b]), b == 18 || b == 19 ? 8 : 1);
    mbar_fence_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tslot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = tslot;
  const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((KNN_TC_N >> 3) << 17) |
                         ((KNN_TC_M >> 4) << 24);
  const float eps = sgt_knn_eps(dim, !three), gamma = sgt_knn_gamma(dim),
              cmax = __uint_as_float(*nmax);
  // places that run on over all query blocks: stage of the copies, stage of the
  // MMAs, accumulator (of the MMAs or of the scan)
  SgtRing load, step, acc;
  unsigned blocks = 0;
  for (int qb = blockIdx.x; qb < nq; qb += gridDim.x, blocks++) {
    const unsigned total = (unsigned)ntile * (unsigned)nch;  // pipeline steps of a query block
    if (warp == 9) {
      if (lane == 0) {  // copies: step g is chunk g % nch of tile g / nch
        bool ok = true;
        if (resident) {
          // every MMA of the last query block has been waited for (its tiles
          // were scanned), so its image can be replaced
          mbar_expect_tx(bar_a, parts * res_part);
          for (int p = 0; p < parts; p++)
            bulk_g2s(sm0 + p * res_part, imgA + ((size_t)qb * 2 + p) * res_part, res_part, bar_a);
        }
        for (unsigned g = 0; g < total; g++, load.next(nst)) {
          const int st = load.at;
          ok = mbar_wait_or(bar_free(st), load.phase ^ 1u, &gave_up);
          if (!ok) break;
          const int tile = (int)(g / (unsigned)nch), ch = (int)(g % (unsigned)nch);
          const int uc = min(ku, U - ch * ku);
          const unsigned sb = st0 + st * st_bytes;
          mbar_expect_tx(bar_full(st), parts * uc * 16u * (KNN_TC_N + (resident ? 0 : KNN_TC_M)));
          for (int p = 0; p < parts; p++) {
            if (!resident)
              bulk_g2s(sb + p * apart, imgA + (((size_t)qb * 2 + p) * U + ch * ku) * KNN_TC_M * 16,
                       uc * KNN_TC_M * 16u, bar_full(st));
            bulk_g2s(sb + a_bytes + p * bpart,
                     imgB + (((size_t)tile * 2 + p) * U + ch * ku) * KNN_TC_N * 16,
                     uc * KNN_TC_N * 16u, bar_full(st));
          }
        }
      }
    } else if (warp == 8) {
      if (lane == 0) {  // MMAs
        bool ok = true;
        if (resident) ok = mbar_wait_or(bar_a, blocks & 1, &gave_up);
        for (unsigned g = 0; g < total && ok; g++) {
          const int st = step.at, ch = (int)(g % (unsigned)nch), ab = acc.at;
          if (ch == 0)  // the accumulator has been scanned
            ok = mbar_wait_or(bar_scan(ab), acc.phase ^ 1u, &gave_up);
          ok = ok && mbar_wait_or(bar_full(st), step.phase, &gave_up);
          if (!ok) break;
          tc_fence_after();
          const unsigned sb = st0 + st * st_bytes;
          const unsigned aa = resident ? sm0 + ch * apart : sb, bb = sb + a_bytes;
          const unsigned alo = resident ? res_part : apart;
          const int ks = min(ku, U - ch * ku) / 2;
          const unsigned dt = tmem + (unsigned)ab * KNN_TC_N;
          for (int term = 0; term < (three ? 3 : 1); term++) {
            // hi.hi, hi.lo, lo.hi; a K step of 16 dimensions is two units
            unsigned long long da = umma_desc(aa + (term == 2 ? alo : 0u), KNN_TC_M * 16, 128);
            unsigned long long db = umma_desc(bb + (term == 1 ? bpart : 0u), KNN_TC_N * 16, 128);
            for (int s = 0; s < ks; s++) {
              umma_bf16(dt, da, db, idesc, ch > 0 || term > 0 || s > 0 ? 1u : 0u);
              da += 2 * KNN_TC_M;
              db += 2 * KNN_TC_N;
            }
          }
          umma_commit(bar_free(st));
          step.next(nst);
          if (ch == nch - 1) {
            umma_commit(bar_acc(ab));
            acc.next(2);
          }
        }
      }
    } else {
      const int row = (warp & 3) * 32 + lane, half = warp >> 2;
      const int q = qb * KNN_TC_M + row;
      float2 *buf = bufs + ((size_t)blockIdx.x * KNN_TC_SCAN + t) * CAP;
      float2 *wbuf = bufs + ((size_t)blockIdx.x * KNN_TC_SCAN + warp * 32) * CAP;
      float thr = q < n ? -INFINITY : INFINITY;
      int cnt = 0;
      bool ok = true;
      s_live[t] = -INFINITY;
      asm volatile("bar.sync 1, %0;" ::"n"(KNN_TC_SCAN) : "memory");  // the scanning warps
      for (int tile = 0; tile < ntile; tile++, acc.next(2)) {
        const int ab = acc.at;
        ok = __all_sync(0xffffffffu, mbar_wait_or(bar_acc(ab), acc.phase, &gave_up));
        if (!ok) break;
        tc_fence_after();
        // L keys of the other half of the query's columns lie above its
        // threshold: what is not above that is no neighbour either
        thr = fmaxf(thr, s_live[t ^ 128]);
        const unsigned tcol = tmem + ((unsigned)((warp & 3) * 32) << 16) +
                              (unsigned)ab * KNN_TC_N + (unsigned)half * 128u;
        float v[32], nv[32];
        __syncwarp();
        tmem_ld32(tcol, nv);
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += 32) {
          tmem_wait(nv);
#pragma unroll
          for (int h = 0; h < 32; h++) v[h] = nv[h];
          __syncwarp();
          if (c0 < 96) tmem_ld32(tcol + (unsigned)c0 + 32u, nv);  // in flight meanwhile
          const int j0 = tile * KNN_TC_N + half * 128 + c0;
          // by all 32 columns, then by fours: a warp seldom has a key to append
          // once the lists have settled
          float m4[8];
#pragma unroll
          for (int h = 0; h < 8; h++)
            m4[h] = fmaxf(fmaxf(v[4 * h], v[4 * h + 1]), fmaxf(v[4 * h + 2], v[4 * h + 3]));
          const float m32 = fmaxf(fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])),
                                  fmaxf(fmaxf(m4[4], m4[5]), fmaxf(m4[6], m4[7])));
          if (!__any_sync(0xffffffffu, m32 > thr)) continue;
#pragma unroll
          for (int h = 0; h < 8; h++)
            if (__any_sync(0xffffffffu, m4[h] > thr)) {
#pragma unroll
              for (int g = 4 * h; g < 4 * h + 4; g++)
                if (v[g] > thr) buf[cnt++] = make_float2(v[g], __int_as_float(j0 + g));
            }
          // room for the next 32 columns
          unsigned full = __ballot_sync(0xffffffffu, cnt > CAP - 32);
          while (full) {
            const int s = __ffs(full) - 1;
            full &= full - 1;
            const int c = __shfl_sync(0xffffffffu, cnt, s);
            __syncwarp();
            const float nt = knn_select<L, CAP>(wbuf + (size_t)s * CAP, c);
            if (lane == s) {
              cnt = L;
              thr = fmaxf(thr, nt);
              s_live[t] = thr;
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_scan(ab));
      }
      s_cnt[t] = cnt;
      s_thr[t] = thr;
      if (!ok) gave_up = 1;
    }
    __syncthreads();
    if (gave_up) break;  // block-uniform: written before the barrier
    if (warp < 8) {
      // re-rank: a warp per query.  All copies into the operand memory and all
      // MMAs that read it have been waited for; the warps share it.
      float *stage = reinterpret_cast<float *>(smem + warp * KNN_RR_BYTES);
      for (int r = warp; r < KNN_TC_M; r += 8) {
        const int q = qb * KNN_TC_M + r;
        if (q >= n) break;
        constexpr int E = CAP / 32;
        const float2 *b0 = bufs + ((size_t)blockIdx.x * KNN_TC_SCAN + r) * CAP;
        const float2 *b1 = b0 + (size_t)128 * CAP;
        const int c0 = s_cnt[r], c1 = s_cnt[128 + r];
        float tail = fmaxf(s_thr[r], s_thr[128 + r]);  // no dropped key is above it
        unsigned u[2 * E];
        int j[2 * E];
#pragma unroll
        for (int i = 0; i < 2 * E; i++) {
          const int e = lane + 32 * (i % E);
          const bool in = e < (i < E ? c0 : c1);
          const float2 v = in ? (i < E ? b0 : b1)[e] : make_float2(0.f, 0.f);
          j[i] = __float_as_int(v.y);
          u[i] = in && j[i] != q ? knn_ordered(v.x) : 0u;  // without the query itself
        }
        unsigned T = 1;  // everything
        const int have = c0 + c1;
        if (have > L) {
          T = knn_kth<2 * E>(u, L);
          if (T == 0) T = 1;  // fewer than L entries besides the query
          else tail = fmaxf(tail, knn_unordered(T));
        }
        // only a candidate whose key is within the bound of the k-th key can
        // be among the k nearest: those of the k best keys have distances of
        // at most far, times 1 + gamma as they are formed (a NaN bound keeps
        // all)
        // (products may lose terms below the smallest normal number: 1e-37 a
        // dimension covers them)
        const float qn = nrm[q], bound = eps * (qn + cmax) + 1e-37f * (float)dim;
        if (have > k) {
          const unsigned K = knn_kth<2 * E>(u, k);
          const float kth = knn_unordered(K), far = fmaxf(qn - 2.f * kth + bound, 0.f);
          const unsigned cut = K == 0 ? 0u : knn_ordered(kth - (bound + 1.1f * gamma * far));
          if (bound == bound && cut > T && cut <= K) T = cut;
        }
        int m = 0;
        __syncwarp();
#pragma unroll
        for (int pass = 0; pass < 2; pass++)
#pragma unroll
          for (int i = 0; i < 2 * E; i++) {
            const bool keep = pass == 0 ? u[i] > T : u[i] == T;
            const unsigned mk = __ballot_sync(0xffffffffu, keep);
            const int slot = m + __popc(mk & ((1u << lane) - 1u));
            if (keep && slot < L) s_idx[warp][slot] = j[i];
            m += __popc(mk);
          }
        m = min(m, L);
        if (m + lane < (m + 31) / 32 * 32) s_idx[warp][m + lane] = q;
        __syncwarp();
        knn_rerank(X, dim, q, m, s_idx[warp], s_d[warp], stage);
        __syncwarp();
        // the k nearest by (distance, index): each entry's rank is the number
        // of entries before it
        float dk = INFINITY;
        for (int e = lane; e < m; e += 32) {
          const float d = s_d[warp][e];
          const int ji = s_idx[warp][e];
          int rank = 0;
          for (int o = 0; o < m; o++) rank += knn_less(s_d[warp][o], s_idx[warp][o], d, ji);
          if (rank < k) {
            idx[(long)q * k + rank] = ji;
            d2[(long)q * k + rank] = d;
          }
          if (rank == k - 1) dk = d;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dk = fminf(dk, __shfl_xor_sync(0xffffffffu, dk, o));
        // settled: nothing was dropped, or the distance of all that was, as it
        // would be formed, is larger than the k-th (false for NaN: such queries
        // are redone too)
        const float near = qn - 2.f * tail - bound;
        const bool settled = m >= k && ((tail == -INFINITY && bound < INFINITY) ||
                                        near - 1.1f * gamma * near > dk);
        if (!settled && lane == 0) redo[atomicAdd(nredo, 1)] = q;
        __syncwarp();
      }
    }
    // order this memory's plain accesses before the next block's bulk copies
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // the lists are free for the next query block
  }
  if (gave_up) {
    // let the copies and MMAs in flight finish before the memory is released
    if (t == KNN_TC_SCAN + 32) {
      atomicExch(err, 1);
      if (resident) mbar_wait(bar_a, blocks & 1);  // (issued as this query block began)
      while (load.back(nst)) mbar_wait(bar_full(load.at), load.phase);
    }
    // MMAs complete in order: the last step's commit and the last tile's
    if (t == KNN_TC_SCAN) {
      if (step.back(nst)) mbar_wait(bar_free(step.at), step.phase);
      if (acc.back(2)) mbar_wait(bar_acc(acc.at), acc.phase);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

}  // namespace

static sgt_status knn_simt(sgt_ctx *ctx, int n, int dim, const float *X, int k,
                           const int *qlist, int nq, int *idx, float *d2) {
  const size_t smem = sizeof(float) * (size_t)(KNN_Q + KNN_C) * KNN_LD;
  cudaError_t e = cudaFuncSetAttribute(k_knn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e == cudaSuccess && nq > 0) {
    const int nb = (nq + KNN_Q - 1) / KNN_Q;
    k_knn<<<nb, KNN_Q, smem, sgti_stream(ctx)>>>(X, n, dim, k, qlist, nq, idx, d2);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess)
    return sgti_fail(ctx, SGT_ERR_CUDA, std::string("sgt_knn: ") + cudaGetErrorString(e));
  return SGT_OK;
}

template <int L, int CAP>
static cudaError_t knn_tc_launch(int nb, cudaStream_t s, const unsigned char *imgA,
                                 const unsigned char *imgB, const float *nrm,
                                 const unsigned *nmax, const int *inexact, const float *X, int n,
                                 int dim, int U, int k, float2 *bufs, int *idx, float *d2,
                                 int *redo, int *cnt) {
  cudaError_t e = cudaFuncSetAttribute(
      k_knn_tc<L, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KNN_TC_SMEM);
  if (e != cudaSuccess) return e;
  k_knn_tc<L, CAP><<<nb, KNN_TC_THREADS, KNN_TC_SMEM, s>>>(
      imgA, imgB, nrm, nmax, inexact, X, n, dim, U, k, bufs, idx, d2, redo, cnt, cnt + 1);
  return cudaGetLastError();
}

static sgt_status knn_tc(sgt_ctx *ctx, int n, int dim, const float *X, int k, int *idx,
                         float *d2, int *n_redo) {
  cudaStream_t s = sgti_stream(ctx);
  // units of 8 dimensions, in pairs (one MMA): the dimensions and three columns
  const int U = ((dim + 3 + 15) / 16) * 2;
  const int nq = (n + KNN_TC_M - 1) / KNN_TC_M, ntile = (n + KNN_TC_N - 1) / KNN_TC_N;
  const size_t a_bytes = (size_t)nq * 2 * U * KNN_TC_M * 16;
  const size_t b_bytes = (size_t)ntile * 2 * U * KNN_TC_N * 16;
  const int nb = std::min(nq, sgti_sm_count(ctx));
  // list length (neighbours and a margin) and buffer capacity
  const int cap = k <= 32 ? 256 : (k <= 96 ? 384 : 448);
  char *buf = nullptr;
  const size_t o_nrm = a_bytes + b_bytes;
  const size_t o_buf = o_nrm + sizeof(float) * (((size_t)n + 3) / 4 * 4);
  const size_t o_max = o_buf + sizeof(float2) * (size_t)nb * KNN_TC_SCAN * cap;
  const size_t o_cnt = o_max + 16, o_redo = o_cnt + 16;
  const size_t total = o_redo + sizeof(int) * (size_t)n;
  cudaError_t e = sgti_alloc(ctx, (void **)&buf, total, s);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();  // not sticky: clear it for the caller's next check
    return sgti_fail(ctx, SGT_ERR_NO_MEMORY, "sgt_knn: tensor-core operand images");
  }
  unsigned char *imgA = reinterpret_cast<unsigned char *>(buf);
  unsigned char *imgB = imgA + a_bytes;
  float *nrm = reinterpret_cast<float *>(buf + o_nrm);
  float2 *bufs = reinterpret_cast<float2 *>(buf + o_buf);
  unsigned *nmax = reinterpret_cast<unsigned *>(buf + o_max);
  int *inexact = reinterpret_cast<int *>(buf + o_max + 4);
  int *cnt = reinterpret_cast<int *>(buf + o_cnt);  // [0] queries to redo, [1] error
  int *redo = reinterpret_cast<int *>(buf + o_redo);
  int hc[2] = {0, 0};
  e = cudaMemsetAsync(buf + o_max, 0, 32, s);
  if (e == cudaSuccess) {
    k_knn_norms<<<std::min((n + 255) / 256, 148 * 4), 256, 0, s>>>(X, n, dim, nrm, nmax, inexact);
    k_knn_split<<<148 * 8, 256, 0, s>>>(X, nrm, n, dim, U, KNN_TC_M, nq, 0, (uint4 *)imgA);
    k_knn_split<<<148 * 8, 256, 0, s>>>(X, nrm, n, dim, U, KNN_TC_N, ntile, 1, (uint4 *)imgB);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    if (k <= 32)
      e = knn_tc_launch<64, 256>(nb, s, imgA, imgB, nrm, nmax, inexact, X, n, dim, U, k, bufs,
                                 idx, d2, redo, cnt);
    else if (k <= 96)
      e = knn_tc_launch<128, 384>(nb, s, imgA, imgB, nrm, nmax, inexact, X, n, dim, U, k,
                                  bufs, idx, d2, redo, cnt);
    else
      e = knn_tc_launch<192, 448>(nb, s, imgA, imgB, nrm, nmax, inexact, X, n, dim, U, k,
                                  bufs, idx, d2, redo, cnt);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  sgt_status st = SGT_OK;
  if (e != cudaSuccess)
    st = sgti_fail(ctx, SGT_ERR_CUDA, std::string("sgt_knn: ") + cudaGetErrorString(e));
  else if (hc[1])
    st = sgti_fail(ctx, SGT_ERR_CUDA, "sgt_knn: a tensor-core pipeline wait timed out");
  else
    st = knn_simt(ctx, n, dim, X, k, redo, hc[0], idx, d2);  // queries the filter could not settle
  if (st == SGT_OK && n_redo) *n_redo = hc[0];
  cudaFreeAsync(buf, s);
  return st;
}

extern "C" sgt_status sgt_knn_ex(sgt_ctx *ctx, int n, int dim, const float *X, int k, int *idx,
                                 float *d2, int method, int *n_redo) {
  if (!ctx || !X || !idx || !d2) return SGT_ERR_INVALID_ARG;
  if (n < 2 || dim < 1 || k < 1) return sgti_fail(ctx, SGT_ERR_INVALID_ARG, "sgt_knn: sizes");
  if (method < SGT_KNN_AUTO || method > SGT_KNN_TENSOR)
    return sgti_fail(ctx, SGT_ERR_INVALID_ARG, "sgt_knn: method");
  if (k > KNN_MAXK || k >= n)
    return sgti_fail(ctx, SGT_ERR_UNSUPPORTED,
                     "sgt_knn: k must be below n and at most " + std::to_string(KNN_MAXK));
  const bool tc_ok = dim <= KNN_TC_MAXDIM && k <= KNN_TC_MAXK && n <= (1 << 28);
  if (method == SGT_KNN_TENSOR && !tc_ok)
    return sgti_fail(ctx, SGT_ERR_UNSUPPORTED,
                     "sgt_knn: the tensor-core filter takes dim <= 64 and k <= 32");
  if (cudaSetDevice(sgti_device(ctx)) != cudaSuccess)
    return sgti_fail(ctx, SGT_ERR_CUDA, "sgt_knn: set device");
  if (n_redo) *n_redo = 0;
  sgt_status st;
  if (method == SGT_KNN_TENSOR || (method == SGT_KNN_AUTO && n >= sgt_knn_min_n(dim, k) && n <= (1 << 28))) {
    st = knn_tc(ctx, n, dim, X, k, idx, d2, n_redo);
    // the filter's operand images (about 8 bytes per point and dimension)
    // did not fit: the automatic choice falls back to the SIMT search
    if (st == SGT_ERR_NO_MEMORY && method == SGT_KNN_AUTO)
      st = knn_simt(ctx, n, dim, X, k, nullptr, n, idx, d2);
  } else {
    st = knn_simt(ctx, n, dim, X, k, nullptr, n, idx, d2);
  }
  if (st != SGT_OK) return st;
  // like the other preparation operators, return with the result ready
  const cudaError_t e = cudaStreamSynchronize(sgti_stream(ctx));
  if (e != cudaSuccess)
    return sgti_fail(ctx, SGT_ERR_CUDA, std::string("sgt_knn: ") + cudaGetErrorString(e));
  return SGT_OK;
}

extern "C" sgt_status sgt_knn(sgt_ctx *ctx, int n, int dim, const float *X, int k, int *idx,
                              float *d2) {
  return sgt_knn_ex(ctx, n, dim, X, k, idx, d2, SGT_KNN_AUTO, nullptr);
}
