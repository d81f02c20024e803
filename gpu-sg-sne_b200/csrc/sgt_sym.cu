// sgt_sym.cu -- (P + P^T) * scale on the device, bit-identical to the host
// sgt_symmetrize (CU/graph_rescaling.cu:266-398 builds the same pattern with
// legacy cuSPARSE csrgeam; scale 1/(2n) at CU/graph_rescaling.cu:378-379).
//
// The host version sorts each row of P stably by column, builds P^T by a
// counting sort that visits rows in order, and merges row r of P with row r
// of P^T, taking P's entries first on equal columns and summing equal
// columns in that order.  Here every nonzero t of P (rows in order) emits two
// entries: (r, c) into the first half of a buffer and (c, r) into the second
// half, both halves in t order.  A stable LSD radix sort on the key (row,
// column) then yields, per output row, the host's merge sequence exactly:
// columns ascending, P (the first half) before P^T, input order within each.
// Runs of equal (row, column) are summed one after another in FP32 and scaled,
// as the host does.  The sort is CUB's device radix sort (this is
// preprocessing, not the iteration); its passes over memory bound the whole,
// so a key holds only the bits that n needs, in 32 bits up to n = 65536: 4
// passes over 8 bytes an entry instead of 7 over 12 with 49-bit keys.
#include "../../include/sgtsne_b200.h"
#include "sgt_internal.h"

#include <algorithm>
#include <string>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

namespace {

constexpr int SYM_THREADS = 256;
constexpr int SYM_ROW_BITS = 24;  // n <= 2^24 rows

// A block takes runs of SYM_THREADS nonzeros.  Their rows lie between the rows
// of the run's ends, so only two threads search all of rowptr.
template <typename K>
__global__ void k_sym_emit(int n, long nnz, int bits, const int *__restrict__ rowptr,
                           const int *__restrict__ col, const float *__restrict__ val,
                           K *__restrict__ keys, float *__restrict__ vals,
                           int *__restrict__ bad) {
  __shared__ int ends[2];
  // largest r in [lo, hi) with rowptr[r] <= t
  auto row_of = [&](long t, int lo, int hi) {
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (rowptr[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
  };
  for (long t0 = blockIdx.x * (long)blockDim.x; t0 < nnz; t0 += (long)gridDim.x * blockDim.x) {
    const long tl = min(t0 + (long)blockDim.x, nnz) - 1, t = t0 + threadIdx.x;
    if (threadIdx.x == 0) ends[0] = row_of(t0, 0, n);
    if (threadIdx.x == 32) ends[1] = row_of(tl, 0, n);
    __syncthreads();
    const int first = ends[0], last = ends[1];
    __syncthreads();
    if (t > tl) continue;
    const int r = row_of(t, first, last + 1), c = col[t];
    if (c < 0 || c >= n) {
      atomicOr(bad, 1);
      keys[t] = keys[nnz + t] = 0;
      vals[t] = vals[nnz + t] = 0.f;
      continue;
    }
    const float v = val[t];
    keys[t] = (K)r << bits | (K)c;
    vals[t] = v;
    keys[nnz + t] = (K)c << bits | (K)r;
    vals[nnz + t] = v;
  }
}

// head[i] = 1 where (row, column) changes
template <typename K>
__global__ void k_sym_heads(long m, const K *__restrict__ keys, int *__restrict__ head) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < m;
       i += (long)gridDim.x * blockDim.x)
    head[i] = (i == 0 || keys[i - 1] != keys[i]) ? 1 : 0;
}

// out_rowptr[r]: the run heads before the first key of row r or above (a
// search per row: counting the heads with an atomic each cost a tenth of the
// whole)
template <typename K>
__global__ void k_sym_rowptr(int n, long m, int bits, const K *__restrict__ keys,
                             const int *__restrict__ head, const int *__restrict__ pos,
                             int *__restrict__ out_rowptr) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= n; r += gridDim.x * blockDim.x) {
    long lo = 0, hi = m;  // first i with a row >= r
    while (lo < hi) {
      const long mid = (lo + hi) >> 1;
      if ((int)(keys[mid] >> bits) < r) lo = mid + 1; else hi = mid;
    }
    out_rowptr[r] = lo < m ? pos[lo] : pos[m - 1] + head[m - 1];
  }
}

// run heads sum their run in sorted order and write the output entry
template <typename K>
__global__ void k_sym_reduce(long m, int bits, const K *__restrict__ keys,
                             const float *__restrict__ vals, const int *__restrict__ head,
                             const int *__restrict__ pos, float scale, int *__restrict__ out_col,
                             float *__restrict__ out_val) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < m;
       i += (long)gridDim.x * blockDim.x) {
    if (!head[i]) continue;
    const K k = keys[i];
    float acc = vals[i];
    for (long j = i + 1; j < m && keys[j] == k; j++) acc += vals[j];
    const int p = pos[i];
    out_col[p] = (int)(k & (((K)1 << bits) - 1));
    out_val[p] = acc * scale;
  }
}

// bits a row or column index below n takes (at least one)
int sym_bits(int n) {
  int b = 1;
  while (((n - 1) >> b) != 0) b++;
  return b;
}

template <typename K>
sgt_status sym_run(sgt_ctx *ctx, int n, long nnz, const int *rowptr, const int *col,
                   const float *val, float scale, int *out_rowptr, int *out_col,
                   float *out_val, long *out_nnz) {
  cudaStream_t s = sgti_stream(ctx);
  const long m = 2 * nnz;
  K *k0 = nullptr, *k1 = nullptr;
  float *v0 = nullptr, *v1 = nullptr;
  int *head = nullptr, *pos = nullptr, *bad = nullptr;
  void *tmp = nullptr;
  size_t tmp_sort = 0, tmp_scan = 0;
  cudaError_t e = cudaSuccess;
  auto ok = [&](cudaError_t x) { if (e == cudaSuccess) e = x; return e == cudaSuccess; };
  const int bits = sym_bits(n);
  cub::DeviceRadixSort::SortPairs(nullptr, tmp_sort, k0, k1, v0, v1, (int)m, 0, 2 * bits, s);
  cub::DeviceScan::ExclusiveSum(nullptr, tmp_scan, head, pos, (int)m, s);
  const size_t tmp_bytes = std::max(tmp_sort, tmp_scan);
  ok(sgti_alloc(ctx, (void **)&k0, sizeof(K) * m, s));
  ok(sgti_alloc(ctx, (void **)&k1, sizeof(K) * m, s));
  ok(sgti_alloc(ctx, (void **)&v0, sizeof(float) * m, s));
  ok(sgti_alloc(ctx, (void **)&v1, sizeof(float) * m, s));
  ok(sgti_alloc(ctx, (void **)&head, sizeof(int) * m, s));
  ok(sgti_alloc(ctx, (void **)&pos, sizeof(int) * m, s));
  ok(sgti_alloc(ctx, (void **)&bad, sizeof(int), s));
  ok(sgti_alloc(ctx, (void **)&tmp, tmp_bytes, s));
  int hbad = 0, total = 0;
  if (e == cudaSuccess) {
    const int nb = (int)std::min<long>((nnz + SYM_THREADS - 1) / SYM_THREADS, 148L * 16);
    const int mb = (int)std::min<long>((m + SYM_THREADS - 1) / SYM_THREADS, 148L * 16);
    const int rb = (int)std::min<long>((n + SYM_THREADS) / SYM_THREADS, 148L * 16);
    ok(cudaMemsetAsync(bad, 0, sizeof(int), s));
    if (e == cudaSuccess) {
      k_sym_emit<K><<<nb, SYM_THREADS, 0, s>>>(n, nnz, bits, rowptr, col, val, k0, v0, bad);
      ok(cudaGetLastError());
    }
    size_t tb = tmp_bytes;
    ok(cub::DeviceRadixSort::SortPairs(tmp, tb, k0, k1, v0, v1, (int)m, 0, 2 * bits, s));
    if (e == cudaSuccess) {
      k_sym_heads<K><<<mb, SYM_THREADS, 0, s>>>(m, k1, head);
      ok(cudaGetLastError());
    }
    tb = tmp_bytes;
    ok(cub::DeviceScan::ExclusiveSum(tmp, tb, head, pos, (int)m, s));
    if (e == cudaSuccess) {
      k_sym_rowptr<K><<<rb, SYM_THREADS, 0, s>>>(n, m, bits, k1, head, pos, out_rowptr);
      k_sym_reduce<K><<<mb, SYM_THREADS, 0, s>>>(m, bits, k1, v1, head, pos, scale, out_col,
                                                 out_val);
      ok(cudaGetLastError());
    }
    ok(cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    ok(cudaMemcpyAsync(&total, out_rowptr + n, sizeof(int), cudaMemcpyDeviceToHost, s));
    ok(cudaStreamSynchronize(s));
  }
  for (void *p : {(void *)k0, (void *)k1, (void *)v0, (void *)v1, (void *)head, (void *)pos,
                  (void *)bad, tmp})
    if (p) cudaFreeAsync(p, s);
  if (e != cudaSuccess)
    return sgti_fail(ctx, e == cudaErrorMemoryAllocation ? SGT_ERR_NO_MEMORY : SGT_ERR_CUDA,
                     std::string("sgt_symmetrize_device: ") + cudaGetErrorString(e));
  if (hbad) return sgti_fail(ctx, SGT_ERR_INVALID_ARG, "sgt_symmetrize_device: column out of range");
  *out_nnz = total;
  return SGT_OK;
}

}  // namespace

extern "C" sgt_status sgt_symmetrize_device(sgt_ctx *ctx, int n, long nnz, const int *rowptr,
                                            const int *col, const float *val, float scale,
                                            int *out_rowptr, int *out_col, float *out_val,
                                            long *out_nnz) {
  if (!ctx || !rowptr || !col || !val || !out_rowptr || !out_col || !out_val || !out_nnz)
    return SGT_ERR_INVALID_ARG;
  if (n < 1 || nnz < 0) return SGT_ERR_INVALID_ARG;
  if (n > (1 << SYM_ROW_BITS))
    return sgti_fail(ctx, SGT_ERR_UNSUPPORTED, "sgt_symmetrize_device: n above 2^24");
  if (2 * nnz > 0x7fffffffL)
    return sgti_fail(ctx, SGT_ERR_UNSUPPORTED, "sgt_symmetrize_device: 2 nnz above 2^31");
  cudaStream_t s = sgti_stream(ctx);
  const long m = 2 * nnz;
  if (cudaSetDevice(sgti_device(ctx)) != cudaSuccess)
    return sgti_fail(ctx, SGT_ERR_CUDA, "sgt_symmetrize_device: set device");
  if (m == 0) {
    if (cudaMemsetAsync(out_rowptr, 0, sizeof(int) * ((size_t)n + 1), s) != cudaSuccess)
      return sgti_fail(ctx, SGT_ERR_CUDA, "sgt_symmetrize_device: memset");
    *out_nnz = 0;
    return SGT_OK;
  }
  return 2 * sym_bits(n) <= 32
             ? sym_run<unsigned>(ctx, n, nnz, rowptr, col, val, scale, out_rowptr, out_col,
                                 out_val, out_nnz)
             : sym_run<unsigned long long>(ctx, n, nnz, rowptr, col, val, scale, out_rowptr,
                                           out_col, out_val, out_nnz);
}
