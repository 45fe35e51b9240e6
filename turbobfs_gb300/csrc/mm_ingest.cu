/*
 * mm_ingest.cu -- graphs built on the device from edge lists and from
 * Matrix Market text.
 *
 *   csc_from_edges_device  edge list (on the device) -> CSC, with the
 *                          construction of the host builder
 *                          tbfs_csc_from_edges: symmetrise (each entry and
 *                          its mirror, a self loop twice), drop self loops,
 *                          sort each column, drop repeats.  Built by stable
 *                          radix sorts, so without sorting a column keeps the
 *                          input order of its entries, exactly as the host
 *                          builder lays it out.
 *   mm_parse_device        the data lines of a Matrix Market coordinate
 *                          file (already in device memory) -> edge list,
 *                          entry k from the k-th data line.
 *
 * These replace the reference's host preparation -- readMMfile_uw and the
 * CP_RP_ug / SSCCSC_uw / SSCCOOC_uw builders
 * (TurboBFS_CSC_TD/readMMfilef.c:56-70, TurboBFS_CSC_TD/sparseformatransf.c:
 * 60-104, TurboBFS_COOC_TD/sparseformatransf.c:62-95) -- which the host
 * reader tbfs_mm_read restates sequentially.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "tbfs_graphgen.h"
#include "tbfs_internal.h"

namespace tbfs {
namespace {

constexpr int kThreads = 256;
constexpr int kTextPer = 16;                       /* bytes a thread looks at */
constexpr int kTextTile = kThreads * kTextPer;     /* bytes a block looks at  */

__device__ __forceinline__ unsigned long long gtid() {
  return (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
}
__device__ __forceinline__ unsigned long long gstride() {
  return (unsigned long long)gridDim.x * blockDim.x;
}

int grid_for(long long work) {
  long long g = (work + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > 65535LL * 8) g = 65535LL * 8;
  return (int)g;
}

/* ---- edge list -> CSC ---- */

/* entry e of the pair list: (column, row); with symmetrise edge k gives
 * e = 2k (dst <- src) and e = 2k+1 (src <- dst).  Dropped or invalid edges
 * get column n, which sorts last and is cut off. */
__global__ void edge_pairs_kernel(const int *src, const int *dst, long long m, int n,
                                  unsigned flags, unsigned *key, unsigned *val, int *bad) {
  const bool sym = (flags & TBFS_BUILD_SYMMETRIZE) != 0u;
  const bool noloop = (flags & TBFS_BUILD_DROP_LOOPS) != 0u;
  for (unsigned long long k = gtid(); k < (unsigned long long)m; k += gstride()) {
    const int u = src[k], v = dst[k];
    const bool ok = u >= 0 && u < n && v >= 0 && v < n;
    if (!ok) atomicOr(bad, 1);
    const bool drop = !ok || (noloop && u == v);
    const unsigned long long e = sym ? 2 * k : k;
    key[e] = drop ? (unsigned)n : (unsigned)v;
    val[e] = ok ? (unsigned)u : 0u;
    if (sym) {
      key[e + 1] = drop ? (unsigned)n : (unsigned)u;
      val[e + 1] = ok ? (unsigned)v : 0u;
    }
  }
}

/* pair i is a real entry (column < n) and, with dedup, differs from pair i-1
 * (the pairs are sorted by column, then row) */
__device__ __forceinline__ bool kept(const unsigned *key, const unsigned *val, long long i, int n,
                                     int dedup) {
  return key[i] < (unsigned)n &&
         !(dedup && i > 0 && key[i] == key[i - 1] && val[i] == val[i - 1]);
}

constexpr int kKeepPer = 8; /* pairs per thread, strided by the block */
constexpr int kKeepTile = kThreads * kKeepPer;

__device__ int block_excl_sum(int x, int *smem, int *total);

/* counts[tile] = kept pairs among the tile's kKeepTile */
__global__ void keep_count_kernel(const unsigned *key, const unsigned *val, long long len, int n,
                                  int dedup, int *counts) {
  __shared__ int smem[33];
  const long long base = (long long)blockIdx.x * kKeepTile + threadIdx.x;
  int c = 0;
#pragma unroll 4
  for (int i = 0; i < kKeepPer; ++i) {
    const long long j = base + (long long)i * kThreads;
    if (j < len && kept(key, val, j, n, dedup)) ++c;
  }
  int total;
  block_excl_sum(c, smem, &total);
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

/* The kept pairs' rows at their compacted positions (offs: exclusive prefix
 * of the tile counts), and cp[c] = the position of the first kept pair of a
 * column >= c: where the column changes, the pair writes the columns between
 * (the last kGap of them; the rest, set to -1 before, is fill_starts' work).
 * Two passes over the sorted pairs (90 us for 8.4 M), where flags, column
 * counts by atomics, two scans and the compaction took 200. */
constexpr int kGap = 64;
__global__ void keep_write_kernel(const unsigned *key, const unsigned *val, long long len, int n,
                                  int dedup, const int *offs, int *ic, int *cp) {
  __shared__ int s_w[kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int run = offs[blockIdx.x];
  for (int i = 0; i < kKeepPer; ++i) {
    const long long j = (long long)blockIdx.x * kKeepTile + (long long)i * kThreads + threadIdx.x;
    const bool in = j < len;
    const bool k = in && kept(key, val, j, n, dedup);
    const unsigned m = __ballot_sync(0xffffffffu, k);
    if (lane == 0) s_w[w] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int ww = 0; ww < kThreads / 32; ++ww) {
      const int c = s_w[ww];
      before += ww < w ? c : 0;
      all += c;
    }
    const int pos = run + before + __popc(m & ((1u << lane) - 1u));
    if (k) ic[pos] = (int)val[j];
    if (in) { /* columns after the previous pair's, up to this one's (n: dropped) */
      const long long c1 = key[j] < (unsigned)n ? (long long)key[j] : (long long)n;
      long long c0 = 0;
      if (j > 0) c0 = (key[j - 1] < (unsigned)n ? (long long)key[j - 1] : (long long)n) + 1;
      if (c0 < c1 - kGap) c0 = c1 - kGap;
      for (long long c = c0; c <= c1; ++c) cp[c] = pos;
    }
    run += all;
    __syncthreads();
  }
}

/* ---- Matrix Market data lines -> edge list ---- */

__device__ __forceinline__ bool blank(char c) { return c == ' ' || c == '\t' || c == '\r'; }
__device__ __forceinline__ bool digit(char c) { return c >= '0' && c <= '9'; }

/* p starts a data line: the first byte of a line whose first non-blank
 * byte is a digit (comment lines start with '%', empty lines have none) */
__device__ __forceinline__ bool entry_start(const char *t, long long len, long long p) {
  if (p >= len || (p > 0 && t[p - 1] != '\n')) return false;
  long long q = p;
  while (q < len && blank(t[q])) ++q;
  return q < len && digit(t[q]);
}

__device__ int block_excl_sum(int x, int *smem, int *total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) smem[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int v = lane < kThreads / 32 ? smem[lane] : 0;
    int vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) vi += t;
    }
    if (lane < kThreads / 32) smem[lane] = vi - v;
    if (lane == 31) smem[32] = vi;
  }
  __syncthreads();
  const int r = incl - x + smem[w];
  *total = smem[32];
  __syncthreads();
  return r;
}

/* counts[tile] = data lines starting in the tile's kTextTile bytes */
__global__ void mm_count_kernel(const char *t, long long len, int *counts) {
  __shared__ int smem[33];
  const long long p0 = (long long)blockIdx.x * kTextTile + (long long)threadIdx.x * kTextPer;
  int c = 0;
#pragma unroll 4
  for (int i = 0; i < kTextPer; ++i) c += entry_start(t, len, p0 + i) ? 1 : 0;
  int total;
  block_excl_sum(c, smem, &total);
  if (threadIdx.x == 0) counts[blockIdx.x] = total;
}

/* reads the unsigned decimal at t[*q..), advancing *q; false without digits
 * or past 2^40 (far beyond any int32 index) */
__device__ bool read_uint(const char *t, long long len, long long *q, unsigned long long *x) {
  long long r = *q;
  unsigned long long v = 0;
  int nd = 0;
  while (r < len && digit(t[r])) {
    v = v * 10u + (unsigned long long)(t[r] - '0');
    if (v > (1ull << 40)) return false;
    ++r;
    ++nd;
  }
  *q = r;
  *x = v;
  return nd > 0;
}

/* Entry k (the k-th data line, k < nz): row i and column j, 1-based, as the
 * edge i-1 -> j-1.  A line that does not hold two indices with 1 <= i <= M,
 * 1 <= j <= N and i <= N records its k in *bad (the smallest wins). */
__global__ void mm_parse_kernel(const char *t, long long len, const int *offs, long long nz,
                                long long M, long long N, int *src, int *dst,
                                unsigned long long *bad) {
  __shared__ int smem[33];
  const long long p0 = (long long)blockIdx.x * kTextTile + (long long)threadIdx.x * kTextPer;
  unsigned starts = 0; /* bit i: p0 + i starts a data line */
#pragma unroll 4
  for (int i = 0; i < kTextPer; ++i)
    if (entry_start(t, len, p0 + i)) starts |= 1u << i;
  int total;
  long long k = (long long)offs[blockIdx.x] + block_excl_sum(__popc(starts), smem, &total);
  while (starts) {
    const int i = __ffs(starts) - 1;
    starts &= starts - 1u;
    if (k < nz) {
      long long q = p0 + i;
      while (q < len && blank(t[q])) ++q;
      unsigned long long a = 0, b = 0;
      bool ok = read_uint(t, len, &q, &a);
      if (ok) {
        const long long q0 = q;
        while (q < len && blank(t[q])) ++q;
        ok = q > q0 && read_uint(t, len, &q, &b);
      }
      ok = ok && a >= 1 && b >= 1 && (long long)a <= M && (long long)b <= N && (long long)a <= N;
      if (ok) {
        src[k] = (int)(a - 1);
        dst[k] = (int)(b - 1);
      } else {
        atomicMin(bad, (unsigned long long)k);
        src[k] = 0;
        dst[k] = 0;
      }
    }
    ++k;
  }
}

}  // namespace

cudaError_t csc_from_edges_device(const int *src, const int *dst, long long m, int n,
                                  unsigned flags, int **cp_out, int **ic_out, long long *nnz_out,
                                  int *bad_out, cudaStream_t s) {
  *cp_out = nullptr;
  *ic_out = nullptr;
  *nnz_out = 0;
  *bad_out = 0;
  const bool sym = (flags & TBFS_BUILD_SYMMETRIZE) != 0u;
  const bool dedup = (flags & TBFS_BUILD_DEDUP) != 0u;
  const bool sorted = dedup || (flags & TBFS_BUILD_SORT) != 0u;
  const long long len = sym ? 2 * m : m;
  if (len > INT32_MAX) return cudaErrorInvalidValue;
  const size_t L = (size_t)(len > 0 ? len : 1);
  const long long tiles = (len + kKeepTile - 1) / kKeepTile;
  unsigned *buf = nullptr;
  int *counts = nullptr, *cp = nullptr, *ic = nullptr;
  cudaError_t e = tbfs::dev_alloc(&buf, 4 * L * sizeof(unsigned));
  /* tile counts, their scan's scratch, the flag */
  const size_t part = (size_t)scan_partials(tiles + 1);
  if (e == cudaSuccess) e = tbfs::dev_alloc(&counts, ((size_t)tiles + 1 + part + 1) * sizeof(int));
  int *dflag = counts ? counts + tiles + 1 + part : nullptr;
  if (e == cudaSuccess) e = tbfs::dev_alloc(&cp, ((size_t)n + 1) * sizeof(int));
  if (e == cudaSuccess) e = cudaMemsetAsync(dflag, 0, sizeof(int), s);
  unsigned *key = buf, *val = buf + L, *kt = buf + 2 * L, *vt = buf + 3 * L;
  if (e == cudaSuccess && m > 0) {
    edge_pairs_kernel<<<grid_for(m), kThreads, 0, s>>>(src, dst, m, n, flags, key, val, dflag);
    e = cudaGetLastError();
  }
  /* rows ascending inside a column: sort by row first, then (stably) by column */
  if (e == cudaSuccess && sorted)
    e = stable_sort_pairs(&val, &key, len, key_bits((unsigned)(n - 1)), &vt, &kt, s);
  if (e == cudaSuccess) e = stable_sort_pairs(&key, &val, len, key_bits((unsigned)n), &kt, &vt, s);
  /* the kept pairs: their number, then their rows and the column starts */
  int nnz = 0;
  if (e == cudaSuccess && len > 0) {
    e = cudaMemsetAsync(counts + tiles, 0, sizeof(int), s);
    if (e == cudaSuccess)
      keep_count_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(key, val, len, n, dedup ? 1 : 0, counts);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = exclusive_scan_ws(counts, tiles + 1, counts, counts + tiles + 1, s);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(&nnz, counts + tiles, sizeof(int), cudaMemcpyDeviceToHost, s);
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(bad_out, dflag, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = tbfs::dev_alloc(&ic, (size_t)(nnz > 0 ? nnz : 1) * sizeof(int));
  if (e == cudaSuccess && len > 0) {
    e = cudaMemsetAsync(cp, 0xff, ((size_t)n + 1) * sizeof(int), s);
    if (e == cudaSuccess)
      keep_write_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(key, val, len, n, dedup ? 1 : 0,
                                                             counts, ic, cp);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = fill_starts(key, len, n, nnz, cp, s);
  } else if (e == cudaSuccess) {
    e = cudaMemsetAsync(cp, 0, ((size_t)n + 1) * sizeof(int), s);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  tbfs::dev_free(buf);
  tbfs::dev_free(counts);
  if (e != cudaSuccess) {
    tbfs::dev_free(cp);
    tbfs::dev_free(ic);
    return e;
  }
  *cp_out = cp;
  *ic_out = ic;
  *nnz_out = nnz;
  return cudaSuccess;
}

cudaError_t mm_parse_device(const char *text, long long len, long long nz, long long M,
                            long long N, int *src, int *dst, long long *lines_out,
                            long long *bad_out, cudaStream_t s) {
  *lines_out = 0;
  *bad_out = -1;
  const long long tiles = (len + kTextTile - 1) / kTextTile;
  if (tiles + 1 > INT32_MAX) return cudaErrorInvalidValue;
  int *offs = nullptr;
  unsigned long long *bad = nullptr;
  cudaError_t e = tbfs::dev_alloc(&offs, (size_t)(tiles + 1) * sizeof(int));
  if (e == cudaSuccess) e = tbfs::dev_alloc(&bad, sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMemsetAsync(offs, 0, (size_t)(tiles + 1) * sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0xff, sizeof(unsigned long long), s);
  if (e == cudaSuccess && tiles > 0) {
    mm_count_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(text, len, offs);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = exclusive_scan(offs, tiles + 1, offs, s);
  if (e == cudaSuccess && tiles > 0) {
    mm_parse_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(text, len, offs, nz, M, N, src, dst, bad);
    e = cudaGetLastError();
  }
  int lines = 0;
  unsigned long long b = ~0ull;
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&lines, offs + tiles, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&b, bad, sizeof(b), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  tbfs::dev_free(offs);
  tbfs::dev_free(bad);
  if (e != cudaSuccess) return e;
  *lines_out = lines;
  *bad_out = b == ~0ull ? -1 : (long long)b;
  return cudaSuccess;
}

}  // namespace tbfs
