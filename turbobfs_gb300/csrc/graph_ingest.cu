/*
 * graph_ingest.cu -- device-side preparation of a resident graph:
 *   validate_csc         bounds check of a CSC before any traversal reads it
 *   counting_sort_lists  (key, val) pairs -> ptr[n+1] / idx[nnz] lists; used
 *                        for COOC -> CSC (key = column) and for the transpose
 *                        CSC -> out-lists (key = row id)
 *   expand_columns       column id of every CSC entry
 *   symmetric_check      whether the CSC equals its transpose (keyed multiset hash)
 *   stable_sort_pairs    LSD radix sort of (key, val) pairs, 8 bits a pass,
 *                        stable: equal keys keep their input order
 * Replaces the host-side format builders of the reference
 * (TurboBFS_CSC_TD/sparseformatransf.c:28-120,
 * TurboBFS_COOC_TD/sparseformatransf.c:62-95) for graphs already on the GPU.
 * counting_sort_lists is stable too, so a list keeps the input order of its
 * entries: a COOC list the file order, a transposed list ascending columns.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "tbfs_internal.h"

namespace tbfs {
namespace {

constexpr int kThreads = 256;
/* elements per block in the scan passes: short arrays are scanned in small
 * tiles, so that they still fill the chip (one pass over the tile sums then
 * takes a few rounds of one block) */
constexpr int kScanTile = 4096, kScanTileSmall = 1024;
constexpr long long kScanSmall = 1 << 20;

__device__ __forceinline__ unsigned long long gtid() {
  return (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
}
__device__ __forceinline__ unsigned long long gstride() {
  return (unsigned long long)gridDim.x * blockDim.x;
}

/* flag bit 1: col_ptr malformed; bit 2: row id out of range.  Four row ids per
 * load where the array is 16-byte aligned (quads); a warp reports once.
 * 31 M entries: 83 us with one entry per thread, 24 us so. */
__global__ void validate_kernel(const int *cp, const int *ic, int n, long long nnz, long long quads,
                                int *flag) {
  int bad = 0;
  for (unsigned long long v = gtid(); v < (unsigned long long)n; v += gstride())
    if (cp[v] > cp[v + 1]) bad |= 1;
  if (gtid() == 0 && (cp[0] != 0 || (long long)cp[n] != nnz)) bad |= 1;
  const unsigned un = (unsigned)n;
  const int4 *q4 = reinterpret_cast<const int4 *>(ic);
  for (unsigned long long q = gtid(); q < (unsigned long long)quads; q += gstride()) {
    const int4 t = __ldg(q4 + q);
    if ((unsigned)t.x >= un || (unsigned)t.y >= un || (unsigned)t.z >= un || (unsigned)t.w >= un)
      bad |= 2;
  }
  for (unsigned long long k = 4ull * quads + gtid(); k < (unsigned long long)nnz; k += gstride())
    if ((unsigned)ic[k] >= un) bad |= 2;
  bad = (int)__reduce_or_sync(0xffffffffu, (unsigned)bad);
  if (bad && (threadIdx.x & 31) == 0) atomicOr(flag, bad);
}

/* flag bit 2: a key outside [0, n) */
__global__ void key_check_kernel(const int *keys, long long nnz, int n, int *flag) {
  bool bad = false;
  for (unsigned long long k = gtid(); k < (unsigned long long)nnz; k += gstride())
    bad |= (unsigned)keys[k] >= (unsigned)n;
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 2);
}

/* ptr[c] = first position whose key is >= c, for c in [0, n]; the keys are
 * sorted: a position writes the columns between its predecessor's key and its
 * own, so that no counting pass with atomics is needed (8 M random keys: 207
 * us of atomics and a scan, 25 us so).  Of a run of more than kGap empty
 * columns only the last kGap are written; the others, set to -1 before, take
 * the start of the next column that has entries (fill_starts_kernel). */
constexpr int kGap = 64;
__global__ void list_starts_kernel(const unsigned *keys, long long len, int n, int *ptr) {
  for (unsigned long long i = gtid(); i < (unsigned long long)len; i += gstride()) {
    const long long hi = (long long)keys[i];
    long long lo = i > 0 ? (long long)keys[i - 1] + 1 : 0;
    if (lo < hi - kGap) lo = hi - kGap;
    for (long long c = lo; c <= hi; ++c) ptr[c] = (int)i;
  }
}

__global__ void fill_starts_kernel(const unsigned *keys, long long len, int n, int total,
                                   int *ptr) {
  for (unsigned long long c = gtid(); c <= (unsigned long long)n; c += gstride()) {
    if (ptr[c] >= 0) continue;
    long long lo = 0, hi = len; /* first key >= c */
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if ((unsigned long long)keys[mid] < c) lo = mid + 1;
      else hi = mid;
    }
    ptr[c] = lo < len && keys[lo] < (unsigned)n ? ptr[keys[lo]] : total;
  }
}

/* SplitMix64's output function (S. Vigna; a bijection of 64-bit words) */
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

/* Sum over the entries u -> v (u in column v) of h({u, v}), counted positive
 * where u < v and negative where u > v, for two keyed hashes h_k of the
 * unordered pair, mix64(((min << 32) | max) ^ k), modulo 2^64: one hash per
 * entry and key, where h_k(u, v) - h_k(v, u) would take two.  A warp takes
 * chunks of kSymChunk consecutive entries, four in flight per lane; a lane
 * follows its entries' columns along col_ptr.  8 M entries: 240 us with 4096
 * entries per warp (a grid of two warps per scheduler) and four hashes each,
 * 52 us so. */
constexpr int kSymChunk = 512;
__global__ void symmetric_hash_kernel(const int *cp, const int *ic, int n, long long nnz,
                                      unsigned long long k1, unsigned long long k2,
                                      unsigned long long *out) {
  const unsigned lane = threadIdx.x & 31;
  const long long nchunks = (nnz + kSymChunk - 1) / kSymChunk;
  unsigned long long d1 = 0, d2 = 0;
  for (long long c = gtid() >> 5; c < nchunks; c += gstride() >> 5) {
    const long long e0 = c * kSymChunk;
    const long long e1 = e0 + kSymChunk < nnz ? e0 + kSymChunk : nnz;
    int col = (int)dev::warp_find_owner(cp, (unsigned)n, (unsigned)e0);
    long long end = __ldg(cp + col + 1);
    for (long long k = e0 + lane; k < e1; k += 128) {
      unsigned u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = k + 32 * j < e1 ? (unsigned)__ldg(ic + k + 32 * j) : 0u;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const long long kk = k + 32 * j;
        if (kk >= e1) break;
        while (end <= kk) end = __ldg(cp + ++col + 1);
        const unsigned v = (unsigned)col;
        if (u[j] == v) continue;
        const unsigned a = u[j] < v ? u[j] : v, b = u[j] < v ? v : u[j];
        const unsigned long long x = ((unsigned long long)a << 32) | b;
        const unsigned long long h1 = mix64(x ^ k1), h2 = mix64(x ^ k2);
        d1 += u[j] < v ? h1 : 0ull - h1;
        d2 += u[j] < v ? h2 : 0ull - h2;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    d1 += __shfl_xor_sync(0xffffffffu, d1, o);
    d2 += __shfl_xor_sync(0xffffffffu, d2, o);
  }
  if (lane == 0 && (d1 | d2)) {
    atomicAdd(out, d1);
    atomicAdd(out + 1, d2);
  }
}

/* col[k] = column of entry k: a warp takes kExpandChunk consecutive entries, a
 * lane follows its entries' columns along col_ptr (a warp per column wrote 15
 * entries of 32 lanes: 51 us for 8 M entries, 37 so) */
constexpr int kExpandChunk = 512;
__global__ void expand_kernel(const int *cp, int n, long long nnz, int *col) {
  const unsigned lane = threadIdx.x & 31;
  const long long nchunks = (nnz + kExpandChunk - 1) / kExpandChunk;
  for (long long c = gtid() >> 5; c < nchunks; c += gstride() >> 5) {
    const long long e0 = c * kExpandChunk;
    const long long e1 = e0 + kExpandChunk < nnz ? e0 + kExpandChunk : nnz;
    int v = (int)dev::warp_find_owner(cp, (unsigned)n, (unsigned)e0);
    long long end = __ldg(cp + v + 1);
    for (long long k = e0 + lane; k < e1; k += 32) {
      while (end <= k) end = __ldg(cp + ++v + 1);
      col[k] = v;
    }
  }
}

/* ---- stable LSD radix sort of (key, val) pairs ----
 * A pass sorts by the digit (key >> shift) & mask, of at most 8 bits.  Tiles
 * of kRadixTile consecutive pairs; hist[d * ntiles + t] counts digit d in tile
 * t, and its exclusive scan (digit-major) is where tile t's pairs of digit d
 * start.  The scatter reads each tile in order -- warp w its 512-pair slice,
 * 32 pairs a round -- and ranks equal digits by lane (match_any), so the
 * output keeps the input order among equal digits; the tile is put in digit
 * order in shared memory first, so that the stores of a digit are consecutive
 * (8.4 M pairs: 148 us with every lane storing its own pair, 62 us so). */
constexpr int kRadixTile = 4096;
constexpr int kRadixWarps = kThreads / 32;
constexpr int kRadixRounds = kRadixTile / kThreads; /* rounds of 32 pairs per warp */

__global__ void radix_hist_kernel(const unsigned *keys, long long len, int shift, unsigned mask,
                                  int ntiles, int *hist) {
  __shared__ int h[256];
  for (int i = threadIdx.x; i < 256; i += kThreads) h[i] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kRadixTile;
  for (int i = threadIdx.x; i < kRadixTile; i += kThreads) {
    const long long j = base + i;
    if (j < len) atomicAdd(&h[(keys[j] >> shift) & mask], 1);
  }
  __syncthreads();
  for (int d = threadIdx.x; d <= (int)mask; d += kThreads)
    hist[(long long)d * ntiles + blockIdx.x] = h[d];
}

__device__ int block_excl_scan(int x, int *smem, int *total);

__global__ void __launch_bounds__(kThreads, 4) radix_scatter_kernel(
    const unsigned *keys, const unsigned *vals, long long len, int shift, unsigned mask,
    int ntiles, const int *offs, unsigned *ko, unsigned *vo) {
  static_assert(kThreads == 256, "one thread per digit");
  __shared__ int cnt[kRadixWarps][256];
  __shared__ int s_off[256]; /* global position of local position 0 of the digit */
  __shared__ int s_scan[33];
  __shared__ unsigned s_k[kRadixTile], s_v[kRadixTile];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const long long t0 = (long long)blockIdx.x * kRadixTile;
  const long long base = t0 + (long long)w * (kRadixTile / kRadixWarps);
  for (int d = lane; d < 256; d += 32) cnt[w][d] = 0;
  unsigned k[kRadixRounds];
  int rank[kRadixRounds]; /* among the warp's pairs of the same digit */
#pragma unroll
  for (int r = 0; r < kRadixRounds; ++r) {
    const long long j = base + r * 32 + lane;
    k[r] = j < len ? keys[j] : 0u;
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < kRadixRounds; ++r) {
    const bool ok = base + r * 32 + lane < len;
    const unsigned d = ok ? (k[r] >> shift) & mask : 256u + (unsigned)lane;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    rank[r] = ok ? cnt[w][d] + __popc(peers & lt) : 0;
    __syncwarp();
    if (ok && (peers & lt) == 0u) cnt[w][d] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  { /* digit d: earlier warps' counts, where its run starts in the tile and
     * in the output */
    const int d = threadIdx.x;
    int tot = 0;
    for (int ww = 0; ww < kRadixWarps; ++ww) tot += cnt[ww][d];
    int all;
    int run = block_excl_scan(tot, s_scan, &all);
    s_off[d] = d <= (int)mask ? offs[(long long)d * ntiles + blockIdx.x] - run : 0;
    for (int ww = 0; ww < kRadixWarps; ++ww) {
      const int c = cnt[ww][d];
      cnt[ww][d] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRadixRounds; ++r) {
    const long long j = base + r * 32 + lane;
    if (j < len) {
      const int pos = cnt[w][(k[r] >> shift) & mask] + rank[r];
      s_k[pos] = k[r];
      s_v[pos] = vals[j];
    }
  }
  __syncthreads();
  const int m = len - t0 < kRadixTile ? (int)(len - t0) : kRadixTile;
  for (int i = threadIdx.x; i < m; i += kThreads) {
    const unsigned key = s_k[i];
    const int pos = s_off[(key >> shift) & mask] + i;
    ko[pos] = key;
    vo[pos] = s_v[i];
  }
}

/* ---- exclusive scan of int32 counts (three passes) ---- */

__device__ int block_excl_scan(int x, int *smem, int *total) {
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
    int v = lane < (kThreads / 32) ? smem[lane] : 0;
    int vi = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, vi, o);
      if (lane >= o) vi += t;
    }
    if (lane < (kThreads / 32)) smem[lane] = vi - v;
    if (lane == 31) smem[32] = vi;
  }
  __syncthreads();
  const int r = incl - x + smem[w];
  *total = smem[32];
  __syncthreads();
  return r;
}

template <int TILE>
__global__ void scan_reduce_kernel(const int *in, long long len, int *partial) {
  __shared__ int smem[33];
  const long long base = (long long)blockIdx.x * TILE;
  int s = 0;
#pragma unroll
  for (int i = threadIdx.x; i < TILE; i += kThreads) {
    const long long j = base + i;
    if (j < len) s += in[j];
  }
  int total;
  block_excl_scan(s, smem, &total);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

__global__ void scan_partials_kernel(int *partial, int nparts) {
  __shared__ int smem[33];
  int carry = 0;
  for (int b0 = 0; b0 < nparts; b0 += kThreads) {
    const int i = b0 + threadIdx.x;
    const int x = i < nparts ? partial[i] : 0;
    int total;
    const int ex = block_excl_scan(x, smem, &total);
    if (i < nparts) partial[i] = ex + carry;
    carry += total;
  }
}

/* out[j] = exclusive prefix of in[] (in and out may alias) */
template <int TILE>
__global__ void scan_apply_kernel(const int *in, long long len, const int *partial,
                                  int *out) {
  __shared__ int smem[33];
  const long long base = (long long)blockIdx.x * TILE;
  int carry = partial[blockIdx.x];
  constexpr int kPer = TILE / kThreads;
  /* each thread owns kPer consecutive elements */
  int vals[kPer];
  int s = 0;
  const long long mine = base + (long long)threadIdx.x * kPer;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    vals[i] = (mine + i < len) ? in[mine + i] : 0;
    s += vals[i];
  }
  int total;
  int ex = block_excl_scan(s, smem, &total) + carry;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (mine + i < len) out[mine + i] = ex;
    ex += vals[i];
  }
}

int grid_for(long long work) {
  long long g = (work + kThreads - 1) / kThreads;
  if (g < 1) g = 1;
  if (g > 65535LL * 8) g = 65535LL * 8;
  return (int)g;
}

}  // namespace

/* the most partial sums a scan of up to len ints needs */
long long scan_partials_most(long long len) {
  const long long a = (len + kScanTile - 1) / kScanTile;
  const long long m = len < kScanSmall ? len : kScanSmall;
  const long long b = (m + kScanTileSmall - 1) / kScanTileSmall;
  return a > b ? a : b;
}

long long scan_partials(long long len) {
  const int tile = len <= kScanSmall ? kScanTileSmall : kScanTile;
  return (len + tile - 1) / tile;
}

/* exclusive scan over len ints with the caller's partial-sum scratch; queued
 * on s, no synchronisation */
cudaError_t exclusive_scan_ws(const int *in, long long len, int *out, int *partial,
                              cudaStream_t s) {
  const long long tiles = scan_partials(len);
  if (tiles == 0) return cudaSuccess;
  const bool small = len <= kScanSmall;
  if (small) scan_reduce_kernel<kScanTileSmall><<<(unsigned)tiles, kThreads, 0, s>>>(in, len, partial);
  else scan_reduce_kernel<kScanTile><<<(unsigned)tiles, kThreads, 0, s>>>(in, len, partial);
  scan_partials_kernel<<<1, kThreads, 0, s>>>(partial, (int)tiles);
  if (small)
    scan_apply_kernel<kScanTileSmall><<<(unsigned)tiles, kThreads, 0, s>>>(in, len, partial, out);
  else
    scan_apply_kernel<kScanTile><<<(unsigned)tiles, kThreads, 0, s>>>(in, len, partial, out);
  return cudaGetLastError();
}

/* exclusive scan over len ints, in place allowed; synchronises the stream */
cudaError_t exclusive_scan(const int *in, long long len, int *out, cudaStream_t s) {
  const long long tiles = scan_partials(len);
  if (tiles == 0) return cudaSuccess;
  int *partial = nullptr;
  cudaError_t e = tbfs::dev_alloc(&partial, (size_t)tiles * sizeof(int));
  if (e != cudaSuccess) return e;
  e = exclusive_scan_ws(in, len, out, partial, s);
  cudaError_t e2 = cudaStreamSynchronize(s);
  tbfs::dev_free(partial);
  return e != cudaSuccess ? e : e2;
}

cudaError_t validate_csc(const int *cp, const int *ic, int n, long long nnz, int *d_flag,
                         cudaStream_t s) {
  const long long quads = (reinterpret_cast<uintptr_t>(ic) & 15u) == 0 ? nnz >> 2 : 0;
  const long long work = quads ? quads : nnz;
  const int grid = grid_for(work > n ? work : n);
  validate_kernel<<<grid < 4864 ? grid : 4864, kThreads, 0, s>>>(cp, ic, n, nnz, quads, d_flag);
  return cudaGetLastError();
}

int key_bits(unsigned max_key) {
  int b = 0;
  while (b < 32 && (max_key >> b) != 0u) ++b;
  return b;
}

cudaError_t stable_sort_pairs(unsigned **keys, unsigned **vals, long long len, int bits,
                              unsigned **ktmp, unsigned **vtmp, cudaStream_t s) {
  if (len <= 1 || bits <= 0) return cudaSuccess;
  const long long tiles = (len + kRadixTile - 1) / kRadixTile;
  if (tiles * 256 > INT32_MAX) return cudaErrorInvalidValue;
  const int passes = (bits + 7) / 8, per = (bits + passes - 1) / passes;
  const size_t counts = (size_t)tiles << per;
  int *hist = nullptr;
  cudaError_t e = tbfs::dev_alloc(
      &hist, (counts + (size_t)scan_partials_most((long long)counts)) * sizeof(int));
  if (e != cudaSuccess) return e;
  for (int p = 0; p < passes && e == cudaSuccess; ++p) {
    const int shift = p * per, w = bits - shift < per ? bits - shift : per;
    const unsigned mask = (1u << w) - 1u;
    radix_hist_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(*keys, len, shift, mask, (int)tiles,
                                                           hist);
    e = exclusive_scan_ws(hist, tiles << w, hist, hist + counts, s);
    if (e != cudaSuccess) break;
    radix_scatter_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(*keys, *vals, len, shift, mask,
                                                              (int)tiles, hist, *ktmp, *vtmp);
    e = cudaGetLastError();
    unsigned *t = *keys;
    *keys = *ktmp;
    *ktmp = t;
    t = *vals;
    *vals = *vtmp;
    *vtmp = t;
  }
  const cudaError_t e2 = tbfs::dev_free(hist); /* waits for the device */
  return e != cudaSuccess ? e : e2;
}

cudaError_t fill_starts(const unsigned *keys, long long len, int n, int total, int *ptr,
                        cudaStream_t s) {
  fill_starts_kernel<<<grid_for((long long)n + 1), kThreads, 0, s>>>(keys, len, n, total, ptr);
  return cudaGetLastError();
}

/* starts of the columns of sorted keys (all below n) */
static cudaError_t list_starts(const unsigned *keys, long long len, int n, int *ptr,
                               cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(ptr, 0xff, ((size_t)n + 1) * sizeof(int), s);
  if (e != cudaSuccess) return e;
  if (len > 0) list_starts_kernel<<<grid_for(len), kThreads, 0, s>>>(keys, len, n, ptr);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return fill_starts(keys, len, n, (int)len, ptr, s);
}

cudaError_t counting_sort_lists(const int *keys, const int *vals, long long nnz, int n,
                                int *ptr_out, int *idx_out, int *d_flag, cudaStream_t s) {
  const int kgrid = grid_for(nnz);
  key_check_kernel<<<kgrid < 4864 ? kgrid : 4864, kThreads, 0, s>>>(keys, nnz, n, d_flag);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  int flag = 0;
  if ((e = cudaMemcpyAsync(&flag, d_flag, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return e;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  if (flag) /* a key out of range: the caller reports it */
    return cudaMemsetAsync(ptr_out, 0, ((size_t)n + 1) * sizeof(int), s);
  /* stable: sort copies of the pairs by key, the values are the lists */
  const size_t m = (size_t)(nnz > 0 ? nnz : 1);
  unsigned *buf = nullptr;
  if ((e = tbfs::dev_alloc(&buf, 4 * m * sizeof(unsigned))) != cudaSuccess) return e;
  unsigned *k = buf, *v = buf + m, *kt = buf + 2 * m, *vt = buf + 3 * m;
  e = cudaMemcpyAsync(k, keys, (size_t)nnz * sizeof(int), cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(v, vals, (size_t)nnz * sizeof(int), cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess)
    e = stable_sort_pairs(&k, &v, nnz, key_bits((unsigned)(n > 0 ? n - 1 : 0)), &kt, &vt, s);
  if (e == cudaSuccess) e = list_starts(k, nnz, n, ptr_out, s);
  if (e == cudaSuccess && nnz)
    e = cudaMemcpyAsync(idx_out, v, (size_t)nnz * sizeof(int), cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = validate_csc(ptr_out, idx_out, n, nnz, d_flag, s); /* values out of range */
  const cudaError_t e2 = tbfs::dev_free(buf); /* waits for the device */
  return e != cudaSuccess ? e : e2;
}

cudaError_t symmetric_check(const int *cp, const int *ic, int n, long long nnz,
                            unsigned long long key1, unsigned long long key2, bool *symmetric,
                            cudaStream_t s) {
  *symmetric = false;
  unsigned long long *acc = nullptr, h[2] = {0, 0};
  cudaError_t e = tbfs::dev_alloc(&acc, 2 * sizeof(unsigned long long));
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(acc, 0, 2 * sizeof(unsigned long long), s);
  if (e == cudaSuccess && nnz > 0) {
    const long long warps = (nnz + kSymChunk - 1) / kSymChunk;
    const long long blocks = (warps * 32 + kThreads - 1) / kThreads;
    symmetric_hash_kernel<<<(unsigned)(blocks < 4864 ? blocks : 4864), kThreads, 0, s>>>(
        cp, ic, n, nnz, key1, key2, acc);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, acc, sizeof h, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  tbfs::dev_free(acc);
  if (e == cudaSuccess) *symmetric = h[0] == 0 && h[1] == 0;
  return e;
}

cudaError_t expand_columns(const int *cp, int n, long long nnz, int *col_of_entry, cudaStream_t s) {
  if (nnz <= 0) return cudaSuccess;
  const long long warps = (nnz + kExpandChunk - 1) / kExpandChunk;
  const int grid = grid_for(warps * 32);
  expand_kernel<<<grid < 4864 ? grid : 4864, kThreads, 0, s>>>(cp, n, nnz, col_of_entry);
  return cudaGetLastError();
}

/* ---- degree-based grouping ----
 * Vertices are put into kGroups groups by degree relative to the mean
 * (group 0: degree < 2*mean; group g: 2^g*mean <= degree < 2^(g+1)*mean),
 * hottest group first, original order kept inside each group.  This is the
 * degree-based grouping of Faldu, Diamond and Grot (IISWC 2019): hubs end up
 * packed at the front, so the traversal's per-vertex gathers concentrate in
 * a few cache lines, while a graph without hubs keeps its layout (all its
 * vertices fall into group 0 and the order is the identity). */

namespace {

constexpr int kGroups = 16;
constexpr int kGroupTile = 256; /* vertices per single-warp block */

__device__ __forceinline__ int degree_group(const int *cp, int v, float inv_mean2) {
  const float t = (float)(cp[v + 1] - cp[v]) * inv_mean2; /* degree / (2*mean) */
  if (t < 1.0f) return 0;
  const int g = 1 + (int)floorf(log2f(t));
  return g < kGroups - 1 ? g : kGroups - 1;
}

/* counts[slot(g, b)] with slot = (kGroups-1-g) * nblocks + b */
__global__ void group_count_kernel(const int *cp, int n, float inv_mean2, int *counts) {
  __shared__ int c[kGroups];
  const int lane = threadIdx.x;
  if (lane < kGroups) c[lane] = 0;
  __syncwarp();
  const long long base = (long long)blockIdx.x * kGroupTile;
  for (int i = lane; i < kGroupTile; i += 32) {
    const long long v = base + i;
    if (v < n) atomicAdd(&c[degree_group(cp, (int)v, inv_mean2)], 1);
  }
  __syncwarp();
  if (lane < kGroups) counts[(size_t)(kGroups - 1 - lane) * gridDim.x + blockIdx.x] = c[lane];
}

/* stable scatter: one warp walks its tile in order, ranking equal groups
 * with __match_any_sync */
__global__ void group_scatter_kernel(const int *cp, int n, float inv_mean2, const int *offsets,
                                     int *perm, int *inv) {
  __shared__ int off[kGroups + 1];
  const int lane = threadIdx.x;
  if (lane < kGroups) off[lane] = offsets[(size_t)(kGroups - 1 - lane) * gridDim.x + blockIdx.x];
  __syncwarp();
  const long long base = (long long)blockIdx.x * kGroupTile;
  unsigned lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  for (int c0 = 0; c0 < kGroupTile; c0 += 32) {
    const long long v = base + c0 + lane;
    const int g = v < n ? degree_group(cp, (int)v, inv_mean2) : kGroups;
    const unsigned m = __match_any_sync(0xffffffffu, g);
    const int rank = __popc(m & lt);
    if (g < kGroups) {
      const int pos = off[g] + rank;
      perm[pos] = (int)v;
      inv[v] = pos;
    }
    __syncwarp();
    if (g < kGroups && (m >> lane) == 1u) off[g] += __popc(m); /* last lane of its group */
    __syncwarp();
  }
}

__global__ void permuted_degree_kernel(const int *cp, const int *perm, int n, int *deg2) {
  for (unsigned long long i = gtid(); i < (unsigned long long)n; i += gstride()) {
    const int v = perm[i];
    deg2[i] = cp[v + 1] - cp[v];
  }
}

/* New list i is old list perm[i] with every entry renamed by inv, in the same
 * order.  Short lists (< 32 entries) are copied by one lane each; longer ones
 * are collected in `longs`, those for a warp each from the front (their
 * number in cnt[0]), those of kHugeList entries and more, for a block each,
 * from the back (cnt[1]). */
constexpr int kHugeList = 4096;
__global__ void permuted_short_lists_kernel(const int *cp, const int *ic, const int *perm,
                                            const int *inv, const int *cp2, int n, int *ic2,
                                            int *longs, int *cnt) {
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  for (unsigned long long base = gtid() & ~31ull; base < (unsigned long long)n; base += gstride()) {
    const unsigned long long i = base + lane;
    int b = 0, len = 0, o = 0;
    if (i < (unsigned long long)n) {
      const int v = perm[i];
      b = cp[v];
      len = cp[v + 1] - b;
      o = cp2[i];
    }
    if (len < 32)
      for (int t = 0; t < len; ++t) ic2[o + t] = inv[ic[b + t]];
    /* append the long ones, one atomic per warp and kind */
    const unsigned bw = __ballot_sync(0xffffffffu, len >= 32 && len < kHugeList);
    const unsigned bh = __ballot_sync(0xffffffffu, len >= kHugeList);
    if (bw) {
      int pos = 0;
      if (lane == 0) pos = atomicAdd(cnt, __popc(bw));
      pos = __shfl_sync(0xffffffffu, pos, 0);
      if (len >= 32 && len < kHugeList) longs[pos + __popc(bw & lt)] = (int)i;
    }
    if (bh) {
      int pos = 0;
      if (lane == 0) pos = atomicAdd(cnt + 1, __popc(bh));
      pos = __shfl_sync(0xffffffffu, pos, 0);
      if (len >= kHugeList) longs[n - 1 - pos - __popc(bh & lt)] = (int)i;
    }
  }
}

__global__ void permuted_long_lists_kernel(const int *cp, const int *ic, const int *perm,
                                           const int *inv, const int *cp2, const int *longs,
                                           const int *cnt, int n, int *ic2) {
  const int nw = cnt[0], nh = cnt[1];
  for (int j = blockIdx.x; j < nh; j += gridDim.x) {
    const int i = longs[n - 1 - j];
    const int v = perm[i];
    const int b = cp[v], len = cp[v + 1] - b, o = cp2[i];
    for (int t = threadIdx.x; t < len; t += blockDim.x) ic2[o + t] = inv[ic[b + t]];
  }
  const int lane = threadIdx.x & 31;
  for (long long j = (long long)(gtid() >> 5); j < nw; j += (long long)(gstride() >> 5)) {
    const int i = longs[j];
    const int v = perm[i];
    const int b = cp[v], len = cp[v + 1] - b, o = cp2[i];
    for (int t = lane; t < len; t += 128) {
      int u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) u[q] = t + 32 * q < len ? __ldg(ic + b + t + 32 * q) : 0;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (t + 32 * q < len) ic2[o + t + 32 * q] = __ldg(inv + u[q]);
    }
  }
}

}  // namespace

cudaError_t degree_group_relabel(const int *cp, const int *ic, int n, long long nnz,
                                 int *perm, int *inv, int *cp2, int *ic2, bool *identity,
                                 cudaStream_t s) {
  const int nblocks = (int)((n + (long long)kGroupTile - 1) / kGroupTile);
  const float inv_mean2 = nnz > 0 ? (float)((double)n / (2.0 * (double)nnz)) : 0.0f;
  int *counts = nullptr;
  const size_t nslots = (size_t)kGroups * nblocks;
  cudaError_t e = tbfs::dev_alloc(&counts, (nslots + 1) * sizeof(int));
  if (e != cudaSuccess) return e;
  group_count_kernel<<<nblocks, 32, 0, s>>>(cp, n, inv_mean2, counts);
  e = cudaGetLastError();
  /* how many vertices sit outside group 0: if none, the order is the identity */
  int tail_first = 0;
  if (e == cudaSuccess)
    e = exclusive_scan(counts, (long long)nslots + 1, counts, s);
  if (e == cudaSuccess)
    e = cudaMemcpy(&tail_first, counts + (size_t)(kGroups - 1) * nblocks, sizeof(int),
                   cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) {
    *identity = tail_first == 0;
    if (!*identity) {
      group_scatter_kernel<<<nblocks, 32, 0, s>>>(cp, n, inv_mean2, counts, perm, inv);
      permuted_degree_kernel<<<grid_for(n), kThreads, 0, s>>>(cp, perm, n, cp2);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemsetAsync(cp2 + n, 0, sizeof(int), s);
      if (e == cudaSuccess) e = exclusive_scan(cp2, (long long)n + 1, cp2, s);
      int *longs = nullptr; /* long lists' new ids, the two counts after them */
      if (e == cudaSuccess) e = tbfs::dev_alloc(&longs, ((size_t)n + 2) * sizeof(int));
      if (e == cudaSuccess) e = cudaMemsetAsync(longs + n, 0, 2 * sizeof(int), s);
      if (e == cudaSuccess) {
        permuted_short_lists_kernel<<<grid_for(n), kThreads, 0, s>>>(cp, ic, perm, inv, cp2, n,
                                                                    ic2, longs, longs + n);
        permuted_long_lists_kernel<<<2432, kThreads, 0, s>>>(cp, ic, perm, inv, cp2, longs,
                                                             longs + n, n, ic2);
        e = cudaGetLastError();
      }
      const cudaError_t e2 = tbfs::dev_free(longs); /* waits for the device */
      if (e == cudaSuccess) e = e2;
    }
  }
  tbfs::dev_free(counts);
  return e;
}

}  // namespace tbfs
