/*
 * brandes.cu -- betweenness centrality: the forward traversal of the engine
 * (depths S and path counts sigma, exactly what the reference computes) plus
 * Brandes' dependency sweep (U. Brandes, "A faster algorithm for betweenness
 * centrality", J. Math. Sociology 25(2), 2001):
 *
 *   delta[v] = sum over out-list entries v -> w with S[w] = S[v] + 1 of
 *              sigma[v] / sigma[w] * (1 + delta[w]),
 *   bc[v]   += delta[v] for every root s != v,
 * computed in the factored form delta[v] = sigma[v] * sum q[w] with
 * q[w] = (1 + delta[w]) / sigma[w], stored once w is final: one division
 * per vertex instead of one per entry, and one gather per entry.
 *
 * The sweep runs level by level from the deepest level up, in one persistent
 * cooperative launch for up to kMaxSweepRoots roots at once: step D works on
 * level D of every root whose traversal reached that deep, so the roots share
 * the grid barriers and fill the GPU where one root's level would not.
 * Vertices are grouped by depth and, within it, by the class of their
 * out-list, with one block-aggregated counting sort for all roots of a launch.
 * Every delta is a pull over the vertex's own out-list in a fixed order, so
 * the result does not depend on scheduling:
 *   out-degree < 32: one lane sums the terms in list order;
 *   otherwise the list is cut into segments of kSeg entries (one segment up
 *   to kSeg); in a segment, lane l sums the entries l, l+32, l+64, ... in
 *   order and the 32 partial sums meet in a butterfly (xor 16, 8, 4, 2, 1);
 *   the segments' sums are added in segment order.
 * A hub's segments are separate work items of the level, so a list of 10^5
 * entries is summed by tens of warps at once; its segment sums are combined
 * after a grid barrier.
 * All operations are correctly rounded IEEE double with no contraction into
 * fused multiply-adds, so a CPU restatement of the same order reproduces
 * every bit.  Each root's delta is kept and bc adds them up after the sweep,
 * in the order of the roots given.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "device_common.cuh"
#include "tbfs.h"
#include "tbfs_internal.h"

namespace tbfs {
namespace {

using dev::FULL;
using dev::grid_barrier;

constexpr int kBlock = 256;
constexpr int kSmemKeys = 11264;  /* depth-and-class keys counted in shared memory per block */
constexpr int kTile = 4096;       /* vertices per block of the counting sort   */
constexpr int kWarpDegree = 32;   /* out-degree from which a warp sums a vertex */
constexpr int kSeg = 2048;        /* entries per segment of a hub's list        */

struct __align__(128) SweepCtl {
  int status, timeout_level;
  unsigned work[4]; /* dynamic work counter of level d in work[d % 4] */
  int pad0[26];
  GridBarrier bar;
};

constexpr int kMaxSweepRoots = 32; /* roots per sweep launch (one lane each in the plan) */

/* Out-list classes of a level, in list order; the lists of a lane each in four
 * classes by length, so that the lanes of a chunk have about as much to add
 * (one class where the keys of six would not fit shared memory). */
enum { C_HUB = 0, C_WARP = 1, C_LANE = 2, kClasses = 6, kClassesFew = 3 };

/* one root's arrays (internal numbering) */
struct RootSweep {
  int *S;                            /* depths of the forward traversal      */
  unsigned long long *sig;           /* path counts                          */
  int *list;                         /* vertices grouped by depth and class  */
  int *off;                          /* class c of level d starts at list[off[classes d + c]] */
  int *fill;                         /* next free position of each           */
  int levels, classes;
  int root;                          /* the root (caller numbering in the host's
                                        copy, internal in the kernels')       */
  double *q[2];                      /* (1 + delta[v]) / sigma[v] in q[depth % 2],
                                        zero where it is not computed yet     */
  double *dl;                        /* delta[v] (0 at the root), zero on entry */
  /* segments of kSeg entries of the hubs (out-degree > kSeg): those of level d
   * are seg[d] .. seg[d + 1], seg_pos[s] = list position of segment s's hub,
   * hseg[i] = first segment of the hub at position i, part[s] = its sum */
  int *seg, *seg_fill, *seg_pos, *hseg;
  double *part;
};

struct SweepParams {
  const int *rp, *jr; /* out-lists (internal numbering) */
  const int *inv;     /* caller id -> internal id, or null */
  const RootSweep *rs;
  int k;              /* roots of the launch            */
  int dmax;           /* largest number of levels       */
  SweepCtl *ctl;
  long long timeout_ns;
};

/* v, of depth d, is final with the sum acc of its children's q: its delta and q */
__device__ __forceinline__ void finish(const RootSweep &R, int d, int v, double acc) {
  const double sv = (double)__ldg(R.sig + v);
  const double dv = __dmul_rn(sv, acc);
  R.q[d & 1][v] = __ddiv_rn(__dadd_rn(1.0, dv), sv);
  if (v != R.root) R.dl[v] = dv;
}

/* The sum of q[w] over the entries k0, k0 + step, ... < e with S[w] = d + 1, in
 * that order.  No depth is looked at: an out-neighbour w of a vertex of depth d
 * has S[w] <= d + 1, and in the array of d + 1's parity only depths d + 1,
 * d + 3, ... are computed, the others 0.0, which leaves the sum as it is, to
 * the bit: one gather per entry where the depth and then a child's q took
 * two, the second waiting for the first.  Eight entries' loads are issued
 * before they are added. */
__device__ __forceinline__ double sum_entries(const SweepParams &p, const RootSweep &R, int d,
                                              int k0, int e, int step) {
  const double *q = R.q[(d + 1) & 1];
  double acc = 0.0;
  int k = k0;
  for (; k + 7 * step < e; k += 8 * step) {
    int w[8];
    double t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = __ldg(p.jr + k + j * step);
#pragma unroll
    for (int j = 0; j < 8; ++j) t[j] = q[w[j]];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc = __dadd_rn(acc, t[j]);
  }
  for (; k < e; k += 4 * step) {
    int w[4];
    double t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = k + j * step < e ? __ldg(p.jr + k + j * step) : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = w[j] >= 0 ? q[w[j]] : 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (w[j] >= 0) acc = __dadd_rn(acc, t[j]);
  }
  return acc;
}

/* the terms of [b, e) summed lane-strided over the warp, then the butterfly;
 * every lane returns the same value (lane 0's order) */
__device__ __forceinline__ double warp_sum(const SweepParams &p, const RootSweep &R, int d, int b,
                                           int e) {
  const int lane = threadIdx.x & 31;
  double acc = sum_entries(p, R, d, b + lane, e, 32);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc = __dadd_rn(acc, __shfl_xor_sync(FULL, acc, o));
  return __shfl_sync(FULL, acc, 0);
}

/* The butterfly of eight lists at once: a[i] is this lane's part of list i's
 * sum, and lanes 4 i .. 4 i + 3 return list i's.  Where two lists are left in a
 * register pair, a lane keeps one and hands the other to the lane it would
 * have been added from: the adds are those of warp_sum, one for two lists (9
 * instead of 40).  FP64 runs at two lanes per clock and SM here, so an add of
 * a whole warp costs 16 clocks, and the division of one list by one lane as
 * much as that of eight by eight. */
__device__ __forceinline__ double warp_sum8(double (&a)[8]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = 4, o = 16; h > 0; h >>= 1, o >>= 1) { /* lists left per lane: 2h -> h */
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const double keep = up ? a[i + h] : a[i], give = up ? a[i] : a[i + h];
      a[i] = __dadd_rn(keep, __shfl_xor_sync(FULL, give, o));
    }
  }
  a[0] = __dadd_rn(a[0], __shfl_xor_sync(FULL, a[0], 2));
  return __dadd_rn(a[0], __shfl_xor_sync(FULL, a[0], 1));
}

/* Items of step D for root R: hub segments, groups of `per` lists a warp sums,
 * chunks of 32 short lists -- or, at the root's deepest level, chunks of 32 positions whose
 * q = 1 / sigma (no children).  cnt[0..3]: segments, warp lists (not yet in
 * groups), chunks, hubs to combine afterwards. */
__device__ __forceinline__ void step_counts(const RootSweep &R, int D, unsigned (&cnt)[4]) {
  cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0u;
  if (D >= R.levels) return;
  const int *o = R.off + R.classes * D;
  const int lo = __ldg(o), hi = __ldg(o + R.classes);
  if (D == R.levels - 1) {
    cnt[2] = (unsigned)(hi - lo + 31) / 32u;
    return;
  }
  const int w = __ldg(o + C_WARP), l = __ldg(o + C_LANE);
  cnt[0] = (unsigned)(__ldg(R.seg + D + 1) - __ldg(R.seg + D));
  cnt[1] = (unsigned)(l - w);
  cnt[2] = (unsigned)(hi - l + 31) / 32u;
  cnt[3] = (unsigned)(w - lo);
}

/* phase A item `it` of root R at step D */
__device__ __forceinline__ void sweep_item(const SweepParams &p, const RootSweep &R, int D,
                                           unsigned it, unsigned per) {
  const int lane = threadIdx.x & 31;
  const int *o = R.off + R.classes * D;
  const int hi = __ldg(o + R.classes);
  if (D == R.levels - 1) { /* the root's deepest level: no children */
    const int i = __ldg(o) + (int)it * 32 + lane;
    if (i < hi) {
      const int v = __ldg(R.list + i);
      R.q[D & 1][v] = __ddiv_rn(1.0, (double)__ldg(R.sig + v));
    }
    return;
  }
  const int s_lo = __ldg(R.seg + D), w = __ldg(o + C_WARP), l = __ldg(o + C_LANE);
  const unsigned ns = (unsigned)(__ldg(R.seg + D + 1) - s_lo), nm = (unsigned)(l - w);
  const unsigned ng = (nm + per - 1u) / per;
  if (it < ns) { /* segment sg of a hub */
    const int sg = s_lo + (int)it;
    const int i = __ldg(R.seg_pos + sg);
    const int v = __ldg(R.list + i);
    const int b = __ldg(p.rp + v) + (sg - __ldg(R.hseg + i)) * kSeg;
    const int e = min(b + kSeg, __ldg(p.rp + v + 1));
    const double acc = warp_sum(p, R, D, b, e);
    if (lane == 0) R.part[sg] = acc;
  } else if (it < ns + ng) { /* one-segment lists, the whole warp on each */
    const int i0 = w + (int)((it - ns) * per), i1 = min(i0 + (int)per, l);
    double a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      a[j] = 0.0;
      if (i0 + j < i1) {
        const int v = __ldg(R.list + i0 + j);
        a[j] = sum_entries(p, R, D, __ldg(p.rp + v) + lane, __ldg(p.rp + v + 1), 32);
      }
    }
    __syncwarp();
    const double acc = warp_sum8(a);
    const int i = i0 + (((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1));
    if ((lane & 3) == 0 && i < i1) finish(R, D, __ldg(R.list + i), acc);
  } else { /* short lists, one lane each */
    const int i = l + (int)(it - ns - ng) * 32 + lane;
    if (i < hi) {
      const int v = __ldg(R.list + i);
      finish(R, D, v, sum_entries(p, R, D, __ldg(p.rp + v), __ldg(p.rp + v + 1), 1));
    }
  }
}

/* smallest r with pre[r + 1] > x (pre[0] = 0, nondecreasing, k entries) */
__device__ __forceinline__ int root_of(const unsigned *pre, int k, unsigned x) {
  int lo = 0, hi = k - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (pre[mid + 1] > x) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

__global__ void __launch_bounds__(kBlock) sweep_kernel(const SweepParams p) {
  __shared__ unsigned s_pa[kMaxSweepRoots + 1], s_pb[kMaxSweepRoots + 1];
  __shared__ RootSweep s_rs[kMaxSweepRoots];
  __shared__ unsigned s_per;
  const int lane = threadIdx.x & 31;
  const unsigned gwarp = (blockIdx.x * kBlock + threadIdx.x) >> 5;
  const unsigned nwarps = (gridDim.x * kBlock) >> 5;
  const unsigned gthread = blockIdx.x * kBlock + threadIdx.x;
  const unsigned nthreads = gridDim.x * kBlock;
  for (int r = threadIdx.x; r < p.k; r += kBlock) {
    s_rs[r] = p.rs[r];
    if (p.inv) s_rs[r].root = __ldg(p.inv + s_rs[r].root);
  }
  __syncthreads();
  for (int D = p.dmax - 1; D >= 0; --D) {
    /* the step's plan, identical in every CTA: per root, its phase-A items
     * and hubs to combine, as prefixes over the roots */
    if (threadIdx.x < 32) { /* lane r: root r's counts, then prefixes over the lanes */
      unsigned c[4] = {0u, 0u, 0u, 0u};
      if (lane < p.k) step_counts(s_rs[lane], D, c);
      /* lists per warp item: as many as leave two items for every warp */
      unsigned all = __reduce_add_sync(FULL, c[1]) / (2u * nwarps);
      const unsigned per = all < 1u ? 1u : all > 8u ? 8u : all;
      if (lane == 0) s_per = per;
      const unsigned a = c[0] + (c[1] + per - 1u) / per + c[2], b = c[3];
      unsigned ia = a, ib = b;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned ta = __shfl_up_sync(FULL, ia, o), tb = __shfl_up_sync(FULL, ib, o);
        if (lane >= o) {
          ia += ta;
          ib += tb;
        }
      }
      if (lane < p.k) {
        s_pa[lane] = ia - a;
        s_pb[lane] = ib - b;
      }
      if (lane == p.k - 1) {
        s_pa[p.k] = ia;
        s_pb[p.k] = ib;
      }
    }
    /* work counter of step D-2 (last used at step D+2) */
    if (gthread == 0) p.ctl->work[(D + 2) & 3] = 0u;
    __syncthreads();
    const unsigned items = s_pa[p.k], hubs = s_pb[p.k], per = s_per;
    /* items: static first, then claimed; each root's long items come first */
    unsigned it = gwarp;
    while (it < items) {
      const int r = root_of(s_pa, p.k, it);
      sweep_item(p, s_rs[r], D, it - s_pa[r], per);
      if (items <= nwarps) break;
      unsigned nxt = 0;
      if (lane == 0) nxt = nwarps + atomicAdd(&p.ctl->work[D & 3], 1u);
      it = __shfl_sync(FULL, nxt, 0);
    }
    if (hubs > 0) { /* the hubs of level D: their segment sums in order */
      if (!grid_barrier(p.ctl, p.timeout_ns, D)) return;
      for (unsigned t = gthread; t < hubs; t += nthreads) {
        const int r = root_of(s_pb, p.k, t);
        const RootSweep &R = s_rs[r];
        const int i = __ldg(R.off + R.classes * D) + (int)(t - s_pb[r]);
        const int v = __ldg(R.list + i);
        const int s0 = __ldg(R.hseg + i);
        const int s1 = s0 + (__ldg(p.rp + v + 1) - __ldg(p.rp + v) + kSeg - 1) / kSeg;
        double acc = __ldcg(R.part + s0);
        for (int sg = s0 + 1; sg < s1; ++sg) acc = __dadd_rn(acc, __ldcg(R.part + sg));
        finish(R, D, v, acc);
      }
    }
    if (!grid_barrier(p.ctl, p.timeout_ns, D)) return;
  }
}

/* bc[v] += dl_r[v] for the roots r of a launch, in order (dl is 0 where the
 * root did not reach v and at the root itself) */
__global__ void bc_add_kernel(double *bc, const double *dl, int k, int n) {
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (long long)gridDim.x * blockDim.x) {
    double x = bc[v];
    for (int r = 0; r < k; ++r) x = __dadd_rn(x, dl[(size_t)r * n + v]);
    bc[v] = x;
  }
}

/* ---- vertices grouped by depth and class (counting sort, block-aggregated),
 * for all roots of a launch at once: blockIdx.y is the root.  Sixteen launches
 * and a wait per root (a sort by depth, then flags, prefixes and position maps
 * of the classes) took 105 us of an RMAT-18 root; three launches for sixteen
 * roots take 80 us in all. ---- */

/* key of v (classes * depth + class), or -1 if the root does not reach it; segs = its
 * segments if it is a hub */
__device__ __forceinline__ int sort_key(const RootSweep &R, const int *rp, int v, int &segs) {
  const int d = __ldg(R.S + v);
  segs = 0;
  if (d < 0) return -1;
  const int deg = __ldg(rp + v + 1) - __ldg(rp + v);
  if (deg > kSeg) {
    segs = (deg + kSeg - 1) / kSeg;
    return R.classes * d + C_HUB;
  }
  int c = C_WARP;
  if (deg < kWarpDegree) {
    c = C_LANE;
    if (R.classes == kClasses) c += deg >= 16 ? 0 : deg >= 8 ? 1 : deg >= 4 ? 2 : 3;
  }
  return R.classes * d + c;
}

/* off[key] = vertices of that key, seg[d] = segments of level d (zero before) */
__global__ void level_count_kernel(const RootSweep *rs, const int *rp, int n) {
  __shared__ int h[kSmemKeys];
  const RootSweep R = rs[blockIdx.y];
  const int keys = R.classes * R.levels;
  const bool local = keys <= kSmemKeys;
  if (local)
    for (int k = threadIdx.x; k < keys; k += blockDim.x) h[k] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kTile;
  for (int j = threadIdx.x; j < kTile; j += blockDim.x) {
    const long long v = base + j;
    if (v >= n) break;
    int segs;
    const int k = sort_key(R, rp, (int)v, segs);
    if (k < 0) continue;
    atomicAdd(local ? &h[k] : &R.off[k], 1);
    if (segs) atomicAdd(&R.seg[k / R.classes], segs);
  }
  __syncthreads();
  if (local)
    for (int k = threadIdx.x; k < keys; k += blockDim.x)
      if (h[k]) atomicAdd(&R.off[k], h[k]);
}

/* a[0..len] -> exclusive prefix, copied to b, by one block */
__device__ void block_prefix(int *a, int *b, int len, int *s_warp) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int carry = 0;
  for (int i0 = 0; i0 <= len; i0 += blockDim.x) {
    const int i = i0 + threadIdx.x;
    const int x = i < len ? a[i] : 0;
    int inc = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    int before = carry, all = 0;
    for (int ww = 0; ww < (int)(blockDim.x >> 5); ++ww) {
      const int t = s_warp[ww];
      before += ww < w ? t : 0;
      all += t;
    }
    if (i <= len) a[i] = b[i] = before + inc - x;
    carry += all;
    __syncthreads();
  }
}

__global__ void level_prefix_kernel(const RootSweep *rs) {
  __shared__ int s_warp[32];
  const RootSweep R = rs[blockIdx.y];
  if (blockIdx.x == 0) block_prefix(R.off, R.fill, R.classes * R.levels, s_warp);
  else block_prefix(R.seg, R.seg_fill, R.levels, s_warp);
}

/* list[...] = vertices by key, and the hubs' segments */
__global__ void level_fill_kernel(const RootSweep *rs, const int *rp, int n) {
  __shared__ int h[kSmemKeys];
  const RootSweep R = rs[blockIdx.y];
  const int keys = R.classes * R.levels;
  const bool local = keys <= kSmemKeys;
  if (local)
    for (int k = threadIdx.x; k < keys; k += blockDim.x) h[k] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kTile;
  if (local) {
    for (int j = threadIdx.x; j < kTile; j += blockDim.x) {
      const long long v = base + j;
      if (v >= n) break;
      int segs;
      const int k = sort_key(R, rp, (int)v, segs);
      if (k >= 0) atomicAdd(&h[k], 1);
    }
    __syncthreads();
    /* reserve this block's range of every key, then hand out positions */
    for (int k = threadIdx.x; k < keys; k += blockDim.x)
      if (h[k]) h[k] = atomicAdd(&R.fill[k], h[k]);
    __syncthreads();
  }
  for (int j = threadIdx.x; j < kTile; j += blockDim.x) {
    const long long v = base + j;
    if (v >= n) break;
    int segs;
    const int k = sort_key(R, rp, (int)v, segs);
    if (k < 0) continue;
    const int i = atomicAdd(local ? &h[k] : &R.fill[k], 1);
    R.list[i] = (int)v;
    if (segs) {
      const int s0 = atomicAdd(&R.seg_fill[k / R.classes], segs);
      R.hseg[i] = s0;
      for (int t = 0; t < segs; ++t) R.seg_pos[s0 + t] = i;
    }
  }
}

/* out[j] = in[inv[j]] (or in[j]) */
__global__ void gather_double_kernel(const double *in, const int *inv, int n, double *out) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < n) out[j] = in[inv ? inv[j] : j];
}

}  // namespace
}  // namespace tbfs

using tbfs::RootSweep;
using tbfs::SweepCtl;
using tbfs::SweepParams;

namespace {

tbfs_status bfail(cudaError_t e, const char *what) {
  tbfs_set_error("tbfs_brandes: %s: %s", what, cudaGetErrorString(e));
  return e == cudaErrorMemoryAllocation ? TBFS_ERR_OUT_OF_MEMORY : TBFS_ERR_CUDA;
}

#define BTRY(call, what)                            \
  do {                                              \
    cudaError_t e_ = (call);                        \
    if (e_ != cudaSuccess) return bfail(e_, what);  \
  } while (0)

/* the call's device memory, one block */
struct Scratch {
  char *base = nullptr;
  size_t used = 0;
  ~Scratch() { tbfs::dev_free(base); }
  template <class T>
  T *take(size_t count) {
    T *p = reinterpret_cast<T *>(base + used);
    used += (count * sizeof(T) + 255) / 256 * 256;
    return p;
  }
};

}  // namespace

extern "C" tbfs_status tbfs_brandes(tbfs_graph *g, const int32_t *roots, int32_t k,
                                    const tbfs_options *opt, double *bc, int32_t *overflow) {
  tbfs_options o;
  tbfs_options_init(&o);
  if (opt) o = *opt;
  if (!g || k < 0 || (k > 0 && !roots) || !bc) {
    tbfs_set_error("tbfs_brandes: null graph, roots or bc, or k < 0");
    return TBFS_ERR_INVALID_ARG;
  }
  for (int32_t i = 0; i < k; ++i)
    if (roots[i] < 0 || roots[i] >= g->n) {
      tbfs_set_error("tbfs_brandes: root %d (index %d) outside [0, n)", roots[i], i);
      return TBFS_ERR_INVALID_ARG;
    }
  BTRY(cudaSetDevice(g->device), "cudaSetDevice");
  cudaStream_t s = (cudaStream_t)o.stream;
  const size_t n = (size_t)g->n;
  /* roots per sweep launch: up to kMaxSweepRoots, fewer on large graphs
   * (each root holds about 80 n bytes while its launch runs) */
  int K = k < tbfs::kMaxSweepRoots ? (k > 0 ? k : 1) : tbfs::kMaxSweepRoots;
  while (K > 1 && (double)K * 80.0 * (double)n > 16e9) K /= 2;
  /* segments: each hub has deg > kSeg, so sum of ceil(deg / kSeg) < 2 nnz / kSeg + 1 */
  const size_t seg_cap = (size_t)(2 * g->nnz / tbfs::kSeg + 1);
  /* keys of at most n levels: six classes up to kSmemKeys keys, else three */
  const size_t key_cap = std::max((size_t)tbfs::kSmemKeys, tbfs::kClassesFew * (n + 1)) + 1;
  std::vector<RootSweep> rs((size_t)K);
  Scratch w;
  double *dl = nullptr, *qs = nullptr, *sum = nullptr;
  int *offs = nullptr, *segs = nullptr;
  RootSweep *rs_dev = nullptr;
  SweepCtl *ctl = nullptr;
  for (int pass = 0; pass < 2; ++pass) { /* sizes first, then the views */
    w.used = 0;
    dl = w.take<double>((size_t)K * n);
    qs = w.take<double>((size_t)K * 2 * n);
    sum = w.take<double>(n);
    rs_dev = w.take<RootSweep>((size_t)K);
    ctl = w.take<SweepCtl>(1);
    offs = w.take<int>((size_t)K * key_cap);
    segs = w.take<int>((size_t)K * (n + 2));
    for (int j = 0; j < K; ++j) {
      RootSweep &R = rs[(size_t)j];
      R.S = w.take<int>(n);
      R.sig = w.take<unsigned long long>(n);
      R.list = w.take<int>(n);
      R.off = offs + (size_t)j * key_cap;
      R.fill = w.take<int>(key_cap);
      R.q[0] = qs + (size_t)j * 2 * n;
      R.q[1] = R.q[0] + n;
      R.dl = dl + (size_t)j * n;
      R.seg = segs + (size_t)j * (n + 2);
      R.seg_fill = w.take<int>(n + 2);
      R.seg_pos = w.take<int>(seg_cap);
      R.hseg = w.take<int>(n);
      R.part = w.take<double>(seg_cap);
    }
    if (pass == 0) BTRY(tbfs::dev_alloc(&w.base, w.used), "alloc");
  }
  BTRY(cudaMemsetAsync(sum, 0, n * sizeof(double), s), "clear");
  /* grid of the sweep: all SMs, as occupancy allows (cooperative) */
  int sms = 0, per = 0;
  BTRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device), "attribute");
  BTRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, tbfs::sweep_kernel, tbfs::kBlock, 0),
       "occupancy");
#ifndef TBFS_SWEEP_PER_SM
#define TBFS_SWEEP_PER_SM 4 /* 4 CTAs of 256 per SM measured 11 % faster than 2 */
#endif
  if (per > TBFS_SWEEP_PER_SM) per = TBFS_SWEEP_PER_SM;
  const unsigned grid = (unsigned)(sms * (per > 0 ? per : 1));
  const unsigned tiles = (unsigned)((n + tbfs::kTile - 1) / tbfs::kTile);
  const unsigned cgrid = (unsigned)((n + 1 + 255) / 256);
  const long long timeout = o.timeout_ns > 0 ? o.timeout_ns : 4000000000LL;
  int32_t ovf_roots = 0;
  tbfs_options fo = o;
  fo.want_sigma = 1;
  fo.outputs_on_device = 1;
  fo.level_trace = nullptr;
  fo.level_trace_cap = 0;
  for (int32_t r0 = 0; r0 < k; r0 += K) {
    const int kk = k - r0 < K ? k - r0 : K;
    int dmax = 0;
    size_t key_max = 0;
    BTRY(cudaMemsetAsync(dl, 0, (size_t)kk * n * sizeof(double), s), "clear");
    BTRY(cudaMemsetAsync(qs, 0, (size_t)kk * 2 * n * sizeof(double), s), "clear");
    /* the forward traversals, one after another without a wait between them */
    tbfs::BfsCtl *fc = nullptr;
    {
      std::vector<tbfs::ForwardRoot> fr((size_t)kk);
      for (int j = 0; j < kk; ++j)
        fr[(size_t)j] = {roots[r0 + j], rs[(size_t)j].S, rs[(size_t)j].sig};
      tbfs_status st = tbfs::forward_internal(g, fr.data(), kk, fo, s, &fc);
      if (st != TBFS_OK) return st;
    }
    BTRY(cudaStreamSynchronize(s), "forward traversal");
    for (int j = 0; j < kk; ++j) {
      if (fc[j].status != 0) {
        tbfs_set_error("tbfs_brandes: forward traversal: grid barrier wait exceeded its budget");
        return TBFS_ERR_TIMEOUT;
      }
      if (fc[j].sigma_overflow) ++ovf_roots;
      rs[(size_t)j].levels = fc[j].levels;
      rs[(size_t)j].classes =
          tbfs::kClasses * fc[j].levels <= tbfs::kSmemKeys ? tbfs::kClasses : tbfs::kClassesFew;
      key_max = std::max(key_max, (size_t)(rs[(size_t)j].classes * (long long)fc[j].levels));
      rs[(size_t)j].root = roots[r0 + j];
      dmax = fc[j].levels > dmax ? fc[j].levels : dmax;
    }
    BTRY(cudaMemcpyAsync(rs_dev, rs.data(), (size_t)kk * sizeof(RootSweep), cudaMemcpyHostToDevice,
                         s),
         "sweep descriptors");
    /* vertices by depth and class */
    BTRY(cudaMemset2DAsync(offs, key_cap * sizeof(int), 0,
                           (key_max + 1) * sizeof(int), (size_t)kk, s),
         "clear");
    BTRY(cudaMemset2DAsync(segs, (n + 2) * sizeof(int), 0, ((size_t)dmax + 1) * sizeof(int),
                           (size_t)kk, s),
         "clear");
    const dim3 by_root(tiles, (unsigned)kk);
    tbfs::level_count_kernel<<<by_root, tbfs::kBlock, 0, s>>>(rs_dev, g->rp, g->n);
    tbfs::level_prefix_kernel<<<dim3(2, (unsigned)kk), 1024, 0, s>>>(rs_dev);
    tbfs::level_fill_kernel<<<by_root, tbfs::kBlock, 0, s>>>(rs_dev, g->rp, g->n);
    BTRY(cudaGetLastError(), "vertices by depth");
    BTRY(cudaMemsetAsync(ctl, 0, sizeof(SweepCtl), s), "clear");
    SweepParams p;
    p.rp = g->rp;
    p.jr = g->jr;
    p.inv = g->inv;
    p.rs = rs_dev;
    p.k = kk;
    p.dmax = dmax;
    p.ctl = ctl;
    p.timeout_ns = timeout;
    void *args[] = {&p};
    BTRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(tbfs::sweep_kernel), dim3(grid),
                                     dim3(tbfs::kBlock), args, 0, s),
         "dependency sweep");
    tbfs::bc_add_kernel<<<cgrid, 256, 0, s>>>(sum, dl, kk, g->n);
    BTRY(cudaGetLastError(), "bc sums");
    SweepCtl sc;
    BTRY(cudaMemcpyAsync(&sc, ctl, sizeof(sc), cudaMemcpyDeviceToHost, s), "read sweep status");
    BTRY(cudaStreamSynchronize(s), "dependency sweep");
    if (sc.status != 0) {
      tbfs_set_error("tbfs_brandes: sweep: grid barrier wait exceeded its budget");
      return TBFS_ERR_TIMEOUT;
    }
  }
  /* results in the caller's numbering */
  double *dst = bc;
  if (!o.outputs_on_device) dst = dl; /* free again */
  tbfs::gather_double_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(sum, g->inv, g->n, dst);
  BTRY(cudaGetLastError(), "gather");
  if (!o.outputs_on_device)
    BTRY(cudaMemcpyAsync(bc, dst, n * sizeof(double), cudaMemcpyDeviceToHost, s), "copy bc");
  BTRY(cudaStreamSynchronize(s), "results");
  if (overflow) *overflow = ovf_roots;
  return TBFS_OK;
}
