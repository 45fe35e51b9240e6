/*
 * bfs_engine.cu -- one persistent, cooperatively launched kernel runs a whole
 * direction-optimizing BFS: every level is a phase separated by a
 * hand-written grid barrier, and the top-down / bottom-up decision is taken
 * on the device from counters the previous phase produced.  No host round
 * trip happens between levels.
 *
 * What it replaces in the reference: the per-level host loops of
 * TurboBFS_CSC_TD/bfsgputdcsc_sc.cu:95-119 (two launches and two event
 * syncs per level, host reads a managed flag), the bottom-up loop of
 * TurboBFS_CSC_BU/bfsgpubucsc_sc.cu:81-95, and the host-side switch of
 * TurboBFS_CSC_TDBU/bfsgputdbucsc_sc.cu:119-153 (managed float sizef).
 *
 * Level d (frontier F_d = vertices at depth d, held as a queue) discovers
 * F_{d+1} either
 *   top-down : edge-balanced push over the out-edges of F_d; an unvisited
 *              target is claimed with atomicCAS(S, -1, d+1) and appended to
 *              the next queue, and (with path counts) every edge that lands
 *              on a vertex at depth d+1 adds sigma[u] to it; or
 *   bottom-up: every unvisited vertex scans its in-list.  Depths only: it
 *              stops at the first in-neighbour in F_d (frontier bitmap).
 *              With path counts: it sums its in-neighbours' counts, which
 *              discovers and counts in one pass (pull_item).
 *
 * Path counts.  sigma[v] = sum of sigma[u] over the entries u->v with
 * S[u] = S[v]-1.  The counts of even and odd depths are kept in two arrays,
 * both zero where nothing was counted.  An in-neighbour of a vertex still
 * unvisited in phase d has depth d, or is unvisited itself: nothing above
 * level d can reach it first.  So the sum over ALL in-neighbours of the array
 * of d's parity is exactly the sum over the parents (a neighbour found in
 * this phase is counted in the other array), and it is nonzero exactly when
 * the vertex has a parent: a bottom-up level needs one gather per list entry
 * and no frontier test.  This holds while no count has wrapped to zero; once
 * an overflow is recorded the parents are found by their depth instead.
 * Before, a bottom-up level stopped at the first parent and the next phase
 * read the lists again for the counts (a push of 52 M entries with 40 M L2
 * reductions on RMAT-22's heaviest level).
 * Counts are exact in uint64 arithmetic; any sum that reaches 2^63 sets
 * ctl->sigma_overflow (overflow is reported, never rounded).
 *
 * Edge-balanced expansion: each queue entry carries the vertex, the
 * exclusive prefix of out-degrees (its offset in the level's flattened edge
 * space) and the start of its list.  A warp takes a contiguous range of
 * flattened edges, stages 128 queue entries at a time in shared memory, and
 * every lane handles kEPT consecutive edges per round, so that many list
 * reads, then that many depth gathers, are in flight per lane.  On graphs
 * without long out-lists (kShortList, kNarrowList) the kernel
 * instances bfs_persistent_kernel<true, .> cut small top-down levels into
 * items of kShortEntries whole queue entries instead, which need no owner
 * search (the chain of dependent L2 round trips is what a small level
 * costs), and run narrow levels without the global queue (narrow_levels);
 * other graphs run the instance compiled without these.
 *
 * Direction rule (device side; after Beamer, Asanovic, Patterson,
 * "Direction-optimizing breadth-first search", SC 2012): a level runs
 * bottom-up when alpha times the frontier's out-edges exceed the unexplored
 * edges plus the cost of visiting every vertex's word; a frontier of more
 * than n/beta vertices does not leave bottom-up, a smaller one does at once
 * without path counts, and with them when the levels' excess has paid for it
 * (kLeaveCost).  The comparisons are in fp32: every thread evaluates them at
 * every level, and fp64 issues slowly on this part (in fp64 they cost about 0.7
 * us per level).
 *
 * Memory model.  Queues and counters are read with ld.global.cg (L2).
 * Depth and path-count gathers use ordinary (L1-cacheable) loads: every
 * value a test acts on -- S == d-1, S == d, S == d+1 claimed earlier in this
 * phase only through an atomic's return value, sigma of a finished level --
 * was written before the last grid barrier, whose gpu-scope acquire makes it
 * visible to every later load of the CTA.  A plain load can return a stale
 * -1 for a vertex claimed during this phase; the engine then only attempts
 * an atomicCAS, whose return value is authoritative.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "device_common.cuh"
#include "tbfs_internal.h"

#ifndef TBFS_EPT
#define TBFS_EPT 6
#endif
#ifndef TBFS_SHORT_CAS_FIRST
#define TBFS_SHORT_CAS_FIRST 1 /* aligned items claim with the CAS alone */
#endif
namespace tbfs {
namespace {

using dev::FULL;
using dev::add_chk;
using dev::global_ns;
using dev::grid_barrier;
using dev::warp_find_owner;
constexpr int kBlock = 1024;       /* threads of a full CTA, one CTA per SM */
/* ... on short-list graphs: levels that are latency alone want registers (a
 * barrier's acquire drops L1, so a spilled value costs a round trip to L2) */
constexpr int kShortBlock = 512;
constexpr long long kLargeEntries = 48 << 20; /* list entries from which a frontier
                                                 filter is used (bfs_launch) */
constexpr int kLargeVertices = 400000; /* vertices from which AUTO takes all threads */
constexpr int kBlockStep = 256;    /* threads per unit of ctas_per_sm */
constexpr int kFilterBits = 1 << 18; /* frontier filter in shared memory (32 KB) */
constexpr int kWin = 128;          /* queue entries staged per warp window */
constexpr int kEPT = TBFS_EPT;     /* most consecutive edges per lane/round */
/* queue entries per item of a small level of a short-list graph: 128 edges, one
 * round of at most 4 per lane, if the lists have kShortList entries */
constexpr unsigned kShortEntries = 8;
constexpr float kBuWordCost = 4.0f; /* a bitmap word of a bottom-up level, in list entries */
enum { DIR_TD = 0, DIR_BU = 1 };

/* A bottom-up level with path counts scans every unvisited vertex's whole
 * list where one without stops at the first parent, so it must beat the push
 * by more: alpha is scaled by this (15 -> 5.25).  RMAT-22, a level of 21.3 M
 * out-edges with 107 M unexplored: top-down 417 us, bottom-up 301; of 9.9 M
 * with 118 M: top-down 247. */
constexpr float kSigmaAlpha = 0.35f;
/* unexplored entries from which a bottom-up level with path counts is cut
 * into items of equal cost (a few hundred entries per warp) ... */
constexpr float kHeavyEntries = 3e5f;
constexpr float kHeavyShare = 0.25f; /* ... and of all entries: else words of
                                        visited hubs make most of the items */
/* entries per frontier vertex from which a frontier filter pays: every CTA
 * reads the whole queue to fill its own */
constexpr float kFilterGain = 300.0f;
/* Leaving bottom-up with path counts, in list entries (~270 K take a
 * microsecond): a bottom-up level reads every vertex's depth and no queue, which
 * together cost more than a top-down one by kScanVertex per vertex less
 * kQueueCost (narrow levels: plus kNarrowGain); leaving costs one pass over the
 * depths, that collects the queue, and kLeaveCost.  A level's excess alone seldom
 * pays for that, but the tail of a deep graph has many: they are added up, and
 * the traversal leaves once they would have.  (RMAT of 2^22 and a chain of 2000,
 * us per level of the chain: 13.9 bottom-up, 7.5 top-down, RMAT of 2^20 8.3 and
 * 7.1, of 2^16 6.4 and 6.6.  With one level's excess compared, as little as
 * kLeaveCost unexplored entries kept every level of the tail bottom-up.) */
constexpr float kScanVertex = 0.48f, kQueueCost = 1.8e5f, kNarrowGain = 9e5f;
constexpr float kLeaveCost = 2.2e5f;

/* Shared memory of a warp that expands: a window of queue entries. */
struct ExpandWin {
  /* sigma of the entry as low and high words in separate arrays, so that
   * neighbouring entries fall in different banks */
  unsigned lo[kWin], hi[kWin];
  int v[kWin];                  /* vertex of the entry                      */
  int a[kWin];                  /* list index of its first window edge      */
  unsigned s[kWin + 1];         /* window-relative start of its edges       */
};

/* Append, for every lane, the entries j < N with bit j of `take` set to the
 * next level's queue (q, e, a): one 64-bit atomic per warp reserves
 * (count << 32 | out-edge sum), so queue positions and edge offsets come from
 * the same reservation and e[] stays the exclusive prefix of out-degrees in
 * queue order.  Must be called by all 32 lanes. */
template <int N>
__device__ __forceinline__ void warp_append(unsigned take, const int (&vv)[N],
                                            const int (&dg)[N], const int (&ad)[N], int *q,
                                            int *e, int *a, unsigned long long *ctr) {
  const int lane = threadIdx.x & 31;
  const int cnt = __popc(take);
  int dsum = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if ((take >> j) & 1u) dsum += dg[j];
  int ic = cnt, id = dsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int tc = __shfl_up_sync(FULL, ic, o);
    const int td = __shfl_up_sync(FULL, id, o);
    if (lane >= o) {
      ic += tc;
      id += td;
    }
  }
  const int tot_c = __shfl_sync(FULL, ic, 31);
  if (tot_c == 0) return;
  const int tot_d = __shfl_sync(FULL, id, 31);
  unsigned long long base = 0;
  if (lane == 31)
    base = atomicAdd(ctr, ((unsigned long long)tot_c << 32) | (unsigned)tot_d);
  base = __shfl_sync(FULL, base, 31);
  unsigned pos = (unsigned)(base >> 32) + (unsigned)(ic - cnt);
  unsigned eo = (unsigned)base + (unsigned)(id - dsum);
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if ((take >> j) & 1u) {
      q[pos] = vv[j];
      e[pos] = (int)eo;
      a[pos] = ad[j];
      ++pos;
      eo += (unsigned)dg[j];
    }
  }
}


/* A level's queue: entries i < qn with vertex q[i], edge offset e[i], list
 * start a[i]; qe is the total of its out-degrees. */
struct Queue {
  const int *q, *e, *a;
  unsigned qn, qe;
};

/* Output queue of the level being discovered. */
struct NextQueue {
  int *q, *e, *a;
  unsigned long long *ctr;
};

__device__ __forceinline__ bool bit_of(const unsigned *bm, int v) {
  return (bm[(unsigned)v >> 5] >> ((unsigned)v & 31u)) & 1u;
}

/* One warp expands the flattened out-edge range [E0, E1) of queue Q: claims
 * unvisited targets at depth d+1 into `nx` (depths only: and bitmap nb).
 * SIG: every edge whose target is at depth d+1 afterwards adds its source's
 * count (src) to the target's (dst); CHK: each add is checked for overflow. */
template <bool SIG, bool CHK = true, bool ALIGNED = false>
__device__ __forceinline__ void expand_chunk(const BfsParams &p, int d, const Queue &Q,
                                             unsigned E0, unsigned E1, unsigned ept,
                                             const NextQueue &nx,
                                             const unsigned long long *src,
                                             unsigned long long *dst, unsigned *nb, ExpandWin &w,
                                             bool &ovf, unsigned first = 0, unsigned count = 0) {
  const int lane = threadIdx.x & 31;
  /* ALIGNED item: entries [first, first + count), all their edges, one
   * window; E0 = 0 and E1 = ~0u, so the window offsets below are the
   * entries' own edge offsets and no owner search is needed */
  constexpr bool aligned = ALIGNED;
  unsigned i0 = aligned ? first : warp_find_owner(Q.e, Q.qn, E0);
  unsigned pos = E0;
  while (pos < E1 && i0 < Q.qn) {
    unsigned nw = (Q.qn - i0) < (unsigned)kWin ? (Q.qn - i0) : (unsigned)kWin;
    if (aligned && count < nw) nw = count;
    for (unsigned k = lane; k < nw; k += 32) {
      const unsigned i = i0 + k;
      const unsigned eb = (unsigned)__ldcg(Q.e + i);
      const unsigned b = eb > pos ? eb : pos;
      const unsigned bc = b < E1 ? b : E1;
      const int v = __ldcg(Q.q + i);
      w.v[k] = v;
      w.a[k] = __ldcg(Q.a + i) + (int)(b - eb);
      w.s[k] = bc - pos;
      if (SIG && !aligned) {
        const unsigned long long x = src[v];
        w.lo[k] = (unsigned)x;
        w.hi[k] = (unsigned)(x >> 32);
      }
    }
    if (lane == 0) {
      const unsigned ee = (i0 + nw < Q.qn) ? (unsigned)__ldcg(Q.e + i0 + nw) : Q.qe;
      w.s[nw] = (ee < E1 ? ee : E1) - pos;
    }
    __syncwarp();
    /* window edges t in [s[0], s[nw]): s[0] = 0 for an edge chunk, the
     * first entry's edge offset for an entry-aligned item */
    const unsigned t_beg = aligned ? w.s[0] : 0u, tot = w.s[nw];
    if (aligned) { /* one round when it fits: (edges + 31) / 32 per lane */
      const unsigned per = (tot - t_beg + 31u) / 32u;
      ept = per < 1u ? 1u : (per > ept ? ept : per);
    }
    const unsigned round = 32u * ept;
    for (unsigned base = t_beg; base < tot; base += round) {
      const unsigned t0 = base + (unsigned)lane * ept;
      const unsigned tend = t0 + ept < tot ? t0 + ept : tot;
      int u[kEPT], kk[kEPT];
      unsigned valid = 0;
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        kk[j] = 0;
        u[j] = 0;
      }
      if (t0 < tot) {
        unsigned lo = 0, hi = nw - 1; /* largest k with s[k] <= t0 */
        while (lo < hi) {
          const unsigned mid = (lo + hi + 1) >> 1;
          if (w.s[mid] <= t0) lo = mid;
          else hi = mid - 1;
        }
        unsigned k = lo;
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          const unsigned t = t0 + j;
          if (t < tend) {
            while (w.s[k + 1] <= t) ++k;
            u[j] = w.a[k] + (int)(t - w.s[k]);
            kk[j] = (int)k;
            valid |= 1u << j;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kEPT; ++j) /* list reads, all in flight */
        if ((valid >> j) & 1u) u[j] = __ldg(p.jr + u[j]);
      /* an aligned item reads its entries' path counts with the list
       * entries instead of staging them first: one round trip fewer */
      unsigned long long xs[kEPT];
      if (aligned && SIG) {
#pragma unroll
        for (int j = 0; j < kEPT; ++j) xs[j] = ((valid >> j) & 1u) ? src[w.v[kk[j]]] : 0ull;
      }
      int su[kEPT]; /* depth of the target */
      /* an aligned item may claim with the CAS alone: its return value is
       * the depth the plain read would have given */
      constexpr bool cas_first = aligned && TBFS_SHORT_CAS_FIRST;
      int ad[kEPT], dg[kEPT];
      if (cas_first) {
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          su[j] = -2;
          ad[j] = 0;
          dg[j] = 0;
          if ((valid >> j) & 1u) {
            su[j] = atomicCAS(p.S + u[j], -1, d + 1);
            ad[j] = __ldg(p.rp + u[j]);
            dg[j] = __ldg(p.rp + u[j] + 1) - ad[j];
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < kEPT; ++j) su[j] = ((valid >> j) & 1u) ? p.S[u[j]] : -2;
      }
      unsigned hit = 0; /* targets at depth d+1 after this edge */
      unsigned take = 0;
      if (cas_first) {
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          if (su[j] == -1) take |= 1u << j;
          else if (su[j] == d + 1) hit |= 1u << j;
        }
      } else {
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          if (su[j] == -1) {
            const int old = atomicCAS(p.S + u[j], -1, d + 1);
            if (old == -1) take |= 1u << j;
            else if (old == d + 1) hit |= 1u << j;
          } else if (su[j] == d + 1) {
            hit |= 1u << j;
          }
        }
      }
      hit |= take;
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        if (!cas_first) {
          ad[j] = 0;
          dg[j] = 0;
        }
        if ((take >> j) & 1u) {
          if (!cas_first) {
            ad[j] = __ldg(p.rp + u[j]);
            dg[j] = __ldg(p.rp + u[j] + 1) - ad[j];
          }
          if (!SIG) atomicOr(nb + ((unsigned)u[j] >> 5), 1u << ((unsigned)u[j] & 31u));
        }
      }
      warp_append<kEPT>(take, u, dg, ad, nx.q, nx.e, nx.a, nx.ctr);
      if (SIG) {
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          if ((hit >> j) & 1u) {
            const unsigned long long x =
                aligned ? xs[j]
                        : ((unsigned long long)w.hi[kk[j]] << 32) | (unsigned long long)w.lo[kk[j]];
            if (CHK) add_chk(atomicAdd(dst + u[j], x), x, ovf);
            else atomicAdd(dst + u[j], x); /* result unused: a reduction, no round trip */
          }
        }
      }
    }
    __syncwarp();
    if (aligned) break;
    pos += tot;
    i0 += nw;
  }
}

/* How one expansion of queue Q is cut into work items (edge chunks).
 * Small frontiers use fewer edges per lane (down to one), so their work is
 * spread over more warps and each lane's chain of dependent loads is short;
 * large frontiers use kEPT for memory-level parallelism.  About four chunks
 * per warp keep the dynamic scheduler balanced. */
struct ExpandPlan {
  unsigned ept, ch, nch;
};

__device__ __forceinline__ ExpandPlan plan_expand(unsigned qe, unsigned nwarps, unsigned max_ept) {
  ExpandPlan pl;
  const unsigned per_lane = (qe + 32u * nwarps - 1) / (32u * nwarps);
  pl.ept = per_lane < 1u ? 1u : (per_lane > max_ept ? max_ept : per_lane);
  const unsigned round = 32u * pl.ept;
  unsigned ch = (qe + 4u * nwarps - 1) / (4u * nwarps);
  ch = (ch + round - 1) / round * round;
  if (ch < round) ch = round;
  if (ch > 16u * round) ch = 16u * round;
  pl.ch = ch;
  pl.nch = (qe + ch - 1) / ch;
  return pl;
}

/* a top-down level: queue, how it is cut, where its counts come from and go */
struct ExpandTask {
  Queue Q;
  ExpandPlan pl;
  const unsigned long long *src;
  unsigned long long *dst;
  bool chk;                /* check every add for overflow */
};

template <bool SIG>
__device__ __forceinline__ void run_expand_item(const BfsParams &p, int d, const ExpandTask &t,
                                                unsigned c, const NextQueue &nx, unsigned *nb,
                                                ExpandWin &w, bool &ovf) {
  const unsigned E0 = c * t.pl.ch;
  const unsigned E1 = E0 + t.pl.ch < t.Q.qe ? E0 + t.pl.ch : t.Q.qe;
  if (!SIG || t.chk)
    expand_chunk<SIG>(p, d, t.Q, E0, E1, t.pl.ept, nx, t.src, t.dst, nb, w, ovf);
  else
    expand_chunk<SIG, false>(p, d, t.Q, E0, E1, t.pl.ept, nx, t.src, t.dst, nb, w, ovf);
}

/* One item of a small top-down level of a short-list graph: queue entries
 * [first, first + kShortEntries) with all their edges (ALIGNED expand_chunk:
 * no owner search). */
template <bool SIG>
__device__ __forceinline__ void run_short_item(const BfsParams &p, int d, const ExpandTask &t,
                                               unsigned first, unsigned max_ept,
                                               const NextQueue &nx, unsigned *nb, ExpandWin &w,
                                               bool &ovf) {
  const unsigned ept = max_ept < 4u ? max_ept : 4u;
  if (!SIG || t.chk)
    expand_chunk<SIG, true, true>(p, d, t.Q, 0u, ~0u, ept, nx, t.src, t.dst, nb, w, ovf, first,
                                  kShortEntries);
  else
    expand_chunk<SIG, false, true>(p, d, t.Q, 0u, ~0u, ept, nx, t.src, t.dst, nb, w, ovf, first,
                                   kShortEntries);
}

/* ---- bottom-up levels ----
 * With path counts, a bottom-up level only counts what it finds (per lane, added up once per
 * warp at the end of the phase): a following bottom-up level needs no queue,
 * and a top-down one collects it from the depths (collect_queue).  Appending
 * during the level, and one work counter for items of two words, cost two
 * atomics on one address per 64 vertices, which L2 takes at ~0.75 G/s: 84 us
 * for a level of RMAT-22 with next to nothing to do. */
struct Found {
  unsigned n, e; /* vertices, their out-edges */
};

/* 32-vertex words a warp looks at together */
constexpr int kBuWords = 8;

/* queue of level d from the depths */
constexpr int kCollectWords = 8;
__device__ __forceinline__ void collect_queue(const BfsParams &p, int d, int *q, int *e, int *a,
                                              unsigned warp, unsigned nwarps) {
  const unsigned lane = threadIdx.x & 31, nwords = ((unsigned)p.n + 31u) >> 5;
  for (unsigned word = warp * kCollectWords; word < nwords; word += nwarps * kCollectWords) {
    int v[kCollectWords], dg[kCollectWords], ad[kCollectWords];
    unsigned take = 0;
#pragma unroll
    for (int j = 0; j < kCollectWords; ++j) {
      v[j] = (int)((word + j) * 32u + lane);
      if (v[j] < p.n && p.S[v[j]] == d) take |= 1u << j;
    }
    if (!__any_sync(FULL, take != 0u)) continue;
#pragma unroll
    for (int j = 0; j < kCollectWords; ++j) {
      dg[j] = ad[j] = 0;
      if ((take >> j) & 1u) {
        ad[j] = __ldg(p.rp + v[j]);
        dg[j] = __ldg(p.rp + v[j] + 1) - ad[j];
      }
    }
    warp_append<kCollectWords>(take, v, dg, ad, q, e, a, &p.ctl->collect);
  }
}

/* Where a bottom-up level finds the counts of level d. */
struct Counts {
  const unsigned long long *src;
  /* frontier filter in the CTA's shared memory: bit u % kFilterBits set for
   * every u in F_d; null where it would not pay */
  const unsigned *filter;
  bool by_depth; /* counts may be zero: parents are found by their depth d */
  int d;
  const int *S;
  bool own; /* no in-list has more than kOwn entries */
};

/* exact sum of counts: 64 bits and the carries out of them */
struct Sum {
  unsigned lo, hi, c;
};

__device__ __forceinline__ void sum_add(Sum &s, unsigned lo, unsigned hi, unsigned c) {
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
      : "+r"(s.lo), "+r"(s.hi), "+r"(s.c)
      : "r"(lo), "r"(hi), "r"(c));
}

/* Entries [lo, hi) of a list by the whole warp: the exact sum of their counts,
 * and whether there is a parent among them. */
__device__ __forceinline__ void sum_exact(const BfsParams &p, const Counts &c, unsigned lo,
                                          unsigned hi, Sum &s, bool &par) {
  s = {0u, 0u, 0u};
  par = false;
  for (unsigned k = lo + (threadIdx.x & 31); k < hi; k += 32u) {
    const int u = __ldg(p.ic + k);
    const unsigned long long x = c.src[u];
    sum_add(s, (unsigned)x, (unsigned)(x >> 32), 0u);
    if (c.by_depth && p.S[u] == c.d) par = true;
  }
  __syncwarp();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned l = __shfl_xor_sync(FULL, s.lo, o), h = __shfl_xor_sync(FULL, s.hi, o);
    const unsigned y = __shfl_xor_sync(FULL, s.c, o);
    sum_add(s, l, h, y);
  }
  par = c.by_depth ? __any_sync(FULL, par) : (s.lo | s.hi | s.c) != 0u;
}

/* Fast sums keep 32 bits: exact while every count is below 2^20 (a list they
 * are used for has at most kHubLen entries); `big` collects the other bits, and
 * a list that shows any is summed again exactly. */
constexpr unsigned kBigCount = ~((1u << 20) - 1u);
static_assert(kHubLen <= 1 << 12, "fast sums must fit 32 bits");

/* the counts of u[0..U) (-1: none) as 32 bits; big collects the other bits.  By
 * depth: 1 for a parent, 0 for others; only lists with a parent are then
 * summed (a level of a grid of 2048 x 2048, all bottom-up: 590 us with every
 * list summed, 30 so) */
template <bool FILTER, int U>
__device__ __forceinline__ void get_fast(const Counts &c, const int (&u)[U], unsigned (&y)[U],
                                         unsigned &big) {
  unsigned long long x[U];
  bool on[U];
#pragma unroll
  for (int j = 0; j < U; ++j) on[j] = u[j] >= 0;
  if (c.by_depth) {
    int sv[U];
#pragma unroll
    for (int j = 0; j < U; ++j) sv[j] = on[j] ? c.S[u[j]] : -1;
#pragma unroll
    for (int j = 0; j < U; ++j) y[j] = sv[j] == c.d ? 1u : 0u;
    return;
  }
  if (FILTER) {
    unsigned f[U];
#pragma unroll
    for (int j = 0; j < U; ++j) f[j] = c.filter[((unsigned)u[j] >> 5) & (kFilterBits / 32u - 1u)];
#pragma unroll
    for (int j = 0; j < U; ++j) on[j] = on[j] && (__funnelshift_r(f[j], f[j], (unsigned)u[j]) & 1u);
  }
#pragma unroll
  for (int j = 0; j < U; ++j) {
    x[j] = 0ull;
    if (on[j]) x[j] = c.src[u[j]];
  }
#pragma unroll
  for (int j = 0; j < U; ++j) {
    y[j] = (unsigned)x[j];
    big |= (unsigned)(x[j] >> 32) | (y[j] & kBigCount);
  }
}

template <bool FILTER, int U>
__device__ __forceinline__ void add_fast(const Counts &c, const int (&u)[U], unsigned &acc,
                                         unsigned &big) {
  unsigned y[U];
  get_fast<FILTER, U>(c, u, y, big);
#pragma unroll
  for (int j = 0; j < U; ++j) acc += y[j];
}

/* Bottom-up discovery with path counts over the vertices [v_lo, v_hi), in
 * groups of 128 (four to a lane), by the length of an unvisited vertex's list:
 * the lane reads up to kOwn entries alone, two of each of its four lists a
 * step; 8 lanes read a list of up to kHalf, the next lists' entries
 * requested before these entries' counts arrive; the whole warp reads a longer
 * one, one pass ahead.  Lists over p.hub_len are left to pull_segment.
 * What bounds a level is latency (a list entry from DRAM and a count from L2
 * are each 700-1500 cycles away with 8 warps per scheduler) and, next to it,
 * instructions.  RMAT-22's heaviest level (76.6 M entries; 5 % in lists of up to
 * 8 entries, 20 % up to 32, 70 % over 64) took 1150 us with groups of one
 * width by the mean length (three quarters of the lanes idle), 376 with the
 * lists laid end to end (100 instructions per 32 entries to find an entry's
 * list and split the sums), 300-355 with 96-bit sums and lists sorted by
 * length in shared memory, 300 word by word without the lookahead, 252 so
 * (against 75 for an early-exit scan and 324 for a push of the counts after
 * it). */
constexpr unsigned kOwn = 8, kHalf = 48; /* kOwn > 2^3 - 1: deg_bits < 4 */
constexpr int kWords = 4; /* words of a group */
static_assert(kWords * 32 <= kWin, "a group's vertices must fit the window");

template <bool FILTER>
__device__ __forceinline__ void pull_range(const BfsParams &p, Found &fd, const Counts &c,
                                           unsigned long long *dst, int v_lo, int v_hi,
                                           ExpandWin &w, bool &ovf) {
  const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
  for (; v_lo < v_hi; v_lo += 32 * kWords) {
    unsigned lo[kWords], hi[kWords]; /* lists the lane reads alone; else hi = lo */
    unsigned mids = 0u, longs = 0u, other = 0u, on = 0u;
    {
#pragma unroll
      for (int j = 0; j < kWords; ++j) {
        const int v = v_lo + 32 * j + (int)lane;
        if (v < v_hi && p.S[v] == -1) on |= 1u << j;
      }
#pragma unroll
      for (int j = 0; j < kWords; ++j) {
        const int v = v_lo + 32 * j + (int)lane;
        lo[j] = hi[j] = 0u;
        if ((on >> j) & 1u) {
          lo[j] = (unsigned)__ldg(p.cp + v);
          hi[j] = (unsigned)__ldg(p.cp + v + 1);
        }
      }
      bool any = false;
#pragma unroll
      for (int j = 0; j < kWords; ++j) {
        unsigned len = hi[j] - lo[j];
        if (len > p.hub_len) len = 0u;
        if (len == 0u) {
          hi[j] = lo[j];
          on &= ~(1u << j);
        }
        any |= len != 0u;
        if (c.own) continue;
        /* to the window: the lists for 8 lanes from the front of v[], those
         * for a warp from its back, both by slot; bounds in lo[], hi[] */
        const bool exact = len > (unsigned)kHubLen;
        const bool is_l = len > kHalf && !exact, is_m = len > kOwn && len <= kHalf && !exact;
        const unsigned mm = __ballot_sync(FULL, is_m), ml = __ballot_sync(FULL, is_l);
        if (((on >> j) & 1u) && (len > kOwn || exact)) {
          other |= 1u << j;
          w.lo[32 * j + lane] = lo[j];
          w.hi[32 * j + lane] = hi[j];
          w.s[32 * j + lane] = 0u;
          w.a[32 * j + lane] = exact ? 1 : 0; /* big */
          if (is_m) w.v[mids + __popc(mm & lt)] = 32 * j + (int)lane;
          if (is_l) w.v[kWin - 1u - longs - __popc(ml & lt)] = 32 * j + (int)lane;
          hi[j] = lo[j];
        }
        mids += __popc(mm);
        longs += __popc(ml);
      }
      if (!__any_sync(FULL, any)) continue;
    }
    __syncwarp();
    if (longs) {
      /* passes of 128 entries, requested one ahead */
      unsigned i = kWin - longs, k = 0u; /* next request: list, first entry */
      auto request = [&](int (&u)[4], int &slot, bool &last) {
        slot = -1;
        if (i >= (unsigned)kWin) return;
        slot = w.v[i];
        const unsigned b = w.lo[slot] + k, e = w.hi[slot];
        const int *a = p.ic + b + lane;
#pragma unroll
        for (int j = 0; j < 4; ++j) u[j] = b + lane + 32u * j < e ? __ldg(a + 32 * j) : -1;
        k += 128u;
        last = b + 128u >= e;
        if (last) {
          ++i;
          k = 0u;
        }
      };
      int u0[4], u1[4], s0, s1;
      bool l0 = false, l1 = false;
      request(u0, s0, l0);
      unsigned a = 0u, b = 0u;
      while (s0 >= 0) {
        request(u1, s1, l1);
        add_fast<FILTER, 4>(c, u0, a, b);
        if (l0) {
          a = __reduce_add_sync(FULL, a);
          b = __reduce_or_sync(FULL, b);
          if (lane == 0) {
            w.s[s0] = a;
            w.a[s0] = (int)b;
          }
          a = b = 0u;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) u0[j] = u1[j];
        s0 = s1;
        l0 = l1;
      }
    }
    if (mids) {
      constexpr int U = kHalf / 8;
      int u[U], t[U];
      auto request = [&](unsigned i) {
        i += lane >> 3;
        const int slot = w.v[i < mids ? i : 0u];
        const unsigned b = w.lo[slot] + (lane & 7u), e = i < mids ? w.hi[slot] : 0u;
        const int *a = p.ic + b;
#pragma unroll
        for (int j = 0; j < U; ++j) u[j] = b + 8u * j < e ? __ldg(a + 8 * j) : -1;
      };
      request(0u);
      for (unsigned i = 0u; i < mids; i += 4u) {
#pragma unroll
        for (int j = 0; j < U; ++j) t[j] = u[j];
        if (i + 4u < mids) request(i + 4u);
        unsigned a = 0u, b = 0u;
        add_fast<FILTER, U>(c, t, a, b);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          a += __shfl_xor_sync(FULL, a, o);
          b |= __shfl_xor_sync(FULL, b, o);
        }
        if ((lane & 7u) == 0u && i + (lane >> 3) < mids) {
          const int slot = w.v[i + (lane >> 3)];
          w.s[slot] = a;
          w.a[slot] = (int)b;
        }
      }
    }
    unsigned acc[kWords], big = 0u; /* big: bit j for the lane's list j */
    unsigned most = 0u;
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
      acc[j] = 0u;
      const unsigned n = hi[j] - lo[j];
      most = most > n ? most : n;
    }
    most = __reduce_max_sync(FULL, most);
    for (unsigned t = 0u; t < most; t += 2u) {
      int u[2 * kWords];
#pragma unroll
      for (int j = 0; j < kWords; ++j) {
        const unsigned k = lo[j] + t;
        u[2 * j] = k < hi[j] ? __ldg(p.ic + k) : -1;
        u[2 * j + 1] = k + 1u < hi[j] ? __ldg(p.ic + k + 1u) : -1;
      }
      unsigned b = 0u, x[2 * kWords];
      get_fast<FILTER, 2 * kWords>(c, u, x, b);
#pragma unroll
      for (int j = 0; j < kWords; ++j) acc[j] += x[2 * j] + x[2 * j + 1];
      if (b) big = ~0u; /* any of the lane's: all its lists again */
    }
    __syncwarp();
    /* vertices with a parent: depth and count */
#pragma unroll
    for (int j = 0; j < kWords; ++j) {
      const int v = v_lo + 32 * j + (int)lane;
      const bool here = (on >> j) & 1u;
      unsigned b = lo[j], e = hi[j], x = acc[j], s_hi = 0u;
      bool redo = here && big != 0u;
      if ((other >> j) & 1u) {
        b = w.lo[32 * j + lane];
        e = w.hi[32 * j + lane];
        x = w.s[32 * j + lane];
        redo = w.a[32 * j + lane] != 0;
      }
      const unsigned n_par = x; /* by depth: parents */
      if (c.by_depth && here && x != 0u) {
        if ((other >> j) & 1u) {
          redo = true;
        } else { /* a short list: the lane alone */
          unsigned long long sum = 0ull;
          for (unsigned k = b; k < e; ++k) sum = add_chk(sum, c.src[__ldg(p.ic + k)], ovf);
          x = (unsigned)sum;
          s_hi = (unsigned)(sum >> 32);
        }
      }
      bool found = x != 0u || s_hi != 0u || (c.by_depth && n_par != 0u);
      for (unsigned m = __ballot_sync(FULL, redo); m; m &= m - 1u) {
        const int l = __ffs(m) - 1;
        Sum s;
        bool par;
        sum_exact(p, c, __shfl_sync(FULL, b, l), __shfl_sync(FULL, e, l), s, par);
        if ((int)lane == l) {
          x = s.lo;
          s_hi = s.hi;
          found = par;
          if (s.c | (s.hi >> 31)) ovf = true;
        }
      }
      if (here && found) {
        p.S[v] = c.d + 1;
        dst[v] = ((unsigned long long)s_hi << 32) | x;
        fd.n += 1u;
        fd.e += p.symmetric ? e - b : (unsigned)(__ldg(p.rp + v + 1) - __ldg(p.rp + v));
      }
    }
    __syncwarp();
  }
}

/* entries [lo, hi) of the list of v by the whole warp */
__device__ __forceinline__ void pull_segment(const BfsParams &p, Found &fd, const Counts &c,
                                             unsigned long long *dst, int v, int lo, int hi,
                                             bool &ovf) {
  const unsigned lane = threadIdx.x & 31;
  unsigned acc = 0u, big = 0u;
  for (unsigned k = (unsigned)lo + lane; k - lane < (unsigned)hi; k += 256u) {
    int u[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j] = k + 32u * j < (unsigned)hi ? __ldg(p.ic + k + 32 * j) : -1;
    add_fast<false, 8>(c, u, acc, big);
  }
  if (c.by_depth) big = acc;
  Sum s = {__reduce_add_sync(FULL, acc), 0u, 0u};
  bool par = s.lo != 0u;
  if (__any_sync(FULL, big != 0u)) sum_exact(p, c, (unsigned)lo, (unsigned)hi, s, par);
  if (lane == 0 && par) {
    const unsigned long long x = ((unsigned long long)s.hi << 32) | s.lo;
    add_chk(atomicAdd(dst + v, x), x, ovf);
    if (s.c) ovf = true;
    if (atomicCAS(p.S + v, -1, c.d + 1) == -1) {
      fd.n += 1u;
      fd.e += (unsigned)(__ldg(p.rp + v + 1) - __ldg(p.rp + v));
    }
  }
}

/* The same for 32 segments of the graph's hub list, kHubLen entries of a longer
 * list each, by the whole warp: i0, i0 + step, ...: neighbours in the list are
 * mostly of one vertex, so that a warp taking 32 in a row would read a whole
 * list alone (87 us of a level whose other work took 70).  Segments of a vertex meet
 * in its count by atomics; the one whose claim of the depth succeeds counts
 * the vertex as found. */
__device__ __forceinline__ void pull_segments(const BfsParams &p, Found &fd, const Counts &c,
                                              unsigned long long *dst, unsigned i0, unsigned step,
                                              unsigned n_seg, bool &ovf) {
  const int lane = threadIdx.x & 31;
  int vs = 0, los = 0, his = 0;
  bool on = false;
  const unsigned i = i0 + (unsigned)lane * step;
  if (i < n_seg) {
    vs = __ldg(p.hub_seg + 2 * i);
    los = __ldg(p.hub_seg + 2 * i + 1);
    const int sv = __ldcg(p.S + vs); /* -1, or d+1 by another segment of this phase */
    on = sv == -1 || sv == c.d + 1;
    if (on) his = __ldg(p.cp + vs + 1);
  }
  for (unsigned m = __ballot_sync(FULL, on); m; m &= m - 1u) {
    const int l = __ffs(m) - 1;
    const int v = __shfl_sync(FULL, vs, l), lo = __shfl_sync(FULL, los, l);
    const int end = __shfl_sync(FULL, his, l), hi = end - lo < kHubLen ? end : lo + kHubLen;
    pull_segment(p, fd, c, dst, v, lo, hi, ovf);
  }
}

/* Bottom-up discovery, depths only.  A warp takes nw <= kBuWords consecutive
 * 32-vertex words (fewer on small graphs, so that every warp has some); lane i owns vertex 32*word+i of each, so the depth checks,
 * list bounds and the first gathers of all kBuWords vertices are in flight
 * together.  An unvisited vertex scans its in-list until the first
 * neighbour in F_d (bitmap cb); the scan advances every still-searching
 * vertex of the lane by one entry per step.  The warp owns its words of the
 * next level's bitmap nb and writes them whole. */
__device__ __forceinline__ void bu_tile(const BfsParams &p, int d, const NextQueue &nx, const unsigned *cb,
                        unsigned *nb, unsigned word, unsigned nw) {
  const int lane = threadIdx.x & 31;
  const unsigned nwords = ((unsigned)p.n + 31u) >> 5;
  {
    int v[kBuWords], k[kBuWords], ke[kBuWords];
    unsigned search = 0; /* bit j: vertex j unvisited and still searching */
#pragma unroll
    for (int j = 0; j < kBuWords; ++j) {
      v[j] = (int)((word + j) * 32u + (unsigned)lane);
      k[j] = 0;
      ke[j] = 0;
      if ((unsigned)j < nw && v[j] < p.n && p.S[v[j]] == -1) search |= 1u << j;
    }
#pragma unroll
    for (int j = 0; j < kBuWords; ++j)
      if ((search >> j) & 1u) {
        k[j] = __ldg(p.cp + v[j]);
        ke[j] = __ldg(p.cp + v[j] + 1);
      }
    unsigned found = 0;
    while (search) { /* two list entries per searching vertex per step */
      int u0[kBuWords], u1[kBuWords];
#pragma unroll
      for (int j = 0; j < kBuWords; ++j) {
        if (((search >> j) & 1u) && k[j] >= ke[j]) search &= ~(1u << j); /* list exhausted */
        const bool on = (search >> j) & 1u;
        u0[j] = on ? __ldg(p.ic + k[j]) : 0;
        u1[j] = (on && k[j] + 1 < ke[j]) ? __ldg(p.ic + k[j] + 1) : -1;
      }
#pragma unroll
      for (int j = 0; j < kBuWords; ++j) {
        if ((search >> j) & 1u) {
          if (bit_of(cb, u0[j]) || (u1[j] >= 0 && bit_of(cb, u1[j]))) {
            found |= 1u << j;
            search &= ~(1u << j);
          } else {
            k[j] += 2;
          }
        }
      }
    }
    int dg[kBuWords], ad[kBuWords];
#pragma unroll
    for (int j = 0; j < kBuWords; ++j) {
      dg[j] = 0;
      ad[j] = 0;
      if ((found >> j) & 1u) {
        p.S[v[j]] = d + 1;
        ad[j] = __ldg(p.rp + v[j]);
        dg[j] = __ldg(p.rp + v[j] + 1) - ad[j];
      }
    }
#pragma unroll
    for (int j = 0; j < kBuWords; ++j) {
      const unsigned bits = __ballot_sync(FULL, (found >> j) & 1u);
      if (lane == 0 && (unsigned)j < nw && word + j < nwords) nb[word + j] = bits;
    }
    warp_append<kBuWords>(found, v, dg, ad, nx.q, nx.e, nx.a, nx.ctr);
  }
}

/* ---- narrow levels of short-list graphs ----
 * A deep graph has thousands of levels of a few thousand vertices, and such a
 * level costs the chain of its dependent round trips to L2, not its work:
 * counter, queue entries, list entries, claim, reservation in the next queue,
 * barrier.  In a narrow level every CTA keeps the vertices it finds in its own
 * shared memory and expands them itself in the next one.  Nothing of the
 * queue goes through L2 then; the lists of the kept vertices, and where their
 * targets' lists are, are read while the barrier is waited for; and what all
 * CTAs have to know, the size of the level, comes back with the barrier.
 * Left between two barriers: one claim.
 *   A CTA whose vertices have more than its share of the level's edges
 * (keep_limit) sends its finds to the global queue, which the next level
 * shares out evenly, so that a frontier that starts in one CTA spreads.  One
 * that does not grow drifts into few CTAs: the faster one claims first.  So
 * every kShareEvery levels, and when a CTA has found more than kRound, all
 * finds of the next level go to the global queue.  (With only the finds beyond
 * kRound sent there: such a vertex is expanded three round trips after the
 * kept ones and loses its targets to them; who had much got more, and 84 % of
 * a grid's levels used the queue.)
 *   Grid of 2048 x 2048 with path counts, us per level: 6.5 with every level
 * through the global queue, 3.1 so (depths only: 2.5).  What is left is the
 * claim, the fence and the barrier's two trips, ~700 clocks each, and DRAM
 * misses (0.2 us: a grid of 512 x 512, which fits L2, takes 2.9).  With 256
 * threads 4.0; sharing every 12 or 96 levels instead of 32: +2 %, +0 %. */
constexpr unsigned kKeep = 256, kRound = 64;
constexpr int kShareEvery = 32;
/* out-edges of a CTA's kept vertices up to which it keeps what it finds, in a
 * level of qe (Erdos-Renyi, 4096 vertices: one CTA ran 336 vertices, found by
 * eight of its own, in 15 us) */
__device__ __forceinline__ unsigned keep_limit(unsigned qe) { return 64u + 4u * qe / gridDim.x; }
/* mean vertices per CTA up to which a level is narrow, its most out-edges;
 * half of both to start.  Up to there a push of all edges costs less than a
 * bottom-up level's ~6 us, so the direction rule is not asked. */
constexpr unsigned kNarrow = 64, kNarrowEdges = 1u << 16;
/* A barrier's 64-bit sum: arrivals, the level's vertices, their out-edges,
 * CTAs that used the global queue, CTAs that kept more than kRound (modulo 32:
 * missed, it costs time only).  narrow_limit keeps the others apart. */
constexpr int kSumCount = 9, kSumEdges = 27, kSumSpill = 51, kSumCrowd = 59;
constexpr unsigned kSumGrid = 240;
static_assert(kSumGrid < 1u << (kSumCount - 1) && kSumGrid < 1u << (kSumCrowd - kSumSpill), "CTAs");

struct NarrowState {
  int v[2][kKeep], a[2][kKeep], deg[2][kKeep]; /* kept vertices of level d in [d & 1] */
  unsigned found[3], edges[3]; /* by this CTA for level d in [d % 3]; out-edges  */
  unsigned long long last[2];    /* the barrier words after their last use        */
  unsigned long long sum;
  int ok;
};

/* One entry (v; list a, deg entries; deg = 0: none) per 2^sub lanes; su, ad,
 * dg: depth, list start and list length of the lane's first target u.  su may
 * have been read while other CTAs were in level d - 1 or d already: a target
 * with su in [0, d] is no child.  Called by all 32 lanes. */
template <bool SIG>
__device__ __forceinline__ void narrow_expand(const BfsParams &p, NarrowState &ns, int d, int sub,
                                              int v, int a, int deg, int u, int su, int ad, int dg,
                                              bool chk, unsigned cap,
                                              const NextQueue &nx,
                                              const unsigned long long *src,
                                              unsigned long long *dst, bool &ovf) {
  const int lane = threadIdx.x & 31, b = (d + 1) & 1;
  const unsigned lt = (1u << lane) - 1u;
  const unsigned long long x = SIG && deg > 0 ? __ldcg(src + v) : 0ull;
  for (int j = lane & ((1 << sub) - 1);;) {
    int old = -2;
    if (j < deg && (su < 0 || su == d + 1)) old = atomicCAS(p.S + u, -1, d + 1);
    const bool won = old == -1;
    if (SIG && (won || old == d + 1)) {
      if (chk) add_chk(atomicAdd(dst + u, x), x, ovf);
      else atomicAdd(dst + u, x);
    }
    const unsigned m = __ballot_sync(FULL, won);
    if (m) {
      const unsigned es = __reduce_add_sync(FULL, won ? (unsigned)dg : 0u);
      unsigned pos = 0;
      if (lane == 0) {
        pos = atomicAdd(&ns.found[(d + 1) % 3], (unsigned)__popc(m));
        atomicAdd(&ns.edges[(d + 1) % 3], es);
      }
      pos = __shfl_sync(FULL, pos, 0);
      const bool over = pos + (unsigned)__popc(m) > cap;
      pos += (unsigned)__popc(m & lt);
      if (won && pos < cap) {
        ns.v[b][pos] = u;
        ns.a[b][pos] = ad;
        ns.deg[b][pos] = dg;
      }
      if (over) {
        const int vv[1] = {u}, gg[1] = {dg}, aa[1] = {ad};
        warp_append<1>(won && pos >= cap ? 1u : 0u, vv, gg, aa, nx.q, nx.e, nx.a, nx.ctr);
      }
    }
    j += 1 << sub;
    if (!__any_sync(FULL, j < deg)) break;
    if (j < deg) {
      u = __ldg(p.jr + a + j);
      su = -1;
      ad = __ldg(p.rp + u);
      dg = __ldg(p.rp + u + 1) - ad;
    }
  }
}

/* lanes (as a power of two) of an entry, when `n` entries are for `warps` */
__device__ __forceinline__ int narrow_sub(unsigned n, unsigned warps) {
  return n <= warps ? 5 : n <= 2u * warps ? 4 : 3;
}

/* what the rest of the kernel knows of the traversal at level d */
struct LevelState {
  int d, td, sig_bits;
  long long m_u, visited, edges;
};

enum NarrowEnd { NARROW_DONE, NARROW_LEAVE, NARROW_TIMEOUT, NARROW_INJECTED };

/* Runs narrow levels from l.d on, whose qn vertices with qe out-edges are in
 * the global queue.  NARROW_LEAVE: level l.d is in the global queue again,
 * to be run otherwise. */
template <bool SIG>
__device__ __forceinline__ NarrowEnd narrow_levels(const BfsParams &p, NarrowState &ns,
                                                   LevelState &l, unsigned qn, unsigned qe,
                                                   bool &ovf) {
  BfsCtl *ctl = p.ctl;
  const unsigned tid = threadIdx.x, lane = tid & 31u, wid = tid >> 5, nw = blockDim.x >> 5;
  const unsigned gtid = blockIdx.x * blockDim.x + tid, nthreads = gridDim.x * blockDim.x;
  const unsigned gwarp = wid * gridDim.x + blockIdx.x, nwarps = gridDim.x * nw;
  /* the warp that waits for the barrier gets kept vertices last */
  const unsigned kwid = wid == 0u ? nw - 1u : wid - 1u;
  const unsigned nwords = ((unsigned)p.n + 31u) >> 5;
  if (!SIG) { /* depths only: no level in between needs its bitmap */
    for (unsigned i = gtid; i < nwords; i += nthreads)
      p.fb[l.d % 3][i] = p.fb[(l.d + 2) % 3][i] = 0u;
  }
  if (tid < 3) ns.found[tid] = ns.edges[tid] = 0u;
  __syncthreads();
  bool global = true, ovf_seen = false; /* vertices of the level are in the global queue */
  unsigned mine = 0; /* kept by this CTA */
  int kept_levels = 0;
  bool crowded = false;
  int sub = 3, v = 0, a = 0, deg = 0, u = 0, su = -1, ad = 0, dg = 0;
  for (;;) {
    const int d = l.d, b = d & 1, c0 = d % 3, c1 = (d + 1) % 3, c2 = (d + 2) % 3;
    ++l.td;
    l.visited += qn;
    l.edges += qe;
    l.m_u -= qe;
    if (gtid == 0) {
      ctl->qctr[c2] = 0ull;
      ctl->work[(d + 2) & 3] = 0u;
      if (p.trace && d < p.trace_cap - 1) {
        long long *rec = p.trace + 4 * (long long)d;
        rec[0] = (long long)global_ns();
        rec[1] = qn;
        rec[2] = qe;
        rec[3] = DIR_TD;
      }
    }
    if (tid == 0) ns.found[c2] = ns.edges[c2] = 0u;
    const unsigned long long gq = global ? __ldcg(&ctl->qctr[c0]) : 0ull;
    const bool chk = SIG && !ovf_seen && !(p.deg_bits > 0 && l.sig_bits + p.deg_bits <= 63);
    const bool share = crowded || ++kept_levels > kShareEvery;
    const unsigned cap = share || (mine && ns.edges[c0] > keep_limit(qe)) ? 0u : kKeep;
    if (share) kept_levels = 0;
    const NextQueue nx = {p.q[b ^ 1], p.e[b ^ 1], p.a[b ^ 1], &ctl->qctr[c1]};
    const unsigned long long *src = b ? p.sigma_odd : p.sigma;
    unsigned long long *dst = b ? p.sigma : p.sigma_odd;
    /* kept vertices: the first round's loads are done */
    unsigned i = kwid << (5 - sub);
    if (i < mine)
      narrow_expand<SIG>(p, ns, d, sub, v, a, deg, u, su, ad, dg, chk, cap, nx, src, dst, ovf);
    for (i += nw << (5 - sub); i < mine; i += nw << (5 - sub)) {
      const unsigned k = i + (lane >> sub);
      const int j = (int)(lane & ((1u << sub) - 1u));
      deg = k < mine ? ns.deg[b][k] : 0;
      v = a = u = ad = dg = 0;
      if (deg) v = ns.v[b][k], a = ns.a[b][k];
      if (j < deg) {
        u = __ldg(p.jr + a + j);
        ad = __ldg(p.rp + u);
        dg = __ldg(p.rp + u + 1) - ad;
      }
      narrow_expand<SIG>(p, ns, d, sub, v, a, deg, u, -1, ad, dg, chk, cap, nx, src, dst, ovf);
    }
    /* a share of the global queue */
    const unsigned gn = (unsigned)(gq >> 32);
    const int gsub = narrow_sub(gn, nwarps);
    for (i = gwarp << (5 - gsub); i < gn; i += nwarps << (5 - gsub)) {
      const unsigned k = i + (lane >> gsub);
      const int j = (int)(lane & ((1u << gsub) - 1u));
      v = a = deg = u = ad = dg = 0;
      if (k < gn) {
        v = __ldcg(p.q[b] + k);
        a = __ldcg(p.a[b] + k);
        deg = (int)((k + 1u < gn ? (unsigned)__ldcg(p.e[b] + k + 1u) : (unsigned)gq) -
                    (unsigned)__ldcg(p.e[b] + k));
      }
      if (j < deg) {
        u = __ldg(p.jr + a + j);
        ad = __ldg(p.rp + u);
        dg = __ldg(p.rp + u + 1) - ad;
      }
      narrow_expand<SIG>(p, ns, d, gsub, v, a, deg, u, -1, ad, dg, chk, cap, nx, src, dst, ovf);
    }
    if (p.inject_barrier_skip > 0 && blockIdx.x == 0 && d == p.inject_barrier_skip - 1)
      return NARROW_INJECTED;
    if (SIG && __any_sync(FULL, ovf) && lane == 0) atomicOr(&ctl->sigma_overflow, 1);

    /* Barrier with a sum, as grid_barrier otherwise: a level's arrivals add
     * 2^(kSumCount - 1), whose bit changes with the last one, and each adds
     * its CTA's figures above.  The sum is the difference to the word after
     * its last use; two words are used in turn, so that a CTA already at the
     * next barrier does not change what a slower one is still to read. */
    __syncthreads();
    constexpr unsigned kFlip = 1u << (kSumCount - 1);
    const unsigned found = ns.found[c1];
    mine = found < cap ? found : cap;
    if (tid == 0) {
      const unsigned long long add =
          (blockIdx.x == 0 ? kFlip - (gridDim.x - 1u) : 1u) +
          ((unsigned long long)found << kSumCount) +
          ((unsigned long long)ns.edges[c1] << kSumEdges) +
          (found > cap ? 1ull << kSumSpill : 0ull) +
          (cap && found > kRound ? 1ull << kSumCrowd : 0ull);
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&ctl->sum[b].word), "l"(add)
                   : "memory");
    }
    /* meanwhile: the lists of the kept vertices, and the depths of their
     * targets, some of which may be level d + 2's already */
    sub = narrow_sub(mine, nw - 1u);
    {
      const unsigned k = (kwid << (5 - sub)) + (lane >> sub);
      const int j = (int)(lane & ((1u << sub) - 1u));
      deg = k < mine ? ns.deg[b ^ 1][k] : 0;
      v = a = u = ad = dg = 0;
      su = -1;
      if (deg) v = ns.v[b ^ 1][k], a = ns.a[b ^ 1][k];
      if (j < deg) {
        u = __ldg(p.jr + a + j);
        su = __ldcg(p.S + u);
        if (SIG) /* its count, to be added to: 3.46 -> 3.25 us per level */
          asm volatile("prefetch.global.L2 [%0];" ::"l"(src + u));
        ad = __ldg(p.rp + u);
        dg = __ldg(p.rp + u + 1) - ad;
      }
      if (SIG && !ovf_seen) ovf_seen = __ldcg(&ctl->sigma_overflow) != 0;
    }
    if (tid == 0) {
      const unsigned long long last = ns.last[b];
      const unsigned long long t0 = global_ns();
      unsigned long long w;
      unsigned spins = 0;
      int ok = 1;
      for (;;) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];"
                     : "=l"(w)
                     : "l"(&ctl->sum[b].word)
                     : "memory");
        if (((w ^ last) & kFlip) != 0ull) break;
        if ((++spins & 31u) == 0) {
          if (dev::ld_volatile(&ctl->status) != 0) {
            ok = 0;
            break;
          }
          if ((long long)(global_ns() - t0) > p.timeout_ns) {
            atomicCAS(&ctl->status, 0, (int)TBFS_ERR_TIMEOUT);
            atomicCAS(&ctl->timeout_level, 0, d + 2);
            ok = 0;
            break;
          }
        }
      }
      ns.ok = ok;
      ns.sum = w - last;
      ns.last[b] = w;
    }
    __syncthreads();
    if (!ns.ok) return NARROW_TIMEOUT;
    const unsigned long long sum = ns.sum;
    qn = (unsigned)(sum >> kSumCount) & ((1u << (kSumEdges - kSumCount)) - 1u);
    qe = (unsigned)(sum >> kSumEdges) & ((1u << (kSumSpill - kSumEdges)) - 1u);
    global = ((sum >> kSumSpill) & ((1u << (kSumCrowd - kSumSpill)) - 1u)) != 0ull;
    crowded = (sum >> kSumCrowd) != 0ull;
    l.sig_bits = l.sig_bits + p.deg_bits < 64 ? l.sig_bits + p.deg_bits : 64;
    ++l.d;
    if (qn == 0u) return NARROW_DONE;
    if (qn > p.narrow || qe > kNarrowEdges) {
      if (wid < (mine + 31u) / 32u) { /* level d + 1 to the global queue */
        const unsigned k = tid;
        const int vv[1] = {k < mine ? ns.v[b ^ 1][k] : 0};
        const int gg[1] = {k < mine ? ns.deg[b ^ 1][k] : 0};
        const int aa[1] = {k < mine ? ns.a[b ^ 1][k] : 0};
        warp_append<1>(k < mine ? 1u : 0u, vv, gg, aa, nx.q, nx.e, nx.a, nx.ctr);
      }
      if (!grid_barrier(ctl, p.timeout_ns, d)) return NARROW_TIMEOUT;
      if (!SIG) { /* and its bitmap */
        for (unsigned k = gtid; k < qn; k += nthreads) {
          const unsigned t = (unsigned)__ldcg(nx.q + k);
          atomicOr(p.fb[c1] + (t >> 5), 1u << (t & 31u));
        }
        if (!grid_barrier(ctl, p.timeout_ns, d)) return NARROW_TIMEOUT;
      }
      return NARROW_LEAVE;
    }
  }
}

template <bool SHORT, bool SIG>
__global__ void __launch_bounds__(SHORT ? kShortBlock : kBlock, 1)
    bfs_persistent_kernel(const BfsParams p) {
  /* a window per warp, then the frontier filter (instance <false, true>) */
  extern __shared__ __align__(16) unsigned char s_dyn[];
  ExpandWin *s_win = reinterpret_cast<ExpandWin *>(s_dyn);
  ExpandWin &win = s_win[threadIdx.x >> 5];
  unsigned *s_filter =
      !SHORT && p.filter ? reinterpret_cast<unsigned *>(s_win + (blockDim.x >> 5)) : nullptr;
  const unsigned gtid = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned nthreads = gridDim.x * blockDim.x;
  const unsigned nwarps = nthreads >> 5;
  BfsCtl *ctl = p.ctl;
  constexpr bool want_sigma = SIG;
  NarrowState *narrow = nullptr;
  if constexpr (SHORT) {
    __shared__ NarrowState s_narrow;
    narrow = &s_narrow;
    if (threadIdx.x == 0) narrow->last[0] = narrow->last[1] = 0ull;
  }
  const int root = p.inv ? __ldg(p.inv + p.root) : p.root; /* internal numbering */

  /* init: S = -1, counts 0, root at depth 0 with one path; depths only:
   * F_0 = {root} in bitmap 0, the other bitmaps empty.  With path counts (a
   * pass over the results ends the traversal) a vertex without in-list is
   * kNoList until then, so that bottom-up levels need not look at it again:
   * 43 % of RMAT-22's vertices. */
  constexpr int kNoList = -2;
  if (want_sigma) {
    for (unsigned i0 = gtid; i0 < (unsigned)p.n; i0 += 4u * nthreads) {
      int len[4];
#pragma unroll
      for (unsigned j = 0; j < 4u; ++j) {
        const unsigned i = i0 + j * nthreads;
        len[j] = i < (unsigned)p.n ? __ldg(p.cp + i + 1) - __ldg(p.cp + i) : 0;
      }
#pragma unroll
      for (unsigned j = 0; j < 4u; ++j) {
        const unsigned i = i0 + j * nthreads;
        if (i < (unsigned)p.n) {
          p.S[i] = (int)i == root ? 0 : len[j] ? -1 : kNoList;
          p.sigma_odd[i] = 0ull; /* may be the same array (bfs_launch) */
          p.sigma[i] = (int)i == root ? 1ull : 0ull;
        }
      }
    }
  } else {
    for (unsigned i = gtid; i < (unsigned)p.n; i += nthreads) p.S[i] = (int)i == root ? 0 : -1;
  }
  const unsigned nwords = ((unsigned)p.n + 31u) >> 5;
  if (!want_sigma) {
    for (unsigned i = gtid; i < nwords; i += nthreads) {
      p.fb[0][i] = i == ((unsigned)root >> 5) ? 1u << ((unsigned)root & 31u) : 0u;
      p.fb[1][i] = 0u;
      p.fb[2][i] = 0u;
    }
  }
  const unsigned n_hub = want_sigma && p.hub_count ? (unsigned)__ldg(p.hub_count) : 0u;
  if (gtid == 0) {
    const int a = __ldg(p.rp + root);
    p.q[0][0] = root;
    p.e[0][0] = 0;
    p.a[0][0] = a;
    const unsigned deg = (unsigned)(__ldg(p.rp + root + 1) - a);
    ctl->qctr[0] = (1ull << 32) | deg;
  }
  const bool started = grid_barrier(ctl, p.timeout_ns, -1);

  int d = 0, dir = DIR_TD, td = 0, bu = 0;
  long long m_u = p.out_edges_total, visited = 0, edges = 0;
  const float alpha = want_sigma ? p.alpha * kSigmaAlpha : p.alpha;
  const bool own = p.deg_bits > 0 && p.deg_bits < 4; /* in-lists of at most kOwn entries */
  bool ovf = false, done = false;
  /* Bound on the bits of the path counts of F_d: sigma(F_0) = 1, and a count
   * of F_{d+1} sums at most max-in-degree counts of F_d, so it has at most
   * deg_bits more bits.  Pushes into a level whose bound is at most 63 bits
   * cannot overflow and add without the check (a reduction whose result
   * is not waited for); so do pushes once an overflow has been recorded,
   * since the flag is per traversal. */
  int sig_bits = 1;
  float excess = 0.0f; /* of bottom-up levels over top-down ones, in list entries */
  while (started) {
    const unsigned long long cur = __ldcg(&ctl->qctr[d % 3]);
    /* read with the counter, so that both loads are in flight together */
    const bool ovf_seen = want_sigma && __ldcg(&ctl->sigma_overflow) != 0;
    const unsigned qn = (unsigned)(cur >> 32);
    const unsigned qe = (unsigned)cur;
    if (qn == 0) {
      done = true;
      break;
    }
    if constexpr (SHORT) {
      if (dir == DIR_TD && p.mode != TBFS_MODE_BOTTOM_UP && qn <= p.narrow / 2u &&
          qe <= kNarrowEdges / 2u) {
        LevelState l = {d, td, sig_bits, m_u, visited, edges};
        const NarrowEnd end = narrow_levels<SIG>(p, *narrow, l, qn, qe, ovf);
        d = l.d;
        td = l.td;
        sig_bits = l.sig_bits;
        m_u = l.m_u;
        visited = l.visited;
        edges = l.edges;
        if (end == NARROW_LEAVE) continue;
        done = end == NARROW_DONE;
        break;
      }
    }
    visited += qn;
    edges += qe;
    /* slot (d+2)%3 held F_{d-1}, read by every CTA before the last barrier;
     * clear it for F_{d+2}, which phase d+1 fills */
    if (gtid == 0) ctl->qctr[(d + 2) % 3] = 0ull;

    m_u -= qe; /* out-edges of the vertices not reached yet */
    const bool no_queue = want_sigma && dir == DIR_BU; /* F_d has no queue yet */
    if (p.mode == TBFS_MODE_TOP_DOWN) {
      dir = DIR_TD;
    } else if (p.mode == TBFS_MODE_BOTTOM_UP) {
      dir = DIR_BU;
    } else if ((float)qe * alpha > (float)m_u + kBuWordCost * (float)nwords) {
      /* a bottom-up level also visits every vertex's word: without that
       * term, the tail of a deep graph (few unexplored edges left) switched
       * to bottom-up levels three times as costly as top-down ones */
      dir = DIR_BU;
    } else if (dir == DIR_BU) {
      /* leave unless the frontier is large; with path counts when the bottom-up
       * levels cost more, summed up, than top-down ones and the pass that
       * collects the queue */
      if ((float)qn * p.beta <= (float)p.n) {
        if (want_sigma) {
          const float scan = kScanVertex * (float)p.n;
          const float fixed = SHORT && p.narrow ? kNarrowGain : -kQueueCost;
          excess = fmaxf(0.0f, excess + (float)m_u + scan + fixed - (float)qe * alpha);
          if (excess > kLeaveCost + kQueueCost + fixed + scan) dir = DIR_TD;
        } else {
          dir = DIR_TD;
        }
      }
    }
    if (dir == DIR_TD) excess = 0.0f;
    if (gtid == 0 && p.trace && d < p.trace_cap - 1) {
      long long *rec = p.trace + 4 * (long long)d;
      rec[0] = (long long)global_ns();
      rec[1] = qn;
      rec[2] = qe;
      rec[3] = dir;
    }

    const int bc = d & 1, bn = bc ^ 1, b3 = (d + 1) % 3;
    const NextQueue nx = {p.q[bn], p.e[bn], p.a[bn], &ctl->qctr[b3]};
    /* depths only -- bitmaps: F_d read; F_{d+1} written; F_{d+2}'s cleared
     * (its previous contents, F_{d-1}, were last read in phase d-1) */
    const unsigned *bm_cur = p.fb[d % 3];
    unsigned *bm_next = p.fb[b3];
    if (!want_sigma) {
      unsigned *bm_clear = p.fb[(d + 2) % 3];
      for (unsigned i = gtid; i < nwords; i += nthreads) bm_clear[i] = 0u;
    }
    /* counts of level d and of level d+1 */
    const unsigned long long *src = bc ? p.sigma_odd : p.sigma;
    unsigned long long *dst = bc ? p.sigma : p.sigma_odd;
    /* work counter of phase d+2 (last used in phase d-2) */
    if (gtid == 0) ctl->work[(d + 2) & 3] = 0u;

    /* this phase's work: an expansion, or hub segments and word tiles */
    ExpandTask A = {{p.q[bc], p.e[bc], p.a[bc], qn, qe}, {1, 1, 0}, src, dst, false};
    const unsigned max_ept =
        p.max_ept > 0 && p.max_ept < kEPT ? (unsigned)p.max_ept : (unsigned)kEPT;
    unsigned n_seg = 0, n_all = 0, n_static = nwarps, tiles = 0, per_item = 1;
    const unsigned *filter = nullptr;
    bool short_level = false, heavy = false;
    Found fd = {0u, 0u};
    if (dir == DIR_TD) {
      ++td;
      if (no_queue) {
        collect_queue(p, d, p.q[bc], p.e[bc], p.a[bc],
                      (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps);
        if (!grid_barrier(ctl, p.timeout_ns, d)) break;
      }
      A.chk = want_sigma && !ovf_seen && !(p.deg_bits > 0 && sig_bits + p.deg_bits <= 63);
      /* a small top-down level of a graph with short lists: items of
       * kShortEntries queue entries each, no owner search (expand_chunk) and
       * no edge-chunk plan */
      short_level = SHORT && qn <= kShortEntries * nwarps;
      if (!short_level) {
        A.pl = plan_expand(qe, nwarps, max_ept);
        n_all = A.pl.nch;
      }
    } else {
      ++bu;
      if (gtid == 0) ctl->collect = 0ull;
      n_seg = (n_hub + 31u) / 32u; /* 32 segments looked at per item */
      /* lists of about one length need no items of equal cost (grid of 1100 x
       * 1100, all bottom-up: 19.5 us per level with them, 12.8 without) */
      heavy = want_sigma && p.tile && !own && (float)m_u > kHeavyEntries &&
              (float)m_u > kHeavyShare * (float)p.nnz;
      if (heavy && s_filter && !no_queue && qn <= kFilterBits / 4u &&
          (float)m_u > kFilterGain * (float)qn) {
        filter = s_filter;
        for (unsigned i = threadIdx.x; i < kFilterBits / 32u; i += blockDim.x) s_filter[i] = 0u;
        __syncthreads();
        for (unsigned i = threadIdx.x; i < qn; i += 8u * blockDim.x) {
          int u[8]; /* eight in flight: every CTA reads the whole queue */
#pragma unroll
          for (unsigned j = 0; j < 8u; ++j)
            u[j] = i + j * blockDim.x < qn ? __ldcg(p.q[bc] + i + j * blockDim.x) : -1;
#pragma unroll
          for (unsigned j = 0; j < 8u; ++j)
            if (u[j] >= 0)
              atomicOr(s_filter + (((unsigned)u[j] >> 5) & (kFilterBits / 32u - 1u)),
                       1u << ((unsigned)u[j] & 31u));
        }
        __syncthreads();
      }
      if (heavy) { /* items of equal cost */
        tiles = (unsigned)(((long long)p.nnz + (long long)kTileVertex * p.n) / kTileCost) + 1u;
        per_item = tiles / (4u * nwarps);
        per_item = per_item < 1u ? 1u : (per_item > 8u ? 8u : per_item);
      } else { /* words, at least one for every warp of a small graph */
        tiles = nwords;
        per_item = (nwords + nwarps - 1u) / nwarps;
        const unsigned most = want_sigma ? (unsigned)kWords : (unsigned)kBuWords;
        per_item = per_item > most ? most : per_item;
      }
      n_all = n_seg + (tiles + per_item - 1u) / per_item;
      /* even work needs no counter */
      if (want_sigma && !heavy) n_static = (n_all / nwarps + 1u) * nwarps;
    }
    const Counts C = {src, filter, ovf_seen, d, p.S, own};
    unsigned *wctr = &ctl->work[d & 3];
    const int lane = threadIdx.x & 31;
    /* work items: the first n_static statically (one per warp, or several),
     * the rest from the level's counter past the static range, so that a
     * small level costs no same-address atomics.  Static items go round-robin
     * over the CTAs (item i to CTA i % grid), so that a small level's work
     * spreads over as many SMs as it has items instead of filling the first
     * CTAs' warps */
    unsigned item = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (short_level) {
      const unsigned first = item * kShortEntries;
      if (first < qn) run_short_item<SIG>(p, d, A, first, max_ept, nx, bm_next, win, ovf);
    }
    while (item < n_all) {
      if (dir == DIR_TD) {
        run_expand_item<SIG>(p, d, A, item, nx, bm_next, win, ovf);
      } else if (item < n_seg) {
        pull_segments(p, fd, C, dst, item, n_seg, n_hub, ovf);
      } else {
        const unsigned t = (item - n_seg) * per_item;
        if constexpr (!SIG) {
          bu_tile(p, d, nx, bm_cur, bm_next, t, per_item);
        } else if (heavy) {
          const int ve = __ldg(p.tile + (t + per_item < tiles ? t + per_item : tiles));
          if (filter) pull_range<true>(p, fd, C, dst, __ldg(p.tile + t), ve, win, ovf);
          else pull_range<false>(p, fd, C, dst, __ldg(p.tile + t), ve, win, ovf);
        } else {
          const int v = (int)(t * 32u), e = v + 32 * (int)per_item;
          pull_range<false>(p, fd, C, dst, v, e < p.n ? e : p.n, win, ovf);
        }
      }
      /* The next item: static, or claimed once this one is done.  Claimed beside
       * it, the counter's round trip is hidden, but a warp that is slow with its
       * item keeps the next one from the others, and a level has one to four items
       * per warp (us, claimed beside / after: depths bottom-up on Erdos-Renyi of
       * 2 M of 6 689 / 573, RMAT-22 423 / 417, top-down 1616 / 1547). */
      item += nwarps;
      if (item >= n_static) {
        if (n_all <= n_static) break;
        if (lane == 0) item = n_static + atomicAdd(wctr, 1u);
        item = __shfl_sync(FULL, item, 0);
      }
    }
    if (dir == DIR_BU) {
      const unsigned fn = __reduce_add_sync(FULL, fd.n), fe = __reduce_add_sync(FULL, fd.e);
      if (lane == 0 && fn) atomicAdd(nx.ctr, ((unsigned long long)fn << 32) | fe);
    }
    /* test hook: CTA 0 leaves without arriving; the others' waits expire */
    if (p.inject_barrier_skip > 0 && blockIdx.x == 0 && d == p.inject_barrier_skip - 1) break;
    if (want_sigma) { /* overflow recorded now: seen by every CTA after the barrier */
      const bool any_ovf = __any_sync(FULL, ovf);
      if (any_ovf && (threadIdx.x & 31) == 0) atomicOr(&ctl->sigma_overflow, 1);
    }
    if (!grid_barrier(ctl, p.timeout_ns, d)) break;
    sig_bits = sig_bits + p.deg_bits < 64 ? sig_bits + p.deg_bits : 64;
    ++d;
  }
  if (__any_sync(FULL, ovf) && (threadIdx.x & 31) == 0) atomicOr(&ctl->sigma_overflow, 1);
  /* results are final after the last barrier.  Renumbered graphs: gathered
   * into the caller's numbering, kOut vertices per thread and round so that
   * their dependent loads (id, depth, count of the depth's parity) overlap;
   * coalesced stores.  Otherwise: counts of odd depths join the others, and
   * kNoList becomes -1, also when the traversal was given up and the arrays are
   * the caller's (a CTA still in the last level sees an unvisited vertex with an
   * empty list). */
  constexpr int kOut = 4;
  if (done && p.perm) {
    for (unsigned i0 = gtid; i0 < (unsigned)p.n; i0 += kOut * nthreads) {
      int o[kOut], sv[kOut];
      unsigned long long x[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        const unsigned i = i0 + j * nthreads;
        o[j] = i < (unsigned)p.n ? __ldg(p.inv + i) : -1;
      }
#pragma unroll
      for (int j = 0; j < kOut; ++j) sv[j] = o[j] >= 0 ? p.S[o[j]] : -1;
      if (want_sigma) {
#pragma unroll
        for (int j = 0; j < kOut; ++j)
          x[j] = sv[j] < 0 ? 0ull : (sv[j] & 1) ? p.sigma_odd[o[j]] : p.sigma[o[j]];
      }
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        const unsigned i = i0 + j * nthreads;
        if (i < (unsigned)p.n) {
          p.S_out[i] = sv[j] < 0 ? -1 : sv[j];
          if (want_sigma) p.sigma_out[i] = x[j];
        }
      }
    }
  } else if (!p.perm && want_sigma) {
    for (unsigned i0 = gtid; i0 < (unsigned)p.n; i0 += kOut * nthreads) {
      bool odd[kOut];
      unsigned long long x[kOut];
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        const unsigned i = i0 + j * nthreads;
        odd[j] = false;
        if (i < (unsigned)p.n) {
          const int sv = p.S[i];
          odd[j] = sv > 0 && (sv & 1);
          if (sv == kNoList) p.S[i] = -1;
        }
      }
#pragma unroll
      for (int j = 0; j < kOut; ++j) x[j] = odd[j] ? p.sigma_odd[i0 + j * nthreads] : 0ull;
#pragma unroll
      for (int j = 0; j < kOut; ++j)
        if (odd[j]) p.sigma[i0 + j * nthreads] = x[j];
    }
  }
  if (gtid == 0) {
    ctl->levels = d;
    ctl->td_levels = td;
    ctl->bu_levels = bu;
    ctl->visited = visited;
    ctl->edges = edges;
    if (p.trace) {
      const int slot = d < p.trace_cap - 1 ? d : p.trace_cap - 1;
      long long *rec = p.trace + 4 * (long long)slot;
      rec[0] = (long long)global_ns();
      rec[1] = 0;
      rec[2] = 0;
      rec[3] = -1;
    }
  }
}

}  // namespace

/* shared memory of a CTA of `block` threads */
static size_t bfs_smem(int block, bool filter) {
  return (size_t)(block / 32) * sizeof(ExpandWin) + (filter ? kFilterBits / 8 : 0);
}

/* the instance for graphs with (or without) short out-lists, with (or
 * without) path counts */
static const void *bfs_kernel(bool short_lists, bool sigma) {
  if (sigma)
    return short_lists ? reinterpret_cast<const void *>(bfs_persistent_kernel<true, true>)
                       : reinterpret_cast<const void *>(bfs_persistent_kernel<false, true>);
  return short_lists ? reinterpret_cast<const void *>(bfs_persistent_kernel<true, false>)
                     : reinterpret_cast<const void *>(bfs_persistent_kernel<false, false>);
}

cudaError_t bfs_geometry(int device, LaunchGeom *out) {
  int sms = 0, coop = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  if (e != cudaSuccess) return e;
  if (!coop) return cudaErrorNotSupported;
  int smem_sm = 0;
  e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
  if (e != cudaSuccess) return e;
  for (int k = 0; k < 4; ++k) { /* carve out what a CTA needs, the rest is L1 */
    const void *fn = bfs_kernel((k & 1) != 0, (k & 2) != 0);
    const int most = (k & 1) ? kShortBlock : kBlock;
    const size_t need = bfs_smem(most, k == 2);
    /* without the filter: a launch with one takes its part of L1 */
    const size_t held = bfs_smem(most, false) + sizeof(NarrowState) + 1024;
    const int carve = (int)((100 * held + (size_t)smem_sm - 1) / (size_t)smem_sm);
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                               carve < 100 ? carve : 100);
    int fit = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, fn, most, need);
    if (e != cudaSuccess) return e;
    if (fit < 1) return cudaErrorInvalidConfiguration;
  }
  out->block = kBlock;
  out->grid = sms;
  out->sms = sms;
  out->per_sm = kBlock / kBlockStep;
  return cudaSuccess;
}

/* Most vertices of a narrow level, 0: none.  Of lists of at most m entries, so
 * many vertices find less than 2^18, with less than 2^24 out-edges, and the
 * fields of a barrier's sum stay apart (also if all vertices are found). */
static unsigned narrow_limit(const BfsParams &p, int grid) {
  const long long m = p.max_list;
  if (m <= 0 || m > kNarrowList || grid > (int)kSumGrid) return 0;
  const long long found = (1 << (kSumEdges - kSumCount)) - 1, edges = (1 << (kSumSpill - kSumEdges)) - 1;
  long long most = (long long)kNarrow * grid;
  if (p.n > found || p.n * m > edges) most = std::min({most, found / m, edges / (m * m)});
  return (unsigned)most;
}

cudaError_t bfs_launch(const BfsParams &p0, const LaunchGeom &g, cudaStream_t s) {
  /* One CTA per SM, of 256 threads per unit of ctas_per_sm.  By default (and at
   * most) 2 on short-list graphs, whose levels are many and small; 4 for depths
   * only and bottom-up levels, if only possible ones from kLargeVertices, which
   * want every warp; else 3, which leaves more L1 and costs less at every barrier (us
   * per BFS with path counts at 3 / 4: RMAT 2^17 of 16 57 / 61, 2^18 of 16 67 /
   * 71, of 32 106 / 110, 2^19 of 8 98 / 93, of 24 98 / 88, 2^20 of 16 137 / 129,
   * 2^21 of 16 191 / 184, 2^22 of 32 468 / 417; Erdos-Renyi of 300 K of 30 81 / 85,
   * of 2 M of 20 257 / 255; bottom-up only, directed, 1 M of 8 538 / 487). */
  BfsParams p = p0;
  /* bottom-up levels alone, large ones, want threads, not the short-list
   * instance's registers (grid of 2048 x 2048: 32 / 28 us per level, depths) */
  const bool pulls = p.mode == TBFS_MODE_BOTTOM_UP && p.n > 1 << 20;
  const bool short_lists = p.short_lists != 0 && !pulls;
  const bool sigma = p.sigma != nullptr;
  const bool full = !sigma || p.mode == TBFS_MODE_BOTTOM_UP ||
                    (p.mode == TBFS_MODE_AUTO && p.n > kLargeVertices);
  const int want = p.ctas_per_sm > 0 ? p.ctas_per_sm : short_lists ? 2 : full ? 4 : 3;
  int block = want < g.per_sm ? kBlockStep * want : g.block;
  if (short_lists && block > kShortBlock) block = kShortBlock;
  p.narrow = short_lists ? narrow_limit(p, g.grid) : 0u;
  /* top-down levels alone do not need even and odd depths apart: half the memory
   * to add to (ms per BFS apart / together: RMAT-22 1.59 / 1.49, Erdos-Renyi of
   * 8 M of 8 2.22 / 2.14) */
  if (p.mode == TBFS_MODE_TOP_DOWN) p.sigma_odd = p.sigma;
  /* The frontier filter pays where the gathers it saves miss L1 even so: its 32
   * KB come off that.  (us per BFS with / without: RMAT 2^18 of 24 87 / 82, 2^19
   * of 8 97 / 92, 2^20 of 16 137 / 134, 2^21 of 16 191 / 189, of 32 218 / 224.) */
  p.filter = !short_lists && sigma && p.tile && p.nnz > kLargeEntries;
  void *args[] = {&p};
  return cudaLaunchCooperativeKernel(bfs_kernel(short_lists, sigma), dim3(g.grid), dim3(block), args,
                                     bfs_smem(block, p.filter), s);
}

}  // namespace tbfs
