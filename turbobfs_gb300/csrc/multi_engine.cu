/*
 * multi_engine.cu -- many independent traversals, each (graph, root) its own
 * instance, advancing together in one persistent cooperative launch: one
 * grid barrier per level for all of them.  Instances may live on different
 * graphs (a packed arena of many small graphs, or separately resident
 * graphs of a server) and start at different times: every instance keeps its
 * own level counter, queues and statistics in its descriptor, so a launch can
 * stop after a number of levels and a later launch can carry on with new
 * instances admitted beside the unfinished ones (continuous batching).
 *
 * Per level and instance the step is the reference's top-down semiring
 * iteration (TurboBFS_CSC_TD/bfsgputdcsc_sc.cu:159-208: f_t = A^T f over the
 * frontier, sigma += f, S = d), done as a push over the out-edges of the
 * instance's frontier queue:
 *   - an edge u -> v with S[v] == -1 claims v with atomicCAS(S[v], -1, d+1)
 *     and appends it to the next queue;
 *   - every edge that lands on a vertex at depth d+1 (claimed now, by this
 *     edge or another) adds sigma[u] to sigma[v] with a 64-bit atomicAdd;
 *     sigma[u] is final because u was claimed a level earlier.
 * Work is edge-balanced across all instances: each CTA computes the same
 * prefix of per-instance work items (rounds of 128 consecutive frontier
 * out-edges, 4 per lane, with fewer rounds per item on small levels) in
 * shared memory; a warp takes its first item by its global index and later
 * ones from a counter, locates the instance by binary search in the prefix,
 * and the owner of each edge by a 32-ary search over the instance's
 * out-degree prefix (first round) followed by a shuffle search in a window
 * of 64 queue entries.
 *
 * Small levels stay out of that: an instance whose frontier fits one CTA is
 * run by that CTA alone, level after level, with its queue in shared memory
 * and no grid barrier (local_run), while the other CTAs advance the wide
 * instances.  A phase is then one level of every wide instance and as many
 * of the others as fit in its time.  Launches with a large instance run a kernel
 * without that (multi_local).
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "device_common.cuh"
#include "tbfs_internal.h"

namespace tbfs {
namespace {

using dev::FULL;
using dev::grid_barrier;

/* Two instances of the kernel.  With one large CTA per SM a CTA can run an
 * instance alone (below); with three of 256 threads, and an L1 not given away to
 * the tables for that, the levels that all CTAs share are faster.  multi_local
 * has the rule. */
constexpr int kLocalBlock = 768, kSharedBlock = 256, kSharedPerSm = 3;
constexpr int kEPT = 4;                   /* consecutive edges per lane per round */
constexpr unsigned kRoundEdges = 32 * kEPT;
constexpr int kMaxRounds = 8;             /* rounds per item, fewer on small levels */

constexpr int kInitBlock = 256;

/* ---- instances run by one CTA ----
 * A level that all CTAs share costs ~11 us, however small: plan, work prefix,
 * queue entries, owners, lists, claims, reservation and barrier are dependent
 * round trips to L2 or follow one.  One CTA with the queue in shared memory
 * has two or three (list entry, depth, where the found one's list is) and two
 * __syncthreads.  What bounds a larger level is the SM's path to L2, one
 * scattered access per 1-3 clocks (and an atomic in ~4), so as little as
 * possible goes there: lists are read by consecutive lanes, the queue and its
 * counts stay in shared memory, and since nobody else touches the instance
 * meanwhile, the vertices found by a level are the keys of a hash table whose
 * slots add up the counts, stored once; a vertex whose kProbe slots are taken
 * by others is claimed and counted in L2.  (A claim and an add in L2 per edge,
 * both ends of every target's list and the source's count from L2: 9 us for
 * a level of 2300 edges.)
 *   A level of up to kLocalEnter edges costs no more so than shared, twice as many
 * beside more than kFew other instances, since a shared level is longer then; an
 * instance is given back when it has outgrown half as many again, or the queue.
 * (192 graphs of 2^10 to 2^18 vertices: 12.5 -> 5.2 ms, of which 3.3 ms were two
 * memsets and two copies per graph on the host; 28 queries to a server of 14 such
 * graphs: 8.3 -> 5.2 ms.  Us per level of a grid of 2^14 vertices 10.2 -> 3.3.
 * Limits of 4096 alone / of 8192 alone / halved beside shared instances, ms: a
 * 1024 x 1024 grid 9.4 / 10.2 / 9.7, six of 700 x 700 9.6 / 5.9 / 8.5, 192 other
 * graphs of up to 2^18 vertices 5.3 / 5.3 / 11.0, 64 of up to 2^20 13.6 / 11.6 /
 * 16.2, 512 of them 37.6 / 26.4 / 36.1.) */
constexpr unsigned kLocalQueue = 2048;
constexpr unsigned kSlotBits = 12, kSlots = 1u << kSlotBits, kProbe = 24;
constexpr unsigned kNoKey = 0xffffffffu, kNoSlot = 0xffffu;
constexpr unsigned kLocalEnter = 4096, kFew = 4;
/* A CTA gives its instance back for the next phase after this long: alone, so
 * that no CTA waits long at the barrier; beside shared instances, about the
 * time of a shared level (of kLocalEdges edges per clock), since a large deep
 * instance waits for it at every one of its levels.  (In clocks of ~0.5 ns: the
 * ns timer is slow to read.) */
constexpr long long kLocalAlone = 500000, kLocalBeside = 20000, kLocalEdges = 8;
constexpr int kLocalMine = 16;            /* instances of one CTA in a phase */
constexpr unsigned kLocalGrid = kMultiMaxSlots / kLocalMine + 1; /* CTAs for that */
constexpr unsigned kIsLocal = 0x80000000u;
/* Vertices of a launch's largest unfinished instance up to which the kernel with
 * one-CTA instances runs it (multi_local).  The levels of larger ones are mostly
 * shared, and the small ones beside them wait for those; a server whose large
 * queries take 10 % longer is that much nearer to saturation.  Us per shared
 * level of one grid, kernel without / with: 512 x 512 9.3 / 5.2, 1024 x 1024 8.8 /
 * 8.1, 1448 x 1448 9.0 / 8.9, 2048 x 2048 10.0 / 10.4, 4096 x 4096 10.3 / 11.5;
 * 64 graphs of up to 4096 x 4096 served at 400 queries/s, p50 / p99 14 / 100 ms
 * without and, all in the kernel with, 15-25 / 137-632. */
constexpr int kLocalVertices = 1 << 20;

struct LocalShared {
  int v[2][kLocalQueue], a[2][kLocalQueue]; /* level d in [d & 1]: vertex, list start */
  unsigned e[2][kLocalQueue];               /* exclusive prefix of out-degrees        */
  unsigned long long cnt[2][kLocalQueue];   /* path counts                            */
  unsigned key[kSlots], lo[kSlots], hi[kSlots]; /* vertices of the next level, counts */
  unsigned long long ctr[3];                /* level d: (count << 32) | out-edges     */
  int leave[2];
  unsigned short slot[kLocalQueue];         /* of the next level's entries            */
};

/* u's slot in the table, entered if it is not there (*is_new); kNoSlot if all its
 * slots are others'.  Entries only come during a level, so every thread that
 * looks for u finds the same answer. */
__device__ __forceinline__ unsigned find_slot(LocalShared &L, unsigned u, bool *is_new) {
  unsigned s = (u * 0x9e3779b1u) >> (32 - kSlotBits);
  for (unsigned p = 0; p < kProbe; ++p, s = (s + 1u) & (kSlots - 1u)) {
    const unsigned k = atomicCAS(&L.key[s], kNoKey, u);
    if (k == kNoKey || k == u) {
      *is_new = k != u;
      return s;
    }
  }
  return kNoSlot;
}

/* Append, for every lane and every bit j of take, (v[j], out-degree dg[j])
 * to a queue: one 64-bit atomic per warp reserves (count << 32 | edge sum),
 * so e[] stays the exclusive prefix of out-degrees in queue order.  All 32
 * lanes call. */
template <int N>
__device__ __forceinline__ void enqueue_n(unsigned take, const int (&v)[N], const unsigned (&dg)[N],
                                          int *q, unsigned *e, unsigned long long *ctr) {
  const int lane = threadIdx.x & 31;
  if (!__any_sync(FULL, take != 0u)) return;
  const unsigned cnt = __popc(take);
  unsigned dsum = 0;
#pragma unroll
  for (int j = 0; j < N; ++j)
    if ((take >> j) & 1u) dsum += dg[j];
  unsigned ic = cnt, id = dsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned tc = __shfl_up_sync(FULL, ic, o);
    const unsigned td = __shfl_up_sync(FULL, id, o);
    if (lane >= o) {
      ic += tc;
      id += td;
    }
  }
  const unsigned tot_c = __shfl_sync(FULL, ic, 31), tot_d = __shfl_sync(FULL, id, 31);
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(ctr, ((unsigned long long)tot_c << 32) | tot_d);
  base = __shfl_sync(FULL, base, 0);
  unsigned pos = (unsigned)(base >> 32) + ic - cnt;
  unsigned eo = (unsigned)base + id - dsum;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    if ((take >> j) & 1u) {
      q[pos] = v[j];
      e[pos] = eo;
      ++pos;
      eo += dg[j];
    }
  }
}

/* largest o < cnt with e[o] <= t, per lane (fallback of the window search) */
__device__ __forceinline__ unsigned lane_owner(const unsigned *e, unsigned cnt, unsigned t) {
  unsigned lo = 0, hi = cnt;
  while (hi - lo > 1) {
    const unsigned mid = (lo + hi) >> 1;
    if (__ldcg(e + mid) <= t)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

/* Waits until every CTA has read what it plans the phase from: `want` arrivals
 * at ctl->planned.  An instance's queue counters, level and done flag are read
 * by all CTAs at the start of a phase and, for an instance that one CTA runs,
 * written by that CTA within the same phase: it may not do so before the last
 * of the others has them (a CTA that starts late, or is held up, would plan
 * another phase than the rest, and an instance be run twice or by nobody).
 * The arrivals of a phase are long there when an instance's first level is
 * done.  Bounded like the grid barrier; called by the whole CTA. */
__device__ __forceinline__ bool plans_read(MultiCtl *ctl, unsigned want, long long timeout_ns,
                                           unsigned ph) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned long long t0 = dev::global_ns();
    unsigned spins = 0;
    while ((int)(dev::ld_acquire_u32(&ctl->planned) - want) < 0) {
      if ((++spins & 31u) != 0) continue;
      if (dev::ld_volatile(&ctl->status) != 0) {
        ok = 0;
        break;
      }
      if ((long long)(dev::global_ns() - t0) > timeout_ns) {
        atomicCAS(&ctl->status, 0, (int)TBFS_ERR_TIMEOUT);
        atomicCAS(&ctl->timeout_level, 0, (int)ph + 2);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

/* This CTA runs instance D from level d on (qn vertices, qe out-edges) until
 * it is finished or has outgrown a CTA (`most` edges), the clock t_end, or a
 * stop request.
 * planned: arrivals after which D's counters may be written (plans_read);
 * false: they did not come in time. */
__device__ __forceinline__ bool local_run(const MultiParams &P, InstDesc &D, LocalShared &L, int d,
                                          unsigned qn, unsigned qe, unsigned most, unsigned ph,
                                          unsigned planned, long long t_end) {
  const int t = threadIdx.x, lane = t & 31;
  const unsigned wid = (unsigned)t >> 5;
  const int *rp = D.rp, *jr = D.jr;
  int *S = D.S;
  unsigned long long *sig = D.sig;
  for (unsigned i = t; i < qn; i += kLocalBlock) {
    const int v = __ldcg(D.q[d % 3] + i);
    L.v[d & 1][i] = v;
    L.e[d & 1][i] = __ldcg(D.e[d % 3] + i);
    L.a[d & 1][i] = __ldg(rp + v);
    if (sig) L.cnt[d & 1][i] = __ldcg(sig + v);
  }
  for (unsigned i = t; i < kSlots; i += kLocalBlock) {
    L.key[i] = kNoKey;
    L.lo[i] = L.hi[i] = 0u;
  }
  if (t < 3) L.ctr[t] = 0ull;
  __syncthreads();
  const int bits = D.deg_bits;
  const bool ovf_seen = __ldcg(&D.ovf) != 0;
  long long visited = 0, edges = 0;
  bool ovf = false;
  for (;;) {
    const int b = d & 1, c1 = (d + 1) % 3;
    visited += qn;
    edges += qe;
    int stop = 0;
    const long long t_level = clock64();
    if (t == 0) {
      L.ctr[(d + 2) % 3] = 0ull;
      stop = dev::ld_volatile(&P.ctl->stop[ph & 1u]);
    }
    const bool chk = sig && !ovf_seen && !(bits > 0 && 1 + (long long)(d + 1) * bits <= 63);
    /* a contiguous piece of the level's edges per warp, up to kEPT rounds of
     * 32 in flight */
    const unsigned steps = (qe + kLocalBlock - 1u) / kLocalBlock;
    const unsigned lim = min(qe, (wid + 1u) * steps * 32u);
    const bool early = steps <= 2u; /* latency counts: where the targets' lists are, unasked */
    const unsigned *le = L.e[b];
    unsigned base = wid * steps * 32u, i0 = 0;
    if (base < qe) { /* largest entry with e <= base */
      unsigned hi = qn;
      while (hi - i0 > 1) {
        const unsigned mid = (i0 + hi) >> 1;
        if (le[mid] <= base) i0 = mid;
        else hi = mid;
      }
    }
    for (; base < lim; base += 32u * kEPT) {
      int u[kEPT];
      unsigned k[kEPT];
      bool on[kEPT];
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        /* owner within the 32 entries from the last one's; past them (many
         * empty lists) step by step */
        const unsigned tj = base + 32u * j + lane;
        on[j] = tj < lim;
        u[j] = 0;
        k[j] = 0;
        if (base + 32u * j >= lim) continue; /* the whole warp */
        const unsigned w = i0 + lane < qn ? le[i0 + lane] : 0xffffffffu;
        unsigned o = 0;
#pragma unroll
        for (int h = 16; h > 0; h >>= 1)
          if (__shfl_sync(FULL, w, (int)(o + h)) <= tj) o += h;
        o += i0;
        if (on[j]) {
          while (o + 1 < qn && le[o + 1] <= tj) ++o;
          k[j] = o;
          u[j] = __ldg(jr + L.a[b][o] + (int)(tj - le[o]));
        }
        i0 = __shfl_sync(FULL, o, 31);
      }
      int sv[kEPT], ad[kEPT];
      unsigned dg[kEPT];
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        sv[j] = 0;
        ad[j] = 0;
        dg[j] = 0u;
        if (on[j]) {
          sv[j] = __ldcg(S + u[j]);
          if (early) {
            ad[j] = __ldg(rp + u[j]);
            dg[j] = (unsigned)__ldg(rp + u[j] + 1);
          }
        }
      }
      unsigned cnt = 0, dsum = 0, won = 0, sl[kEPT];
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        sl[j] = kNoSlot;
        /* not reached before this level (d + 1: just claimed by another lane) */
        on[j] = on[j] && (sv[j] == -1 || sv[j] == d + 1);
        if (on[j]) {
          bool is_new = false;
          sl[j] = find_slot(L, (unsigned)u[j], &is_new);
          if (is_new) S[u[j]] = d + 1;
          if (sl[j] == kNoSlot) is_new = atomicCAS(S + u[j], -1, d + 1) == -1;
          if (is_new) won |= 1u << j;
        }
        if (!early && ((won >> j) & 1u)) {
          ad[j] = __ldg(rp + u[j]);
          dg[j] = (unsigned)__ldg(rp + u[j] + 1);
        }
      }
      if (sig) { /* low words of all, then the carries and high words */
        unsigned long long x[kEPT];
        unsigned up[kEPT];
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          up[j] = 0u;
          x[j] = on[j] ? L.cnt[b][k[j]] : 0ull;
          if (on[j] && sl[j] != kNoSlot) up[j] = atomicAdd(&L.lo[sl[j]], (unsigned)x[j]);
        }
#pragma unroll
        for (int j = 0; j < kEPT; ++j) {
          if (on[j] && sl[j] != kNoSlot) {
            const unsigned carry = up[j] + (unsigned)x[j] < up[j] ? 1u : 0u;
            const unsigned xh = (unsigned)(x[j] >> 32), add = xh + carry;
            if (add < xh) ovf = true;
            if (add) {
              const unsigned old = atomicAdd(&L.hi[sl[j]], add);
              if (old + add < old || (old + add) >> 31) ovf = true;
            }
          } else if (on[j]) {
            if (chk) dev::add_chk(atomicAdd(sig + u[j], x[j]), x[j], ovf);
            else atomicAdd(sig + u[j], x[j]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        dg[j] -= (unsigned)ad[j];
        if ((won >> j) & 1u) {
          ++cnt;
          dsum += dg[j];
        }
      }
      if (!__any_sync(FULL, cnt)) continue;
      unsigned ic = cnt, id = dsum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned tc = __shfl_up_sync(FULL, ic, o), td = __shfl_up_sync(FULL, id, o);
        if (lane >= o) {
          ic += tc;
          id += td;
        }
      }
      unsigned long long at = 0;
      if (lane == 31) at = atomicAdd(&L.ctr[c1], ((unsigned long long)ic << 32) | id);
      at = __shfl_sync(FULL, at, 31);
      unsigned pos = (unsigned)(at >> 32) + ic - cnt, eo = (unsigned)at + id - dsum;
#pragma unroll
      for (int j = 0; j < kEPT; ++j) {
        if ((won >> j) & 1u) {
          if (pos < kLocalQueue) {
            L.slot[pos] = (unsigned short)sl[j];
            L.v[b ^ 1][pos] = u[j];
            L.a[b ^ 1][pos] = ad[j];
            L.e[b ^ 1][pos] = eo;
          } else { /* more than fit: where the instance's queue has them */
            D.q[c1][pos] = u[j];
            D.e[c1][pos] = eo;
          }
          ++pos;
          eo += dg[j];
        }
      }
    }
    if (t == 0) { /* no time for another such level */
      const long long now = clock64();
      L.leave[b] = stop || now + (now - t_level) > t_end;
    }
    __syncthreads();
    ++d;
    const unsigned long long cur = L.ctr[c1];
    qn = (unsigned)(cur >> 32);
    qe = (unsigned)cur;
    /* the counts to memory, and the table empty again */
    if (qn <= kLocalQueue) {
      for (unsigned i = t; i < qn; i += kLocalBlock) {
        const unsigned s = L.slot[i];
        const int v = L.v[b ^ 1][i];
        if (s != kNoSlot) {
          const unsigned long long x = ((unsigned long long)L.hi[s] << 32) | L.lo[s];
          if (sig) sig[v] = L.cnt[b ^ 1][i] = x;
          L.key[s] = kNoKey;
          L.lo[s] = L.hi[s] = 0u;
        } else if (sig) {
          L.cnt[b ^ 1][i] = __ldcg(sig + v);
        }
      }
    } else if (sig) { /* the instance leaves */
      for (unsigned s = t; s < kSlots; s += kLocalBlock)
        if (L.key[s] != kNoKey) sig[L.key[s]] = ((unsigned long long)L.hi[s] << 32) | L.lo[s];
    }
    if (qn == 0u || qn > kLocalQueue || qe > most || L.leave[b]) {
      for (unsigned i = t; i < qn && i < kLocalQueue; i += kLocalBlock) {
        D.q[c1][i] = L.v[b ^ 1][i];
        D.e[c1][i] = L.e[b ^ 1][i];
      }
      if (__any_sync(FULL, ovf) && lane == 0) atomicExch(&D.ovf, 1);
      if (!plans_read(P.ctl, planned, P.timeout_ns, ph)) return false;
      if (t == 0) {
        D.ctr[c1] = cur;
        D.ctr[(d + 1) % 3] = 0ull;
        D.ctr[(d + 2) % 3] = 0ull;
        D.d = d;
        D.levels = d;
        D.visited = __ldcg(&D.visited) + visited;
        D.edges = __ldcg(&D.edges) + edges;
        if (qn == 0u) {
          D.done = 1;
          if (P.stop_on_done) *(volatile int *)&P.ctl->stop[ph & 1u] = 1;
        }
      }
      __syncthreads(); /* before the next instance's queue */
      return true;
    }
    __syncthreads();
  }
}

template <bool LOCAL>
__global__ void __launch_bounds__(LOCAL ? kLocalBlock : kSharedBlock, LOCAL ? 1 : kSharedPerSm)
    multi_bfs_kernel(const MultiParams P) {
  constexpr int kBlock = LOCAL ? kLocalBlock : kSharedBlock;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ int s_mine[LOCAL ? kLocalMine : 1]; /* this CTA's instances */
  constexpr int kWarps = kBlock / 32;
  __shared__ unsigned s_pre[kMultiMaxSlots + 1]; /* item prefix over slots      */
  __shared__ int s_d[kMultiMaxSlots];            /* level each slot runs next   */
  __shared__ unsigned s_qn[kMultiMaxSlots], s_qe[kMultiMaxSlots];
  __shared__ unsigned long long s_wsum[kWarps];  /* per-warp edge sums          */
  __shared__ int s_wact[kWarps];
  __shared__ unsigned long long s_wscan[kWarps]; /* per-warp item sums          */
  InstDesc *I = P.inst;
  const int ns = P.nslots;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const long long tid = (long long)blockIdx.x * kBlock + t;
  MultiCtl *ctl = P.ctl;

  for (int i = t; i < ns; i += kBlock) s_d[i] = __ldcg(&I[i].d);
  __syncthreads();

  const bool use_local = LOCAL && gridDim.x >= kLocalGrid;
  unsigned enter = kLocalEnter;
  unsigned planned = 0; /* arrivals at ctl->planned up to this phase */
  unsigned ph = 0;
  for (; ph < (unsigned)P.max_phases; ++ph) {
    /* the host's "request waiting" flag (mapped host memory, a slow read):
     * issued now, used at the end of the level */
    int wake_now = 0;
    if (tid == 0 && P.wake) wake_now = *P.wake;
    const long long t_begin = clock64();
    if (LOCAL && t < kLocalMine) s_mine[t] = -1;
    /* ---- plan: identical in every CTA (reads counters finished before the
     * last barrier: a shared instance's of this level are only added to, and
     * those of an instance run by one CTA are written once all CTAs have read
     * them, plans_read); block sums and scans by warp shuffles ---- */
    constexpr int kPer = (kMultiMaxSlots + kBlock - 1) / kBlock;
    /* every read of the plan in one round trip: the previous level's stop
     * word, each slot's done flag and queue counter, and (CTA 0) the totals
     * its bookkeeping adds to */
    const bool stop_prev = ph > 0 && __ldcg(&ctl->stop[(ph - 1) & 1u]) != 0;
    unsigned long long qvs[kPer];
    long long vis[kPer], edg[kPer];
    bool dns[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = t * kPer + j;
      qvs[j] = 0ull;
      vis[j] = edg[j] = 0;
      dns[j] = true;
      if (i < ns) {
        dns[j] = __ldcg(&I[i].done) != 0;
        qvs[j] = __ldcg(&I[i].ctr[s_d[i] % 3]);
        if (blockIdx.x == 0) {
          vis[j] = I[i].visited;
          edg[j] = I[i].edges;
        }
      }
    }
    /* a stop requested during the previous level ends the launch before
     * any bookkeeping of this one */
    if (stop_prev) break;
    unsigned qes[kPer];
    bool loc[kPer];
    unsigned long long esum = 0;
    int act = 0, fin = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = t * kPer + j;
      qes[j] = 0;
      loc[j] = false;
      if (i < ns) {
        const int d = s_d[i];
        const bool done = dns[j];
        const unsigned long long qv = done ? 0ull : qvs[j];
        const unsigned qn = (unsigned)(qv >> 32), qe = (unsigned)qv;
        loc[j] = use_local && qn && qn <= kLocalQueue && qe <= enter;
        s_qn[i] = loc[j] ? qn | kIsLocal : qn;
        s_qe[i] = qe;
        if (qn) {
          act |= loc[j] ? 1 : 2;
          if (!loc[j]) {
            qes[j] = qe;
            esum += qe;
          }
        }
        /* bookkeeping of a shared instance, by CTA 0 */
        if (blockIdx.x == 0 && !done && !loc[j]) {
          if (qn) {
            I[i].ctr[(d + 2) % 3] = 0ull;
            I[i].levels = d + 1;
            I[i].visited = vis[j] + qn;
            I[i].edges = edg[j] + qe;
          } else {
            I[i].done = 1;
            fin = 1;
          }
        }
      }
    }
    if (fin && P.stop_on_done) ctl->stop[ph & 1u] = 1; /* CTA 0 only; read after the barrier */
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) esum += __shfl_xor_sync(FULL, esum, o);
    const int wact = (__any_sync(FULL, act & 1) ? 1 : 0) | (__any_sync(FULL, act & 2) ? 2 : 0);
    if (lane == 0) {
      s_wsum[wid] = esum;
      s_wact[wid] = wact;
    }
    __syncthreads();
    unsigned long long etot = 0;
    int any_act = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      etot += s_wsum[w];
      any_act |= s_wact[w];
    }
    if (!any_act) break;
    if (LOCAL && (any_act & 1)) { /* this CTA has read them */
      planned += gridDim.x;
      if (t == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(&ctl->planned), "r"(1u)
                     : "memory");
    }
    /* rounds per item: enough items for every warp on small levels */
    const unsigned nwarps = gridDim.x * kWarps;
    const unsigned long long per_warp =
        min(etot, 0xffffffffull) / ((unsigned long long)kRoundEdges * nwarps);
    const unsigned rounds = (unsigned)max(1ull, min((unsigned long long)kMaxRounds, per_warp));
    const unsigned iedges = kRoundEdges * rounds;
    unsigned items[kPer];
    unsigned long long sum = 0; /* instances shared << 48 | run by one CTA << 32 | items */
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      items[j] = (qes[j] + iedges - 1) / iedges;
      sum += items[j] + (loc[j] ? 1ull << 32 : 0ull) + (items[j] ? 1ull << 48 : 0ull);
    }
    /* exclusive scan of the per-thread sums: within the warp by shuffles,
     * across the warps from their totals */
    unsigned long long inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long x = __shfl_up_sync(FULL, inc, o);
      if (lane >= o) inc += x;
    }
    if (lane == 31) s_wscan[wid] = inc;
    __syncthreads();
    unsigned long long wbase = 0, wtot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const unsigned long long v = s_wscan[w];
      if (w < wid) wbase += v;
      wtot += v;
    }
    const unsigned total = (unsigned)wtot;
    unsigned run = (unsigned)(wbase + inc - sum);
    unsigned rank = (unsigned)((wbase + inc - sum) >> 32) & 0xffffu;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = t * kPer + j;
      if (i < ns) s_pre[i] = run;
      run += items[j];
      if (LOCAL && loc[j]) { /* instance `rank` of the local ones, on CTA 1 and up */
        if (rank % (gridDim.x - 1u) + 1u == blockIdx.x) s_mine[rank / (gridDim.x - 1u)] = i;
        ++rank;
      }
    }
    if (t == 0) s_pre[ns] = total;
    __syncthreads();
    if (tid == 0) ctl->work[(ph + 2) & 3u] = 0u;

    /* ---- claim items: the first one statically (global warp index), the
     * rest from the phase's counter, so that a level with few items costs
     * no same-address atomics ---- */
    unsigned it = (unsigned)wid * gridDim.x + blockIdx.x; /* round-robin over the CTAs */
    for (;; ) {
      if (it >= total) break;
      /* slot of the item: largest i with s_pre[i] <= it */
      unsigned lo = 0, hi = (unsigned)ns;
      while (hi - lo > 1) {
        const unsigned mid = (lo + hi) >> 1;
        if (s_pre[mid] <= it)
          lo = mid;
        else
          hi = mid;
      }
      const int i = (int)lo;
      InstDesc &D = I[i];
      const int d = s_d[i];
      const unsigned qn = s_qn[i], qe = s_qe[i];
      const int *q = D.q[d % 3];
      const unsigned *e = D.e[d % 3];
      int *qn_q = D.q[(d + 1) % 3];
      unsigned *qn_e = D.e[(d + 1) % 3];
      unsigned long long *ctr1 = &D.ctr[(d + 1) % 3];
      const int *rp = D.rp, *jr = D.jr;
      int *S = D.S;
      unsigned long long *sig = D.sig;
      /* counts of level d+1 have at most 1 + (d+1) deg_bits bits: below 64
       * they cannot overflow, and neither need be checked once the
       * instance's overflow is recorded; such adds are reductions whose old
       * value nobody waits for */
      const bool chk = sig && !(D.deg_bits > 0 && 1 + (long long)(d + 1) * D.deg_bits <= 63) &&
                       __ldcg(&D.ovf) == 0;
      const unsigned t0 = (it - s_pre[i]) * iedges;
      bool ovf = false;
      unsigned o0 = 0xffffffffu; /* owner of the round's first edge, once known */
      for (unsigned r = 0; r < rounds; ++r) {
        const unsigned tb = t0 + r * kRoundEdges;
        if (tb >= qe) break;
        /* owners: a 32-ary search for the item's first edge, afterwards the
         * owner of the previous round's last edge; a window of 32 queue
         * entries from there is searched with shuffles, edges beyond it
         * (runs of empty lists) by a binary search of their own */
        if (o0 == 0xffffffffu) o0 = dev::warp_find_owner(reinterpret_cast<const int *>(e), qn, tb);
        /* the window's queue entries come with their prefixes; their list
         * starts and path counts follow in one more round trip, so that an
         * edge inside the window needs only its list entry */
        const unsigned wi = o0 + lane;
        const bool in0 = wi < qn, in1 = wi + 32 < qn;
        const unsigned ew0 = in0 ? __ldcg(e + wi) : 0xffffffffu;
        const unsigned ew1 = in1 ? __ldcg(e + wi + 32) : 0xffffffffu;
        const int qw0 = in0 ? __ldcg(q + wi) : 0;
        const int qw1 = in1 ? __ldcg(q + wi + 32) : 0;
        const unsigned eend = o0 + 64 < qn ? __ldcg(e + o0 + 64) : 0xffffffffu;
        const int aw0 = in0 ? __ldg(rp + qw0) : 0;
        const int aw1 = in1 ? __ldg(rp + qw1) : 0;
        unsigned long long gw0 = 0ull, gw1 = 0ull;
        if (sig) {
          gw0 = in0 ? sig[qw0] : 0ull;
          gw1 = in1 ? sig[qw1] : 0ull;
        }
        unsigned tk[kEPT], off[kEPT], ow[kEPT];
        int u[kEPT], a[kEPT];
        unsigned long long su[kEPT];
#pragma unroll
        for (int k = 0; k < kEPT; ++k) {
          tk[k] = tb + kEPT * lane + k;
          unsigned j = 0; /* largest window index with e <= tk */
#pragma unroll
          for (int s = 32; s > 0; s >>= 1) {
            const unsigned c = j + s;
            const unsigned a0 = __shfl_sync(FULL, ew0, (int)(c & 31));
            const unsigned a1 = __shfl_sync(FULL, ew1, (int)(c & 31));
            if (c < 64 && (c < 32 ? a0 : a1) <= tk[k]) j = c;
          }
          const int src = (int)(j & 31);
          const bool hi = j >= 32;
          const unsigned b0 = __shfl_sync(FULL, ew0, src), b1 = __shfl_sync(FULL, ew1, src);
          const int u0 = __shfl_sync(FULL, qw0, src), u1 = __shfl_sync(FULL, qw1, src);
          const int c0 = __shfl_sync(FULL, aw0, src), c1 = __shfl_sync(FULL, aw1, src);
          const unsigned long long g0 = __shfl_sync(FULL, gw0, src);
          const unsigned long long g1 = __shfl_sync(FULL, gw1, src);
          ow[k] = o0 + j;
          off[k] = tk[k] - (hi ? b1 : b0);
          u[k] = hi ? u1 : u0;
          a[k] = hi ? c1 : c0;
          su[k] = hi ? g1 : g0;
          if (tk[k] < qe && tk[k] >= eend) { /* past the window: owner of its own */
            const unsigned oo = lane_owner(e, qn, tk[k]);
            ow[k] = oo;
            off[k] = tk[k] - __ldcg(e + oo);
            u[k] = __ldcg(q + oo);
            a[k] = __ldg(rp + u[k]);
            su[k] = sig ? sig[u[k]] : 0ull;
          }
        }
        int v[kEPT], sv[kEPT];
        unsigned dgo[kEPT];
#pragma unroll
        for (int k = 0; k < kEPT; ++k) v[k] = tk[k] < qe ? __ldg(jr + a[k] + (int)off[k]) : 0;
#pragma unroll
        for (int k = 0; k < kEPT; ++k) sv[k] = tk[k] < qe ? S[v[k]] : 0;
        /* degrees of the unvisited targets, in flight with the claims */
        int r0[kEPT], r1[kEPT];
#pragma unroll
        for (int k = 0; k < kEPT; ++k) {
          r0[k] = 0;
          r1[k] = 0;
          if (tk[k] < qe && sv[k] == -1) {
            r0[k] = __ldg(rp + v[k]);
            r1[k] = __ldg(rp + v[k] + 1);
          }
        }
        unsigned take = 0;
#pragma unroll
        for (int k = 0; k < kEPT; ++k) {
          if (tk[k] < qe && sv[k] == -1) {
            sv[k] = atomicCAS(S + v[k], -1, d + 1);
            if (sv[k] == -1) {
              take |= 1u << k;
              sv[k] = d + 1;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < kEPT; ++k) dgo[k] = ((take >> k) & 1u) ? (unsigned)(r1[k] - r0[k]) : 0u;
        if (sig) {
#pragma unroll
          for (int k = 0; k < kEPT; ++k) {
            if (tk[k] < qe && sv[k] == d + 1) {
              const unsigned long long x = su[k];
              if (chk) {
                const unsigned long long old = atomicAdd(sig + v[k], x);
                const unsigned long long s2 = old + x;
                if (s2 < old || (s2 >> 63)) ovf = true;
              } else {
                atomicAdd(sig + v[k], x); /* result unused: a reduction */
              }
            }
          }
        }
        enqueue_n<kEPT>(take, v, dgo, qn_q, qn_e, ctr1);
        o0 = __shfl_sync(FULL, ow[kEPT - 1], 31); /* owner of the round's last edge */
      }
      if (__any_sync(FULL, ovf) && lane == 0) atomicExch(&D.ovf, 1);
      if (total <= nwarps) break;
      unsigned nx = 0;
      if (lane == 0) nx = nwarps + atomicAdd(&ctl->work[ph & 3u], 1u);
      it = __shfl_sync(FULL, nx, 0);
    }
    if (LOCAL && (any_act & 1)) { /* instances run by single CTAs */
      LocalShared &L = *reinterpret_cast<LocalShared *>(s_dyn);
      const long long level = kLocalBeside + (long long)(etot / kLocalEdges);
      const long long most = (any_act & 2) && level < kLocalAlone ? level : kLocalAlone;
      const long long span = most < P.timeout_ns / 4 ? most : P.timeout_ns / 4;
      const long long t_end = t_begin + span;
      int mine = 0;
      while (mine < kLocalMine && s_mine[mine] >= 0) ++mine;
      for (int m = 0; m < mine; ++m) { /* equal parts of the time */
        const int i = s_mine[m];
        if (!local_run(P, I[i], L, s_d[i], s_qn[i] & ~kIsLocal, s_qe[i], enter + enter / 2,
                       ph, planned,
                       t_begin + span * (m + 1) / mine))
          return;
      }
      /* CTA 0 has none: it watches for requests until all others arrived */
      if (tid == 0 && P.wake) {
        const unsigned others = gridDim.x - 1u;
        while (!wake_now && clock64() < t_end &&
               (dev::ld_acquire_u32(&ctl->bar.arrive) & 0x7fffffffu) != others)
          wake_now = *P.wake;
        if (wake_now) *(volatile int *)&ctl->stop[ph & 1u] = 1;
      }
    }
    enter = (unsigned)(wtot >> 48) + ((unsigned)(wtot >> 32) & 0xffffu) > kFew ? 2 * kLocalEnter
                                                                               : kLocalEnter;
    /* a waiting request (host flag) ends the launch after this level */
    if (tid == 0 && wake_now) ctl->stop[ph & 1u] = 1;
    if (!grid_barrier(ctl, P.timeout_ns, (int)ph)) return;
    for (int i = t; i < ns; i += kBlock) {
      if (LOCAL && (s_qn[i] & kIsLocal)) s_d[i] = __ldcg(&I[i].d);
      else if (s_qn[i]) s_d[i] += 1;
    }
    __syncthreads();
  }
  /* the level each instance runs next, for the following launch */
  if (blockIdx.x == 0)
    for (int i = t; i < ns; i += kBlock) I[i].d = s_d[i];
  if (tid == 0) ctl->phases = (int)ph;
}

/* new instances: depths -1 and counts 0, 0 and 1 at the root, queue {root}.
 * One launch for all of them (blockIdx.y): two memsets per instance took 2.4 us
 * of the host each, and more than a small traversal. */
__global__ void __launch_bounds__(kInitBlock) multi_init_kernel(InstDesc *I, const int *slots) {
  InstDesc &D = I[slots[blockIdx.y]];
  const int r = D.inv ? D.inv[D.root] : D.root;
  int *S = D.S;
  unsigned long long *sig = D.sig;
  const long long n = D.n, step = (long long)gridDim.x * kInitBlock * 4;
  for (long long i = ((long long)blockIdx.x * kInitBlock + threadIdx.x) * 4; i < n; i += step) {
    if (i + 4 <= n) { /* both arrays start on 256 bytes */
      *reinterpret_cast<int4 *>(S + i) =
          make_int4(i == r ? 0 : -1, i + 1 == r ? 0 : -1, i + 2 == r ? 0 : -1, i + 3 == r ? 0 : -1);
      if (sig) {
        *reinterpret_cast<ulonglong2 *>(sig + i) = make_ulonglong2(i == r, i + 1 == r);
        *reinterpret_cast<ulonglong2 *>(sig + i + 2) = make_ulonglong2(i + 2 == r, i + 3 == r);
      }
    } else {
      for (long long k = i; k < n; ++k) {
        S[k] = k == r ? 0 : -1;
        if (sig) sig[k] = k == r ? 1ull : 0ull;
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    D.q[0][0] = r;
    D.e[0][0] = 0u;
    D.ctr[0] = (1ull << 32) | (unsigned)(D.rp[r + 1] - D.rp[r]);
  }
}

/* results in the caller's numbering: out[j] = S[inv[j]] */
__global__ void multi_gather_kernel(const int *S, const unsigned long long *sig, const int *inv,
                                    int n, int *S_out, unsigned long long *sig_out) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const int v = inv ? inv[j] : (int)j;
  S_out[j] = S[v];
  if (sig_out) sig_out[j] = sig[v];
}

/* results of all instances (blockIdx.y), each at its place in the packed outputs */
__global__ void __launch_bounds__(kInitBlock) multi_pack_kernel(const InstDesc *I, int *S_out,
                                                                unsigned long long *sig_out) {
  const InstDesc &D = I[blockIdx.y];
  const long long step = (long long)gridDim.x * kInitBlock;
  for (long long i = (long long)blockIdx.x * kInitBlock + threadIdx.x; i < D.n; i += step) {
    S_out[D.out + i] = D.S[i];
    if (sig_out) sig_out[D.out + i] = D.sig[i];
  }
}

}  // namespace

static const void *multi_kernel(bool local) {
  return local ? reinterpret_cast<const void *>(multi_bfs_kernel<true>)
               : reinterpret_cast<const void *>(multi_bfs_kernel<false>);
}

static size_t multi_smem(bool local) { return local ? sizeof(LocalShared) : 0; }

bool multi_local(int n_most) { return n_most <= kLocalVertices; }

cudaError_t multi_geometry(int device, MultiGeom *out) {
  int sms = 0, coop = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  if (e != cudaSuccess) return e;
  if (!coop) return cudaErrorNotSupported;
  e = cudaFuncSetAttribute(multi_kernel(true), cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)multi_smem(true));
  for (int local = 0; local < 2 && e == cudaSuccess; ++local) {
    const int block = local ? kLocalBlock : kSharedBlock, most = local ? 1 : kSharedPerSm;
    int per = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, multi_kernel(local != 0), block,
                                                      multi_smem(local != 0));
    if (e == cudaSuccess && per < 1) e = cudaErrorInvalidConfiguration;
    out->shape[local].block = block;
    out->shape[local].grid = sms * std::min(per, most);
  }
  return e;
}

cudaError_t multi_launch(const MultiParams &p, const MultiGeom &g, bool local, cudaStream_t s) {
  void *args[] = {const_cast<MultiParams *>(&p)};
  const LaunchGeom &shape = g.shape[local ? 1 : 0];
  return cudaLaunchCooperativeKernel(multi_kernel(local), dim3(shape.grid), dim3(shape.block), args,
                                     multi_smem(local), s);
}

/* blocks (x) for the k instances of a launch, the largest of n vertices, each
 * thread with `per` of them: as many as the largest asks for while all
 * together are at most ~16 per SM */
static unsigned inst_blocks(int n, int k, int per) {
  const long long want = ((long long)n + (long long)kInitBlock * per - 1) / ((long long)kInitBlock * per);
  const long long most = 2432 / k + 1;
  return (unsigned)std::max(1ll, std::min(want, most));
}

cudaError_t multi_init(InstDesc *inst, const int *slots, int k, int n_most, cudaStream_t s) {
  if (k <= 0) return cudaSuccess;
  multi_init_kernel<<<dim3(inst_blocks(n_most, k, 4), (unsigned)k), kInitBlock, 0, s>>>(inst, slots);
  return cudaGetLastError();
}

cudaError_t multi_pack(const InstDesc *inst, int k, int n_most, int *S_out,
                       unsigned long long *sig_out, cudaStream_t s) {
  if (k <= 0) return cudaSuccess;
  multi_pack_kernel<<<dim3(inst_blocks(n_most, k, 1), (unsigned)k), kInitBlock, 0, s>>>(inst, S_out,
                                                                                     sig_out);
  return cudaGetLastError();
}

cudaError_t multi_gather(const int *S, const unsigned long long *sig, const int *inv, int n,
                         int *S_out, unsigned long long *sig_out, cudaStream_t s) {
  multi_gather_kernel<<<(unsigned)(((long long)n + 255) / 256), 256, 0, s>>>(S, sig, inv, n, S_out,
                                                                            sig_out);
  return cudaGetLastError();
}

}  // namespace tbfs
