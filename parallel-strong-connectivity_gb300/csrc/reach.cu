// Single-source reachability on the device (REACH, src/reach.hpp:21-243).
//
// A search "side" is one direction from one source.  The first pivot of SCC
// needs a forward and a backward side; both run in the same launches, so the
// two latency-bound searches overlap.  Each round, per side:
//   push: the frontier is a u32 queue; warps expand 32 frontier vertices at a
//         time with the balanced warp expansion, claim targets on the visited
//         bitmap and append winners with one warp-aggregated atomic (the
//         reference's hashbag insert + pack); vertices above kHeavyDeg
//         out-edges go to a heavy list that the whole grid expands next;
//   VGC:  (local search, reach.hpp:114-171) one frontier vertex per warp runs
//         a local BFS in a shared-memory queue of up to tau vertices before
//         spilling the rest to the next frontier — used while the frontier is
//         small, where rounds, not bandwidth, bound the search.  Steady or
//         low-degree searches leave the rounds altogether (k_reach_async);
//   pull: the frontier is a bitmap; a warp takes 4 to 32 words of the visited
//         bitmap, lists the vertices that are neither visited nor without
//         in-edges (a bitmap per direction, built once per handle: no pull can
//         reach those) in shared memory, and scans the in-edges of the listed
//         ones until a frontier bit is found; the visited / next-frontier words
//         are written with one store each (the reference's dense_update).
// On graphs of up to kRrMaxEdges edges push and pull rounds run in one resident
// launch instead (k_reach_rounds; its pull rounds take 32 consecutive vertices per
// warp and know no unreachable ones).
// The push/pull switch follows the reference's rule (REACH::judge, reach.hpp:86-112):
// push while frontier vertices + their out-edges < m / pull_div (20).  After a
// push round the out-edge count is exact (gathered by the kernels); after a
// pull round it is exact for a frontier under 2^14 vertices and otherwise
// estimated from 50 sampled frontier vertices, as the reference's
// dense_sample does (reach.hpp:192-206).
//
// Expansion issues K edges per lane before using any of them, so the loads of
// E and the claims on the bitmap overlap instead of forming one dependent
// memory round trip per edge.
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "async_rules.h"
#include "common.cuh"
#include "engines.cuh"
#include "levels.cuh"
#include "pull.cuh"

namespace psc {

constexpr int kReachBlock = 256;
constexpr int kVgcBlock = 128;  // VGC blocks: 4 warps
constexpr int kVgcQueue = 512;  // VGC queue entries per warp (8 KB of 16-byte entries)
// VGC: edges in flight per lane.  Sparse graphs (fewer than 8 edges per vertex
// on average) use 4: fewer registers, 6 instead of 5 resident blocks per SM,
// more local searches at once (kNN 10^7: 16.8 -> 16.3 ms, grid 4096^2:
// 17.6 -> 16.3 ms); denser ones and batches use 8 (a 1024-graph batch: 16.2
// instead of 19.1 ms).
constexpr int kVgcKWide = 8;
constexpr int kVgcKNarrow = 4;
constexpr int kPushK = 4;       // push: edges in flight per lane
constexpr int kHeavyK = 4;      // heavy vertices: edges in flight per lane
constexpr uint64_t kHeavyChunk = 32 * kHeavyK;  // edges of one heavy-list work unit

// One search side as the kernels see it.
struct ReachSide {
  const uint64_t* off;  // adjacency of the search direction
  const uint32_t* E;
  const uint32_t* qin;  // current frontier (queue)
  uint64_t nin;
  uint32_t* vis;        // visited bitmap
  uint32_t* qout;       // next frontier (queue)
  uint64_t* heavy;      // heavy list: vertex << 32 | first chunk (see heavy_push)
  Counters* ctr;
  const VRec* rec;      // adjacency records, for k_reach_async (or null)
};

// Lists a vertex with more than kHeavyDeg out-edges for k_reach_heavy.  Its
// edges are cut into chunks of kHeavyChunk; one 64-bit atomic on ctr->heavy =
// count << kPackShift | chunks gives the entry its slot and its first chunk,
// so entries in slot order have increasing first chunks.
__device__ __forceinline__ void heavy_push(const ReachSide& S, uint32_t u, uint64_t deg) {
  const unsigned long long old = atomicAdd(
      &S.ctr->heavy, (1ull << kPackShift) + (deg + kHeavyChunk - 1) / kHeavyChunk);
  S.heavy[old >> kPackShift] = ((uint64_t)u << 32) | (old & kPackMask);
}

__global__ void k_reach_init(uint32_t* vis, uint32_t* q, uint32_t src) {
  vis[src >> 5] = 1u << (src & 31);
  q[0] = src;
}

// Several sources at once (one per graph of a batch).
__global__ void k_reach_init_multi(uint32_t* vis, uint32_t* q, const uint32_t* __restrict__ srcs,
                                   uint64_t ns) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ns;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = srcs[i];
    atomicOr(&vis[v >> 5], 1u << (v & 31));
    q[i] = v;
  }
}

__device__ __forceinline__ int find_src(const WarpExpandSmem& sm, uint32_t gi) {
  int lo = 0, hi = 31;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (sm.excl[mid] <= gi)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Balanced expansion of the 32 lanes' ranges [beg, beg+deg) with K edges per
// lane in flight: K loads of E, then a read of each target's bitmap word, then
// atomicOr claims only for targets still unvisited.  emit(tm, v) gets the
// lane's K candidates and the mask of those it claimed (warp-collective).
template <int K, class Emit>
__device__ __forceinline__ void expand_claim(WarpExpandSmem& sm, uint64_t beg, uint32_t deg,
                                             const uint32_t* __restrict__ E, uint32_t* vis,
                                             Emit&& emit) {
  const unsigned lane = lane_id();
  uint32_t incl = deg;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(kFull, incl, o);
    if ((int)lane >= o) incl += t;
  }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  sm.excl[lane] = incl - deg;
  sm.beg[lane] = beg;
  __syncwarp();
  for (uint32_t base = 0; base < total; base += 32 * K) {
    uint32_t v[K];
    uint32_t pre = 0, tm = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t gi = base + k * 32 + lane;
      v[k] = 0xFFFFFFFFu;
      if (gi < total) {
        const int s = find_src(sm, gi);
        v[k] = __ldg(&E[sm.beg[s] + (gi - sm.excl[s])]);
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
      if (v[k] != 0xFFFFFFFFu && !(__ldcg(&vis[v[k] >> 5]) & (1u << (v[k] & 31)))) pre |= 1u << k;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (pre & (1u << k)) {
        const uint32_t b = 1u << (v[k] & 31);
        if (!(atomicOr(&vis[v[k] >> 5], b) & b)) tm |= 1u << k;
      }
    emit(tm, v);
  }
  __syncwarp();
}

__device__ __forceinline__ void flush_side_counters(Counters* c0, Counters* c1,
                                                    unsigned long long s0, unsigned long long s1,
                                                    unsigned long long n0, unsigned long long n1,
                                                    unsigned long long x0, unsigned long long x1) {
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  n0 = warp_sum(n0);
  n1 = warp_sum(n1);
  x0 = warp_sum(x0);
  x1 = warp_sum(x1);
  if (lane_id() == 0) {
    if (s0 | n0 | x0) {
      atomicAdd(&c0->edges, s0);
      atomicAdd(&c0->next_edges, n0);
      atomicAdd(&c0->expanded, x0);
    }
    if (s1 | n1 | x1) {
      atomicAdd(&c1->edges, s1);
      atomicAdd(&c1->next_edges, n1);
      atomicAdd(&c1->expanded, x1);
    }
  }
}

// Push round for up to two sides: 32 frontier vertices per warp step.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_reach_push(ReachSide s0, ReachSide s1) {
  __shared__ WarpExpandSmem sm[BLOCK / 32];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint64_t gw = (uint64_t)blockIdx.x * (BLOCK / 32) + wid;
  const uint64_t nw = (uint64_t)gridDim.x * (BLOCK / 32);
  const uint64_t c0 = (s0.nin + 31) / 32, c1 = (s1.nin + 31) / 32;
  unsigned long long scanned0 = 0, scanned1 = 0, nedges0 = 0, nedges1 = 0, exp0 = 0, exp1 = 0;
  for (uint64_t c = gw; c < c0 + c1; c += nw) {
    const int sd = c < c0 ? 0 : 1;
    const ReachSide S = sd ? s1 : s0;
    const uint64_t i = (sd ? c - c0 : c) * 32 + lane;
    uint64_t beg = 0;
    uint32_t deg = 0;
    if (i < S.nin) {
      const uint32_t u = S.qin[i];
      beg = S.off[u];
      uint64_t d = S.off[u + 1] - beg;
      (sd ? exp1 : exp0)++;
      if (d > kHeavyDeg) {
        heavy_push(S, u, d);
        d = 0;
      }
      deg = (uint32_t)d;
    }
    (sd ? scanned1 : scanned0) += deg;
    expand_claim<kPushK>(sm[wid], beg, deg, S.E, S.vis, [&](uint32_t tm, const uint32_t* v) {
      warp_append_batch<kPushK>(tm, v, S.qout, &S.ctr->next);
#pragma unroll
      for (int k = 0; k < kPushK; k++)
        if (tm & (1u << k)) (sd ? nedges1 : nedges0) += S.off[v[k] + 1] - S.off[v[k]];
    });
  }
  flush_side_counters(s0.ctr, s1.ctr, scanned0, scanned1, nedges0, nedges1, exp0, exp1);
}

// Local-queue entry: a claimed vertex with its adjacency range.
struct QEnt {
  uint64_t beg;
  uint32_t v;
  uint32_t deg;
};

// Places this lane's claimed candidates (bit k of tm <=> w[k] claimed) into the
// warp's local queue while it has room, then spills the rest to the global
// frontier: one warp scan and at most one global atomic for the whole warp.
template <int K>
__device__ __forceinline__ void vgc_place(uint32_t tm, const uint32_t* w, const uint64_t* vb,
                                          const uint64_t* ve, QEnt* Q, uint32_t& tail, uint32_t tq,
                                          uint32_t* qout, unsigned long long* next_ctr,
                                          unsigned long long& nedges) {
  const unsigned lane = lane_id();
  const uint32_t cnt = __popc(tm);
  uint32_t incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if ((int)lane >= o) incl += t;
  }
  const uint32_t total = __shfl_sync(kFull, incl, 31);
  if (total == 0) return;
  const uint32_t room = tail < tq ? tq - tail : 0;
  const uint32_t nloc = total < room ? total : room;
  unsigned long long sbase = 0;
  if (total > nloc && lane == 0) sbase = atomicAdd(next_ctr, (unsigned long long)(total - nloc));
  sbase = __shfl_sync(kFull, sbase, 0);
  uint32_t r = incl - cnt;
#pragma unroll
  for (int k = 0; k < K; k++)
    if (tm & (1u << k)) {
      const uint64_t vd = ve[k] - vb[k];
      if (r < nloc) {
        Q[tail + r] = QEnt{vb[k], w[k], (uint32_t)(vd < 0xFFFFFFFFull ? vd : 0xFFFFFFFFull)};
      } else {
        qout[sbase + (r - nloc)] = w[k];
        nedges += vd;
      }
      r++;
    }
  tail += nloc;
  __syncwarp();
}

// Claims of one batch: a claimed vertex enters the queue with its adjacency
// range, so the next wave needs no dependent load.  SPEC: the range is loaded
// alongside the claim (off the claim's latency chain, but wasted traffic when
// the claim fails), for latency-bound rounds; otherwise only after a claim
// succeeds, for rounds with more frontier than resident warps.
template <int K, bool SPEC>
__device__ __forceinline__ uint32_t vgc_claim(const uint32_t* w, uint64_t* vb, uint64_t* ve,
                                              const uint64_t* __restrict__ off, uint32_t* vis) {
  if (SPEC) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      vb[k] = ve[k] = 0;
      if (w[k] != 0xFFFFFFFFu) {
        vb[k] = __ldg(&off[w[k]]);
        ve[k] = __ldg(&off[w[k] + 1]);
      }
    }
  }
  uint32_t tm = 0;
#pragma unroll
  for (int k = 0; k < K; k++)
    if (w[k] != 0xFFFFFFFFu) {
      const uint32_t b = 1u << (w[k] & 31);
      if (!(atomicOr(&vis[w[k] >> 5], b) & b)) tm |= 1u << k;
    }
  if (!SPEC) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      vb[k] = ve[k] = 0;
      if (tm & (1u << k)) {
        vb[k] = __ldg(&off[w[k]]);
        ve[k] = __ldg(&off[w[k] + 1]);
      }
    }
  }
  return tm;
}

// A frontier vertex with tau..kHeavyDeg out-edges: the warp walks them with
// K edges per lane in flight.
template <int K>
__device__ __forceinline__ void vgc_direct(const ReachSide& S, uint64_t ub, uint64_t du,
                                           unsigned long long& nedges) {
  const unsigned lane = lane_id();
  const uint64_t ue = ub + du;
  for (uint64_t b = ub; b < ue; b += 32 * K) {
    uint32_t v[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint64_t e = b + k * 32 + lane;
      v[k] = e < ue ? __ldg(&S.E[e]) : 0xFFFFFFFFu;
    }
    uint32_t tm = 0;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (v[k] != 0xFFFFFFFFu && bit_set(S.vis, v[k])) tm |= 1u << k;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (tm & (1u << k)) nedges += S.off[v[k] + 1] - S.off[v[k]];
    warp_append_batch<K>(tm, v, S.qout, &S.ctr->next);
  }
}

// VGC round for up to two sides.  Each warp takes a chunk of up to `chunk`
// frontier vertices (one when the frontier is small, up to 32 when it is much
// larger than the grid, so every warp has work).  Chunk vertices with
// 0 < deg < tau seed a local BFS in a shared-memory queue of tq =
// min(tau, QCAP) entries: each wave takes up to 32 queued vertices and claims
// their neighbours on the bitmap (balanced expansion, K edges per lane in
// flight), keeping claimed vertices in the queue while it has room and
// spilling the rest to the next frontier.  Queued vertices with more than tq
// out-edges, and whatever is left in the queue when it fills or after
// max_waves waves, are spilled too.
// Other chunk vertices are expanded directly (heavy ones by the whole grid).
template <int BLOCK, int QCAP, int K, bool SPEC>
__global__ void __launch_bounds__(BLOCK)
    k_reach_vgc(ReachSide s0, ReachSide s1, uint32_t tau, uint32_t chunk, uint32_t hlim) {
  __shared__ WarpExpandSmem sm[BLOCK / 32];
  __shared__ QEnt sq[BLOCK / 32][QCAP];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint64_t gw = (uint64_t)blockIdx.x * (BLOCK / 32) + wid;
  const uint64_t nw = (uint64_t)gridDim.x * (BLOCK / 32);
  const uint32_t tq = tau < (uint32_t)QCAP ? tau : (uint32_t)QCAP;
  // A round lasts as long as its longest local search.  Searches that stay
  // narrow (a few vertices per wave) stop after max_waves waves and spill
  // their queue, like a full one: on the kNN 10^7 graph waves hold 8 vertices
  // on average, and this cap (56 at tau = 512) cut the first-pivot phase by
  // 12 % at the cost of 7 % more rounds.
  const uint32_t max_waves = tq / 9 > 8 ? tq / 9 : 8;
  uint32_t C = chunk < tq ? chunk : tq;
  C = C < 1 ? 1 : C > 32 ? 32 : C;
  QEnt* Q = sq[wid];
  unsigned long long scanned0 = 0, scanned1 = 0, nedges0 = 0, nedges1 = 0, exp0 = 0, exp1 = 0;
  unsigned long long wv0 = 0, wv1 = 0;  // waves (warp-uniform)
  const uint64_t c0 = (s0.nin + C - 1) / C, c1 = (s1.nin + C - 1) / C;
  for (uint64_t c = gw; c < c0 + c1; c += nw) {
    const int sd = c < c0 ? 0 : 1;
    const ReachSide S = sd ? s1 : s0;
    unsigned long long& nedges = sd ? nedges1 : nedges0;
    const uint64_t first = (sd ? c - c0 : c) * C;
    const uint64_t left = S.nin - first;
    const uint32_t cnt = left < C ? (uint32_t)left : C;
    uint32_t u = 0;
    uint64_t ub = 0, du = 0;
    if (lane < cnt) {
      u = S.qin[first + lane];
      ub = S.off[u];
      du = S.off[u + 1] - ub;
      (sd ? exp1 : exp0)++;
      if (du > hlim) heavy_push(S, u, du);
    }
    uint32_t big = __ballot_sync(kFull, lane < cnt && du >= tq && du <= hlim);
    while (big) {
      const int l = __ffs(big) - 1;
      big &= big - 1;
      const uint64_t bb = __shfl_sync(kFull, ub, l), bd = __shfl_sync(kFull, du, l);
      if (lane == 0) (sd ? scanned1 : scanned0) += bd;
      vgc_direct<K>(S, bb, bd, nedges);
    }
    const bool seed = lane < cnt && du > 0 && du < tq && du <= hlim;
    const uint32_t smask = __ballot_sync(kFull, seed);
    if (seed) Q[__popc(smask & ((1u << lane) - 1))] = QEnt{ub, u, (uint32_t)du};
    const uint32_t nseed = __popc(smask);
    __syncwarp();
    uint32_t head = 0, tail = nseed, nwave = 0;
    while (head < tail && (head == 0 || tail < tq) && nwave++ < max_waves) {
      const uint32_t wave = min(32u, tail - head);
      uint64_t beg = 0;
      uint32_t deg = 0, x = 0, xdeg = 0;
      bool spill_self = false;
      if (lane < wave) {
        const QEnt q = Q[head + lane];
        x = q.v;
        beg = q.beg;
        xdeg = q.deg;
        deg = q.deg;
        if (deg > tq) {
          spill_self = true;
          deg = 0;
        }
        if (head + lane >= nseed) (sd ? exp1 : exp0)++;
      }
      head += wave;
      (sd ? wv1 : wv0)++;
      __syncwarp();
      if (__any_sync(kFull, spill_self)) {
        unsigned long long pos = warp_append(&S.ctr->next, spill_self);
        if (spill_self) {
          S.qout[pos] = x;
          nedges += xdeg;
        }
      }
      (sd ? scanned1 : scanned0) += deg;
      // balanced expansion over the wave's edges, 32*K per batch
      uint32_t incl = deg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += t;
      }
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      sm[wid].excl[lane] = incl - deg;
      sm[wid].beg[lane] = beg;
      __syncwarp();
      for (uint32_t base = 0; base < total; base += 32 * K) {
        uint32_t w[K];
        uint64_t vb[K], ve[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t gi = base + k * 32 + lane;
          w[k] = 0xFFFFFFFFu;
          if (gi < total) {
            const int src = find_src(sm[wid], gi);
            w[k] = __ldg(&S.E[sm[wid].beg[src] + (gi - sm[wid].excl[src])]);
          }
        }
        const uint32_t tm = vgc_claim<K, SPEC>(w, vb, ve, S.off, S.vis);
        vgc_place<K>(tm, w, vb, ve, Q, tail, tq, S.qout, &S.ctr->next, nedges);
      }
    }
    // spill what is left in the queue with one reservation
    const uint32_t rem = tail - head;
    if (rem) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&S.ctr->next, (unsigned long long)rem);
      base = __shfl_sync(kFull, base, 0);
      for (uint32_t k = lane; k < rem; k += 32) {
        const QEnt q = Q[head + k];
        S.qout[base + k] = q.v;
        nedges += q.deg;
      }
    }
    __syncwarp();
  }
  if (lane == 0) {
    if (wv0) atomicAdd(&s0.ctr->waves, wv0);
    if (wv1) atomicAdd(&s1.ctr->waves, wv1);
  }
  flush_side_counters(s0.ctr, s1.ctr, scanned0, scanned1, nedges0, nedges1, exp0, exp1);
}

// ---------------------------------------------------------------------------
// Local searches without rounds.  In rounds of VGC searches every vertex that
// a search spills waits for the round's longest search: on kNN 10^7 a round
// lasted 150 us with a tenth of the warps at work.  Here one launch of the
// resident grid runs the whole sparse part of a search: a warp's local search
// goes on until its queue is empty, gives what it holds beyond kAsyncKeep vertices
// away whenever warps are idle, and an idle warp waits for a vertex, not for a
// round.
//
// Idle warps hold tickets (consecutive indexes drawn from ctl->head) and poll the
// slot of their ticket; givers reserve slots from ctl->tail and write vertex ids
// into them, so a slot has one writer and one reader and needs no lock.  A
// vertex enters the slots at most once while the launch runs (it is claimed once, and
// a ticket's vertices are expanded before any of them could be given away, see
// async_rules.h).  ctl->fin counts the
// vertices taken from the slots whose searches have ended; when it equals
// ctl->tail nothing is queued and nobody works, and whoever sees that marks the
// side done.  Idle warps look at the flags every 16 polls only, so the first one that sees
// the end marks the slots of all tickets (a search of a few vertices 84 -> 66 us).  No warp waits for a block that may not be running: all work is
// held by running warps or lies in the slots.  Every wait is bounded, and any
// condition that this launch should not handle sets a stop bit: warps then
// put their queues into the slots and leave, and the host goes on from
// what was not taken (k_async_collect).  Stop bits: a vertex with more than
// kHeavyDeg out-edges, a backlog that full-width rounds expand faster, the end
// of the prepared slots, a wait that reached its bound.
// ---------------------------------------------------------------------------
constexpr uint32_t kTaken = 0xFFFFFFFEu;  // a slot whose vertex was taken (ids are smaller)
constexpr uint32_t kAsyncDone = 1, kAsyncHeavy = 2, kAsyncWide = 4, kAsyncFull = 8, kAsyncYield = 16;
constexpr uint32_t kAsyncStop = kAsyncHeavy | kAsyncWide | kAsyncFull | kAsyncYield;
constexpr uint32_t kAsyncSpin = 1u << 16;  // polls of one wait: some 50 ms

// Two lines: the flags are polled by idle warps, and every access to one line
// takes its turn in the L2 (with the flags beside head and tail, and polled four
// times as often, a wave took 3,400 cycles instead of 2,050).
struct __align__(128) AsyncCtl {
  uint32_t head, tail, pad0[30];
  uint32_t fin, flags, marked, pad1[29];
};
static_assert(sizeof(AsyncCtl) == 2 * sizeof(Counters), "two counter sets hold it");
// Counter sets of a launch: the control words of both sides, then their counters.
constexpr int kAsyncSet = 4, kAsyncSets = 6;

// The slots of up to two sides (kNone behind the starting frontier), and the counter sets
// from kAsyncSet on: zero, with both sides' control words.  A side without a frontier is done
// from the start.
__global__ void k_async_prepare(const uint32_t* __restrict__ q0, uint32_t nf0, uint32_t* slot0,
                                const uint32_t* __restrict__ q1, uint32_t nf1, uint32_t* slot1,
                                uint32_t slots, Counters* ctr) {
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < slots; i += stride) {
    slot0[i] = i < nf0 ? __ldg(&q0[i]) : kNone;
    if (slot1) slot1[i] = i < nf1 ? __ldg(&q1[i]) : kNone;
  }
  if (blockIdx.x == 0) {
    unsigned long long* z = (unsigned long long*)(ctr + kAsyncSet);
    for (uint32_t i = threadIdx.x; i < kAsyncSets * sizeof(Counters) / 8; i += blockDim.x) z[i] = 0;
    __syncthreads();
    if (threadIdx.x == 0) {
      AsyncCtl* c = (AsyncCtl*)(ctr + kAsyncSet);
      c[0].tail = nf0;
      c[0].flags = nf0 ? 0u : kAsyncDone;
      c[1].tail = nf1;
      c[1].flags = nf1 ? 0u : kAsyncDone;
    }
  }
}

__device__ __forceinline__ uint2 ld_head_tail(const AsyncCtl* c) {
  uint2 x;
  asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];"
               : "=r"(x.x), "=r"(x.y)
               : "l"(&c->head)
               : "memory");
  return x;
}
__device__ __forceinline__ uint32_t ld_flags(const AsyncCtl* c) {
  return *(const volatile uint32_t*)&c->flags;
}

// One warp's part in the hand-over of vertices on one side.
struct AsyncLink {
  AsyncCtl* C;
  AsyncCtl *c0, *c1;  // both sides: a stop is for both
  volatile uint32_t* slot;
  uint32_t slots, nw;  // prepared slots; warps of the grid
  uint32_t most;       // vertices that a warp takes at a time

  __device__ void stop(uint32_t why) const {
    atomicOr(&c0->flags, why);
    atomicOr(&c1->flags, why);
  }

  // The warp's search has ended (`items` vertices taken for it): accounts for
  // them, then waits for vertices.  Returns the mask of lanes that got one (v),
  // or 0 with *fl = the flags that ended the wait.  tk: the lane's ticket.
  __device__ __forceinline__ unsigned wait(uint32_t items, bool quit, uint32_t& tk, uint32_t& v,
                                           uint32_t* flags) const {
    const unsigned lane = lane_id();
    if (items && lane == 0) {
      const uint32_t f = atomicAdd(&C->fin, items) + items;
      __threadfence();
      if (f == *(volatile uint32_t*)&C->tail) atomicOr(&C->flags, kAsyncDone);
    }
    const bool none = !__any_sync(kFull, tk != kNone);
    uint32_t first = 0, take = 0, fl = 0;
    if (lane == 0) {
      const uint2 c = ld_head_tail(C);
      fl = quit ? kAsyncHeavy : ld_flags(C);
      if (!fl && none) {
        take = async_take((int32_t)(c.y - c.x), nw, most);
        first = atomicAdd(&C->head, take);
      }
    }
    fl = __shfl_sync(kFull, fl, 0);
    first = __shfl_sync(kFull, first, 0);
    take = __shfl_sync(kFull, take, 0);
    if (lane < take) tk = first + lane;
    v = kNone;
    unsigned got = 0;
    // (the tickets' own looks at the flags, 16 polls apart, do not fall together)
    for (uint32_t spin = 1 + (first & 15u); !fl; spin++) {
      if (tk != kNone && tk < slots) v = slot[tk];
      got = __ballot_sync(kFull, v != kNone);
      if (got) break;
      if ((spin & 15u) == 0) {
        if (lane == 0) {
          fl = ld_flags(C);
          if (!fl && spin >= kAsyncSpin) {
            stop(kAsyncYield);
            fl = kAsyncYield;
          }
        }
        fl = __shfl_sync(kFull, fl, 0);
      } else {
        __nanosleep(spin < 64 ? 100 : 400);
      }
    }
    if (got) got = __ballot_sync(kFull, v < kTaken);  // (none: the mark of a side that is done)
    if (fl == kAsyncDone) {
      // the first to see it marks the slots of all tickets, for the others
      uint32_t end = 0;
      if (lane == 0 && atomicExch(&C->marked, 1u) == 0) end = min(*(volatile uint32_t*)&C->head, slots);
      end = __shfl_sync(kFull, end, 0);
      for (uint32_t i = *(volatile uint32_t*)&C->tail + lane; i < end; i += 32) slot[i] = kTaken;
    }
    if (v < kTaken) {
      slot[tk] = kTaken;
      tk = kNone;
    }
    *flags = fl;
    return got;
  }

  // Reserves n slots (lane 0's atomic); the result is the same in all lanes.
  __device__ __forceinline__ uint32_t reserve(uint32_t n) const {
    uint32_t pos = 0;
    if (lane_id() == 0) {
      pos = atomicAdd(&C->tail, n);
      if (pos + n > slots) stop(kAsyncFull);
    }
    return __shfl_sync(kFull, pos, 0);
  }

  // How many of the `held` queued vertices to give to idle warps, from a look
  // at head and tail.
  __device__ __forceinline__ uint32_t share(const uint2& ht, uint32_t held,
                                            uint32_t backlog_max) const {
    const int32_t hungry = (int32_t)(ht.x - ht.y);
    if (hungry < 0 && (uint32_t)-hungry > backlog_max && lane_id() == 0) stop(kAsyncWide);
    return async_give(hungry, held);
  }

  // Puts the last n of the ring's vertices (places [t - n, t)) into the slots.
  __device__ __forceinline__ void put(const uint32_t* V, uint32_t mask, uint32_t& t,
                                      uint32_t n) const {
    const uint32_t pos = reserve(n);
    t -= n;
    for (uint32_t i = lane_id(); i < n; i += 32) slot[pos + i] = V[(t + i) & mask];
    __syncwarp();
  }
};

// Of every wave: `look` reads head and tail when there may be something to give
// away, `check` the stop bits now and then.  Both are used only under the same
// (warp-uniform) conditions, so that nothing waits for them before the end.
constexpr uint32_t kAsyncLook = kAsyncKeep - 4;

// Any degrees: balanced expansion over up to 32 queued vertices per wave, K
// edges per lane in flight; while the queued vertices have at most 8 out-edges,
// eight lanes per vertex and 16 vertices per wave, which needs neither the prefix
// sum nor the search (batch of 256 graphs, 3.3e6 vertices in this launch: SCC 3.49
// -> 3.30 ms).  S.qout holds the slots; the first `slots` of them
// are prepared (kNone or the starting frontier).
template <int BLOCK, int QCAP, int K>
__global__ void __launch_bounds__(BLOCK)
    k_reach_async(ReachSide s0, ReachSide s1, AsyncCtl* c0, AsyncCtl* c1, uint32_t slots,
                  uint32_t backlog_max) {
  static_assert((QCAP & (QCAP - 1)) == 0, "ring queue");
  __shared__ WarpExpandSmem ssm[BLOCK / 32];
  __shared__ uint64_t shdr[BLOCK / 32][QCAP];  // adj_hdr of a queued vertex
  __shared__ uint32_t sv[BLOCK / 32][QCAP];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint32_t gw = blockIdx.x * (BLOCK / 32) + wid;
  WarpExpandSmem& sm = ssm[wid];
  uint64_t* H = shdr[wid];
  uint32_t* V = sv[wid];
  unsigned long long edges[2] = {0, 0}, expanded[2] = {0, 0};
  bool leave = false;
  for (int turn = 0; turn < 2 && !leave; turn++) {
    const int sd = (int)((gw + turn) & 1);
    const uint64_t* __restrict__ off = sd ? s1.off : s0.off;
    const uint32_t* __restrict__ E = sd ? s1.E : s0.E;
    uint32_t* vis = sd ? s1.vis : s0.vis;
    const AsyncLink L{sd ? c1 : c0, c0, c1, sd ? s1.qout : s0.qout, slots,
                      (uint32_t)(gridDim.x * (BLOCK / 32)), kAsyncTake};
    uint32_t tk = kNone;               // this lane's ticket
    uint32_t h = 0, t = 0, items = 0;  // ring queue [h, t); vertices taken for this search
    unsigned long long ed = 0, ex = 0;
    bool quit = false;  // this warp met a heavy vertex
    uint32_t nwave = 0;
    for (;;) {
      if (h == t) {
        uint32_t v, fl;
        const unsigned got = L.wait(items, quit, tk, v, &fl);
        if (!got) {
          leave = (fl & kAsyncStop) != 0;  // stopped: all sides; done: the other side is next
          break;
        }
        if (v != kNone) {
          const uint32_t at = __popc(got & ((1u << lane) - 1u));
          V[at] = v;
          H[at] = adj_hdr(__ldg(&off[v]), __ldg(&off[v + 1]));
        }
        items = __popc(got);
        h = 0;
        t = items;
        __syncwarp();
      }
      uint32_t wave = min(32u, t - h);
      const bool look = t - h > kAsyncLook, check = (++nwave & 7u) == 0;
      uint2 ht;
      uint32_t flags;
      if (look) ht = ld_head_tail(L.C);
      if (check) flags = ld_flags(L.C);
      uint64_t beg = 0;
      uint32_t deg = 0, x = 0;
      if (lane < wave) {
        const uint64_t r = H[(h + lane) & (QCAP - 1)];
        x = V[(h + lane) & (QCAP - 1)];
        beg = r >> 24;
        deg = (uint32_t)(r & 0xFFFFFFull);
      }
      const uint32_t h0 = h;
      const bool few = !__any_sync(kFull, deg > 8);
      if (few) wave = min(wave, kAsyncFewWave);
      h += wave;
      // Claims the lane's candidates w[0 .. N) (steps from lim on have none), their
      // ranges loaded alongside, and queues the new ones.
      auto claim = [&](const uint32_t* w, uint32_t lim, auto nn) {
        constexpr int N = decltype(nn)::value;
        uint32_t old[N];
        uint64_t r[N];
        unsigned m[N];
        uint32_t tot = 0;
#pragma unroll
        for (int k = 0; k < N; k++) {
          old[k] = ~0u;
          r[k] = 0;
          if ((uint32_t)k < lim && w[k] != kNone) {
            old[k] = atomicOr(&vis[w[k] >> 5], 1u << (w[k] & 31));
            r[k] = adj_hdr(__ldg(&off[w[k]]), __ldg(&off[w[k] + 1]));
          }
        }
        // a vertex without out-edges is done once it is claimed
#pragma unroll
        for (int k = 0; k < N; k++) {
          m[k] = __ballot_sync(kFull, !((old[k] >> (w[k] & 31)) & 1u) && (r[k] & 0xFFFFFFull));
          tot += __popc(m[k]);
        }
        if (tot == 0) return;
        const uint32_t room = QCAP - (t - h);
        const uint32_t nloc = tot < room ? tot : room;
        uint32_t spill = 0;
        if (tot > nloc) spill = L.reserve(tot - nloc);
        uint32_t b = 0;
#pragma unroll
        for (int k = 0; k < N; k++) {
          if ((m[k] >> lane) & 1u) {
            const uint32_t at = b + __popc(m[k] & ((1u << lane) - 1u));
            if (at < nloc) {
              H[(t + at) & (QCAP - 1)] = r[k];
              V[(t + at) & (QCAP - 1)] = w[k];
            } else {
              L.slot[spill + (at - nloc)] = w[k];
            }
          }
          b += __popc(m[k]);
        }
        t += nloc;
        __syncwarp();
      };
      if (few) {
        // eight lanes per entry, lane j takes its target j (no scan, no search)
        const unsigned grp = lane >> 3, j = lane & 7;
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const uint32_t i = 4 * k + grp;
          const uint64_t r = i < wave ? H[(h0 + i) & (QCAP - 1)] : 0ull;
          w[k] = j < (r & 0xFFFFFFull) ? __ldg(&E[(r >> 24) + j]) : kNone;
        }
        if (lane < wave) {
          ex++;
          ed += deg;
        }
        __syncwarp();  // the entries are read: their places may be written
        claim(w, 4u, std::integral_constant<int, 4>());
      } else {
        ex += lane < wave;
        const bool big = deg > kHeavyDeg;
        if (__any_sync(kFull, big)) {  // not for this launch: back to the slots
          quit = true;  // (so a warp puts back at most what it took, see kAsyncSlack)
          if (big) {
            L.slot[atomicAdd(&L.C->tail, 1u)] = x;
            deg = 0;
            L.stop(kAsyncHeavy);
          }
        }
        ed += deg;
        uint32_t incl = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(kFull, incl, o);
          if ((int)lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        __syncwarp();
        sm.excl[lane] = incl - deg;
        sm.beg[lane] = beg;
        __syncwarp();
        for (uint32_t base = 0; base < total; base += 32 * K) {
          uint32_t w[K];
#pragma unroll
          for (int k = 0; k < K; k++) {
            w[k] = kNone;
            if (base + k * 32 < total) {
              const uint32_t gi = base + k * 32 + lane;
              if (gi < total) {
                const int src = find_src(sm, gi);
                w[k] = __ldg(&E[sm.beg[src] + (gi - sm.excl[src])]);
              }
            }
          }
          claim(w, (total - base + 31) / 32, std::integral_constant<int, K>());
        }
      }
      if (look) {
        const uint32_t give = L.share(ht, t - h, backlog_max);
        if (give) L.put(V, QCAP - 1, t, give);
      }
      if ((quit || (check && (flags & kAsyncStop))) && t != h) L.put(V, QCAP - 1, t, t - h);
    }
    edges[sd] = ed;
    expanded[sd] = ex;
  }
  flush_side_counters(s0.ctr, s1.ctr, edges[0], edges[1], 0, 0, expanded[0], expanded[1]);
}

// Low degrees, with records: the queue holds the records themselves, so a
// wave's targets are in shared memory and its only trip is the claim (a record
// comes with it, one 256-bit load).  What is left is the warp's own work, which
// took more than the trip (2,100 of 3,500 cycles a wave on the grid) when the
// edges were spread over the lanes by a scan and a search: here eight lanes
// belong to an entry, lane j to its target j, four entries per step and up to
// kLowWave per wave, and new vertices are placed by ballots.  A vertex with more
// than kRecEdges targets comes back to the front of the queue with its next
// ones, which its lanes load during the wave (at most kLowWave such entries,
// which are never given away: kAsyncKeep stay).
// A wave holds 6 to 8 entries on average, so there is code for 4, 8 and 12 of them.
// Reach of the first pivot (both sides): kNN 10^7 (depth about 3,700) in rounds
// 10.1 ms, k_reach_async 8.6, this 4.3 (always 12 entries 4.5, 8 or 12 4.8, 4 or 12
// 4.5); 4096^2 grid 8.2, 7.8, 4.2 (4.2, 4.7, 4.4).  Waves of 8 / 12 /
// 16 entries: 4.6 / 4.5 / 4.9 ms on kNN; kAsyncKeep 12 / 16 / 20: 4.5 / 4.5 / 4.7;
// 1 / 2 / 3 / 5 blocks per SM: 5.9 / 5.0 / 4.9 / 5.0 (waves of 16), so three.
template <int BLOCK, int QCAP>
__global__ void __launch_bounds__(BLOCK)
    k_reach_async_low(ReachSide s0, ReachSide s1, AsyncCtl* c0, AsyncCtl* c1, uint32_t slots,
                      uint32_t backlog_max) {
  static_assert((QCAP & (QCAP - 1)) == 0 && QCAP >= 64, "ring queue");
  __shared__ uint4 srec[BLOCK / 32][QCAP][2];
  __shared__ uint32_t sv[BLOCK / 32][QCAP];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const unsigned grp = lane >> 3, j = lane & 7, lt = (1u << lane) - 1u;
  const uint32_t gw = blockIdx.x * (BLOCK / 32) + wid;
  uint4(*R)[2] = srec[wid];
  uint32_t* V = sv[wid];
  unsigned long long edges[2] = {0, 0}, expanded[2] = {0, 0};
  bool leave = false;
  for (int turn = 0; turn < 2 && !leave; turn++) {
    const int sd = (int)((gw + turn) & 1);
    const VRec* __restrict__ rec = sd ? s1.rec : s0.rec;
    const uint32_t* __restrict__ E = sd ? s1.E : s0.E;
    uint32_t* vis = sd ? s1.vis : s0.vis;
    const AsyncLink L{sd ? c1 : c0, c0, c1, sd ? s1.qout : s0.qout, slots,
                      (uint32_t)(gridDim.x * (BLOCK / 32)), kAsyncTakeLow};
    uint32_t tk = kNone;               // this lane's ticket
    uint32_t h = 0, t = 0, items = 0;  // ring queue [h, t); vertices taken for this search
    uint32_t ed = 0;
    unsigned long long ex = 0;
    uint32_t nwave = 0;
    for (;;) {
      if (h == t) {
        edges[sd] += ed;
        ed = 0;
        uint32_t v, fl;
        const unsigned got = L.wait(items, false, tk, v, &fl);
        if (!got) {
          leave = (fl & kAsyncStop) != 0;  // stopped: all sides; done: the other side is next
          break;
        }
        if (v != kNone) {
          const uint32_t at = (h + __popc(got & lt)) & (QCAP - 1);
          V[at] = v;
          ld_rec(rec + v, R[at][0], R[at][1]);
        }
        items = __popc(got);
        t = h + items;
        ex += lane == 0 ? items : 0;
        __syncwarp();
      }
      const uint32_t n = min((uint32_t)kLowWave, t - h);
      const bool look = t - h > kAsyncLook, check = (++nwave & 7u) == 0;
      uint2 ht;
      uint32_t flags;
      if (look) ht = ld_head_tail(L.C);
      if (check) flags = ld_flags(L.C);
      auto step = [&](auto kk) {
        constexpr int K = decltype(kk)::value;
        // target j of entry 4 k + grp, and the one kRecEdges further on
        uint32_t w[K], old[K], nx[K], lo[K], more = 0;
        uint4 ra[K], rb[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t* word = (const uint32_t*)&R[(h + 4 * k + grp) & (QCAP - 1)][0];
          lo[k] = word[0];
          w[k] = word[2 + (j < (unsigned)kRecEdges ? j : 0)];
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t deg = 4 * k + grp < n ? lo[k] & 0xFFFFFFu : 0u;
          if (j >= (unsigned)kRecEdges || j >= deg) w[k] = kNone;
          more |= (deg > (uint32_t)kRecEdges ? 1u : 0u) << k;
        }
        const bool any_more = __any_sync(kFull, more);
        if (any_more) {
#pragma unroll
          for (int k = 0; k < K; k++) {
            const uint64_t beg =
                ((uint64_t)((const uint32_t*)&R[(h + 4 * k + grp) & (QCAP - 1)][0])[1] << 8) | (lo[k] >> 24);
            nx[k] = kNone;
            if (((more >> k) & 1u) && j < (unsigned)kRecEdges && kRecEdges + j < (lo[k] & 0xFFFFFFu))
              nx[k] = __ldg(&E[beg + kRecEdges + j]);
          }
        }
        // the claims, with the candidates' records
#pragma unroll
        for (int k = 0; k < K; k++) {
          old[k] = ~0u;
          ra[k].x = 0;
          if (w[k] != kNone) {
            old[k] = atomicOr(&vis[w[k] >> 5], 1u << (w[k] & 31));
            ld_rec(rec + w[k], ra[k], rb[k]);
            ed++;
          }
        }
        // place the claimed ones (a vertex without out-edges is done)
        unsigned m[K];
        uint32_t tot = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
          m[k] = __ballot_sync(kFull, !((old[k] >> (w[k] & 31)) & 1u) && (ra[k].x & 0xFFFFFFu));
          tot += __popc(m[k]);
        }
        const uint32_t room = QCAP - (t - h);
        const uint32_t nloc = min(tot, room);
        uint32_t at = t;
#pragma unroll
        for (int k = 0; k < K; k++) {
          const uint32_t q = at + __popc(m[k] & lt);
          if (((m[k] >> lane) & 1u) && q - t < nloc) {
            R[q & (QCAP - 1)][0] = ra[k];
            R[q & (QCAP - 1)][1] = rb[k];
            V[q & (QCAP - 1)] = w[k];
          }
          at += __popc(m[k]);
        }
        if (tot > nloc) {  // a full queue: the rest goes to the slots
          const uint32_t spill = L.reserve(tot - nloc);
          at = t;
#pragma unroll
          for (int k = 0; k < K; k++) {
            const uint32_t q = at + __popc(m[k] & lt) - t;
            if (((m[k] >> lane) & 1u) && q >= nloc) L.slot[spill + (q - nloc)] = w[k];
            at += __popc(m[k]);
          }
        }
        t += nloc;
        if (lane == 0) ex += nloc;
        // entries with targets left return to the front, in the places just read
        const uint32_t h0 = h;
        h += n;
        if (any_more) {
#pragma unroll
          for (int k = K - 1; k >= 0; k--) {
            const unsigned back = __ballot_sync(kFull, j == 0 && ((more >> k) & 1u));
            if (back) {
              // the group's own entry moves from place 4 k + grp to place (h - 1 - later ones)
              const bool mv = (more >> k) & 1u;
              const uint32_t from = (h0 + 4 * k + grp) & (QCAP - 1);
              const uint32_t to = (h - 1 - __popc(back >> (8 * grp + 1))) & (QCAP - 1);
              uint32_t lo = 0, hi = 0, x = 0;
              if (mv && j == 0) {
                const uint2 hd = *(const uint2*)&R[from][0];
                lo = hd.x;
                hi = hd.y;
                x = V[from];
              }
              __syncwarp();
              if (mv) {
                uint32_t* word = (uint32_t*)&R[to][0];
                if (j < (unsigned)kRecEdges) word[2 + j] = nx[k];
                if (j == 0) {
                  const uint64_t r = ((((uint64_t)hi << 32) | lo) + ((uint64_t)kRecEdges << 24)) - kRecEdges;
                  word[0] = (uint32_t)r;
                  word[1] = (uint32_t)(r >> 32);
                  V[to] = x;
                }
              }
              __syncwarp();
              h -= __popc(back);
            }
          }
        }
        __syncwarp();
      };
      if (n <= 4)
        step(std::integral_constant<int, 1>());
      else if (n <= 8)
        step(std::integral_constant<int, 2>());
      else
        step(std::integral_constant<int, kLowWave / 4>());
      if (look) {
        const uint32_t give = L.share(ht, t - h, backlog_max);
        if (give) L.put(V, QCAP - 1, t, give);
      }
      if (check && (flags & kAsyncStop) && t != h) L.put(V, QCAP - 1, t, t - h);
    }
    edges[sd] += ed;
    expanded[sd] = ex;
  }
  flush_side_counters(s0.ctr, s1.ctr, edges[0], edges[1], 0, 0, expanded[0], expanded[1]);
}

// What a stopped launch left in the slots becomes the frontier (ctr->next,
// ctr->next_edges): vertices not taken, and all those behind the prepared slots.
__global__ void k_async_collect(const uint32_t* __restrict__ slot, const AsyncCtl* C, uint32_t slots,
                                const uint64_t* __restrict__ off, uint32_t* q, Counters* ctr) {
  if (C->fin == C->tail) return;
  const uint64_t total = C->tail;
  unsigned long long e = 0;
  for (uint64_t base = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; base < total;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = base + lane_id();
    const uint32_t v = i < total ? slot[i] : kNone;
    const bool left = v < kTaken;
    const unsigned long long pos = warp_append(&ctr->next, left);
    if (left) {
      q[pos] = v;
      e += off[v + 1] - off[v];
    }
  }
  e = warp_sum(e);
  if (lane_id() == 0 && e) atomicAdd(&ctr->next_edges, e);
}

// Heavy vertices of both sides: the chunks of a side's heavy list are cut
// into one contiguous range per warp; a warp finds the entry of its first
// chunk once, then claims kHeavyChunk edges per step (every entry has a
// chunk, so the next entry is at most one step away).  What a warp claims
// collects in shared memory and goes to the next frontier kHeavyBuf / 2 and more
// vertices at a time: one reservation per chunk was an atomic on the same word
// every 3 ns, and the chunks waited for it.
// R-MAT 2^26, 1.7e7 edges of both sides: 443 -> 225 us (8 instead of 4 edges in flight
// per lane without the buffer 325; with it, 4 or 8 edges and 512 or 1,024 entries
// 220 to 229; 16 edges 300).
constexpr uint32_t kHeavyBuf = 512;
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_reach_heavy(ReachSide s0, ReachSide s1) {
  __shared__ uint32_t bufs[BLOCK / 32][kHeavyBuf];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  uint32_t* buf = bufs[wid];
  const uint64_t gw = (uint64_t)blockIdx.x * (BLOCK / 32) + wid;
  const uint64_t nw = (uint64_t)gridDim.x * (BLOCK / 32);
#pragma unroll 1
  for (int sd = 0; sd < 2; sd++) {
    const ReachSide S = sd ? s1 : s0;
    if (!S.ctr) continue;
    const unsigned long long packed = S.ctr->heavy;
    const uint64_t nh = packed >> kPackShift, total = packed & kPackMask;
    const uint64_t per = (total + nw - 1) / nw;
    const uint64_t c_beg = gw * per, c_end = c_beg + per < total ? c_beg + per : total;
    if (nh == 0 || c_beg >= c_end) continue;
    uint64_t h = 0, hi = nh - 1;  // last entry whose first chunk is <= c_beg
    while (h < hi) {
      const uint64_t mid = (h + hi + 1) >> 1;
      if ((uint32_t)__ldg(&S.heavy[mid]) <= c_beg)
        h = mid;
      else
        hi = mid - 1;
    }
    uint64_t ent = __ldg(&S.heavy[h]);
    uint64_t cs = (uint32_t)ent, cn = h + 1 < nh ? (uint32_t)__ldg(&S.heavy[h + 1]) : total;
    uint64_t beg = S.off[ent >> 32], end = S.off[(ent >> 32) + 1];
    unsigned long long scanned = 0, next_edges = 0;
    uint32_t held = 0;  // claimed vertices in buf (warp-uniform)
    auto flush = [&] {
      __syncwarp();
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&S.ctr->next, (unsigned long long)held);
      base = __shfl_sync(kFull, base, 0);
#pragma unroll 4
      for (uint32_t i = lane; i < held; i += 32) {
        const uint32_t v = buf[i];
        S.qout[base + i] = v;
        next_edges += S.off[v + 1] - S.off[v];
      }
      __syncwarp();
      held = 0;
    };
    for (uint64_t c = c_beg; c < c_end; c++) {
      if (c >= cn) {
        h++;
        ent = __ldg(&S.heavy[h]);
        cs = cn;
        cn = h + 1 < nh ? (uint32_t)__ldg(&S.heavy[h + 1]) : total;
        beg = S.off[ent >> 32];
        end = S.off[(ent >> 32) + 1];
      }
      const uint64_t e0 = beg + (c - cs) * kHeavyChunk;
      uint32_t v[kHeavyK], tm = 0;
#pragma unroll
      for (int k = 0; k < kHeavyK; k++) {
        const uint64_t e = e0 + k * 32 + lane;
        v[k] = 0;
        if (e < end) {
          scanned++;
          v[k] = __ldg(&S.E[e]);
        }
      }
#pragma unroll
      for (int k = 0; k < kHeavyK; k++)
        if (e0 + k * 32 + lane < end && bit_set(S.vis, v[k])) tm |= 1u << k;
#pragma unroll
      for (int k = 0; k < kHeavyK; k++) {
        const uint32_t mk = __ballot_sync(kFull, (tm >> k) & 1u);
        if ((tm >> k) & 1u) buf[held + __popc(mk & ((1u << lane) - 1u))] = v[k];
        held += __popc(mk);
      }
      if (held > kHeavyBuf - kHeavyChunk) flush();
    }
    if (held) flush();
    scanned = warp_sum(scanned);
    next_edges = warp_sum(next_edges);
    if (lane == 0) {
      if (scanned) atomicAdd(&S.ctr->heavy_edges, scanned);
      if (next_edges) atomicAdd(&S.ctr->next_edges, next_edges);
    }
  }
}

// Pull round: B_* is the reverse direction of the search.  A warp takes `wps` words
// of the visited bitmap (at most 32, one per lane), lists the vertices that are
// neither visited nor dead in shared memory, and scans the in-lists of the listed
// ones for a frontier vertex, 32 * kPullB vertices at a time: the ranges of all, the
// first in-edges of all, their frontier bits (dense rounds often hit at once), then
// each vertex alone up to kPullSolo in-edges, kPullP in flight, then the long
// in-lists left over by the whole warp, 32 * kPullP edges per step, until a hit.
//
// What bounds it: four dependent trips to memory per step (words, range, first
// in-edge, frontier bit).  Without the list a lane owned a fixed vertex, two thirds
// of the lanes of a first pull round on R-MAT 2^26 and 98 % of a second had nothing
// to do, and the steps were as many as the bitmap has words.
// R-MAT 2^26 (6.7e7 vertices, 6.1e8 edges), per side: first pull 480 -> 330 us (tiles
// staged by bulk copies before), second 315 -> 65 us.  SCC 5.02 -> 4.15 ms.
// dead (optional): bitmap of vertices without in-edges in this direction, which no
// pull can reach; they keep their visited bit clear, and still count as unvisited
// (the work of the reference's dense round).  The next round's out-edge count is
// left to k_pull_out_edges, off this chain.
// (vertices per lane and blocks an SM, SCC of R-MAT 2^26 / load and SCC of 2^22: 2 and
// 6 4.12 / 4.90 ms, 4 and 4 4.11 / 4.94, 8 and 4 4.48 / 5.11; scanning a lane's
// vertices together instead of one after the other 4.26 / 4.97)
constexpr int kPullB = 2;

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1536 / BLOCK)
    k_reach_pull(const uint64_t* __restrict__ B_off, const uint32_t* __restrict__ B_E,
                 const uint32_t* __restrict__ fb_in, uint32_t* vis, uint32_t* fb_out, uint64_t n,
                 Counters* ctr, const uint32_t* __restrict__ dead, uint32_t wps) {
  constexpr int B = kPullB;
  __shared__ uint16_t lists[BLOCK / 32][1024];
  __shared__ uint32_t founds[BLOCK / 32][32];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  uint16_t* list = lists[wid];
  uint32_t* found = founds[wid];
  const uint64_t gw = (uint64_t)blockIdx.x * (BLOCK / 32) + wid;
  const uint64_t nw = (uint64_t)gridDim.x * (BLOCK / 32);
  const uint64_t nwords = (n + 31) >> 5;
  unsigned long long cnt = 0, scanned = 0, unvisited = 0;
  for (uint64_t base = gw * wps; base < nwords; base += nw * wps) {
    const uint64_t w = base + lane;
    const bool mine = lane < wps && w < nwords;
    const uint32_t vw = mine ? vis[w] : ~0u;
    const uint32_t dw = mine && dead ? __ldg(&dead[w]) : 0u;
    uint32_t un = ~vw;
    if (mine && w * 32 + 32 > n) un &= (1u << (n & 31)) - 1u;
    unvisited += __popc(un);
    uint32_t live = un & ~dw;
    const uint32_t c = __popc(live);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, o);
      if ((int)lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    if (total == 0) {
      if (mine) fb_out[w] = 0;
      continue;
    }
    found[lane] = 0;
    for (uint32_t r = incl - c; live; live &= live - 1)
      list[r++] = (uint16_t)(lane * 32 + (__ffs(live) - 1));
    __syncwarp();
    const uint64_t v0 = base * 32;
    for (uint32_t i0 = 0; i0 < total; i0 += 32 * B) {
      uint32_t li[B], x[B];
      uint64_t j[B], e[B], lim[B];
      bool f[B];
#pragma unroll
      for (int k = 0; k < B; k++) {
        const uint32_t i = i0 + k * 32 + lane;
        li[k] = i < total ? list[i] : 0u;
        j[k] = e[k] = 0;
        if (i < total) {
          j[k] = __ldg(&B_off[v0 + li[k]]);
          e[k] = __ldg(&B_off[v0 + li[k] + 1]);
        }
        scanned -= j[k];
      }
#pragma unroll
      for (int k = 0; k < B; k++) {
        lim[k] = e[k] < j[k] + kPullSolo ? e[k] : j[k] + kPullSolo;
        x[k] = j[k] < lim[k] ? __ldg(&B_E[j[k]]) : kNone;
      }
#pragma unroll
      for (int k = 0; k < B; k++) {
        f[k] = x[k] != kNone && fb_test(fb_in, x[k]);
        if (j[k] < lim[k]) j[k]++;
      }
#pragma unroll
      for (int k = 0; k < B; k++)
        if (!f[k]) f[k] = pull_scan(B_E, fb_in, j[k], lim[k]);
#pragma unroll
      for (int k = 0; k < B; k++) scanned += j[k];
#pragma unroll
      for (int k = 0; k < B; k++) {
        pull_long(B_E, fb_in, __ballot_sync(kFull, !f[k] && j[k] < e[k]), j[k], e[k], f[k], scanned);
        if (f[k]) atomicOr(&found[li[k] >> 5], 1u << (li[k] & 31));
      }
    }
    __syncwarp();
    if (mine) {
      const uint32_t fw = found[lane];
      fb_out[w] = fw;
      if (fw) vis[w] = vw | fw;
      cnt += __popc(fw);
    }
    __syncwarp();
  }
  cnt = warp_sum(cnt);
  scanned = warp_sum(scanned);
  unvisited = warp_sum(unvisited);
  if (lane == 0) {
    if (cnt) atomicAdd(&ctr->next, cnt);
    if (scanned) atomicAdd(&ctr->edges, scanned);
    if (unvisited) atomicAdd(&ctr->unvisited, unvisited);
  }
}

// A pull round on the resident blocks of the kernel, words per warp step as many
// as give every warp two steps (4 to 32); 4 in a batch of graphs, where the hubs of
// every member lie side by side, and those of a member whose pivot missed its large component
// are scanned whole, by one warp with 32 words (first pivots of 512 graphs 6.9 ms with 32, 5.6
// with 4; one graph, R-MAT 2^26: 3.54 ms of SCC with 32, 3.77 with 8, 4.26 with 4).
template <int BLOCK>
static void launch_pull(int num_sms, cudaStream_t st, const uint64_t* B_off, const uint32_t* B_E,
                        const uint32_t* fb_in, uint32_t* vis, uint32_t* fb_out, uint64_t n,
                        Counters* ctr, const uint32_t* dead, bool batch = false) {
  static int per_sm = [] {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_reach_pull<BLOCK>, BLOCK, 0) !=
            cudaSuccess ||
        b < 1) {
      cudaGetLastError();
      b = 1;
    }
    return b;
  }();
  const uint64_t nwords = (n + 31) / 32, cap = (uint64_t)num_sms * per_sm;
  uint32_t wps = batch ? 4 : 32;
  while (wps > 4 && nwords < 2 * cap * (BLOCK / 32) * wps) wps /= 2;
  const uint64_t want = (nwords + wps * (BLOCK / 32) - 1) / (wps * (BLOCK / 32));
  k_reach_pull<BLOCK><<<(unsigned)std::max<uint64_t>(1, std::min(want, cap)), BLOCK, 0, st>>>(
      B_off, B_E, fb_in, vis, fb_out, n, ctr, dead, wps);
}

constexpr uint64_t kPullExactBelow = 1u << 14;
constexpr uint32_t kSampleProbes = 32 * 64;
constexpr uint32_t kSampleHits = 50;
constexpr int kSampleK = 8;  // probes per lane in flight (70 -> 29 us when 2 % are hits)
static_assert(kSampleProbes % (32 * kSampleK) == 0, "whole batches");

__global__ void k_pull_out_edges(const uint32_t* __restrict__ fb, const uint64_t* __restrict__ A_off,
                                 uint64_t n, uint32_t seed, Counters* ctr) {
  const unsigned lane = lane_id();
  const uint64_t nf = *(volatile unsigned long long*)&ctr->next;
  if (nf < kPullExactBelow) {
    const uint64_t nwords = (n + 31) >> 5;
    unsigned long long sum = 0;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nwords;
         w += (uint64_t)gridDim.x * blockDim.x) {
      uint32_t word = fb[w];
      while (word) {
        const uint64_t v = w * 32 + (__ffs(word) - 1);
        word &= word - 1;
        sum += A_off[v + 1] - A_off[v];
      }
    }
    sum = warp_sum(sum);
    if (lane == 0 && sum) atomicAdd(&ctr->next_edges, sum);
    return;
  }
  if (blockIdx.x != 0 || threadIdx.x >= 32) return;
  unsigned long long sum = 0;
  uint32_t hits = 0;
  for (uint32_t base = 1; base <= kSampleProbes && hits < kSampleHits; base += 32 * kSampleK) {
    uint32_t idx[kSampleK], word[kSampleK];
#pragma unroll
    for (int k = 0; k < kSampleK; k++) {
      idx[k] = (uint32_t)(hash32(seed + base + k * 32 + lane) % n);
      word[k] = __ldg(&fb[idx[k] >> 5]);
    }
#pragma unroll
    for (int k = 0; k < kSampleK; k++) {
      const bool hit = (word[k] >> (idx[k] & 31)) & 1u;
      const uint32_t m = __ballot_sync(kFull, hit);
      const uint32_t rank = __popc(m & ((1u << lane) - 1));
      if (hit && hits + rank < kSampleHits) sum += A_off[idx[k] + 1] - A_off[idx[k]];
      hits += __popc(m);
    }
  }
  sum = warp_sum(sum);
  if (hits > kSampleHits) hits = kSampleHits;
  if (lane == 0) ctr->next_edges = hits ? nf * (sum / hits) : 0;
}

// ---------------------------------------------------------------------------
// Resident rounds, for graphs of up to kRrMaxEdges edges.  A round is 5 to 40 us of
// work, and launched from the host about 30 more (a
// memset, one to three kernels, a read-back, a wait, twice that for heavy
// vertices).  k_reach_rounds runs push and pull rounds of both sides back to
// back on a resident grid, one grid barrier per round (two when heavy vertices
// were listed).  Every round leaves its frontier as a queue and as a bitmap, so a
// change between push and pull needs no conversion: three bitmaps rotate (read,
// written, cleared).  The switch is the host loop's, with exact out-edge counts.
// First-pivot phase, host rounds -> this: R-MAT 2^12 0.26 -> 0.12 ms, 2^16 0.34 ->
// 0.17, 2^18 0.46 -> 0.20, 2^20 (1.6e7 edges) 0.47 -> 0.32, 2^21 (3.2e7) 0.56 ->
// 0.43, 64-graph batch 0.90 -> 0.67; 3x10^6 vertices with 1.2e7 edges 0.73 -> 0.71.
// ---------------------------------------------------------------------------
constexpr int kRrThreads = 512;
constexpr int kRrWarps = kRrThreads / 32;
constexpr uint64_t kRrHeavy = 256;        // out-edges of a vertex left to the grid
constexpr uint64_t kRrMaxEdges = 1 << 25;  // larger graphs: full-width rounds
constexpr int kRrCtr = 4;                 // counter sets 4-9: three rounds, two sides
constexpr int kRrState = 10;

struct RrState {
  uint32_t arrive, failed, rounds[2];
  unsigned long long nf[2], nf_edges[2], prev_nf[2];
  unsigned long long edges[2], expanded[2], unvisited[2];
  uint32_t done, odd;  // the frontiers lie in q[odd]
  unsigned long long zeros;
};
static_assert(sizeof(RrState) <= 2 * sizeof(Counters), "two counter sets hold it");

struct RrSide {
  const uint64_t *off, *B_off;  // search direction, reverse direction
  const uint32_t *E, *B_E;
  uint32_t* vis;
  uint32_t* q[2];
  uint32_t* fb[3];
  uint64_t* heavy;
  uint64_t nf;
};

struct RrArgs {
  RrSide s[2];
  int ns;
  uint64_t n, threshold;
  uint32_t max_rounds;
  // first launch of a search: the sources, and (optional) the count of trimmed
  // vertices, with which there is one source or none
  const uint32_t* srcs;
  const uint64_t* zeros;
  Counters* ctr;
  RrState* st;
};

// A vertex claimed by a push round joins the next frontier in both forms.
template <int K>
__device__ __forceinline__ void rr_emit(const RrSide& S, uint32_t tm, const uint32_t* v,
                                        uint32_t* qout, uint32_t* fb_out, Counters* c,
                                        unsigned long long& next_edges) {
  warp_append_batch<K>(tm, v, qout, &c->next);
#pragma unroll
  for (int k = 0; k < K; k++)
    if (tm & (1u << k)) {
      atomicOr(&fb_out[v[k] >> 5], 1u << (v[k] & 31));
      next_edges += S.off[v[k] + 1] - S.off[v[k]];
    }
}

__global__ void __launch_bounds__(kRrThreads, 1) k_reach_rounds(RrArgs a) {
  __shared__ WarpExpandSmem ssm[kRrWarps];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5, tid = threadIdx.x;
  const uint64_t gw = (uint64_t)blockIdx.x * kRrWarps + wid, nw = (uint64_t)gridDim.x * kRrWarps;
  const uint64_t gt = (uint64_t)blockIdx.x * kRrThreads + tid, nt = (uint64_t)gridDim.x * kRrThreads;
  const uint64_t nwords = (a.n + 31) >> 5;
  const bool lead = blockIdx.x == 0 && tid == 0;
  WarpExpandSmem& sm = ssm[wid];
  uint32_t target = 0;
  auto barrier = [&]() { return grid_barrier(&a.st->arrive, &a.st->failed, target); };
  uint64_t nf0 = a.s[0].nf, nf1 = a.ns > 1 ? a.s[1].nf : 0, ne0 = 0, ne1 = 0, pf0 = 0, pf1 = 0;
  uint32_t rd0 = 0, rd1 = 0, round = 0;
  unsigned long long t_e[2] = {0, 0}, t_x[2] = {0, 0}, t_u[2] = {0, 0};  // lead thread
  for (int k = 0; k < a.ns; k++)
    for (uint64_t w = gt; w < nwords; w += nt) {
      a.s[k].fb[1][w] = 0;
      a.s[k].fb[2][w] = 0;
      if (a.srcs) a.s[k].vis[w] = 0;
    }
  uint64_t zeros = 0;
  if (a.zeros) {
    zeros = *a.zeros;
    nf0 = nf1 = zeros < a.n ? 1 : 0;
    if (a.ns < 2) nf1 = 0;
  }
  if (!barrier()) return;
  if (a.srcs) {
    for (int k = 0; k < a.ns; k++)
      for (uint64_t i = gt; i < (k ? nf1 : nf0); i += nt) {
        const uint32_t v = __ldg(&a.srcs[i]);
        atomicOr(&a.s[k].vis[v >> 5], 1u << (v & 31));
        a.s[k].q[0][i] = v;
      }
    if (!barrier()) return;
  }
  for (; (nf0 | nf1) && round < a.max_rounds; round++) {
    Counters* c0 = a.ctr + kRrCtr + 2 * (round % 3);
    if (blockIdx.x == 0 && tid < 2 * sizeof(Counters) / 8)  // last read a barrier ago
      ((unsigned long long*)(a.ctr + kRrCtr + 2 * ((round + 1) % 3)))[tid] = 0;
    for (int k = 0; k < a.ns; k++) {
      const RrSide& S = a.s[k];
      const uint64_t nf = k ? nf1 : nf0, ne = k ? ne1 : ne0;
      uint32_t* clear = S.fb[(round + 2) % 3];
      for (uint64_t w = gt; w < nwords; w += nt) clear[w] = 0;
      if (nf == 0) continue;
      Counters* c = c0 + k;
      const uint32_t* qin = S.q[round & 1];
      uint32_t* qout = S.q[(round + 1) & 1];
      const uint32_t* fb_in = S.fb[round % 3];
      uint32_t* fb_out = S.fb[(round + 1) % 3];
      unsigned long long scanned = 0, next_edges = 0, expanded = 0, unvisited = 0;
      if (round == 0 || nf + ne < a.threshold) {
        // --- push: 32 vertices per warp step, fewer when that leaves warps idle
        const uint64_t per = (nf + nw - 1) / nw;
        const uint32_t chunk = (uint32_t)(per > 32 ? 32 : per);
        for (uint64_t b = gw * chunk; b < nf; b += nw * chunk) {
          uint64_t beg = 0, d = 0;
          if (lane < chunk && b + lane < nf) {
            const uint32_t u = ld_cg(&qin[b + lane]);
            beg = S.off[u];
            d = S.off[u + 1] - beg;
            expanded++;
            if (d > kRrHeavy) {
              const unsigned long long old =
                  atomicAdd(&c->heavy, (1ull << kPackShift) + (d + kHeavyChunk - 1) / kHeavyChunk);
              S.heavy[old >> kPackShift] = ((uint64_t)u << 32) | (old & kPackMask);
              d = 0;
            }
          }
          scanned += d;
          expand_claim<kPushK>(sm, beg, (uint32_t)d, S.E, S.vis,
                               [&](uint32_t tm, const uint32_t* v) {
                                 rr_emit<kPushK>(S, tm, v, qout, fb_out, c, next_edges);
                               });
        }
      } else {
        // --- pull: a warp owns 32 consecutive vertices at a time
        for (uint64_t w = gw; w < nwords; w += nw) {
          const uint32_t vw = __ldcg(&S.vis[w]);
          const uint64_t v = w * 32 + lane;
          const bool t = v < a.n && !((vw >> lane) & 1u);
          uint64_t j = 0, e = 0;
          bool found = false;
          if (t) {
            const uint64_t b = S.B_off[v];
            e = S.B_off[v + 1];
            j = b;
            found = pull_scan<true>(S.B_E, fb_in, j, e < b + kPullSolo ? e : b + kPullSolo);
            scanned += j - b;
            unvisited++;
          }
          pull_long<true>(S.B_E, fb_in, __ballot_sync(kFull, t && !found && j < e), j, e, found,
                          scanned);
          const uint32_t mk = __ballot_sync(kFull, found);
          if (mk) {
            if (lane == 0) {
              fb_out[w] = mk;
              S.vis[w] = vw | mk;
            }
            const unsigned long long pos = warp_append(&c->next, found);
            if (found) {
              qout[pos] = (uint32_t)v;
              next_edges += S.off[v + 1] - S.off[v];
            }
          }
        }
      }
      scanned = warp_sum(scanned);
      next_edges = warp_sum(next_edges);
      expanded = warp_sum(expanded);
      unvisited = warp_sum(unvisited);
      if (lane == 0) {
        if (scanned) atomicAdd(&c->edges, scanned);
        if (next_edges) atomicAdd(&c->next_edges, next_edges);
        if (expanded) atomicAdd(&c->expanded, expanded);
        if (unvisited) atomicAdd(&c->unvisited, unvisited);
      }
    }
    if (!barrier()) return;
    if (__ldcg(&c0->heavy) | (a.ns > 1 ? __ldcg(&c0[1].heavy) : 0)) {
      // --- heavy vertices: their chunks in one contiguous range per warp
      for (int k = 0; k < a.ns; k++) {
        const RrSide& S = a.s[k];
        Counters* c = c0 + k;
        const unsigned long long packed = __ldcg(&c->heavy);
        const uint64_t nh = packed >> kPackShift, total = packed & kPackMask;
        const uint64_t per = (total + nw - 1) / nw;
        const uint64_t c_beg = gw * per, c_end = c_beg + per < total ? c_beg + per : total;
        unsigned long long scanned = 0, next_edges = 0;
        if (nh && c_beg < c_end) {
          uint64_t h = 0, hi = nh - 1;  // last entry whose first chunk is <= c_beg
          while (h < hi) {
            const uint64_t mid = (h + hi + 1) >> 1;
            if ((uint32_t)ld_cg(&S.heavy[mid]) <= c_beg)
              h = mid;
            else
              hi = mid - 1;
          }
          for (uint64_t x = c_beg; x < c_end;) {
            const uint64_t ent = ld_cg(&S.heavy[h]);
            const uint64_t cs = (uint32_t)ent;
            const uint64_t cn = h + 1 < nh ? (uint32_t)ld_cg(&S.heavy[h + 1]) : total;
            const uint64_t beg = S.off[ent >> 32], end = S.off[(ent >> 32) + 1];
            for (; x < c_end && x < cn; x++) {
              const uint64_t e0 = beg + (x - cs) * kHeavyChunk;
              uint32_t v[kHeavyK], tm = 0;
#pragma unroll
              for (int i = 0; i < kHeavyK; i++) {
                const uint64_t e = e0 + i * 32 + lane;
                v[i] = kNone;
                if (e < end) {
                  scanned++;
                  v[i] = __ldg(&S.E[e]);
                }
              }
#pragma unroll
              for (int i = 0; i < kHeavyK; i++)
                if (v[i] != kNone && bit_set(S.vis, v[i])) tm |= 1u << i;
              rr_emit<kHeavyK>(S, tm, v, S.q[(round + 1) & 1], S.fb[(round + 1) % 3], c, next_edges);
            }
            h++;
          }
        }
        scanned = warp_sum(scanned);
        next_edges = warp_sum(next_edges);
        if (lane == 0) {
          if (scanned) atomicAdd(&c->edges, scanned);
          if (next_edges) atomicAdd(&c->next_edges, next_edges);
        }
      }
      if (!barrier()) return;
    }
    if (lead)
      for (int k = 0; k < a.ns; k++) {
        t_e[k] += __ldcg(&c0[k].edges);
        t_x[k] += __ldcg(&c0[k].expanded);
        t_u[k] += __ldcg(&c0[k].unvisited);
      }
    if (nf0) {
      rd0++;
      pf0 = nf0;
      nf0 = __ldcg(&c0->next);
      ne0 = __ldcg(&c0->next_edges);
    }
    if (nf1) {
      rd1++;
      pf1 = nf1;
      nf1 = __ldcg(&c0[1].next);
      ne1 = __ldcg(&c0[1].next_edges);
    }
  }
  if (lead) {
    RrState& s = *a.st;
    s.rounds[0] = rd0;
    s.rounds[1] = rd1;
    s.nf[0] = nf0;
    s.nf[1] = nf1;
    s.nf_edges[0] = ne0;
    s.nf_edges[1] = ne1;
    s.prev_nf[0] = pf0;
    s.prev_nf[1] = pf1;
    for (int k = 0; k < 2; k++) {
      s.edges[k] = t_e[k];
      s.expanded[k] = t_x[k];
      s.unvisited[k] = t_u[k];
    }
    s.odd = round & 1;
    s.zeros = zeros;
    s.done = 1;
  }
}

__global__ void k_queue_to_bitmap(const uint32_t* __restrict__ q, uint64_t nq, uint32_t* fb) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t v = q[i];
    atomicOr(&fb[v >> 5], 1u << (v & 31));
  }
}

// Unordered compaction of a bitmap into a queue (counter: ctr->aux0).
__global__ void k_bitmap_to_queue(const uint32_t* __restrict__ fb, uint64_t nwords, uint32_t* q,
                                  Counters* ctr) {
  const unsigned lane = lane_id();
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t base = gw * 32; base < nwords; base += nw * 32) {
    const uint64_t w = base + lane;
    uint32_t word = w < nwords ? fb[w] : 0u;
    uint32_t c = __popc(word);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t t = __shfl_up_sync(kFull, incl, o);
      if ((int)lane >= o) incl += t;
    }
    uint32_t total = __shfl_sync(kFull, incl, 31);
    unsigned long long pos = 0;
    if (lane == 0 && total) pos = atomicAdd(&ctr->aux0, (unsigned long long)total);
    pos = __shfl_sync(kFull, pos, 0) + (incl - c);
    while (word) {
      int b = __ffs(word) - 1;
      word &= word - 1;
      q[pos++] = (uint32_t)(w * 32 + b);
    }
  }
}

__global__ void k_bitmap_to_bytes(const uint32_t* __restrict__ vis, uint64_t n, uint8_t* out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = (vis[i >> 5] >> (i & 31)) & 1u;
}

// ---------------------------------------------------------------------------
// Host round loop over one or two sides.
// ---------------------------------------------------------------------------
namespace {

// The VGC kernel of a graph (see kVgcKNarrow): its resident blocks per SM
// (cached on the handle) and its launch.
static bool vgc_narrow(const psc_graph_s* g) { return g->m < 8 * g->n; }

static int vgc_occupancy(psc_graph_s* g) {
  if (!g->vgc_blocks) {
    PSC_CUDA(vgc_narrow(g) ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                 &g->vgc_blocks, k_reach_vgc<kVgcBlock, kVgcQueue, kVgcKNarrow, true>,
                                 kVgcBlock, 0)
                           : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                                 &g->vgc_blocks, k_reach_vgc<kVgcBlock, kVgcQueue, kVgcKWide, true>,
                                 kVgcBlock, 0));
    if (g->vgc_blocks < 1) g->vgc_blocks = 1;
  }
  return PSC_OK;
}

// The search without rounds: with records on graphs of low degree (queue of
// kAsyncRecQueue entries), else in the narrow or wide form of the VGC kernel.
constexpr int kAsyncRecQueue = 128;
constexpr int kAsyncRecBlocks = 3;  // per SM (see k_reach_async_low)
template <class F>
static auto with_async_kernel(const psc_graph_s* g, bool rec, F f) {
  if (rec) return f(k_reach_async_low<kVgcBlock, kAsyncRecQueue>);
  if (vgc_narrow(g)) return f(k_reach_async<kVgcBlock, kVgcQueue, kVgcKNarrow>);
  return f(k_reach_async<kVgcBlock, kVgcQueue, kVgcKWide>);
}

static int launch_async(psc_graph_s* g, bool rec, const ReachSide& a, const ReachSide& b,
                        AsyncCtl* ca, AsyncCtl* cb, uint32_t slots, uint32_t backlog) {
  int& per_sm = g->async_blocks[rec ? 1 : 0];
  return with_async_kernel(g, rec, [&](auto kernel) -> int {
    if (!per_sm) {
      PSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kVgcBlock, 0));
      if (rec) per_sm = std::min(per_sm, kAsyncRecBlocks);
      if (per_sm < 1) per_sm = 1;
    }
    const uint64_t blocks = std::min<uint64_t>((uint64_t)resident_sms(g) * per_sm,
                                               kAsyncMaxWarps / (kVgcBlock / 32));
    kernel<<<(unsigned)blocks, kVgcBlock, 0, g->stream>>>(a, b, ca, cb, slots, backlog);
    return PSC_OK;
  });
}

// spec: speculative range loads (vgc_claim), for rounds whose frontier gives
// each resident warp at most kVgcSpecChunk vertices (latency-bound rounds)
#ifndef PSC_VGC_SPEC_CHUNK
#define PSC_VGC_SPEC_CHUNK 8
#endif
constexpr uint64_t kVgcSpecChunk = PSC_VGC_SPEC_CHUNK;
// Out-degree above which a vertex of a sparse VGC round (one vertex per warp) goes to
// k_reach_heavy: a warp takes some 5 us per 256 edges, so the round waits for its
// largest vertex, and the extra launch costs about what 2,048 edges do (second round
// of R-MAT 2^26: 335 + 225 us with 8,192, 183 + 241 with 2,048, 184 + 244 with 1,024).
constexpr uint32_t kVgcHeavy = 2048;
static void launch_vgc(psc_graph_s* g, unsigned blocks, const ReachSide& a, const ReachSide& b,
                       uint32_t tau, uint32_t chunk, bool spec, uint32_t hlim) {
  cudaStream_t st = g->stream;
  if (vgc_narrow(g)) {
    if (spec)
      k_reach_vgc<kVgcBlock, kVgcQueue, kVgcKNarrow, true><<<blocks, kVgcBlock, 0, st>>>(a, b, tau, chunk, hlim);
    else
      k_reach_vgc<kVgcBlock, kVgcQueue, kVgcKNarrow, false><<<blocks, kVgcBlock, 0, st>>>(a, b, tau, chunk, hlim);
  } else {
    if (spec)
      k_reach_vgc<kVgcBlock, kVgcQueue, kVgcKWide, true><<<blocks, kVgcBlock, 0, st>>>(a, b, tau, chunk, hlim);
    else
      k_reach_vgc<kVgcBlock, kVgcQueue, kVgcKWide, false><<<blocks, kVgcBlock, 0, st>>>(a, b, tau, chunk, hlim);
  }
}

// Adjacency records of one direction (see VRec).
__global__ void k_build_records(const uint64_t* __restrict__ off, const uint32_t* __restrict__ E,
                                uint64_t n, VRec* rec) {
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = off[v], r = adj_hdr(b, off[v + 1]), d = r & 0xFFFFFFull;
    uint32_t e[kRecEdges];
#pragma unroll
    for (int j = 0; j < kRecEdges; j++) e[j] = (uint64_t)j < d ? __ldg(&E[b + j]) : kNone;
    uint4* o = (uint4*)(rec + v);
    o[0] = make_uint4((uint32_t)r, (uint32_t)(r >> 32), e[0], e[1]);
    o[1] = make_uint4(e[2], e[3], e[4], e[5]);
  }
}

// Once per handle and direction (the graph does not change); a symmetric graph
// has one set.  *out is null when there is no memory for them.
int records_once_impl(psc_graph_s* g, bool backward, const VRec** out) {
  const int d = backward && !g->symmetric ? 1 : 0;
  VRec* r = nullptr;
  *out = nullptr;
  const int st = ensure_t(g, d ? B_REC_B : B_REC_F, g->n, &r);
  if (st == PSC_ERR_OOM) return PSC_OK;
  PSC_TRY(st);
  if (!g->rec_known[d]) {
    ProfScope ps(g, F_REACH_VGC);
    k_build_records<<<grid_for(g, g->n, 256), 256, 0, g->stream>>>(d ? g->in_off : g->off,
                                                                   d ? g->in_E : g->E, g->n, r);
    PSC_CUDA(cudaGetLastError());
    g->rec_known[d] = true;
  }
  *out = r;
  return PSC_OK;
}

// Bitmap words of vertices whose range in off is empty (one warp per word),
// and their count.
__global__ void k_dead_bits(const uint64_t* __restrict__ off, uint64_t n, uint32_t* bits,
                            unsigned long long* count) {
  const uint64_t nwords = (n + 31) >> 5;
  unsigned long long c = 0;
  for (uint64_t base = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull;
       base < nwords * 32; base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t v = base + lane_id();
    const uint32_t word = __ballot_sync(kFull, v < n && off[v + 1] == off[v]);
    if (lane_id() == 0) {
      bits[base >> 5] = word;
      c += __popc(word);
    }
  }
  if (lane_id() == 0 && c) atomicAdd(count, c);
}

// Once per handle: the vertices a forward pull can never reach (no in-edge)
// and those a backward pull can never reach (no out-edge).
static int dead_bits_once(psc_graph_s* g) {
  if (g->dead_known) return PSC_OK;
  const uint64_t nwords = (g->n + 31) / 32;
  uint32_t* d;
  PSC_TRY(ensure_t(g, B_DEAD, 2 * (nwords + 1), &d));
  unsigned long long* c = &g->ctr[2].aux0;  // aux0, aux1 of the staging set
  PSC_CUDA(cudaMemsetAsync(c, 0, 2 * sizeof(unsigned long long), g->stream));
  k_dead_bits<<<grid_for(g, nwords * 32, 256), 256, 0, g->stream>>>(g->in_off, g->n, d, c);
  k_dead_bits<<<grid_for(g, nwords * 32, 256), 256, 0, g->stream>>>(g->off, g->n, d + nwords + 1,
                                                                     c + 1);
  PSC_CUDA(cudaGetLastError());
  PSC_TRY(read_counters(g));
  g->dead_count[0] = g->hctr[2].aux0;
  g->dead_count[1] = g->hctr[2].aux1;
  g->dead_known = true;
  return PSC_OK;
}

struct Side {
  bool backward = false;
  uint32_t* vis = nullptr;
  int slot_qa = 0, slot_qb = 0, slot_fa = 0, slot_fb = 0, slot_heavy = 0;
  int cset = 0;  // counter block
  uint64_t nf = 0, nf_edges = 0, prev_nf = 0;
  bool pull = false;
  uint32_t rounds = 0;
  // unvisited vertices that some pull could still reach, after a pull round
  uint64_t live = 0;
};

// Counter sets of k_reach_async: the control words of side k, and its counters.
constexpr int async_ctl_set(int k) { return kAsyncSet + 2 * k; }
constexpr int async_ctr_set(int k) { return kAsyncSet + 4 + k; }
// Rounds of a search with local searches that k_reach_rounds takes.
constexpr uint32_t kRrRounds = 16;

enum Mode { M_NONE, M_VGC, M_PUSH, M_PULL };

ReachSide side_args(psc_graph_s* g, const Side& s) {
  ReachSide r;
  r.off = s.backward ? g->in_off : g->off;
  r.E = s.backward ? g->in_E : g->E;
  r.qin = (const uint32_t*)g->bufs[s.slot_qa].p;
  r.nin = s.nf;
  r.vis = s.vis;
  r.qout = (uint32_t*)g->bufs[s.slot_qb].p;
  r.heavy = (uint64_t*)g->bufs[s.slot_heavy].p;
  r.ctr = g->ctr + s.cset;
  r.rec = nullptr;
  return r;
}

Side make_side(bool backward, uint32_t* vis, int second) {
  Side s;
  s.backward = backward;
  s.vis = vis;
  s.slot_qa = second ? B_QA2 : B_QA;
  s.slot_qb = second ? B_QB2 : B_QB;
  s.slot_fa = second ? B_FB_A2 : B_FB_A;
  s.slot_fb = second ? B_FB_B2 : B_FB_B;
  s.slot_heavy = second ? B_HEAVY2 : B_HEAVY;
  s.cset = second ? 1 : 0;
  return s;
}

}  // namespace

// Largest out-degree (out[0]) and in-degree (out[1]) of the graph.
__global__ void k_max_degrees(const uint64_t* __restrict__ off, const uint64_t* __restrict__ in_off,
                              uint64_t n, unsigned long long* out) {
  unsigned long long a = 0, b = 0;
  for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const unsigned long long x = off[v + 1] - off[v], y = in_off[v + 1] - in_off[v];
    a = x > a ? x : a;
    b = y > b ? y : b;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long x = __shfl_xor_sync(kFull, a, o), y = __shfl_xor_sync(kFull, b, o);
    a = x > a ? x : a;
    b = y > b ? y : b;
  }
  if (lane_id() == 0) {
    if (a) atomicMax(&out[0], a);
    if (b) atomicMax(&out[1], b);
  }
}

// Once per handle (the graph does not change): max_deg, for the choice of the
// search without rounds and of the heavy launches of BFS.
int max_degrees_once(psc_graph_s* g) {
  if (g->deg_known) return PSC_OK;
  unsigned long long* d = &g->ctr[2].aux0;  // aux0, aux1 of the staging set
  PSC_CUDA(cudaMemsetAsync(d, 0, 2 * sizeof(unsigned long long), g->stream));
  k_max_degrees<<<grid_for(g, g->n, 256), 256, 0, g->stream>>>(g->off, g->in_off, g->n, d);
  PSC_CUDA(cudaGetLastError());
  PSC_TRY(read_counters(g));
  g->max_deg[0] = g->hctr[2].aux0;
  g->max_deg[1] = g->hctr[2].aux1;
  g->deg_known = true;
  return PSC_OK;
}

int records_if_low(psc_graph_s* g, bool backward, const VRec** out) {
  *out = nullptr;
  if (g->num_graphs || (g->m >> 40) || g->rec_refused) return PSC_OK;
  PSC_TRY(max_degrees_once(g));
  if (g->max_deg[0] > kRecMaxDeg || g->max_deg[1] > kRecMaxDeg) return PSC_OK;
  return records_once_impl(g, backward, out);
}

// Whether the device holds k_reach_rounds with a block on every SM.
static bool rr_ready(int device) {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static int state[kMaxDev] = {};
  if (device < 0 || device >= kMaxDev) return false;
  std::lock_guard<std::mutex> lock(mu);
  int& st = state[device];
  if (st == 0) {
    int coop = 0, b = 0;
    st = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess && coop &&
                 cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_reach_rounds, kRrThreads, 0) ==
                     cudaSuccess &&
                 b > 0
             ? 1
             : -1;
    cudaGetLastError();
  }
  return st == 1;
}

// Runs the searches of `ns` sides (1 or 2) to completion.  Side k starts from
// srcs[k], or, when d_srcs is given, every side starts from the n_dsrc device
// sources d_srcs.
// zeros (with d_srcs): the device count of trimmed vertices; there is one source
// if it is below n, else none; *n_zeros receives it.
static int reach_sides(psc_graph_s* g, Side* sides, int ns, const uint32_t* srcs, bool local,
                       uint32_t tau, uint32_t pull_div, const uint32_t* d_srcs = nullptr,
                       uint64_t n_dsrc = 0, uint64_t vgc_max = 0, const uint64_t* zeros = nullptr,
                       uint64_t* n_zeros = nullptr) {
  const uint64_t n = g->n, nwords = (n + 31) / 32;
  // heavy-list fields: < 2^24 entries (m / kHeavyDeg), < 2^32 chunks
  if (g->m >> 36) return PSC_ERR_TOO_LARGE;
  // VGC rounds while the frontier is below one vertex per resident warp
  // (unless the caller sets the limit)
  const uint64_t vgc_limit = vgc_max ? vgc_max : (uint64_t)g->num_sms * 64;
  if (pull_div == 0) pull_div = 20;
  const uint64_t threshold = g->m / pull_div;
  const uint64_t slack = !local ? 0 : g->m > kHeavyDeg ? kAsyncSlack : std::min(n, kAsyncSlack);
  // (graphs of low degree have narrow frontiers, so deep ones: not in rounds)
  bool resident = g->m <= kRrMaxEdges && rr_ready(g->device);
  if (resident && local) {
    PSC_TRY(max_degrees_once(g));
    resident = g->max_deg[0] > kRecMaxDeg || g->max_deg[1] > kRecMaxDeg;
  }
  const bool start_there = resident && d_srcs;  // the launch sets its sources itself
  if (zeros && !start_there) {
    PSC_CUDA(cudaMemcpyAsync(&g->hctr->aux0, zeros, 8, cudaMemcpyDeviceToHost, g->stream));
    PSC_CUDA(cudaStreamSynchronize(g->stream));
    *n_zeros = g->hctr->aux0;
    n_dsrc = *n_zeros < n ? 1 : 0;
  }
  for (int k = 0; k < ns; k++) {
    Side& s = sides[k];
    void* p;
    PSC_TRY(ensure(g, s.slot_qa, (n + 1 + slack) * 4, &p));
    PSC_TRY(ensure(g, s.slot_qb, (n + 1 + slack) * 4, &p));
    PSC_TRY(ensure(g, s.slot_fa, (nwords + 1) * 4, &p));
    PSC_TRY(ensure(g, s.slot_fb, (nwords + 1) * 4, &p));
    PSC_TRY(ensure(g, s.slot_heavy, (n + 1) * 8, &p));
    s.nf = d_srcs ? n_dsrc : 1;
    s.nf_edges = 0;
    s.prev_nf = 0;
    s.pull = false;
    s.rounds = 0;
    if (start_there) continue;
    PSC_CUDA(cudaMemsetAsync(s.vis, 0, nwords * 4, g->stream));
    if (!d_srcs)
      k_reach_init<<<1, 1, 0, g->stream>>>(s.vis, (uint32_t*)g->bufs[s.slot_qa].p, srcs[k]);
    else if (n_dsrc)
      k_reach_init_multi<<<grid_for(g, n_dsrc, 256), 256, 0, g->stream>>>(
          s.vis, (uint32_t*)g->bufs[s.slot_qa].p, d_srcs, n_dsrc);
  }
  const bool tr = trace_on();
  bool async = local;
  uint32_t full = 0;  // launches that ended for want of slots
  bool first_launch = start_there;
  for (uint64_t iter = 0;; iter++) {
    if (iter > n + 2) return PSC_ERR_ITER_LIMIT;
    // Small graphs: all rounds in one launch, or the first kRrRounds of a search
    // with local searches (a deep one then goes on below, without rounds).
    if (resident) {
      resident = !local;  // local: once
      RrArgs a = {};
      a.ns = ns;
      a.n = n;
      a.threshold = threshold;
      a.max_rounds = local ? kRrRounds : 1u << 16;
      a.ctr = g->ctr;
      a.st = (RrState*)(g->ctr + kRrState);
      bool any = false;
      for (int k = 0; k < ns; k++) {
        const Side& s = sides[k];
        RrSide& r = a.s[k];
        r.off = s.backward ? g->in_off : g->off;
        r.E = s.backward ? g->in_E : g->E;
        r.B_off = s.backward ? g->off : g->in_off;
        r.B_E = s.backward ? g->E : g->in_E;
        r.vis = s.vis;
        r.q[0] = (uint32_t*)g->bufs[s.slot_qa].p;
        r.q[1] = (uint32_t*)g->bufs[s.slot_qb].p;
        uint32_t* third;
        PSC_TRY(ensure_t(g, k ? B_FB_C2 : B_FB_C, nwords + 1, &third));
        r.fb[0] = third;
        r.fb[1] = (uint32_t*)g->bufs[s.slot_fa].p;
        r.fb[2] = (uint32_t*)g->bufs[s.slot_fb].p;
        r.heavy = (uint64_t*)g->bufs[s.slot_heavy].p;
        r.nf = s.nf;
        any |= s.nf != 0;
      }
      if (first_launch) {
        a.srcs = d_srcs;
        a.zeros = zeros;
        any = true;
        first_launch = false;
      }
      if (any) {
        PSC_TRY(zero_counters(g));
        {
          ProfScope ps(g, F_REACH_PUSH);
          void* args[] = {&a};
          PSC_CUDA(cudaLaunchCooperativeKernel((const void*)k_reach_rounds, dim3(resident_sms(g)),
                                               dim3(kRrThreads), args, 0, g->stream));
        }
        PSC_TRY(read_counters(g));
        const RrState& st = *(const RrState*)(g->hctr + kRrState);
        if (st.failed || !st.done) return PSC_ERR_ITER_LIMIT;
        if (a.zeros) *n_zeros = st.zeros;
        for (int k = 0; k < ns; k++) {
          Side& s = sides[k];
          s.rounds += st.rounds[k];
          s.nf = st.nf[k];
          s.nf_edges = st.nf_edges[k];
          s.prev_nf = st.prev_nf[k];
          if (st.odd) std::swap(g->bufs[s.slot_qa], g->bufs[s.slot_qb]);
          if (g->profiling)
            g->prof[F_REACH_PUSH].bytes +=
                16.0 * (st.expanded[k] + st.unvisited[k]) + 5.0 * st.edges[k];
          if (tr)
            std::fprintf(stderr, "reach side %d resident rounds %u left %llu edges %llu\n", k,
                         st.rounds[k], st.nf[k], st.edges[k]);
        }
        continue;
      }
    }
    // The sparse part of a search in one launch (k_reach_async): from the
    // start on graphs of low degree (their frontiers grow slowly), else once
    // every active side's frontier is steady, well inside VGC range (at least
    // two rounds done, grown at most 1.5x in the last one, far from the pull
    // threshold).  What a stopped launch left goes on in rounds.
    if (async) {
      int act[2], na = 0;
      bool steady = true, sparse = true;
      for (int k = 0; k < ns; k++) {
        const Side& s = sides[k];
        if (s.nf == 0) continue;
        act[na++] = k;
        sparse = sparse && !s.pull && s.nf <= vgc_limit && s.nf <= kAsyncSlots / 4;
        steady = steady && s.rounds >= 2 && 2 * s.nf <= 3 * s.prev_nf &&
                 3 * (s.nf + s.nf_edges) < threshold;
      }
      bool go = na > 0 && sparse;
      if (go && !steady) {
        PSC_TRY(max_degrees_once(g));
        go = g->max_deg[0] <= kRecMaxDeg && g->max_deg[1] <= kRecMaxDeg;
      }
      if (go) {
        const uint32_t slots = async_slots(n, std::max(sides[0].nf, ns > 1 ? sides[1].nf : 0), full);
        // queued vertices whose edges reach the pull threshold, or more than a
        // few rounds' worth of local searches: full-width rounds are faster
        uint64_t backlog = std::max<uint64_t>(threshold * n / std::max<uint64_t>(g->m, 1), 1);
        const bool low = g->deg_known && g->max_deg[0] <= kRecMaxDeg && g->max_deg[1] <= kRecMaxDeg;
        if (low) backlog = n;
        if (!vgc_max) backlog = std::min<uint64_t>(backlog, 4 * vgc_limit);
        ReachSide sd[2] = {};
        bool rec = low;
        AsyncCtl* ctl[2];
        uint32_t nf[2] = {0, 0};
        for (int a = 0; a < 2; a++) {
          ctl[a] = (AsyncCtl*)(g->ctr + async_ctl_set(a));
          if (a >= na) continue;
          const Side& s = sides[act[a]];
          sd[a] = side_args(g, s);
          sd[a].ctr = g->ctr + async_ctr_set(a);
          if (rec) PSC_TRY(records_if_low(g, s.backward, &sd[a].rec));
          rec = rec && sd[a].rec;
          nf[a] = (uint32_t)s.nf;
        }
        k_async_prepare<<<grid_for(g, slots, 256, 4), 256, 0, g->stream>>>(
            sd[0].qin, nf[0], sd[0].qout, sd[1].qin, nf[1], sd[1].qout, slots, g->ctr);
        if (na == 1) {  // the second side is done from the start
          sd[1] = sd[0];
          sd[1].ctr = g->ctr + async_ctr_set(1);
        }
        {
          ProfScope ps(g, F_REACH_VGC);
          PSC_TRY(launch_async(g, rec, sd[0], sd[1], ctl[0], ctl[1], slots,
                               (uint32_t)std::min<uint64_t>(backlog, 0x7FFFFFFFu)));
        }
        PSC_CUDA(cudaGetLastError());
        PSC_TRY(read_counters(g));
        bool stopped = false;
        for (int a = 0; a < na; a++)
          stopped |= (((const AsyncCtl*)(g->hctr + async_ctl_set(a)))->flags & kAsyncStop) != 0;
        if (stopped) {
          for (int a = 0; a < na; a++)
            k_async_collect<<<g->num_sms * 2, 256, 0, g->stream>>>(
                sd[a].qout, ctl[a], slots, sd[a].off, (uint32_t*)sd[a].qin, sd[a].ctr);
          PSC_CUDA(cudaGetLastError());
          PSC_TRY(read_counters(g));
        }
        for (int a = 0; a < na; a++) {
          Side& s = sides[act[a]];
          const AsyncCtl& c = *(const AsyncCtl*)(g->hctr + async_ctl_set(a));
          const Counters& k = g->hctr[async_ctr_set(a)];
          if (g->profiling)
            g->prof[F_REACH_VGC].bytes += 16.0 * k.expanded + 5.0 * k.edges + 5.0 * k.expanded;
          if (tr)
            std::fprintf(stderr, "reach side %d async nf %u left %llu edges %llu expanded %llu "
                         "given %u flags %u\n", act[a], nf[a], k.next, k.edges, k.expanded,
                         c.tail, c.flags);
          if (!(c.flags & kAsyncStop) && c.fin != c.tail) return PSC_ERR_ITER_LIMIT;  // cannot be
          if (c.flags & (kAsyncHeavy | kAsyncWide)) async = false;
          if (c.flags & kAsyncFull) full++;
          s.rounds++;
          s.prev_nf = s.nf;
          s.nf = k.next;
          s.nf_edges = k.next_edges;
        }
        continue;
      }
    }
    Mode mode[2] = {M_NONE, M_NONE};
    bool any = false;
    for (int k = 0; k < ns; k++) {
      Side& s = sides[k];
      if (s.nf == 0) continue;
      any = true;
      s.rounds++;
      // A search that pulls goes on pulling while that looks at less: the live
      // vertices and the bitmaps' words (fifth round of R-MAT 2^26, 2.5e6 frontier and
      // 1e5 live vertices: 0.29 ms pushed, with the bitmaps turned into queues,
      // 0.14 pulled).
      const bool want_pull = (s.nf + s.nf_edges) >= threshold ||
                             (s.pull && s.nf >= s.live + nwords / 4);
      uint32_t* qa = (uint32_t*)g->bufs[s.slot_qa].p;
      uint32_t* fa = (uint32_t*)g->bufs[s.slot_fa].p;
      if (want_pull && !s.pull) {
        PSC_TRY(dead_bits_once(g));
        ProfScope ps(g, F_REACH_PULL);
        PSC_CUDA(cudaMemsetAsync(fa, 0, nwords * 4, g->stream));
        k_queue_to_bitmap<<<grid_for(g, s.nf, 256), 256, 0, g->stream>>>(qa, s.nf, fa);
        s.pull = true;
      } else if (!want_pull && s.pull) {
        ProfScope ps(g, F_REACH_PUSH);
        PSC_CUDA(cudaMemsetAsync(&g->ctr[s.cset].aux0, 0, 8, g->stream));
        k_bitmap_to_queue<<<grid_for(g, nwords, 256), 256, 0, g->stream>>>(fa, nwords, qa,
                                                                         g->ctr + s.cset);
        s.pull = false;
      }
      mode[k] = s.pull ? M_PULL : (local && s.nf <= vgc_limit) ? M_VGC : M_PUSH;
    }
    if (!any) break;
    PSC_TRY(zero_counters(g));
    ReachSide vg[2] = {}, pu[2] = {}, hv[2] = {};
    int nv = 0, np = 0, nh = 0;
    uint64_t v_items = 0, p_items = 0;
    for (int k = 0; k < ns; k++) {
      if (mode[k] == M_VGC) {
        vg[nv++] = side_args(g, sides[k]);
        v_items += sides[k].nf;
      } else if (mode[k] == M_PUSH) {
        pu[np++] = side_args(g, sides[k]);
        p_items += sides[k].nf;
      }
      if (mode[k] == M_VGC || mode[k] == M_PUSH) hv[nh++] = side_args(g, sides[k]);
    }
    if (nv) {
      ProfScope ps(g, F_REACH_VGC);
      // a resident grid; one frontier vertex per warp while the frontier
      // fits it, else chunks of up to 32 so that every warp stays busy
      PSC_TRY(vgc_occupancy(g));
      const uint64_t max_blocks = (uint64_t)g->num_sms * g->vgc_blocks;
      const uint64_t max_warps = max_blocks * (kVgcBlock / 32);
      const uint64_t chunk = std::min<uint64_t>(32, (v_items + max_warps - 1) / max_warps);
      const uint64_t chunks = (v_items + chunk - 1) / chunk;
      const uint64_t blocks = std::min(max_blocks, (chunks + kVgcBlock / 32 - 1) / (kVgcBlock / 32));
      launch_vgc(g, (unsigned)std::max<uint64_t>(1, blocks), vg[0], vg[1], tau, (uint32_t)chunk,
                 chunk <= kVgcSpecChunk, chunk == 1 ? kVgcHeavy : (uint32_t)kHeavyDeg);
    }
    if (np) {
      ProfScope ps(g, F_REACH_PUSH);
      switch (g->block) {
        case 128:
          k_reach_push<128><<<grid_for(g, p_items, 128), 128, 0, g->stream>>>(pu[0], pu[1]);
          break;
        case 512:
          k_reach_push<512><<<grid_for(g, p_items, 512), 512, 0, g->stream>>>(pu[0], pu[1]);
          break;
        default:
          k_reach_push<kReachBlock><<<grid_for(g, p_items, kReachBlock), kReachBlock, 0,
                                      g->stream>>>(pu[0], pu[1]);
      }
    }
    for (int k = 0; k < ns; k++) {
      if (mode[k] != M_PULL) continue;
      Side& s = sides[k];
      ProfScope ps(g, F_REACH_PULL);
      const uint64_t* B_off = s.backward ? g->off : g->in_off;
      const uint32_t* B_E = s.backward ? g->E : g->in_E;
      const uint64_t* A_off = s.backward ? g->in_off : g->off;
      const uint32_t* fa = (const uint32_t*)g->bufs[s.slot_fa].p;
      uint32_t* fbo = (uint32_t*)g->bufs[s.slot_fb].p;
      const uint32_t* dead = (const uint32_t*)g->bufs[B_DEAD].p + (s.backward ? nwords + 1 : 0);
      switch (g->block) {
        case 128:
          launch_pull<128>(g->num_sms, g->stream, B_off, B_E, fa, s.vis, fbo, n, g->ctr + s.cset, dead,
                           g->num_graphs > 1);
          break;
        case 512:
          launch_pull<512>(g->num_sms, g->stream, B_off, B_E, fa, s.vis, fbo, n, g->ctr + s.cset, dead,
                           g->num_graphs > 1);
          break;
        default:
          launch_pull<kReachBlock>(g->num_sms, g->stream, B_off, B_E, fa, s.vis, fbo, n,
                                   g->ctr + s.cset, dead, g->num_graphs > 1);
      }
      k_pull_out_edges<<<grid_for(g, nwords, 256), 256, 0, g->stream>>>(
          fbo, A_off, n, hash32((uint32_t)s.rounds), g->ctr + s.cset);
    }
    PSC_CUDA(cudaGetLastError());
    cudaEvent_t tr_b = nullptr;
    if (tr) {
      tr_b = take_event(g);
      PSC_CUDA(cudaEventRecord(tr_b, g->stream));
    }
    PSC_TRY(read_counters(g));
    // Heavy vertices are rare: the grid-wide walk is launched only for a
    // round that queued some, then the counters are read again.
    bool heavy = false;
    for (int k = 0; k < nh; k++) heavy |= g->hctr[hv[k].ctr - g->ctr].heavy != 0;
    if (heavy) {
      {
        ProfScope ps(g, F_HEAVY);
        k_reach_heavy<kReachBlock><<<g->num_sms * 4, kReachBlock, 0, g->stream>>>(hv[0], hv[1]);
      }
      PSC_CUDA(cudaGetLastError());
      PSC_TRY(read_counters(g));
      if (g->profiling)
        for (int k = 0; k < nh; k++) {
          const Counters& c = g->hctr[hv[k].ctr - g->ctr];
          g->prof[F_HEAVY].bytes += 24.0 * (c.heavy >> kPackShift) + 5.0 * c.heavy_edges;
        }
    }
    if (tr) {
      float us = 0;  // ms since the start of the call
      cudaEventElapsedTime(&us, g->t0, tr_b);
      give_event(g, tr_b);
      for (int k = 0; k < ns; k++)
        if (mode[k] != M_NONE)
          std::fprintf(stderr, "reach side %d round %u mode %s nf %llu next %llu edges %llu "
                       "expanded %llu unvisited %llu live %llu waves %llu t %.3f ms\n",
                       k, sides[k].rounds, mode[k] == M_VGC ? "vgc" : mode[k] == M_PUSH ? "push" : "pull",
                       (unsigned long long)sides[k].nf, g->hctr[sides[k].cset].next,
                       g->hctr[sides[k].cset].edges, g->hctr[sides[k].cset].expanded,
                       g->hctr[sides[k].cset].unvisited, (unsigned long long)sides[k].live,
                       g->hctr[sides[k].cset].waves, us);
    }
    for (int k = 0; k < ns; k++) {
      Side& s = sides[k];
      if (mode[k] == M_NONE) continue;
      const Counters& c = g->hctr[s.cset];
      if (g->profiling) {
        // algorithmic bytes: 16 per adjacency range read, 4 + 1 per edge
        // (target id, visited flag), 5 per new frontier vertex; pull: 16 per
        // unvisited vertex, 5 per scanned in-edge, bitmap words 1/4 byte per vertex
        const int fam = mode[k] == M_VGC ? F_REACH_VGC : mode[k] == M_PUSH ? F_REACH_PUSH
                                                                           : F_REACH_PULL;
        g->prof[fam].bytes += mode[k] == M_PULL
                                  ? 16.0 * c.unvisited + 5.0 * c.edges + 0.25 * n + 1.0 * c.next
                                  : 16.0 * c.expanded + 5.0 * c.edges + 5.0 * c.next;
      }
      if (mode[k] == M_PULL) {  // unvisited minus the dead ones (all but sources) minus found
        const uint64_t gone = g->dead_count[s.backward ? 1 : 0] + c.next;
        s.live = c.unvisited > gone ? c.unvisited - gone : 0;
      }
      if (mode[k] == M_PULL)
        std::swap(g->bufs[s.slot_fa], g->bufs[s.slot_fb]);
      else
        std::swap(g->bufs[s.slot_qa], g->bufs[s.slot_qb]);
      s.prev_nf = s.nf;
      s.nf = c.next;
      s.nf_edges = c.next_edges;
    }
  }
  return PSC_OK;
}

int reach_run(psc_graph_s* g, uint32_t src, bool backward, bool local, uint32_t tau,
              uint32_t pull_div, uint32_t* vis, uint32_t* rounds_out) {
  Side s = make_side(backward, vis, 0);
  PSC_TRY(reach_sides(g, &s, 1, &src, local, tau ? tau : 512, pull_div));
  if (rounds_out) *rounds_out = s.rounds;
  return PSC_OK;
}

int reach_first(psc_graph_s* g, const uint32_t* P, const uint64_t* zeros, bool local, uint32_t tau,
                uint32_t pull_div, uint32_t* vis_f, uint32_t* vis_b, uint32_t* rounds_f,
                uint32_t* rounds_b, uint64_t* n_zeros) {
  Side s[2] = {make_side(false, vis_f, 0), make_side(true, vis_b, 1)};
  PSC_TRY(reach_sides(g, s, 2, nullptr, local, tau ? tau : 512, pull_div, P, 1, 0, zeros, n_zeros));
  if (rounds_f) *rounds_f = s[0].rounds;
  if (rounds_b) *rounds_b = s[1].rounds;
  return PSC_OK;
}

int reach_pair_multi(psc_graph_s* g, const uint32_t* d_srcs, uint64_t n_srcs, bool local,
                     uint32_t tau, uint32_t pull_div, uint32_t* vis_f, uint32_t* vis_b,
                     uint32_t* rounds_f, uint32_t* rounds_b, uint64_t vgc_max) {
  Side s[2] = {make_side(false, vis_f, 0), make_side(true, vis_b, 1)};
  PSC_TRY(reach_sides(g, s, 2, nullptr, local, tau ? tau : 512, pull_div, d_srcs, n_srcs, vgc_max));
  if (rounds_f) *rounds_f = s[0].rounds;
  if (rounds_b) *rounds_b = s[1].rounds;
  return PSC_OK;
}

}  // namespace psc

using namespace psc;

extern "C" int psc_reach(psc_graph_t g, uint32_t src, int dir, int local, uint32_t tau,
                         uint8_t* dst_out, uint32_t* rounds) {
  if (!g || !dst_out || src >= g->n || (dir != 0 && dir != 1)) return PSC_ERR_INVALID;
  CallScope scope(g->device);
  PSC_TRY(call_begin(g));
  uint32_t* vis;
  uint8_t* bytes;
  PSC_TRY(ensure_t(g, B_VIS_F, (g->n + 31) / 32 + 1, &vis));
  PSC_TRY(ensure_t(g, B_AUX0, g->n, &bytes));
  uint32_t r = 0;
  PSC_TRY(reach_run(g, src, dir == 1, local != 0, tau ? tau : 512, 0, vis, &r));
  k_bitmap_to_bytes<<<grid_for(g, g->n, 256), 256, 0, g->stream>>>(vis, g->n, bytes);
  PSC_CUDA(cudaMemcpyAsync(dst_out, bytes, g->n, cudaMemcpyDeviceToHost, g->stream));
  g->stats.reach_rounds = r;
  if (rounds) *rounds = r;
  return call_end(g);
}

// ---------------------------------------------------------------------------
// psc_reach_noalloc: the same reach kernels with their scratch in one
// file-scope device array instead of allocated buffers.
// ---------------------------------------------------------------------------
namespace psc {

constexpr uint64_t kNaMaxN = PSC_NOALLOC_MAX_VERTICES;
constexpr uint64_t kNaWords = kNaMaxN / 32;
// Region sizes are multiples of 64 u32 (256 bytes) so every region, and the
// Counters block at the end, starts 256-byte aligned.
constexpr size_t kNaBitmap = kNaWords + 64;
constexpr size_t kNaQueue = kNaMaxN + 64;
constexpr size_t kNaVis = 0;
constexpr size_t kNaFa = kNaVis + kNaBitmap;
constexpr size_t kNaFb = kNaFa + kNaBitmap;
constexpr size_t kNaQa = kNaFb + kNaBitmap;
constexpr size_t kNaQb = kNaQa + kNaQueue;
constexpr size_t kNaHeavy = kNaQb + kNaQueue;  // u64 entries: two u32 per vertex
constexpr size_t kNaCtr = kNaHeavy + 2 * kNaQueue;
constexpr size_t kNaTotal = kNaCtr + 64;
static_assert(sizeof(Counters) <= 64 * sizeof(uint32_t), "counters fit their region");
static_assert(kNaCtr % 64 == 0, "256-byte aligned counters");

static __device__ __align__(256) uint32_t g_noalloc_scratch[kNaTotal];

struct NoAllocDevice {
  uint32_t* scratch = nullptr;
  int num_sms = 0;
  bool ready = false;
};
constexpr int kNaMaxDevices = 64;
static NoAllocDevice g_na_dev[kNaMaxDevices];
static std::mutex g_na_mu;

// Once per device, with that device current: the array's device address.
static int noalloc_setup(int dev, NoAllocDevice* out) {
  if (dev < 0 || dev >= kNaMaxDevices) return PSC_ERR_INVALID;
  std::lock_guard<std::mutex> lock(g_na_mu);
  NoAllocDevice& d = g_na_dev[dev];
  if (!d.ready) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e);
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_status(e);
    d.scratch = (uint32_t*)p;
    d.num_sms = sms;
    d.ready = true;
  }
  *out = d;
  return PSC_OK;
}

static unsigned na_grid(int sms, uint64_t items, unsigned block) {
  uint64_t want = (items + block - 1) / block;
  uint64_t cap = (uint64_t)sms * 16;
  if (want < 1) want = 1;
  if (want > cap) want = cap;
  return (unsigned)want;
}

}  // namespace psc

extern "C" int psc_reach_noalloc(const uint64_t* d_off, const uint32_t* d_E,
                                 const uint64_t* d_in_off, const uint32_t* d_in_E, uint64_t n,
                                 uint64_t m, uint32_t src, int dir, uint8_t* d_dst, void* stream,
                                 uint32_t* rounds) {
  if (n > kNaMaxN || (m >> 36)) return PSC_ERR_TOO_LARGE;
  if (!d_off || (m && !d_E) || !d_dst || n == 0 || src >= n || (dir != 0 && dir != 1))
    return PSC_ERR_INVALID;
  if ((d_in_off == nullptr) != (d_in_E == nullptr)) return PSC_ERR_INVALID;
  if (!d_in_off) {  // symmetric: the transpose is the graph itself
    d_in_off = d_off;
    d_in_E = d_E;
  }
  int dev = 0;
  PSC_CUDA(cudaGetDevice(&dev));
  NoAllocDevice nd;
  PSC_TRY(noalloc_setup(dev, &nd));
  cudaStream_t s = (cudaStream_t)stream;
  const bool backward = dir == 1;
  const uint64_t* A_off = backward ? d_in_off : d_off;
  const uint32_t* A_E = backward ? d_in_E : d_E;
  const uint64_t* B_off = backward ? d_off : d_in_off;
  const uint32_t* B_E = backward ? d_E : d_in_E;
  const uint64_t nwords = (n + 31) / 32;
  uint32_t* vis = nd.scratch + kNaVis;
  uint32_t* fa = nd.scratch + kNaFa;
  uint32_t* fb = nd.scratch + kNaFb;
  uint32_t* qa = nd.scratch + kNaQa;
  uint32_t* qb = nd.scratch + kNaQb;
  uint64_t* heavy = (uint64_t*)(nd.scratch + kNaHeavy);
  Counters* ctr = (Counters*)(nd.scratch + kNaCtr);
  Counters hc;  // host copy of the counters (stack memory)

  // the caller's arrays are checked before any kernel indexes by them (the
  // check of psc_graph_upload; the flag is a word of the counters region)
  PSC_CUDA(cudaMemsetAsync(ctr, 0, sizeof(Counters), s));
  const unsigned vgrid = na_grid(nd.num_sms, std::max<uint64_t>(n, m), 256);
  k_validate_csr<><<<vgrid, 256, 0, s>>>(d_off, n, d_E, m, &ctr->aux0);
  if (d_in_off != d_off)
    k_validate_csr<><<<vgrid, 256, 0, s>>>(d_in_off, n, d_in_E, m, &ctr->aux0);
  PSC_CUDA(cudaGetLastError());
  PSC_CUDA(cudaMemcpyAsync(&hc, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, s));
  PSC_CUDA(cudaStreamSynchronize(s));
  if (hc.aux0) return PSC_ERR_INVALID;
  // the array keeps the previous call's contents: clear the visited bitmap
  PSC_CUDA(cudaMemsetAsync(vis, 0, nwords * 4, s));
  k_reach_init<<<1, 1, 0, s>>>(vis, qa, src);
  const uint64_t threshold = m / 20;
  uint64_t nf = 1, nf_edges = 0;
  LvGate gate;
  bool pull = false;
  uint32_t r = 0;
  const bool cluster = levels_ready<ReachClaim>(dev);
  while (nf > 0) {
    const bool want_pull = (nf + nf_edges) >= threshold;
    // narrow push rounds run back to back on one cluster (levels.cuh)
    if (cluster && !want_pull && !pull && gate.enter(r, nf, nf_edges)) {
      PSC_CUDA(cudaMemsetAsync(ctr, 0, sizeof(Counters), s));
      PSC_TRY(launch_levels(LvArgs{A_off, A_E, qa, nf, qb, threshold, r, ctr}, ReachClaim{vis}, s));
      PSC_CUDA(cudaMemcpyAsync(&hc, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, s));
      PSC_CUDA(cudaStreamSynchronize(s));
      gate.ran(hc.aux0);
      if (hc.aux0) {  // else the first round was too wide: one of the whole grid
        r += (uint32_t)hc.aux0;
        if (r > n + 2) return PSC_ERR_ITER_LIMIT;
        std::swap(qa, qb);
        nf = hc.next;
        nf_edges = hc.next_edges;
        continue;
      }
    }
    r++;
    if (r > n + 2) return PSC_ERR_ITER_LIMIT;
    if (want_pull && !pull) {
      PSC_CUDA(cudaMemsetAsync(fa, 0, nwords * 4, s));
      k_queue_to_bitmap<<<na_grid(nd.num_sms, nf, 256), 256, 0, s>>>(qa, nf, fa);
      pull = true;
    } else if (!want_pull && pull) {
      PSC_CUDA(cudaMemsetAsync(ctr, 0, sizeof(Counters), s));
      k_bitmap_to_queue<<<na_grid(nd.num_sms, nwords, 256), 256, 0, s>>>(fa, nwords, qa, ctr);
      pull = false;
      gate.pulled();
    }
    PSC_CUDA(cudaMemsetAsync(ctr, 0, sizeof(Counters), s));
    if (!pull) {
      ReachSide side{A_off, A_E, qa, nf, vis, qb, heavy, ctr};
      ReachSide none{};
      k_reach_push<kReachBlock><<<na_grid(nd.num_sms, nf, kReachBlock), kReachBlock, 0, s>>>(side,
                                                                                          none);
      PSC_CUDA(cudaGetLastError());
      PSC_CUDA(cudaMemcpyAsync(&hc, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, s));
      PSC_CUDA(cudaStreamSynchronize(s));
      // vertices above the heavy threshold were listed: the whole grid
      // expands them before the round ends
      if (hc.heavy)
        k_reach_heavy<kReachBlock><<<nd.num_sms * 4, kReachBlock, 0, s>>>(side, none);
      std::swap(qa, qb);
      if (!hc.heavy) {
        nf = hc.next;
        nf_edges = hc.next_edges;
        continue;
      }
    } else {
      launch_pull<kReachBlock>(nd.num_sms, s, B_off, B_E, fa, vis, fb, n, ctr, nullptr);
      k_pull_out_edges<<<na_grid(nd.num_sms, nwords, 256), 256, 0, s>>>(fb, A_off, n,
                                                                        hash32(r), ctr);
      std::swap(fa, fb);
    }
    PSC_CUDA(cudaGetLastError());
    PSC_CUDA(cudaMemcpyAsync(&hc, ctr, sizeof(Counters), cudaMemcpyDeviceToHost, s));
    PSC_CUDA(cudaStreamSynchronize(s));
    nf = hc.next;
    nf_edges = hc.next_edges;
  }
  k_bitmap_to_bytes<<<na_grid(nd.num_sms, n, 256), 256, 0, s>>>(vis, n, d_dst);
  PSC_CUDA(cudaGetLastError());
  PSC_CUDA(cudaStreamSynchronize(s));
  if (rounds) *rounds = r;
  return PSC_OK;
}
