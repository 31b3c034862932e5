// Multi-search on the device (SCC::multi_search / multi_search_safe,
// src/scc.hpp:144-275), forward and backward in the same launches.
//
// Per direction ("side") the state is the closure table {(v, pivot)} — 64-bit
// keys v<<32 | pivot label in an open-addressing table with linear probing
// and atomicCAS inserts (the reference's resizable_table, keyed here by the
// hash of the whole pair) — and a frontier of pairs that are new to the table.
// A sub-round offers each frontier pair (u, l) to every out-neighbour w of u
// inside u's subproblem (labels[w] == labels[u]); new pairs form the next
// frontier, so each pair is expanded once.  The closure, and therefore the
// partition, is the reference's.
//
//   VGC (scc.hpp:177-219): while a side's frontier is small, one pair per
//     warp runs a local BFS for its pivot in a shared-memory queue (entries
//     carry the vertex's adjacency range, loaded alongside the claim), up to
//     tau vertices, spilling the rest as pairs;
//   expand: larger frontiers, 32 pairs per warp step with the balanced
//     expansion;
//   heavy: pairs of vertices with more than kHeavyDeg out-edges, expanded by
//     the whole grid.
// Claims are batched: a lane loads K target ids, then their labels (and in
// VGC their adjacency ranges), then issues the first table probes, so the
// memory round trips of K edges overlap.
//
// Table growth: the host keeps the load at most 1/2 between sub-rounds.  An
// insert that still gives up (kProbeLimit probes) re-queues its source pair;
// the host grows the table before the next sub-round and the pair is expanded
// again, finding the pairs it already placed.  This replaces the reference's
// restart of the whole search (scc.hpp:263-272) with the same fixed point.
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "common.cuh"
#include "engines.cuh"

namespace psc {

constexpr int kMsBlock = 256;
constexpr int kMsVgcBlock = 128;
constexpr int kMsVgcQueue = 512;
constexpr int kMsK = 8;        // VGC: edges in flight per lane
constexpr int kMsExpandK = 4;  // expand: fewer registers, more warps
// An insert gives up after this many probes: the table is too full.  Every further insert
// of the sub-round would spend as many, so the work at hand stops there and comes back
// as pairs, after the table has grown (4 R-MAT and kNN graphs of 2^16 to 2^20 vertices in
// a batch, a first pivot outside the giant component, so that hubs meet the small tables of
// a first batch: 129 -> 5.7 ms of multi-search).
constexpr uint32_t kProbeLimit = 256;

struct MsSide {
  const uint64_t* off;
  const uint32_t* E;
  const uint64_t* Fin;  // frontier pairs
  uint64_t nin;
  unsigned long long* T;
  uint64_t mask;
  uint64_t* Fout;
  uint64_t* Fheavy;
  uint32_t* hflag;
  Counters* ctr;
  uint32_t vgc_budget;  // new pairs one VGC local search may insert
};

constexpr int kMsHeavyK = 4;  // heavy pairs: edges in flight per lane
constexpr uint64_t kMsHeavyChunk = 32 * kMsHeavyK;
constexpr uint32_t kRequeued = 0x80000000u;  // hflag bit: the pair was re-queued

// Lists a pair whose vertex has more than kHeavyDeg out-edges for k_ms_heavy.
// Its edges are cut into chunks of kMsHeavyChunk; one 64-bit atomic on
// ctr->heavy = count << kPackShift | chunks gives the pair its slot and its
// first chunk (hflag, below the kRequeued bit), increasing with the slot.
__device__ __forceinline__ void ms_heavy_push(const MsSide& S, uint64_t key, uint64_t deg) {
  const unsigned long long old = atomicAdd(
      &S.ctr->heavy, (1ull << kPackShift) + (deg + kMsHeavyChunk - 1) / kMsHeavyChunk);
  const uint64_t hh = old >> kPackShift;
  S.Fheavy[hh] = key;
  S.hflag[hh] = (uint32_t)(old & kPackMask);
}

// Per-warp source data of one expansion step.
struct MsSrc {
  uint64_t sub[32];
  uint32_t lab[32];
  uint32_t fail;
};

// Seeds both sides of a batch: pair (front[i], label) into each side's table
// and frontier.
__global__ void k_ms_seed(const uint32_t* __restrict__ front, uint64_t nf, uint64_t label_offset,
                          const uint32_t* __restrict__ front_labels, unsigned long long* T0,
                          uint64_t mask0, uint64_t* F0, unsigned long long* T1, uint64_t mask1,
                          uint64_t* F1) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nf;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t lab = front_labels ? front_labels[i] : (uint32_t)(label_offset + i);
    const uint64_t key = ((uint64_t)front[i] << 32) | (uint64_t)lab;
    uint32_t pr = 0;
    table_insert(T0, mask0, key, (uint32_t)(mask0 + 1 < 0xFFFFFFFFull ? mask0 + 1 : 0xFFFFFFFFu), &pr);
    table_insert(T1, mask1, key, (uint32_t)(mask1 + 1 < 0xFFFFFFFFull ? mask1 + 1 : 0xFFFFFFFFu), &pr);
    F0[i] = key;
    F1[i] = key;
  }
}

__global__ void k_rehash(const unsigned long long* __restrict__ T, uint64_t cap,
                         unsigned long long* T2, uint64_t mask2) {
  uint32_t pr = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint64_t e = T[i];
    if (e != kEmpty) table_insert(T2, mask2, e, 0xFFFFFFFFu, &pr);
  }
}

// Linear probing from slot h (the first probe is already done by the caller).
__device__ __forceinline__ int table_insert_from(unsigned long long* T, uint64_t mask, uint64_t key,
                                                 uint64_t h, uint32_t limit, uint32_t* probes) {
  for (uint32_t i = 0; i < limit; i++) {
    h = (h + 1) & mask;
    uint64_t cur = __ldcg(&T[h]);
    if (cur == key) {
      *probes += i + 1;
      return 0;
    }
    if (cur == kEmpty) {
      uint64_t old = atomicCAS(&T[h], (unsigned long long)kEmpty, (unsigned long long)key);
      if (old == kEmpty) {
        *probes += i + 1;
        return 1;
      }
      if (old == key) {
        *probes += i + 1;
        return 0;
      }
    }
  }
  *probes += limit;
  return -1;
}

// Batched claim over the 32 lanes' adjacency ranges (K edges per lane in
// flight).  A candidate w of source lane s is offered pivot src.lab[s] if
// labels[w] == src.sub[s].  DIRECT: the first probe is an atomicCAS (one
// round trip, for latency-bound rounds); otherwise a load, then a CAS only on
// an empty slot.  PF: also load w's adjacency range.  A failed insert sets bit
// s of src.fail.  emit(tm, keys) gets the lane's K candidate pairs and the mask
// of those newly inserted (warp-collective).
template <int K, bool DIRECT, bool PF, class Emit>
__device__ __forceinline__ void ms_expand_claim(WarpExpandSmem& sm, MsSrc& src, uint64_t beg,
                                                uint32_t deg, const uint64_t* __restrict__ off,
                                                const uint32_t* __restrict__ E,
                                                const uint64_t* labels,
                                                unsigned long long* T, uint64_t mask,
                                                uint32_t& probes, Emit&& emit) {
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
    uint32_t w[K];
    int sl[K];
    uint64_t key[K], old[K], h[K], vb[K], ve[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t gi = base + k * 32 + lane;
      w[k] = 0xFFFFFFFFu;
      sl[k] = 0;
      if (gi < total) {
        int lo = 0, hi = 31;
        while (lo < hi) {
          int mid = (lo + hi + 1) >> 1;
          if (sm.excl[mid] <= gi)
            lo = mid;
          else
            hi = mid - 1;
        }
        sl[k] = lo;
        w[k] = __ldg(&E[sm.beg[lo] + (gi - sm.excl[lo])]);
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      key[k] = kEmpty;
      vb[k] = ve[k] = 0;
      if (w[k] != 0xFFFFFFFFu) {
        const uint64_t lw = ld_cg(&labels[w[k]]);
        if (PF) {
          vb[k] = __ldg(&off[w[k]]);
          ve[k] = __ldg(&off[w[k] + 1]);
        }
        if (lw == src.sub[sl[k]]) key[k] = ((uint64_t)w[k] << 32) | src.lab[sl[k]];
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      old[k] = kEmpty;
      h[k] = 0;
      if (key[k] != kEmpty) {
        h[k] = hash64(key[k]) & mask;
        if (DIRECT)
          old[k] = atomicCAS(&T[h[k]], (unsigned long long)kEmpty, (unsigned long long)key[k]);
        else
          old[k] = __ldcg(&T[h[k]]);
      }
    }
    uint32_t tm = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (key[k] != kEmpty) {
        int r;
        probes++;
        if (DIRECT) {
          r = old[k] == kEmpty ? 1 : old[k] == key[k] ? 0
                                  : table_insert_from(T, mask, key[k], h[k], kProbeLimit - 1, &probes);
        } else if (old[k] == key[k]) {
          r = 0;
        } else if (old[k] == kEmpty) {
          const uint64_t o2 =
              atomicCAS(&T[h[k]], (unsigned long long)kEmpty, (unsigned long long)key[k]);
          r = o2 == kEmpty ? 1 : o2 == key[k] ? 0
                             : table_insert_from(T, mask, key[k], h[k], kProbeLimit - 1, &probes);
        } else {
          r = table_insert_from(T, mask, key[k], h[k], kProbeLimit - 1, &probes);
        }
        if (r == 1) tm |= 1u << k;
        if (r < 0) atomicOr(&src.fail, 1u << sl[k]);
      }
    }
    emit(tm, key);
  }
  __syncwarp();
}

__device__ __forceinline__ void flush_ms_counters(Counters* c0, Counters* c1,
                                                  unsigned long long s0, unsigned long long s1,
                                                  unsigned long long r0, unsigned long long r1,
                                                  unsigned long long p0, unsigned long long p1,
                                                  unsigned long long x0, unsigned long long x1,
                                                  unsigned long long i0, unsigned long long i1) {
  i0 = warp_sum(i0);
  i1 = warp_sum(i1);
  if (lane_id() == 0) {
    if (i0) atomicAdd(&c0->inserted, i0);
    if (i1) atomicAdd(&c1->inserted, i1);
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  r0 = warp_sum(r0);
  r1 = warp_sum(r1);
  p0 = warp_sum(p0);
  p1 = warp_sum(p1);
  x0 = warp_sum(x0);
  x1 = warp_sum(x1);
  if (lane_id() == 0) {
    if (s0 | r0 | p0 | x0) {
      atomicAdd(&c0->edges, s0);
      atomicAdd(&c0->probes, p0);
      atomicAdd(&c0->expanded, x0);
      if (r0) {
        atomicAdd(&c0->fail, r0);
        atomicAdd(&c0->aux1, r0);
      }
    }
    if (s1 | r1 | p1 | x1) {
      atomicAdd(&c1->edges, s1);
      atomicAdd(&c1->probes, p1);
      atomicAdd(&c1->expanded, x1);
      if (r1) {
        atomicAdd(&c1->fail, r1);
        atomicAdd(&c1->aux1, r1);
      }
    }
  }
}

// Expansion sub-round for up to two sides: 32 pairs per warp step (warp gw of
// nw, with its own sm and src).
__device__ __forceinline__ void ms_expand_round(const MsSide& s0, const MsSide& s1,
                                                const uint64_t* labels, WarpExpandSmem& sm,
                                                MsSrc& src, uint64_t gw, uint64_t nw) {
  const unsigned lane = lane_id();
  const uint64_t c0 = (s0.nin + 31) / 32, c1 = (s1.nin + 31) / 32;
  unsigned long long sc0 = 0, sc1 = 0, rq0 = 0, rq1 = 0, ex0 = 0, ex1 = 0, in0 = 0, in1 = 0;
  uint32_t pr0 = 0, pr1 = 0;
  for (uint64_t c = gw; c < c0 + c1; c += nw) {
    const int sd = c < c0 ? 0 : 1;
    const MsSide S = sd ? s1 : s0;
    const uint64_t i = (sd ? c - c0 : c) * 32 + lane;
    uint64_t beg = 0, key = 0, sub = 0;
    uint32_t deg = 0;
    if (i < S.nin) {
      key = ld_cg(&S.Fin[i]);
      const uint32_t u = (uint32_t)(key >> 32);
      beg = S.off[u];
      uint64_t d = S.off[u + 1] - beg;
      sub = ld_cg(&labels[u]);
      (sd ? ex1 : ex0)++;
      if (d > kHeavyDeg) {
        ms_heavy_push(S, key, d);
        d = 0;
      }
      deg = (uint32_t)d;
    }
    (sd ? sc1 : sc0) += deg;
    src.sub[lane] = sub;
    src.lab[lane] = (uint32_t)key;
    if (lane == 0) src.fail = 0;
    __syncwarp();
    uint32_t probes = 0;
    ms_expand_claim<kMsExpandK, false, false>(
        sm, src, beg, deg, S.off, S.E, labels, S.T, S.mask, probes,
        [&](uint32_t tm, const uint64_t* keys) {
          (sd ? in1 : in0) += __popc(tm);
          warp_append_batch<kMsExpandK>(tm, keys, S.Fout, &S.ctr->next);
        });
    (sd ? pr1 : pr0) += probes;
    __syncwarp();
    const bool rq = (src.fail >> lane) & 1u;
    unsigned long long pos = warp_append(&S.ctr->next, rq);
    if (rq) {
      S.Fout[pos] = key;
      (sd ? rq1 : rq0)++;
    }
    __syncwarp();
  }
  flush_ms_counters(s0.ctr, s1.ctr, sc0, sc1, rq0, rq1, pr0, pr1, ex0, ex1, in0, in1);
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, (768 / BLOCK) > 0 ? (768 / BLOCK) : 1)
    k_ms_expand(MsSide s0, MsSide s1, const uint64_t* labels) {
  __shared__ WarpExpandSmem sm[BLOCK / 32];
  __shared__ MsSrc ssrc[BLOCK / 32];
  const unsigned wid = threadIdx.x >> 5;
  ms_expand_round(s0, s1, labels, sm[wid], ssrc[wid],
                  (uint64_t)blockIdx.x * (BLOCK / 32) + wid, (uint64_t)gridDim.x * (BLOCK / 32));
}

struct MsQEnt {
  uint64_t beg;
  uint32_t v;
  uint32_t deg;
};

// Claims of one batch for pivot lab inside subproblem sub: each candidate's
// label and adjacency range are loaded together, then the first table probes
// (atomicCAS) of all K candidates are issued before any is resolved.  Returns
// the mask of new pairs; failed: the mask of inserts that gave up.
template <int K, bool ADJ = true>
__device__ __forceinline__ uint32_t ms_vgc_claim(const uint32_t* w, uint64_t* vb, uint64_t* ve,
                                                 uint64_t sub, uint32_t lab,
                                                 const uint64_t* __restrict__ off,
                                                 const uint64_t* labels,
                                                 unsigned long long* T, uint64_t mask,
                                                 uint32_t& probes, uint32_t& failed) {
  uint64_t key[K], old[K], h[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    key[k] = kEmpty;
    vb[k] = ve[k] = 0;
    if (w[k] != 0xFFFFFFFFu) {
      const uint64_t lw = ld_cg(&labels[w[k]]);
      if (ADJ) {
        vb[k] = __ldg(&off[w[k]]);
        ve[k] = __ldg(&off[w[k] + 1]);
      }
      if (lw == sub) key[k] = ((uint64_t)w[k] << 32) | lab;
    }
  }
#pragma unroll
  for (int k = 0; k < K; k++) {
    old[k] = kEmpty;
    h[k] = 0;
    if (key[k] != kEmpty) {
      h[k] = hash64(key[k]) & mask;
      old[k] = atomicCAS(&T[h[k]], (unsigned long long)kEmpty, (unsigned long long)key[k]);
    }
  }
  uint32_t tm = 0;
#pragma unroll
  for (int k = 0; k < K; k++)
    if (key[k] != kEmpty) {
      probes++;
      const int r = old[k] == kEmpty ? 1 : old[k] == key[k] ? 0
                    : table_insert_from(T, mask, key[k], h[k], kProbeLimit - 1, &probes);
      if (r == 1) tm |= 1u << k;
      if (r < 0) failed |= 1u << k;
    }
  return tm;
}

// Places this lane's new pairs (bit k of tm) into the warp's queue while it
// has room, then spills (w, lab) pairs: a ballot per step, at most one atomic.
// Returns the warp's new pairs.
template <int K>
__device__ __forceinline__ uint32_t ms_vgc_place(uint32_t tm, const uint32_t* w, const uint64_t* vb,
                                                 const uint64_t* ve, uint32_t lab, MsQEnt* Q,
                                                 uint32_t& tail, uint32_t tq, uint64_t* Fout,
                                                 unsigned long long* next_ctr) {
  const unsigned lane = lane_id();
  unsigned m[K];
  uint32_t total = 0;
#pragma unroll
  for (int k = 0; k < K; k++) {
    m[k] = __ballot_sync(kFull, (tm >> k) & 1u);
    total += __popc(m[k]);
  }
  if (total == 0) return 0;
  const uint32_t room = tq - tail;
  const uint32_t nloc = total < room ? total : room;
  unsigned long long sbase = 0;
  if (total > nloc) {
    if (lane == 0) sbase = atomicAdd(next_ctr, (unsigned long long)(total - nloc));
    sbase = __shfl_sync(kFull, sbase, 0);
  }
  uint32_t b = 0;
#pragma unroll
  for (int k = 0; k < K; k++) {
    if ((m[k] >> lane) & 1u) {
      const uint32_t r = b + __popc(m[k] & ((1u << lane) - 1u));
      if (r < nloc) {
        const uint64_t vd = ve[k] - vb[k];
        Q[tail + r] = MsQEnt{vb[k], w[k], (uint32_t)(vd < 0xFFFFFFFFull ? vd : 0xFFFFFFFFull)};
      } else {
        Fout[sbase + (r - nloc)] = ((uint64_t)w[k] << 32) | lab;
      }
    }
    b += __popc(m[k]);
  }
  tail += nloc;
  __syncwarp();
  return total;
}

// VGC sub-round for up to two sides: one frontier pair (u, l) per warp.  If
// 0 < deg(u) < tau the warp runs a local BFS for pivot l inside u's
// subproblem in a shared-memory queue of tq = min(tau, QCAP) vertices: each
// wave offers l along the edges of up to 32 queued vertices (while those have at
// most 8 out-edges, eight lanes per vertex and up to 4 K vertices, else the
// balanced expansion over all of them); a new
// pair stays in the queue while there is room, else spills to the next
// frontier.  Queued vertices with more than tq out-edges and the queue's
// remainder spill too.  A queued vertex whose expansion hit a failed insert is
// re-queued as a pair, and the search ends there.
// (warp gw of nw, with its own sm and queue Q; kMsK edges in flight per lane)
template <int kMsK, int QCAP>
__device__ __forceinline__ void ms_vgc_round(const MsSide& s0, const MsSide& s1,
                                             const uint64_t* labels, uint32_t tau,
                                             WarpExpandSmem& sm, MsQEnt* Q, uint64_t gw,
                                             uint64_t nw) {
  const unsigned lane = lane_id();
  const uint32_t tq = tau < (uint32_t)QCAP ? tau : (uint32_t)QCAP;
  unsigned long long sc0 = 0, sc1 = 0, rq0 = 0, rq1 = 0, ex0 = 0, ex1 = 0, in0 = 0, in1 = 0;
  uint32_t pr0 = 0, pr1 = 0;
  if (lane == 0) sm.fail = 0;
  __syncwarp();
  for (uint64_t i = gw; i < s0.nin + s1.nin; i += nw) {
    const int sd = i < s0.nin ? 0 : 1;
    const MsSide S = sd ? s1 : s0;
    const uint64_t key = ld_cg(&S.Fin[sd ? i - s0.nin : i]);
    const uint32_t u = (uint32_t)(key >> 32);
    const uint32_t lab = (uint32_t)key;
    const uint64_t sub = ld_cg(&labels[u]);
    const uint64_t ub = S.off[u], ue = S.off[u + 1];
    const uint64_t du = ue - ub;
    auto emit = [&](bool take, uint32_t w) {
      unsigned long long pos = warp_append(&S.ctr->next, take);
      if (take) S.Fout[pos] = ((uint64_t)w << 32) | lab;
    };
    if (lane == 0) (sd ? ex1 : ex0)++;
    uint32_t probes = 0;
    if (!(du > 0 && du < tq)) {
      if (du > kHeavyDeg) {
        if (lane == 0) ms_heavy_push(S, key, du);
        continue;
      }
      // a vertex with tau..kHeavyDeg out-edges: the warp walks them with
      // kMsK edges per lane in flight
      if (lane == 0) (sd ? sc1 : sc0) += du;
      bool failed = false;
      for (uint64_t b = ub; b < ue; b += 32 * kMsK) {
        uint32_t w[kMsK];
        uint64_t vb[kMsK], ve[kMsK], keys[kMsK];
#pragma unroll
        for (int k = 0; k < kMsK; k++) {
          const uint64_t e = b + k * 32 + lane;
          w[k] = e < ue ? __ldg(&S.E[e]) : 0xFFFFFFFFu;
        }
        uint32_t fm = 0;
        const uint32_t tm = ms_vgc_claim<kMsK, false>(w, vb, ve, sub, lab, S.off, labels, S.T,
                                                      S.mask, probes, fm);
        (sd ? in1 : in0) += __popc(tm);
#pragma unroll
        for (int k = 0; k < kMsK; k++) keys[k] = ((uint64_t)w[k] << 32) | lab;
        warp_append_batch<kMsK>(tm, keys, S.Fout, &S.ctr->next);
        failed = __any_sync(kFull, fm != 0);
        if (failed) break;  // (the pair comes back whole: see kProbeLimit)
      }
      (sd ? pr1 : pr0) += probes;
      const bool rq = failed && lane == 0;
      emit(rq, u);
      if (rq) (sd ? rq1 : rq0)++;
      continue;
    }
    if (lane == 0) Q[0] = MsQEnt{ub, u, (uint32_t)du};
    __syncwarp();
    // the local search stops at tq queued vertices, or once it has inserted
    // its share of the table's free room (the first wave always runs)
    uint32_t head = 0, tail = 1, ins = 0;
    while (head < tail && tail < tq && (head == 0 || ins < S.vgc_budget)) {
      uint32_t wave = min(32u, tail - head);
      uint64_t beg = 0;
      uint32_t deg = 0, x = 0;
      if (lane < wave) {
        const MsQEnt q = Q[head + lane];
        x = q.v;
        beg = q.beg;
        deg = q.deg;
      }
      const uint32_t head0 = head;
      bool fk = false;  // an insert of this lane failed
      if (!__any_sync(kFull, deg > 8)) {
        // eight lanes per vertex, lane j takes its target j (no scan, no search)
        wave = min(wave, 4u * kMsK);
        head += wave;
        const unsigned grp = lane >> 3, j = lane & 7;
        uint32_t w[kMsK];
        uint64_t vb[kMsK], ve[kMsK];
#pragma unroll
        for (int k = 0; k < kMsK; k++) {
          w[k] = 0xFFFFFFFFu;
          if (4 * k + grp < wave) {
            const MsQEnt& q = Q[head0 + 4 * k + grp];
            if (j < q.deg) w[k] = __ldg(&S.E[q.beg + j]);
          }
        }
        if (lane < wave) {
          (sd ? sc1 : sc0) += deg;
          if (head0 + lane > 0) (sd ? ex1 : ex0)++;
        }
        uint32_t fm = 0;
        const uint32_t tm = ms_vgc_claim<kMsK>(w, vb, ve, sub, lab, S.off, labels, S.T, S.mask,
                                               probes, fm);
        if (fm) {
          fk = true;
#pragma unroll
          for (int k = 0; k < kMsK; k++)
            if ((fm >> k) & 1u) atomicOr(&sm.fail, 1u << (4 * k + grp));
        }
        (sd ? in1 : in0) += __popc(tm);
        ins += ms_vgc_place<kMsK>(tm, w, vb, ve, lab, Q, tail, tq, S.Fout, &S.ctr->next);
      } else {
        head += wave;
        const bool spill_self = deg > tq;
        if (spill_self) deg = 0;
        if (lane < wave && head0 + lane > 0) (sd ? ex1 : ex0)++;
        if (__any_sync(kFull, spill_self)) emit(spill_self, x);
        (sd ? sc1 : sc0) += deg;
        uint32_t incl = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(kFull, incl, o);
          if ((int)lane >= o) incl += t;
        }
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        sm.excl[lane] = incl - deg;
        sm.beg[lane] = beg;
        __syncwarp();
        for (uint32_t base = 0; base < total; base += 32 * kMsK) {
          uint32_t w[kMsK];
          int sl[kMsK];
          uint64_t vb[kMsK], ve[kMsK];
#pragma unroll
          for (int k = 0; k < kMsK; k++) {
            const uint32_t gi = base + k * 32 + lane;
            w[k] = 0xFFFFFFFFu;
            sl[k] = 0;
            if (gi < total) {
              int lo = 0, hi = 31;
              while (lo < hi) {
                int mid = (lo + hi + 1) >> 1;
                if (sm.excl[mid] <= gi)
                  lo = mid;
                else
                  hi = mid - 1;
              }
              sl[k] = lo;
              w[k] = __ldg(&S.E[sm.beg[lo] + (gi - sm.excl[lo])]);
            }
          }
          uint32_t fm = 0;
          const uint32_t tm = ms_vgc_claim<kMsK>(w, vb, ve, sub, lab, S.off, labels, S.T, S.mask,
                                                 probes, fm);
          // a failure is charged to the source lane of the failed edge
          if (fm) {
            fk = true;
#pragma unroll
            for (int k = 0; k < kMsK; k++)
              if ((fm >> k) & 1u) atomicOr(&sm.fail, 1u << sl[k]);
          }
          (sd ? in1 : in0) += __popc(tm);
          ins += ms_vgc_place<kMsK>(tm, w, vb, ve, lab, Q, tail, tq, S.Fout, &S.ctr->next);
        }
      }
      (sd ? pr1 : pr0) += probes;
      probes = 0;
      __syncwarp();
      if (__any_sync(kFull, fk)) {  // a vertex with a failed insert comes back as a pair
        const bool rq = ((sm.fail >> lane) & 1u) && lane < wave;
        __syncwarp();
        if (lane == 0) sm.fail = 0;
        __syncwarp();
        emit(rq, x);
        if (rq) (sd ? rq1 : rq0)++;
        break;
      }
    }
    // spill what is left in the queue with one reservation
    const uint32_t rem = tail - head;
    if (rem) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&S.ctr->next, (unsigned long long)rem);
      base = __shfl_sync(kFull, base, 0);
      for (uint32_t k = lane; k < rem; k += 32)
        S.Fout[base + k] = ((uint64_t)Q[head + k].v << 32) | lab;
    }
    __syncwarp();
  }
  flush_ms_counters(s0.ctr, s1.ctr, sc0, sc1, rq0, rq1, pr0, pr1, ex0, ex1, in0, in1);
}

template <int BLOCK, int QCAP>
__global__ void __launch_bounds__(BLOCK)
    k_ms_vgc(MsSide s0, MsSide s1, const uint64_t* labels, uint32_t tau) {
  __shared__ WarpExpandSmem sm[BLOCK / 32];
  __shared__ MsQEnt sq[BLOCK / 32][QCAP];
  const unsigned wid = threadIdx.x >> 5;
  ms_vgc_round<kMsK, QCAP>(s0, s1, labels, tau, sm[wid], sq[wid],
                           (uint64_t)blockIdx.x * (BLOCK / 32) + wid,
                           (uint64_t)gridDim.x * (BLOCK / 32));
}

// Heavy pairs of both sides: the chunks of a side's heavy list are cut into
// one contiguous range per warp; a warp finds the pair of its first chunk
// once, then offers kMsHeavyChunk edges per step (a heavy pair has more than
// 64 chunks, so the next pair is at most one step away).  A step with a
// failed insert re-queues its pair once (kRequeued), whichever warp failed
// first.
__device__ __forceinline__ void ms_heavy_round(const MsSide& s0, const MsSide& s1,
                                               const uint64_t* labels, uint64_t gw, uint64_t nw) {
  constexpr int K = kMsHeavyK;
  const unsigned lane = lane_id();
#pragma unroll 1
  for (int sd = 0; sd < 2; sd++) {
    const MsSide S = sd ? s1 : s0;
    if (!S.ctr) continue;
    const unsigned long long packed = __ldcg(&S.ctr->heavy);
    const uint64_t nh = packed >> kPackShift, total = packed & kPackMask;
    const uint64_t per = (total + nw - 1) / nw;
    const uint64_t c_beg = gw * per, c_end = c_beg + per < total ? c_beg + per : total;
    if (nh == 0 || c_beg >= c_end) continue;
    // first chunks: hflag below the kRequeued bit (fixed while other warps set that bit)
    auto first_chunk = [&](uint64_t i) -> uint64_t { return ld_cg(&S.hflag[i]) & ~kRequeued; };
    uint64_t h = 0, hi = nh - 1;  // last pair whose first chunk is <= c_beg
    while (h < hi) {
      const uint64_t mid = (h + hi + 1) >> 1;
      if (first_chunk(mid) <= c_beg)
        h = mid;
      else
        hi = mid - 1;
    }
    uint64_t key = ld_cg(&S.Fheavy[h]), cs = first_chunk(h), cn = h + 1 < nh ? first_chunk(h + 1) : total;
    uint64_t sub = ld_cg(&labels[key >> 32]), beg = S.off[key >> 32], end = S.off[(key >> 32) + 1];
    unsigned long long scanned = 0, requeued = 0, ins = 0;
    uint32_t probes = 0;
    bool over = false;  // this warp has seen an insert of the pair fail
    for (uint64_t c = c_beg; c < c_end; c++) {
      if (over && c < cn) continue;
      if (c >= cn) {
        over = false;
        h++;
        key = ld_cg(&S.Fheavy[h]);
        cs = cn;
        cn = h + 1 < nh ? first_chunk(h + 1) : total;
        sub = ld_cg(&labels[key >> 32]);
        beg = S.off[key >> 32];
        end = S.off[(key >> 32) + 1];
      }
      const uint64_t e0 = beg + (c - cs) * kMsHeavyChunk;
      const uint32_t lab = (uint32_t)key;
      uint32_t w[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint64_t e = e0 + k * 32 + lane;
        w[k] = 0xFFFFFFFFu;
        if (e < end) {
          scanned++;
          w[k] = __ldg(&S.E[e]);
        }
      }
      uint64_t nk[K];
      uint32_t tm = 0;
      bool failed = false;
#pragma unroll
      for (int k = 0; k < K; k++) {
        nk[k] = 0;
        if (w[k] != 0xFFFFFFFFu && ld_cg(&labels[w[k]]) == sub) {
          nk[k] = ((uint64_t)w[k] << 32) | lab;
          const int r = table_insert(S.T, S.mask, nk[k], kProbeLimit, &probes);
          if (r == 1) tm |= 1u << k;
          failed |= r < 0;
        }
      }
      ins += __popc(tm);
      warp_append_batch<K>(tm, nk, S.Fout, &S.ctr->next);
      bool rq = false;
      over = __any_sync(kFull, failed);
      if (over && lane == 0) rq = !(atomicOr(&S.hflag[h], kRequeued) & kRequeued);
      const unsigned long long pos = warp_append(&S.ctr->next, rq);
      if (rq) {
        S.Fout[pos] = key;
        requeued++;
      }
    }
    scanned = warp_sum(scanned);
    requeued = warp_sum(requeued);
    ins = warp_sum(ins);
    const unsigned long long pr = warp_sum((unsigned long long)probes);
    if (lane == 0) {
      if (ins) atomicAdd(&S.ctr->inserted, ins);
      if (scanned) atomicAdd(&S.ctr->heavy_edges, scanned);
      if (pr) atomicAdd(&S.ctr->heavy_probes, pr);
      if (requeued) {
        atomicAdd(&S.ctr->fail, requeued);
        atomicAdd(&S.ctr->aux1, requeued);
      }
    }
  }
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
    k_ms_heavy(MsSide s0, MsSide s1, const uint64_t* labels) {
  ms_heavy_round(s0, s1, labels, (uint64_t)blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5),
                 (uint64_t)gridDim.x * (BLOCK / 32));
}

// ---------------------------------------------------------------------------
// Resident batches.  A prefix-doubling batch is small for most of a solve (1,
// 2, 3, 5, 8, ... pivots) and a chain of dependent steps: select the live
// centres of its window, seed the tables, sub-rounds until no pair is new,
// partition.  Launched step by step that costs about 8 launches and 2 waits, 60
// to 85 us per batch whatever it holds; here one cooperative launch of a block
// per SM runs batch after batch with a grid barrier (about 1.5 us) between
// steps, and every block takes the same decisions from the same counters.
// Two table sets alternate, so that the next batch's tables are cleared while
// this batch is partitioned.  A batch that outgrows its tables (load above 1/2 or
// a failed insert) ends the launch between two sub-rounds; the host grows tables
// and frontiers and the next launch goes on from there.  A window too large for
// the tables from the start goes to the host's full-width kernels (ms_pair).
// 12 warps a block, 2 edges in flight per lane: 16 warps (spills) and 4 edges were
// 5 to 7 % slower on kNN and grid.  Multi-search phase, before -> now: R-MAT 2^16
// (8 batches) 0.38 -> 0.12 ms, kNN 10^7 (26) 2.23 -> 1.20, 4096^2 grid (29) 3.52 ->
// 1.71, R-MAT 2^26 (24) 1.58 -> 0.56, 256-graph batch (19) 2.91 -> 1.53.
// ---------------------------------------------------------------------------
constexpr int kMbThreads = 384;
constexpr int kMbWarps = kMbThreads / 32;
constexpr int kMbK = 2;  // VGC edges in flight per lane
constexpr int kMbCtr = 4;    // counter sets 4-9: three sub-rounds in rotation, two sides
constexpr int kMbState = 16; // counter sets 16-17

enum MbWhy : uint32_t { MB_RUNNING = 0, MB_DONE = 1, MB_HOST = 2, MB_GROW = 3 };

struct MbState {
  uint32_t arrive, failed, why, pad;
  unsigned long long cur, step, label_offset, round, ne[2];
  unsigned long long batches, subrounds;
  unsigned long long edges, probes, expanded, pairs, heavy, heavy_edges, heavy_probes;
  unsigned long long slots;
  // a batch interrupted between two sub-rounds (MB_GROW)
  unsigned long long cap, nf, n0, n1, e0, e1;
  uint32_t set, buf;
  unsigned long long n_remaining;
};
static_assert(sizeof(MbState) <= 2 * sizeof(Counters) && kMbState + 2 <= kCounterSets,
              "the state fits its counter sets");

struct MbShared {
  MsQEnt q[kMbWarps][kMsVgcQueue];
  WarpExpandSmem sm[kMbWarps];
  MsSrc src[kMbWarps];
  uint32_t wcnt[kMbWarps + 1];
  uint32_t before, total;
};

struct MbArgs {
  const uint64_t *off, *in_off;
  const uint32_t *E, *in_E;
  uint64_t* labels;
  MsRun run;
  double beta;
  uint32_t tau;
  int local;
  uint64_t vgc_limit, cap_max;
  unsigned long long* T[2][2];  // [set][side]
  uint64_t* F[2][2];            // [side][buffer]
  uint64_t* Fh[2];
  uint32_t* hf[2];
  uint32_t* counts;  // per block
  // an interrupted batch to go on with (cap 0: none)
  uint64_t cap, nf, n0, n1, e0, e1;
  uint32_t set, buf;
  Counters* ctr;
  MbState* st;
};

// Slots of a batch's tables: at least 4 per candidate, 4 times the last
// batch's entries (batches grow by beta; twice, where that is a lot to clear and
// to scan), and room for VGC local searches.
__host__ __device__ inline uint64_t mb_cap(uint64_t window, uint64_t ne0, uint64_t ne1,
                                           uint64_t vgc_limit, uint32_t tau) {
  const uint64_t ne = ne0 > ne1 ? ne0 : ne1;
  const uint64_t vgc = window <= vgc_limit ? window * (tau < 64 ? tau : 64) : 0;
  const uint64_t last = ne <= (1ull << 18) ? 4 * ne : 2 * ne;
  uint64_t want = 4 * window > last ? 4 * window : last;
  const uint64_t room = 2 * (window + vgc);
  // (the VGC room is a wish: local searches stop at their share of the table)
  if (room > want) want = room < (1ull << 20) ? room : (want > (1ull << 20) ? want : (1ull << 20));
  uint64_t c = 1ull << 13;
  while (c < want) c <<= 1;
  return c;
}

__device__ __forceinline__ void mb_seed(unsigned long long* T0, unsigned long long* T1,
                                        uint64_t mask, uint64_t* F0, uint64_t* F1, uint64_t r,
                                        uint32_t v, uint32_t label) {
  const uint64_t key = ((uint64_t)v << 32) | label;
  uint32_t pr = 0;
  table_insert(T0, mask, key, 0xFFFFFFFFu, &pr);  // at most a quarter full
  table_insert(T1, mask, key, 0xFFFFFFFFu, &pr);
  F0[r] = key;
  F1[r] = key;
}

// GRAPHS: a batch of graphs (windows of many graphs per round).
template <bool GRAPHS>
__global__ void __launch_bounds__(kMbThreads, 1) k_ms_batches(MbArgs a) {
  extern __shared__ __align__(16) unsigned char mb_raw[];
  MbShared& sh = *reinterpret_cast<MbShared*>(mb_raw);
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5, tid = threadIdx.x;
  const uint64_t gw = (uint64_t)blockIdx.x * kMbWarps + wid, nw = (uint64_t)gridDim.x * kMbWarps;
  const uint64_t gt = (uint64_t)blockIdx.x * kMbThreads + tid, nt = (uint64_t)gridDim.x * kMbThreads;
  const bool lead = blockIdx.x == 0 && tid == 0;
  uint32_t target = 0;
  auto barrier = [&]() { return grid_barrier(&a.st->arrive, &a.st->failed, target); };
  if (lane == 0) sh.sm[wid].fail = 0;
  __syncwarp();

  if (a.run.n_rem_dev) a.run.n_remaining = *a.run.n_rem_dev;
  uint64_t cur = a.run.cur, step = a.run.step, label_offset = a.run.label_offset;
  uint64_t round = a.run.round, ne0 = a.run.ne[0], ne1 = a.run.ne[1];
  uint64_t batches = 0, subs = 0, slots = 0;
  unsigned long long t_edges = 0, t_probes = 0, t_exp = 0, t_pairs = 0, t_heavy = 0, t_he = 0,
                     t_hp = 0;  // lead thread
  int set = (int)a.set;
  uint64_t clean = 0;  // slots of this set known to be empty
  uint64_t nf = 0, n0 = 0, n1 = 0, e0 = 0, e1 = 0, cap = 0;
  int buf = 0;
  bool resume = a.cap != 0;
  uint32_t why = MB_RUNNING;

  // the next window: plain centres [cur, cur + W), or round's windows
  const uint64_t *wstart = nullptr, *wpre = nullptr;
  const uint32_t* wg = nullptr;
  uint32_t nwin = 0;
  auto window_size = [&]() -> uint64_t {
    if (GRAPHS) {
      if (round >= a.run.rounds) return 0;
      nwin = (uint32_t)__ldg(&a.run.heads[2 * round + 1]);
      const uint64_t* w = a.run.sched + __ldg(&a.run.heads[2 * round]);
      wg = (const uint32_t*)w;
      wstart = w + nwin;
      wpre = w + 2 * (uint64_t)nwin;
      return __ldg(&wpre[nwin]);
    }
    const uint64_t left = a.run.n_remaining - cur;
    return step < left ? step : left;
  };
  auto win_of = [&](uint64_t j) -> uint32_t { return last_le(wpre, nwin, j); };
  auto centre = [&](uint64_t j, uint32_t w) -> uint32_t {
    return GRAPHS ? __ldg(&a.run.centres[wstart[w] + (j - wpre[w])])
                  : __ldg(&a.run.centres[cur + j]);
  };
  auto advance = [&](uint64_t W) {
    if (GRAPHS) {
      round++;
    } else {
      cur += W;
      step = (uint64_t)ceil((double)step * a.beta);
      if (step > a.run.n_remaining) step = a.run.n_remaining;
      if (step == 0) step = 1;
    }
  };

  for (;;) {
    const uint64_t W = window_size();
    if (W == 0) {
      why = MB_DONE;
      break;
    }
    cap = resume ? a.cap : mb_cap(W, ne0, ne1, a.vgc_limit, a.tau);
    if (cap > a.cap_max) {
      nf = W;
      why = MB_HOST;
      break;
    }
    const uint64_t mask = cap - 1;
    unsigned long long* T0 = set ? a.T[1][0] : a.T[0][0];
    unsigned long long* T1 = set ? a.T[1][1] : a.T[0][1];
    uint64_t* F0 = a.F[0][0];
    uint64_t* F1 = a.F[1][0];
    if (!resume && cap > clean) {
      for (uint64_t i = clean + gt; i < cap; i += nt) {
        T0[i] = kEmpty;
        T1[i] = kEmpty;
      }
      clean = cap;
      if (!barrier()) return;
    }
    // --- select the live centres in order, and seed both sides with them
    nf = 0;
    if (resume) {
      nf = a.nf;
    } else if (!GRAPHS && W <= (uint64_t)kMbThreads) {
      // every block selects the whole window; rank r is seeded by block r % grid
      uint32_t v = 0;
      bool sel = false;
      if (tid < W) {
        v = centre(tid, 0);
        sel = !(ld_cg(&a.labels[v]) & kTopBit);
      }
      const unsigned m = __ballot_sync(kFull, sel);
      if (lane == 0) sh.wcnt[wid] = __popc(m);
      __syncthreads();
      uint32_t r = __popc(m & ((1u << lane) - 1u)), tot = 0;
      for (int w = 0; w < kMbWarps; w++) {
        const uint32_t c = sh.wcnt[w];
        if (w < (int)wid) r += c;
        tot += c;
      }
      nf = tot;
      if (sel && r % gridDim.x == blockIdx.x)
        mb_seed(T0, T1, mask, F0, F1, r, v, (uint32_t)(label_offset + r));
      __syncthreads();
    } else {
      const uint64_t per = (W + gridDim.x - 1) / gridDim.x;
      const uint64_t j0 = per * blockIdx.x < W ? per * blockIdx.x : W;
      const uint64_t j1 = j0 + per < W ? j0 + per : W;
      uint32_t c = 0;
      for (uint64_t j = j0 + tid; j < j1; j += kMbThreads) {
        const uint32_t w = GRAPHS ? win_of(j) : 0;
        c += !(ld_cg(&a.labels[centre(j, w)]) & kTopBit);
      }
      if (tid == 0) sh.before = sh.total = 0;
      __syncthreads();
      c = __reduce_add_sync(kFull, c);
      if (lane == 0 && c) atomicAdd(&sh.total, c);
      __syncthreads();
      if (tid == 0) {
        a.counts[blockIdx.x] = sh.total;
        sh.total = 0;
      }
      if (!barrier()) return;
      for (uint32_t b = tid; b < gridDim.x; b += kMbThreads) {
        const uint32_t x = ld_cg(&a.counts[b]);
        if (x) {
          atomicAdd(&sh.total, x);
          if (b < blockIdx.x) atomicAdd(&sh.before, x);
        }
      }
      __syncthreads();
      nf = sh.total;
      uint64_t base = sh.before;
      for (uint64_t t0 = j0; t0 < j1; t0 += kMbThreads) {
        const uint64_t j = t0 + tid;
        uint32_t v = 0, w = 0;
        bool sel = false;
        if (j < j1) {
          w = GRAPHS ? win_of(j) : 0;
          v = centre(j, w);
          sel = !(ld_cg(&a.labels[v]) & kTopBit);
        }
        const unsigned m = __ballot_sync(kFull, sel);
        if (lane == 0) sh.wcnt[wid] = __popc(m);
        __syncthreads();
        uint64_t r = base + __popc(m & ((1u << lane) - 1u));
        uint32_t tot = 0;
        for (int x = 0; x < kMbWarps; x++) {
          const uint32_t cx = sh.wcnt[x];
          if (x < (int)wid) r += cx;
          tot += cx;
        }
        if (GRAPHS) {
          // pivot r belongs to window w; a window's first item knows its base
          if (j < j1 && j == wpre[w]) a.run.fb[w] = r;
          if (sel) {
            a.run.front[r] = v;
            a.run.win[r] = w;
          }
        } else if (sel) {
          mb_seed(T0, T1, mask, F0, F1, r, v, (uint32_t)(label_offset + r));
        }
        base += tot;
        __syncthreads();
      }
      if (GRAPHS && nf) {
        if (lead) a.run.fb[nwin] = nf;
        if (!barrier()) return;
        for (uint64_t r = gt; r < nf; r += nt) {
          const uint32_t w = ld_cg(&a.run.win[r]);
          const uint64_t lab = ld_cg(&a.run.lo[__ldg(&wg[w])]) + (r - ld_cg(&a.run.fb[w]));
          mb_seed(T0, T1, mask, F0, F1, r, ld_cg(&a.run.front[r]), (uint32_t)lab);
        }
      }
    }
    if (nf == 0) {
      advance(W);
      // counts[] is rewritten by the next window only after another barrier
      if (!barrier()) return;
      continue;
    }
    if (resume) {
      n0 = a.n0;
      n1 = a.n1;
      e0 = a.e0;
      e1 = a.e1;
      buf = (int)a.buf;
      resume = false;
    } else {
      if (!barrier()) return;
      n0 = n1 = e0 = e1 = nf;
      buf = 0;
    }

    // --- sub-rounds
    bool give_up = false;
    while (n0 | n1) {
      Counters* c0 = a.ctr + kMbCtr + 2 * (subs % 3);
      Counters* c1 = c0 + 1;
      unsigned long long* z = (unsigned long long*)(a.ctr + kMbCtr + 2 * ((subs + 1) % 3));
      if (blockIdx.x == 0 && tid < 2 * sizeof(Counters) / 8) z[tid] = 0;  // last read a barrier ago
      subs++;
      auto side = [&](int k) {
        MsSide s;
        s.off = k ? a.in_off : a.off;
        s.E = k ? a.in_E : a.E;
        s.Fin = buf ? a.F[k][1] : a.F[k][0];
        s.Fout = buf ? a.F[k][0] : a.F[k][1];
        s.nin = k ? n1 : n0;
        s.T = k ? T1 : T0;
        s.mask = mask;
        s.Fheavy = a.Fh[k];
        s.hflag = a.hf[k];
        s.ctr = k ? c1 : c0;
        const uint64_t ne = k ? e1 : e0;
        const uint64_t room = cap / 2 > ne ? cap / 2 - ne : 0;
        const uint64_t share = room / (s.nin ? s.nin : 1);
        s.vgc_budget = (uint32_t)(share < 0xFFFFFFFFull ? share : 0xFFFFFFFFull);
        return s;
      };
      MsSide s0 = side(0), s1 = side(1);
      const bool v0 = a.local && n0 <= a.vgc_limit, v1 = a.local && n1 <= a.vgc_limit;
      if ((v0 && n0) || (v1 && n1)) {
        MsSide x0 = s0, x1 = s1;
        if (!v0) x0.nin = 0;
        if (!v1) x1.nin = 0;
        ms_vgc_round<kMbK, kMsVgcQueue>(x0, x1, a.labels, a.tau, sh.sm[wid], sh.q[wid], gw, nw);
      }
      if (!v0 || !v1) {
        MsSide x0 = s0, x1 = s1;
        if (v0) x0.nin = 0;
        if (v1) x1.nin = 0;
        ms_expand_round(x0, x1, a.labels, sh.sm[wid], sh.src[wid], gw, nw);
        if (lane == 0) sh.sm[wid].fail = 0;
      }
      if (!barrier()) return;
      if (__ldcg(&c0->heavy) | __ldcg(&c1->heavy)) {
        ms_heavy_round(s0, s1, a.labels, gw, nw);
        if (!barrier()) return;
      }
      if (lead) {
        t_edges += __ldcg(&c0->edges) + __ldcg(&c1->edges);
        t_probes += __ldcg(&c0->probes) + __ldcg(&c1->probes);
        t_exp += __ldcg(&c0->expanded) + __ldcg(&c1->expanded);
        t_pairs += n0 + n1;
        t_heavy += (__ldcg(&c0->heavy) >> kPackShift) + (__ldcg(&c1->heavy) >> kPackShift);
        t_he += __ldcg(&c0->heavy_edges) + __ldcg(&c1->heavy_edges);
        t_hp += __ldcg(&c0->heavy_probes) + __ldcg(&c1->heavy_probes);
      }
      n0 = __ldcg(&c0->next);
      n1 = __ldcg(&c1->next);
      e0 += __ldcg(&c0->inserted);
      e1 += __ldcg(&c1->inserted);
      buf ^= 1;
      if ((n0 | n1) &&
          ((__ldcg(&c0->fail) | __ldcg(&c1->fail)) || 2 * e0 > cap || 2 * e1 > cap)) {
        give_up = true;
        break;
      }
    }
    if (give_up) {
      why = MB_GROW;
      break;
    }
    // --- partition (scc.hpp:437-464), and clear the other set for the next batch
    batches++;
    slots += 2 * cap;
    const uint64_t this_w = W;
    if (GRAPHS) {
      for (uint32_t w = gt; w < nwin; w += nt)
        a.run.lo[__ldg(&wg[w])] =
            ld_cg(&a.run.lo[__ldg(&wg[w])]) + ld_cg(&a.run.fb[w + 1]) - ld_cg(&a.run.fb[w]);
    } else {
      label_offset += nf;
    }
    const bool small0 = e0 <= e1;  // the side with fewer entries probes the other
    const ulonglong2* Ps = (const ulonglong2*)(small0 ? T0 : T1);
    const ulonglong2* Pl = (const ulonglong2*)(small0 ? T1 : T0);
    const unsigned long long* Tl = small0 ? T1 : T0;
    for (uint64_t i = gt; i < cap; i += nt) {  // cap/2 pairs of slots of each table
      const bool small = i < cap / 2;
      const ulonglong2 e2 = __ldcg(small ? &Ps[i] : &Pl[i - cap / 2]);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint64_t e = h ? e2.y : e2.x;
        if (e == kEmpty) continue;
        const uint32_t v = (uint32_t)(e >> 32);
        const uint64_t l = e & kValMask;
        bool both = false;
        if (small) {
          uint64_t s = hash64(e) & mask;
          for (uint64_t x = 0; x <= mask; x++) {
            const uint64_t o = __ldcg(&Tl[s]);
            both = o == e;
            if (both || o == kEmpty) break;
            s = (s + 1) & mask;
          }
        }
        const uint64_t val = both ? (l | kTopBit) : l;
        if (ld_cg(&a.labels[v]) < val)
          atomicMax((unsigned long long*)&a.labels[v], (unsigned long long)val);
      }
    }
    ne0 = e0;
    ne1 = e1;
    advance(this_w);
    set ^= 1;
    clean = 0;
    const uint64_t next_w = window_size();
    if (next_w) {
      const uint64_t next_cap = mb_cap(next_w, ne0, ne1, a.vgc_limit, a.tau);
      if (next_cap <= a.cap_max) {
        unsigned long long* N0 = set ? a.T[1][0] : a.T[0][0];
        unsigned long long* N1 = set ? a.T[1][1] : a.T[0][1];
        const ulonglong2 none = make_ulonglong2(kEmpty, kEmpty);
        for (uint64_t i = gt; i < next_cap / 2; i += nt) {
          ((ulonglong2*)N0)[i] = none;
          ((ulonglong2*)N1)[i] = none;
        }
        clean = next_cap;
      }
    }
    if (!barrier()) return;
  }
  if (lead) {
    MbState& s = *a.st;
    s.cur = cur;
    s.step = step;
    s.label_offset = label_offset;
    s.round = round;
    s.ne[0] = ne0;
    s.ne[1] = ne1;
    s.batches = batches;
    s.subrounds = subs;
    s.edges = t_edges;
    s.probes = t_probes;
    s.expanded = t_exp;
    s.pairs = t_pairs;
    s.heavy = t_heavy;
    s.heavy_edges = t_he;
    s.heavy_probes = t_hp;
    s.slots = slots;
    s.n_remaining = a.run.n_remaining;
    s.cap = cap;
    s.nf = nf;
    s.n0 = n0;
    s.n1 = n1;
    s.e0 = e0;
    s.e1 = e1;
    s.set = (uint32_t)set;
    s.buf = (uint32_t)buf;
    s.why = why;
  }
}

static uint64_t pow2_at_least(uint64_t x) {
  uint64_t c = 1;
  while (c < x) c <<= 1;
  return c;
}

// Slots that leave the local searches from nf pairs (up to min(tau, 64) new pairs each)
// room below half load, at most 2^27; 0 when there are none.
static uint64_t ms_vgc_room(bool local, uint64_t nf, uint64_t ne, uint32_t tau, uint64_t vgc_limit) {
  if (!local || nf > vgc_limit) return 0;
  return std::min<uint64_t>(1ull << 27,
                            pow2_at_least(2 * (ne + nf * std::min<uint32_t>(tau, 64))));
}

// Rehash the table in slot tslot into a new table of capacity cap2.
// (in a buffer of at least `room` slots).
static int ms_grow(psc_graph_s* g, int tslot, uint64_t cap, uint64_t cap2, uint64_t room = 0) {
  cudaEvent_t ea = take_event(g), eb = take_event(g);
  PSC_CUDA(cudaEventRecord(ea, g->stream));
  unsigned long long *T, *T2;
  T = (unsigned long long*)g->bufs[tslot].p;
  PSC_TRY(ensure_t(g, B_TS, std::max(cap2, room), &T2));
  PSC_CUDA(cudaMemsetAsync(T2, 0xFF, cap2 * 8, g->stream));
  {
    ProfScope ps(g, F_TABLE);
    ps.bytes = 8.0 * cap + 8.0 * cap2;
    k_rehash<<<grid_for(g, cap, 256), 256, 0, g->stream>>>(T, cap, T2, cap2 - 1);
  }
  PSC_CUDA(cudaGetLastError());
  swap_bufs(g, tslot, B_TS);
  g->stats.table_grows++;
  PSC_CUDA(cudaEventRecord(eb, g->stream));
  g->grow_events.emplace_back(ea, eb);
  return PSC_OK;
}

namespace {

struct MsState {
  bool backward;
  int t_slot, a_slot, b_slot, h_slot, f_slot, cset;
  uint64_t cap = 0, ne = 0, nf = 0;
  bool grow = false;
};

MsSide ms_args(psc_graph_s* g, const MsState& s) {
  MsSide r;
  r.off = s.backward ? g->in_off : g->off;
  r.E = s.backward ? g->in_E : g->E;
  r.Fin = (const uint64_t*)g->bufs[s.a_slot].p;
  r.nin = s.nf;
  r.T = (unsigned long long*)g->bufs[s.t_slot].p;
  r.mask = s.cap - 1;
  r.Fout = (uint64_t*)g->bufs[s.b_slot].p;
  r.Fheavy = (uint64_t*)g->bufs[s.h_slot].p;
  r.hflag = (uint32_t*)g->bufs[s.f_slot].p;
  r.ctr = g->ctr + s.cset;
  // VGC local searches share the room left below half load, so one
  // sub-round cannot fill the table
  const uint64_t room = s.cap / 2 > s.ne ? s.cap / 2 - s.ne : 0;
  const uint64_t share = room / (s.nf ? s.nf : 1);
  r.vgc_budget = (uint32_t)(share < 0xFFFFFFFFull ? share : 0xFFFFFFFFull);
  return r;
}

}  // namespace

int ms_pair(psc_graph_s* g, const uint32_t* front, uint64_t n_front, uint64_t label_offset,
            const uint64_t* labels, const psc_params_t* p, const uint64_t prev_ne[2],
            MsResult out[2], const uint32_t* front_labels, uint64_t vgc_max) {
  // heavy-list fields: < 2^24 pairs (m / kHeavyDeg), first chunks < 2^31
  if (g->m >> 36) return PSC_ERR_TOO_LARGE;
  const uint32_t tau = p->tau ? p->tau : 512;
  const bool local = p->local_scc != 0;
  const uint64_t vgc_limit = vgc_max ? vgc_max : (uint64_t)g->num_sms * 32;
  MsState st[2];
  st[0] = MsState{false, B_TF, B_PA, B_PB, B_PH, B_AUX1, 0};
  st[1] = MsState{true, B_TB, B_PA2, B_PB2, B_PH2, B_HF2, 1};
  for (int k = 0; k < 2; k++) {
    MsState& s = st[k];
    const uint64_t want0 = (local && n_front <= vgc_limit) ? n_front * std::min<uint32_t>(tau, 64) : 0;
    s.cap = pow2_at_least(std::max<uint64_t>(
        {4096, 4 * n_front, 2 * prev_ne[k], std::min<uint64_t>(1ull << 27, 2 * (n_front + want0))}));
    void* q;
    PSC_TRY(ensure(g, s.t_slot, s.cap * 8 + 16, &q));
    PSC_CUDA(cudaMemsetAsync(q, 0xFF, s.cap * 8, g->stream));
    PSC_TRY(ensure(g, s.a_slot, s.cap * 8 + 16, &q));
    PSC_TRY(ensure(g, s.b_slot, s.cap * 8 + 16, &q));
    PSC_TRY(ensure(g, s.h_slot, s.cap * 8 + 16, &q));
    PSC_TRY(ensure(g, s.f_slot, s.cap * 4 + 16, &q));
    s.nf = s.ne = n_front;
  }
  {
    ProfScope ps(g, F_MS_SEED);
    ps.bytes = 40.0 * n_front;
    k_ms_seed<<<grid_for(g, n_front, 256), 256, 0, g->stream>>>(
        front, n_front, label_offset, front_labels, (unsigned long long*)g->bufs[st[0].t_slot].p,
        st[0].cap - 1, (uint64_t*)g->bufs[st[0].a_slot].p,
        (unsigned long long*)g->bufs[st[1].t_slot].p, st[1].cap - 1,
        (uint64_t*)g->bufs[st[1].a_slot].p);
  }
  for (;;) {
    bool any = false;
    for (auto& s : st) {
      if (s.nf == 0) continue;
      any = true;
      g->stats.subrounds++;
      // room for the VGC local searches of this sub-round: up to
      // min(tq, 64) new pairs each, while the table stays below 2^27 slots
      const uint64_t room = ms_vgc_room(local, s.nf, s.ne, tau, vgc_limit);
      const bool vgc_room = room > s.cap;
      if (s.grow || 2 * s.ne > s.cap || vgc_room) {
        // keep the load at most 1/2 (1/4 right after growing)
        uint64_t cap2 = pow2_at_least(std::max<uint64_t>(4 * s.ne, 2 * s.cap));
        if (vgc_room) cap2 = std::max(cap2, room);
        if (cap2 > (1ull << 40)) return PSC_ERR_TABLE_FULL;
        PSC_TRY(ms_grow(g, s.t_slot, s.cap, cap2));
        s.cap = cap2;
        void* q;
        PSC_TRY(ensure_keep(g, s.a_slot, s.cap * 8 + 16, s.nf * 8, &q));
        PSC_TRY(ensure(g, s.b_slot, s.cap * 8 + 16, &q));
        PSC_TRY(ensure(g, s.h_slot, s.cap * 8 + 16, &q));
        PSC_TRY(ensure(g, s.f_slot, s.cap * 4 + 16, &q));
      }
    }
    if (!any) break;
    PSC_TRY(zero_counters(g));
    MsSide vg[2] = {}, ex[2] = {}, hv[2] = {};
    int nv = 0, ne = 0, nh = 0;
    uint64_t v_items = 0, e_items = 0;
    bool is_vgc[2] = {false, false};
    for (int k = 0; k < 2; k++) {
      if (st[k].nf == 0) continue;
      MsSide a = ms_args(g, st[k]);
      is_vgc[k] = local && st[k].nf <= vgc_limit;
      if (is_vgc[k]) {
        vg[nv++] = a;
        v_items += st[k].nf;
      } else {
        ex[ne++] = a;
        e_items += st[k].nf;
      }
      hv[nh++] = a;
    }
    if (nv) {
      ProfScope ps(g, F_MS_VGC);
      // a resident grid, one pair per warp at a time
      if (!g->ms_vgc_blocks) {
        PSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &g->ms_vgc_blocks, k_ms_vgc<kMsVgcBlock, kMsVgcQueue>, kMsVgcBlock, 0));
        if (g->ms_vgc_blocks < 1) g->ms_vgc_blocks = 1;
      }
      const uint64_t max_blocks = (uint64_t)g->num_sms * g->ms_vgc_blocks;
      const uint64_t blocks =
          std::min(max_blocks, (v_items + kMsVgcBlock / 32 - 1) / (kMsVgcBlock / 32));
      k_ms_vgc<kMsVgcBlock, kMsVgcQueue><<<(unsigned)std::max<uint64_t>(1, blocks), kMsVgcBlock, 0,
                                           g->stream>>>(vg[0], vg[1], labels, tau);
    }
    if (ne) {
      ProfScope ps(g, F_MS_EXPAND);
      switch (p->block) {
        case 128:
          k_ms_expand<128><<<grid_for(g, e_items, 128), 128, 0, g->stream>>>(ex[0], ex[1], labels);
          break;
        case 512:
          k_ms_expand<512><<<grid_for(g, e_items, 512), 512, 0, g->stream>>>(ex[0], ex[1], labels);
          break;
        default:
          k_ms_expand<kMsBlock><<<grid_for(g, e_items, kMsBlock), kMsBlock, 0, g->stream>>>(
              ex[0], ex[1], labels);
      }
    }
    PSC_CUDA(cudaGetLastError());
    PSC_TRY(read_counters(g));
    // Heavy pairs are rare: the grid-wide walk is launched only for a round
    // that queued some, then the counters are read again.
    if ((st[0].nf && g->hctr[st[0].cset].heavy) || (st[1].nf && g->hctr[st[1].cset].heavy)) {
      {
        ProfScope ps(g, F_HEAVY);
        k_ms_heavy<kMsBlock><<<g->num_sms * 4, kMsBlock, 0, g->stream>>>(hv[0], hv[1], labels);
      }
      PSC_CUDA(cudaGetLastError());
      PSC_TRY(read_counters(g));
      if (g->profiling)
        for (int k = 0; k < 2; k++)
          if (st[k].nf) {
            const Counters& c = g->hctr[st[k].cset];
            g->prof[F_HEAVY].bytes +=
                28.0 * (c.heavy >> kPackShift) + 12.0 * c.heavy_edges + 8.0 * c.heavy_probes;
          }
    }
    if (trace_on()) {
      cudaEvent_t tr = take_event(g);
      PSC_CUDA(cudaEventRecord(tr, g->stream));
      PSC_CUDA(cudaEventSynchronize(tr));
      float ms = 0;  // since the start of the call
      cudaEventElapsedTime(&ms, g->t0, tr);
      give_event(g, tr);
      for (int k = 0; k < 2; k++)
        if (st[k].nf)
          std::fprintf(stderr, "ms side %d mode %s nf %llu next %llu edges %llu probes %llu "
                       "expanded %llu cap %llu ne %llu t %.3f ms\n",
                       k, is_vgc[k] ? "vgc" : "expand", (unsigned long long)st[k].nf,
                       g->hctr[st[k].cset].next, g->hctr[st[k].cset].edges,
                       g->hctr[st[k].cset].probes, g->hctr[st[k].cset].expanded,
                       (unsigned long long)st[k].cap, (unsigned long long)st[k].ne, ms);
    }
    for (int k = 0; k < 2; k++) {
      MsState& s = st[k];
      if (s.nf == 0) continue;
      const Counters& c = g->hctr[s.cset];
      if (g->profiling) {
        // 8 per frontier pair read + 16 per adjacency range + 4 per edge (ids)
        // + 8 per edge (label compare) + 8 per probe + 8 per appended pair
        g->prof[is_vgc[k] ? F_MS_VGC : F_MS_EXPAND].bytes +=
            8.0 * s.nf + 16.0 * c.expanded + 12.0 * c.edges + 8.0 * c.probes + 8.0 * c.next;
      }
      s.ne += c.inserted;
      s.grow = c.fail > 0;
      std::swap(g->bufs[s.a_slot], g->bufs[s.b_slot]);
      s.nf = c.next;
    }
  }
  for (int k = 0; k < 2; k++) {
    out[k].cap = st[k].cap;
    out[k].ne = st[k].ne;
  }
  return PSC_OK;
}

bool ms_run_ready(psc_graph_s* g) {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static int state[kMaxDev] = {};
  if (g->device < 0 || g->device >= kMaxDev) return false;
  std::lock_guard<std::mutex> lock(mu);
  int& st = state[g->device];
  if (st == 0) {
    st = -1;
    int coop = 0, b0 = 0, b1 = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, g->device) == cudaSuccess && coop &&
        cudaFuncSetAttribute(k_ms_batches<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(MbShared)) == cudaSuccess &&
        cudaFuncSetAttribute(k_ms_batches<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(MbShared)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_ms_batches<false>, kMbThreads,
                                                      sizeof(MbShared)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_ms_batches<true>, kMbThreads,
                                                      sizeof(MbShared)) == cudaSuccess &&
        b0 > 0 && b1 > 0)
      st = 1;
    cudaGetLastError();
  }
  return st == 1;
}

// Largest window of the resident launch (a batch's tables have four slots per
// candidate at least).
constexpr uint64_t kMbWindow = 1 << 18;

// Tables to begin with: 2^20 slots hold every batch of the R-MAT 2^26, kNN 10^7
// and 4096^2 grid solves; a smaller graph's tables are smaller.
static uint64_t mb_cap_max(const psc_graph_s* g) {
  return std::min<uint64_t>(1ull << 20, std::max<uint64_t>(1ull << 13, pow2_at_least(16 * g->n)));
}

static int ms_run_resident(psc_graph_s* g, uint64_t* labels, const psc_params_t* p, MsRun* run,
                           uint64_t window) {
  if (g->m >> 36) return PSC_ERR_TOO_LARGE;  // heavy-list fields, as in ms_pair
  MbArgs a = {};
  a.off = g->off;
  a.in_off = g->in_off;
  a.E = g->E;
  a.in_E = g->in_E;
  a.labels = labels;
  a.beta = p->beta;
  a.tau = p->tau ? p->tau : 512;
  a.local = p->local_scc != 0;
  a.vgc_limit = run->vgc_max ? run->vgc_max : (uint64_t)g->num_sms * 32;
  a.cap_max = mb_cap_max(g);
  // windows of more than kMbWindow candidates are full-width work: ms_pair; others
  // get the tables that they need
  if (window > kMbWindow) return PSC_OK;
  a.cap_max = std::max(a.cap_max, mb_cap(window, run->ne[0], run->ne[1], a.vgc_limit, a.tau));
  static const int kT[2][2] = {{B_TF, B_TB}, {B_TF2, B_TB2}}, kF[2][2] = {{B_PA, B_PB}, {B_PA2, B_PB2}};
  PSC_TRY(ensure_t(g, B_BLOCKS, (size_t)g->num_sms, &a.counts));
  a.ctr = g->ctr;
  a.st = (MbState*)(g->ctr + kMbState);
  const MbState& s = *(const MbState*)(g->hctr + kMbState);
  for (;;) {
    a.run = *run;
    for (int x = 0; x < 2; x++)
      for (int k = 0; k < 2; k++) {
        PSC_TRY(ensure_t(g, kT[x][k], a.cap_max, &a.T[x][k]));
        PSC_TRY(ensure_t(g, kF[x][k], a.cap_max, &a.F[x][k]));
      }
    PSC_TRY(ensure_t(g, B_PH, a.cap_max, &a.Fh[0]));
    PSC_TRY(ensure_t(g, B_PH2, a.cap_max, &a.Fh[1]));
    PSC_TRY(ensure_t(g, B_AUX1, a.cap_max, &a.hf[0]));
    PSC_TRY(ensure_t(g, B_HF2, a.cap_max, &a.hf[1]));
    PSC_TRY(zero_counters(g));
    {
      ProfScope ps(g, F_MS_VGC);
      void* args[] = {&a};
      PSC_CUDA(cudaLaunchCooperativeKernel(
          run->sched ? (const void*)k_ms_batches<true> : (const void*)k_ms_batches<false>,
          dim3(resident_sms(g)), dim3(kMbThreads), args, sizeof(MbShared), g->stream));
    }
    PSC_TRY(read_counters(g));
    if (s.failed || s.why == MB_RUNNING) return PSC_ERR_ITER_LIMIT;
    run->n_remaining = s.n_remaining;
    run->n_rem_dev = nullptr;
    run->cur = s.cur;
    run->step = s.step;
    run->label_offset = s.label_offset;
    run->round = s.round;
    run->ne[0] = s.ne[0];
    run->ne[1] = s.ne[1];
    g->stats.batches += s.batches;
    g->stats.subrounds += 2 * s.subrounds;
    if (g->profiling) {
      // as for the separate kernels (see ms_pair and scc_partition)
      g->prof[F_MS_VGC].bytes += 8.0 * s.pairs + 16.0 * s.expanded + 12.0 * s.edges + 8.0 * s.probes;
      g->prof[F_HEAVY].bytes += 28.0 * s.heavy + 12.0 * s.heavy_edges + 8.0 * s.heavy_probes;
      g->prof[F_PARTITION].bytes += 8.0 * s.slots;
    }
    if (trace_on())
      std::fprintf(stderr, "ms resident: %llu batches, %llu sub-rounds, pairs %llu edges %llu why %u\n",
                   s.batches, s.subrounds, s.pairs, s.edges, s.why);
    a.cap = 0;
    a.set = 0;
    if (s.why == MB_HOST && s.nf <= kMbWindow) {  // a larger table is all it needs
      a.cap_max = s.cap;
      continue;
    }
    if (s.why != MB_GROW) break;
    // grow both tables of the batch at hand to a quarter load, with room for the local
    // searches of the next sub-round as ms_pair makes it (the other set and what a
    // sub-round writes anew need not keep their contents)
    uint64_t cap2 = std::max<uint64_t>(4 * std::max(s.e0, s.e1), 2 * s.cap);
    for (int k = 0; k < 2; k++)
      cap2 = std::max(cap2, ms_vgc_room(a.local, k ? s.n1 : s.n0, k ? s.e1 : s.e0, a.tau, a.vgc_limit));
    cap2 = pow2_at_least(cap2);
    if (cap2 > (1ull << 40)) return PSC_ERR_TABLE_FULL;
    a.cap = cap2;
    a.nf = s.nf;
    a.n0 = s.n0;
    a.n1 = s.n1;
    a.e0 = s.e0;
    a.e1 = s.e1;
    a.set = s.set;
    a.buf = s.buf;
    a.cap_max = std::max(a.cap_max, cap2);
    const uint64_t keep[2] = {a.n0, a.n1}, old_cap = s.cap;
    for (int k = 0; k < 2; k++) {
      PSC_TRY(ms_grow(g, kT[a.set][k], old_cap, cap2, a.cap_max));
      void* q;
      PSC_TRY(ensure_keep(g, kF[k][a.buf], a.cap_max * 8 + 16, keep[k] * 8, &q));
    }
  }
  run->done = s.why == MB_DONE;
  return PSC_OK;
}

// Without room for two sets of tables the batch at hand is left to ms_pair, from its start
// (an interrupted one has written no label).
int ms_run(psc_graph_s* g, uint64_t* labels, const psc_params_t* p, MsRun* run, uint64_t window) {
  const int st = ms_run_resident(g, labels, p, run, window);
  if (st != PSC_ERR_OOM) return st;
  for (int b : {B_TF2, B_TB2}) PSC_TRY(release_buf(g, b));
  if (run->n_rem_dev) {
    PSC_CUDA(cudaMemcpyAsync(&g->hctr->aux0, run->n_rem_dev, 8, cudaMemcpyDeviceToHost, g->stream));
    PSC_CUDA(cudaStreamSynchronize(g->stream));
    run->n_remaining = g->hctr->aux0;
    run->n_rem_dev = nullptr;
  }
  run->done = run->sched ? run->round >= run->rounds : run->cur >= run->n_remaining;
  return PSC_OK;
}

}  // namespace psc
