// Connectivity on the device (src/Connectivity.h:37-119): a low-diameter
// decomposition followed by union-find over the edges that leave the largest
// cluster.  The input graph is symmetric (as the reference requires).
//
// LDD (src/ldd.hpp:325-417) as an exponential-shift multi-source BFS: 1024
// candidate centres hash32(1024 + i) % n are fixed up front; round r adds the
// next floor(exp(r * beta)) of them that are still unlabelled, and every round
// grows all clusters by one hop — a frontier vertex u offers label[u] to its
// neighbours, and atomicCAS(label[v], NONE, label[u]) lets the first offer
// win (the reference's compare_and_swap, ldd.hpp:226,253).  Rounds switch
// between push (queue) and pull (bitmap) by the reference's rule.  Vertices
// no cluster reaches are their own centre.
//
// Union-find (union_find_rules.h) as hook-and-compress: parent = LDD label;
// for every vertex outside the most frequent cluster (get_max_label,
// Connectivity.h:13-35, 10^4 hashed samples), every edge runs the lock-free
// unite: find both roots with path halving, link the larger root under the
// smaller with atomicCAS, retry on contention.  A final pass compresses every
// vertex to its root.  Spanning forest: the LDD tree edges (v, parent[v]) plus
// the edges whose unite linked two trees (Connectivity.h:99-117).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "engines.cuh"
#include "scan.cuh"

namespace psc {

constexpr int kCcBlock = 256;
constexpr int kLddSamples = 1024;   // ldd.hpp:462
constexpr int kMaxLabelSamples = 10000;  // Connectivity.h:14

__global__ void k_cc_init(uint32_t* label, uint32_t* parent, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    label[i] = kNone;
    if (parent) parent[i] = (uint32_t)i;
  }
}

// New centres perm[start .. start+count): claim the unlabelled ones and add
// them to the frontier (queue, or bitmap in pull mode).
__global__ void k_ldd_centres(const uint32_t* __restrict__ perm, uint32_t start, uint32_t count,
                              uint32_t* label, uint32_t* q, uint32_t* fb, Counters* ctr) {
  const unsigned lane = lane_id();
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < count;
       base += gridDim.x * blockDim.x) {
    const uint32_t i = base + lane;
    bool take = false;
    uint32_t c = 0;
    if (i < count) {
      c = perm[start + i];
      take = atomicCAS(&label[c], kNone, c) == kNone;
    }
    if (fb) {
      if (take) atomicOr(&fb[c >> 5], 1u << (c & 31));
      const unsigned m = __ballot_sync(kFull, take);
      if (lane == 0 && m) atomicAdd(&ctr->next, (unsigned long long)__popc(m));
    } else {
      unsigned long long pos = warp_append(&ctr->next, take);
      if (take) q[pos] = c;
    }
  }
}

// Big frontier vertices of an LDD round (out-degree >= the VGC queue size),
// listed by k_ldd_vgc with one 64-bit atomic on ctr->heavy = count <<
// kLddPackShift | chunks that gives each entry (vertex << 32 | first chunk)
// its slot and its first chunk of kLddChunk edges, increasing with the slot.
// The chunks of all entries are cut into one contiguous range per warp of the
// grid; a warp finds the entry of its first chunk once, then offers its
// vertex's label to kLddChunk edges per step (atomicCAS from NONE, as in the
// other LDD rounds).  A hub's edges are spread over the whole grid instead of
// one warp.  Field widths: count < 2^30, chunks < 2^34 (m < 2^36).
constexpr int kLddHeavyK = 4;
constexpr uint64_t kLddChunk = 32 * kLddHeavyK;
constexpr int kLddPackShift = 34;
constexpr uint64_t kLddPackMask = (1ull << kLddPackShift) - 1;

// (warp gw of nw)
__device__ __forceinline__ void ldd_heavy_round(const uint64_t* __restrict__ off,
                                                const uint32_t* __restrict__ E,
                                                const uint64_t* big, uint32_t* label,
                                                uint32_t* parent, uint32_t* qout, Counters* ctr,
                                                uint64_t gw, uint64_t nw) {
  constexpr int K = kLddHeavyK;
  const unsigned lane = lane_id();
  const unsigned long long packed = __ldcg(&ctr->heavy);
  const uint64_t nh = packed >> kLddPackShift, total = packed & kLddPackMask;
  const uint64_t per = (total + nw - 1) / nw;
  const uint64_t c_beg = gw * per, c_end = c_beg + per < total ? c_beg + per : total;
  if (nh == 0 || c_beg >= c_end) return;
  uint64_t h = 0, hi = nh - 1;  // last entry whose first chunk is <= c_beg
  while (h < hi) {
    const uint64_t mid = (h + hi + 1) >> 1;
    if ((uint32_t)ld_cg(&big[mid]) <= c_beg)
      h = mid;
    else
      hi = mid - 1;
  }
  uint64_t ent = ld_cg(&big[h]);
  uint64_t cs = (uint32_t)ent, cn = h + 1 < nh ? (uint32_t)ld_cg(&big[h + 1]) : total;
  uint32_t u = (uint32_t)(ent >> 32), lu = ld_cg(&label[u]);
  uint64_t beg = off[u], end = off[u + 1];
  unsigned long long scanned = 0, next_edges = 0;
  for (uint64_t c = c_beg; c < c_end; c++) {
    if (c >= cn) {
      h++;
      ent = ld_cg(&big[h]);
      cs = cn;
      cn = h + 1 < nh ? (uint32_t)ld_cg(&big[h + 1]) : total;
      u = (uint32_t)(ent >> 32);
      lu = ld_cg(&label[u]);
      beg = off[u];
      end = off[u + 1];
    }
    const uint64_t e0 = beg + (c - cs) * kLddChunk;
    uint32_t v[K], tm = 0, pre = 0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint64_t e = e0 + k * 32 + lane;
      v[k] = kNone;
      if (e < end) {
        scanned++;
        v[k] = __ldg(&E[e]);
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
      if (v[k] != kNone && __ldcg(&label[v[k]]) == kNone) pre |= 1u << k;
#pragma unroll
    for (int k = 0; k < K; k++)
      if ((pre & (1u << k)) && atomicCAS(&label[v[k]], kNone, lu) == kNone) {
        tm |= 1u << k;
        if (parent) parent[v[k]] = u;
      }
    warp_append_batch<K>(tm, v, qout, &ctr->next);
#pragma unroll
    for (int k = 0; k < K; k++)
      if (tm & (1u << k)) next_edges += off[v[k] + 1] - off[v[k]];
  }
  scanned = warp_sum(scanned);
  next_edges = warp_sum(next_edges);
  if (lane == 0) {
    if (scanned) atomicAdd(&ctr->edges, scanned);
    if (next_edges) atomicAdd(&ctr->next_edges, next_edges);
  }
}

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
    k_ldd_heavy(const uint64_t* __restrict__ off, const uint32_t* __restrict__ E,
                const uint64_t* big, uint32_t* label, uint32_t* parent, uint32_t* qout,
                Counters* ctr) {
  ldd_heavy_round(off, E, big, label, parent, qout, ctr,
                  (uint64_t)blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5),
                  (uint64_t)gridDim.x * (BLOCK / 32));
}

// VGC round (the reference's sparse_update with its local queue,
// ldd.hpp:88-161): each warp takes a chunk of up to `chunk` frontier
// vertices (one while the frontier fits the grid, up to 32 when it is much
// larger).  A chunk vertex with 0 < deg < tq seeds a local BFS in the warp's
// shared-memory queue of tq = min(tau, kLddQueue) entries: each wave takes up
// to 32 queued vertices, offers each one's label along its edges (balanced
// expansion, kLddK edges per lane in flight, atomicCAS from NONE), keeps the
// vertices it claims in the queue while there is room and spills the rest to
// the next frontier, as is whatever is left when the queue fills.  Queued
// vertices with deg > tq spill too; chunk vertices with deg >= tq go to the
// `big` list, whose edges k_ldd_heavy spreads over the grid afterwards.
constexpr int kLddQueue = 512;
constexpr int kLddVgcBlock = 128;
constexpr int kLddK = 8;

struct LEnt {
  uint64_t beg;
  uint32_t v;
  uint32_t deg;
};

// (warp gw of nw, with its own sm and queue Q, QL)
template <int QCAP, int kLddK>
__device__ __forceinline__ void ldd_vgc_round(const uint64_t* __restrict__ off,
                                              const uint32_t* __restrict__ E, const uint32_t* qin,
                                              uint64_t nin, uint32_t* label, uint32_t* parent,
                                              uint32_t* qout, uint64_t* big, uint32_t tau,
                                              uint32_t chunk, Counters* ctr, WarpExpandSmem& sm,
                                              LEnt* Q, uint32_t* QL, uint64_t gw, uint64_t nw) {
  const unsigned lane = lane_id();
  const uint32_t tq = tau < (uint32_t)QCAP ? tau : (uint32_t)QCAP;
  uint32_t C = chunk < tq ? chunk : tq;
  C = C < 1 ? 1 : C > 32 ? 32 : C;
  unsigned long long scanned = 0, next_edges = 0;
  const uint64_t nchunks = (nin + C - 1) / C;
  for (uint64_t c = gw; c < nchunks; c += nw) {
    const uint64_t first = c * C;
    const uint64_t left = nin - first;
    const uint32_t cnt = left < C ? (uint32_t)left : C;
    uint32_t u = 0, lu = 0;
    uint64_t ub = 0, du = 0;
    if (lane < cnt) {
      u = ld_cg(&qin[first + lane]);
      ub = off[u];
      du = off[u + 1] - ub;
      lu = ld_cg(&label[u]);
    }
    if (lane < cnt && du >= tq) {
      const unsigned long long old = atomicAdd(
          &ctr->heavy, (1ull << kLddPackShift) + (du + kLddChunk - 1) / kLddChunk);
      big[old >> kLddPackShift] = ((uint64_t)u << 32) | (old & kLddPackMask);
    }
    const bool seed = lane < cnt && du > 0 && du < tq;
    const uint32_t smask = __ballot_sync(kFull, seed);
    if (seed) {
      const uint32_t at = __popc(smask & ((1u << lane) - 1));
      Q[at] = LEnt{ub, u, (uint32_t)du};
      QL[at] = lu;
    }
    __syncwarp();
    uint32_t head = 0, tail = __popc(smask);
    while (head < tail && (head == 0 || tail < tq)) {
      const uint32_t wave = min(32u, tail - head);
      uint64_t beg = 0;
      uint32_t deg = 0, x = 0, xl = 0, xdeg = 0;
      bool spill_self = false;
      if (lane < wave) {
        const LEnt q = Q[head + lane];
        x = q.v;
        xl = QL[head + lane];
        beg = q.beg;
        deg = q.deg;
        xdeg = q.deg;
        if (deg > tq) {
          spill_self = true;
          deg = 0;
        }
      }
      head += wave;
      __syncwarp();
      if (__any_sync(kFull, spill_self)) {
        const unsigned long long pos = warp_append(&ctr->next, spill_self);
        if (spill_self) {
          qout[pos] = x;
          next_edges += xdeg;
        }
      }
      scanned += deg;
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
      for (uint32_t base = 0; base < total; base += 32 * kLddK) {
        uint32_t w[kLddK], wl[kLddK], wp[kLddK];
        uint64_t vb[kLddK], ve[kLddK];
#pragma unroll
        for (int k = 0; k < kLddK; k++) {
          const uint32_t gi = base + k * 32 + lane;
          w[k] = kNone;
          wl[k] = 0;
          wp[k] = 0;
          if (gi < total) {
            int lo = 0, hi = 31;
            while (lo < hi) {
              const int mid = (lo + hi + 1) >> 1;
              if (sm.excl[mid] <= gi)
                lo = mid;
              else
                hi = mid - 1;
            }
            w[k] = __ldg(&E[sm.beg[lo] + (gi - sm.excl[lo])]);
            wl[k] = QL[head - wave + lo];
            wp[k] = Q[head - wave + lo].v;
          }
        }
        // claims: the adjacency range is loaded alongside (used if claimed)
        uint32_t tm = 0;
#pragma unroll
        for (int k = 0; k < kLddK; k++) {
          vb[k] = ve[k] = 0;
          if (w[k] != kNone && __ldcg(&label[w[k]]) == kNone) {
            vb[k] = __ldg(&off[w[k]]);
            ve[k] = __ldg(&off[w[k] + 1]);
            tm |= 1u << k;
          }
        }
#pragma unroll
        for (int k = 0; k < kLddK; k++)
          if (tm & (1u << k)) {
            if (atomicCAS(&label[w[k]], kNone, wl[k]) == kNone) {
              if (parent) parent[w[k]] = wp[k];
            } else {
              tm &= ~(1u << k);
            }
          }
        // place: into the queue while it has room, then spill
        const uint32_t cntk = __popc(tm);
        uint32_t inc = cntk;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(kFull, inc, o);
          if ((int)lane >= o) inc += t;
        }
        const uint32_t tot = __shfl_sync(kFull, inc, 31);
        if (tot) {
          const uint32_t room = tail < tq ? tq - tail : 0;
          const uint32_t nloc = tot < room ? tot : room;
          unsigned long long sbase = 0;
          if (tot > nloc && lane == 0) sbase = atomicAdd(&ctr->next, (unsigned long long)(tot - nloc));
          sbase = __shfl_sync(kFull, sbase, 0);
          uint32_t r = inc - cntk;
#pragma unroll
          for (int k = 0; k < kLddK; k++)
            if (tm & (1u << k)) {
              const uint64_t vd = ve[k] - vb[k];
              if (r < nloc) {
                Q[tail + r] = LEnt{vb[k], w[k], (uint32_t)(vd < 0xFFFFFFFFull ? vd : 0xFFFFFFFFull)};
                QL[tail + r] = wl[k];
              } else {
                qout[sbase + (r - nloc)] = w[k];
                next_edges += vd;
              }
              r++;
            }
          tail += nloc;
          __syncwarp();
        }
      }
    }
    // spill what is left in the queue with one reservation
    const uint32_t rem = tail - head;
    if (rem) {
      unsigned long long b0 = 0;
      if (lane == 0) b0 = atomicAdd(&ctr->next, (unsigned long long)rem);
      b0 = __shfl_sync(kFull, b0, 0);
      for (uint32_t k = lane; k < rem; k += 32) {
        qout[b0 + k] = Q[head + k].v;
        next_edges += Q[head + k].deg;
      }
    }
    __syncwarp();
  }
  scanned = warp_sum(scanned);
  next_edges = warp_sum(next_edges);
  if (lane == 0) {
    if (scanned) atomicAdd(&ctr->edges, scanned);
    if (next_edges) atomicAdd(&ctr->next_edges, next_edges);
  }
}

template <int BLOCK, int QCAP>
__global__ void __launch_bounds__(BLOCK)
    k_ldd_vgc(const uint64_t* __restrict__ off, const uint32_t* __restrict__ E,
              const uint32_t* qin, uint64_t nin, uint32_t* label, uint32_t* parent,
              uint32_t* qout, uint64_t* big, uint32_t tau, uint32_t chunk, Counters* ctr) {
  __shared__ WarpExpandSmem sm[BLOCK / 32];
  __shared__ LEnt sq[BLOCK / 32][QCAP];
  __shared__ uint32_t slab[BLOCK / 32][QCAP];
  const unsigned wid = threadIdx.x >> 5;
  ldd_vgc_round<QCAP, kLddK>(off, E, qin, nin, label, parent, qout, big, tau, chunk, ctr, sm[wid],
                             sq[wid], slab[wid], (uint64_t)blockIdx.x * (BLOCK / 32) + wid,
                             (uint64_t)gridDim.x * (BLOCK / 32));
}

// ---------------------------------------------------------------------------
// Resident rounds.  Most rounds of a decomposition are narrow: on R-MAT 2^24 20
// of 27 hold fewer than 100 vertices and no edge to offer, yet cost three launches
// and two or three waits, 52 us each.  k_ldd_rounds runs rounds back to back on a
// resident grid with a grid barrier between the steps (new centres, expansion,
// big vertices), until the schedule is exhausted and nothing is left, or a round
// turns wide (the pull switch, or more edges than kLddWideEdges): that round,
// whose centres are in place, goes to the host's full-width kernels.
//
// LOW, for graphs with adjacency records: the expansion of k_reach_async_low with
// labels (eight lanes per entry, the records in the queue, one trip per hop), its
// searches cut after ldd_waves() waves so that a round lasts as long as its hops.
// Device time of connectivity, before -> now: symmetrised kNN 10^6 3.38 -> 0.81
// ms, kNN 8x10^6 6.96 -> 2.95, grid 2048 x 4000 7.75 -> 2.25, R-MAT 2^24 3.12 ->
// 1.95.  Cut after 6 / 10 / 16 / 24 waves: kNN 10^6 0.69 / 0.81 / 0.91 / 1.03, the grid
// 2.56 / 2.25 / 2.12 / 2.14, kNN 8x10^6 3.19 / 2.95 / 3.10 / 2.99.
// ---------------------------------------------------------------------------
constexpr int kLrThreads = 384;
constexpr int kLrWarps = kLrThreads / 32;
constexpr int kLrRing = 128;
constexpr uint64_t kLddWideEdges = 1 << 18;
constexpr int kLrCtr = 4;     // counter sets 4-6: three rounds in rotation
constexpr int kLrState = 10;  // counter sets 10-13
constexpr uint32_t kLrRounds = 64;  // rounds with new centres of one launch

enum LrWhy : uint32_t { LR_RUNNING = 0, LR_DONE = 1, LR_WIDE = 2, LR_PAUSE = 3 };

struct LrState {
  uint32_t arrive, failed, why, round;
  unsigned long long nf, nf_edges, edges, front, next;
  uint32_t odd, sampled;           // the frontier lies in q[odd]
  uint32_t fresh[kLrRounds];       // new centres of the launch's rounds
};
static_assert(sizeof(LrState) <= 4 * sizeof(Counters) && kLrState + 4 <= kCounterSets,
              "the state fits its counter sets");

struct LrLow {
  uint4 rec[kLrRing][2];
  uint32_t v[kLrRing], lab[kLrRing];
};
struct LrWide {
  LEnt q[kLddQueue];
  uint32_t lab[kLddQueue];
  WarpExpandSmem sm;
};

struct LrArgs {
  const uint64_t* off;
  const uint32_t* E;
  const VRec* rec;
  uint32_t *label, *parent;
  uint32_t* q[2];
  uint64_t* big;
  const uint32_t* perm;  // candidates, G per index
  uint64_t G;
  const uint32_t* work;  // candidate indexes offered in round 1, 2, ... (0 from n_work on)
  uint32_t n_work, round, sampled;
  uint32_t waves;  // of a search on records (ldd_waves)
  uint64_t nf, nf_edges, threshold;
  Counters* ctr;
  LrState* st;
};

// One expansion round over qin[0 .. nin) (see above).
__device__ __forceinline__ void ldd_low_round(const LrArgs& a, const uint32_t* qin, uint64_t nin,
                                              uint32_t* qout, Counters* ctr, LrLow& Q, uint64_t gw,
                                              uint64_t nw) {
  constexpr int K = kLrWave / 4;
  const unsigned lane = lane_id(), grp = lane >> 3, j = lane & 7, lt = (1u << lane) - 1u;
  const uint64_t per = (nin + nw - 1) / nw;
  const uint32_t C = (uint32_t)(per < 1 ? 1 : per > 32 ? 32 : per);
  unsigned long long next_edges = 0;
  uint32_t scanned = 0;
  for (uint64_t c = gw; c < (nin + C - 1) / C; c += nw) {
    const uint64_t left = nin - c * C;
    const uint32_t cnt = left < C ? (uint32_t)left : C;
    __syncwarp();
    if (lane < cnt) {
      const uint32_t u = ld_cg(&qin[c * C + lane]);
      Q.v[lane] = u;
      Q.lab[lane] = ld_cg(&a.label[u]);
      ld_rec(a.rec + u, Q.rec[lane][0], Q.rec[lane][1]);
    }
    uint32_t h = 0, t = cnt;
    __syncwarp();
    for (uint32_t wave = 0; h != t && wave < a.waves; wave++) {
      const uint32_t n = min((uint32_t)kLrWave, t - h);
      // target j of entry 4 k + grp, and the one kRecEdges further on
      uint32_t w[K], old[K], nx[K], lo[K], lab[K], src[K], more = 0;
      uint4 ra[K], rb[K];
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t q = (h + 4 * k + grp) & (kLrRing - 1);
        const uint32_t* word = (const uint32_t*)&Q.rec[q][0];
        lo[k] = word[0];
        w[k] = word[2 + (j < (unsigned)kRecEdges ? j : 0)];
        lab[k] = Q.lab[q];
        src[k] = Q.v[q];
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
              ((uint64_t)((const uint32_t*)&Q.rec[(h + 4 * k + grp) & (kLrRing - 1)][0])[1] << 8) |
              (lo[k] >> 24);
          nx[k] = kNone;
          if (((more >> k) & 1u) && j < (unsigned)kRecEdges && kRecEdges + j < (lo[k] & 0xFFFFFFu))
            nx[k] = __ldg(&a.E[beg + kRecEdges + j]);
        }
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        old[k] = 0;
        ra[k].x = 0;
        if (w[k] != kNone) {
          old[k] = atomicCAS(&a.label[w[k]], kNone, lab[k]);
          ld_rec(a.rec + w[k], ra[k], rb[k]);
          scanned++;
        }
      }
      unsigned m[K];
      uint32_t tot = 0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const bool won = w[k] != kNone && old[k] == kNone;
        if (won && a.parent) a.parent[w[k]] = src[k];
        m[k] = __ballot_sync(kFull, won);
        tot += __popc(m[k]);
      }
      const uint32_t room = kLrRing - (t - h);
      const uint32_t nloc = min(tot, room);
      unsigned long long spill = 0;
      if (tot > nloc) {  // a full queue: the rest waits for the next round
        if (lane == 0) spill = atomicAdd(&ctr->next, (unsigned long long)(tot - nloc));
        spill = __shfl_sync(kFull, spill, 0);
      }
      uint32_t at = 0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        const uint32_t q = at + __popc(m[k] & lt);
        if ((m[k] >> lane) & 1u) {
          if (q < nloc) {
            const uint32_t to = (t + q) & (kLrRing - 1);
            Q.rec[to][0] = ra[k];
            Q.rec[to][1] = rb[k];
            Q.v[to] = w[k];
            Q.lab[to] = lab[k];
          } else {
            qout[spill + (q - nloc)] = w[k];
            next_edges += ra[k].x & 0xFFFFFFu;
          }
        }
        at += __popc(m[k]);
      }
      t += nloc;
      // entries with targets left return to the front, in the places just read
      const uint32_t h0 = h;
      h += n;
      if (any_more) {
#pragma unroll
        for (int k = K - 1; k >= 0; k--) {
          const unsigned back = __ballot_sync(kFull, j == 0 && ((more >> k) & 1u));
          if (back) {
            const bool mv = (more >> k) & 1u;
            const uint32_t to = (h - 1 - __popc(back >> (8 * grp + 1))) & (kLrRing - 1);
            uint32_t hi = 0;
            if (mv && j == 0)
              hi = ((const uint32_t*)&Q.rec[(h0 + 4 * k + grp) & (kLrRing - 1)][0])[1];
            __syncwarp();
            if (mv) {
              uint32_t* word = (uint32_t*)&Q.rec[to][0];
              if (j < (unsigned)kRecEdges) word[2 + j] = nx[k];
              if (j == 0) {
                const uint64_t r =
                    ((((uint64_t)hi << 32) | lo[k]) + ((uint64_t)kRecEdges << 24)) - kRecEdges;
                word[0] = (uint32_t)r;
                word[1] = (uint32_t)(r >> 32);
                Q.v[to] = src[k];
                Q.lab[to] = lab[k];
              }
            }
            __syncwarp();
            h -= __popc(back);
          }
        }
      }
      __syncwarp();
    }
    // what is left waits for the next round
    const uint32_t rem = t - h;
    if (rem) {
      unsigned long long base = 0;
      if (lane == 0) base = atomicAdd(&ctr->next, (unsigned long long)rem);
      base = __shfl_sync(kFull, base, 0);
      for (uint32_t k = lane; k < rem; k += 32) {
        const uint32_t q = (h + k) & (kLrRing - 1);
        qout[base + k] = Q.v[q];
        next_edges += Q.rec[q][0].x & 0xFFFFFFu;
      }
    }
  }
  next_edges = warp_sum(next_edges);
  const unsigned long long e = warp_sum((unsigned long long)scanned);
  if (lane == 0) {
    if (e) atomicAdd(&ctr->edges, e);
    if (next_edges) atomicAdd(&ctr->next_edges, next_edges);
  }
}

template <bool LOW>
__global__ void __launch_bounds__(kLrThreads, 1) k_ldd_rounds(LrArgs a) {
  extern __shared__ __align__(16) unsigned char lr_raw[];
  const unsigned wid = threadIdx.x >> 5, tid = threadIdx.x;
  const uint64_t gw = (uint64_t)blockIdx.x * kLrWarps + wid, nw = (uint64_t)gridDim.x * kLrWarps;
  const bool lead = blockIdx.x == 0 && tid == 0;
  uint32_t target = 0;
  auto barrier = [&]() { return grid_barrier(&a.st->arrive, &a.st->failed, target); };
  uint64_t nf = a.nf, nf_edges = a.nf_edges;
  uint32_t round = a.round, sampled = a.sampled, why = LR_RUNNING, odd = 0;
  const uint32_t round0 = round;
  unsigned long long t_edges = 0, t_front = 0, t_next = 0;
  for (;;) {
    if (nf == 0 && round >= a.n_work) {
      why = LR_DONE;
      break;
    }
    if (round - round0 >= (round < a.n_work ? kLrRounds : kLrMaxRounds)) {
      why = LR_PAUSE;
      break;
    }
    // --- new centres join the frontier behind its nf vertices
    const uint32_t work = round < a.n_work ? __ldg(&a.work[round]) : 0;
    Counters* c = a.ctr + kLrCtr + round % 3;
    if (blockIdx.x == 0 && tid < sizeof(Counters) / 8)  // last read a barrier ago
      ((unsigned long long*)(a.ctr + kLrCtr + (round + 1) % 3))[tid] = 0;
    uint32_t* qin = odd ? a.q[1] : a.q[0];
    if (work) {
      const uint64_t count = work * a.G;
      for (uint64_t base = ((uint64_t)blockIdx.x * kLrThreads + tid) & ~31ull; base < count;
           base += (uint64_t)gridDim.x * kLrThreads) {
        const uint64_t i = base + lane_id();
        bool take = false;
        uint32_t v = 0;
        if (i < count) {
          v = __ldg(&a.perm[sampled * a.G + i]);
          take = atomicCAS(&a.label[v], kNone, v) == kNone;
        }
        const unsigned long long pos = warp_append(&c->aux1, take);
        if (take) qin[nf + pos] = v;
      }
      if (!barrier()) return;
      const uint64_t fresh = __ldcg(&c->aux1);
      if (lead) a.st->fresh[round - round0] = (uint32_t)fresh;
      nf += fresh;
      sampled += work;
    } else if (lead && round < a.n_work) {
      a.st->fresh[round - round0] = 0;
    }
    round++;
    if (nf == 0) {  // (a barrier has passed since the counters were zeroed)
      continue;
    }
    if (nf + nf_edges >= a.threshold || nf_edges > kLddWideEdges || nf > kLddWideEdges) {
      why = LR_WIDE;
      break;
    }
    // --- expansion, then the big vertices it set aside
    uint32_t* qout = odd ? a.q[0] : a.q[1];
    if constexpr (LOW) {
      LrLow* Q = reinterpret_cast<LrLow*>(lr_raw);
      ldd_low_round(a, qin, nf, qout, c, Q[wid], gw, nw);
    } else {
      LrWide* W = reinterpret_cast<LrWide*>(lr_raw);
      const uint64_t per = (nf + nw - 1) / nw;
      ldd_vgc_round<kLddQueue, 4>(a.off, a.E, qin, nf, a.label, a.parent, qout, a.big, kLddQueue,
                                  (uint32_t)(per > 32 ? 32 : per), c, W[wid].sm, W[wid].q,
                                  W[wid].lab, gw, nw);
    }
    if (!barrier()) return;
    if (!LOW && (__ldcg(&c->heavy) >> kLddPackShift)) {
      ldd_heavy_round(a.off, a.E, a.big, a.label, a.parent, qout, c, gw, nw);
      if (!barrier()) return;
    }
    t_front += nf;
    nf = __ldcg(&c->next);
    nf_edges = __ldcg(&c->next_edges);
    if (lead) {
      t_edges += __ldcg(&c->edges);
      t_next += nf;
    }
    odd ^= 1;
  }
  if (lead) {
    LrState& s = *a.st;
    s.nf = nf;
    s.nf_edges = nf_edges;
    s.round = round;
    s.sampled = sampled;
    s.odd = odd;
    s.edges = t_edges;
    s.front = t_front;
    s.next = t_next;
    s.why = why;
  }
}

// Pull round (ldd.hpp:163-247): every unlabelled vertex takes the label of
// its first neighbour in the frontier bitmap.  A warp owns 32 consecutive
// vertices and writes their next-frontier word with one store.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
    k_ldd_pull(const uint64_t* __restrict__ off, const uint32_t* __restrict__ E,
               const uint32_t* __restrict__ fb_in, uint32_t* label, uint32_t* parent,
               uint32_t* fb_out, uint64_t n, Counters* ctr) {
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint64_t gw = (uint64_t)blockIdx.x * (BLOCK / 32) + wid;
  const uint64_t nw = (uint64_t)gridDim.x * (BLOCK / 32);
  const uint64_t nwords = (n + 31) >> 5;
  unsigned long long cnt = 0, scanned = 0, next_edges = 0;
  for (uint64_t w = gw; w < nwords; w += nw) {
    const uint64_t v = w * 32 + lane;
    bool found = false;
    if (v < n && label[v] == kNone) {
      const uint64_t b = off[v], e = off[v + 1];
      uint64_t j = b;
      for (; j < e; j++) {
        const uint32_t x = __ldg(&E[j]);
        if ((__ldg(&fb_in[x >> 5]) >> (x & 31)) & 1u) {
          label[v] = label[x];
          if (parent) parent[v] = x;
          found = true;
          break;
        }
      }
      scanned += (found ? j + 1 : j) - b;
      if (found) next_edges += e - b;
    }
    const uint32_t mask = __ballot_sync(kFull, found);
    if (lane == 0) {
      fb_out[w] = mask;
      cnt += __popc(mask);
    }
  }
  scanned = warp_sum(scanned);
  next_edges = warp_sum(next_edges);
  if (lane == 0) {
    if (cnt) atomicAdd(&ctr->next, cnt);
    if (scanned) atomicAdd(&ctr->edges, scanned);
    if (next_edges) atomicAdd(&ctr->next_edges, next_edges);
  }
}

__global__ void k_cc_queue_to_bitmap(const uint32_t* __restrict__ q, uint64_t nq, uint32_t* fb) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t v = q[i];
    atomicOr(&fb[v >> 5], 1u << (v & 31));
  }
}

__global__ void k_cc_bitmap_to_queue(const uint32_t* __restrict__ fb, uint64_t nwords, uint32_t* q,
                                     Counters* ctr) {
  const unsigned lane = lane_id();
  const uint64_t gw = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t base = gw * 32; base < nwords; base += nw * 32) {
    const uint64_t w = base + lane;
    uint32_t word = w < nwords ? fb[w] : 0u;
    const uint32_t c = __popc(word);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, o);
      if ((int)lane >= o) incl += t;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    unsigned long long pos = 0;
    if (lane == 0 && total) pos = atomicAdd(&ctr->aux0, (unsigned long long)total);
    pos = __shfl_sync(kFull, pos, 0) + (incl - c);
    while (word) {
      const int b = __ffs(word) - 1;
      word &= word - 1;
      q[pos++] = (uint32_t)(w * 32 + b);
    }
  }
}

__global__ void k_set_u64(unsigned long long* p, unsigned long long v) { *p = v; }

__global__ void k_ldd_finish(uint32_t* label, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    if (label[i] == kNone) label[i] = (uint32_t)i;
}

// Candidate centres (ldd.hpp:463-466), sample-major: entry i * G + k is
// hash32(1024 + i) % size of graph k.
__global__ void k_ldd_candidates(const uint64_t* __restrict__ base, const uint64_t* __restrict__ size,
                                 uint64_t n, uint64_t G, uint32_t* perm) {
  const uint64_t count = (uint64_t)kLddSamples * G;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = i % G, h = hash32((uint32_t)(kLddSamples + i / G));
    perm[i] = base ? (uint32_t)(base[k] + h % size[k]) : (uint32_t)(h % n);
  }
}

// Most frequent of kMaxLabelSamples hashed label samples (get_max_label,
// Connectivity.h:13-35; ties go to the smallest label, as the reference's scan of
// the sorted samples does): one block counts them in a shared-memory hash
// table, the samples of a warp that agree together.  (Copied to the host and
// sorted there this took 0.35 ms of every call.)
constexpr uint32_t kModeSlots = 1 << 14;
static_assert(kMaxLabelSamples < (int)kModeSlots, "the table never fills");

__global__ void __launch_bounds__(1024)
    k_label_mode(const uint32_t* __restrict__ label, uint64_t n, uint64_t seed, uint32_t* out) {
  extern __shared__ uint32_t mode_sm[];  // keys, then counts
  uint32_t *key = mode_sm, *cnt = mode_sm + kModeSlots;
  __shared__ unsigned long long best;
  for (uint32_t i = threadIdx.x; i < kModeSlots; i += 1024) {
    key[i] = kNone;
    cnt[i] = 0;
  }
  if (threadIdx.x == 0) best = 0;
  __syncthreads();
  for (uint32_t base = threadIdx.x & ~31u; base < (uint32_t)kMaxLabelSamples; base += 1024) {
    const uint32_t i = base + lane_id();
    const uint32_t x = i < (uint32_t)kMaxLabelSamples ? label[hash64(i + seed) % n] : kNone;
    const unsigned peers = __match_any_sync(kFull, x);
    if (x != kNone && (int)lane_id() == __ffs(peers) - 1) {
      uint32_t h = hash32(x) & (kModeSlots - 1);
      for (;;) {
        const uint32_t o = atomicCAS(&key[h], kNone, x);
        if (o == kNone || o == x) break;
        h = (h + 1) & (kModeSlots - 1);
      }
      atomicAdd(&cnt[h], (uint32_t)__popc(peers));
    }
  }
  __syncthreads();
  unsigned long long b = 0;  // count, then the smallest label
  for (uint32_t i = threadIdx.x; i < kModeSlots; i += 1024)
    if (cnt[i]) {
      const unsigned long long v = ((unsigned long long)cnt[i] << 32) | (uint32_t)~key[i];
      b = v > b ? v : b;
    }
  if (b) atomicMax(&best, b);
  __syncthreads();
  if (threadIdx.x == 0) *out = ~(uint32_t)best;
}

// find with path halving (union_find_rules.h:80-90, split/halve variants)
__device__ __forceinline__ uint32_t uf_find(uint32_t* p, uint32_t x) {
  uint32_t px = __ldcg(&p[x]);
  while (px != x) {
    const uint32_t gx = __ldcg(&p[px]);
    if (gx != px) atomicCAS(&p[x], px, gx);
    x = px;
    px = gx;
  }
  return x;
}

// Unite over the edges [first, last) of the adjacency list of every vertex
// whose root is not its graph's groot (Connectivity.h:74-93).  Link the larger root
// under the smaller (UniteRemCAS links high -> low,
// union_find_rules.h:193-225).
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK)
    k_uf_edges(const uint64_t* __restrict__ off, const uint32_t* __restrict__ E, uint64_t n,
               uint32_t* parent, const uint32_t* __restrict__ cluster,
               const uint32_t* __restrict__ gid, const uint32_t* __restrict__ groot,
               uint32_t first, uint32_t last, uint32_t* forest, Counters* ctr) {
  __shared__ WarpExpandSmem sm[BLOCK / 32];
  __shared__ uint32_t s_u[BLOCK];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint64_t gw = (uint64_t)blockIdx.x * (BLOCK / 32) + wid;
  const uint64_t nw = (uint64_t)gridDim.x * (BLOCK / 32);
  unsigned long long scanned = 0;
  for (uint64_t base = gw * 32; base < n; base += nw * 32) {
    const uint64_t i = base + lane;
    uint64_t beg = 0, rem = 0;
    if (i < n && uf_find(parent, (uint32_t)i) != groot[gid ? gid[i] : 0]) {
      const uint64_t b = off[i], d = off[i + 1] - b;
      const uint64_t lo = d < first ? d : first, hi = d < last ? d : last;
      beg = b + lo;
      rem = hi - lo;
    }
    scanned += rem;
    s_u[wid * 32 + lane] = (uint32_t)i;
    // adjacency lists in pieces of at most 2^26 edges (32-bit warp scan)
    while (__any_sync(kFull, rem > 0)) {
      const uint32_t piece = (uint32_t)(rem < (1ull << 26) ? rem : (1ull << 26));
      warp_expand(sm[wid], beg, piece, [&](bool act, int s, uint64_t e) {
        bool linked = false;
        uint32_t x = 0, y = 0;
        // an edge inside one LDD cluster joins nothing (both ends already
        // share the cluster's centre as an ancestor)
        if (act) {
          x = s_u[wid * 32 + s];
          y = __ldg(&E[e]);
          if (__ldg(&cluster[y]) == __ldg(&cluster[x])) act = false;
        }
        if (act) {
          for (;;) {
            uint32_t rx = uf_find(parent, x), ry = uf_find(parent, y);
            if (rx == ry) break;
            if (rx < ry) {
              const uint32_t t = rx;
              rx = ry;
              ry = t;
            }
            if (atomicCAS(&parent[rx], rx, ry) == rx) {
              linked = true;
              break;
            }
          }
        }
        if (forest) {
          const unsigned long long pos = warp_append(&ctr->aux1, linked);
          if (linked) {
            forest[2 * pos] = x;
            forest[2 * pos + 1] = y;
          }
        }
      });
      beg += piece;
      rem -= piece;
    }
    __syncwarp();
  }
  scanned = warp_sum(scanned);
  if (lane == 0 && scanned) atomicAdd(&ctr->edges, scanned);
}

__global__ void k_uf_final(uint32_t* parent, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    parent[i] = uf_find(parent, (uint32_t)i);
}

// Most frequent LDD label among kGraphSamples hashed samples of each graph of
// a batch (ties to the smallest label, as the single-graph scan of sorted
// samples): one block per graph, a bitonic sort in shared memory.
constexpr int kGraphSamples = 256;

__global__ void __launch_bounds__(kGraphSamples)
    k_graph_modes(const uint32_t* __restrict__ label, const uint64_t* __restrict__ mbase,
                  const uint64_t* __restrict__ msize, const uint32_t* __restrict__ mk,
                  uint32_t* groot) {
  __shared__ uint32_t a[kGraphSamples];
  const uint32_t t = threadIdx.x;
  const uint64_t b = mbase[blockIdx.x], sz = msize[blockIdx.x];
  const uint64_t seed = hash64(sz + 1);
  a[t] = label[b + hash64(t + seed) % sz];
  __syncthreads();
  for (uint32_t k = 2; k <= (uint32_t)kGraphSamples; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      const uint32_t p = t ^ j;
      if (p > t) {
        const uint32_t x = a[t], y = a[p];
        if ((x > y) == ((t & k) == 0)) {
          a[t] = y;
          a[p] = x;
        }
      }
      __syncthreads();
    }
  }
  if (t == 0) {
    uint32_t best = a[0], best_cnt = 0;
    for (uint32_t i = 0; i < (uint32_t)kGraphSamples;) {
      uint32_t j = 1;
      while (i + j < (uint32_t)kGraphSamples && a[i + j] == a[i]) j++;
      if (j > best_cnt) {
        best_cnt = j;
        best = a[i];
      }
      i += j;
    }
    groot[mk[blockIdx.x]] = best;
  }
}

// Roots of the given labels after a compressing pass: groot[k] = label[groot[k]].
__global__ void k_gather_roots(const uint32_t* __restrict__ label, const uint32_t* __restrict__ mk,
                               uint32_t count, uint32_t* groot) {
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < count; j += gridDim.x * blockDim.x) {
    const uint32_t k = mk ? mk[j] : j;
    groot[k] = label[groot[k]];
  }
}

// LDD tree edges (v, parent[v]) for v != parent[v], appended to the forest.
__global__ void k_ldd_tree_edges(const uint32_t* __restrict__ tree, uint64_t n, uint32_t* forest,
                                 Counters* ctr) {
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = base + lane_id();
    const bool t = i < n && tree[i] != (uint32_t)i;
    const unsigned long long pos = warp_append(&ctr->aux1, t);
    if (t) {
      forest[2 * pos] = (uint32_t)i;
      forest[2 * pos + 1] = tree[i];
    }
  }
}

// Graphs of a batch with at least one vertex (the whole graph when the
// handle holds no batch): their vertex bases and sizes.
static void ldd_members(const psc_graph_s* g, std::vector<uint64_t>& base,
                        std::vector<uint64_t>& size) {
  base.clear();
  size.clear();
  if (g->num_graphs > 1) {
    for (uint32_t k = 0; k < g->num_graphs; k++)
      if (g->vbase[k + 1] > g->vbase[k]) {
        base.push_back(g->vbase[k]);
        size.push_back(g->vbase[k + 1] - g->vbase[k]);
      }
  } else {
    base.push_back(0);
    size.push_back(g->n);
  }
}

static size_t lr_smem(bool low) { return kLrWarps * (low ? sizeof(LrLow) : sizeof(LrWide)); }

// Whether the device holds k_ldd_rounds with a block on every SM (and its
// shared-memory limits are set); asked once per device.
static bool lr_ready(psc_graph_s* g) {
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
        cudaFuncSetAttribute(k_ldd_rounds<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)lr_smem(false)) == cudaSuccess &&
        cudaFuncSetAttribute(k_ldd_rounds<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)lr_smem(true)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b0, k_ldd_rounds<false>, kLrThreads,
                                                      lr_smem(false)) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_ldd_rounds<true>, kLrThreads,
                                                      lr_smem(true)) == cudaSuccess &&
        b0 > 0 && b1 > 0)
      st = 1;
    cudaGetLastError();
  }
  return st == 1;
}

// LDD into d_label (centre ids); tree (optional) receives BFS parents.  In a
// batch every graph draws its own candidate centres (hash32(1024 + i) % n_k,
// as a graph alone would) and all graphs add them on the same schedule, so
// the centre list is laid out sample-major: entry i * G + k.
int ldd_run(psc_graph_s* g, double beta, uint32_t* d_label, uint32_t* tree) {
  const uint64_t n = g->n, m = g->m, nwords = (n + 31) / 32;
  if (m >> 36) return PSC_ERR_TOO_LARGE;  // big-list fields (k_ldd_heavy)
  const unsigned tb = kCcBlock;
  std::vector<uint64_t> mb, ms;
  ldd_members(g, mb, ms);
  const uint64_t G = mb.size();
  const uint64_t ncent = (uint64_t)kLddSamples * G;
  uint32_t *qa, *qb, *fa, *fb, *perm, *work_d;
  PSC_TRY(ensure_t(g, B_QA, n + ncent + 1, &qa));
  PSC_TRY(ensure_t(g, B_QB, n + ncent + 1, &qb));
  PSC_TRY(ensure_t(g, B_FB_A, nwords + 1, &fa));
  PSC_TRY(ensure_t(g, B_FB_B, nwords + 1, &fb));
  PSC_TRY(ensure_t(g, B_AUX2, ncent + kLddSamples, &perm));
  work_d = perm + ncent;
  // candidate indexes offered in round 1, 2, ... until all are (ldd.hpp:343-373)
  std::vector<uint32_t> work_of;
  for (uint32_t sum = 0; sum < (uint32_t)kLddSamples; sum += work_of.back())
    work_of.push_back((uint32_t)std::min<double>(
        std::floor(std::exp((double)(work_of.size() + 1) * beta)), (double)(kLddSamples - sum)));
  PSC_CUDA(cudaMemcpyAsync(work_d, work_of.data(), work_of.size() * 4, cudaMemcpyHostToDevice,
                           g->stream));
  {
    uint64_t* members = nullptr;
    if (g->num_graphs > 1) {
      PSC_TRY(ensure_t(g, B_GRAPHS, 2 * (size_t)G + (size_t)g->num_graphs + G + 2, &members));
      PSC_CUDA(cudaMemcpyAsync(members, mb.data(), G * 8, cudaMemcpyHostToDevice, g->stream));
      PSC_CUDA(cudaMemcpyAsync(members + G, ms.data(), G * 8, cudaMemcpyHostToDevice, g->stream));
    }
    ProfScope ps(g, F_CC);
    k_ldd_candidates<<<grid_for(g, ncent, 256), 256, 0, g->stream>>>(
        members, members ? members + G : nullptr, n, G, perm);
  }
  {
    ProfScope ps(g, F_CC);
    k_cc_init<<<grid_for(g, n, tb), tb, 0, g->stream>>>(d_label, tree, n);
  }
  const uint64_t threshold = m / 20;
  uint64_t nf = 0, nf_edges = 0;
  uint32_t sampled = 0, round = 0;
  bool pull = false;
  g->ldd_trace.clear();
  const VRec* rec = nullptr;
  const bool resident = lr_ready(g);
  if (resident) PSC_TRY(records_if_low(g, false, &rec));
  bool centres_in = false;  // the round's centres are in place already
  while (nf > 0 || sampled < (uint32_t)kLddSamples) {
    if (round > n + kLddSamples + 2) return PSC_ERR_ITER_LIMIT;
    if (resident && !pull && !centres_in && nf + nf_edges < std::max<uint64_t>(threshold, 1) &&
        nf <= kLddWideEdges && nf_edges <= kLddWideEdges) {
      LrArgs a = {};
      PSC_TRY(ensure_t(g, B_HEAVY, n + 1, &a.big));
      if (g->rec_refused) rec = nullptr;  // (that may have taken their room)
      a.off = g->off;
      a.E = g->E;
      a.rec = rec;
      a.label = d_label;
      a.parent = tree;
      a.q[0] = qa;
      a.q[1] = qb;
      a.perm = perm;
      a.G = G;
      a.work = work_d;
      a.n_work = (uint32_t)work_of.size();
      a.round = round;
      a.sampled = sampled;
      a.waves = ldd_waves(std::max(g->max_deg[0], g->max_deg[1]));
      a.nf = nf;
      a.nf_edges = nf_edges;
      a.threshold = threshold;
      a.ctr = g->ctr;
      a.st = (LrState*)(g->ctr + kLrState);
      PSC_TRY(zero_counters(g));
      {
        ProfScope ps(g, F_CC);
        void* args[] = {&a};
        PSC_CUDA(cudaLaunchCooperativeKernel(
            rec ? (const void*)k_ldd_rounds<true> : (const void*)k_ldd_rounds<false>,
            dim3(resident_sms(g)), dim3(kLrThreads), args, lr_smem(rec != nullptr), g->stream));
      }
      PSC_TRY(read_counters(g));
      const LrState& st = *(const LrState*)(g->hctr + kLrState);
      if (st.failed || st.why == LR_RUNNING) return PSC_ERR_ITER_LIMIT;
      for (uint32_t r = round; r < st.round; r++) {
        const uint32_t w = r < work_of.size() ? work_of[r] : 0;
        g->ldd_trace.insert(g->ldd_trace.end(), {sampled, w, w ? st.fresh[r - round] : 0});
        sampled += w;
      }
      if (trace_on())
        std::fprintf(stderr, "ldd resident rounds %u to %u, nf %llu edges %llu why %u\n", round + 1,
                     st.round, st.nf, st.edges, st.why);
      if (g->profiling)
        g->prof[F_CC].bytes += 16.0 * st.front + 8.0 * st.edges + 8.0 * st.next;
      round = st.round;
      nf = st.nf;
      nf_edges = st.nf_edges;
      if (st.odd) {
        std::swap(qa, qb);
        swap_bufs(g, B_QA, B_QB);
      }
      centres_in = st.why == LR_WIDE;
      continue;
    }
    if (!centres_in) {
      const uint32_t work = round < work_of.size() ? work_of[round] : 0;
      round++;
      uint32_t new_centres = 0;
      const uint32_t first = sampled;
      if (work > 0) {
        // new centres join the frontier: appended after the nf queued vertices
        // (counter block 1 is the queue cursor) or set in the frontier bitmap
        PSC_TRY(zero_counters(g));
        k_set_u64<<<1, 1, 0, g->stream>>>(&g->ctr[1].next, pull ? 0ull : (unsigned long long)nf);
        ProfScope ps(g, F_CC);
        k_ldd_centres<<<grid_for(g, work * G, 256), 256, 0, g->stream>>>(
            perm, (uint32_t)(sampled * G), (uint32_t)(work * G), d_label, pull ? nullptr : qa,
            pull ? fa : nullptr, g->ctr + 1);
        sampled += work;
        PSC_TRY(read_counters(g));
        new_centres = (uint32_t)(pull ? g->hctr[1].next : g->hctr[1].next - nf);
        nf = pull ? nf + g->hctr[1].next : g->hctr[1].next;
      }
      g->ldd_trace.insert(g->ldd_trace.end(), {first, work, new_centres});
    }
    centres_in = false;
    if (nf == 0) continue;
    const bool want_pull = (nf + nf_edges) >= threshold;
    if (want_pull && !pull) {
      PSC_CUDA(cudaMemsetAsync(fa, 0, nwords * 4, g->stream));
      k_cc_queue_to_bitmap<<<grid_for(g, nf, 256), 256, 0, g->stream>>>(qa, nf, fa);
      pull = true;
    } else if (!want_pull && pull) {
      PSC_TRY(zero_counters(g));
      k_cc_bitmap_to_queue<<<grid_for(g, nwords, 256), 256, 0, g->stream>>>(fa, nwords, qa, g->ctr);
      pull = false;
    }
    PSC_TRY(zero_counters(g));
    if (!pull) {
      // VGC round on a resident grid, then the big-degree frontier vertices
      // it set aside, their edges cut into chunks over the whole grid, into
      // the same queue
      if (!g->ldd_vgc_blocks) {
        PSC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &g->ldd_vgc_blocks, k_ldd_vgc<kLddVgcBlock, kLddQueue>, kLddVgcBlock, 0));
        if (g->ldd_vgc_blocks < 1) g->ldd_vgc_blocks = 1;
      }
      const uint64_t max_blocks = (uint64_t)g->num_sms * g->ldd_vgc_blocks;
      const uint64_t max_warps = max_blocks * (kLddVgcBlock / 32);
      const uint64_t chunk = std::min<uint64_t>(32, (nf + max_warps - 1) / max_warps);
      const uint64_t chunks = (nf + chunk - 1) / chunk;
      const uint64_t blocks =
          std::min(max_blocks, (chunks + kLddVgcBlock / 32 - 1) / (kLddVgcBlock / 32));
      uint64_t* big;
      PSC_TRY(ensure_t(g, B_HEAVY, n + 1, &big));
      {
        ProfScope ps(g, F_CC);
        k_ldd_vgc<kLddVgcBlock, kLddQueue>
            <<<(unsigned)std::max<uint64_t>(1, blocks), kLddVgcBlock, 0, g->stream>>>(
                g->off, g->E, qa, nf, d_label, tree, qb, big, kLddQueue, (uint32_t)chunk, g->ctr);
      }
      PSC_CUDA(cudaGetLastError());
      PSC_TRY(read_counters(g));
      if (g->hctr[0].heavy >> kLddPackShift) {
        ProfScope ps(g, F_CC);
        k_ldd_heavy<kCcBlock><<<g->num_sms * 4, kCcBlock, 0, g->stream>>>(
            g->off, g->E, big, d_label, tree, qb, g->ctr);
      }
      std::swap(qa, qb);
      swap_bufs(g, B_QA, B_QB);
    } else {
      ProfScope ps(g, F_CC);
      k_ldd_pull<kCcBlock><<<grid_for(g, nwords * 32, tb), tb, 0, g->stream>>>(
          g->off, g->E, fa, d_label, tree, fb, n, g->ctr);
      std::swap(fa, fb);
      swap_bufs(g, B_FB_A, B_FB_B);
    }
    PSC_CUDA(cudaGetLastError());
    PSC_TRY(read_counters(g));
    if (trace_on()) {  // ms since the start of the call (the stream is idle here)
      cudaEvent_t ev = take_event(g);
      PSC_CUDA(cudaEventRecord(ev, g->stream));
      PSC_CUDA(cudaEventSynchronize(ev));
      float ms = 0;
      cudaEventElapsedTime(&ms, g->t0, ev);
      give_event(g, ev);
      std::fprintf(stderr, "ldd round %u mode %s nf %llu next %llu edges %llu t %.3f ms\n", round,
                   pull ? "pull" : "push", (unsigned long long)nf, g->hctr[0].next,
                   g->hctr[0].edges, ms);
    }
    if (g->profiling) {
      // algorithmic bytes: push / VGC: 16 per frontier vertex (range), 8 per
      // edge (target id, label CAS), 8 per new vertex; pull: both bitmaps,
      // 8 per scanned in-edge, 4 per new vertex
      const Counters& c = g->hctr[0];
      g->prof[F_CC].bytes += pull ? 0.25 * n + 8.0 * c.edges + 4.0 * c.next
                                  : 16.0 * nf + 8.0 * c.edges + 8.0 * c.next;
    }
    nf = g->hctr[0].next;
    nf_edges = g->hctr[0].next_edges;
  }
  g->stats.reach_rounds = round;
  {
    ProfScope ps(g, F_CC);
    k_ldd_finish<<<grid_for(g, n, tb), tb, 0, g->stream>>>(d_label, n);
  }
  PSC_CUDA(cudaGetLastError());
  return PSC_OK;
}

// k_label_mode's shared memory, allowed once per device.
static int mode_ready(int device) {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static bool done[kMaxDev] = {};
  std::lock_guard<std::mutex> lock(mu);
  if (device >= 0 && device < kMaxDev && done[device]) return PSC_OK;
  PSC_CUDA(cudaFuncSetAttribute(k_label_mode, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(kModeSlots * 8)));
  if (device >= 0 && device < kMaxDev) done[device] = true;
  return PSC_OK;
}

int cc_run(psc_graph_s* g, double beta, uint32_t* d_label, uint32_t* d_forest, uint64_t* n_forest) {
  const uint64_t n = g->n;
  const unsigned tb = kCcBlock;
  uint32_t* tree = nullptr;
  if (d_forest) PSC_TRY(ensure_t(g, B_TMP32, n + 1, &tree));
  PSC_TRY(ldd_run(g, beta, d_label, tree));
  std::vector<uint64_t> mb, ms;
  ldd_members(g, mb, ms);
  const bool batched = g->num_graphs > 1;
  uint32_t *groot = nullptr, *mk = nullptr;
  const uint32_t G = (uint32_t)mb.size();
  uint64_t* mw;
  PSC_TRY(ensure_t(g, B_GRAPHS, 2 * (size_t)G + (size_t)g->num_graphs + G + 2, &mw));
  groot = (uint32_t*)(mw + 2 * (size_t)G);
  std::vector<uint32_t> hk;
  if (batched) {
    // a batch: each graph's most frequent cluster (ldd_run left the members'
    // bases and sizes in mw)
    mk = groot + g->num_graphs + 1;
    for (uint32_t k = 0; k < g->num_graphs; k++)
      if (g->vbase[k + 1] > g->vbase[k]) hk.push_back(k);
    PSC_CUDA(cudaMemcpyAsync(mk, hk.data(), hk.size() * 4, cudaMemcpyHostToDevice, g->stream));
    ProfScope ps(g, F_UF);
    k_graph_modes<<<G, kGraphSamples, 0, g->stream>>>(d_label, mw, mw + G, mk, groot);
  } else {
    PSC_TRY(mode_ready(g->device));
    ProfScope ps(g, F_UF);
    k_label_mode<<<1, 1024, kModeSlots * 8, g->stream>>>(d_label, n, hash64(n + 1), groot);
  }
  const uint32_t* gid = batched ? g->d_gid : nullptr;
  // LDD labels are centre ids and every centre labels itself, so the label
  // array is already a depth-1 union-find forest; groot is its own root.
  PSC_TRY(zero_counters(g));
  uint32_t* forest = d_forest;
  if (forest) {
    ProfScope ps(g, F_CC);
    k_ldd_tree_edges<<<grid_for(g, n, 256), 256, 0, g->stream>>>(tree, n, forest, g->ctr);
  }
  // the LDD clusters, kept unchanged while the unions rewrite d_label
  uint32_t* cluster;
  PSC_TRY(ensure_t(g, B_AUX1, n + 1, &cluster));
  PSC_CUDA(cudaMemcpyAsync(cluster, d_label, n * 4, cudaMemcpyDeviceToDevice, g->stream));
  // Two passes over the edges of vertices outside the largest component:
  // first each one's first kUfSample edges (adjacency lists are sorted, so
  // these reach low-id hubs, which join most vertices to the largest
  // component), then, after compressing, the rest of the edges of the
  // vertices still outside it.  Every edge is still offered to the union
  // from one side: an edge skipped on both sides joins two vertices already
  // in the largest component.
  constexpr uint32_t kUfSample = 2;
  // algorithmic bytes of a union pass: per vertex its range, its two labels
  // and its cluster; per offered edge the target id and its label
  auto uf_bytes = [&](unsigned long long edges0) -> int {
    if (!g->profiling) return PSC_OK;
    PSC_TRY(read_counters(g));
    g->prof[F_UF].bytes += 28.0 * n + 8.0 * (g->hctr[0].edges - edges0) + 8.0 * n;
    return PSC_OK;
  };
  {
    ProfScope ps(g, F_UF);
    k_uf_edges<kCcBlock><<<grid_for(g, n, tb), tb, 0, g->stream>>>(
        g->off, g->E, n, d_label, cluster, gid, groot, 0, kUfSample, forest, g->ctr);
  }
  {
    ProfScope ps(g, F_UF);
    k_uf_final<<<grid_for(g, n, tb), tb, 0, g->stream>>>(d_label, n);
  }
  PSC_TRY(uf_bytes(0));
  const unsigned long long uf_edges1 = g->profiling ? g->hctr[0].edges : 0;
  {
    ProfScope ps(g, F_UF);
    k_gather_roots<<<(G + 255) / 256, 256, 0, g->stream>>>(d_label, mk, G, groot);
  }
  {
    ProfScope ps(g, F_UF);
    k_uf_edges<kCcBlock><<<grid_for(g, n, tb), tb, 0, g->stream>>>(
        g->off, g->E, n, d_label, cluster, gid, groot, kUfSample, 0xFFFFFFFFu, forest, g->ctr);
  }
  {
    ProfScope ps(g, F_UF);
    k_uf_final<<<grid_for(g, n, tb), tb, 0, g->stream>>>(d_label, n);
  }
  PSC_TRY(uf_bytes(uf_edges1));
  PSC_CUDA(cudaGetLastError());
  if (trace_on()) {
    cudaEvent_t ev = take_event(g);
    PSC_CUDA(cudaEventRecord(ev, g->stream));
    PSC_CUDA(cudaEventSynchronize(ev));
    float ms = 0;
    cudaEventElapsedTime(&ms, g->t0, ev);
    give_event(g, ev);
    std::fprintf(stderr, "cc union-find done t %.3f ms\n", ms);
  }
  if (n_forest) {
    PSC_TRY(read_counters(g));
    *n_forest = g->hctr[0].aux1;
  }
  return PSC_OK;
}

}  // namespace psc

using namespace psc;

extern "C" int psc_cc(psc_graph_t g, double beta, uint32_t* labels_out, uint32_t* forest_out,
                      uint64_t* n_forest) {
  if (!g || !labels_out || !(beta > 0)) return PSC_ERR_INVALID;
  if ((forest_out == nullptr) != (n_forest == nullptr)) return PSC_ERR_INVALID;
  CallScope scope(g->device);
  PSC_TRY(call_begin(g));
  uint32_t *d, *df = nullptr;
  PSC_TRY(ensure_t(g, B_AUX0, g->n + 1, &d));
  if (forest_out) PSC_TRY(ensure_t(g, B_AUX3, 2 * g->n + 2, &df));
  uint64_t nfor = 0;
  PSC_TRY(cc_run(g, beta, d, df, forest_out ? &nfor : nullptr));
  PSC_CUDA(cudaMemcpyAsync(labels_out, d, g->n * 4, cudaMemcpyDeviceToHost, g->stream));
  if (forest_out) {
    *n_forest = nfor;
    if (nfor) PSC_CUDA(cudaMemcpyAsync(forest_out, df, nfor * 8, cudaMemcpyDeviceToHost, g->stream));
  }
  return call_end(g);
}

extern "C" int psc_ldd_rounds(psc_graph_t g, uint32_t* out, uint32_t cap, uint32_t* rounds) {
  if (!g || !rounds || (cap && !out)) return PSC_ERR_INVALID;
  const uint32_t r = (uint32_t)(g->ldd_trace.size() / 3);
  *rounds = r;
  if (r > cap) return PSC_ERR_CAPACITY;
  std::copy(g->ldd_trace.begin(), g->ldd_trace.end(), out);
  return PSC_OK;
}

extern "C" int psc_ldd(psc_graph_t g, double beta, uint32_t* label_out, uint32_t* parent_out) {
  if (!g || !label_out || !(beta > 0)) return PSC_ERR_INVALID;
  CallScope scope(g->device);
  PSC_TRY(call_begin(g));
  uint32_t *d, *dp = nullptr;
  PSC_TRY(ensure_t(g, B_AUX0, g->n + 1, &d));
  if (parent_out) PSC_TRY(ensure_t(g, B_TMP32, g->n + 1, &dp));
  PSC_TRY(ldd_run(g, beta, d, dp));
  PSC_CUDA(cudaMemcpyAsync(label_out, d, g->n * 4, cudaMemcpyDeviceToHost, g->stream));
  if (parent_out)
    PSC_CUDA(cudaMemcpyAsync(parent_out, dp, g->n * 4, cudaMemcpyDeviceToHost, g->stream));
  return call_end(g);
}
