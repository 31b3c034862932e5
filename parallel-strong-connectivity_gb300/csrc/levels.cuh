// Level-synchronous search on one thread-block cluster: narrow levels of a
// BFS (src/bfs.hpp:200-238) or of a push-only reachability search
// (src/reach.hpp:173-190) run back to back inside one launch.
//
// What bounds it: a narrow level is a chain of dependent memory round trips
// (target id, then the claim), and between levels everybody has to agree on
// the next frontier.  Launched from the host, a level costs a memset, a
// kernel, a read-back and a wait, 23 us on the grid and kNN graphs for well
// under 10 us of work; a grid-wide barrier costs 1.3 us and more.  So the
// levels run on one cluster of 16 blocks (the largest non-portable size), whose
// hardware barrier takes a few hundred ns, and the frontier never leaves
// the cluster: a claimed vertex goes with its adjacency range straight into the
// shared memory of the block that will expand it (distributed shared memory),
// dealt out round-robin, so every block gets 1/16 of each source's claims.  Each
// (source, destination) pair of blocks has its own segment, so a slot needs only
// an atomic in the source's own shared memory, and the segment lengths are
// written once per level.  A level is then: read the own segments, load targets,
// claim (the ranges of the candidates are loaded alongside), store, barrier.
// Entries of at most kLvFew edges are expanded by eight lanes each, which needs
// neither the prefix sum nor the search of the balanced expansion (BFS 7.46 -> 6.49
// ms and reachability 5.58 -> 5.17 on the graphs below), by code for 4, 8, 16 or 32
// entries, so that a warp with three entries does not step through empty places
// (6.76 -> 6.08 and 4.69 -> 4.13; with 8 or 32 entries only, 6.2 to 8.1 and 5.1).
// BFS of a 1021 x 2043 grid (2,813 levels): 49.8 -> 6.1 ms, 2.1 us per level;
// backward push reachability on kNN 1.5e6: 37.6 -> 4.6 ms.
//
// The cluster hands the search back to the host's wide rounds when a level
// outgrows it (more than kLvMaxEdges edges, a vertex of more than kLvMaxDeg, which one warp
// would expand alone, a full segment, or the push/pull switch): every vertex of the next frontier is then written to the
// caller's queue.  No wait depends on anything but the hardware barrier, which
// all threads of the cluster reach the same number of times (every branch
// around it is taken on values that all blocks read from the same segment
// lengths).
#pragma once
#include <cooperative_groups.h>

#include <mutex>
#include <type_traits>

#include "common.cuh"

namespace psc {

constexpr int kLvBlocks = 16;    // blocks of the cluster
constexpr int kLvThreads = 512;  // one warp per segment
constexpr int kLvCap = 256;      // entries of one segment
constexpr int kLvK = 8;          // edges in flight per lane, balanced expansion
constexpr int kLvStep = 32;      // entries a warp takes at a time
constexpr uint32_t kLvFew = 24;  // edges of an entry that eight lanes expand
// Frontiers that enter the cluster, and the edges of a level that it keeps.
// 16 SMs claim about 10 edges per ns, so a level of 2^16 edges takes about as
// long as a host round of the whole GPU costs before it does any work.
constexpr uint64_t kLvMaxFront = 8192;
constexpr uint64_t kLvMaxEdges = 1 << 16;
// Out-edges of one vertex: four steps of a warp.  (Without this bound a hub of up to 65,536 was
// expanded by one warp: allocation-free reachability from the hub of R-MAT 2^20 0.29 ms with host
// rounds alone, 1.76 with the cluster, now 0.30; BFS of R-MAT 2^18 0.92 -> 0.17.)
constexpr uint32_t kLvMaxDeg = 1024;
// Edge sums are kept in 32 bits: a vertex, a warp and a block count for at
// most kLvSat each, far above kLvMaxEdges (16 * kLvSat < 2^32).
constexpr uint32_t kLvSat = 1u << 20;
static_assert(kLvThreads / 32 == kLvBlocks, "warp w expands the segment of block w");
static_assert(kLvMaxFront <= (uint64_t)kLvBlocks * kLvBlocks * kLvCap, "an entering frontier fits");

struct LvShared {
  // entries from each source block, double-buffered: beg << 24 | min(deg, 2^24 - 1)
  uint64_t rng[2][kLvBlocks][kLvCap];
  uint32_t vid[2][kLvBlocks][kLvCap];
  // per source block: claims of its last level, and the out-edges of those (at most
  // kLvSat; kLvSat too when a segment ran over, which ends the launch the same way)
  uint32_t edges[2][kLvBlocks];
  uint32_t claims[2][kLvBlocks];
  // this block's level in progress, double-buffered
  uint32_t my_edges[2];
  uint32_t my_claims[2];
  WarpExpandSmem sm[kLvThreads / 32];
};

struct LvArgs {
  const uint64_t* off;  // adjacency of the search direction
  const uint32_t* E;
  const uint32_t* qin;  // entering frontier
  uint64_t nin;
  uint32_t* qout;       // the frontier when the cluster hands back
  uint64_t threshold;   // hand back when frontier + out-edges reach this (pull switch)
  uint32_t level;       // levels done before this launch
  Counters* ctr;        // next / next_edges: the frontier handed back; aux0: levels run here;
                        // expanded / edges: vertices and edges of those levels
};

// Claims of the two searches: issue() is the atomic, won() says from its
// result whether this caller got v (apart, so that a lane's atomics overlap).
struct BfsClaim {
  uint32_t* dist;
  __device__ uint32_t issue(uint32_t v, uint32_t level) const {
    return atomicCAS(&dist[v], kNone, level);
  }
  __device__ bool won(uint32_t, uint32_t old) const { return old == kNone; }
};
struct ReachClaim {
  uint32_t* vis;
  __device__ uint32_t issue(uint32_t v, uint32_t) const {
    return atomicOr(&vis[v >> 5], 1u << (v & 31));
  }
  __device__ bool won(uint32_t v, uint32_t old) const { return !((old >> (v & 31)) & 1u); }
};

// Edges that a vertex counts for in the sums (kLvSat ends the launch).
__device__ __forceinline__ uint32_t lv_edges(uint64_t r) {
  const uint32_t d = (uint32_t)(r & 0xFFFFFFull);
  return d > kLvMaxDeg ? kLvSat : d;
}

// Whether narrow push levels should go to the cluster: from the second level on, and not
// while they grow so fast that the next one or two will be wide (a launch of the cluster
// costs some 5 us more than a host round: BFS of R-MAT 2^12 122 us with host rounds alone,
// 133 with one cluster level among them).  Launches that came back after a level or two
// (hubs) hold the next ones off, as does a pull round, after which few levels are left.
struct LvGate {
  uint64_t prev = 0;  // out-edges of the last level
  uint32_t rest = 0, penalty = 1;
  bool enter(uint32_t level, uint64_t nf, uint64_t nf_edges) {
    const bool slow = nf_edges <= 4 * (prev > 8 ? prev : 8);
    prev = nf_edges;
    if (level == 0 || !slow || nf > kLvMaxFront || nf_edges > kLvMaxEdges) return false;
    if (rest == 0) return true;
    rest--;
    return false;
  }
  void pulled() { rest = 3; }
  void ran(uint64_t levels) {
    rest = levels < 3 ? penalty : 0;
    penalty = levels < 3 ? (penalty < 64 ? 2 * penalty : 64) : 1;
  }
};

__device__ __forceinline__ uint64_t lv_pack(uint64_t beg, uint64_t end) {
  const uint64_t d = end - beg;
  return (beg << 24) | (d < 0xFFFFFFull ? d : 0xFFFFFFull);
}

template <class Claim>
__global__ void __launch_bounds__(kLvThreads) k_levels(LvArgs a, Claim claim) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) unsigned char lv_raw[];
  LvShared& sh = *reinterpret_cast<LvShared*>(lv_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank();
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  WarpExpandSmem& sm = sh.sm[wid];

  // entering frontier: vertex i goes to block i % 16, segment (i / 16) % 16
  if (threadIdx.x < kLvBlocks) {
    sh.claims[0][threadIdx.x] = 0;
    sh.edges[0][threadIdx.x] = 0;
  }
  if (threadIdx.x < 2) {
    sh.my_claims[threadIdx.x] = 0;
    sh.my_edges[threadIdx.x] = 0;
  }
  __syncthreads();
  const uint64_t mine = a.nin > rank ? (a.nin - rank + kLvBlocks - 1) / kLvBlocks : 0;
  uint32_t e_in = 0;
  for (uint64_t k = threadIdx.x; k < mine; k += kLvThreads) {
    const uint32_t u = a.qin[rank + k * kLvBlocks];
    const uint64_t r = lv_pack(a.off[u], a.off[u + 1]);
    sh.rng[0][k % kLvBlocks][k / kLvBlocks] = r;
    sh.vid[0][k % kLvBlocks][k / kLvBlocks] = u;
    e_in = min(e_in + lv_edges(r), kLvSat);
  }
  e_in = __reduce_add_sync(kFull, min(e_in, kLvSat));
  if (lane == 0 && e_in) atomicAdd(&sh.my_edges[1], e_in);
  cluster.sync();  // every block's arrays are set before others write to them
  if (threadIdx.x < kLvBlocks) {
    LvShared* d = cluster.map_shared_rank(&sh, threadIdx.x);
    d->edges[0][rank] = min(sh.my_edges[1], kLvSat);
    d->claims[0][rank] = (uint32_t)mine;
  }
  __syncthreads();
  if (threadIdx.x == 0) sh.my_edges[1] = 0;
  cluster.sync();

  // entries of segment s (this warp's) in the level to come
  uint32_t seg = wid < mine ? (uint32_t)((mine - wid + kLvBlocks - 1) / kLvBlocks) : 0;
  uint32_t cur = 0, levels = 0;
  unsigned long long done_v = 0, done_e = 0;
  for (;;) {
    // what all blocks claimed last level (the same numbers in every block)
    const uint32_t nf = __reduce_add_sync(kFull, lane < kLvBlocks ? sh.claims[cur][lane] : 0u);
    const uint32_t ne = __reduce_add_sync(kFull, lane < kLvBlocks ? sh.edges[cur][lane] : 0u);
    const bool stop = nf == 0 || ne > kLvMaxEdges || nf > 2 * kLvMaxFront ||
                      (levels && (uint64_t)nf + ne >= a.threshold);
    if (stop) {
      // the frontier goes back to the caller's queue (a run-over segment's
      // surplus is there already); ctr->next counts it
      const uint32_t n_seg = seg < (uint32_t)kLvCap ? seg : (uint32_t)kLvCap;
      unsigned long long base = 0;
      if (lane == 0 && n_seg) base = atomicAdd(&a.ctr->next, (unsigned long long)n_seg);
      base = __shfl_sync(kFull, base, 0);
      unsigned long long e = 0;  // exact: the push/pull switch is decided on it
      for (uint32_t at = lane; at < n_seg; at += 32) {
        const uint32_t u = sh.vid[cur][wid][at];
        a.qout[base + at] = u;
        e += a.off[u + 1] - a.off[u];
      }
      e = warp_sum(e);
      if (lane == 0 && e) atomicAdd(&a.ctr->next_edges, e);
      if (rank == 0 && threadIdx.x == 0) {
        a.ctr->aux0 = levels;
        a.ctr->expanded = done_v;
        a.ctr->edges = done_e;
      }
      break;
    }
    levels++;
    done_v += nf;
    done_e += ne;
    const uint32_t level = a.level + levels;
    const uint32_t nxt = cur ^ 1;
    uint32_t my_e = 0;
    // Deals the lane's claims (bit k of tm: v[k] with range r[k]).
    auto deal = [&](uint32_t tm, const uint32_t* v, const uint64_t* r, auto kk) {
      constexpr int N = decltype(kk)::value;
      unsigned m[N];
      uint32_t total = 0;
#pragma unroll
      for (int k = 0; k < N; k++) {
        m[k] = __ballot_sync(kFull, (tm >> k) & 1u);
        total += __popc(m[k]);
      }
      if (total == 0) return;
      uint32_t j = 0;
      if (lane == 0) j = atomicAdd(&sh.my_claims[cur], total);
      j = __shfl_sync(kFull, j, 0);
#pragma unroll
      for (int k = 0; k < N; k++) {
        if ((m[k] >> lane) & 1u) {
          const uint32_t i = j + __popc(m[k] & ((1u << lane) - 1u)), at = i / kLvBlocks;
          if (at < (uint32_t)kLvCap) {
            LvShared* d = cluster.map_shared_rank(&sh, (i + rank) % kLvBlocks);
            d->rng[nxt][rank][at] = r[k];
            d->vid[nxt][rank][at] = v[k];
          } else {
            a.qout[atomicAdd(&a.ctr->next, 1ull)] = v[k];
            atomicAdd(&a.ctr->next_edges, (unsigned long long)(a.off[v[k] + 1] - a.off[v[k]]));
            my_e = kLvSat;
          }
          my_e = min(my_e + lv_edges(r[k]), kLvSat);
        }
        j += __popc(m[k]);
      }
    };
    auto claim_all = [&](const uint32_t* v, uint64_t* r, auto kk) {
      constexpr int N = decltype(kk)::value;
      uint32_t old[N], tm = 0;
#pragma unroll
      for (int k = 0; k < N; k++) {
        r[k] = 0;
        old[k] = 0;
        if (v[k] != kNone) {
          old[k] = claim.issue(v[k], level);
          r[k] = lv_pack(__ldg(&a.off[v[k]]), __ldg(&a.off[v[k] + 1]));
        }
      }
#pragma unroll
      for (int k = 0; k < N; k++)
        if (v[k] != kNone && claim.won(v[k], old[k])) tm |= 1u << k;
      deal(tm, v, r, kk);
    };
    for (uint32_t i0 = 0; i0 < seg; i0 += kLvStep) {
      // low degrees: eight lanes per entry, lane j takes edges j, j + 8, ...
      const unsigned grp = lane >> 3, ej = lane & 7;
      auto few = [&](auto kk) {
        constexpr int N = decltype(kk)::value;
        uint64_t rr[N], r[N];
        uint32_t v[N];
        bool big = false;
#pragma unroll
        for (int k = 0; k < N; k++) {
          const uint32_t i = i0 + 4 * k + grp;
          rr[k] = i < seg ? sh.rng[cur][wid][i] : 0ull;
          big |= (rr[k] & 0xFFFFFFull) > kLvFew;
        }
        if (__any_sync(kFull, big)) return false;
        for (uint32_t j = ej;; j += 8) {
          bool more = false;
#pragma unroll
          for (int k = 0; k < N; k++) {
            const uint32_t d = (uint32_t)(rr[k] & 0xFFFFFFull);
            v[k] = j < d ? __ldg(&a.E[(rr[k] >> 24) + j]) : kNone;
            more |= j + 8 < d;
          }
          claim_all(v, r, kk);
          if (!__any_sync(kFull, more)) return true;
        }
      };
      const uint32_t left = seg - i0;
      if (left <= 4    ? few(std::integral_constant<int, 1>())
          : left <= 8  ? few(std::integral_constant<int, 2>())
          : left <= 16 ? few(std::integral_constant<int, 4>())
                       : few(std::integral_constant<int, kLvStep / 4>()))
        continue;
      // balanced expansion: the warp walks the concatenated ranges of the step's
      // entries, up to kLvK edges per lane in flight (the steps that nobody needs
      // are skipped as a whole)
      uint64_t beg = 0;
      uint32_t deg = 0;
      if (lane < (unsigned)kLvStep && i0 + lane < seg) {
        const uint64_t x = sh.rng[cur][wid][i0 + lane];
        beg = x >> 24;
        deg = (uint32_t)(x & 0xFFFFFFull);
      }
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
      for (uint32_t b = 0; b < total; b += 32 * kLvK) {
        uint32_t v[kLvK];
        uint64_t r[kLvK];
#pragma unroll
        for (int k = 0; k < kLvK; k++) {
          v[k] = kNone;
          if (b + k * 32 < total) {
            const uint32_t gi = b + k * 32 + lane;
            if (gi < total) {
              int lo = 0, hi = 31;
              while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (sm.excl[mid] <= gi)
                  lo = mid;
                else
                  hi = mid - 1;
              }
              v[k] = __ldg(&a.E[sm.beg[lo] + (gi - sm.excl[lo])]);
            }
          }
        }
        claim_all(v, r, std::integral_constant<int, kLvK>());
      }
      __syncwarp();
    }
    if (seg) {
      my_e = __reduce_add_sync(kFull, my_e);
      if (lane == 0 && my_e) atomicAdd(&sh.my_edges[cur], min(my_e, kLvSat));
    }
    if (threadIdx.x == 0) {  // the next level's sums (last read a barrier ago)
      sh.my_claims[nxt] = 0;
      sh.my_edges[nxt] = 0;
    }
    __syncthreads();
    if (threadIdx.x < kLvBlocks) {
      LvShared* d = cluster.map_shared_rank(&sh, threadIdx.x);
      d->claims[nxt][rank] = sh.my_claims[cur];
      d->edges[nxt][rank] = min(sh.my_edges[cur], kLvSat);
    }
    cluster.sync();
    cur = nxt;
    // source w's claims j with (j + w) % 16 == rank came to this block
    const uint32_t J = sh.claims[cur][wid], o = (rank + kLvBlocks - wid) % kLvBlocks;
    seg = J > o ? (J - o + kLvBlocks - 1) / kLvBlocks : 0;
  }
  cluster.sync();  // no block leaves while others may still write to its shared memory
}

// Whether the current device runs k_levels (a cluster of 16 blocks with its
// shared memory); asked once per device and instance.
template <class Claim>
bool levels_ready(int device) {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static int state[kMaxDev] = {};
  if (device < 0 || device >= kMaxDev) return false;
  std::lock_guard<std::mutex> lock(mu);
  if (state[device] == 0) {
    state[device] = -1;
    if (cudaFuncSetAttribute(k_levels<Claim>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(LvShared)) == cudaSuccess &&
        cudaFuncSetAttribute(k_levels<Claim>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
            cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = kLvBlocks;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.gridDim = dim3(kLvBlocks);
      cfg.blockDim = dim3(kLvThreads);
      cfg.dynamicSmemBytes = sizeof(LvShared);
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, k_levels<Claim>, &cfg) == cudaSuccess &&
          clusters > 0)
        state[device] = 1;
    }
    cudaGetLastError();
  }
  return state[device] == 1;
}

// One launch of k_levels; the counters must be zero.
template <class Claim>
int launch_levels(const LvArgs& a, Claim claim, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kLvBlocks;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(kLvBlocks);
  cfg.blockDim = dim3(kLvThreads);
  cfg.dynamicSmemBytes = sizeof(LvShared);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  PSC_CUDA(cudaLaunchKernelEx(&cfg, k_levels<Claim>, a, claim));
  return PSC_OK;
}

}  // namespace psc
