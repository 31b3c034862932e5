// Device transpose (make_directed, src/graph.hpp:222-245): the in-lists,
// sorted by source as the reference's sort-based transpose leaves them, from
// a stable radix sort of the (target, source) pairs by target.
#include "common.cuh"
#include "engines.cuh"
#include "scan.cuh"

namespace psc {

// ---------------------------------------------------------------------------
// Radix transpose: the (target, source) pairs of all edges, generated in CSR
// order (sorted by source), sorted by target with a stable LSD radix sort of
// kRsBits-bit digits.  Stability keeps every in-list ordered by source, as
// the reference's sort-based transpose leaves it.
//
// What bounds it is the traffic of the passes (16 bytes per pair and pass), as
// long as nothing else is read: the histograms of all digits come from one read of
// the keys, and a pass finds the places of its tiles' digit runs while it runs,
// by looking back over the tiles before it (decoupled look-back, after D. Merrill and
// M. Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016, and
// its use for radix passes by A. Adinets and D. Merrill, "Onesweep", 2022: a tile
// publishes its digit counts, later their prefix sums), so there is no histogram pass
// and no scan per digit.  Tiles are numbered by a ticket, so the tiles that one waits for
// are running or done; every wait is bounded.  A tile that gives up sets *failed: keys
// that no pass wrote must not be used as places, so every later kernel of the sort,
// and the offsets made of it, then writes nothing (k_rs_pass, k_bounds).
// R-MAT 2^22, 6.6e7 edges, 3 passes: histogram 0.37, scan 0.03 and scatter 0.60 ms
// per pass -> one read of 0.08 ms and 0.49 per pass; sources 0.35 -> 0.15, offsets
// 0.28 -> 0.08.
// ---------------------------------------------------------------------------
constexpr int kRsBits = 8;
constexpr int kRsBins = 1 << kRsBits;
constexpr int kRsBlock = 256;
constexpr int kRsTile = 4608;  // pairs per block and pass (12 per thread)
constexpr int kEsTile = 3072;  // edges per block of k_edge_sources (4608: 163 instead of 126 us)
#ifndef PSC_ES_WIDE
#define PSC_ES_WIDE (16 * kEsTile)
#endif
constexpr uint64_t kEsWide = PSC_ES_WIDE;
constexpr int kRsMaxPasses = 4;
constexpr int kRsLook = 4;
#ifndef PSC_RS_SPIN
#define PSC_RS_SPIN (1u << 22)
#endif
constexpr uint32_t kRsSpin = PSC_RS_SPIN;  // polls of one wait
// Status word of a (tile, digit): nothing yet, the tile's count, or the count of
// all tiles up to it.
constexpr uint64_t kRsCount = 1ull << 62, kRsPrefix = 2ull << 62, kRsValue = kRsCount - 1;

// src[e] = the vertex whose adjacency holds edge e.  A block takes kEsTile
// consecutive edges: each vertex whose list begins inside the tile marks its first
// edge, and a running maximum over the marks gives every edge its owner (instead
// of a binary search per edge).  A tile whose edges lie among more than kEsWide
// vertices, nearly all of them without edges, is searched after all: the walk over the
// vertices is one block's.  Upload and transpose of 6e7 vertices with 1e5 edges at both
// ends 104 -> 3.0 ms, spread evenly 6.2 -> 3.1; 32,768 vertices a tile (2^25 vertices, 3.1e6
// edges) walked 2.18, searched 2.27 ms; 65,536 2.13 and 2.11.
__device__ __forceinline__ uint64_t edge_owner(const uint64_t* __restrict__ off, uint64_t n,
                                               uint64_t e) {
  uint64_t lo = 0, hi = n - 1;
  while (lo < hi) {  // largest u with off[u] <= e
    const uint64_t mid = (lo + hi + 1) >> 1;
    if (__ldg(&off[mid]) <= e)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// owner[2 t], owner[2 t + 1]: the owners of the first and the last edge of tile t
// (searched for all tiles at once: inside the tile's block the 20-odd dependent
// steps were most of its time).
__global__ void k_tile_owners(const uint64_t* __restrict__ off, uint64_t n, uint64_t m,
                              uint32_t* owner) {
  const uint64_t ends = 2 * ((m + kEsTile - 1) / kEsTile);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ends;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t e0 = (i >> 1) * kEsTile;
    const uint64_t e1 = e0 + kEsTile < m ? e0 + kEsTile : m;
    owner[i] = (uint32_t)edge_owner(off, n, (i & 1) ? e1 - 1 : e0);
  }
}

// (eight blocks an SM: the walk lives on loads in flight)
__global__ void __launch_bounds__(kRsBlock, 8)
    k_edge_sources(const uint64_t* __restrict__ off, const uint32_t* __restrict__ owner,
                   uint64_t m, uint32_t* src) {
  constexpr int NW = kRsBlock / 32, PER = kEsTile / NW;
  __shared__ uint32_t mark[kEsTile];
  __shared__ uint32_t wmax[NW];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5, tid = threadIdx.x;
  const uint64_t ntiles = (m + kEsTile - 1) / kEsTile;
  for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint64_t e0 = tile * kEsTile;
    const uint64_t e1 = e0 + kEsTile < m ? e0 + kEsTile : m;
    const uint64_t v0 = __ldg(&owner[2 * tile]), v1 = __ldg(&owner[2 * tile + 1]);
    if (v1 - v0 > kEsWide) {
      constexpr int K = 4;  // searches of a thread side by side
      const uint64_t* o = off + v0;
#pragma unroll 1
      for (uint64_t eb = e0 + tid; eb < e1; eb += K * kRsBlock) {
        uint32_t lo[K], len[K];  // the owner lies in [lo, lo + len]
#pragma unroll
        for (int k = 0; k < K; k++) {
          lo[k] = 0;
          len[k] = (uint32_t)(v1 - v0);  // (n < 2^32 - 1)
        }
        for (int step = 32 - __clz((uint32_t)(v1 - v0)); step > 0; step--) {
#pragma unroll
          for (int k = 0; k < K; k++) {
            const uint32_t half = (len[k] + 1) >> 1;
            if (half) {
              const bool up = __ldg(&o[lo[k] + half]) <= eb + k * kRsBlock;
              lo[k] += up ? half : 0u;
              len[k] = up ? len[k] - half : half - 1;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < K; k++)
          if (eb + k * kRsBlock < e1) src[eb + k * kRsBlock] = (uint32_t)v0 + lo[k];
      }
      continue;
    }
    for (int i = tid; i < kEsTile; i += kRsBlock) mark[i] = 0;
    __syncthreads();
    for (uint64_t v = v0 + 1 + tid; v <= v1; v += kRsBlock)
      atomicMax(&mark[__ldg(&off[v]) - e0], (uint32_t)(v - v0));
    __syncthreads();
    uint32_t run = 0;  // maximum so far of the warp's part
    for (int c = 0; c < PER / 32; c++) {
      uint32_t x = mark[wid * PER + c * 32 + lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if ((int)lane >= o && y > x) x = y;
      }
      x = x > run ? x : run;
      mark[wid * PER + c * 32 + lane] = x;
      run = __shfl_sync(kFull, x, 31);
    }
    if (lane == 0) wmax[wid] = run;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < (int)wid; w++) before = wmax[w] > before ? wmax[w] : before;
    for (int c = 0; c < PER / 32; c++) {
      const uint64_t i = wid * PER + c * 32 + lane;
      const uint32_t x = mark[i];
      if (e0 + i < e1) src[e0 + i] = (uint32_t)v0 + (x > before ? x : before);
    }
    __syncthreads();
  }
}

// Counts of every digit of every pass in one read of the keys (per-warp
// histograms in shared memory).
template <int PASSES>
__global__ void __launch_bounds__(kRsBlock)
    k_rs_count(const uint32_t* __restrict__ keys, uint64_t m, unsigned long long* hist) {
  __shared__ uint32_t h[kRsBlock / 32][PASSES][kRsBins];
  const unsigned wid = threadIdx.x >> 5;
  uint32_t* all = &h[0][0][0];
  for (int i = threadIdx.x; i < kRsBlock / 32 * PASSES * kRsBins; i += kRsBlock) all[i] = 0;
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * kRsBlock;
  const uint64_t t = (uint64_t)blockIdx.x * kRsBlock + threadIdx.x;
  auto add = [&](uint32_t k) {
#pragma unroll
    for (int p = 0; p < PASSES; p++) atomicAdd(&h[wid][p][(k >> (p * kRsBits)) & (kRsBins - 1)], 1u);
  };
  const uint64_t nq = m / 4;
  const uint4* k4 = reinterpret_cast<const uint4*>(keys);  // (pool memory: 16-byte aligned)
  for (uint64_t q = t; q < nq; q += stride) {
    const uint4 x = __ldg(&k4[q]);
    add(x.x);
    add(x.y);
    add(x.z);
    add(x.w);
  }
  for (uint64_t i = nq * 4 + t; i < m; i += stride) add(keys[i]);
  __syncthreads();
  for (int i = threadIdx.x; i < PASSES * kRsBins; i += kRsBlock) {
    unsigned long long c = 0;
    for (int w = 0; w < kRsBlock / 32; w++) c += h[w][i / kRsBins][i % kRsBins];
    if (c) atomicAdd(&hist[i], c);
  }
}

// Digit starts of a pass: the exclusive sums of its counts, in place.
__global__ void __launch_bounds__(kRsBins) k_rs_starts(unsigned long long* hist) {
  __shared__ uint64_t sm[33];
  unsigned long long* h = hist + (uint64_t)blockIdx.x * kRsBins;
  uint64_t all;
  const uint64_t start = block_excl_scan<kRsBins>(h[threadIdx.x], sm, &all);
  h[threadIdx.x] = start;
}

// One stable pass.  Each warp owns a twelfth of the tile, consecutive pairs
// (chunks of 32 in order, lanes in order), held in registers.  The tile is sorted
// by digit in shared memory (warp counts, a block scan over digits, ranked
// placement), then written out so that consecutive threads write consecutive
// positions of one digit's run: coalesced stores instead of one sector per pair.
// 384 threads and three blocks an SM: the pass is a chain of ballots, shared-memory
// round trips and block barriers, so it lives on warps in flight; the values are
// loaded only behind the ranking, which keeps the registers low enough for it.
// (load and solve of R-MAT 2^22, 6.7e7 edges: 256 threads x 12 pairs 5.17 ms, 384 x 12
// 5.02, 384 x 8 and 512 x 8 5.04, 384 x 10 5.12, 512 x 12 5.19.)
constexpr int kRpBlock = 384;
constexpr int kRsPer = kRsTile / kRpBlock;  // keys per thread
static_assert(kRsTile % kRpBlock == 0 && kRsTile % kRsBlock == 0, "whole chunks per warp");

// (Pairs as 64-bit words between passes were measured and dropped: 0.61 ms a pass
// instead of 0.53 then, the ranked placement then meets twice the bank conflicts.)
__global__ void __launch_bounds__(kRpBlock, 3)
    k_rs_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint64_t m,
              int shift, const unsigned long long* __restrict__ starts, uint32_t* ticket,
              unsigned long long* status, uint32_t* kout, uint32_t* vout,
              unsigned long long* failed) {
  constexpr int NW = kRpBlock / 32;
  constexpr int PER_WARP = kRsTile / NW;
  static_assert(kRsBins <= kRpBlock, "one digit per thread in the digit scan");
  __shared__ uint32_t skey[kRsTile];
  __shared__ uint32_t sval[kRsTile];
  __shared__ uint32_t wcnt[NW][kRsBins];
  __shared__ uint64_t gbase[kRsBins];
  __shared__ uint64_t scan_sm[33];
  __shared__ uint32_t s_tile, s_bad;
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5, tid = threadIdx.x;
  const unsigned lt = (1u << lane) - 1;
  if (tid == 0) {
    s_tile = atomicAdd(ticket, 1u);
    s_bad = *(volatile unsigned long long*)failed != 0;
  }
  for (int b = lane; b < kRsBins; b += 32) wcnt[wid][b] = 0;
  __syncthreads();
  if (s_bad) return;  // an earlier pass gave up (or a tile of this one: its waiters do too)
  const uint64_t tile = s_tile;
  const uint64_t tbase = tile * kRsTile;
  const uint64_t base = tbase + (uint64_t)wid * PER_WARP;
  const uint32_t tcount = (uint32_t)(m - tbase < (uint64_t)kRsTile ? m - tbase : kRsTile);
  uint32_t key[kRsPer], val[kRsPer];
#pragma unroll
  for (int c = 0; c < kRsPer; c++) {
    const uint64_t i = base + c * 32 + lane;
    key[c] = i < m ? __ldg(&kin[i]) : 0u;
  }
  // rank of each pair among the warp's pairs of its digit: lanes of a chunk with the
  // same digit are found by one ballot per digit bit (by atomicOr of lane masks in
  // shared memory: 0.63 ms a pass instead of 0.52)
  uint32_t rank[kRsPer];
#pragma unroll
  for (int c = 0; c < kRsPer; c++) {
    const bool in = base + c * 32 + lane < m;
    const uint32_t d = (key[c] >> shift) & (kRsBins - 1);
    unsigned p = __ballot_sync(kFull, in);
#pragma unroll
    for (int b = 0; b < kRsBits; b++) {
      const bool bit = (d >> b) & 1u;
      const unsigned v = __ballot_sync(kFull, bit);
      p &= bit ? v : ~v;
    }
    const uint32_t at = wcnt[wid][d];
    __syncwarp();
    rank[c] = at + __popc(p & lt);
    if (in && (p & lt) == 0) wcnt[wid][d] = at + __popc(p);
    __syncwarp();
  }
#pragma unroll
  for (int c = 0; c < kRsPer; c++) {
    const uint64_t i = base + c * 32 + lane;
    val[c] = i < m ? __ldg(&vin[i]) : 0u;
  }
  __syncthreads();
  // digit tid: the tile's count is published, then its start in the sorted tile
  // and each warp's base inside it
  const bool dig = kRpBlock == kRsBins || tid < kRsBins;
  uint32_t total = 0;
#pragma unroll
  for (int w = 0; w < NW; w++) total += dig ? wcnt[w][tid] : 0u;
  volatile unsigned long long* row = status + tile * kRsBins + tid;
  if (dig) *row = (tile ? kRsCount : kRsPrefix) | total;
  uint64_t all = 0;
  const uint32_t start = (uint32_t)block_excl_scan<kRpBlock>(total, scan_sm, &all);
  uint32_t run = start;
#pragma unroll
  for (int w = 0; w < NW; w++) {
    if (dig) {
      const uint32_t c = wcnt[w][tid];
      wcnt[w][tid] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kRsPer; c++) {
    if (base + c * 32 + lane < m) {
      const uint32_t lp = wcnt[wid][(key[c] >> shift) & (kRsBins - 1)] + rank[c];
      skey[lp] = key[c];
      sval[lp] = val[c];
    }
  }
  // look back, kRsLook tiles' words at a time (8 / 16 / 32 at a time: 1 / 2 / 8 %
  // slower; the pass is bound by instructions, not by this wait)
  uint64_t before = 0;
  bool open = dig && tile > 0;
  for (uint64_t t = tile; open;) {
    unsigned long long x[kRsLook];
#pragma unroll
    for (int k = 0; k < kRsLook; k++)
      x[k] = t > (uint64_t)k ? *(volatile unsigned long long*)(status + (t - 1 - k) * kRsBins + tid)
                             : kRsPrefix;
#pragma unroll
    for (int k = 0; k < kRsLook; k++) {
      if (!open) break;
      uint32_t spin = 0;
      while (!(x[k] >> 62)) {
        if (++spin > kRsSpin ||
            ((spin & 1023u) == 0 && *(volatile unsigned long long*)failed)) {
          s_bad = 1;
          open = false;
          break;
        }
        x[k] = *(volatile unsigned long long*)(status + (t - 1 - k) * kRsBins + tid);
      }
      before += x[k] & kRsValue;
      if (x[k] >> 63) open = false;
    }
    t -= t < (uint64_t)kRsLook ? t : (uint64_t)kRsLook;
    if (t == 0) open = false;
  }
  if (dig && tile) *row = kRsPrefix | (before + total);
  if (dig) gbase[tid] = starts[tid] + before - start;
  __syncthreads();
  if (s_bad) {
    if (tid == 0) *failed = 1;
    return;
  }
  for (uint32_t j = tid; j < tcount; j += kRpBlock) {
    const uint32_t k = skey[j];
    const uint64_t pos = gbase[(k >> shift) & (kRsBins - 1)] + j;
    kout[pos] = k;
    vout[pos] = sval[j];
  }
}

// off[v] = first place of the sorted array t[0 .. m) with t >= v, for v in [0, n]:
// the places between two neighbours t[i - 1] < t[i] belong to v in (t[i - 1], t[i]].
// Gaps of more than kGapLong ids are listed (end of the range, value, start) and
// filled by the whole grid afterwards.
constexpr uint32_t kGapLong = 64;

struct GapEnt {
  uint64_t first, last, value;  // off[first .. last] = value
};

// Nothing is written when the sort that made t gave up (*failed).
__global__ void k_bounds(const uint32_t* __restrict__ t, uint64_t m, uint64_t n, uint64_t* off,
                         GapEnt* gaps, unsigned long long* ngaps,
                         const unsigned long long* __restrict__ failed) {
  if (*failed) return;
  // ids after the one before place i, up to the one at place i
  auto place = [&](uint64_t i, uint64_t a, uint64_t b) {
    if (b + 1 > a + kGapLong) {
      gaps[atomicAdd(ngaps, 1ull)] = GapEnt{a, b, i};
    } else {
      for (uint64_t v = a; v <= b; v++) off[v] = i;
    }
  };
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t nq = m / 4;
  const uint4* t4 = reinterpret_cast<const uint4*>(t);  // (pool memory: 16-byte aligned)
  for (uint64_t q = g; q < nq; q += stride) {
    const uint4 x = __ldg(&t4[q]);
    const uint64_t a = q ? (uint64_t)__ldg(&t[4 * q - 1]) + 1 : 0;
    place(4 * q, a, x.x);
    place(4 * q + 1, (uint64_t)x.x + 1, x.y);
    place(4 * q + 2, (uint64_t)x.y + 1, x.z);
    place(4 * q + 3, (uint64_t)x.z + 1, x.w);
  }
  for (uint64_t i = nq * 4 + g; i <= m; i += stride)
    place(i, i ? (uint64_t)t[i - 1] + 1 : 0, i < m ? t[i] : n);
}

__global__ void k_fill_gaps(const GapEnt* __restrict__ gaps, const unsigned long long* __restrict__ ngaps,
                            uint64_t* off) {
  const uint64_t ng = *ngaps;
  const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t gt = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // short lists of long gaps: every gap over the grid; else a warp per gap
  if (ng < 64) {
    for (uint64_t g = 0; g < ng; g++) {
      const GapEnt e = gaps[g];
      for (uint64_t v = e.first + gt; v <= e.last; v += nt) off[v] = e.value;
    }
  } else {
    for (uint64_t g = gt >> 5; g < ng; g += nt >> 5) {
      const GapEnt e = gaps[g];
      for (uint64_t v = e.first + (gt & 31); v <= e.last; v += 32) off[v] = e.value;
    }
  }
}

static int fill_bounds(psc_graph_s* g, const uint32_t* t, uint64_t m, uint64_t* off) {
  const uint64_t n = g->n;
  GapEnt* gaps;
  PSC_TRY(ensure_t(g, B_SCAN3, n / kGapLong + 2, &gaps));
  unsigned long long* ngaps = &g->ctr[3].aux0;  // staging set
  PSC_CUDA(cudaMemsetAsync(ngaps, 0, 8, g->stream));
  {
    ProfScope ps(g, F_TRANSPOSE);
    ps.bytes = 4.0 * m + 8.0 * n;
    k_bounds<<<grid_for(g, m + 1, 256), 256, 0, g->stream>>>(t, m, n, off, gaps, ngaps,
                                                             &g->ctr[3].aux1);
    k_fill_gaps<<<g->num_sms * 4, 256, 0, g->stream>>>(gaps, ngaps, off);
  }
  PSC_CUDA(cudaGetLastError());
  return PSC_OK;
}

static int digit_passes(uint64_t n) {
  int bits = 1;
  while (bits < 32 && ((uint64_t)1 << bits) < n) bits++;
  return (bits + kRsBits - 1) / kRsBits;
}

// Scratch of a sort: digit counts of every pass, tickets and status words.
struct RsScratch {
  unsigned long long *hist, *status, *failed;
  uint32_t* ticket;
};

static int rs_scratch(psc_graph_s* g, uint64_t cnt, RsScratch* r) {
  const uint64_t ntiles = (cnt + kRsTile - 1) / kRsTile;
  PSC_TRY(ensure_t(g, B_AUX3, ntiles * kRsBins, &r->status));
  PSC_TRY(ensure_t(g, B_SCAN2, kRsMaxPasses * kRsBins + 2, &r->hist));
  r->ticket = (uint32_t*)(r->hist + kRsMaxPasses * kRsBins);
  r->failed = &g->ctr[3].aux1;  // staging set, read by rs_check and fill_bounds
  PSC_CUDA(cudaMemsetAsync(r->failed, 0, 8, g->stream));
  return PSC_OK;
}

// The owners use the status words' room (a sort clears those before each pass).
static void launch_edge_sources(psc_graph_s* g, const RsScratch& r, uint32_t* src) {
  const uint64_t ntiles = (g->m + kEsTile - 1) / kEsTile;
  uint32_t* owner = (uint32_t*)r.status;
  k_tile_owners<<<grid_for(g, 2 * ntiles, 128), 128, 0, g->stream>>>(g->off, g->n, g->m, owner);
  k_edge_sources<<<(unsigned)std::min<uint64_t>(ntiles, g->num_sms * 8), kRsBlock, 0, g->stream>>>(
      g->off, owner, g->m, src);
}

// The digit counts of all passes over keys.
static int rs_count(psc_graph_s* g, const uint32_t* keys, uint64_t cnt, int passes,
                    const RsScratch& r) {
  PSC_CUDA(cudaMemsetAsync(r.hist, 0, kRsMaxPasses * kRsBins * 8, g->stream));
  ProfScope ps(g, F_TRANSPOSE);
  ps.bytes = 4.0 * cnt;
  const unsigned grid = (unsigned)std::min<uint64_t>((cnt + kRsTile - 1) / kRsTile, g->num_sms * 6);
  switch (passes) {
    case 1: k_rs_count<1><<<grid, kRsBlock, 0, g->stream>>>(keys, cnt, r.hist); break;
    case 2: k_rs_count<2><<<grid, kRsBlock, 0, g->stream>>>(keys, cnt, r.hist); break;
    case 3: k_rs_count<3><<<grid, kRsBlock, 0, g->stream>>>(keys, cnt, r.hist); break;
    default: k_rs_count<4><<<grid, kRsBlock, 0, g->stream>>>(keys, cnt, r.hist); break;
  }
  k_rs_starts<<<passes, kRsBins, 0, g->stream>>>(r.hist);
  PSC_CUDA(cudaGetLastError());
  return PSC_OK;
}

// All passes over cnt pairs: from (kin, vin), by way of pair[0] and pair[1] (cnt
// keys, then cnt values, each), into (kout, vout).
static int rs_sort(psc_graph_s* g, uint64_t cnt, int passes, const uint32_t* kin,
                   const uint32_t* vin, uint64_t* pair[2], const RsScratch& r, uint32_t* kout,
                   uint32_t* vout) {
  const uint64_t ntiles = (cnt + kRsTile - 1) / kRsTile;
  PSC_TRY(rs_count(g, kin, cnt, passes, r));
  for (int p = 0; p < passes; p++) {
    PSC_CUDA(cudaMemsetAsync(r.status, 0, ntiles * kRsBins * 8, g->stream));
    PSC_CUDA(cudaMemsetAsync(r.ticket, 0, 4, g->stream));
    ProfScope ps(g, F_TRANSPOSE);
    ps.bytes = 16.0 * cnt;
    const bool first = p == 0, last = p + 1 == passes;
    const uint32_t* ki = first ? kin : (const uint32_t*)pair[(p + 1) & 1];
    uint32_t* ko = last ? kout : (uint32_t*)pair[p & 1];
    k_rs_pass<<<(unsigned)ntiles, kRpBlock, 0, g->stream>>>(
        ki, first ? vin : ki + cnt, cnt, p * kRsBits, r.hist + (uint64_t)p * kRsBins, r.ticket,
        r.status, ko, last ? vout : ko + cnt, r.failed);
    PSC_CUDA(cudaGetLastError());
  }
  return PSC_OK;
}

// Waits for the sorts queued so far; an error if one gave up a wait.
static int rs_check(psc_graph_s* g) {
  PSC_TRY(read_counters(g));
  return g->hctr[3].aux1 ? PSC_ERR_ITER_LIMIT : PSC_OK;
}

int build_transpose(psc_graph_s* g) {
  const uint64_t n = g->n, m = g->m;
  if (m == 0) {
    PSC_CUDA(cudaMemsetAsync(g->in_off, 0, (n + 1) * 8, g->stream));
    return PSC_OK;
  }
  const int passes = digit_passes(n);
  uint32_t *src, *key;
  uint64_t* pair[2];
  PSC_TRY(ensure_t(g, B_AUX0, m, &src));
  PSC_TRY(ensure_t(g, B_QA, m, &key));
  PSC_TRY(ensure_t(g, B_AUX1, m, &pair[0]));
  PSC_TRY(ensure_t(g, B_AUX2, m, &pair[1]));
  RsScratch r;
  PSC_TRY(rs_scratch(g, m, &r));
  {
    ProfScope ps(g, F_TRANSPOSE);
    ps.bytes = 16.0 * n + 4.0 * m;
    launch_edge_sources(g, r, src);
  }
  PSC_TRY(rs_sort(g, m, passes, g->E, src, pair, r, key, g->in_E));
  PSC_TRY(fill_bounds(g, key, m, g->in_off));
  return rs_check(g);
}


// ---------------------------------------------------------------------------
// Device symmetrisation (make_symmetric, src/graph.hpp:187-220): every edge in
// both directions, each adjacency list sorted, duplicates and self-loops
// dropped.  The 2m pairs (a, b) -- a's list holds b -- are sorted by b and
// then stably by a with the radix passes above (an LSD sort of the key
// (a, b)); one compaction keeps the first pair of every run of equal pairs
// when a != b, writing the targets; the offsets come from the kept sources.
// ---------------------------------------------------------------------------
__global__ void k_sym_pairs(const uint32_t* __restrict__ E, const uint32_t* __restrict__ src,
                            uint64_t m, uint32_t* key, uint32_t* val) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t a = src[i], b = E[i];
    key[i] = b;  // first pass set: sort by the target
    val[i] = a;
    key[m + i] = a;  // the reverse edge b -> a
    val[m + i] = b;
  }
}

struct SymKeep {  // first of a run of equal (a, b) pairs, a != b
  const uint32_t* A;
  const uint32_t* B;
  __device__ uint32_t operator()(uint64_t i) const {
    const uint32_t a = A[i], b = B[i];
    if (a == b) return 0u;
    return (i == 0 || A[i - 1] != a || B[i - 1] != b) ? 1u : 0u;
  }
};

struct SymEmit {
  const uint32_t* A;
  const uint32_t* B;
  uint32_t* a_out;
  uint32_t* b_out;
  __device__ void operator()(uint64_t i, uint64_t excl, uint32_t v) const {
    if (v) {
      a_out[excl] = A[i];
      b_out[excl] = B[i];
    }
  }
};

int build_symmetric(psc_graph_s* g) {
  const uint64_t n = g->n, m = g->m;
  uint64_t* off_s = nullptr;
  uint32_t* E_s = nullptr;
  uint64_t ms = 0;
  if (m > 0) {
    const uint64_t c = 2 * m;
    const int passes = digit_passes(n);
    uint32_t *k, *v;  // the pairs, between and after the sorts
    uint64_t* pair[2];
    PSC_TRY(ensure_t(g, B_AUX0, c, &k));
    PSC_TRY(ensure_t(g, B_QA, c, &v));
    PSC_TRY(ensure_t(g, B_AUX1, c, &pair[0]));
    PSC_TRY(ensure_t(g, B_AUX2, c, &pair[1]));
    RsScratch r;
    PSC_TRY(rs_scratch(g, c, &r));
    uint32_t* src = (uint32_t*)pair[0];
    {
      ProfScope ps(g, F_TRANSPOSE);
      ps.bytes = 16.0 * n + 4.0 * m;
      launch_edge_sources(g, r, src);
    }
    {
      ProfScope ps(g, F_TRANSPOSE);
      ps.bytes = 8.0 * m + 16.0 * m;
      k_sym_pairs<<<grid_for(g, m, 256), 256, 0, g->stream>>>(g->E, src, m, k, v);
    }
    // by target, then stably by source (a single pass cannot end where it begins)
    uint32_t* k1 = passes == 1 ? (uint32_t*)pair[0] : k;
    uint32_t* v1 = passes == 1 ? (uint32_t*)pair[1] : v;
    PSC_TRY(rs_sort(g, c, passes, k, v, pair, r, k1, v1));
    PSC_TRY(rs_sort(g, c, passes, v1, k1, pair, r, v, k));
    PSC_TRY(rs_check(g));
    const uint32_t *A = v, *B = k;  // sources, targets
    PSC_TRY(release_buf(g, B_AUX3));
    PSC_TRY(release_buf(g, B_SCAN2));
    // the kept pairs: sources and targets
    uint32_t *asel = (uint32_t*)pair[0], *bsel = (uint32_t*)pair[1];
    PSC_TRY(scan_emit_flags(g, c, SymKeep{A, B}, SymEmit{A, B, asel, bsel}, &ms, F_TRANSPOSE,
                            8.0, 8.0));
    PSC_CUDA(cudaMallocAsync((void**)&E_s, (ms ? ms : 1) * 4, g->stream));
    if (ms) PSC_CUDA(cudaMemcpyAsync(E_s, bsel, ms * 4, cudaMemcpyDeviceToDevice, g->stream));
    PSC_CUDA(cudaMallocAsync((void**)&off_s, (n + 1) * 8, g->stream));
    PSC_TRY(fill_bounds(g, asel, ms, off_s));
    PSC_TRY(release_buf(g, B_AUX0));
    PSC_TRY(release_buf(g, B_AUX1));
    PSC_TRY(release_buf(g, B_AUX2));
    PSC_TRY(release_buf(g, B_QA));
    PSC_TRY(release_buf(g, B_SCAN3));
  } else {
    PSC_CUDA(cudaMallocAsync((void**)&E_s, 4, g->stream));
    PSC_CUDA(cudaMallocAsync((void**)&off_s, (n + 1) * 8, g->stream));
    PSC_CUDA(cudaMemsetAsync(off_s, 0, (n + 1) * 8, g->stream));
  }
  PSC_CUDA(cudaStreamSynchronize(g->stream));
  if (g->in_off && g->in_off != g->off) cudaFreeAsync(g->in_off, g->stream);
  if (g->in_E && g->in_E != g->E) cudaFreeAsync(g->in_E, g->stream);
  cudaFreeAsync(g->off, g->stream);
  cudaFreeAsync(g->E, g->stream);
  g->off = g->in_off = off_s;
  g->E = g->in_E = E_s;
  g->m = ms;
  g->symmetric = true;
  PSC_CUDA(cudaGetLastError());
  return PSC_OK;
}

}  // namespace psc
