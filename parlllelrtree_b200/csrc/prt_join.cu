// Breadth-first batched join: every query descends the tree level by level,
// all queries at once.  A frontier item is (query, node); a group of G lanes
// (G = fanout rounded up to a power of two) tests the node's entries against
// the query box, a warp ballot compacts the hits, and one atomicAdd per warp
// reserves their slots in the next frontier (or, at the leaf level, in the
// pair output).  Frontier counts stay on the device and every launch
// grid-strides over the current count, so a whole join is a fixed sequence of
// launches with no host round trip until the final count is read.
//
// Two forms of that step: expand_kernel reserves output slots with atomics
// (prt_join into a buffer of known capacity, the allocation-free join, the
// graph pipeline); or the hits of a level are counted per tile of the frontier
// first and written at their places by a second launch, so that frontiers and
// pairs stay in (query, entry) order and need no sort (prt_join_begin).  Window
// counts visit the tree depth first instead, a warp per query with the
// counters in registers (counts_kernel).  The last two prune: a query that
// contains the box of an entry intersects every record below it, so nothing below
// is tested.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include "prt_internal.cuh"

namespace prt {
namespace {

constexpr int kJoinBlock = 256;

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

struct JoinLevel {
  const void *mbr;          // entries of node level l (Box<T>)
  int64_t n_entries;        // entries at level l
  const uint2 *in;          // frontier (query, node); nullptr = (q, 0) for all queries
  const unsigned long long *in_count;
  int64_t in_cap;
  uint2 *out;               // next frontier, or pairs at the leaf level
  unsigned long long *out_count;
  int64_t out_cap;
  int leaf;                 // 1: emit (entry, query) pairs
  int64_t nq;
  long long *counts;        // optional per-query reference counters
  int td_slots;
};

// One block iteration takes kJoinRounds rounds of kGroups items per warp: the
// frontier items of all rounds are loaded first, then their node entries, so
// each warp has that many independent loads in flight; the hits of the whole
// iteration are reserved with one atomicAdd per block.  Measured on the
// 1M-window join of the 10M-box tree (F = 16) with the grid sized to one
// resident wave: 3, 4, 6 rounds take 3.00, 3.29, 3.07 ms.
constexpr int kJoinRounds = 3;

template <typename T, int G>
__global__ void __launch_bounds__(kJoinBlock) expand_kernel(JoinLevel J, const Box<T> *__restrict__ queries,
                                                            int fanout) {
  const Box<T> *mbr = reinterpret_cast<const Box<T> *>(J.mbr);
  const int lane = threadIdx.x & 31;
  const int sub = lane / G;           // group within the warp
  const int e = lane % G;             // entry within the node
  constexpr int kGroups = 32 / G;
  constexpr int kWarps = kJoinBlock / 32;
  const uint32_t gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (sub * G));
  const uint32_t lt = lanemask_lt();
  int64_t count = J.in ? (int64_t)min((unsigned long long)J.in_cap, *J.in_count) : J.nq;
  __shared__ uint32_t s_wcount[2][kWarps];
  __shared__ unsigned long long s_base[2];
  const int warp = threadIdx.x >> 5;
  const int64_t per_warp = (int64_t)kJoinRounds * kGroups;
  const int64_t per_block = (int64_t)kWarps * per_warp;
  int par = 0;
  for (int64_t bb = blockIdx.x * per_block; bb < count; bb += (int64_t)gridDim.x * per_block, par ^= 1) {
    const int64_t wb = bb + warp * per_warp;
    uint32_t q[kJoinRounds], node[kJoinRounds];
#pragma unroll
    for (int r = 0; r < kJoinRounds; r++) {
      const int64_t item = wb + r * kGroups + sub;
      q[r] = 0;
      node[r] = 0;
      if (item < count) {
        if (J.in) {
          const uint2 it = J.in[item];
          q[r] = it.x;
          node[r] = it.y;
        } else {
          q[r] = (uint32_t)item;
        }
      }
    }
    uint32_t ballots[kJoinRounds];
    uint32_t wtot = 0;
#pragma unroll
    for (int r = 0; r < kJoinRounds; r++) {
      const int64_t item = wb + r * kGroups + sub;
      const bool live = item < count;
      bool hit = false;
      if (live && e < fanout) {
        const Box<T> qb = load_box(queries, q[r]);
        const Box<T> eb = load_box(mbr, (int64_t)node[r] * fanout + e);  // padded slots intersect nothing
        hit = overlaps(eb, qb);
      }
      ballots[r] = __ballot_sync(0xffffffffu, hit);
      wtot += __popc(ballots[r]);
      if (J.counts && live && e == 0) {
        const int k = __popc(ballots[r] & gmask);
        const int64_t fill = J.td_slots ? fanout : min((int64_t)fanout, J.n_entries - (int64_t)node[r] * fanout);
        unsigned long long *c = reinterpret_cast<unsigned long long *>(&J.counts[3 * (int64_t)q[r]]);
        atomicAdd(&c[0], (unsigned long long)fill);
        if (k > 1) atomicAdd(&c[1], (unsigned long long)(k - 1));
        if (J.leaf && k) atomicAdd(&c[2], (unsigned long long)k);
      }
    }
    // one reservation per block iteration (warp counts double-buffered by
    // iteration parity, so one barrier separates the writes and the reads)
    if (lane == 0) s_wcount[par][warp] = wtot;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t tot = 0;
#pragma unroll
      for (int w = 0; w < kWarps; w++) tot += s_wcount[par][w];
      s_base[par] = tot ? atomicAdd(J.out_count, (unsigned long long)tot) : 0ull;
    }
    __syncthreads();
    if (wtot) {
      unsigned long long slot = s_base[par];
#pragma unroll
      for (int w = 0; w < kWarps; w++) slot += w < warp ? s_wcount[par][w] : 0u;
#pragma unroll
      for (int r = 0; r < kJoinRounds; r++) {
        if (ballots[r] >> lane & 1u) {
          const unsigned long long at = slot + __popc(ballots[r] & lt);
          const uint32_t entry = node[r] * (uint32_t)fanout + (uint32_t)e;
          if ((int64_t)at < J.out_cap) J.out[at] = J.leaf ? make_uint2(entry, q[r]) : make_uint2(q[r], entry);
        }
        slot += __popc(ballots[r]);
      }
    }
  }
}

// Resident blocks per SM of expand_kernel<T, G> (once per instantiation): the
// grid is exactly one wave, since a block beyond it would process its share
// of every grid-stride loop after the others.
template <typename T, int G>
int expand_blocks() {
  static std::atomic<int> per_sm{0};
  int b = per_sm.load(std::memory_order_relaxed);
  if (b == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, expand_kernel<T, G>, kJoinBlock, 0) != cudaSuccess || b < 1) {
      cudaGetLastError();
      b = 4;
    }
    per_sm.store(b, std::memory_order_relaxed);
  }
  return kSMs * b;
}

template <typename T>
int launch_expand(const JoinLevel &J, const void *queries, int fanout, cudaStream_t s) {
  const Box<T> *q = reinterpret_cast<const Box<T> *>(queries);
  if (fanout <= 2) {
    PRT_PROF("expand", s);
    expand_kernel<T, 2><<<expand_blocks<T, 2>(), kJoinBlock, 0, s>>>(J, q, fanout);
  }
  else if (fanout <= 4) {
    PRT_PROF("expand", s);
    expand_kernel<T, 4><<<expand_blocks<T, 4>(), kJoinBlock, 0, s>>>(J, q, fanout);
  }
  else if (fanout <= 8) {
    PRT_PROF("expand", s);
    expand_kernel<T, 8><<<expand_blocks<T, 8>(), kJoinBlock, 0, s>>>(J, q, fanout);
  }
  else if (fanout <= 16) {
    PRT_PROF("expand", s);
    expand_kernel<T, 16><<<expand_blocks<T, 16>(), kJoinBlock, 0, s>>>(J, q, fanout);
  }
  else {
    PRT_PROF("expand", s);
    expand_kernel<T, 32><<<expand_blocks<T, 32>(), kJoinBlock, 0, s>>>(J, q, fanout);
  }
  return PRT_OK;
}

// Overlapping pairs of sibling entries (the reference's RtreeSearch1,
// BotomUp-rtree.cu:574-590, TopDown-rtree.cu:78-93): for every node of every
// level, the entry pairs j < i < fill whose boxes intersect.  One warp per
// node, lane i holds entry i and counts its overlaps with the entries before
// it, which it receives by shuffles; one atomic per warp.
template <typename T>
__global__ void __launch_bounds__(256) sibling_kernel(const Box<T> *__restrict__ lv, int64_t n_entries, int fanout,
                                                      unsigned long long *__restrict__ total) {
  const int lane = threadIdx.x & 31;
  const int64_t nodes = (n_entries + fanout - 1) / fanout;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long acc = 0;
  for (int64_t node = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; node < nodes; node += nw) {
    const int64_t first = node * fanout;
    const int fill = (int)min((int64_t)fanout, n_entries - first);
    Box<T> b = empty_box<T>();
    if (lane < fill) b = load_box(lv, first + lane);
    unsigned c = 0;
    for (int j = 0; j < fill - 1; j++) {
      Box<T> o;
      o.x1 = __shfl_sync(0xffffffffu, b.x1, j);
      o.y1 = __shfl_sync(0xffffffffu, b.y1, j);
      o.x2 = __shfl_sync(0xffffffffu, b.x2, j);
      o.y2 = __shfl_sync(0xffffffffu, b.y2, j);
      c += (j < lane && lane < fill && overlaps(b, o)) ? 1u : 0u;
    }
    acc += c;
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0 && acc) atomicAdd(total, acc);
}

// Frontier capacity that worked last time (grows across calls; shared by the
// process's threads, so it is atomic).
std::atomic<int64_t> g_frontier_hint{1 << 20};

int check_join(const prt_tree *t, const void *d_queries, int coord, int64_t nq, const void *d_pairs, int64_t cap) {
  PRT_CHECK(t != nullptr, PRT_ERR_INVALID, "tree is NULL");
  PRT_CHECK(coord == t->coord, PRT_ERR_INVALID, "query coordinate type %d differs from the tree's %d", coord,
            t->coord);
  PRT_CHECK(nq >= 0 && nq < (1ll << 31), PRT_ERR_INVALID, "nq=%lld", (long long)nq);
  PRT_CHECK(cap >= 0, PRT_ERR_INVALID, "cap < 0");
  PRT_CHECK((reinterpret_cast<uintptr_t>(d_queries) & 15) == 0 && (reinterpret_cast<uintptr_t>(d_pairs) & 7) == 0,
            PRT_ERR_INVALID, "d_queries must be 16-byte and d_pairs 8-byte aligned");
  return PRT_OK;
}

void raise_frontier_hint(int64_t fcap) {
  int64_t seen = g_frontier_hint.load(std::memory_order_relaxed);
  while (seen < fcap && !g_frontier_hint.compare_exchange_weak(seen, fcap, std::memory_order_relaxed)) {
  }
}

// Runs the traversal.  pairs may be nullptr with cap 0 (count only).
int run_join(const prt_tree *t, const void *d_queries, int coord, int64_t nq, uint2 *d_pairs, int64_t cap,
             int64_t *h_count, cudaStream_t s, long long *d_counts = nullptr, int td_slots = 0) {
  if (h_count) *h_count = 0;
  int ra = check_join(t, d_queries, coord, nq, d_pairs, cap);
  if (ra) return ra;
  if (nq == 0) return PRT_OK;
  const TreeLevels &L = t->lv;
  const size_t bs = 4 * coord_size(t->coord);
  int64_t fcap = std::max<int64_t>(g_frontier_hint.load(std::memory_order_relaxed), 4 * nq);
  for (int attempt = 0; attempt < 8; attempt++) {
    unsigned long long *cnt = nullptr;
    uint2 *fr[2] = {nullptr, nullptr};
    int rc = dalloc(&cnt, PRT_MAX_LEVELS + 2, s);
    if (!rc && L.levels > 1) rc = dalloc(&fr[0], fcap, s);
    if (!rc && L.levels > 2) rc = dalloc(&fr[1], fcap, s);
    if (!rc) {
      cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(unsigned long long) * (PRT_MAX_LEVELS + 2), s);
      if (e == cudaSuccess && d_counts) e = cudaMemsetAsync(d_counts, 0, sizeof(long long) * 3 * nq, s);
      if (e != cudaSuccess) rc = cuda_status(e, "memset");
    }
    // level L-1 (root node) down to 0
    int cur = -1;
    for (int l = L.levels - 1; l >= 0 && !rc; l--) {
      JoinLevel J;
      J.mbr = reinterpret_cast<const char *>(t->d_mbr) + L.offset[l] * bs;
      J.n_entries = L.count[l];
      J.in = cur < 0 ? nullptr : fr[cur];
      J.in_count = cur < 0 ? nullptr : &cnt[l + 1];
      J.in_cap = fcap;
      J.leaf = l == 0;
      int nxt = cur < 0 ? 0 : 1 - cur;
      J.out = J.leaf ? d_pairs : fr[nxt];
      J.out_count = J.leaf ? &cnt[PRT_MAX_LEVELS] : &cnt[l];
      J.out_cap = J.leaf ? cap : fcap;
      J.nq = nq;
      J.counts = d_counts;
      J.td_slots = td_slots;
      rc = dispatch_coord(t->coord, [&](auto tag) {
        using T = decltype(tag);
        return launch_expand<T>(J, d_queries, t->fanout, s);
      });
      cur = nxt;
    }
    if (!rc) {
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) rc = cuda_status(e, "join launch");
    }
    std::vector<unsigned long long> h(PRT_MAX_LEVELS + 2, 0);
    if (!rc) {
      cudaError_t e = cudaMemcpyAsync(h.data(), cnt, sizeof(unsigned long long) * (PRT_MAX_LEVELS + 2),
                                      cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) rc = cuda_status(e, "join");
    }
    dfree(cnt, s);
    dfree(fr[0], s);
    dfree(fr[1], s);
    if (rc) return rc;
    unsigned long long worst = 0;
    for (int l = 1; l < L.levels; l++) worst = std::max(worst, h[l]);
    if ((int64_t)worst > fcap) {
      fcap = (int64_t)(worst + worst / 4 + 1024);
      raise_frontier_hint(fcap);
      continue;
    }
    int64_t np = (int64_t)h[PRT_MAX_LEVELS];
    if (h_count) *h_count = np;
    if (np > cap && d_pairs) {
      set_error("join: %lld pairs exceed capacity %lld", (long long)np, (long long)cap);
      return PRT_ERR_CAPACITY;
    }
    return PRT_OK;
  }
  set_error("join: frontier kept overflowing");
  return PRT_ERR_CAPACITY;
}

__global__ void pair_key_kernel(const uint2 *__restrict__ p, int64_t n, uint64_t *__restrict__ k,
                                uint32_t *__restrict__ v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint2 x = p[i];
    k[i] = ((uint64_t)x.y << 32) | x.x;
    v[i] = x.x;
  }
}

__global__ void pair_unkey_kernel(const uint64_t *k0, const uint64_t *k1, const int *sel, int64_t n,
                                  uint2 *__restrict__ p) {
  const uint64_t *k = *sel ? k1 : k0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t x = k[i];
    p[i] = make_uint2((uint32_t)x, (uint32_t)(x >> 32));
  }
}

// ------------------------------------------------------------------ ordered traversal

// Bit 31 of a frontier item's node: the query contains the node's box, so it
// intersects every entry of it (entries are below 2^30).
constexpr uint32_t kContained = 0x80000000u;

// Containment implies intersection only for proper boxes (x1 <= x2, y1 <= y2,
// no NaN): an empty polygon's box, say, intersects nothing but lies inside
// its parent.  The build notes whether a tree has an improper record.
__device__ __forceinline__ bool all_proper(const unsigned *flags) { return (*flags & kTreeImproper) == 0; }

template <typename T>
__device__ __forceinline__ bool contains(const Box<T> &q, const Box<T> &b) {
  return q.x1 <= b.x1 && b.x2 <= q.x2 && q.y1 <= b.y1 && b.y2 <= q.y2;
}

// The frontier is cut into tiles of up to kTileItems items, smaller ones where
// that spreads a small frontier over every block (kTilesPerBlock each), and
// kSuperTiles tiles share a word of pair counts, so that a tile finds the hits
// before it from two short sums and no block waits for another (a look-back
// between the tiles of one launch cost 15-20 us a level in polls of the same
// few lines: the five levels of a 100k-window join took 211 us against 106).
constexpr int kTileItems = 1024;
constexpr int kTilesPerBlock = 2;
constexpr int kSuperTiles = 256;

struct OrderedLevel {
  const void *mbr;          // entries of node level l (Box<T>)
  int64_t n_entries;
  const uint2 *in;          // frontier (query, node | kContained); nullptr = (q, 0) for all queries
  const unsigned long long *in_count;
  int64_t in_cap;
  int64_t nq;
  uint32_t *masks, *conts;  // per item: entries hit; entries the query contains
  uint32_t *tile_count;     // hits per tile
  unsigned long long *super_count;  // and per kSuperTiles tiles (zeroed)
  uint2 *out;               // next frontier, or (entry, query) pairs at the leaf level
  unsigned long long *out_count;
  int64_t out_cap;
  int leaf;
  int64_t blocks;           // grid of the hits launch: the tiles' size goes by it
  const unsigned *flags;    // the tree's
};

struct Tiling {
  int64_t count, per_tile, tiles;
  int rounds;
};

template <int G>
__device__ __forceinline__ Tiling tiling(const OrderedLevel &J) {
  constexpr int kGroups = kJoinBlock / G;
  Tiling t;
  t.count = J.in ? (int64_t)min((unsigned long long)J.in_cap, *J.in_count) : J.nq;
  const int64_t wave = J.blocks * kTilesPerBlock * kGroups;
  t.rounds = (int)min(max((t.count + wave - 1) / wave, (int64_t)1), (int64_t)(kTileItems / kGroups));
  t.per_tile = (int64_t)t.rounds * kGroups;
  t.tiles = (t.count + t.per_tile - 1) / t.per_tile;
  return t;
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The hits of every item of a level: a group of G lanes per item, lane e for
// entry e, three rounds of loads in flight.
template <typename T, int G>
__global__ void __launch_bounds__(kJoinBlock) ordered_hits_kernel(OrderedLevel J, const Box<T> *__restrict__ queries,
                                                                  int fanout) {
  __shared__ uint32_t s_sum[2][kJoinBlock / 32];
  const Box<T> *mbr = reinterpret_cast<const Box<T> *>(J.mbr);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / G, e = lane % G;
  constexpr int kGroups = kJoinBlock / G, kWarpGroups = 32 / G;
  const uint32_t gsel = G == 32 ? 0xffffffffu : (1u << G) - 1u;
  const Tiling t = tiling<G>(J);
  const bool prune = !J.leaf && all_proper(J.flags);
  int par = 0;
  for (int64_t tile = blockIdx.x; tile < t.tiles; tile += gridDim.x, par ^= 1) {
    const int64_t first = tile * t.per_tile;
    const int items = (int)min(t.per_tile, t.count - first);
    uint32_t sum = 0;
    for (int r0 = 0; r0 < t.rounds; r0 += kJoinRounds) {
      uint2 it[kJoinRounds];
      bool live[kJoinRounds];
#pragma unroll
      for (int r = 0; r < kJoinRounds; r++) {
        const int i = (r0 + r) * kGroups + warp * kWarpGroups + sub;
        live[r] = i < items && r0 + r < t.rounds;
        it[r] = make_uint2(0u, 0u);
        if (live[r]) it[r] = J.in ? J.in[first + i] : make_uint2((uint32_t)(first + i), 0u);
      }
      bool hit[kJoinRounds], in[kJoinRounds];
#pragma unroll
      for (int r = 0; r < kJoinRounds; r++) {
        hit[r] = in[r] = false;
        if (live[r] && e < fanout) {
          if (it[r].y & kContained) {
            hit[r] = in[r] = (int64_t)(it[r].y & ~kContained) * fanout + e < J.n_entries;
          } else {
            const Box<T> qb = load_box(queries, it[r].x);
            const Box<T> eb = load_box(mbr, (int64_t)it[r].y * fanout + e);  // padded slots intersect nothing
            hit[r] = overlaps(eb, qb);
            in[r] = hit[r] && prune && contains(qb, eb);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < kJoinRounds; r++) {
        const int i = (r0 + r) * kGroups + warp * kWarpGroups + sub;
        const uint32_t hb = __ballot_sync(0xffffffffu, hit[r]) >> (sub * G) & gsel;
        const uint32_t cb = J.leaf ? 0u : __ballot_sync(0xffffffffu, in[r]) >> (sub * G) & gsel;
        if (live[r] && e == 0) {
          J.masks[first + i] = hb;
          if (!J.leaf) J.conts[first + i] = cb;
          sum += __popc(hb);
        }
      }
    }
    sum = warp_sum(sum);
    if (lane == 0) s_sum[par][warp] = sum;
    __syncthreads();  // the sums are double-buffered: one barrier a tile
    if (threadIdx.x == 0) {
      uint32_t total = 0;
      for (int w = 0; w < kJoinBlock / 32; w++) total += s_sum[par][w];
      J.tile_count[tile] = total;
      if (total) {
        atomicAdd(&J.super_count[tile / kSuperTiles], (unsigned long long)total);
        atomicAdd(J.out_count, (unsigned long long)total);
      }
    }
  }
}

// Writes a level's hits in item order, entry order within an item: the next
// frontier, or the pairs.
template <int G>
__global__ void __launch_bounds__(kJoinBlock) ordered_emit_kernel(OrderedLevel J, int fanout) {
  __shared__ uint32_t s_mask[kTileItems], s_cont[kTileItems], s_off[kTileItems];
  __shared__ uint2 s_item[kTileItems];
  __shared__ uint32_t s_warp[kJoinBlock / 32];
  __shared__ unsigned long long s_before[kJoinBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = threadIdx.x % G;
  constexpr int kGroups = kJoinBlock / G;
  const Tiling t = tiling<G>(J);
  for (int64_t tile = blockIdx.x; tile < t.tiles; tile += gridDim.x) {
    const int64_t first = tile * t.per_tile;
    const int items = (int)min(t.per_tile, t.count - first);
    // the hits of the tiles before this one
    unsigned long long before = 0;
    const int64_t super = tile / kSuperTiles;
    for (int64_t k = threadIdx.x; k < super; k += kJoinBlock) before += J.super_count[k];
    for (int64_t k = super * kSuperTiles + threadIdx.x; k < tile; k += kJoinBlock) before += J.tile_count[k];
    for (int o = 16; o; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) s_before[warp] = before;
    for (int i = threadIdx.x; i < items; i += kJoinBlock) {
      s_mask[i] = J.masks[first + i];
      s_cont[i] = J.leaf ? 0u : J.conts[first + i];
      s_item[i] = J.in ? J.in[first + i] : make_uint2((uint32_t)(first + i), 0u);
    }
    __syncthreads();
    unsigned long long base = 0;
    for (int w = 0; w < kJoinBlock / 32; w++) base += s_before[w];
    // the items' offsets in the tile: consecutive items per thread
    const int per = (items + kJoinBlock - 1) / kJoinBlock, mine = threadIdx.x * per;
    uint32_t sum = 0;
    for (int i = mine; i < min(mine + per, items); i++) sum += __popc(s_mask[i]);
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t at = incl - sum;
    for (int w = 0; w < warp; w++) at += s_warp[w];
    for (int i = mine; i < min(mine + per, items); i++) {
      s_off[i] = at;
      at += __popc(s_mask[i]);
    }
    __syncthreads();
    for (int i = threadIdx.x / G; i < items; i += kGroups) {
      const uint32_t m = s_mask[i];
      if (m >> e & 1u) {
        const unsigned long long to = base + s_off[i] + __popc(m & ((1u << e) - 1u));
        const uint2 it = s_item[i];
        const uint32_t entry = (it.y & ~kContained) * (uint32_t)fanout + (uint32_t)e;
        if ((int64_t)to < J.out_cap)
          J.out[to] = J.leaf ? make_uint2(entry, it.x)
                             : make_uint2(it.x, entry | ((s_cont[i] >> e & 1u) ? kContained : 0u));
      }
    }
    __syncthreads();
  }
}

template <typename T, int G>
int ordered_blocks() {
  static std::atomic<int> per_sm{0};
  int b = per_sm.load(std::memory_order_relaxed);
  if (b == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, ordered_hits_kernel<T, G>, kJoinBlock, 0) != cudaSuccess ||
        b < 1) {
      cudaGetLastError();
      b = 4;
    }
    per_sm.store(b, std::memory_order_relaxed);
  }
  return kSMs * b;
}

// f(tag, std::integral_constant<int, G>) for the group size of a fanout.
template <typename F>
int dispatch_group(int coord, int fanout, F &&f) {
  return dispatch_coord(coord, [&](auto tag) {
    if (fanout <= 2) return f(tag, std::integral_constant<int, 2>{});
    if (fanout <= 4) return f(tag, std::integral_constant<int, 4>{});
    if (fanout <= 8) return f(tag, std::integral_constant<int, 8>{});
    if (fanout <= 16) return f(tag, std::integral_constant<int, 16>{});
    return f(tag, std::integral_constant<int, 32>{});
  });
}

// An ordered join up to its pair count: the leaf frontier with its hit masks.
struct Ordered {
  void *scratch = nullptr;   // counters, super-tile and tile counts
  uint2 *fr[2] = {nullptr, nullptr};
  uint32_t *masks = nullptr, *conts = nullptr;
  OrderedLevel leaf;
  int64_t count = 0;
  int fanout = 0;
};

void ordered_free(Ordered &o, cudaStream_t s) {
  dfree(o.scratch, s);
  dfree(o.fr[0], s);
  dfree(o.fr[1], s);
  dfree(o.masks, s);
  dfree(o.conts, s);
  o.scratch = nullptr;
  o.fr[0] = o.fr[1] = nullptr;
  o.masks = o.conts = nullptr;
}

// Writes a level's hits.
int ordered_emit(const OrderedLevel &J, int fanout, cudaStream_t s) {
  const unsigned grid = (unsigned)std::min<int64_t>(J.blocks * kTilesPerBlock, (int64_t)kSMs * 8);
  return dispatch_group(PRT_COORD_F32, fanout, [&](auto, auto g) {
    PRT_PROF("join_emit", s);
    ordered_emit_kernel<decltype(g)::value><<<grid, kJoinBlock, 0, s>>>(J, fanout);
    return PRT_OK;
  });
}

// Runs an ordered join of nq >= 1 queries up to the pair count.
int run_ordered(const prt_tree *t, const void *d_queries, int64_t nq, Ordered &o, cudaStream_t s) {
  const TreeLevels &L = t->lv;
  const size_t bs = 4 * coord_size(t->coord);
  o.fanout = t->fanout;
  int64_t blocks = 1;
  int rc = dispatch_group(t->coord, t->fanout, [&](auto tag, auto g) {
    blocks = ordered_blocks<decltype(tag), decltype(g)::value>();
    return PRT_OK;
  });
  if (rc) return rc;
  int64_t fcap = std::max<int64_t>(g_frontier_hint.load(std::memory_order_relaxed), 4 * nq);
  for (int attempt = 0; attempt < 8; attempt++) {
    // per level: its hits (PRT_MAX_LEVELS + 2 counters in all), then its
    // super-tile counts; the tile counts of one level at a time
    const int64_t tiles = std::max<int64_t>(blocks * kTilesPerBlock, fcap / kTileItems) + 2;
    const int64_t supers = tiles / kSuperTiles + 1;
    const size_t zeroed = 8 * (size_t)(PRT_MAX_LEVELS + 2 + supers * L.levels);
    rc = dmalloc(&o.scratch, zeroed + 4 * (size_t)tiles, s);
    if (!rc && L.levels > 1) rc = dalloc(&o.fr[0], fcap, s);
    if (!rc && L.levels > 2) rc = dalloc(&o.fr[1], fcap, s);
    if (!rc) rc = dalloc(&o.masks, L.levels > 1 ? fcap : nq, s);
    if (!rc && L.levels > 1) rc = dalloc(&o.conts, fcap, s);
    unsigned long long *cnt = static_cast<unsigned long long *>(o.scratch);
    unsigned long long *super = cnt + PRT_MAX_LEVELS + 2;
    if (!rc) {
      cudaError_t e = cudaMemsetAsync(o.scratch, 0, zeroed, s);
      if (e != cudaSuccess) rc = cuda_status(e, "memset");
    }
    int cur = -1;
    for (int l = L.levels - 1; l >= 0 && !rc; l--) {
      OrderedLevel J;
      memset(&J, 0, sizeof J);
      J.mbr = reinterpret_cast<const char *>(t->d_mbr) + L.offset[l] * bs;
      J.n_entries = L.count[l];
      J.in = cur < 0 ? nullptr : o.fr[cur];
      J.in_count = cur < 0 ? nullptr : &cnt[l + 1];
      J.in_cap = fcap;
      J.nq = nq;
      J.leaf = l == 0;
      const int nxt = cur < 0 ? 0 : 1 - cur;
      J.masks = o.masks;
      J.conts = o.conts;
      J.super_count = super + supers * l;
      J.tile_count = reinterpret_cast<uint32_t *>(super + supers * L.levels);
      J.out = J.leaf ? nullptr : o.fr[nxt];
      J.out_count = J.leaf ? &cnt[PRT_MAX_LEVELS] : &cnt[l];
      J.out_cap = fcap;
      J.blocks = blocks;
      J.flags = t->d_flags;
      rc = dispatch_group(t->coord, t->fanout, [&](auto tag, auto g) {
        using T = decltype(tag);
        PRT_PROF("expand", s);
        ordered_hits_kernel<T, decltype(g)::value><<<(unsigned)blocks, kJoinBlock, 0, s>>>(
            J, reinterpret_cast<const Box<T> *>(d_queries), t->fanout);
        return PRT_OK;
      });
      if (J.leaf) o.leaf = J;
      else if (!rc) rc = ordered_emit(J, t->fanout, s);
      cur = nxt;
    }
    unsigned long long h[PRT_MAX_LEVELS + 1];
    if (!rc) {
      cudaError_t e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(h, cnt, sizeof h, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) rc = cuda_status(e, "join");
    }
    unsigned long long worst = 0;
    for (int l = 1; l < L.levels && !rc; l++) worst = std::max(worst, h[l]);
    if (!rc && (int64_t)worst <= fcap) {
      o.count = (int64_t)h[PRT_MAX_LEVELS];
      return PRT_OK;
    }
    ordered_free(o, s);
    if (rc) return rc;
    fcap = (int64_t)(worst + worst / 4 + 1024);
    raise_frontier_hint(fcap);
  }
  set_error("join: frontier kept overflowing");
  return PRT_ERR_CAPACITY;
}

// ------------------------------------------------------------------ window counts

// A level as the walk needs it: entries are numbered over the whole tree
// (below 2^32), a node by its first entry.  The child of entry x of this level
// starts at x * fanout + child (mod 2^32).
struct CountsLevel {
  uint32_t child;
  uint32_t last;   // first entry of the level's last node
  uint32_t fill;   // and the entries it has
  uint32_t first;  // first entry of the level
};

struct CountsTree {
  const void *mbr;
  int levels;
  CountsLevel lv[PRT_MAX_LEVELS];
};

// A subtree left to a later launch: a node and its level, query q.
struct CountsItem {
  uint32_t q, node;
  int32_t level;
};

struct CountsQueue {
  const CountsItem *in;          // work of this launch (nullptr: the root for every query)
  const unsigned long long *n_in;
  CountsItem *out;               // work left over
  unsigned long long *out_count;
  int64_t out_cap;
  unsigned *ticket;              // batches taken beyond the warps' first ones
};

// Per-query counters (entries examined, sum of max(0, hits - 1) per visited
// node, leaf hits).  A warp walks the tree for one query: the nodes still to
// visit are on a stack in shared memory, 32 / G of them (G: lanes per node) are
// tested in one round, counts_rounds rounds' loads are in flight together, and
// the counters stay in registers: nothing is written but the result, where a
// breadth-first frontier costs 16 bytes and three atomics a node.  One node at a
// time where their entries might not fit the stack.  An entry the query
// contains is not visited: its subtree's counters follow from the level sizes.
// A query that is not done after kCountsSteps steps (a long thin window, a tree
// that cannot be pruned) leaves what is on its stack to the next launch, where
// every node is a work item of its own.
// Bound by instruction issue (0.77 per cycle and scheduler): some 110 instructions a
// step and 60 a query.  From kCountsBatched queries on a warp therefore takes several
// and tests them against the root a lane each: 1M windows of 1e-4..1e-2 on 10M boxes
// 2.32 -> 1.82 ms at F = 16 (breadth first 3.55), on 10k and 100k boxes 0.62 -> 0.49 and
// 0.82 -> 0.68 ms (breadth first 0.50 and 0.74).
// Without batches, 10M boxes: 1 and 3 rounds at F = 16 2.67 and 2.10 ms, 5
// blocks per SM 2.42; two walks per warp 2.71.  Nodes of 8 entries and fewer keep the
// warp too little to do per round (313k windows on 740k boxes, F = 8: 409 us against
// 325): they go breadth first (kCountsWideFanout).
constexpr int kCountsBlock = 256;
constexpr int kCountsSteps = 256;
constexpr int kCountsWideFanout = 9;  // fanouts from here on go depth first
// Calls of so many queries batch them, kCountsBatch at a time, a warp's first batch by
// its index and the next ones from a counter.  Batches dealt out in advance differ in
// what their walks cost and in how many a warp gets: 1M windows on 10M boxes 2.08 ms,
// 1.82 from the counter, 300k 0.79 and 0.68, 131k 0.45 and 0.41 (batches of 16 1.85,
// 0.73 and 0.46; of 4 1.82, 0.66 and 0.38, but 3 to 6% slower on 10k and 1M boxes, where
// a walk is short and the root's share in it large).
constexpr int64_t kCountsBatched = 1 << 17;
constexpr int kCountsBatch = 8;
// Queries that leave most warps idle (kCountsFew times as many could be resident)
// hand what is left of a walk on after kCountsFewSteps, to launches that are made at
// once, kCountsChain in all, as a wait for each would cost more than they do.  2M
// boxes, F = 16: 100 windows across the whole extent 139 -> 83 us (breadth first 80), 100
// of 0.1 by 0.1 where nothing can be pruned 359 -> 112 (128); 100 small windows, for
// which there is nothing left, 53 -> 58 (66).  Not on trees of under kCountsLong nodes,
// where walks are short.  With a look at what is left before the later launches small
// windows stay at 53, and long ones take 126 and 157.
constexpr int kCountsFew = 8, kCountsFewSteps = 24, kCountsChain = 3;
constexpr int64_t kCountsLong = 1024;

template <int G>
constexpr int counts_rounds() { return G == 32 ? 4 : G == 16 ? 2 : 1; }
template <int G>
constexpr int counts_pop() { return counts_rounds<G>() * (32 / G); }

// Stack entries of a warp: a step that takes `pop` nodes must leave room for a
// walk that takes one at a time (fanout - 1 more per level).
inline int counts_stack(int levels, int fanout, int pop) { return (2 * levels + pop) * (fanout - 1) + 1; }

// Shared memory of a block's warps with kBatch: a batch's queries, the root's
// entries that each hits and contains, and the root's entries.
template <typename T>
struct CountsBatch {
  Box<T> query[kCountsBlock / 32][kCountsBatch];
  uint2 hits[kCountsBlock / 32][kCountsBatch];
  Box<T> root[32];
};

// kBatch: a warp takes kCountsBatch queries at a time, a lane of it testing each against
// the root, and then walks for those that hit something there (trees of two
// levels and more, not for left-over work).
template <typename T, int G, bool kBatch>
__global__ void __launch_bounds__(kCountsBlock, sizeof(T) == 4 ? 4 : 3)
    counts_kernel(CountsTree t, const Box<T> *__restrict__ queries, int64_t nq, int max_steps, int fanout,
                  int td_slots, int stack_cap, const unsigned *__restrict__ flags, long long *__restrict__ counts, CountsQueue Q) {
  extern __shared__ __align__(32) unsigned char s_raw[];
  constexpr int kNodes = 32 / G, kRounds = counts_rounds<G>(), kPop = counts_pop<G>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / G, e = lane % G;
  const uint32_t gmask = (G == 32 ? 0xffffffffu : (1u << G) - 1u) << (lane - e);
  const uint32_t lt = lanemask_lt();
  const bool on = e < fanout;
  cudaGridDependencySynchronize();
  const int64_t work = !kBatch && Q.in ? (int64_t)min(*Q.n_in, (unsigned long long)Q.out_cap) : nq;
  if (work == 0) return;
  CountsBatch<T> &B = *reinterpret_cast<CountsBatch<T> *>(s_raw);
  CountsLevel *s_lv = reinterpret_cast<CountsLevel *>(s_raw + (kBatch ? sizeof(CountsBatch<T>) : 0));
  uint2 *stack = reinterpret_cast<uint2 *>(s_lv + t.levels) + warp * stack_cap;  // (node, level)
  const Box<T> *mbr = reinterpret_cast<const Box<T> *>(t.mbr) + e;
  for (int l = threadIdx.x; l < t.levels; l += kCountsBlock) s_lv[l] = t.lv[l];
  if (kBatch && threadIdx.x < fanout)
    B.root[threadIdx.x] = load_box(reinterpret_cast<const Box<T> *>(t.mbr), (int64_t)t.lv[t.levels - 1].first + threadIdx.x);
  __syncthreads();
  const bool prune = all_proper(flags);
  const int room = stack_cap - (t.levels + kPop) * (fanout - 1);  // most entries a kPop step may start from
  const uint32_t leaf_last = s_lv[0].last, leaf_lack = fanout - s_lv[0].fill;
  const uint32_t warps = gridDim.x * (kCountsBlock / 32);
  constexpr int step = kBatch ? kCountsBatch : 1;
  for (int64_t w = (int64_t)(blockIdx.x * (kCountsBlock / 32) + warp) * step; w < work;) {
    uint32_t next = 0;
    if (kBatch && lane == 0) next = atomicAdd(Q.ticket, 1u);
    uint32_t todo = 1u;  // queries of the batch to walk for
    CountsItem it{(uint32_t)w, s_lv[t.levels - 1].first, t.levels - 1};
    if constexpr (kBatch) {
      const uint32_t fill = s_lv[t.levels - 1].fill;
      uint32_t hits = 0, conts = 0;
      __syncwarp();
      if (lane < step && w + lane < nq) {
        const Box<T> q = load_box(queries, w + lane);
        for (uint32_t j = 0; j < fill; j++) {
          const Box<T> r = B.root[j];
          hits |= (overlaps(r, q) ? 1u : 0u) << j;
          conts |= (prune && contains(q, r) ? 1u : 0u) << j;
        }
        B.query[warp][lane] = q;
        B.hits[warp][lane] = make_uint2(hits, conts & hits);
        if (hits == 0) {
          long long *out = &counts[3 * (w + lane)];
          out[0] = td_slots ? fanout : fill;
          out[1] = out[2] = 0;
        }
      }
      todo = __ballot_sync(0xffffffffu, hits != 0);
      __syncwarp();
    } else if (Q.in) {
      it = Q.in[w];
    }
    for (; todo; todo &= todo - 1) {
      Box<T> qb;
      int sp, steps = 0;
      // the group's nodes, the same on its lanes: visited, entries that levels'
      // last nodes lack, sum of max(hits, 1), leaf hits
      uint32_t visits = 0, lack = 0, c1 = 0, c2 = 0;
      // this lane's contained subtrees: nodes, entries, leaf entries (a tree has
      // fewer than 2^32 entries)
      uint32_t d_nodes = 0, d_entries = 0, d_leaf = 0;
      // adds the subtree below an entry whose child starts at x, of level m
      auto add_subtree = [&](uint32_t x, uint32_t m) {
        uint32_t n = 1;  // its nodes of level m, [x, end)
        for (;; m--) {
          const CountsLevel M = s_lv[m];
          const uint32_t end = min(x + n * (uint32_t)fanout, M.last + M.fill);  // all n nodes are in the tree
          d_nodes += n;
          n = end - x;
          d_entries += n;
          if (m == 0) break;
          x = x * (uint32_t)fanout + M.child;
        }
        d_leaf += n;
      };
      if constexpr (kBatch) {
        const int j = __ffs(todo) - 1;
        it.q = (uint32_t)w + j;
        qb = B.query[warp][j];
        const uint2 h = B.hits[warp][j];
        const CountsLevel L = s_lv[t.levels - 1];
        if (g == 0) {
          visits = 1;
          c1 = __popc(h.x);
          lack = fanout - L.fill;
        }
        const uint32_t x = (L.first + e) * (uint32_t)fanout + L.child;
        const uint32_t pb = h.x & ~h.y;
        if (g == 0 && (pb >> e & 1u)) stack[__popc(pb & lt)] = make_uint2(x, t.levels - 2);
        if (g == 0 && (h.y >> e & 1u)) add_subtree(x, t.levels - 2);
        sp = __popc(pb);
      } else {
        qb = load_box(queries, it.q);
        __syncwarp();
        if (lane == 0) stack[0] = make_uint2(it.node, (uint32_t)it.level);
        sp = 1;
      }
      __syncwarp();
      while (sp > 0) {
        const int pop = sp <= room ? min(sp, kPop) : 1;
        uint2 nd[kRounds];
        Box<T> b[kRounds];
#pragma unroll
        for (int r = 0; r < kRounds; r++) {
          nd[r] = make_uint2(0u, 0xffffffffu);
          if (r * kNodes + g < pop) {
            nd[r] = stack[sp - 1 - r * kNodes - g];
            if (on) b[r] = load_box(mbr, nd[r].x);
          }
        }
        sp -= pop;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kRounds; r++) {
          if (r * kNodes >= pop) break;
          const bool live = nd[r].y != 0xffffffffu;
          const bool hit = live && on && overlaps(b[r], qb);
          const int k = __popc(__ballot_sync(0xffffffffu, hit) & gmask);
          const bool inner = live && nd[r].y != 0;
          if (live) {
            visits++;
            c1 += max(k, 1);
            if (!inner) {
              c2 += k;
              if (nd[r].x == leaf_last) lack += leaf_lack;
            }
          }
          if (__any_sync(0xffffffffu, inner)) {
            const bool in = hit && inner && prune && contains(qb, b[r]);
            const bool push = hit && inner && !in;
            const uint32_t pb = __ballot_sync(0xffffffffu, push);
            if (inner) {
              const CountsLevel L = s_lv[nd[r].y];
              if (nd[r].x == L.last) lack += fanout - L.fill;
              const uint32_t x = (nd[r].x + e) * (uint32_t)fanout + L.child;  // the entry's child
              if (push) stack[sp + __popc(pb & lt)] = make_uint2(x, nd[r].y - 1u);
              if (in) add_subtree(x, nd[r].y - 1u);
            }
            sp += __popc(pb);
          }
        }
        __syncwarp();
        if (++steps >= (kBatch ? kCountsSteps : max_steps) && sp > 0) {
          // too long a walk: the rest of it to the next launch, if that has room
          unsigned long long at = 0;
          if (lane == 0) at = atomicAdd(Q.out_count, (unsigned long long)sp);
          at = __shfl_sync(0xffffffffu, at, 0);
          const int fits = (int)min((long long)sp, max(0ll, (long long)Q.out_cap - (long long)at));
          for (int k = lane; k < fits; k += 32) Q.out[at + k] = CountsItem{it.q, stack[sp - 1 - k].x, (int32_t)stack[sp - 1 - k].y};
          sp -= fits;
          steps = 0;
          __syncwarp();
        }
      }
      if (e != 0) visits = lack = c1 = c2 = 0;
      const uint32_t r0 = __reduce_add_sync(
          0xffffffffu, td_slots ? (visits + d_nodes) * (uint32_t)fanout : visits * (uint32_t)fanout - lack + d_entries);
      const uint32_t r1 = __reduce_add_sync(0xffffffffu, c1 - visits + (d_entries - d_nodes));
      const uint32_t r2 = __reduce_add_sync(0xffffffffu, c2 + d_leaf);
      if (lane < 3) {
        unsigned long long *out = reinterpret_cast<unsigned long long *>(&counts[3 * (int64_t)it.q + lane]);
        const unsigned long long v = lane == 0 ? r0 : lane == 1 ? r1 : r2;
        if (!kBatch && Q.in) atomicAdd(out, v);
        else *out = v;
      }
    }
    w = kBatch ? (int64_t)(warps + __shfl_sync(0xffffffffu, next, 0)) * step : w + warps;
  }
}

}  // namespace
}  // namespace prt

using namespace prt;

struct prt_join_state {
  prt::Ordered o;
  cudaStream_t stream = nullptr;
};

extern "C" {

int prt_join(const prt_tree *t, const void *d_queries, int coord_type, int64_t nq, prt_pair *d_pairs, int64_t cap,
             int64_t *h_count, void *stream) {
  return run_join(t, d_queries, coord_type, nq, reinterpret_cast<uint2 *>(d_pairs), d_pairs ? cap : 0, h_count,
                  reinterpret_cast<cudaStream_t>(stream));
}

int prt_join_sorted(const prt_tree *t, const void *d_queries, int coord_type, int64_t nq, prt_pair *d_pairs,
                    int64_t cap, int64_t *h_count, void *stream) {
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  int64_t np = 0;
  int rc = run_join(t, d_queries, coord_type, nq, reinterpret_cast<uint2 *>(d_pairs), d_pairs ? cap : 0, &np,
                    s);
  if (h_count) *h_count = np;
  if (rc || np == 0) return rc;
  PRT_CHECK(np < (1ll << 30), PRT_ERR_INVALID, "join_sorted: %lld pairs (sort limit 2^30)", (long long)np);
  unsigned char *scr = nullptr;
  rc = dmalloc(reinterpret_cast<void **>(&scr), 64 + np * (8 + 8 + 4 + 4), s);
  if (rc) return rc;
  unsigned *err = reinterpret_cast<unsigned *>(scr);
  int *sel = reinterpret_cast<int *>(scr + 8);
  uint64_t *k0 = reinterpret_cast<uint64_t *>(scr + 64), *k1 = k0 + np;
  uint32_t *v0 = reinterpret_cast<uint32_t *>(k1 + np), *v1 = v0 + np;
  cudaMemsetAsync(err, 0, 8, s);
  int g = grid_for(np, 256, 16);
  {
    PRT_PROF("pair_key", s);
    pair_key_kernel<<<g, 256, 0, s>>>(reinterpret_cast<const uint2 *>(d_pairs), np, k0, v0);
  }
  rc = radix_sort_pairs<uint64_t>(k0, v0, k1, v1, np, 64, sel, err, s);
  if (!rc) {
    PRT_PROF("pair_unkey", s);
    pair_unkey_kernel<<<g, 256, 0, s>>>(k0, k1, sel, np, reinterpret_cast<uint2 *>(d_pairs));
  }
  unsigned herr = 0;
  if (!rc) {
    cudaError_t e = cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) rc = cuda_status(e, "join_sorted");
  }
  dfree(scr, s);
  if (!rc && (herr & kErrTimeout)) {
    set_error("join_sorted: sort look-back timed out");
    rc = PRT_ERR_TIMEOUT;
  }
  return rc;
}

int prt_join_begin(const prt_tree *t, const void *d_queries, int coord_type, int64_t nq, prt_join_state **out,
                   int64_t *h_count, void *stream) {
  PRT_CHECK(out && h_count, PRT_ERR_INVALID, "NULL argument");
  *out = nullptr;
  *h_count = 0;
  int rc = check_join(t, d_queries, coord_type, nq, nullptr, 0);
  if (rc) return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  prt_join_state *st = new (std::nothrow) prt_join_state();
  PRT_CHECK(st != nullptr, PRT_ERR_NOMEM, "no host memory");
  st->stream = s;
  if (nq > 0) rc = run_ordered(t, d_queries, nq, st->o, s);
  if (rc) {
    delete st;
    return rc;
  }
  *h_count = st->o.count;
  *out = st;
  return PRT_OK;
}

int prt_join_finish(prt_join_state *st, prt_pair *d_pairs) {
  PRT_CHECK(st != nullptr, PRT_ERR_INVALID, "state is NULL");
  int rc = PRT_OK;
  if (d_pairs && st->o.count > 0) {
    if ((reinterpret_cast<uintptr_t>(d_pairs) & 7) != 0) {
      set_error("d_pairs must be 8-byte aligned");
      rc = PRT_ERR_INVALID;
    } else {
      prt::OrderedLevel J = st->o.leaf;
      J.out = reinterpret_cast<uint2 *>(d_pairs);
      J.out_cap = st->o.count;
      rc = ordered_emit(J, st->o.fanout, st->stream);
      cudaError_t e = cudaGetLastError();
      if (!rc && e != cudaSuccess) rc = cuda_status(e, "join pairs");
    }
  }
  ordered_free(st->o, st->stream);
  delete st;
  return rc;
}

int prt_query_counts(const prt_tree *t, const void *d_queries, int coord_type, int64_t nq, int td_slots,
                     int64_t *d_counts, void *stream) {
  PRT_CHECK(d_counts != nullptr, PRT_ERR_INVALID, "d_counts is NULL");
  int rc = check_join(t, d_queries, coord_type, nq, nullptr, 0);
  if (rc || nq == 0) return rc;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (t->fanout < kCountsWideFanout) {
    int64_t np = 0;
    return run_join(t, d_queries, coord_type, nq, nullptr, 0, &np, s, reinterpret_cast<long long *>(d_counts), td_slots);
  }
  CountsTree c;
  c.mbr = t->d_mbr;
  c.levels = t->lv.levels;
  int64_t all_nodes = 0;
  for (int l = 0; l < c.levels; l++) {
    const int64_t nodes = t->lv.padded[l] / t->fanout, first = t->lv.offset[l];
    all_nodes += nodes;
    c.lv[l].first = (uint32_t)first;
    c.lv[l].last = (uint32_t)(first + (nodes - 1) * t->fanout);
    c.lv[l].fill = (uint32_t)(t->lv.count[l] - (nodes - 1) * t->fanout);
    c.lv[l].child = l > 0 ? (uint32_t)(t->lv.offset[l - 1] - first * t->fanout) : 0u;
  }
  // two work queues for the walks that are left over, and the counts of what the
  // launches leave
  constexpr int64_t kQueue = 1 << 20;
  CountsItem *queue = nullptr;
  unsigned long long *left = nullptr;
  rc = dalloc(&queue, 2 * kQueue, s);
  if (!rc) rc = dalloc(&left, kCountsChain + 2, s);
  int chain = 1, round = 0;  // launches until the host looks
  unsigned long long n_left = 1;
  while (!rc && n_left > 0) {
    cudaError_t e = cudaMemsetAsync(left, 0, 8 * (kCountsChain + 1), s);
    int last = 0;
    for (int i = 0; i < chain && e == cudaSuccess && !rc; i++, round++) {
      CountsQueue Q;
      Q.in = round ? queue + ((round - 1) & 1) * kQueue : nullptr;
      Q.n_in = i ? &left[i - 1] : left + kCountsChain + 1;
      Q.ticket = reinterpret_cast<unsigned *>(left + kCountsChain);
      Q.out = queue + (round & 1) * kQueue;
      Q.out_count = &left[last = i];
      Q.out_cap = kQueue;
      rc = dispatch_group(t->coord, t->fanout, [&](auto tag, auto g) {
        using T = decltype(tag);
        constexpr int G = std::max(decltype(g)::value, 16), kWarps = kCountsBlock / 32;  // smaller ones went above
        const int cap = counts_stack(c.levels, t->fanout, counts_pop<G>());
        auto launch = [&](auto kernel, size_t smem, int batch) {
          smem += sizeof(CountsLevel) * c.levels + sizeof(uint2) * (size_t)kWarps * cap;
          int b = 0;
          PRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel, kCountsBlock, smem));
          const int64_t resident = (int64_t)kSMs * std::max(b, 1);
          if (!Q.in && nq * kCountsFew < resident * kWarps && all_nodes >= kCountsLong) chain = kCountsChain;
          const int64_t per = (int64_t)kWarps * batch;
          const int64_t blocks = Q.in ? resident : std::min<int64_t>((nq + per - 1) / per, resident);
          const int steps = i + 1 < chain ? kCountsFewSteps : kCountsSteps;
          PRT_PROF("counts", s);
          PRT_CUDA(launch_dependent(kernel, (int)blocks, kCountsBlock, smem, s, c,
                                    reinterpret_cast<const Box<T> *>(d_queries), nq, steps, t->fanout, td_slots,
                                    cap, t->d_flags, reinterpret_cast<long long *>(d_counts), Q));
          return PRT_OK;
        };
        if (!Q.in && c.levels > 1 && nq >= kCountsBatched) return launch(counts_kernel<T, G, true>, sizeof(CountsBatch<T>), kCountsBatch);
        return launch(counts_kernel<T, G, false>, 0, 1);
      });
    }
    if (!rc && e == cudaSuccess) e = cudaMemcpyAsync(&n_left, &left[last], 8, cudaMemcpyDeviceToHost, s);
    if (!rc && e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (!rc && e != cudaSuccess) rc = cuda_status(e, "query counts");
    if (rc || n_left == 0) break;
    chain = 1;
    // the count of what this round left, where the next one's first launch reads it
    e = cudaMemcpyAsync(left + kCountsChain + 1, &left[last], 8, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) rc = cuda_status(e, "query counts");
  }
  dfree(queue, s);
  dfree(left, s);
  return rc;
}

int prt_tree_sibling_overlaps(const prt_tree *t, int64_t *h_count, void *stream) {
  PRT_CHECK(t && h_count, PRT_ERR_INVALID, "NULL argument");
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  *h_count = 0;
  unsigned long long *d = nullptr;
  int rc = dalloc(&d, 1, s);
  if (rc) return rc;
  cudaError_t e = cudaMemsetAsync(d, 0, 8, s);
  const size_t bs = 4 * coord_size(t->coord);
  for (int l = 0; l < t->lv.levels && e == cudaSuccess; l++) {
    const int64_t nodes = (t->lv.count[l] + t->fanout - 1) / t->fanout;
    const void *lv = reinterpret_cast<const char *>(t->d_mbr) + t->lv.offset[l] * bs;
    rc = dispatch_coord(t->coord, [&](auto tag) {
      using T = decltype(tag);
      PRT_PROF("sibling", s);
      sibling_kernel<T><<<grid_for(nodes * 32, 256, 8), 256, 0, s>>>(reinterpret_cast<const Box<T> *>(lv),
                                                                     t->lv.count[l], t->fanout, d);
      return PRT_OK;
    });
    e = cudaGetLastError();
  }
  unsigned long long h = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, 8, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  dfree(d, s);
  if (e != cudaSuccess) return cuda_status(e, "sibling overlaps");
  *h_count = (int64_t)h;
  return rc;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free join.
//
// prt_join takes its frontier buffers and level counters from the
// stream-ordered allocator.  Some callers may not allocate device memory at
// the moment they join: a host process that hands the whole device budget to
// its own pool and treats any other allocation as a failure, or an embedding
// that forbids the library from calling cudaMalloc / cudaMallocAsync at all.
// prt_join_noalloc runs the same breadth-first traversal with its scratch in
// the file-scope array below instead: the caller passes the queries and the
// pair buffer, and the library allocates nothing.  The call still waits for
// its stream once, at the end, to read the level and pair counts.
//
// The array is reserved on every GPU that loads the library, for the life of
// the process.  Its device address is looked up once per device
// (cudaGetSymbolAddress, with that device current) on the first call made
// there and kept for the process, so make that first call before any stream
// capture, and do not call again on a device after cudaDeviceReset (the kept
// address would be stale).  All calls on a device share the one array and its
// contents stay from one call to the next (every call clears the counters):
// calls that can overlap on the GPU (different streams, or host threads) race
// on it and must be serialised by the caller.
#include <mutex>

namespace prt {
namespace {

// Frontier items per buffer: two (query, node) buffers of 4 Mi items each
// (64 MiB) plus the level counters.
constexpr int64_t kNoAllocFrontier = 1ll << 22;
constexpr size_t kNoAllocCounterBytes = 512;  // 64 x uint64, room for PRT_MAX_LEVELS + 2
constexpr size_t kNoAllocBytes = kNoAllocCounterBytes + 2 * sizeof(uint2) * (size_t)kNoAllocFrontier;

static __device__ __align__(256) unsigned char g_join_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
unsigned char *g_noalloc_addr[256] = {nullptr};  // per device, set on first use

int noalloc_scratch(unsigned char **out) {
  int dev = 0;
  PRT_CUDA(cudaGetDevice(&dev));
  PRT_CHECK(dev >= 0 && dev < 256, PRT_ERR_INVALID, "device %d out of range", dev);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_join_scratch);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(join scratch)");
    g_noalloc_addr[dev] = reinterpret_cast<unsigned char *>(p);
  }
  *out = g_noalloc_addr[dev];
  return PRT_OK;
}

}  // namespace
}  // namespace prt

extern "C" {

int prt_join_noalloc(const prt_tree *t, const void *d_queries, int coord_type, int64_t nq, prt_pair *d_pairs,
                     int64_t cap, int64_t *h_count, void *stream) {
  using namespace prt;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  PRT_CHECK(t != nullptr, PRT_ERR_INVALID, "tree is NULL");
  PRT_CHECK(coord_type == t->coord, PRT_ERR_INVALID, "query coordinate type %d differs from the tree's %d",
            coord_type, t->coord);
  PRT_CHECK(nq >= 0 && nq < (1ll << 31), PRT_ERR_INVALID, "nq=%lld", (long long)nq);
  PRT_CHECK(cap >= 0 && (cap == 0 || d_pairs != nullptr), PRT_ERR_INVALID, "pair buffer");
  PRT_CHECK((reinterpret_cast<uintptr_t>(d_queries) & 15) == 0 && (reinterpret_cast<uintptr_t>(d_pairs) & 7) == 0,
            PRT_ERR_INVALID, "d_queries must be 16-byte and d_pairs 8-byte aligned");
  PRT_CHECK(t->lv.levels + 2 <= (int)(kNoAllocCounterBytes / 8), PRT_ERR_INVALID, "tree too deep");
  if (h_count) *h_count = 0;
  if (nq == 0) return PRT_OK;
  unsigned char *scr = nullptr;
  int rc = noalloc_scratch(&scr);
  if (rc) return rc;
  unsigned long long *cnt = reinterpret_cast<unsigned long long *>(scr);
  uint2 *fr[2] = {reinterpret_cast<uint2 *>(scr + kNoAllocCounterBytes),
                  reinterpret_cast<uint2 *>(scr + kNoAllocCounterBytes) + kNoAllocFrontier};
  // the counters must start at zero; the frontier buffers are written before read
  PRT_CUDA(cudaMemsetAsync(cnt, 0, kNoAllocCounterBytes, s));
  const TreeLevels &L = t->lv;
  const size_t bs = 4 * coord_size(t->coord);
  const int leaf_slot = PRT_MAX_LEVELS;  // counter of emitted pairs
  int cur = -1;
  for (int l = L.levels - 1; l >= 0 && !rc; l--) {
    JoinLevel J;
    J.mbr = reinterpret_cast<const char *>(t->d_mbr) + L.offset[l] * bs;
    J.n_entries = L.count[l];
    J.in = cur < 0 ? nullptr : fr[cur];
    J.in_count = cur < 0 ? nullptr : &cnt[l + 1];
    J.in_cap = kNoAllocFrontier;
    J.leaf = l == 0;
    int nxt = cur < 0 ? 0 : 1 - cur;
    J.out = J.leaf ? reinterpret_cast<uint2 *>(d_pairs) : fr[nxt];
    J.out_count = J.leaf ? &cnt[leaf_slot] : &cnt[l];
    J.out_cap = J.leaf ? cap : kNoAllocFrontier;
    J.nq = nq;
    J.counts = nullptr;
    J.td_slots = 0;
    rc = dispatch_coord(t->coord, [&](auto tag) {
      using T = decltype(tag);
      return launch_expand<T>(J, d_queries, t->fanout, s);
    });
    cur = nxt;
  }
  if (rc) return rc;
  PRT_CUDA(cudaGetLastError());
  unsigned long long h[PRT_MAX_LEVELS + 2];
  PRT_CUDA(cudaMemcpyAsync(h, cnt, sizeof h, cudaMemcpyDeviceToHost, s));
  PRT_CUDA(cudaStreamSynchronize(s));
  for (int l = 1; l < L.levels; l++) {
    if ((int64_t)h[l] > kNoAllocFrontier) {
      set_error("prt_join_noalloc: a frontier of %llu (query, node) items exceeds the fixed scratch of %lld items; "
                "use prt_join or fewer queries per call",
                h[l], (long long)kNoAllocFrontier);
      return PRT_ERR_CAPACITY;
    }
  }
  const int64_t np = (int64_t)h[leaf_slot];
  if (h_count) *h_count = np;
  if (np > cap) {
    set_error("prt_join_noalloc: %lld pairs exceed capacity %lld", (long long)np, (long long)cap);
    return PRT_ERR_CAPACITY;
  }
  return PRT_OK;
}

}  // extern "C"

namespace prt {

// Breadth-first join into caller-owned buffers, nothing synchronised: the
// capture-safe form used by the graph pipeline (prt_pipeline_*).
int join_enqueue(const prt_tree *t, const void *d_queries, int64_t nq, uint2 *d_pairs, int64_t cap, uint2 *fr0,
                 uint2 *fr1, int64_t fcap, unsigned long long *cnt, cudaStream_t s) {
  PRT_CHECK(t != nullptr && nq >= 0, PRT_ERR_INVALID, "join_enqueue arguments");
  if (nq == 0) return PRT_OK;
  const TreeLevels &L = t->lv;
  const size_t bs = 4 * coord_size(t->coord);
  uint2 *fr[2] = {fr0, fr1};
  int cur = -1;
  int rc = PRT_OK;
  for (int l = L.levels - 1; l >= 0 && !rc; l--) {
    JoinLevel J;
    J.mbr = reinterpret_cast<const char *>(t->d_mbr) + L.offset[l] * bs;
    J.n_entries = L.count[l];
    J.in = cur < 0 ? nullptr : fr[cur];
    J.in_count = cur < 0 ? nullptr : &cnt[l + 1];
    J.in_cap = fcap;
    J.leaf = l == 0;
    int nxt = cur < 0 ? 0 : 1 - cur;
    J.out = J.leaf ? d_pairs : fr[nxt];
    J.out_count = J.leaf ? &cnt[PRT_MAX_LEVELS] : &cnt[l];
    J.out_cap = J.leaf ? cap : fcap;
    J.nq = nq;
    J.counts = nullptr;
    J.td_slots = 0;
    rc = dispatch_coord(t->coord, [&](auto tag) {
      using T = decltype(tag);
      return launch_expand<T>(J, d_queries, t->fanout, s);
    });
    cur = nxt;
  }
  if (rc) return rc;
  PRT_CUDA(cudaGetLastError());
  return PRT_OK;
}

}  // namespace prt
