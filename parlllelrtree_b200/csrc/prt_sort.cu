// Onesweep LSD radix sort of (key, uint32 value) pairs.
//
// One upsweep kernel histograms every 8-bit digit of every key at once; a
// tiny plan kernel scans the histograms and marks passes whose digit differs
// between keys (the others are skipped without a host round trip, so the whole
// sort can be captured in a CUDA graph).  Each remaining pass is ONE kernel:
// a CTA takes the next tile in launch order (atomic ticket), ranks its keys
// with a warp-level multisplit (lanes with the same digit found by one ballot
// per digit bit), learns its global digit offsets by decoupled look-back over the
// preceding tiles (bounded spin, an error flag instead of a hang), stages the tile
// in shared memory in digit order and writes it out in coalesced runs.  Stable:
// ranks follow the original order within a warp, then warp order, then tile order.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "prt_internal.cuh"

namespace prt {
namespace {

constexpr int kRadix = 256;
constexpr int kSortBlock = 256;
constexpr int kSortWarps = kSortBlock / 32;
#ifndef PRT_SORT_MIN_BLOCKS
// resident blocks per SM the 32-bit-key pass is compiled for: 4 (64
// registers, a 56-byte spill) against 3 (80 registers): 0.0872 ->
// 0.0830-0.0840 ms per 10M-key pass, measured with the look-back batch below.
// The 64-bit-key pass stays at 3: its 58 KB tile fits no more per SM.
#define PRT_SORT_MIN_BLOCKS 4
#endif
// Keys per thread of a tile, by the number of keys that are sorted.  A pass
// over few keys takes as long as one tile's chain of rankings and the look-back
// over the tiles: 16, 8, 4 keys per thread take 7.7, 5.7, 3.6 us for 4k
// keys, 9.6, 7.7, 7.7 for 150k, 9.8, 9.1, 9.8 for 300k and 11.7, 11.9, 14.0 for
// 600k (32-bit keys); at 10M, where the pass is bound by instruction issue, 84,
// 107 and 163 us.
inline int sort_items(int64_t n) { return n <= 200000 ? 4 : n <= 600000 ? 8 : 16; }
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1;

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename KeyT>
__global__ void __launch_bounds__(256) hist_kernel(const KeyT *__restrict__ keys, int64_t n, int passes,
                                                   uint32_t *__restrict__ ghist) {
  extern __shared__ uint32_t sh[];  // passes * 256
  for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (sizeof(KeyT) == 4 && (reinterpret_cast<uintptr_t>(keys) & 15) == 0) {
    // four keys per 16-byte load
    const uint4 *k4 = reinterpret_cast<const uint4 *>(keys);
    for (int64_t i = i0; i < n / 4; i += stride) {
      const uint4 q = k4[i];
      const KeyT kk[4] = {(KeyT)q.x, (KeyT)q.y, (KeyT)q.z, (KeyT)q.w};
#pragma unroll
      for (int j = 0; j < 4; j++)
        for (int p = 0; p < passes; p++) atomicAdd(&sh[p * kRadix + (int)((kk[j] >> (8 * p)) & 0xFF)], 1u);
    }
    i0 += (n / 4) * 4;
  }
  for (int64_t i = i0; i < n; i += stride) {
    KeyT k = keys[i];
    for (int p = 0; p < passes; p++) atomicAdd(&sh[p * kRadix + (int)((k >> (8 * p)) & 0xFF)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x)
    if (sh[i]) atomicAdd(&ghist[i], sh[i]);
}

// Exclusive scan of one value per thread over a block of kRadix threads.
__device__ __forceinline__ uint32_t scan_digits(uint32_t v, uint32_t *s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t off = 0;
#pragma unroll
  for (int w = 0; w < kRadix / 32; w++) off += w < warp ? s_warp[w] : 0u;
  return off + incl - v;
}

// Digit offsets of pass p and whether it moves anything (a pass whose digit is
// the same for all keys of every run is skipped), one block per run and pass:
// goff[(p * runs + run) * 256 + d] = the run's first position + the run's
// exclusive digit scan; bit p of *active (cleared before) is set when some run
// has more than one digit in pass p.  hist holds hist_passes x 256 counts per run.
__global__ void __launch_bounds__(kRadix) plan_kernel(const uint32_t *__restrict__ hist, int64_t n, int64_t run_len,
                                                      int64_t runs, int hist_passes, int passes,
                                                      uint32_t *__restrict__ goff, unsigned *active) {
  __shared__ uint32_t s_warp[kRadix / 32];
  const int64_t run = blockIdx.x / passes;
  const int p = (int)(blockIdx.x % passes);
  const int64_t start = run * run_len;
  const int64_t len = min(run_len, n - start);
  const uint32_t c = hist[(run * hist_passes + p) * kRadix + threadIdx.x];
  if (__syncthreads_or((int64_t)c != len && c != 0) && threadIdx.x == 0) atomicOr(active, 1u << p);
  goff[((int64_t)p * runs + run) * kRadix + threadIdx.x] = (uint32_t)start + scan_digits(c, s_warp);
}

template <typename KeyT, int kItems>
struct PassSmem {
  KeyT keys[kSortBlock * kItems];
  uint32_t vals[kSortBlock * kItems];
  uint32_t warp_hist[kSortWarps][kRadix];
  uint32_t digit_start[kRadix];  // tile-local exclusive start of each digit
  uint32_t global_start[kRadix];
  uint32_t scan_tmp[kSortWarps];
  int tile;
};

#ifndef PRT_SORT_LOOKBATCH
#define PRT_SORT_LOOKBATCH 4  // 2, 4, 8, 16 measured: 4 best at 4 blocks per SM
#endif
#ifndef PRT_SORT_BACKOFF_NS
#define PRT_SORT_BACKOFF_NS 0  // pause between look-back polls that found nothing new
#endif
constexpr int kLookBatch = PRT_SORT_LOOKBATCH;  // predecessor statuses read per look-back step

template <typename KeyT, int kItems, bool kRuns>
__global__ void __launch_bounds__(kSortBlock, sizeof(KeyT) == 4 ? PRT_SORT_MIN_BLOCKS : 3)
    onesweep_pass(KeyT *keys0, uint32_t *vals0, KeyT *keys1, uint32_t *vals1, int64_t n, int shift,
                  int passes, const unsigned *__restrict__ active, int *d_sel,
                  const uint32_t *__restrict__ goff, uint32_t *status, unsigned *tile_ticket, unsigned *err, WaitLimit wl, int64_t run_len,
                  int tiles_per_run) {
  constexpr int kTile = kSortBlock * kItems;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PassSmem<KeyT, kItems> &S = *reinterpret_cast<PassSmem<KeyT, kItems> *>(smem_raw);
  // the buffers swap at every active pass
  const int pass = shift / 8;
  const unsigned act = *active;
  const bool moves = act >> pass & 1u;
  const bool from = __popc(act & ((1u << pass) - 1u)) & 1;
  if (pass == passes - 1 && blockIdx.x == 0 && threadIdx.x == 0) *d_sel = from != moves;
  if (!moves) return;
  const KeyT *src_k = from ? keys1 : keys0;
  const uint32_t *src_v = from ? vals1 : vals0;
  KeyT *dst_k = from ? keys0 : keys1;
  uint32_t *dst_v = from ? vals0 : vals1;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int d = tid;  // kSortBlock == kRadix: thread d owns digit d
  if (tid == 0) S.tile = (int)atomicAdd(tile_ticket, 1u);
  for (int i = tid; i < kSortWarps * kRadix; i += kSortBlock) (&S.warp_hist[0][0])[i] = 0;
  __syncthreads();
  const int tile = S.tile;
  // the tile's run (kRuns: runs of run_len keys are sorted independently), its
  // first tile, its place and its digit offsets
  int first = 0;
  int64_t base = (int64_t)tile * kTile, end = n;
  if constexpr (kRuns) {
    const int run = tile / tiles_per_run;
    first = run * tiles_per_run;
    base = run * run_len + (int64_t)(tile - first) * kTile;
    end = min(n, (run + 1) * run_len);
    goff += run * kRadix;
  }
  const int valid = (int)min((int64_t)kTile, end - base);
  const int wb = warp * 32 * kItems;  // this warp's first item in the tile

  KeyT k[kItems];
  uint32_t v[kItems];
  if (valid == kTile) {
    const KeyT *pk = src_k + base + wb + lane;
    const uint32_t *pv = src_v + base + wb + lane;
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      k[i] = pk[i * 32];
      v[i] = pv[i * 32];
    }
  } else {
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      const int li = wb + i * 32 + lane;
      k[i] = 0;
      v[i] = 0;
      if (li < valid) {
        k[i] = src_k[base + li];
        v[i] = src_v[base + li];
      }
    }
  }
  // 1. stable ranks and the warps' digit histograms in one sweep: lanes with the
  //    same digit are found by one ballot per digit bit; all of them read the
  //    warp's counter and the lowest bumps it.  Items are ranked in index order
  //    (item slot i of lane l is tile position wb + 32 i + l), which makes the pass
  //    stable.  Full tiles, all but one per run, go without the checks per item
  //    (10M 32-bit keys: 86 -> 82 us a pass).
  const uint32_t lt = lanemask_lt();
  uint32_t *wh = S.warp_hist[warp];
  uint32_t dr[kItems];  // rank << 9 | digit (256 + lane: no item)
  if (valid == kTile) {
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      const uint32_t dg = (uint32_t)((k[i] >> shift) & 0xFF);
      uint32_t peers = 0xffffffffu;
#pragma unroll
      for (int b = 0; b < 8; b++) {
        const uint32_t m = __ballot_sync(0xffffffffu, (dg >> b) & 1u);
        peers &= ((dg >> b) & 1u) ? m : ~m;
      }
      const uint32_t before = __popc(peers & lt);
      const uint32_t cnt = wh[dg];
      __syncwarp();
      if (before == 0) wh[dg] = cnt + __popc(peers);
      dr[i] = ((cnt + before) << 9) | dg;
      __syncwarp();  // this item's counter updates before the next item's reads
    }
  } else {
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      const int li = wb + i * 32 + lane;
      const bool ok = li < valid;
      const uint32_t dg = ok ? (uint32_t)((k[i] >> shift) & 0xFF) : 256u + lane;
      uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
      for (int b = 0; b < 8; b++) {
        const uint32_t m = __ballot_sync(0xffffffffu, (dg >> b) & 1u);
        peers &= ((dg >> b) & 1u) ? m : ~m;
      }
      if (!ok) peers = 1u << lane;
      const int leader = __ffs(peers) - 1;
      uint32_t cnt = 0;
      if (lane == leader && ok) {
        cnt = wh[dg];
        wh[dg] = cnt + __popc(peers);
      }
      cnt = __shfl_sync(0xffffffffu, cnt, leader);
      dr[i] = ((cnt + __popc(peers & lt)) << 9) | dg;
      __syncwarp();  // this item's counter updates before the next item's reads
    }
  }
  __syncthreads();
  // 2. digit d: exclusive prefix over the warps and the tile's count, which
  //    is published at once for the later tiles' look-back
  uint32_t total = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    const uint32_t c = S.warp_hist[w][d];
    S.warp_hist[w][d] = total;
    total += c;
  }
  uint32_t *st = status + (int64_t)tile * kRadix + d;
  if (tile == first) atomicExch(st, kFlagPrefix | ((goff[d] + total) & kCountMask));
  else atomicExch(st, kFlagAgg | (total & kCountMask));
  // tile-local exclusive scan over digits: shuffle scan per warp of 32
  // digits, then the 8 warp totals
  uint32_t incl = total;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) S.scan_tmp[warp] = incl;
  __syncthreads();
  uint32_t woff = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) woff += w < warp ? S.scan_tmp[w] : 0u;
  S.digit_start[d] = woff + incl - total;
  __syncthreads();
  // 3. stage the tile in digit order before the look-back: the items leave
  //    the registers, which the look-back's batches then use
  if (valid == kTile) {
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      const uint32_t dg = dr[i] & 255u;
      const uint32_t pos = S.digit_start[dg] + wh[dg] + (dr[i] >> 9);
      S.keys[pos] = k[i];
      S.vals[pos] = v[i];
    }
  } else {
#pragma unroll
    for (int i = 0; i < kItems; i++) {
      const uint32_t dg = dr[i] & 511u;
      if (dg < 256u) {
        const uint32_t pos = S.digit_start[dg] + wh[dg] + (dr[i] >> 9);
        S.keys[pos] = k[i];
        S.vals[pos] = v[i];
      }
    }
  }

  // 4. decoupled look-back for digit d, kLookBatch predecessor statuses per
  //    round trip; every wait is bounded
  uint32_t excl = goff[d];
  if (tile > first) {  // the run's first tile publishes a prefix: the look-back stops there
    uint32_t acc = 0;
    int t = tile - 1;
    int spins = 0;
    bool timed_out = false;
    for (;;) {
      uint32_t sv[kLookBatch];
#pragma unroll
      for (int j = 0; j < kLookBatch; j++) {
        uint32_t sj = 2u << 30;  // before tile 0: an empty prefix (never reached)
        if (t - j >= 0) sj = *reinterpret_cast<volatile uint32_t *>(status + (int64_t)(t - j) * kRadix + d);
        sv[j] = wl.blind ? 0u : sj;
      }
      int used = 0;
      bool done = false;
#pragma unroll
      for (int j = 0; j < kLookBatch; j++) {
        if (done || used < j) continue;  // stop at the first prefix or unpublished status
        const uint32_t f = sv[j] & ~kCountMask;
        if (f == 0u) continue;           // not yet published: retry from here
        acc += sv[j] & kCountMask;
        used = j + 1;
        if (f == kFlagPrefix) done = true;
      }
      if (done) break;
      t -= used;
      if (used == 0) {
        if (++spins > wl.polls) {
          timed_out = true;
          break;
        }
        if (PRT_SORT_BACKOFF_NS > 0) __nanosleep(PRT_SORT_BACKOFF_NS);
      }
    }
    if (timed_out) atomicOr(err, kErrTimeout);
    excl = acc;
    atomicExch(st, kFlagPrefix | ((excl + total) & kCountMask));
  }
  // staged position i of digit dd goes to global_start[dd] + i - digit_start[dd]
  S.global_start[d] = excl - S.digit_start[d];
  __syncthreads();

  // 5. write the staged tile out in coalesced runs per digit (a look-back
  //    that timed out leaves the offsets wrong: the bound keeps every write
  //    inside the buffers, and the caller reports the timeout)
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = tid + j * kSortBlock;
    if (i < valid) {
      const KeyT kk = S.keys[i];
      const uint32_t dst = S.global_start[(int)((kk >> shift) & 0xFF)] + (uint32_t)i;
      if (dst < (uint32_t)n) {  // n < 2^30
        dst_k[dst] = kk;
        dst_v[dst] = S.vals[i];
      }
    }
  }
}

// The passes of one sort, with kItems keys per thread.
template <typename KeyT, int kItems, bool kRuns>
cudaError_t launch_passes(KeyT *keys0, uint32_t *vals0, KeyT *keys1, uint32_t *vals1, int64_t n, int64_t run_len,
                          int tpr, int64_t tiles, int64_t runs, int passes, const unsigned *active, int *d_sel, const uint32_t *goff,
                          uint32_t *status, unsigned *tick, unsigned *err, cudaStream_t s) {
  const size_t smem = sizeof(PassSmem<KeyT, kItems>);
  // the shared-memory opt-in is set once per device (not a stream operation,
  // but kept out of graph captures after the first call)
  static bool attr_done[256] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  cudaError_t e = cudaSuccess;
  if (dev < 0 || dev >= 256 || !attr_done[dev]) {
    e = cudaFuncSetAttribute(onesweep_pass<KeyT, kItems, kRuns>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && dev >= 0 && dev < 256) attr_done[dev] = true;
  }
  const WaitLimit wl = wait_limit();
  for (int p = 0; p < passes && e == cudaSuccess; p++) {
    PRT_PROF("onesweep_pass", s);
    onesweep_pass<KeyT, kItems, kRuns><<<(unsigned)tiles, kSortBlock, smem, s>>>(
        keys0, vals0, keys1, vals1, n, 8 * p, passes, active, d_sel, goff + (size_t)p * runs * kRadix,
        status + (size_t)p * tiles * kRadix, tick + p, err, wl, run_len, tpr);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  return e;
}

// Sorts n keys in runs of run_len; d_hist (nullptr: counted here, one run
// only) holds hist_passes digit histograms per run.
template <typename KeyT>
int sort_impl(KeyT *keys0, uint32_t *vals0, KeyT *keys1, uint32_t *vals1, int64_t n, int64_t run_len, int key_bits,
              int *d_sel, unsigned *d_err, cudaStream_t s, const uint32_t *d_hist, int hist_passes) {
  PRT_CHECK(n >= 0 && n < (int64_t)kCountMask, PRT_ERR_INVALID, "radix sort: n=%lld out of range",
            (long long)n);
  const int passes = std::max(1, (key_bits + 7) / 8);
  PRT_CHECK(passes <= (int)sizeof(KeyT), PRT_ERR_INVALID, "radix sort: %d key bits", key_bits);
  if (n == 0) {
    PRT_CUDA(cudaMemsetAsync(d_sel, 0, sizeof(int), s));
    return PRT_OK;
  }
  PRT_CHECK(run_len >= 1, PRT_ERR_INVALID, "radix sort: run length %lld", (long long)run_len);
  const int64_t runs = (n + run_len - 1) / run_len;
  // smaller tiles where the last tile of every run would be mostly empty
  int items = sort_items(n);
  auto tile_of = [](int k) { return (int64_t)kSortBlock * k; };
  while (items > 4 && (run_len + tile_of(items) - 1) / tile_of(items) * tile_of(items) > run_len + run_len / 8) items /= 2;
  const int tpr = (int)((run_len + tile_of(items) - 1) / tile_of(items));
  const int64_t tiles = (runs - 1) * tpr + (n - (runs - 1) * run_len + tile_of(items) - 1) / tile_of(items);
  // scratch: active passes, tickets, histograms and status (cleared), offsets
  const size_t head = 128;
  const size_t hist_b = d_hist ? 0 : sizeof(uint32_t) * (size_t)passes * kRadix;
  const size_t stat_b = sizeof(uint32_t) * (size_t)tiles * kRadix * passes;
  const size_t goff_b = sizeof(uint32_t) * (size_t)runs * passes * kRadix;
  unsigned char *scratch = nullptr;
  int rc = dmalloc(reinterpret_cast<void **>(&scratch), head + hist_b + stat_b + goff_b, s);
  if (rc) return rc;
  unsigned *active = reinterpret_cast<unsigned *>(scratch);
  unsigned *tick = reinterpret_cast<unsigned *>(scratch + 64);
  uint32_t *ghist = reinterpret_cast<uint32_t *>(scratch + head);
  uint32_t *status = reinterpret_cast<uint32_t *>(scratch + head + hist_b);
  uint32_t *goff = reinterpret_cast<uint32_t *>(scratch + head + hist_b + stat_b);
  cudaError_t e = cudaMemsetAsync(scratch, 0, head + hist_b + stat_b, s);
  if (e == cudaSuccess) {
    if (!d_hist) {
      PRT_PROF("hist", s);
      hist_kernel<KeyT><<<grid_for(n, 256, 4), 256, sizeof(uint32_t) * passes * kRadix, s>>>(keys0, n, passes, ghist);
      d_hist = ghist;
      hist_passes = passes;
    }
    {
      PRT_PROF("plan", s);
      plan_kernel<<<(unsigned)(runs * passes), kRadix, 0, s>>>(d_hist, n, run_len, runs, hist_passes, passes, goff,
                                                               active);
    }
    auto go = [&](auto k) {
      constexpr int kItems = decltype(k)::value;
      auto launch = runs > 1 ? launch_passes<KeyT, kItems, true> : launch_passes<KeyT, kItems, false>;
      return launch(keys0, vals0, keys1, vals1, n, run_len, tpr, tiles, runs, passes, active, d_sel, goff, status,
                    tick, d_err, s);
    };
    e = items == 4   ? go(std::integral_constant<int, 4>{})
        : items == 8 ? go(std::integral_constant<int, 8>{})
                     : go(std::integral_constant<int, 16>{});
  }
  dfree(scratch, s);
  if (e != cudaSuccess) return cuda_status(e, "radix sort");
  return PRT_OK;
}

}  // namespace

template <typename KeyT>
int radix_sort_runs(KeyT *keys0, uint32_t *vals0, KeyT *keys1, uint32_t *vals1, int64_t n, int64_t run_len,
                    int key_bits, int *d_sel, unsigned *d_err, cudaStream_t s, const uint32_t *d_hist) {
  return sort_impl<KeyT>(keys0, vals0, keys1, vals1, n, run_len, key_bits, d_sel, d_err, s, d_hist,
                         (int)sizeof(KeyT));
}

template <typename KeyT>
int radix_sort_pairs(KeyT *keys0, uint32_t *vals0, KeyT *keys1, uint32_t *vals1, int64_t n, int key_bits,
                     int *d_sel, unsigned *d_err, cudaStream_t s, const uint32_t *d_hist) {
  return sort_impl<KeyT>(keys0, vals0, keys1, vals1, n, n, key_bits, d_sel, d_err, s, d_hist,
                         std::max(1, (key_bits + 7) / 8));
}

namespace {
std::atomic<int> g_wait_polls{kSpinLimit};
std::atomic<int> g_wait_blind{0};
}  // namespace

WaitLimit wait_limit() { return WaitLimit{g_wait_polls.load(), g_wait_blind.load()}; }

template int radix_sort_runs<uint32_t>(uint32_t *, uint32_t *, uint32_t *, uint32_t *, int64_t, int64_t, int,
                                       int *, unsigned *, cudaStream_t, const uint32_t *);
template int radix_sort_runs<uint64_t>(uint64_t *, uint32_t *, uint64_t *, uint32_t *, int64_t, int64_t, int,
                                       int *, unsigned *, cudaStream_t, const uint32_t *);
template int radix_sort_pairs<uint32_t>(uint32_t *, uint32_t *, uint32_t *, uint32_t *, int64_t, int, int *,
                                        unsigned *, cudaStream_t, const uint32_t *);
template int radix_sort_pairs<uint64_t>(uint64_t *, uint32_t *, uint64_t *, uint32_t *, int64_t, int, int *,
                                        unsigned *, cudaStream_t, const uint32_t *);

}  // namespace prt

extern "C" int prt_debug_wait_limit(int polls, int never_published) {
  using namespace prt;
  g_wait_polls.store(polls > 0 ? polls : kSpinLimit);
  g_wait_blind.store(never_published ? 1 : 0);
  return PRT_OK;
}
