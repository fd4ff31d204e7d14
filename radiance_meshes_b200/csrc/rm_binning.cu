// Stages 2-4 on the GPU: per-tile tet lists ordered by (depth bits, tet id).
//
// The reference emits one 64-bit key per (tile, tet) pair, sorts all N pairs
// with a 7-pass LSD radix sort and then searches the sorted keys for tile
// boundaries (slang/tile_shader.slang:49-125, sort_by_keys/sort_by_keys.cu:9-53,
// tile_shader_slang.py:36-69).  The sort depth is a per-tet quantity, so the
// same order is produced here with far less traffic:
//
//   1. rank the T tets by (depth bits, tet id) with a 4-pass LSD radix sort of
//      32-bit keys (T elements, not N);
//   2. tile populations come from a 2-D difference array (4 atomics per tet,
//      written by the projection kernel) and two prefix passes; an exclusive
//      scan turns them into tile_ranges directly;
//   3. pairs of a tet and a region of 8 x 4 tiles, generated in rank order, go
//      through a stable counting sort on the region id alone (12 bits at 1080p,
//      against the reference's 49-bit keys), and the regions' segments are expanded
//      to tile lists; stability keeps every list in rank order, so nothing is
//      sorted per tile.
//
// Ascending rank inside a tile is ascending (depth bits, tet id), which is what
// the reference's stable sort produces because it emits pairs in tet order.

#include "rm_common.cuh"

namespace rm {

// ---------------------------------------------------------------------------
// Regions: blocks of kRegW x kRegH tiles, one tile per lane of a warp.
// ---------------------------------------------------------------------------
constexpr int kRegShiftX = 3, kRegShiftY = 2;
constexpr int kRegW = 1 << kRegShiftX, kRegH = 1 << kRegShiftY;  // 8 x 4 = 32 tiles

// number of regions a tile rectangle (x0, y0, x1, y1), max exclusive, touches; 0 for an empty one
__device__ __forceinline__ uint32_t regions_touched(int4 rc) {
  if (rc.z <= rc.x || rc.w <= rc.y) return 0u;
  return (uint32_t)((((rc.z - 1) >> kRegShiftX) - (rc.x >> kRegShiftX) + 1) *
                    (((rc.w - 1) >> kRegShiftY) - (rc.y >> kRegShiftY) + 1));
}

// number of valid items: n, or the device-side count if one is given (the visible tets, known only on the device)
__device__ __forceinline__ int64_t valid_items(int64_t n, const uint32_t* n_dev) {
  return n_dev ? min(n, (int64_t)*n_dev) : n;
}

// Counters of one call, zeroed with the tile-coverage arrays before the projection.
struct BinCounters {
  uint32_t n_visible, status, n_deferred;  // written by the projection
  uint32_t ticket[4];                      // next block of each pass of the rank sort
  uint32_t rank_ticket;                    // and of the scan in rank order
  unsigned long long n_keys;   // sum of the tile populations
};

// ---------------------------------------------------------------------------
// Device-wide scan of uint32: block sums, then every block adds up the sums before its own and scans its items.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) >= o) v += n;
  }
  return v;
}

// exclusive scan across the block of one value per thread; returns exclusive prefix, total in *total
template <int THREADS>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total, uint32_t* smem /* THREADS/32 + 1 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = warp_inclusive_scan(v);
  if (lane == 31) smem[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < THREADS / 32 ? smem[lane] : 0;
    uint32_t winc = warp_inclusive_scan(w);
    if (lane < THREADS / 32) smem[lane] = winc - w;
    if (lane == THREADS / 32 - 1) smem[THREADS / 32] = winc;
  }
  __syncthreads();
  uint32_t r = inc - v + smem[warp];
  *total = smem[THREADS / 32];
  __syncthreads();
  return r;
}

// sum of the block sums before this block's, and, if `total` is given, of all n of them (else n is this block's index)
__device__ __forceinline__ uint32_t sums_before(const uint32_t* bsum, uint32_t n, unsigned long long* total) {
  __shared__ unsigned long long before[kScanThreads / 32], all[kScanThreads / 32];
  unsigned long long b = 0, t = 0;
  for (uint32_t i = threadIdx.x; i < n; i += kScanThreads) {
    const uint32_t v = bsum[i];
    if (i < blockIdx.x) b += v;
    t += v;
  }
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    b += __shfl_xor_sync(0xffffffffu, b, o);
    t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  if ((threadIdx.x & 31) == 0) {
    before[threadIdx.x >> 5] = b;
    all[threadIdx.x >> 5] = t;
  }
  __syncthreads();
  b = t = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    b += before[w];
    t += all[w];
  }
  if (total) *total = t;
  return (uint32_t)b;
}

// blocked arrangement: thread t owns items [t*kScanItems, (t+1)*kScanItems) of its block
__device__ __forceinline__ void load_blocked(const uint32_t* in, int64_t base, int64_t n, uint32_t (&v)[kScanItems]) {
  if (base + kScanItems <= n) {
#pragma unroll
    for (int k = 0; k < kScanItems; k += 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(in + base + k);
      v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0u;
  }
}

// ---------------------------------------------------------------------------
// Tile populations from the 2-D difference array, and the tile ranges from those.
// diff is (gh+1) x (gw+1), in `copies` partial arrays one behind the other; their sum is
// left in the first.  After a prefix along x and along y, entry (y,x) is the number of tet
// rectangles covering tile (y,x).  Four steps of little work that depend on nothing but the
// projection: each rides along with one launch of the rank sort, in the first blocks of its
// grid (as launches of their own they took 20 us at 128 x 128 pixels, 54 us at 4K).
// ---------------------------------------------------------------------------
struct TileJob {
  int step;  // 0..3
  int blocks;
  int32_t* diff;
  int copies, gh, gw;
  uint32_t *counts, *bsum, *tile_start;
  int2* ranges;
  BinCounters* counters;
};
constexpr int kJobThreads = 256;

__device__ __forceinline__ int32_t warp_prefix_step(int32_t v, int32_t& carry) {
  v = (int32_t)warp_inclusive_scan((uint32_t)v) + carry;
  carry = __shfl_sync(0xffffffffu, v, 31);
  return v;
}

__device__ __noinline__ void run_tile_job(const TileJob& j) {
  const int lane = threadIdx.x & 31, warp = blockIdx.x * (kJobThreads / 32) + (threadIdx.x >> 5);
  const int64_t G = (int64_t)j.gh * j.gw;
  if (j.step == 0) {  // prefix along x, a warp per row
    if (warp > j.gh) return;
    int32_t* r = j.diff + (int64_t)warp * (j.gw + 1);
    int32_t carry = 0;
    for (int base = 0; base <= j.gw; base += 32) {
      const int x = base + lane;
      int32_t v = 0;
      if (x <= j.gw)
        for (int k = 0; k < j.copies; ++k) v += r[x + (int64_t)k * (j.gh + 1) * (j.gw + 1)];
      v = warp_prefix_step(v, carry);
      if (x <= j.gw) r[x] = v;
    }
  } else if (j.step == 1) {  // prefix along y, a warp per column
    if (warp >= j.gw) return;
    int32_t carry = 0;
    for (int base = 0; base < j.gh; base += 32) {
      const int y = base + lane;
      const int32_t v = warp_prefix_step(y < j.gh ? j.diff[(int64_t)y * (j.gw + 1) + warp] : 0, carry);
      if (y < j.gh) j.counts[(int64_t)y * j.gw + warp] = (uint32_t)v;
    }
  } else {
    __shared__ uint32_t sm[kScanThreads / 32 + 1];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems], s = 0, total;
    load_blocked(j.counts, base, G, v);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) s += v[k];
    uint32_t ex = block_exclusive_scan<kScanThreads>(s, &total, sm);
    if (j.step == 2) {  // block sums of the populations
      if (threadIdx.x == 0) j.bsum[blockIdx.x] = total;
      return;
    }
    // tile_start[g] = exclusive scan of the populations; tile_ranges[g] = (start, start+count), or (0,0) for an empty tile
    // (compute_tile_ranges leaves untouched tiles at their zero fill); the sum of the populations to the counters
    const bool last = blockIdx.x == j.blocks - 1;
    unsigned long long all;
    ex += sums_before(j.bsum, last ? j.blocks : blockIdx.x, last ? &all : nullptr);
    if (last && threadIdx.x == 0) j.counters->n_keys = all;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < G) {
        j.tile_start[base + k] = ex;
        j.ranges[base + k] = v[k] ? make_int2((int)ex, (int)(ex + v[k])) : make_int2(0, 0);
      }
      ex += v[k];
    }
  }
}

// ---------------------------------------------------------------------------
// Rank sort: LSD radix sort of (uint32 key, uint32 tet) pairs, 8 bits per pass, stable.  The digit histograms of all
// four passes are taken in one launch; a pass is one launch, in which a block learns where its runs start from the
// blocks before it (decoupled look-back: Merrill and Garland, "Single-pass parallel prefix scan with decoupled
// look-back", 2016).  Blocks number themselves with a ticket, so those a block waits for are running already.  The
// first pass drops the culled tets (key 0xFFFFFFFF), the others run over the visible ones.
// 16 bytes per tet and pass; bound by the issue of the ballot ranking and the latency of a block's phases (issue slots 41 %,
// alu pipe 48 %, DRAM 7 %).  Histogram, row scan and scatter launches for each pass, over all tets: 248 us for 6.7M tets,
// 1.2 ms for 36M; this, with the tile populations on the way, 224 us and 0.88 ms.
// ---------------------------------------------------------------------------
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
static_assert(kSortThreads == kJobThreads && kSortThreads == kScanThreads, "the tile jobs ride in the sort's blocks");
// Keys per thread.  A mesh that 16 would cut into a few blocks gets 4: the ranking rounds of a warp follow one another,
// and 13k tets in four blocks took 8 us a pass where 13 blocks take 5.  Not beyond 64 blocks: they all run at once, and
// the look-back walks over those that are not done.
constexpr int sort_items(int64_t n) { return n <= 64 * 4 * kSortThreads ? 4 : 16; }
constexpr uint32_t kCulledKey = 0xFFFFFFFFu;
// Look-back words: 0 not there yet; n + 1 a block's own run of n; kRunEnd | n all runs up to and with the block's.
// No wait decides a result: from a word on that is not there after kMaxPolls polls, a block counts what is missing
// itself, from the other blocks' items, which nothing writes while the kernel runs (finish_look_back).
constexpr uint32_t kRunEnd = 1u << 31;
#ifdef RM_BOUNDS_CHECK
constexpr int kMaxPolls = 0;  // the checked build waits for no word, and never sees those of every other block (look_word)
static __device__ unsigned g_recounted;
#else
constexpr int kMaxPolls = 1 << 14;  // about 10 ms per word
#endif
enum Recounted { kRecountRankPass = 1, kRecountRankRects = 2, kRecountRegionPass = 4, kRecountFineLists = 8 };
__device__ __forceinline__ void note_recount(Recounted which) {
#ifdef RM_BOUNDS_CHECK
  atomicOr(&g_recounted, (unsigned)which);
#else
  (void)which;
#endif
}

__global__ void __launch_bounds__(kSortThreads)
k_digit_hist(const uint32_t* keys, int64_t n, uint32_t* __restrict__ hist /* [4][kRadix], zeroed */, TileJob job) {
  after_previous();
  constexpr int kItems = 8, kTile = kItems * kSortThreads;
  if ((int)blockIdx.x < job.blocks) return run_tile_job(job);
  const int64_t block = blockIdx.x - job.blocks, blocks = gridDim.x - job.blocks;
  __shared__ uint32_t h[2][4 * kRadix];  // two copies: half the warps each, against queues on the crowded high digits
  for (int i = threadIdx.x; i < 2 * 4 * kRadix; i += kSortThreads) (&h[0][0])[i] = 0;
  __syncthreads();
  uint32_t* mine = h[(threadIdx.x >> 5) & 1];
  for (int64_t base = block * kTile; base < n; base += blocks * kTile) {
    uint32_t key[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const int64_t i = base + k * kSortThreads + threadIdx.x;
      key[k] = i < n ? keys[i] : kCulledKey;
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      if (key[k] == kCulledKey) continue;
#pragma unroll
      for (int pass = 0; pass < 4; ++pass) atomicAdd(&mine[pass * kRadix + ((key[k] >> (8 * pass)) & 255u)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * kRadix; i += kSortThreads) {
    const uint32_t v = h[0][i] + h[1][i];
    if (v) atomicAdd(hist + i, v);
  }
}

__device__ __forceinline__ uint32_t load_relaxed(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ void store_relaxed(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v));
}

__device__ __forceinline__ uint32_t look_word(const uint32_t* p, uint32_t block) {
#ifdef RM_BOUNDS_CHECK
  if (block & 1u) return 0u;
#else
  (void)block;
#endif
  return load_relaxed(p);
}

// Sum of what the `blocks` blocks before `word` hold, on top of `before`, without waiting; count(b): what block b holds.
template <typename F>
__device__ __forceinline__ uint32_t finish_look_back(uint32_t before, const uint32_t* word, uint32_t blocks, int stride, F count) {
#pragma unroll 1
  while (blocks) {
    --blocks;
    word -= stride;
    uint32_t v = look_word(word, blocks);
    if (v == 0u) v = count(blocks) + 1u;
    if (v & kRunEnd) return before + (v ^ kRunEnd);
    before += v - 1u;
  }
  return before;
}

// Sum of what the `blocks` blocks before `word` hold, the nearest first, `stride` words apart.  AHEAD words are asked for
// at a time: blocks that run together all walk over each other's runs, one round trip to L2 per word otherwise.  Two are
// enough for the rank sort (36M tets: 975, 881, 881 us with 1, 2, 8), whose blocks hold many words each, eight are better
// for the list build (two passes 1180 -> 1012 us, lists 1681 -> 1554 us).  finish(before, word, blocks), where a wait runs
// out, is a call that ends the walk: with the counting inside the loop the rank sort of 36M tets took 1065 us, not 881.
template <uint32_t AHEAD, typename F>
__device__ __forceinline__ uint32_t look_back(const uint32_t* word, uint32_t blocks, int stride, F finish) {
  uint32_t before = 0;
  for (;;) {
    uint32_t v[AHEAD];
#pragma unroll
    for (uint32_t k = 0; k < AHEAD; ++k) v[k] = k < blocks ? look_word(word - (int64_t)(k + 1) * stride, blocks - 1u - k) : kRunEnd;
#pragma unroll
    for (uint32_t k = 0; k < AHEAD; ++k) {
      if (v[k] == 0u) {
        for (int polls = 0; v[k] == 0u && polls < kMaxPolls; ++polls) v[k] = load_relaxed(word - (int64_t)(k + 1) * stride);
        if (v[k] == 0u) return finish(before, word - (int64_t)k * stride, blocks - k);
      }
      if (v[k] & kRunEnd) return before + (v[k] ^ kRunEnd);
      before += v[k] - 1u;
    }
    word -= (int64_t)AHEAD * stride;
    blocks -= AHEAD;
  }
}

// The same for one word per block, by a whole warp, 32 words at a time.
template <typename F>
__device__ __forceinline__ uint32_t warp_look_back(const uint32_t* word, uint32_t blocks, F finish) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t before = 0;
  for (;;) {
    uint32_t v = lane < blocks ? look_word(word - lane - 1, blocks - 1u - lane) : kRunEnd;
    for (int polls = 0; __any_sync(0xffffffffu, v == 0u); ++polls) {
      if (polls == kMaxPolls) return finish(before, word, blocks);
      if (v == 0u) v = load_relaxed(word - lane - 1);
    }
    const uint32_t ends = __ballot_sync(0xffffffffu, (v & kRunEnd) != 0u);
    const uint32_t stop = ends ? (uint32_t)__ffs(ends) - 1u : 32u;
    before += __reduce_add_sync(0xffffffffu, lane < stop ? v - 1u : (lane == stop ? v ^ kRunEnd : 0u));
    if (ends) return before;
    word -= 32;
    blocks -= 32;
  }
}

// Thread d (of 256) places the runs of digit d.  In: cnt[w][d], how many items of the digit warp w of this block holds,
// and the digit's total over all blocks.  Out: cnt[w][d] the offset of the warp's items inside the block's run, lstart[d]
// where the run starts in the block's reordered buffer, dbase[d] what to add to a position there for its global one.
// Returns the number of items of the block.  finish: see look_back.
template <uint32_t AHEAD, typename F>
__device__ __forceinline__ uint32_t place_runs(bool live, uint32_t digit_total, uint32_t tile, uint32_t* __restrict__ look,
                                               int bins, uint32_t* cnt, uint32_t* dbase, uint32_t* lstart, uint32_t* sm,
                                               F finish) {
  const uint32_t d = threadIdx.x;
  uint32_t run = 0;
#pragma unroll
  for (int w = 0; w < kSortWarps; ++w) {
    const uint32_t c = cnt[w * kRadix + d];
    cnt[w * kRadix + d] = run;
    run += c;
  }
  uint32_t* word = look + (int64_t)tile * bins + d;
  if (live) store_relaxed(word, tile == 0 ? kRunEnd | run : run + 1u);
  uint32_t n_block, unused, before = 0;
  const uint32_t ls = block_exclusive_scan<kSortThreads>(run, &n_block, sm);
  const uint32_t digit_base = block_exclusive_scan<kSortThreads>(digit_total, &unused, sm);
  if (live && tile > 0) {
    before = look_back<AHEAD>(word, tile, bins, finish);
    store_relaxed(word, kRunEnd | (before + run));
  }
  lstart[d] = ls;
  dbase[d] = digit_base + before - ls;
  return n_block;
}

// finish_look_back of a pass of the rank sort whose blocks hold `tile` keys; a thread per digit.
__device__ __noinline__ uint32_t count_digits_before(uint32_t before, const uint32_t* word, uint32_t blocks, const uint32_t* keys,
                                                     int tile, int shift) {
  note_recount(kRecountRankPass);
  return finish_look_back(before, word, blocks, kRadix, [&](uint32_t b) {
    uint32_t n = 0;
#pragma unroll 1
    for (int i = 0; i < tile; ++i) {
      const uint32_t key = keys[(int64_t)b * tile + i];
      n += key != kCulledKey && ((key >> shift) & (kRadix - 1)) == threadIdx.x;
    }
    return n;
  });
}

// One stable pass.  The block's pairs are first reordered by digit in shared memory, so that the global stores of one
// digit's run are contiguous.  FIRST: the tet of item i is i.
template <bool FIRST, int kSortItems>
__global__ void __launch_bounds__(kSortThreads, 3)
k_rank_pass(const uint32_t* keys_in, const uint32_t* vals_in, int64_t T, BinCounters* counters, int pass,
            const uint32_t* hist, uint32_t* __restrict__ look /* [blocks][kRadix], zeroed */,
            uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, TileJob job) {
  after_previous();
  constexpr int kSortTile = kSortThreads * kSortItems;
  constexpr int kWarpSpan = 32 * kSortItems;  // consecutive keys owned by one warp
  if ((int)blockIdx.x < job.blocks) return run_tile_job(job);
  __shared__ uint2 sbuf[kSortTile];
  __shared__ uint32_t cnt[kSortWarps * kRadix];  // per-warp digit counts -> offsets
  __shared__ uint32_t dbase[kRadix];
  __shared__ uint32_t lstart[kRadix];
  __shared__ uint32_t sm[kSortThreads / 32 + 1];
  __shared__ uint32_t s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, shift = pass * kRadixBits;
  const int64_t n_out = valid_items(T, &counters->n_visible), n = FIRST ? T : n_out;
  if (threadIdx.x == 0) s_tile = atomicAdd(&counters->ticket[pass], 1u);
  for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortThreads) cnt[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const int64_t bbase = (int64_t)tile * kSortTile;
  if (bbase >= n) return;
  // warp w owns keys [bbase + w*kWarpSpan, +kWarpSpan) in index order (stability)
  const int64_t wbase = bbase + (int64_t)warp * kWarpSpan;
  uint32_t* wc = cnt + warp * kRadix;
  uint32_t key[kSortItems], val[kSortItems], rnk[kSortItems];
  // loads first (in flight together); the warp barriers of the ranking rounds would
  // otherwise serialise them
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    const int64_t i = wbase + k * 32 + lane;
    key[k] = i < n ? keys_in[i] : kCulledKey;  // no visible tet has that key
    val[k] = FIRST ? (uint32_t)i : (i < n ? vals_in[i] : 0u);
  }
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    const bool valid = key[k] != kCulledKey;
    const uint32_t d = (key[k] >> shift) & (kRadix - 1);
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < kRadixBits; ++b) {
      const bool bit = (d >> b) & 1u;
      const uint32_t m = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? m : ~m;
    }
    const uint32_t before = __popc(peers & ((1u << lane) - 1u));
    uint32_t prev = 0;
    if (valid) prev = wc[d];
    __syncwarp();
    if (valid && before == 0) wc[d] = prev + __popc(peers);
    __syncwarp();
    rnk[k] = prev + before;
  }
  __syncthreads();
  const uint32_t n_block = place_runs<2>(
      true, hist[threadIdx.x], tile, look, kRadix, cnt, dbase, lstart, sm,
      [&](uint32_t before, const uint32_t* word, uint32_t blocks) {
        return count_digits_before(before, word, blocks, keys_in, kSortTile, shift);
      });
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kSortItems; ++k) {
    if (key[k] != kCulledKey) {
      const uint32_t q = (key[k] >> shift) & (kRadix - 1);
      sbuf[lstart[q] + wc[q] + rnk[k]] = make_uint2(key[k], val[k]);
    }
  }
  __syncthreads();
  for (uint32_t lp = threadIdx.x; lp < n_block; lp += kSortThreads) {
    const uint2 pr = sbuf[lp];
    const uint32_t g = dbase[(pr.x >> shift) & (kRadix - 1)] + lp;
    if (g >= n_out || !RM_INDEX_OK(g, RM_X_TETS, 13)) continue;
    if (pass < 3) keys_out[g] = pr.x;  // nobody reads the keys of the last pass
    vals_out[g] = pr.y;
  }
}

// finish_look_back of k_rank_rects, by a warp.
__device__ __noinline__ uint32_t count_touched_before(uint32_t before, const uint32_t* word, uint32_t blocks,
                                                      const uint32_t* order, const int4* rect) {
  note_recount(kRecountRankRects);
  // every lane may see another state of a word: the sum is lane 0's, which the count needs no lane to agree with
  return __shfl_sync(0xffffffffu, finish_look_back(before, word, blocks, 1, [&](uint32_t b) {
    uint32_t n = 0;
#pragma unroll 1
    for (int i = 0; i < kScanTile; ++i) n += regions_touched(rect[order[(int64_t)b * kScanTile + i]]);
    return n & 0x3FFFFFFFu;
  }), 0);
}

// Ranked rectangles: rect[order[i]] for every visible rank i, in rank order; the inclusive scan of the number of regions
// each touches; and, by the block of the last rank, the info block.  The list build reads the rectangles in rank order;
// gathering them once, here, is a fraction of the three gathers per pair that it took to read them by tet id.  One launch
// with look-back: the counts change hands in shared memory between the gather's striped order and the scan's blocked one.
__global__ void __launch_bounds__(kScanThreads)
k_rank_rects(const uint32_t* order, const int4* rect, int64_t T, BinCounters* counters,
             uint32_t* __restrict__ look /* zeroed */, int4* __restrict__ ranked, uint32_t* __restrict__ cum,
             RmBinInfo* __restrict__ info, RmBinInfo* __restrict__ host_info) {
  after_previous();
  constexpr int kPad = kScanItems + 1;  // a thread's items in blocked order, spread over the banks
  __shared__ uint32_t touched[kScanThreads * kPad];
  __shared__ uint32_t sm[kScanThreads / 32 + 1];
  __shared__ uint32_t s_tile, s_before;
  if (threadIdx.x == 0) s_tile = atomicAdd(&counters->rank_ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const int64_t first = (int64_t)tile * kScanTile, n = valid_items(T, &counters->n_visible);
  const bool last = first + kScanTile >= n && (first < n || tile == 0);
  if (first >= n && !last) return;
  uint32_t id[kScanItems];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = first + k * kScanThreads + threadIdx.x;
    id[k] = i < n ? order[i] : 0u;
  }
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int j = k * kScanThreads + threadIdx.x;
    uint32_t v = 0;
    if (first + j < n && RM_INDEX_OK(id[k], RM_X_TETS, 13)) {
      const int4 rc = rect[id[k]];
      ranked[first + j] = rc;
      v = regions_touched(rc);
    }
    touched[j / kScanItems * kPad + j % kScanItems] = v;
  }
  __syncthreads();
  uint32_t v[kScanItems], s = 0, total;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += v[k] = touched[threadIdx.x * kPad + k];
  uint32_t ex = block_exclusive_scan<kScanThreads>(s, &total, sm);
  if (threadIdx.x < 32) {
    // more pairs than a list can hold are reported through n_keys: the words only must not lose their flags
    if (threadIdx.x == 0) store_relaxed(look + tile, tile == 0 ? kRunEnd | (total & ~kRunEnd) : (total & 0x3FFFFFFFu) + 1u);
    const uint32_t before =
        tile == 0 ? 0u : warp_look_back(look + tile, tile, [&](uint32_t sum, const uint32_t* word, uint32_t blocks) {
          return count_touched_before(sum, word, blocks, order, rect);
        });
    if (threadIdx.x == 0) {
      if (tile) store_relaxed(look + tile, kRunEnd | ((before + total) & ~kRunEnd));
      s_before = before;
    }
  }
  __syncthreads();
  ex += s_before;
  if (last && threadIdx.x == 0) {
    RmBinInfo r;
    r.n_keys = (int64_t)counters->n_keys;
    r.n_region_keys = (int64_t)(s_before + total);
    r.n_visible = (int32_t)counters->n_visible;
    r.status = counters->status | (counters->n_keys > 0x7fffffffull ? RM_STATUS_KEY_OVERFLOW : 0u);
    *info = r;
    if (host_info) *host_info = r;
  }
  const int64_t base = first + (int64_t)threadIdx.x * kScanItems;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) v[k] = ex += v[k];
  if (base + kScanItems <= n) {
#pragma unroll
    for (int k = 0; k < kScanItems; k += 4)
      *reinterpret_cast<uint4*>(cum + base + k) = make_uint4(v[k], v[k + 1], v[k + 2], v[k + 3]);
  } else {
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
      if (base + k < n) cum[base + k] = v[k];
  }
}

// ---------------------------------------------------------------------------
// Tile lists, built in two levels.
//
// Level 1 (regions).  Work items are the (region, tet) pairs numbered in rank
// order (tets by rank, then region rows, then columns): item j belongs to the
// rank r with cum[r-1] <= j < cum[r].  A stable counting sort on the
// region id leaves every region's segment
// ordered by rank, i.e. by (depth bits, tet id): no per-region sort, no atomics
// on the data path, deterministic.  A tet touches far fewer regions than tiles
// (about 9 times fewer at 1080p with 4 x 4 pixel tiles), so this sort moves a
// fraction of the pairs.  Every sorted entry carries the tet id and a 32-bit
// mask of the region's tiles its rectangle covers.
//   pairs:  the (tet, region) pairs and the digit totals of all passes
//   passes: stable splits on digits of the region id of at most 8 bits, low digit first; a pass is one launch with
//           look-back, like those of the rank sort; the last one writes the entries (tet id, tile mask) and counts
//           every region's entries at the ends of its runs
//
// Level 2 (tiles).  A region's segment is cut into chunks of kChunk entries, one
// warp per chunk, lane l owning tile l of the region.  A lane's tile list is the
// subsequence of entries whose mask has bit l; see k_fine_lists.  Order inside a
// tile is the order of the region's segment: rank order.
// ---------------------------------------------------------------------------
constexpr int kBinThreads = 256;
static_assert(kBinThreads == kSortThreads, "place_runs is shared by the rank sort and the region sort");
constexpr int kBinWarps = kBinThreads / 32;
constexpr int kChunk = 256;        // entries of a region segment handled by one warp
// Pairs per thread: 4 for the few pairs of a small frame, as in the rank sort.
constexpr int bin_items(int64_t n) { return n <= 128 * 4 * kBinThreads ? 4 : 16; }

template <int THREADS>
__device__ __forceinline__ uint32_t block_exclusive_maxscan(uint32_t v, uint32_t* smem /* THREADS/32 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc = max(inc, n);
  }
  if (lane == 31) smem[warp] = inc;
  __syncthreads();
  uint32_t prev = 0;
  for (int w = 0; w < warp; ++w) prev = max(prev, smem[w]);
  uint32_t up = __shfl_up_sync(0xffffffffu, inc, 1);
  uint32_t ex = lane ? max(prev, up) : prev;
  __syncthreads();
  return ex;
}

// First rank r in [0, n] with cum[r] > j0, found by the whole block: 256 probes a round, three rounds for 16M ranks.
__device__ __forceinline__ uint32_t first_rank_above(const uint32_t* __restrict__ cum, uint32_t n, uint32_t j0) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t step = (hi - lo + kBinThreads - 1) / kBinThreads;
    const uint32_t probe = min(lo + (threadIdx.x + 1) * step, hi) - 1;
    const uint32_t c = (uint32_t)__syncthreads_count(__ldg(cum + probe) <= j0);
    if (c == kBinThreads) return hi;
    hi = min(lo + (c + 1) * step, hi) - 1;
    lo += c * step;
  }
  return lo;
}

// Owner table of the block's items: after this call item jl (0 <= jl < items of the
// block) belongs to rank *r0 + own[jl]; win[i] = cum[*r0 + i].
template <int kBinItems>
__device__ __forceinline__ void owners_of_items(const uint32_t* __restrict__ cum, int n_ranked, int64_t j0,
                                                uint32_t start_rank,
                                                uint32_t* win /* kBinTile+1 */, uint16_t* own /* kBinTile */,
                                                uint32_t* s_misc /* 16 words */) {
  constexpr int kBinTile = kBinThreads * kBinItems;
  if (threadIdx.x == 0) {
    s_misc[8] = start_rank;
    s_misc[9] = start_rank > 0 ? cum[start_rank - 1] : 0u;  // items before rank r0
  }
  for (int i = threadIdx.x; i < kBinTile; i += kBinThreads) own[i] = 0;
  __syncthreads();
  const int r0 = (int)s_misc[8];
  for (int i = threadIdx.x; i <= kBinTile; i += kBinThreads) {
    int r = r0 + i;
    uint32_t c = r < n_ranked ? cum[r] : 0xFFFFFFFFu;
    win[i] = c;
    // rank r0+i+1 starts at item c (visible tets have at least one item, so starts are distinct)
    int64_t start = (int64_t)c - j0;
    if (c != 0xFFFFFFFFu && start < kBinTile && r + 1 < n_ranked) own[start] = (uint16_t)(i + 1);
  }
  __syncthreads();
  // inclusive max-scan of own[], thread t owning kBinItems consecutive items
  uint32_t loc[kBinItems];
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < kBinItems; ++k) {
    m = max(m, (uint32_t)own[threadIdx.x * kBinItems + k]);
    loc[k] = m;
  }
  uint32_t ex = block_exclusive_maxscan<kBinThreads>(m, s_misc);
#pragma unroll
  for (int k = 0; k < kBinItems; ++k) own[threadIdx.x * kBinItems + k] = (uint16_t)max(ex, loc[k]);
  __syncthreads();
}

// A (region, tet) pair is (tet, code), code = region << 10 | the part of the region the tet's rectangle covers: first and
// last column (3 bits each), first and last row (2 bits each).
constexpr int kCodeBits = 10;
__device__ __forceinline__ uint32_t region_code(uint32_t region, int gx, int gy, int4 rc) {
  const uint32_t lx0 = max(rc.x - gx * kRegW, 0), lx1 = min(rc.z - gx * kRegW, kRegW) - 1;
  const uint32_t ly0 = max(rc.y - gy * kRegH, 0), ly1 = min(rc.w - gy * kRegH, kRegH) - 1;
  return region << kCodeBits | lx0 << 7 | lx1 << 4 | ly0 << 2 | ly1;
}
// mask of the region's tiles (bit = 8 * row + column)
__device__ __forceinline__ uint32_t code_mask(uint32_t code) {
  const uint32_t lx0 = (code >> 7) & 7u, lx1 = (code >> 4) & 7u, ly0 = (code >> 2) & 3u, ly1 = code & 3u;
  const uint32_t row = (2u << lx1) - (1u << lx0);
  const uint32_t rows = (0x01010101u >> (8 * (3 - ly1))) & ~((1u << (8 * ly0)) - 1u);
  return row * rows;
}

// pair of local item jl
__device__ __forceinline__ uint2 item_pair(int jl, int64_t j0, int r0, uint32_t before_r0, const uint32_t* win,
                                           const uint16_t* own, const uint32_t* __restrict__ order,
                                           const int4* __restrict__ ranked, int reg_w) {
  const int i = own[jl];
  const uint32_t rank = (uint32_t)(r0 + i);
  const uint32_t excl = i > 0 ? win[i - 1] : before_r0;
  const uint32_t local = (uint32_t)(j0 + jl - excl);
  const int4 rc = __ldg(ranked + rank);
  const uint32_t cx0 = (uint32_t)(rc.x >> kRegShiftX);
  const uint32_t w = (uint32_t)((rc.z - 1) >> kRegShiftX) - cx0 + 1u;
  const uint32_t dy = local / w;
  const uint32_t gy = (uint32_t)(rc.y >> kRegShiftY) + dy, gx = cx0 + (local - dy * w);
  return make_uint2(__ldg(order + rank), region_code(gy * (uint32_t)reg_w + gx, (int)gx, (int)gy, rc));
}

// Generates the block's (tet, region) pairs, writes them out, and adds up the digit totals of all passes.
// digit_total: [passes][kRadix], zero so far.  Also zero-fills what the later launches count and look back in.
constexpr int kMaxPasses = 3;
template <int kBinItems>
__global__ void __launch_bounds__(kBinThreads)
k_region_pairs(const uint32_t* __restrict__ cum, const uint32_t* __restrict__ order, int n_tets,
               const uint32_t* __restrict__ n_dev, const int4* __restrict__ ranked, int reg_w, int64_t n_items, int passes,
               int bits, uint32_t* __restrict__ digit_total, uint2* __restrict__ pairs_out, uint4* __restrict__ zero,
               int64_t n_zero) {
  after_previous();
  constexpr int kBinTile = kBinThreads * kBinItems;
  for (int64_t i = (int64_t)blockIdx.x * kBinThreads + threadIdx.x; i < n_zero; i += (int64_t)gridDim.x * kBinThreads)
    zero[i] = make_uint4(0u, 0u, 0u, 0u);
  __shared__ uint32_t win[kBinTile + 4];
  __shared__ uint32_t s_misc[16];
  __shared__ uint16_t own[kBinTile];
  __shared__ uint32_t h[kMaxPasses * kRadix];
  const int64_t j0 = (int64_t)blockIdx.x * kBinTile;
  const int cnt = (int)min((int64_t)kBinTile, n_items - j0);
  const uint32_t n_ranked = (uint32_t)valid_items(n_tets, n_dev);
  for (int i = threadIdx.x; i < passes * kRadix; i += kBinThreads) h[i] = 0;
  owners_of_items<kBinItems>(cum, (int)n_ranked, j0, first_rank_above(cum, n_ranked, (uint32_t)j0), win, own, s_misc);
  const int r0 = (int)s_misc[8];
  const uint32_t before = s_misc[9], bins = 1u << bits;
  for (int jl = threadIdx.x; jl < cnt; jl += kBinThreads) {
    const uint2 pair = item_pair(jl, j0, r0, before, win, own, order, ranked, reg_w);
    const uint32_t region = pair.y >> kCodeBits;
    if (!(RM_INDEX_OK(region, RM_X_REGIONS, 11) && RM_INDEX_OK(pair.x, RM_X_TETS, 13))) continue;
    pairs_out[j0 + jl] = pair;
    for (int q = 0; q < passes; ++q) atomicAdd(&h[q * kRadix + ((region >> (q * bits)) & (bins - 1))], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kRadix; i += kBinThreads)
    if (h[i]) atomicAdd(digit_total + i, h[i]);
}

// What the last pass leaves of the regions: how many entries each has (zeroed), where they start in the sorted entries and
// in the chunks (both with a closing total at index n_regions).
struct RegionTable {
  uint32_t n_regions;
  uint32_t *count, *start, *chunk_base, *done;
};
// By one block: exclusive scans of the counts and of ceil(count / chunk size), together in the halves of 64-bit words,
// eight regions per thread and round.
__device__ __noinline__ void layout_regions(const RegionTable& t) {
  __shared__ unsigned long long warp_sum[kBinWarps];
  constexpr uint32_t kPer = 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long carry = 0;
  for (uint32_t base = 0; base < t.n_regions; base += kBinThreads * kPer) {
    const uint32_t r0 = base + threadIdx.x * kPer;
    unsigned long long v[kPer], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      const uint32_t c = r0 + k < t.n_regions ? __ldcg(t.count + r0 + k) : 0u;
      v[k] = (unsigned long long)((c + kChunk - 1) / kChunk) << 32 | c;
      sum += v[k];
    }
    unsigned long long inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long up = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += up;
    }
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    unsigned long long ex = carry + inc - sum;
#pragma unroll
    for (int w = 0; w < kBinWarps; ++w) {
      if (w < warp) ex += warp_sum[w];
      carry += warp_sum[w];
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      if (r0 + k < t.n_regions) {
        t.start[r0 + k] = (uint32_t)ex;
        t.chunk_base[r0 + k] = (uint32_t)(ex >> 32);
      }
      ex += v[k];
    }
  }
  if (threadIdx.x == 0) {
    t.start[t.n_regions] = (uint32_t)carry;
    t.chunk_base[t.n_regions] = (uint32_t)(carry >> 32);
  }
}

// finish_look_back of k_region_pass; a thread per digit.
__device__ __noinline__ uint32_t count_pairs_before(uint32_t before, const uint32_t* word, uint32_t blocks, const uint2* pairs,
                                                    int tile, int shift, uint32_t bins) {
  note_recount(kRecountRegionPass);
  return finish_look_back(before, word, blocks, (int)bins, [&](uint32_t b) {
    uint32_t n = 0;
#pragma unroll 1
    for (int i = 0; i < tile; ++i) n += ((pairs[(int64_t)b * tile + i].y >> shift) & (bins - 1)) == threadIdx.x;
    return n;
  });
}

// One stable pass on the digit (code >> shift) & (2^BITS - 1).  final == 0: the reordered pairs go to pairs_out;
// final != 0: the sorted entries (tet id, tile mask) are written instead, and the regions' entries are counted: in the
// block's reordered buffer a region's pairs are contiguous, so that the position of a run's first pair is subtracted
// from its region's count and the position behind its last added.
template <int BITS, int kBinItems>
__global__ void __launch_bounds__(kBinThreads, 3)
k_region_pass(const uint2* pairs, int64_t n, int shift, const uint32_t* digit_total,
              uint32_t* __restrict__ ticket, uint32_t* __restrict__ look /* [blocks][2^BITS], zeroed */,
              int final, uint2* __restrict__ pairs_out, uint2* __restrict__ entries,
              RegionTable table) {
  after_previous();
  constexpr int kBinTile = kBinThreads * kBinItems;
  constexpr int kBinSpan = 32 * kBinItems;  // consecutive items owned by one warp
  __shared__ uint2 sbuf[kBinTile];
  __shared__ uint32_t cnt[kBinWarps * kRadix];  // per-warp digit counts -> offsets
  __shared__ uint32_t dbase[kRadix], lstart[kRadix];
  __shared__ uint32_t sm[kBinThreads / 32 + 1];
  __shared__ uint32_t s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr uint32_t bins = 1u << BITS;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  for (int i = threadIdx.x; i < kBinWarps * kRadix; i += kBinThreads) cnt[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const int64_t base = (int64_t)tile * kBinTile;
  if (base >= n) return;
  const int n_block = (int)min((int64_t)kBinTile, n - base);
  uint32_t* wc = cnt + warp * kRadix;
  uint2 pr[kBinItems];
#pragma unroll
  for (int k = 0; k < kBinItems; ++k) {
    const int jl = warp * kBinSpan + k * 32 + lane;
    pr[k] = jl < n_block ? pairs[base + jl] : make_uint2(0u, 0u);
  }
  uint32_t rnk[kBinItems / 2];
#pragma unroll
  for (int k = 0; k < kBinItems; ++k) {
    const bool valid = warp * kBinSpan + k * 32 + lane < n_block;
    const uint32_t digit = (pr[k].y >> shift) & (bins - 1);
    // lanes with the same digit, from one ballot per bit: constant cost, where match.any slows down with the number
    // of distinct values
    uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
      const bool bit = (digit >> b) & 1u;
      const uint32_t m = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? m : ~m;
    }
    const uint32_t before = __popc(peers & ((1u << lane) - 1u));
    uint32_t prev = 0;
    if (valid) prev = wc[digit];
    __syncwarp();
    if (valid && before == 0) wc[digit] = prev + __popc(peers);
    __syncwarp();
    const uint32_t r = prev + before;
    if (k & 1) rnk[k >> 1] |= r << 16; else rnk[k >> 1] = r;
  }
  __syncthreads();
  place_runs<8>(threadIdx.x < bins, threadIdx.x < bins ? digit_total[threadIdx.x] : 0u, tile, look, (int)bins, cnt, dbase,
                lstart, sm, [&](uint32_t before, const uint32_t* word, uint32_t blocks) {
                  return count_pairs_before(before, word, blocks, pairs, kBinTile, shift, bins);
                });
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kBinItems; ++k) {
    if (warp * kBinSpan + k * 32 + lane >= n_block) continue;
    const uint32_t digit = (pr[k].y >> shift) & (bins - 1);
    sbuf[lstart[digit] + wc[digit] + ((rnk[k >> 1] >> (16 * (k & 1))) & 0xFFFFu)] = pr[k];
  }
  __syncthreads();
  for (int lp = threadIdx.x; lp < n_block; lp += kBinThreads) {
    const uint2 p2 = sbuf[lp];
    const uint32_t g = dbase[(p2.y >> shift) & (bins - 1)] + (uint32_t)lp;
    if (g >= n || !RM_INDEX_OK(g, RM_X_PAIRS, 9)) continue;
    if (!final) {
      pairs_out[g] = p2;
      continue;
    }
    entries[g] = make_uint2(p2.x, code_mask(p2.y));
    const uint32_t region = p2.y >> kCodeBits;
    if (!RM_INDEX_OK(region, RM_X_REGIONS, 11)) continue;
    const bool first = lp == 0 || (sbuf[lp - 1].y >> kCodeBits) != region;
    const bool last = lp == n_block - 1 || (sbuf[lp + 1].y >> kCodeBits) != region;
    const uint32_t add = (first ? 0u - (uint32_t)lp : 0u) + (last ? (uint32_t)lp + 1u : 0u);
    if (add) atomicAdd(table.count + region, add);
  }
  if (!final) return;
  // the block that is done last lays out the regions
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(table.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (s_last) layout_regions(table);
}

// ---------------------------------------------------------------------------
// Level 2: from the region segments to the tile lists.
// ---------------------------------------------------------------------------
constexpr int kFineThreads = 128;  // 4 warps = 4 chunks per block
constexpr int kFineWarps = kFineThreads / 32;

// 32 x 32 bit transpose across the warp: lane l ends with bit i = bit l of lane i's word.
__device__ __forceinline__ uint32_t warp_bit_transpose(uint32_t a) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 16; j >= 1; j >>= 1) {
    const uint32_t m = j == 16 ? 0x0000FFFFu : j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu : j == 2 ? 0x33333333u
                                                                                                    : 0x55555555u;
    const uint32_t b = __shfl_xor_sync(0xffffffffu, a, j);
    a = (lane & j) ? (((b >> j) & m) | (a & ~m)) : ((a & m) | ((b & m) << j));
  }
  return a;
}

// Region of a chunk: the last r with chunk_base[r] <= chunk, found by the whole warp, 32 probes a round.
__device__ __forceinline__ uint32_t region_of_chunk(const uint32_t* chunk_base, uint32_t n_regions, uint32_t chunk) {
  uint32_t lo = 0, hi = n_regions;  // first index with chunk_base > chunk lies in [lo, hi]: chunk_base[n_regions] > chunk
  while (lo < hi) {
    const uint32_t step = (hi - lo + 31) / 32;
    const uint32_t probe = min(lo + ((threadIdx.x & 31) + 1) * step, hi) - 1;
    const uint32_t c = __popc(__ballot_sync(0xffffffffu, chunk_base[probe] <= chunk));
    if (c == 32) {
      lo = hi;
    } else {
      hi = min(lo + (c + 1) * step, hi) - 1;
      lo += c * step;
    }
  }
  return lo - 1;
}

// Expands the chunks to tile lists.  A warp reads the masks of its chunk in rounds of 32 entries and transposes them, so
// that lane l holds the bit sets of the entries that cover tile l; publishes how many there are; collects their positions
// in the chunk, one byte each, in shared memory; learns from the region's chunks before it where its tiles' lists go on
// (look-back, as in the sort passes, blocks numbered by a ticket); and writes tile after tile, 32 consecutive list entries
// per store.  Bound by the issue of shared-memory and store instructions.  The lists were written straight from the
// entries before, one store of the covering lanes per round and tile, after a counting launch and one for the cursors:
// 462 us for the three at 6.7M tets, 1080p (142M list entries), 2.85 ms at 36M, 2160p (886M); this 281 us and 1.55 ms.
constexpr int kFineRounds = kChunk / 32;
constexpr int kFineStride = kChunk + 4;  // bytes per tile: the lanes' byte stores fall into different banks

// finish_look_back of k_fine_lists over the chunks of a region, whose entries start at `first`; a lane per tile.
__device__ __noinline__ uint32_t count_covering_before(uint32_t before, const uint32_t* word, uint32_t chunks, const uint2* first) {
  note_recount(kRecountFineLists);
  return finish_look_back(before, word, chunks, 32, [&](uint32_t k) {
    uint32_t n = 0;
#pragma unroll 1
    for (int i = 0; i < kChunk; ++i) n += (first[(int64_t)k * kChunk + i].y >> (threadIdx.x & 31)) & 1u;
    return n;
  });
}

__global__ void __launch_bounds__(kFineThreads)
k_fine_lists(const uint2* entries, const uint32_t* region_start, const uint32_t* chunk_base, uint32_t n_regions, int reg_w,
             int grid_w, int grid_h, const uint32_t* __restrict__ tile_start, uint32_t* __restrict__ ticket,
             uint32_t* __restrict__ look /* zeroed */, uint32_t* __restrict__ digit_total, uint32_t n_keys,
             int32_t* __restrict__ sorted_idx) {
  after_previous();
  __shared__ uint8_t s_pos[kFineWarps][32 * kFineStride];
  __shared__ int32_t s_id[kFineWarps][kChunk];
  __shared__ uint32_t s_block;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_block = atomicAdd(ticket, 1u);
  __syncthreads();
  if (s_block == 0)  // nobody needs them any more; the lists can then be built again from the same first half
    for (int i = threadIdx.x; i < kMaxPasses * kRadix; i += kFineThreads) digit_total[i] = 0;
  const uint32_t chunk = s_block * kFineWarps + warp;
  if (chunk >= chunk_base[n_regions]) return;
  if (!RM_INDEX_OK(chunk, RM_X_CHUNKS, 10)) return;
  const uint32_t r = region_of_chunk(chunk_base, n_regions, chunk);
  const uint32_t k_in_region = chunk - chunk_base[r];
  const uint32_t begin = region_start[r] + k_in_region * kChunk;
  const uint32_t count = min((uint32_t)kChunk, region_start[r + 1] - begin);
  uint8_t* pos = s_pos[warp] + lane * kFineStride;
  int32_t* ids = s_id[warp];
  uint32_t word[kFineRounds], n = 0;
  {
    uint2 en[kFineRounds];
#pragma unroll
    for (int k = 0; k < kFineRounds; ++k) {
      const uint32_t e = 32 * k + lane;
      en[k] = (e < count && RM_INDEX_OK(begin + e, RM_X_PAIRS, 9)) ? entries[begin + e] : make_uint2(0u, 0u);
    }
#pragma unroll
    for (int k = 0; k < kFineRounds; ++k) {
      ids[32 * k + lane] = (int32_t)en[k].x;
      word[k] = __brev(warp_bit_transpose(en[k].y));  // entry 32 k + i at bit 31 - i
      n += __popc(word[k]);
    }
  }
  uint32_t* mine = look + (size_t)chunk * 32 + lane;
  store_relaxed(mine, k_in_region == 0 ? kRunEnd | n : n + 1u);
  uint32_t c = 0;
#pragma unroll
  for (int k = 0; k < kFineRounds; ++k) {
    for (uint32_t w = word[k]; w;) {
      const uint32_t b = 31 - __clz(w);
      w ^= 1u << b;
      pos[c++] = (uint8_t)(32 * k + 31 - b);
    }
  }
  uint32_t before = 0;
  if (k_in_region) {
    before = look_back<8>(mine, k_in_region, 32, [&](uint32_t sum, const uint32_t* word, uint32_t chunks) {
      return count_covering_before(sum, word, chunks, entries + (begin - k_in_region * kChunk));
    });
    store_relaxed(mine, kRunEnd | (before + n));
  }
  const int gy = (int)(r / (uint32_t)reg_w), gx = (int)(r - (uint32_t)gy * (uint32_t)reg_w);
  const int tx = gx * kRegW + (lane & (kRegW - 1)), ty = gy * kRegH + (lane >> kRegShiftX);
  uint32_t at = before;  // first list position of this lane's tile that the chunk fills
  if (tx < grid_w && ty < grid_h && RM_INDEX_OK((int64_t)ty * grid_w + tx, RM_X_TILES, 12))
    at += __ldg(tile_start + (int64_t)ty * grid_w + tx);
  __syncwarp();
  // at + n <= n_keys always holds when the masks agree with the tile populations; the clamp keeps a disagreement from
  // writing outside the list array
  if (at + n > n_keys) n = at < n_keys ? n_keys - at : 0u;
  const uint8_t* from = s_pos[warp] + lane;
  for (int t = 0; t < 32; ++t, from += kFineStride) {
    const int n_t = (int)__shfl_sync(0xffffffffu, n, t), mine_t = n_t - lane;
    const uint32_t at_t = __shfl_sync(0xffffffffu, at, t) + lane;
    int32_t* out = sorted_idx + at_t;
#pragma unroll
    for (int k = 0; k < kFineRounds; ++k) {
      if (32 * k >= n_t) break;
      if (32 * k < mine_t && RM_INDEX_OK(at_t + 32 * k, RM_X_LIST, 8)) out[32 * k] = ids[from[32 * k]];
    }
  }
}

}  // namespace rm

// ---------------------------------------------------------------------------
// Workspace layout (all sub-buffers 256-byte aligned)
// ---------------------------------------------------------------------------
namespace {
struct BinLayout {
  size_t keys_a, keys_b, ord_a, ord_b, ranked, cum, bsum, tile_count, tile_start, zero, counters, digit_hist, region_digits, look,
      rank_look, tile_diff, total;
  size_t zero_bytes;  // [zero, zero + zero_bytes): counters, digit histograms, look-back words, tile coverage
  int sort_items, nblk_sort, diff_copies;
  int64_t nblk_scan_t, nblk_scan_g;
};
inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
// A small tile grid gets several partial difference arrays, dealt to the blocks of the projection: its
// atomics otherwise queue on few addresses (614k tets on the 51 x 51 corners of 16 x 16-pixel tiles: k_project
// 265 us, against 43 us for the same tets on 201 x 201).  128 KB hold 8 copies of that grid and one of any grid
// larger than 127 x 127, where the queues are short; of the smallest grids they hold thousands, which a lane then adds up
// one after another.  A copy for every two blocks of the projection is enough (projection and rank sort of 13k tets on
// 2 x 2 corners 330 us with all that fit, 53 with a copy for 256 tets, 66 for 512; 600k tets 488, 222, 177; on 9 x 9
// corners 46, 39, 37 and 117, 113, 113).
constexpr int64_t kDiffWords = 32768, kTetsPerDiffCopy = 256;
BinLayout make_layout(int64_t T, int64_t G, int gh, int gw) {
  BinLayout L;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align256(off + bytes);
    return o;
  };
  int64_t Tp = T > 0 ? T : 1;
  L.sort_items = rm::sort_items(Tp);
  const int64_t sort_tile = (int64_t)L.sort_items * rm::kSortThreads;
  L.nblk_sort = (int)((Tp + sort_tile - 1) / sort_tile);
  L.nblk_scan_t = (Tp + rm::kScanTile - 1) / rm::kScanTile;
  L.nblk_scan_g = (G + rm::kScanTile - 1) / rm::kScanTile;
  L.keys_a = take(4 * Tp);
  L.keys_b = take(4 * Tp);
  L.ord_a = take(4 * Tp);
  L.ord_b = take(4 * Tp);
  L.ranked = take(16 * Tp);
  L.cum = take(4 * Tp);
  L.bsum = take(4 * (size_t)L.nblk_scan_g + 4);
  L.tile_count = take(4 * (size_t)(G + 1));
  L.tile_start = take(4 * (size_t)(G + 1));
  L.zero = off;
  L.counters = take(sizeof(rm::BinCounters));
  L.digit_hist = take(4 * 4 * rm::kRadix);
  L.region_digits = take(4 * rm::kMaxPasses * rm::kRadix);
  L.look = take(4 * 4 * (size_t)rm::kRadix * L.nblk_sort);
  L.rank_look = take(4 * (size_t)L.nblk_scan_t);
  // (gh+1)*(gw+1) <= G + gh + gw + 1; gh, gw <= G
  const int64_t n_diff = gh >= 0 ? (int64_t)(gh + 1) * (gw + 1) : 4 * G + 4;
  L.diff_copies = 1;
  while (2 * L.diff_copies * n_diff <= kDiffWords && 2 * L.diff_copies * kTetsPerDiffCopy <= T) L.diff_copies *= 2;
  L.tile_diff = take(4 * (size_t)(n_diff > kDiffWords ? n_diff : kDiffWords));
  L.zero_bytes = L.tile_diff + 4 * (size_t)(L.diff_copies * n_diff) - L.zero;
  L.total = off;
  return L;
}
}  // namespace

size_t rm_bin_layout_bytes(int64_t T, int64_t G) {
  // upper bound that does not need gh, gw: (gh+1)(gw+1) <= 2G + 2 for gh, gw >= 1 ... use 4G + 4
  return make_layout(T, G, -1, -1).total;
}

int rm_launch_bin_prepare(int64_t T, const RmCamera* cam, void* ws, size_t ws_bytes, uint32_t** depth_keys,
                          int32_t** tile_diff, int* diff_copies, uint32_t** counters, uint32_t** deferred,
                          cudaStream_t st) {
  const int gh = cam->grid_height, gw = cam->grid_width;
  const int64_t G = (int64_t)gh * gw;
  BinLayout L = make_layout(T, G, gh, gw);
  if (L.total > ws_bytes) return RM_ERR_WORKSPACE;
  char* b = static_cast<char*>(ws);
  *depth_keys = reinterpret_cast<uint32_t*>(b + L.keys_a);
  *tile_diff = reinterpret_cast<int32_t*>(b + L.tile_diff);
  *diff_copies = L.diff_copies;
  *counters = reinterpret_cast<uint32_t*>(b + L.counters);  // n_visible, status, n_deferred
  *deferred = reinterpret_cast<uint32_t*>(b + L.keys_b);    // free until the sort
  RM_CUDA_CHECK(cudaMemsetAsync(b + L.zero, 0, L.zero_bytes, st));
  return RM_OK;
}

// After k_project: rank the tets, build tile_ranges, the rank-ordered inclusive
// scan of the regions every tet touches, and the info block.
int rm_launch_bin_finish(int64_t T, const RmCamera* cam, const int32_t* rect, int32_t* tile_ranges,
                         RmBinInfo* info, RmBinInfo* host_info, void* ws, cudaStream_t st) {
  const int gh = cam->grid_height, gw = cam->grid_width;
  const int64_t G = (int64_t)gh * gw;
  BinLayout L = make_layout(T, G, gh, gw);
  char* b = static_cast<char*>(ws);
  uint32_t* keys[2] = {reinterpret_cast<uint32_t*>(b + L.keys_a), reinterpret_cast<uint32_t*>(b + L.keys_b)};
  uint32_t* ord[2] = {reinterpret_cast<uint32_t*>(b + L.ord_a), reinterpret_cast<uint32_t*>(b + L.ord_b)};
  uint32_t* cum = reinterpret_cast<uint32_t*>(b + L.cum);
  uint32_t* bsum = reinterpret_cast<uint32_t*>(b + L.bsum);
  int32_t* diff = reinterpret_cast<int32_t*>(b + L.tile_diff);
  uint32_t* tcount = reinterpret_cast<uint32_t*>(b + L.tile_count);
  uint32_t* tstart = reinterpret_cast<uint32_t*>(b + L.tile_start);
  uint32_t* digit_hist = reinterpret_cast<uint32_t*>(b + L.digit_hist);
  rm::BinCounters* counters = reinterpret_cast<rm::BinCounters*>(b + L.counters);

  rm_set_extent(RM_X_TETS, T, st);
  rm_set_extent(RM_X_TILES, G, st);
  // Rank the visible tets by (depth bits, id): four stable radix passes that start and end in buffer 0.  Ranks past the
  // visible tets hold nothing that later stages read.  With them, a step each, go the tile populations and tile_ranges.
  rm::TileJob job = {0,        0,      diff, L.diff_copies, gh, gw, tcount, bsum, tstart, reinterpret_cast<int2*>(tile_ranges),
                     counters};
  auto tile_step = [&](int step) {
    job.step = step;
    const int64_t warps = step == 0 ? gh + 1 : gw;
    job.blocks = step < 2 ? (int)((warps + rm::kJobThreads / 32 - 1) / (rm::kJobThreads / 32)) : (int)L.nblk_scan_g;
    return job;
  };
  {
    RmProfScope prof("rank_tets_radix_sort", st);
    const rm::TileJob first = tile_step(0);
    const int64_t hist_blocks = (T + 8 * rm::kSortThreads - 1) / (8 * rm::kSortThreads);
    RM_CUDA_CHECK(rm_launch_behind(T, rm::k_digit_hist, (unsigned)(first.blocks + (hist_blocks < 4 * 148 ? hist_blocks : 4 * 148)),
                                   rm::kSortThreads, 0, st, keys[0], T, digit_hist, first));
    const int nblk = T > 0 ? L.nblk_sort : 0;
    for (int pass = 0; pass < 4; ++pass) {
      const int src = pass & 1, dst = src ^ 1;
      uint32_t* look = reinterpret_cast<uint32_t*>(b + L.look) + (size_t)pass * rm::kRadix * L.nblk_sort;
      rm::TileJob with = job;
      with.blocks = 0;
      if (pass < 3) with = tile_step(pass + 1);
      if (with.blocks + nblk == 0) continue;
      auto kernel = L.sort_items == 4 ? (pass == 0 ? rm::k_rank_pass<true, 4> : rm::k_rank_pass<false, 4>)
                                      : (pass == 0 ? rm::k_rank_pass<true, 16> : rm::k_rank_pass<false, 16>);
      RM_CUDA_CHECK(rm_launch_behind(T, kernel, (unsigned)(with.blocks + nblk), rm::kSortThreads, 0, st, keys[src], ord[src], T,
                                     counters, pass, digit_hist + pass * rm::kRadix, look, keys[dst], ord[dst], with));
    }
  }
  // rectangles in rank order, inclusive scan of the number of regions every visible tet touches, info
  {
    RmProfScope prof("k_rank_rects", st);
    RM_CUDA_CHECK(rm_launch_behind(T, rm::k_rank_rects, (unsigned)L.nblk_scan_t, rm::kScanThreads, 0, st, ord[0],
                                   reinterpret_cast<const int4*>(rect), T, counters,
                                   reinterpret_cast<uint32_t*>(b + L.rank_look), reinterpret_cast<int4*>(b + L.ranked), cum,
                                   info, host_info));
  }
  return RM_OK;
}

namespace {
struct ListPlan {
  int reg_w, reg_h, passes, bits, items, nblk;  // passes of `bits` bits each over the region id
  uint32_t n_regions, max_chunks;
  size_t pairs_a, pairs_b, entries, region_start, chunk_base, zero, zero_bytes, tickets, region_count, look, fine_look,
      total;
};
// region grid, split of the region-id bits into digits, and the scratch layout
bool make_list_plan(int64_t n_region_keys, int gh, int gw, ListPlan* P) {
  P->reg_w = (gw + rm::kRegW - 1) / rm::kRegW;
  P->reg_h = (gh + rm::kRegH - 1) / rm::kRegH;
  const int64_t R = (int64_t)P->reg_w * P->reg_h;
  int bits = 1;
  while (((int64_t)1 << bits) < R) ++bits;
  if (bits > 32 - rm::kCodeBits || n_region_keys > 0x7fffffffll) return false;
  P->n_regions = (uint32_t)R;
  P->passes = (bits + rm::kRadixBits - 1) / rm::kRadixBits;
  P->bits = (bits + P->passes - 1) / P->passes;
  P->items = rm::bin_items(n_region_keys);
  const int64_t tile = (int64_t)P->items * rm::kBinThreads;
  P->nblk = (int)((n_region_keys + tile - 1) / tile);
  P->max_chunks = (uint32_t)(n_region_keys / rm::kChunk + R + 1);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off = align256(off + bytes);
    return o;
  };
  P->pairs_a = take(8 * (size_t)n_region_keys);
  P->pairs_b = take(P->passes > 1 ? 8 * (size_t)n_region_keys : 0);
  P->entries = take(8 * (size_t)n_region_keys);
  P->region_start = take(4 * (size_t)(R + 1));
  P->chunk_base = take(4 * (size_t)(R + 1));
  P->zero = off;
  P->tickets = take(4 * (rm::kMaxPasses + 2));
  P->region_count = take(4 * (size_t)(R + 1));
  P->look = take(4 * ((size_t)P->passes << P->bits) * (size_t)(P->nblk > 0 ? P->nblk : 1));
  P->fine_look = take(4 * 32 * (size_t)P->max_chunks);
  P->zero_bytes = off - P->zero;
  P->total = off;
  return true;
}
}  // namespace

// A kernel for every width of digit: with 8-bit digits throughout, whatever the number of regions, the passes took 222 us in
// place of 197 (6M tets, 4,080 regions: two of 6 bits) and 1079 in place of 1012 (36M, 16,200 regions: two of 7).
template <int ITEMS>
static auto pass_kernel(int bits) {
  static decltype(&rm::k_region_pass<1, ITEMS>) const kernels[rm::kRadixBits + 1] = {
      nullptr, rm::k_region_pass<1, ITEMS>, rm::k_region_pass<2, ITEMS>, rm::k_region_pass<3, ITEMS>,
      rm::k_region_pass<4, ITEMS>, rm::k_region_pass<5, ITEMS>, rm::k_region_pass<6, ITEMS>, rm::k_region_pass<7, ITEMS>,
      rm::k_region_pass<8, ITEMS>};
  return kernels[bits];
}

size_t rm_list_plan_bytes(int64_t n_region_keys, int gh, int gw) {
  ListPlan P;
  if (!make_list_plan(n_region_keys, gh, gw, &P)) return 0;
  return P.total;
}

int rm_launch_build_lists(int64_t T, const RmCamera* cam, int64_t n_keys, int64_t n_region_keys, void* ws, void* scratch,
                          size_t scratch_bytes, int32_t* sorted_idx, cudaStream_t st) {
  if (n_keys == 0) return RM_OK;
  const int gh = cam->grid_height, gw = cam->grid_width;
  const int64_t G = (int64_t)gh * gw;
  BinLayout L = make_layout(T, G, gh, gw);
  ListPlan P;
  if (n_region_keys < 1 || n_region_keys > n_keys || !make_list_plan(n_region_keys, gh, gw, &P))
    return RM_ERR_INVALID_ARG;
  if (P.total > scratch_bytes || (reinterpret_cast<uintptr_t>(scratch) & 255)) return RM_ERR_WORKSPACE;
  rm_set_extent(RM_X_TETS, T, st);
  rm_set_extent(RM_X_TILES, G, st);
  rm_set_extent(RM_X_LIST, n_keys, st);
  rm_set_extent(RM_X_PAIRS, n_region_keys, st);
  rm_set_extent(RM_X_CHUNKS, P.max_chunks, st);
  rm_set_extent(RM_X_REGIONS, P.n_regions, st);
  char* b = static_cast<char*>(ws);
  const uint32_t* order = reinterpret_cast<uint32_t*>(b + L.ord_a);
  const int4* ranked = reinterpret_cast<const int4*>(b + L.ranked);
  rm::BinCounters* counters = reinterpret_cast<rm::BinCounters*>(b + L.counters);
  const uint32_t* cum = reinterpret_cast<uint32_t*>(b + L.cum);
  const uint32_t* tile_start = reinterpret_cast<uint32_t*>(b + L.tile_start);
  char* sb = static_cast<char*>(scratch);
  uint2* pairs[2] = {reinterpret_cast<uint2*>(sb + P.pairs_a), reinterpret_cast<uint2*>(sb + P.pairs_b)};
  uint2* entries = reinterpret_cast<uint2*>(sb + P.entries);
  uint32_t* tickets = reinterpret_cast<uint32_t*>(sb + P.tickets);
  uint32_t* digit_total = reinterpret_cast<uint32_t*>(b + L.region_digits);
  uint32_t* fine_look = reinterpret_cast<uint32_t*>(sb + P.fine_look);
  const rm::RegionTable table = {P.n_regions, reinterpret_cast<uint32_t*>(sb + P.region_count),
                                 reinterpret_cast<uint32_t*>(sb + P.region_start),
                                 reinterpret_cast<uint32_t*>(sb + P.chunk_base), tickets + rm::kMaxPasses + 1};
  {
    RmProfScope prof("k_region_pairs", st);
    auto kernel = P.items == 4 ? rm::k_region_pairs<4> : rm::k_region_pairs<16>;
    RM_CUDA_CHECK(rm_launch(kernel, P.nblk, rm::kBinThreads, 0, st, cum, order, (int)T, &counters->n_visible, ranked,
                            P.reg_w, n_region_keys, P.passes, P.bits, digit_total, pairs[0],
                            reinterpret_cast<uint4*>(sb + P.zero), (int64_t)(P.zero_bytes / sizeof(uint4))));
  }
  {
    RmProfScope prof("k_region_pass", st);
    for (int pass = 0; pass < P.passes; ++pass) {
      uint32_t* look = reinterpret_cast<uint32_t*>(sb + P.look) + ((size_t)pass << P.bits) * P.nblk;
      auto kernel = P.items == 4 ? pass_kernel<4>(P.bits) : pass_kernel<16>(P.bits);
      RM_CUDA_CHECK(rm_launch_behind(n_region_keys, kernel, (unsigned)P.nblk, rm::kBinThreads, 0, st, pairs[pass & 1],
                                     n_region_keys, rm::kCodeBits + pass * P.bits, digit_total + pass * rm::kRadix,
                                     tickets + pass, look, pass == P.passes - 1, pairs[(pass & 1) ^ 1],
                                     entries, table));
    }
  }
  {
    RmProfScope prof("k_fine_lists", st);
    RM_CUDA_CHECK(rm_launch_behind(n_region_keys, rm::k_fine_lists, (unsigned)((P.max_chunks + rm::kFineWarps - 1) / rm::kFineWarps),
                                   rm::kFineThreads, 0, st, entries, table.start, table.chunk_base, P.n_regions, P.reg_w, gw, gh,
                                   tile_start, tickets + rm::kMaxPasses, fine_look, digit_total,
                                   (uint32_t)n_keys, sorted_idx));
  }
  return RM_OK;
}

unsigned rm_bounds_status_binning() { return rm_take_bounds_status(); }

// Checked build: which kinds of look-back words have been counted by waiting blocks since the last call, else 0.
unsigned rm_take_recounted() {
  unsigned v = 0;
#ifdef RM_BOUNDS_CHECK
  const unsigned z = 0;
  cudaDeviceSynchronize();
  cudaMemcpyFromSymbol(&v, rm::g_recounted, sizeof(v));
  cudaMemcpyToSymbol(rm::g_recounted, &z, sizeof(z));
#endif
  return v;
}
