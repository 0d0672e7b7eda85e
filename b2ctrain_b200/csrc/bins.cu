// From depth-ordered splats to per-tile fragment lists, in two levels. Reference semantics: the emission, the tile sort and
// the ranges of bin_and_sort (src/gpu/binning.cu:16-105,117-145): every (tile, splat) pair the exact ellipse test keeps,
// grouped by tile, in depth order inside a tile.
//
// A splat touches tens of tiles, and sorting its (tile, splat) pairs moves 48 bytes a pair and needs one place to do the
// ellipse tests, whose number varies from 1 to thousands a splat. Here the image is divided into BINS of 8x8 tiles. Level 1
// distributes the splats over the bins their boxes overlap (two to five pairs a splat), in depth order; level 2 takes the
// pairs of a bin 256 at a time, tests each splat against the at most 64 tiles of the bin, and writes the hits straight to
// their places. Both levels are a stable counting distribution: count, scan, write; no block ever waits for another, and
// all counts stay on the device.
//   level 1  bin_count    a block per run of depth ranks counts its pairs per bin
//            bin_rows     per bin: scan over the blocks; the last block to finish lays out the bins and cuts them into items
//            bin_scatter  the same blocks write their pairs (splat indices) to their places
//   level 2  item_count   ellipse tests of an item's pairs -> 64-bit hit words, hits per tile
//            item_columns per bin and tile: scan over the bin's items
//            tile_scan    scan over the tiles, row-major -> ranges
//            item_emit    the item's hits to their tiles' lists
// A box that lies in one depth chunk of a view (b2k_render_chunked) skips tiles whose pixels have all saturated: the
// compositing kernel clears their bits in one 64-bit word per bin.
//
// Bound by instruction issue (ellipse tests, bit work) and by launch latency in small views. Against emission of expanded
// pairs and two radix passes over them, sum of the stage's kernels per view: 4K, 6M splats, 37.5M hits 2,660 -> 870 us;
// 1080p, 500k splats, 4.4M hits 330 -> 150; 1024x1024, 1M splats of which a tenth cover hundreds of tiles 1,350 -> 390.
// Inside that, the tests of a warp's 32 pairs shared out by tile row (not a pair per lane): 455 -> 286 us at 4K.
#include "bins.cuh"
#include <algorithm>

namespace b2k {
namespace {

constexpr int L1_THREADS = 256, L1_WARPS = L1_THREADS / 32;
constexpr int SERIAL_BINS = 12;               // a splat over more bins is spread by its whole warp (4K view: 8 -> 12 takes 360 + 338 to 264 + 204 us)
static_assert((size_t)MAX_ITEMS * BIN_TILES <= BINS_TABLE_WORDS, "the counts of the items take the place of level 1's table");
static_assert(MAX_BINS * BIN_TILES / SCAN_TILES <= BINS_SEGMENTS, "one sum per tile_scan block");

__device__ __forceinline__ uint32_t run_len(uint32_t n, uint32_t blocks) {
  const uint32_t per = (n + blocks - 1) / blocks;
  return (per + L1_THREADS - 1) / L1_THREADS * L1_THREADS;
}

// The bins a splat's box overlaps, inside the band.
struct BinSpan { int bx0, by0, w, h, count; };
__device__ __forceinline__ BinSpan span_of(const Box& b, const Band& g) {
  BinSpan s{0, 0, 0, 0, 0};
  if (b.x1 <= b.x0 || b.y1 <= b.y0) return s;
  const int by0 = max(b.y0 / BIN_W, g.bin_row0), by1 = min((b.y1 - 1) / BIN_W + 1, g.bin_row0 + g.bin_rows);
  s.bx0 = b.x0 / BIN_W; s.by0 = by0; s.w = (b.x1 - 1) / BIN_W + 1 - s.bx0;
  s.h = max(by1 - by0, 0);
  s.count = s.w * s.h;
  return s;
}

// Where level 1's pairs lie. A view has fewer pairs than hits as a rule, but a long needle's box overlaps many bins without a hit,
// and a chunk does not test them: pairs may be more than the lists have room for although the hits are not. Up to `cap` they lie
// in the first buffer, and the second and third keep their hit words. More of them, up to ROOM times the lists' room, go on into
// those; then no hit words are kept (S_KEPT) and the emission makes the tests again. Still more do not fit, and their number is reported.
constexpr uint32_t ROOM = 3;
struct Pairs {
  uint32_t *first, *lo, *hi; uint32_t cap;   // cap: entries of each buffer
  __host__ __device__ __forceinline__ uint32_t room() const { return (uint32_t)((unsigned long long)cap * ROOM < 0xFFFF0000ull ? (unsigned long long)cap * ROOM : cap > 0xFFFF0000u ? cap : 0xFFFF0000u); }
  __device__ __forceinline__ uint32_t* at(uint32_t p) const { return p < cap ? first + p : p - cap < cap ? lo + (p - cap) : hi + (p - cap - cap); }   // p < room()
};

// One rank's splat as level 1 sees it.
struct Rank { uint32_t splat, tiles; uint4 hi; Box box; BinSpan span; };
// Walks a list of splats (list(p) for p in [begin, end)) in rounds of blockDim.x, the dependent loads (list entry, then the splat's
// record) one and two rounds ahead of their use.
template <bool WHOLE, class List>
struct RankReader {
  const View& v; const Band& g; const List& list; uint64_t at, end;
  uint32_t i1 = 0u, i2 = 0u, t1 = 0u;
  uint4 h1 = make_uint4(0u, 0u, 0u, 0u);
  __device__ __forceinline__ RankReader(const View& v_, const Band& g_, const List& list_, uint64_t begin, uint64_t end_) : v(v_), g(g_), list(list_), at(begin + threadIdx.x), end(end_) {
    i1 = entry(at); i2 = entry(at + blockDim.x);
    record(at);
  }
  __device__ __forceinline__ uint32_t entry(uint64_t p) const { return p < end ? list(p) : 0u; }
  __device__ __forceinline__ void record(uint64_t p) {
    const bool valid = p < end;
    h1 = valid ? v.hit_info[i1] : make_uint4(0u, 0u, 0u, 0u);
    if (WHOLE) t1 = valid ? v.tile_count[i1] : 0u;
  }
  __device__ __forceinline__ Rank next() {
    Rank k;
    k.splat = i1; k.tiles = t1; k.hi = h1;
    at += blockDim.x;
    i1 = i2;
    record(at);
    i2 = entry(at + blockDim.x);
    if (WHOLE && k.tiles == 0u) k.hi = make_uint4(0u, 0u, 0u, 0u);
    k.box = box_of(k.hi);
    k.span = span_of(k.box, g);
    return k;
  }
};
// Whether a splat goes into bin (bx, by): a chunk asks for a tile of the box that is still alive; the whole view for a hit
// tile, except that a large box takes every bin it overlaps (level 2 finds out) and a box inside one bin has a hit there.
template <bool WHOLE>
__device__ __forceinline__ bool takes_bin(const unsigned long long* s_alive, const uint4& hi, const Box& b, int bx, int by, int bin, int count) {
  if constexpr (WHOLE) return count == 1 || hi.z == 0xFFFFFFFFu || mask_bits(hi, b, bx, by) != 0ull;
  else return (s_alive[bin] & rect_bits(b, bx, by)) != 0ull;   // (looking for all-alive and all-dead bins first measured slower: 204 -> 238 us)
}
// The band's alive words, in shared memory.
__device__ __forceinline__ void load_alive(const View& v, const Band& g, unsigned long long* s_alive) {
  for (int i = threadIdx.x; i < band_bins(g); i += blockDim.x) s_alive[i] = v.alive ? v.alive[g.bin_row0 * g.bins_x + i] : ~0ull;
}
// Running sums over the band's bins that hold a live tile, (bins_x + 1) to a row: any rectangle of bins is counted in four reads.
// In the later chunks most splats lie behind saturated bins only, and would otherwise ask each bin in turn (1M large splats on
// 1024x1024 in four chunks: bin_count 98 -> 49 us a view; 6M small ones on 4K 245 -> 236).
inline size_t live_sums_bytes(const Band& g) { return ((size_t)(g.bins_x + 1) * (g.bin_rows + 1) * sizeof(uint16_t) + 15) / 16 * 16; }
__device__ __forceinline__ void sum_live(const Band& g, const unsigned long long* s_alive, uint16_t* s_sum) {   // synchronises
  const int tid = threadIdx.x, lane = tid & 31, pitch = g.bins_x + 1;
  for (int x = tid; x < pitch; x += blockDim.x) s_sum[x] = 0;
  for (int y = tid >> 5; y < g.bin_rows; y += blockDim.x >> 5) {
    uint16_t* row = s_sum + (y + 1) * pitch;
    uint32_t at = 0;
    if (lane == 0) row[0] = 0;
    for (int x0 = 0; x0 < g.bins_x; x0 += 32) {
      const uint32_t m = __ballot_sync(FULL, x0 + lane < g.bins_x && s_alive[y * g.bins_x + x0 + lane] != 0ull);
      if (x0 + lane < g.bins_x) row[x0 + lane + 1] = (uint16_t)(at + __popc(m & (0xFFFFFFFFu >> (31 - lane))));
      at += __popc(m);
    }
  }
  __syncthreads();
  for (int x = tid; x < pitch; x += blockDim.x) {
    uint32_t at = 0;
    for (int y = 1; y <= g.bin_rows; y++) { at += s_sum[y * pitch + x]; s_sum[y * pitch + x] = (uint16_t)at; }
  }
  __syncthreads();
}
__device__ __forceinline__ bool any_live(const Band& g, const uint16_t* s_sum, const BinSpan& s) {
  const int pitch = g.bins_x + 1;
  const uint16_t *top = s_sum + (s.by0 - g.bin_row0) * pitch + s.bx0, *bottom = top + s.h * pitch;
  return (int)bottom[s.w] - (int)bottom[0] - (int)top[s.w] + (int)top[0] != 0;
}
// The few bins of a lane's own splat that it goes into, as bits in the order of its span; zero for a wide splat.
template <bool WHOLE>
__device__ __forceinline__ uint32_t own_bins(const unsigned long long* s_alive, const Band& g, const Rank& k) {
  uint32_t take = 0u;
  if (k.span.count <= SERIAL_BINS) {
    int bx = k.span.bx0, by = k.span.by0;
    for (int c = 0; c < k.span.count; c++) {
      if (takes_bin<WHOLE>(s_alive, k.hi, k.box, bx, by, (by - g.bin_row0) * g.bins_x + bx, k.span.count)) take |= 1u << c;
      if (++bx == k.span.bx0 + k.span.w) { bx = k.span.bx0; by++; }
    }
  }
  return take;
}
__device__ __forceinline__ int own_bin(const Band& g, const Rank& k, int c) {
  const int dy = c / k.span.w;
  return (k.span.by0 + dy - g.bin_row0) * g.bins_x + k.span.bx0 + c - dy * k.span.w;
}
// The bins of a splat over many of them, shared out over the lanes of a warp: f(local bin). Returns whether the lane called f.
template <bool WHOLE, class F>
__device__ __forceinline__ bool spread_bins(const unsigned long long* s_alive, const Band& g, const uint4& hi, F f) {
  const Box b = box_of(hi);
  const BinSpan s = span_of(b, g);
  bool any = false;
  for (int c = threadIdx.x & 31; c < s.count; c += 32) {
    const int dy = c / s.w, bx = s.bx0 + c - dy * s.w, by = s.by0 + dy, bin = (by - g.bin_row0) * g.bins_x + bx;
    if (takes_bin<WHOLE>(s_alive, hi, b, bx, by, bin, s.count)) { any = true; f(bin); }
  }
  return any;
}
// Splats over many bins are spread by the whole warp, one after the other: f(lane of the splat, splat, local bin) for every
// bin. All lanes call this together; returns whether this lane's own splat is wide and went into any bin.
template <bool WHOLE, class F>
__device__ __forceinline__ bool wide_bins(const unsigned long long* s_alive, const Band& g, const Rank& k, F f) {
  const int lane = threadIdx.x & 31;
  bool took = false;
  for (uint32_t wide = __ballot_sync(FULL, k.span.count > SERIAL_BINS); wide; wide &= wide - 1u) {
    const int src = __ffs(wide) - 1;
    uint4 hi;
    hi.x = __shfl_sync(FULL, k.hi.x, src); hi.y = __shfl_sync(FULL, k.hi.y, src); hi.z = __shfl_sync(FULL, k.hi.z, src); hi.w = __shfl_sync(FULL, k.hi.w, src);
    const uint32_t splat = __shfl_sync(FULL, k.splat, src);
    const bool any = __any_sync(FULL, spread_bins<WHOLE>(s_alive, g, hi, [&](int bin) { f(src, splat, bin); }));
    if (lane == src) took = any;
  }
  return took;
}

// ---- level 1 -----------------------------------------------------------------------------------------------------------

// Pairs per bin of each block's run of ranks. Each warp takes a part of the run by itself. A chunk also leaves the part's splats that go
// anywhere, in order, at the part's place in `live`, and their number in live_counts: in the later chunks most splats lie behind
// saturated tiles, and the write pass never looks at them. (With one list a block, the block met after every 512 ranks and every warp
// added up the warps before it: 478 instructions for 32 ranks, nearly all dead, in the last chunk of a 4K view of 6M splats: 130 us, now 64.)
// The whole view leaves the run's tile count instead (tile_off is its running sum).
constexpr int COUNT_THREADS = 512, PARTS = COUNT_THREADS / 32;
__device__ __forceinline__ uint32_t part_len(uint32_t run) { return (run + COUNT_THREADS - 1) / COUNT_THREADS * 32; }
template <bool WHOLE>
__global__ void __launch_bounds__(COUNT_THREADS) bin_count_kernel(View v, Band g, Tables t, uint32_t* __restrict__ live) {
  after_previous();
  extern __shared__ __align__(16) unsigned long long s_alive[];   // [bins], then [bins] counts
  const int bins = band_bins(g), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(s_alive + (WHOLE ? 0 : bins));
  uint16_t* s_sum = reinterpret_cast<uint16_t*>(s_cnt + bins);   // of a chunk behind the first
  __shared__ uint32_t s_warp[32];
  for (int i = tid; i < bins; i += COUNT_THREADS) s_cnt[i] = 0u;
  if (!WHOLE) load_alive(v, g, s_alive);
  if (blockIdx.x == 0 && tid == 0) {    // this band's counters; the view's with its first band
    t.st[S_DONE_ROWS] = 0u; t.st[S_DONE_TILES] = 0u;
    if (v.first_band) { t.st[S_SLOT] = v.words ? v.words[CW_BASE + v.chunk] : 0u; if (!v.words || v.chunk == 0) t.st[S_OVER] = 0u; if (!v.words) *t.longest = 0u; }
  }
  __syncthreads();
  const bool some_dead = !WHOLE && v.alive;
  if (some_dead) sum_live(g, s_alive, s_sum);
  uint32_t r0, r1;
  view_ranks(v, r0, r1);
  const uint32_t len = run_len(r1 - r0, gridDim.x), part = part_len(len);
  const uint32_t run_end = (uint32_t)min((uint64_t)r0 + (uint64_t)(blockIdx.x + 1) * len, (uint64_t)r1);
  const uint32_t begin = (uint32_t)min((uint64_t)r0 + (uint64_t)blockIdx.x * len + warp * part, (uint64_t)run_end), end = min(begin + part, run_end);
  uint32_t tiles = 0, n_live = 0, waiting = 0;
  auto count = [&](const Rank& k) {     // the bins of a warp's splats, and in a chunk the list of those that go into any
    const uint32_t take = own_bins<WHOLE>(s_alive, g, k);
    for (uint32_t b = take; b; b &= b - 1u) atomicAdd(&s_cnt[own_bin(g, k, __ffs(b) - 1)], 1u);
    const bool wide = wide_bins<WHOLE>(s_alive, g, k, [&](int, uint32_t, int bin) { atomicAdd(&s_cnt[bin], 1u); });
    if constexpr (!WHOLE) {
      const uint32_t on = __ballot_sync(FULL, take != 0u || wide);
      if ((on >> lane) & 1u) live[begin + n_live + __popc(on & ((1u << lane) - 1u))] = k.splat;
      n_live += __popc(on);
    }
  };
  __shared__ uint4 s_hit[WHOLE ? 1 : PARTS][64];
  __shared__ uint32_t s_splat[WHOLE ? 1 : PARTS][64];
  auto queued = [&](uint32_t n) {       // counts the first n of the warp's queue
    __syncwarp();
    Rank k{0u, 0u, make_uint4(0u, 0u, 0u, 0u), Box{0, 0, 0, 0}, BinSpan{0, 0, 0, 0, 0}};
    const int w = WHOLE ? 0 : warp;
    if ((uint32_t)lane < n) { k.splat = s_splat[w][lane]; k.hi = s_hit[w][lane]; }
    k.box = box_of(k.hi); k.span = span_of(k.box, g);
    count(k);
  };
  constexpr int PER = 2;                // ranks of a lane on their way together
  uint32_t next[PER];
#pragma unroll
  for (int u = 0; u < PER; u++) next[u] = begin + u * 32 + lane < end ? v.order[begin + u * 32 + lane] : 0u;
  for (uint32_t at = begin; at < end; at += 32 * PER) {
    Rank k[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) {
      const bool valid = at + u * 32 + lane < end;
      k[u].splat = next[u];
      k[u].hi = valid ? v.hit_info[next[u]] : make_uint4(0u, 0u, 0u, 0u);
      k[u].tiles = WHOLE && valid ? v.tile_count[next[u]] : 0u;
    }
#pragma unroll
    for (int u = 0; u < PER; u++) { const uint32_t p = at + (PER + u) * 32 + lane; next[u] = p < end ? v.order[p] : 0u; }
#pragma unroll
    for (int u = 0; u < PER; u++) {
      if (WHOLE && k[u].tiles == 0u) k[u].hi = make_uint4(0u, 0u, 0u, 0u);
      tiles += k[u].tiles;
      k[u].box = box_of(k[u].hi);
      k[u].span = span_of(k[u].box, g);
      if (!some_dead) { count(k[u]); continue; }
      // Behind the first chunks few splats overlap a bin that holds a live tile. They wait in shared memory until there are a warp's
      // worth of them: with one here and there, nearly every warp went through the bins for a lane or two.
      const bool in = k[u].span.count != 0 && any_live(g, s_sum, k[u].span);
      const uint32_t m = __ballot_sync(FULL, in);
      if (m == 0u) continue;
      const int w = WHOLE ? 0 : warp;
      if (in) { const uint32_t q = waiting + __popc(m & ((1u << lane) - 1u)); s_splat[w][q] = k[u].splat; s_hit[w][q] = k[u].hi; }
      waiting += __popc(m);
      if (waiting >= 32u) {
        queued(32u);
        waiting -= 32u;
        __syncwarp();
        const bool rest = (uint32_t)lane < waiting;
        const uint32_t i = rest ? s_splat[w][32 + lane] : 0u;
        const uint4 h = rest ? s_hit[w][32 + lane] : make_uint4(0u, 0u, 0u, 0u);
        if (rest) { s_splat[w][lane] = i; s_hit[w][lane] = h; }
        __syncwarp();                   // the next to wait may be put where another lane has just read
      }
    }
  }
  if (waiting) queued(waiting);
  __syncthreads();
  for (int i = tid; i < bins; i += COUNT_THREADS) t.cells[(size_t)i * gridDim.x + blockIdx.x] = s_cnt[i];
  if (!WHOLE) {
    if (lane == 0) t.live_counts[blockIdx.x * PARTS + warp] = n_live;
  } else if (v.first_band) {
    uint32_t total;
    block_scan(tiles, s_warp, total);
    if (tid == 0) t.block_sums[blockIdx.x] = total;
  }
}

// A warp per bin turns the bin's counts into offsets. The last block to finish lays out the band: first pair of every bin,
// and the items (runs of pairs of one bin) that level 2 works on. An item is 256 pairs unless that made too many. The band's pairs
// are added up in 64 bits: two million splats over a whole 4K image make more than 2^32, and a sum that wrapped around would
// give items that are too short, and more of them than there is room for.
constexpr int ROWS_THREADS = 512, ROWS_BINS = ROWS_THREADS / 32, ROWS_PER = 16;   // at most 32 * ROWS_PER blocks of level 1
__global__ void __launch_bounds__(ROWS_THREADS) bin_rows_kernel(int blocks, int bins, uint32_t cap, uint32_t room_pairs, Tables t) {
  after_previous();
  __shared__ uint32_t s_warp[32];
  __shared__ unsigned long long s_sums[32];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, bin = blockIdx.x * ROWS_BINS + (tid >> 5);
  if (bin < bins) {
    uint32_t* row = t.cells + (size_t)bin * blocks;
    uint32_t c[ROWS_PER], at = 0;
#pragma unroll
    for (int u = 0; u < ROWS_PER; u++) { const int k = u * 32 + lane; c[u] = k < blocks ? row[k] : 0u; }
#pragma unroll
    for (int u = 0; u < ROWS_PER; u++) {
      if (u * 32 >= blocks) break;
      uint32_t incl = c[u];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { const uint32_t x = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += x; }
      if (u * 32 + lane < blocks) row[u * 32 + lane] = at + incl - c[u];
      at += __shfl_sync(FULL, incl, 31);
    }
    if (lane == 0) t.totals[bin] = at;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(t.st + S_DONE_ROWS, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  constexpr int PER = MAX_BINS / ROWS_THREADS;
  uint32_t tot[PER];
  unsigned long long sum = 0, pairs;
#pragma unroll
  for (int u = 0; u < PER; u++) { const int b = tid * PER + u; tot[u] = b < bins ? __ldcg(t.totals + b) : 0u; sum += tot[u]; }
  unsigned long long at = block_scan(sum, s_sums, pairs) - sum;
  const uint32_t room = MAX_ITEMS - (uint32_t)bins, len = 256u * (uint32_t)(pairs / (256u * room) + 1u);   // items <= pairs / len + bins <= MAX_ITEMS
  uint32_t items = 0, n_items;
#pragma unroll
  for (int u = 0; u < PER; u++) items += (tot[u] + len - 1u) / len;
  uint32_t it = block_scan(items, s_warp, n_items) - items;
  const bool kept = pairs <= cap || pairs > room_pairs;   // the last: a view that does not fit, cut short
  auto in_room = [&](unsigned long long p) { return (uint32_t)(p < room_pairs ? p : room_pairs); };   // pairs beyond the buffers are not written
#pragma unroll
  for (int u = 0; u < PER; u++) {
    const int b = tid * PER + u;
    if (b < bins) { t.base[b] = in_room(at); t.first_item[b] = it; }
    at += tot[u]; it += (tot[u] + len - 1u) / len;
  }
  if (tid == 0) {
    const uint32_t total = (uint32_t)(pairs < 0xFFFFFFFFull ? pairs : 0xFFFFFFFFull);
    t.base[bins] = in_room(pairs); t.first_item[bins] = n_items;
    t.st[S_PAIRS] = total; t.st[S_ITEMS] = n_items; t.st[S_ITEM_LEN] = len; t.st[S_KEPT] = kept ? 1u : 0u;
    if (total > room_pairs && total > t.st[S_OVER]) t.st[S_OVER] = total;   // level 1's own pairs did not fit: the caller grows the buffers
  }
  if (tid < BINS_SEGMENTS) t.segments[tid] = 0u;
}

// The pairs to their places, stable: bit l of s_bits[bin][w] says that lane l of warp w adds a pair to the bin in this round.
// The splat that adds a bin's first pair of the round afterwards moves the bin's place on and clears its bits.
template <bool WHOLE>
__global__ void __launch_bounds__(L1_THREADS) bin_scatter_kernel(View v, Band g, Tables t, Pairs pr, const uint32_t* __restrict__ live,
                                                                 uint32_t* __restrict__ tile_off) {
  after_previous();
  extern __shared__ __align__(16) uint32_t s_bits[];   // [bins][8], then [bins] alive words, then [bins] next free place
  const int bins = band_bins(g), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned long long* s_alive = reinterpret_cast<unsigned long long*>(s_bits + (size_t)bins * L1_WARPS);
  uint32_t* s_next = reinterpret_cast<uint32_t*>(s_alive + (WHOLE ? 0 : bins));
  __shared__ uint32_t s_warp[32], s_wides;
  __shared__ uint4 s_wide[L1_THREADS];
  __shared__ uint2 s_wide_of[L1_THREADS];     // splat, thread
  uint32_t r0, r1;
  view_ranks(v, r0, r1);
  const uint32_t len = run_len(r1 - r0, gridDim.x);
  // The run's ranks, or of a chunk the live splats that the warps of bin_count have listed part by part.
  const uint64_t run = (uint64_t)r0 + (uint64_t)blockIdx.x * len;
  __shared__ uint32_t s_part[PARTS + 1];      // entries of the parts before
  if (!WHOLE) {
    if (warp == 0) {
      const uint32_t c = lane < PARTS ? t.live_counts[blockIdx.x * PARTS + lane] : 0u;
      uint32_t incl = c;
#pragma unroll
      for (int o = 1; o < PARTS; o <<= 1) { const uint32_t u = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += u; }
      if (lane < PARTS) s_part[lane + 1] = incl;
      if (lane == 0) s_part[0] = 0u;
    }
    __syncthreads();
  }
  const uint64_t begin = WHOLE ? run : 0u, end = WHOLE ? (run + len < (uint64_t)r1 ? run + len : (uint64_t)r1) : s_part[PARTS];
  auto list = [&](uint64_t p) -> uint32_t {
    if constexpr (WHOLE) return v.order[p];
    uint32_t k = 0;                           // the part that holds entry p
#pragma unroll
    for (uint32_t step = PARTS / 2; step > 0; step >>= 1) k += s_part[k + step] <= p ? step : 0u;
    return live[run + k * part_len(len) + (p - s_part[k])];
  };
  const bool offsets = WHOLE && v.first_band;
  const uint32_t room = pr.room();
  for (int b = blockIdx.x * L1_WARPS + warp; b < bins; b += gridDim.x * L1_WARPS) {   // the items' bins, a warp per bin
    const uint32_t e = t.first_item[b + 1];
    for (uint32_t k = t.first_item[b] + (uint32_t)lane; k < e; k += 32) t.item_bin[k] = (uint32_t)b;
  }
  if (begin >= end && !(offsets && blockIdx.x == gridDim.x - 1)) return;
  for (int i = tid; i < bins * L1_WARPS; i += L1_THREADS) s_bits[i] = 0u;
  if (tid == 0) s_wides = 0u;
  for (int i = tid; i < bins; i += L1_THREADS) s_next[i] = (uint32_t)min((unsigned long long)t.base[i] + t.cells[(size_t)i * gridDim.x + blockIdx.x], (unsigned long long)room);
  if (!WHOLE) load_alive(v, g, s_alive);
  uint32_t tiles_before = 0;
  if (offsets) {
    uint32_t mine = 0, total;
    for (int b = tid; b < (int)blockIdx.x; b += L1_THREADS) mine += t.block_sums[b];
    block_scan(mine, s_warp, total);
    tiles_before = total;
  }
  __syncthreads();
  auto earlier = [&](int bin, int of_warp, int l) {   // pairs of this round before lane l of a warp
    const uint4* b4 = reinterpret_cast<const uint4*>(s_bits + bin * L1_WARPS);
    const uint4 a = b4[0], b = b4[1];
    const uint32_t w[L1_WARPS] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t n = 0;
#pragma unroll
    for (int k = 0; k < L1_WARPS; k++) n += (uint32_t)__popc(k < of_warp ? w[k] : k == of_warp ? w[k] & ((1u << l) - 1u) : 0u);
    return n;
  };
  auto move_on = [&](int bin) {
    uint4* b4 = reinterpret_cast<uint4*>(s_bits + bin * L1_WARPS);
    const uint4 a = b4[0], b = b4[1];
    const uint32_t added = __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w) + __popc(b.x) + __popc(b.y) + __popc(b.z) + __popc(b.w);
    if (added) { s_next[bin] += added; b4[0] = make_uint4(0u, 0u, 0u, 0u); b4[1] = make_uint4(0u, 0u, 0u, 0u); }
  };
  auto spread = [&](auto put) {
    RankReader<WHOLE, decltype(list)> ranks(v, g, list, begin, end);
    for (uint64_t at = begin; at < end; at += L1_THREADS) {
      const Rank k = ranks.next();
      const uint32_t take = own_bins<WHOLE>(s_alive, g, k);
      for (uint32_t b = take; b; b &= b - 1u) atomicOr(&s_bits[own_bin(g, k, __ffs(b) - 1) * L1_WARPS + warp], 1u << lane);
      // Splats over many bins are listed, and the block's warps share them: behind the first chunks they are most of what is left, and with
      // each to its own warp a few warps spread thirty while the others wait.
      const bool wide = k.span.count > SERIAL_BINS;
      if (wide) { const uint32_t at = atomicAdd(&s_wides, 1u); s_wide[at] = k.hi; s_wide_of[at] = make_uint2(k.splat, (uint32_t)tid); }
      if (offsets) {
        uint32_t total;
        const uint32_t incl = block_scan(k.tiles, s_warp, total);
        if (at + tid < end) tile_off[at + tid] = tiles_before + incl;
        tiles_before += total;
      }
      const bool any_wide = __syncthreads_or(wide);
      const uint32_t wides = any_wide ? s_wides : 0u;
      if (any_wide) {
        for (uint32_t e = warp; e < wides; e += L1_WARPS) {
          const uint32_t of = s_wide_of[e].y;
          spread_bins<WHOLE>(s_alive, g, s_wide[e], [&](int bin) { atomicOr(&s_bits[bin * L1_WARPS + (of >> 5)], 1u << (of & 31u)); });
        }
        __syncthreads();
        if (tid == 0) s_wides = 0u;
      }
      uint32_t first = 0u;
      for (uint32_t b = take; b; b &= b - 1u) {
        const int bin = own_bin(g, k, __ffs(b) - 1);
        const uint32_t n = earlier(bin, warp, lane), pos = s_next[bin] + n;
        put(pos, k.splat);
        if (n == 0u) first |= b & (0u - b);
      }
      for (uint32_t e = warp; e < wides; e += L1_WARPS) {
        const uint2 of = s_wide_of[e];
        spread_bins<WHOLE>(s_alive, g, s_wide[e], [&](int bin) { put(s_next[bin] + earlier(bin, (int)(of.y >> 5), (int)(of.y & 31u)), of.x); });
      }
      __syncthreads();
      if (any_wide) { for (int i = tid; i < bins; i += L1_THREADS) move_on(i); }
      else { for (uint32_t b = first; b; b &= b - 1u) move_on(own_bin(g, k, __ffs(b) - 1)); }
      __syncthreads();
    }
  };
  // (one of two loops: a test of the place against both limits inside it, and the kernel takes 42 us for 39)
  if (t.st[S_KEPT]) spread([&](uint32_t pos, uint32_t splat) { if (pos < pr.cap) pr.first[pos] = splat; });
  else spread([&](uint32_t pos, uint32_t splat) { if (pos < room) *pr.at(pos) = splat; });
  if (offsets && blockIdx.x == gridDim.x - 1 && tid == 0) t.st[S_TOTAL] = tiles_before;   // the view's hits, also when the pairs did not fit
}

// ---- level 2 -----------------------------------------------------------------------------------------------------------

// The pairs of one item and the bin's corner.
struct Item { uint32_t first, end; int bx, by; };
__device__ __forceinline__ Item item_of(const Tables& t, const Band& g, uint32_t it, uint32_t limit) {
  const uint32_t bin = t.item_bin[it], len = t.st[S_ITEM_LEN];
  Item m;
  const unsigned long long first = t.base[bin] + (unsigned long long)(it - t.first_item[bin]) * len;
  m.first = (uint32_t)min(first, (unsigned long long)limit);
  m.end = (uint32_t)min(first + len, (unsigned long long)min(t.base[bin + 1], limit));
  m.bx = (int)bin % g.bins_x; m.by = g.bin_row0 + (int)bin / g.bins_x;
  return m;
}

// Hit word of every pair of an item (bit = row * 8 + column of the tile in its bin), and the item's hits per tile.
template <bool WHOLE>
__global__ void __launch_bounds__(L2_THREADS) item_count_kernel(View v, Band g, Tables t, Pairs pr) {
  after_previous();
  __shared__ WarpShare s_share[L2_WARPS];
  __shared__ uint32_t s_cnt[L2_WARPS][BIN_TILES];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  WarpShare& ws = s_share[warp];
  const uint32_t n_items = t.st[S_ITEMS];
  const bool kept = t.st[S_KEPT] != 0u;
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const Item m = item_of(t, g, it, kept ? pr.cap : pr.room());
    const unsigned long long alive = !WHOLE && v.alive ? v.alive[m.by * g.bins_x + m.bx] : ~0ull;
    uint32_t c_lo = 0, c_hi = 0;   // this warp's hits on tiles `lane` and `lane + 32`
    for (uint32_t p0 = m.first; p0 < m.end; p0 += L2_THREADS) {
      const uint32_t p = p0 + tid;
      unsigned long long hits = 0ull, todo = 0ull;   // todo: tiles to test
      if (p < m.end) {
        const uint32_t i = kept ? pr.first[p] : *pr.at(p);
        const uint4 hi = v.hit_info[i];
        const Box b = box_of(hi);
        if (WHOLE && hi.z != 0xFFFFFFFFu) {
          hits = mask_bits(hi, b, m.bx, m.by);   // the projection has tested this box
        } else {
          todo = rect_bits(b, m.bx, m.by) & alive;
          const float4 q0 = v.proj0[i], q1 = v.proj1[i];
          share_record(ws, q0, q1);
        }
      }
      hits |= shared_tests(ws, todo, m.bx, m.by);
      if (kept && p < m.end) { pr.lo[p] = (uint32_t)hits; pr.hi[p] = (uint32_t)(hits >> 32); }
      c_lo += __popc(transpose_bits((uint32_t)hits)); c_hi += __popc(transpose_bits((uint32_t)(hits >> 32)));
    }
    s_cnt[warp][lane] = c_lo; s_cnt[warp][lane + 32] = c_hi;
    __syncthreads();
    if (tid < BIN_TILES) {
      uint32_t sum = 0;
#pragma unroll
      for (int w = 0; w < L2_WARPS; w++) sum += s_cnt[w][tid];
      t.cells[(size_t)it * BIN_TILES + tid] = sum;
    }
    __syncthreads();
  }
}

// A block per bin: the counts of its items become offsets inside each tile, the totals go to the tiles (ranges[tile].x until
// tile_scan has run) and to the sums of tile_scan's blocks. Groups of 64 threads share a column: sixteen where few bins have long ones,
// four where there are bins enough to fill the GPU (74 -> 29 us over the five chunks of a 4K view).
template <int COL_GROUPS>
__global__ void __launch_bounds__(COL_GROUPS * BIN_TILES) item_columns_kernel(Band g, Tables t, uint2* __restrict__ ranges) {
  after_previous();
  __shared__ uint32_t s_sum[COL_GROUPS][BIN_TILES];
  const int bin = blockIdx.x, tile = threadIdx.x % BIN_TILES, group = threadIdx.x / BIN_TILES;
  const uint32_t i0 = t.first_item[bin], i1 = t.first_item[bin + 1], per = (i1 - i0 + COL_GROUPS - 1) / COL_GROUPS;
  const uint32_t a = min(i0 + group * per, i1), b = min(a + per, i1);
  uint32_t* col = t.cells + tile;
  uint32_t sum = 0;
#pragma unroll 8
  for (uint32_t k = a; k < b; k++) sum += col[(size_t)k * BIN_TILES];
  s_sum[group][tile] = sum;
  __syncthreads();
  uint32_t at = 0, total = 0;
#pragma unroll
  for (int k = 0; k < COL_GROUPS; k++) { const uint32_t s = s_sum[k][tile]; if (k < group) at += s; total += s; }
#pragma unroll 8
  for (uint32_t k = a; k < b; k++) { const uint32_t c = col[(size_t)k * BIN_TILES]; col[(size_t)k * BIN_TILES] = at; at += c; }
  if (group != 0) return;   // two whole warps are left
  const int bx = bin % g.bins_x, by = g.bin_row0 + bin / g.bins_x, x = bx * BIN_W + (tile & 7), y = by * BIN_W + (tile >> 3);
  const bool valid = x < g.tiles_x && y < g.tiles_y;
  const int id = y * g.tiles_x + x;
  if (valid) ranges[id] = make_uint2(total, 0u);
  // One reduction for the warp's tiles of a segment, nearly always all of them: with one for every tile a thousand met in a word (1024x1024
  // over 1M heavy splats, first chunk: 12 -> 3.4 us, and the wait of the scan behind it 12 -> 4.3).
  int segment = valid && total ? (id - g.bin_row0 * BIN_W * g.tiles_x) / SCAN_TILES : BINS_SEGMENTS;
  for (int s = __reduce_min_sync(FULL, segment); s < BINS_SEGMENTS; s = __reduce_min_sync(FULL, segment)) {
    const uint32_t sum_of = __reduce_add_sync(FULL, segment == s ? total : 0u);
    if ((threadIdx.x & 31) == 0) atomicAdd(t.segments + s, sum_of);
    if (segment == s) segment = BINS_SEGMENTS;
  }
}

// Ranges of the band's tiles, row-major: block b starts behind the hits of the blocks before it. Empty tiles get (0, 0);
// ranges end with the buffers. The last block to finish moves the view's slot on. All loads are issued before the one
// scan of the block (two scans one after the other and a fence took 5.4 to 7.8 us, this 2.8 to 5.8).
__global__ void __launch_bounds__(SCAN_TILES) tile_scan_kernel(View v, Band g, Tables t, uint32_t cap, uint2* __restrict__ ranges, uint32_t* __restrict__ num_isect,
                                                               uint32_t* __restrict__ list) {
  after_previous();
  __shared__ uint32_t s_warp[32], s_longest[32], s_slot;
  const int tid = threadIdx.x, lane = tid & 31;
  const int tile0 = g.bin_row0 * BIN_W * g.tiles_x, tiles = (min((g.bin_row0 + g.bin_rows) * BIN_W, g.tiles_y) - g.bin_row0 * BIN_W) * g.tiles_x;
  const int mine = blockIdx.x * SCAN_TILES + tid;
  const uint32_t c = mine < tiles ? ranges[tile0 + mine].x : 0u;
  if (tid == 0) s_slot = t.st[S_SLOT];
  { const uint32_t m = __reduce_max_sync(FULL, c); if (lane == 0) s_longest[tid >> 5] = m; }
  uint32_t all = 0, before = 0;   // hits of the band, and of the blocks before this one: every warp adds them up for itself
  {
    uint32_t seg[BINS_SEGMENTS / 32];
#pragma unroll
    for (int u = 0; u < BINS_SEGMENTS / 32; u++) seg[u] = u * 32 + lane < (int)gridDim.x ? t.segments[u * 32 + lane] : 0u;
#pragma unroll
    for (int u = 0; u < BINS_SEGMENTS / 32; u++) { all += seg[u]; before += u * 32 + lane < (int)blockIdx.x ? seg[u] : 0u; }
    all = __reduce_add_sync(FULL, all); before = __reduce_add_sync(FULL, before);
  }
  uint32_t total;
  const uint32_t in_block = block_scan(c, s_warp, total) - c, slot = s_slot, start = slot + before + in_block;
  if (mine < tiles) ranges[tile0 + mine] = c ? make_uint2(min(start, cap), min(start + c, cap)) : make_uint2(0u, 0u);
  if (tid < 32) { const uint32_t m = __reduce_max_sync(FULL, s_longest[lane]); if (lane == 0 && m) atomicMax(t.longest, m); }
  if (list) {   // the chunk's tiles with a list, for the compositing: long lists from the start, short ones from the end
    const uint32_t longs = __ballot_sync(FULL, c >= LONG_LIST), shorts = __ballot_sync(FULL, c > 0u && c < LONG_LIST), lane_lt = (1u << lane) - 1u;
    uint32_t at_long = 0u, at_short = 0u;
    if (lane == 0 && longs) at_long = atomicAdd(v.words + CW_LONG + v.chunk, (uint32_t)__popc(longs));
    if (lane == 1 && shorts) at_short = atomicAdd(v.words + CW_SHORT + v.chunk, (uint32_t)__popc(shorts));
    at_long = __shfl_sync(FULL, at_long, 0); at_short = __shfl_sync(FULL, at_short, 1);
    if ((longs >> lane) & 1u) list[at_long + __popc(longs & lane_lt)] = (uint32_t)(tile0 + mine);
    if ((shorts >> lane) & 1u) list[g.tiles_x * g.tiles_y - 1 - (int)(at_short + __popc(shorts & lane_lt))] = (uint32_t)(tile0 + mine);
  }
  if (tid == 0 && atomicAdd(t.st + S_DONE_TILES, 1u) == gridDim.x - 1u) {   // every block has read the slot (its first thread did)
    uint32_t end = slot + all;
    if (v.last_band) {
      if (v.words) { v.words[CW_COUNT + v.chunk] = end - v.words[CW_BASE + v.chunk]; v.words[CW_BASE + v.chunk + 1] = (end + 31u) & ~31u; }
      *num_isect = max(v.words ? end : t.st[S_TOTAL], t.st[S_OVER]);
    }
    t.st[S_SLOT] = end;
  }
}

// The hits of an item to their tiles' lists, in the order of the pairs: for each tile the warp takes the 32 pairs of one hit
// word at a time, and the lanes with a hit write side by side.
template <bool WHOLE, bool KEPT>
__device__ __forceinline__ void emit_items(const View& v, const Band& g, const Tables& t, const Pairs& pr, const uint2* __restrict__ ranges, uint32_t* __restrict__ vals,
                                           uint32_t (&s_splat)[L2_THREADS], uint32_t (&s_word)[L2_WARPS][BIN_TILES]) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lane_lt = (1u << lane) - 1u, n_items = t.st[S_ITEMS];
  const uint32_t cap = pr.cap;
  constexpr int TPW = BIN_TILES / L2_WARPS;   // tiles a warp writes
  for (uint32_t it = blockIdx.x; it < n_items; it += gridDim.x) {
    const Item m = item_of(t, g, it, KEPT ? cap : pr.room());
    uint32_t next = 0;   // lane k < TPW: next place of the warp's k-th tile
    if (lane < TPW) {
      const int tile = warp * TPW + lane, x = m.bx * BIN_W + (tile & 7), y = m.by * BIN_W + (tile >> 3);
      if (x < g.tiles_x && y < g.tiles_y) next = ranges[y * g.tiles_x + x].x + t.cells[(size_t)it * BIN_TILES + tile];
    }
    for (uint32_t p0 = m.first; p0 < m.end; p0 += L2_THREADS) {
      const uint32_t p = p0 + tid;
      const bool valid = p < m.end;
      uint32_t splat = 0u, lo = 0u, hi = 0u;
      if (valid) {
        if constexpr (KEPT) { splat = pr.first[p]; lo = pr.lo[p]; hi = pr.hi[p]; }
        else {
          splat = *pr.at(p);
          const unsigned long long hits = hits_again<WHOLE>(v, m.bx, m.by, !WHOLE && v.alive ? v.alive[m.by * g.bins_x + m.bx] : ~0ull, splat);
          lo = (uint32_t)hits; hi = (uint32_t)(hits >> 32);
        }
      }
      s_splat[tid] = splat;
      s_word[warp][lane] = transpose_bits(lo);
      s_word[warp][lane + 32] = transpose_bits(hi);
      __syncthreads();
#pragma unroll
      for (int k = 0; k < TPW; k++) {
        uint32_t pos = __shfl_sync(FULL, next, k);
#pragma unroll
        for (int w = 0; w < L2_WARPS; w++) {
          const uint32_t word = s_word[w][warp * TPW + k];
          if (word == 0u) continue;
          const uint32_t at = pos + __popc(word & lane_lt);
          if (((word >> lane) & 1u) && at < cap) vals[at] = s_splat[w * 32 + lane];
          pos += __popc(word);
        }
        if (lane == k) next = pos;
      }
      __syncthreads();
    }
  }
}
template <bool WHOLE>
__global__ void __launch_bounds__(L2_THREADS, 4) item_emit_kernel(View v, Band g, Tables t, Pairs pr, const uint2* __restrict__ ranges, uint32_t* __restrict__ vals) {
  after_previous();
  __shared__ uint32_t s_splat[L2_THREADS], s_word[L2_WARPS][BIN_TILES];
  if (t.st[S_KEPT]) emit_items<WHOLE, true>(v, g, t, pr, ranges, vals, s_splat, s_word);
  else emit_items<WHOLE, false>(v, g, t, pr, ranges, vals, s_splat, s_word);
}

// Tile ids of the sorted list, for callers of the whole-view binning: a warp per tile.
__global__ void __launch_bounds__(256) fill_keys_kernel(int n_tiles, const uint2* __restrict__ ranges, uint32_t* __restrict__ keys) {
  after_previous();
  const int lane = threadIdx.x & 31;
  for (int tile = blockIdx.x * 8 + (threadIdx.x >> 5); tile < n_tiles; tile += gridDim.x * 8) {
    const uint2 r = ranges[tile];
    for (uint32_t p = r.x + lane; p < r.y; p += 32) keys[p] = (uint32_t)tile;
  }
}

}  // namespace

// Bins the ranks of one depth chunk (words != nullptr) or of the whole view into vals_sorted and `ranges`. Level 1's pairs
// take ctx->keys, the hit words (or more pairs) ctx->vals and ctx->keys_sorted, a chunk's live splats the scratch of the depth sort.
int launch_bins(const B2kCtx* c, int n, uint32_t* words, int chunk, int lo_num, int hi_num, const unsigned long long* alive, uint32_t* tiles_out, uint32_t* tables, cudaStream_t s) {
  const Tables t = bins_tables(tables, words ? words + CW_LONGEST + chunk : c->num_isect + NI_LONGEST);
  static bool attr_set[64] = {false};
  int dev = 0;
  constexpr int smem_max = MAX_BINS * ((L1_WARPS + 1) * (int)sizeof(uint32_t) + 8);
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
    B2K_CUDA(cudaFuncSetAttribute(bin_count_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_BINS * 12 + (MAX_BINS + 1) * 4 + 16));
    B2K_CUDA(cudaFuncSetAttribute(bin_scatter_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    B2K_CUDA(cudaFuncSetAttribute(bin_scatter_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max));
    attr_set[dev] = true;
  }
  const uint32_t cap = (uint32_t)c->isect_cap;
  const Pairs pr{c->keys, c->vals, c->keys_sorted, cap};
  uint2* ranges = (uint2*)c->tile_ranges + (words ? (size_t)chunk * c->n_tiles : 0);
  const int bins_x = div_up(c->tiles_x, BIN_W), bin_rows = div_up(c->tiles_y, BIN_W);
  if (bins_x > MAX_BINS) return B2K_ERR_UNSUPPORTED;   // tile boxes hold twelve bits of a tile's column: the caller's own limit is lower
  const int rows_per_band = MAX_BINS / bins_x;
  View v{c->order, (const uint4*)c->hit_info, c->tile_count, (const float4*)c->proj0, (const float4*)c->proj1, n, words, chunk, lo_num, hi_num, alive, 0, 0};
  const long long most = words ? (long long)n * (hi_num - lo_num) / 256 + 1 : n;   // ranks
  if (!words && walks(c, n)) return launch_walk(c, v, tables, s);
  for (int row = 0; row < bin_rows; row += rows_per_band) {
    Band g{c->tiles_x, c->tiles_y, bins_x, row, std::min(rows_per_band, bin_rows - row)};
    v.first_band = row == 0; v.last_band = row + g.bin_rows == bin_rows;
    const int bins = g.bins_x * g.bin_rows;
    // Blocks of level 1: two per SM, no more than the table holds rows for, none without a rank.
    const int blocks = (int)std::max<long long>(1, std::min<long long>({2LL * sm_count(), 32LL * ROWS_PER, (long long)(BINS_TABLE_WORDS / bins), (most + L1_THREADS - 1) / L1_THREADS}));
    // Items are read on the device: a grid that fills the GPU, or what few splats can make at most.
    const int item_blocks = (int)std::min<long long>(sm_count() * 8LL, bins + most * std::min(bins, 64) / L2_THREADS);
    const int tiles = (std::min((row + g.bin_rows) * BIN_W, c->tiles_y) - row * BIN_W) * c->tiles_x;
#define L(WHOLE) do { \
    const size_t alive_bytes = WHOLE ? 0 : bins * sizeof(unsigned long long); \
    launch_next(bin_count_kernel<WHOLE>, blocks, COUNT_THREADS, alive_bytes + bins * sizeof(uint32_t) + (WHOLE ? 0 : live_sums_bytes(g)), s, v, g, t, c->depth_keys); \
    launch_next(bin_rows_kernel, div_up(bins, ROWS_BINS), ROWS_THREADS, 0, s, blocks, bins, cap, pr.room(), t); \
    launch_next(bin_scatter_kernel<WHOLE>, blocks, L1_THREADS, alive_bytes + bins * (L1_WARPS + 1) * sizeof(uint32_t), s, v, g, t, pr, c->depth_keys, c->tile_off); \
    launch_next(item_count_kernel<WHOLE>, item_blocks, L2_THREADS, 0, s, v, g, t, pr); } while (0)
    if (words) L(false); else L(true);
#undef L
    if (bins >= 2 * sm_count()) launch_next(item_columns_kernel<4>, bins, 4 * BIN_TILES, 0, s, g, t, ranges);
    else launch_next(item_columns_kernel<16>, bins, 16 * BIN_TILES, 0, s, g, t, ranges);
    launch_next(tile_scan_kernel, div_up(tiles, SCAN_TILES), SCAN_TILES, 0, s, v, g, t, cap, ranges, c->num_isect, tiles_out);
    if (words) launch_next(item_emit_kernel<false>, item_blocks, L2_THREADS, 0, s, v, g, t, pr, ranges, c->vals_sorted);
    else launch_next(item_emit_kernel<true>, item_blocks, L2_THREADS, 0, s, v, g, t, pr, ranges, c->vals_sorted);
  }
  return check_launch();
}

int launch_fill_keys(const B2kCtx* c, cudaStream_t s) {
  launch_next(fill_keys_kernel, std::min(div_up(c->n_tiles, 8), sm_count() * 8), 256, 0, s, c->n_tiles, (const uint2*)c->tile_ranges, c->keys_sorted);
  return check_launch();
}

}  // namespace b2k
