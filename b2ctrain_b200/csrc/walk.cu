// From depth-ordered splats to per-tile fragment lists in small views: every bin of 8x8 tiles walks the ranks, tests their boxes, and what
// overlaps the bin comes out in depth order. So level 1 of bins.cu (count, scan, write: three kernels) is gone; a run of ranks has its own
// place for its hit words with every bin, tile totals are added up with reductions, and the emission scans them itself:
//   walk_count   a block per bin and run of 256 ranks: the ranks' hit words in the bin, the hits per tile
//   walk_emit    the same blocks write their hits and tile ids to the tiles' lists; the first one writes the ranges
// Two kernels in place of eight, with the lists, ranges and totals of bins.cu, bit for bit. For whole views only.
// Bound by launch latency and by chains of three dependent loads.
#include "bins.cuh"
#include <algorithm>

namespace b2k {
namespace {

constexpr int WALK_THREADS = 256, WALK_WARPS = WALK_THREADS / 32;
constexpr int RUN = WALK_THREADS;             // ranks of a run: one batch of pairs. A small object lies in two or three bins, and longer runs leave it to a few blocks
constexpr int OFF_RANKS = 4 * WALK_THREADS;   // ranks per block of the running sum of tile counts

struct Walk {
  uint32_t* any;                              // [bin][run] whether any rank of the run has a box over the bin
  uint32_t* cells;                            // [bin][run][64] hits per tile
  uint32_t* totals;                           // [tile] hits
  uint32_t *lo, *hi;                          // [bin][run][RUN] hit words of the ranks
  uint32_t* off_sums;                         // [block of ranks] tile counts
  int runs, off_blocks;
};

// The block's work: the first off_blocks blocks make the running sum of the tile counts, the others take a bin and a run each.
struct Unit { int bin, run, bx, by; size_t at; };
__device__ __forceinline__ Unit unit_of(const Walk& w, const Band& g) {
  const int bins = band_bins(g), k = (int)blockIdx.x - w.off_blocks;
  Unit u;
  u.run = k / bins; u.bin = k - u.run * bins;
  u.bx = u.bin % g.bins_x; u.by = u.bin / g.bins_x;
  u.at = (size_t)u.bin * w.runs + u.run;
  return u;
}
// Tile counts of the block's ranks, in order: thread t holds ranks 4 t .. 4 t + 3.
__device__ __forceinline__ void off_counts(const View& v, uint32_t (&c)[4]) {
  uint32_t i[4];
  const int p = blockIdx.x * OFF_RANKS + threadIdx.x * 4;
#pragma unroll
  for (int u = 0; u < 4; u++) i[u] = p + u < v.n ? v.order[p + u] : 0u;
#pragma unroll
  for (int u = 0; u < 4; u++) c[u] = p + u < v.n ? v.tile_count[i[u]] : 0u;
}

__global__ void __launch_bounds__(WALK_THREADS) walk_count_kernel(View v, Band g, Walk w) {
  after_previous();
  __shared__ uint32_t s_warp[32];
  __shared__ WarpShare s_share[WALK_WARPS];
  __shared__ uint32_t s_cnt[WALK_WARPS][BIN_TILES];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((int)blockIdx.x < w.off_blocks) {
    uint32_t c[4], total;
    off_counts(v, c);
    block_scan(c[0] + c[1] + c[2] + c[3], s_warp, total);
    if (tid == 0) w.off_sums[blockIdx.x] = total;
    return;
  }
  const Unit u = unit_of(w, g);
  const int p = u.run * RUN + tid, x0 = u.bx * BIN_W, y0 = u.by * BIN_W;
  uint32_t i = 0u;
  uint4 hi = make_uint4(0u, 0u, 0u, 0u);
  if (p < v.n) { i = v.order[p]; hi = v.hit_info[i]; }
  const Box b = box_of(hi);
  const bool in = b.x0 < x0 + BIN_W && b.x1 > max(x0, b.x0) && b.y0 < y0 + BIN_W && b.y1 > max(y0, b.y0);
  const bool any = __syncthreads_or(in);
  if (tid == 0) w.any[u.at] = any ? 1u : 0u;
  if (!any) return;
  unsigned long long hits = 0ull, todo = 0ull;
  uint32_t tiles = 0u;                        // zero: hidden since the projection. (Read for every rank with its box, the kernel takes 8.4 us for 7.2.)
  if (in) {
    tiles = v.tile_count[i];
    if (hi.z != 0xFFFFFFFFu) hits = mask_bits(hi, b, u.bx, u.by);    // the projection has tested this box
    else {
      todo = rect_bits(b, u.bx, u.by);
      share_record(s_share[warp], v.proj0[i], v.proj1[i]);
    }
  }
  hits |= shared_tests(s_share[warp], todo, u.bx, u.by);
  if (tiles == 0u) hits = 0ull;
  w.lo[u.at * RUN + tid] = (uint32_t)hits; w.hi[u.at * RUN + tid] = (uint32_t)(hits >> 32);
  const uint32_t c_lo = __popc(transpose_bits((uint32_t)hits)), c_hi = __popc(transpose_bits((uint32_t)(hits >> 32)));   // this warp's hits on tiles `lane` and `lane + 32`
  s_cnt[warp][lane] = c_lo; s_cnt[warp][lane + 32] = c_hi;
  __syncthreads();
  if (tid < BIN_TILES) {
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < WALK_WARPS; k++) sum += s_cnt[k][tid];
    w.cells[u.at * BIN_TILES + tid] = sum;
    const int x = u.bx * BIN_W + (tid & 7), y = u.by * BIN_W + (tid >> 3);
    if (sum) atomicAdd(w.totals + y * g.tiles_x + x, sum);   // a tile outside the image has no hit
  }
}

// The hits of 256 pairs (hit words lo, hi of the thread's splat) to their tiles' lists, in the order of the pairs. next: the tiles' next free
// places, moved on. All threads of a block of 256 call this; it begins and ends with the block in step.
// Up to EMIT_HITS hits a lane goes through its own: each finds its place among the block's hits, tile by tile, in shared memory, and
// they leave from there side by side. Above that (splats over most of the bin) a warp takes a row of tiles and the 32 pairs of one hit
// word at a time, and the lanes with a hit write side by side; for sparse words most of that is spent on lanes without one.
constexpr uint32_t EMIT_HITS = 4096;
struct EmitShare {
  uint32_t word[WALK_WARPS][BIN_TILES];       // bit l: lane l of the warp hits the tile
  uint32_t before[WALK_WARPS][BIN_TILES];     // place, among the block's hits by tile, of the warp's first on the tile
  uint32_t next[BIN_TILES], delta[BIN_TILES]; // next free place of the tile's list; place in the list less place among the block's hits
  uint32_t total, splat[EMIT_HITS];
  unsigned char tile[EMIT_HITS];
};
// put(place, tile, splat)
template <class F>
__device__ __forceinline__ void emit_hits(EmitShare& es, uint32_t splat, uint32_t lo, uint32_t hi, F put) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lane_lt = (1u << lane) - 1u;
  es.word[warp][lane] = transpose_bits(lo);
  es.word[warp][lane + 32] = transpose_bits(hi);
  __syncthreads();
  if (warp == 0) {
    uint32_t c[2][WALK_WARPS], n[2] = {0u, 0u};
#pragma unroll
    for (int q = 0; q < WALK_WARPS; q++)
#pragma unroll
      for (int h = 0; h < 2; h++) { c[h][q] = n[h]; n[h] += __popc(es.word[q][lane + 32 * h]); }
    uint32_t first[2] = {n[0], n[1]};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int h = 0; h < 2; h++) { const uint32_t u = __shfl_up_sync(FULL, first[h], o); if (lane >= o) first[h] += u; }
    const uint32_t half = __shfl_sync(FULL, first[0], 31), all = half + __shfl_sync(FULL, first[1], 31);
    first[0] -= n[0]; first[1] += half - n[1];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int t = lane + 32 * h;
#pragma unroll
      for (int q = 0; q < WALK_WARPS; q++) es.before[q][t] = first[h] + c[h][q];
      es.delta[t] = es.next[t] - first[h];
      es.next[t] += n[h];
    }
    if (lane == 0) es.total = all;
  }
  __syncthreads();
  const uint32_t total = es.total;
  if (total <= EMIT_HITS) {
    auto spread = [&](uint32_t bits, int t0) {
      for (; bits; bits &= bits - 1u) {
        const int t = t0 + __ffs(bits) - 1;
        const uint32_t at = es.before[warp][t] + __popc(es.word[warp][t] & lane_lt);
        es.splat[at] = splat; es.tile[at] = (unsigned char)t;
      }
    };
    spread(lo, 0); spread(hi, 32);
    __syncthreads();
    for (uint32_t j = tid; j < total; j += WALK_THREADS) { const int t = es.tile[j]; put(es.delta[t] + j, t, es.splat[j]); }
  } else {
    es.splat[tid] = splat;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BIN_TILES / WALK_WARPS; k++) {
      const int t = warp * (BIN_TILES / WALK_WARPS) + k;
      for (int q = 0; q < WALK_WARPS; q++) {
        const uint32_t word = es.word[q][t];
        if ((word >> lane) & 1u) put(es.delta[t] + es.before[q][t] + __popc(word & lane_lt), t, es.splat[q * 32 + lane]);
      }
    }
  }
  __syncthreads();
}

// The hits of a bin and run to their tiles' lists, behind those of the bin's earlier runs.
__global__ void __launch_bounds__(WALK_THREADS) walk_emit_kernel(View v, Band g, Walk w, int n_tiles, uint2* __restrict__ ranges, uint32_t* __restrict__ vals,
                                                                 uint32_t* __restrict__ keys, uint32_t cap, uint32_t* __restrict__ tile_off, uint32_t* __restrict__ num_isect) {
  after_previous();
  __shared__ EmitShare s_emit;
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_start[WALK_TILES + WALK_THREADS];
  __shared__ uint32_t s_part[WALK_THREADS / BIN_TILES][BIN_TILES], s_longest[WALK_WARPS];
  const int tid = threadIdx.x;
  if ((int)blockIdx.x < w.off_blocks) {
    uint32_t c[4], mine = 0, total;
    for (int k = tid; k < (int)blockIdx.x; k += WALK_THREADS) mine += w.off_sums[k];
    off_counts(v, c);
    block_scan(mine, s_warp, total);
    uint32_t all, at = total + block_scan(c[0] + c[1] + c[2] + c[3], s_warp, all) - (c[0] + c[1] + c[2] + c[3]);
    const int p = blockIdx.x * OFF_RANKS + tid * 4;
#pragma unroll
    for (int u = 0; u < 4; u++) { at += c[u]; if (p + u < v.n) tile_off[p + u] = at; }
    return;
  }
  const Unit u = unit_of(w, g);
  const bool writes_ranges = (int)blockIdx.x == w.off_blocks;
  const bool any = w.any[u.at] != 0u;
  if (!any && !writes_ranges) return;
  // The hit words, the hits of the bin's earlier runs and the totals are on their way together.
  const int p = u.run * RUN + tid;
  const uint32_t splat = p < v.n ? v.order[p] : 0u, lo = any ? w.lo[u.at * RUN + tid] : 0u, hi = any ? w.hi[u.at * RUN + tid] : 0u;
  constexpr int GROUPS = WALK_THREADS / BIN_TILES;
  {
    const int tile = tid % BIN_TILES, group = tid / BIN_TILES;
    uint32_t sum = 0;
#pragma unroll 8
    for (int k = group; k < u.run; k += GROUPS) {
      const size_t unit = (size_t)u.bin * w.runs + k;
      const uint32_t c = w.cells[unit * BIN_TILES + tile];
      sum += w.any[unit] ? c : 0u;            // the others have not written their cells
    }
    s_part[group][tile] = sum;
  }
  // Scan over the tiles: each thread takes some in a row, by way of shared memory (one word of skew for every thread).
  const int per = (n_tiles + WALK_THREADS - 1) / WALK_THREADS;
  for (int i = tid; i < n_tiles; i += WALK_THREADS) s_start[i + i / per] = w.totals[i];
  __syncthreads();
  uint32_t sum = 0, total;
  const int t0 = tid * per;
  for (int k = 0; k < per; k++) sum += t0 + k < n_tiles ? s_start[t0 + k + tid] : 0u;
  uint32_t start = block_scan(sum, s_warp, total) - sum;
  uint32_t longest = 0u;
  for (int k = 0; k < per; k++) {
    if (t0 + k >= n_tiles) break;
    const uint32_t c = s_start[t0 + k + tid];
    longest = max(longest, c);
    s_start[t0 + k + tid] = start;
    if (writes_ranges) ranges[t0 + k] = c ? make_uint2(min(start, cap), min(start + c, cap)) : make_uint2(0u, 0u);
    start += c;
  }
  longest = __reduce_max_sync(FULL, longest);
  if ((tid & 31) == 0) s_longest[tid >> 5] = longest;
  __syncthreads();
  if (writes_ranges && tid == 0) {
    num_isect[0] = total;
    for (int k = 1; k < WALK_WARPS; k++) longest = max(longest, s_longest[k]);
    num_isect[NI_LONGEST] = longest;
  }
  if (!any) return;
  const int x0 = u.bx * BIN_W, y0 = u.by * BIN_W;
  if (tid < BIN_TILES) {
    const int x = x0 + (tid & 7), y = y0 + (tid >> 3);
    uint32_t next = 0;
    if (x < g.tiles_x && y < g.tiles_y) {
      const int id = y * g.tiles_x + x;
      next = s_start[id + id / per];
#pragma unroll
      for (int k = 0; k < GROUPS; k++) next += s_part[k][tid];
    }
    s_emit.next[tid] = next;
  }
  emit_hits(s_emit, splat, lo, hi, [&](uint32_t at, int t, uint32_t id) {
    if (at < cap) { vals[at] = id; keys[at] = (uint32_t)((y0 + (t >> 3)) * g.tiles_x + x0 + (t & 7)); }
  });
}

// Where the walk is taken: images of few tiles, whose totals every block can scan, and up to this many tests of a rank against a bin.
// Binning behind the sort, us, the general distribution / the walk (tests): 64x64 over 2k splats 30.8 / 13.6, over 200k (0.2M) 65.5 / 31.3;
// 200x150 over 40k (0.5M) 43.7 / 26.2, over 100k (1.2M) 55.1 / 46.7; 333x217 over 20k (0.5M) 43.8 / 24.1, over 60k (1.4M) 48.3 / 46.6;
// 400x300 over 30k (1.1M) 45.6 / 40.3, over 60k (2.1M) 50.3 / 62.8; 512x512 over 8k (0.5M) 50.1 / 36.4, over 16k (1.0M) 50.2 / 52.6.
constexpr long long WALK_TESTS = 1LL << 20;

}  // namespace

bool walks(const B2kCtx* c, int n) {
  const int bins = div_up(c->tiles_x, BIN_W) * div_up(c->tiles_y, BIN_W);
  if (c->n_tiles > WALK_TILES || (long long)n * bins > WALK_TESTS) return false;
  const long long units = (long long)bins * div_up(n, RUN);
  return units * (BIN_TILES + 1) <= (long long)BINS_TABLE_WORDS && units * RUN <= (long long)c->isect_cap;   // (cells; hit words)
}

int launch_walk(const B2kCtx* c, const View& v, uint32_t* tables, cudaStream_t s) {
  const Tables t = bins_tables(tables, c->num_isect + NI_LONGEST);
  const Band g{c->tiles_x, c->tiles_y, div_up(c->tiles_x, BIN_W), 0, div_up(c->tiles_y, BIN_W)};
  const int bins = g.bins_x * g.bin_rows;
  Walk w;
  w.runs = div_up(v.n, RUN); w.off_blocks = div_up(v.n, OFF_RANKS);
  w.cells = t.cells; w.any = t.cells + (size_t)bins * w.runs * BIN_TILES; w.totals = t.tile_totals; w.off_sums = t.item_bin;
  w.lo = c->keys; w.hi = c->vals;
  const int blocks = w.off_blocks + bins * w.runs;
  launch_next(walk_count_kernel, blocks, WALK_THREADS, 0, s, v, g, w);
  launch_next(walk_emit_kernel, blocks, WALK_THREADS, 0, s, v, g, w, c->n_tiles, (uint2*)c->tile_ranges, c->vals_sorted, c->keys_sorted, (uint32_t)c->isect_cap, c->tile_off,
              c->num_isect);
  return check_launch();
}

}  // namespace b2k
