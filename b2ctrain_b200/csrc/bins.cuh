// What the two routes from depth-ordered splats to tile lists share: bins of 8x8 tiles, tile boxes and masks as the projection leaves
// them, ellipse tests of a warp's pairs, block scans, the tables. bins.cu: counting distribution over the bins; walk.cu: every bin
// walks the ranks.
#pragma once
#include "common.cuh"

namespace b2k {

constexpr int BIN_W = 8;                      // tiles along a bin's edge
constexpr int BIN_TILES = BIN_W * BIN_W;
constexpr int MAX_BINS = 2048;                // bins of one band: what a block's tables in shared memory hold; larger images take several bands of bin rows
constexpr int MAX_ITEMS = 8192;               // items of one band: BINS_TABLE_WORDS / 64
constexpr int L2_THREADS = 256, L2_WARPS = L2_THREADS / 32;
constexpr int SCAN_TILES = 1024;              // tiles per block of tile_scan
constexpr unsigned FULL = 0xffffffffu;

// The bins and tiles of one band.
struct Band { int tiles_x, tiles_y, bins_x, bin_row0, bin_rows; };
__device__ __forceinline__ int band_bins(const Band& g) { return g.bins_x * g.bin_rows; }

// What a call works on. words == nullptr: the whole view, from exact hit masks; else depth chunk `chunk` of a chunked view.
struct View {
  const uint32_t* order; const uint4* hit_info; const uint32_t* tile_count; const float4* proj0; const float4* proj1;
  int n; uint32_t* words; int chunk, lo_num, hi_num; const unsigned long long* alive; int first_band, last_band;
};

struct Tables {
  uint32_t* cells;       // [bin][block] of level 1, then [item][64] of level 2
  uint32_t* totals;      // [MAX_BINS] pairs per bin
  uint32_t* base;        // [MAX_BINS + 1] first pair of each bin
  uint32_t* first_item;  // [MAX_BINS + 1]
  uint32_t* item_bin;    // [MAX_ITEMS]
  uint32_t* block_sums;  // [1024] tile counts of level 1's blocks (whole view)
  uint32_t* segments;    // [BINS_SEGMENTS] hits per tile_scan block
  uint32_t* st;          // [16] see S_*
  uint32_t* tile_totals; // [WALK_TILES] hits per tile, of walk.cu
  uint32_t* live_counts; // [512][16] live splats of the parts of level 1's runs (a chunk)
  uint32_t* longest;     // the longest list, for the compositing: of a whole view in ctx->num_isect, of a chunk in its words
};
constexpr int WALK_TILES = 4096;               // tiles of a view that walk.cu takes
inline Tables bins_tables(uint32_t* tables, uint32_t* longest) {
  Tables t;
  t.longest = longest;
  t.cells = tables;
  t.totals = t.cells + BINS_TABLE_WORDS; t.base = t.totals + MAX_BINS; t.first_item = t.base + MAX_BINS + 1; t.item_bin = t.first_item + MAX_BINS + 1;
  t.block_sums = t.item_bin + MAX_ITEMS; t.segments = t.block_sums + 1024; t.st = t.segments + BINS_SEGMENTS; t.tile_totals = t.st + 16; t.live_counts = t.tile_totals + WALK_TILES;
  static_assert(MAX_BINS + 2 * (MAX_BINS + 1) + MAX_ITEMS + 1024 + BINS_SEGMENTS + 16 + WALK_TILES + 512 * 16 <= BINS_EXTRA_WORDS, "scratch");
  return t;
}
enum { S_PAIRS = 0, S_ITEMS, S_ITEM_LEN, S_DONE_ROWS, S_DONE_TILES, S_SLOT, S_OVER, S_TOTAL, S_KEPT };

__device__ __forceinline__ void view_ranks(const View& v, uint32_t& r0, uint32_t& r1) {
  if (!v.words) { r0 = 0u; r1 = (uint32_t)v.n; return; }
  const uint64_t V = v.words[CW_V];
  r0 = (uint32_t)((V * (uint64_t)v.lo_num) >> 8);
  r1 = (uint32_t)((V * (uint64_t)v.hi_num) >> 8);
}

// A splat's tile box, half open; empty when x1 == x0.
struct Box { int x0, y0, x1, y1; };
__device__ __forceinline__ Box box_of(const uint4& hi) {
  Box b;
  if (hi.z == 0xFFFFFFFFu) {
    b.x0 = (int)(hi.x & 0xFFFFu); b.y0 = (int)(hi.x >> 16);
    b.x1 = b.x0 + (int)(hi.y & 0xFFFFu); b.y1 = b.y0 + (int)(hi.y >> 16);
  } else {
    b.x0 = (int)(hi.z & 0xFFFu); b.y0 = (int)((hi.z >> 12) & 0xFFFu);
    b.x1 = b.x0 + (int)(hi.z >> 24); b.y1 = b.y0 + (int)hi.w;
  }
  return b;
}
// The box's tiles inside bin (bx, by), bit = row * 8 + column.
__device__ __forceinline__ unsigned long long rect_bits(const Box& b, int bx, int by) {
  const int lx0 = max(b.x0 - bx * BIN_W, 0), lx1 = min(b.x1 - bx * BIN_W, BIN_W), ly0 = max(b.y0 - by * BIN_W, 0), ly1 = min(b.y1 - by * BIN_W, BIN_W);
  const unsigned long long row = ((1u << (lx1 - lx0)) - 1u) << lx0;
  return (row * 0x0101010101010101ull) & ((~0ull >> (64 - BIN_W * (ly1 - ly0))) << (BIN_W * ly0));
}
// The same from the exact hit mask of a box of at most 64 tiles (row-major inside the box).
__device__ __forceinline__ unsigned long long mask_bits(const uint4& hi, const Box& b, int bx, int by) {
  const unsigned long long mask = ((unsigned long long)hi.y << 32) | hi.x;
  const int xs = max(b.x0, bx * BIN_W), xe = min(b.x1, bx * BIN_W + BIN_W), ys = max(b.y0, by * BIN_W), ye = min(b.y1, by * BIN_W + BIN_W), bw = b.x1 - b.x0;
  unsigned long long out = 0ull;
  for (int y = ys; y < ye; y++)
    out |= ((mask >> ((y - b.y0) * bw + (xs - b.x0))) & ((1ull << (xe - xs)) - 1ull)) << ((y - by * BIN_W) * BIN_W + (xs - bx * BIN_W));
  return out;
}

// Inclusive scan over the block of one value per thread (at most 1024 threads); s_warp holds 32 values. Synchronises.
template <class T>
__device__ __forceinline__ T block_scan(T v, T* s_warp, T& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const T u = __shfl_up_sync(FULL, v, o); if (lane >= o) v += u; }
  __syncthreads();
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  T pre = 0, all = 0;
  for (int w = 0; w < warps; w++) { const T t = s_warp[w]; if (w < warp) pre += t; all += t; }
  total = all;
  return v + pre;
}

// Transposes the 32x32 bit matrix whose row i is lane i's word.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const uint32_t m = o == 16 ? 0x0000FFFFu : o == 8 ? 0x00FF00FFu : o == 4 ? 0x0F0F0F0Fu : o == 2 ? 0x33333333u : 0x55555555u;   // columns without bit o
    const uint32_t y = __shfl_xor_sync(FULL, x, o);
    x = (lane & o) ? (x & ~m) | ((y >> o) & m) : (x & m) | ((y & m) << o);
  }
  return x;
}

// The ellipse tests of a warp's 32 pairs against their bin, shared out by tile row: boxes hold one to 64 tiles of the bin, and with a
// pair per lane most lanes wait for the largest. todo: tiles of the lane's pair to test (rec of the lane's pair where it is not
// zero); returns the hits. All lanes call this.
struct WarpShare { float4 rec[64]; unsigned long long hits[32]; uint32_t unit[32 * BIN_W]; };   // unit: pair | row << 5 | columns << 8
__device__ __forceinline__ void share_record(WarpShare& ws, const float4& q0, const float4& q1) {
  const TileRec rec = make_tile_rec(q0.x, q0.y, q0.z, q0.w, q1.x, q1.w);
  const int lane = threadIdx.x & 31;
  ws.rec[lane * 2] = make_float4(rec.mx, rec.my, rec.c00, rec.c01);
  ws.rec[lane * 2 + 1] = make_float4(rec.c11, rec.power, rec.ia, rec.ib);
}
__device__ __forceinline__ unsigned long long shared_tests(WarpShare& ws, unsigned long long todo, int bx, int by) {
  const int lane = threadIdx.x & 31;
  uint32_t rows = 0u;
#pragma unroll
  for (int r = 0; r < BIN_W; r++) rows |= ((uint32_t)(todo >> (8 * r)) & 0xFFu) ? 1u << r : 0u;
  uint32_t at = __popc(rows);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(FULL, at, o); if (lane >= o) at += u; }
  const uint32_t units = __shfl_sync(FULL, at, 31);
  if (units == 0u) return 0ull;
  at -= __popc(rows);
  for (uint32_t b = rows; b; b &= b - 1u, at++) {
    const int r = __ffs(b) - 1;
    ws.unit[at] = (uint32_t)lane | ((uint32_t)r << 5) | (((uint32_t)(todo >> (8 * r)) & 0xFFu) << 8);
  }
  ws.hits[lane] = 0ull;
  __syncwarp();
  for (uint32_t u = lane; u < units; u += 32) {
    const uint32_t e = ws.unit[u], owner = e & 31u, r = (e >> 5) & 7u;
    const float4 a = ws.rec[owner * 2], b = ws.rec[owner * 2 + 1];
    const TileRec rec{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const TileRow row = tile_row(by * BIN_W + (int)r, rec);
    uint32_t out = 0u;
    for (uint32_t cols = e >> 8; cols; cols &= cols - 1u) {
      const int c = __ffs(cols) - 1;
      if (tile_hit(bx * BIN_W + c, row, rec)) out |= 1u << c;
    }
    reinterpret_cast<unsigned char*>(ws.hits + owner)[r] = (unsigned char)out;
  }
  __syncwarp();
  const unsigned long long hits = ws.hits[lane];
  __syncwarp();
  return hits;
}

// A pair's hit word by itself, where none was kept.
template <bool WHOLE>
__device__ __forceinline__ unsigned long long hits_again(const View& v, int bx, int by, unsigned long long alive, uint32_t i) {
  const uint4 hi = v.hit_info[i];
  const Box b = box_of(hi);
  if (WHOLE && hi.z != 0xFFFFFFFFu) return mask_bits(hi, b, bx, by);
  const float4 q0 = v.proj0[i], q1 = v.proj1[i];
  const TileRec rec = make_tile_rec(q0.x, q0.y, q0.z, q0.w, q1.x, q1.w);
  unsigned long long out = 0ull;
  for (unsigned long long todo = rect_bits(b, bx, by) & alive; todo; todo &= todo - 1ull) {
    const int tile = __ffsll((long long)todo) - 1;
    if (tile_hit(bx * BIN_W + (tile & 7), by * BIN_W + (tile >> 3), rec)) out |= 1ull << tile;
  }
  return out;
}

// The other route (walk.cu): whether it is taken for a whole view of n splats, and the lists by it.
bool walks(const B2kCtx* c, int n);
int launch_walk(const B2kCtx* c, const View& v, uint32_t* tables, cudaStream_t s);

}  // namespace b2k
