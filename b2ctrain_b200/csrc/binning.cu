// Depth order, and the entry points of the binning stage and of the front-to-back chunked renderer. Reference semantics:
// bin_and_sort (src/gpu/binning.cu:109-145); its library sorts and scan are replaced by the radix sort in this file and the
// two-level distribution of bins.cu.
//
// The sort is integer work bound by HBM traffic. Design points:
//  * No host round trip: element counts are read from device memory by grids sized from the SM count, so the whole view is
//    one asynchronous chain.
//  * The radix sort is the wait-free three-kernel form (per-block digit counts, row scan, ranked scatter): no kernel
//    ever spins on another block. Each block owns one contiguous segment and walks it tile by tile, so the count
//    table is 256 x (a few hundred) words whatever the input size.
//  * Scatter is staged through shared memory so global writes go out in digit runs (coalesced), keys and values
//    move as 32-bit words, loads are warp-contiguous.
//  * Sorting is LSD with 8-bit digits and is stable, so order = ascending (key, original position): exactly the
//    order the reference's stable sorts define.
#include "common.cuh"
#include <algorithm>

namespace b2k {
namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 16;
constexpr int COUNT_TILE = SORT_THREADS * SORT_ITEMS;   // 4096 keys per counting step of a CTA
constexpr int SORT_TILE = 4096;                         // pairs per scatter tile (a multiple of COUNT_TILE)
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int RADIX_MAX = 512;                 // widest digit (9 bits): sizes the histogram scratch
constexpr int BLOCKS_PER_SM = 2;               // resident scatter CTAs per SM: one wave covers the input

__device__ __forceinline__ uint32_t seg_len(uint32_t n, uint32_t blocks) {
  uint32_t per = (n + blocks - 1) / blocks;
  return ((per + SORT_TILE - 1) / SORT_TILE) * SORT_TILE;
}
__device__ __forceinline__ uint32_t load_n(const uint32_t* n_ptr, uint32_t n_max) {
  const uint32_t n = *n_ptr;
  return n < n_max ? n : n_max;
}
// A sort may work on a window of its buffers that starts `*off_ptr` elements in (a depth chunk of the view): the
// window's length is clamped to what is left of the buffers.
__device__ __forceinline__ uint32_t load_off(const uint32_t* off_ptr) { return off_ptr ? *off_ptr : 0u; }
__device__ __forceinline__ uint32_t load_n(const uint32_t* n_ptr, uint32_t n_max, uint32_t off) {
  return load_n(n_ptr, off < n_max ? n_max - off : 0u);
}

// Pass kernel 1: digit counts of each block's segment. hist is [RADIX][blocks]. Each lane keeps 16 keys in flight
// (four 128-bit loads) so that a few hundred resident warps cover the HBM latency-bandwidth product.
template <int BITS>
__global__ void __launch_bounds__(SORT_THREADS) radix_count_kernel(const uint32_t* __restrict__ keys_base, const uint32_t* __restrict__ n_ptr, uint32_t n_max,
                                                                   int shift, uint32_t mask, uint32_t* __restrict__ hist, const uint32_t* __restrict__ off_ptr) {
  constexpr int RADIX = 1 << BITS;
  __shared__ uint32_t s_hist[SORT_WARPS][RADIX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < SORT_WARPS * RADIX; i += SORT_THREADS) (&s_hist[0][0])[i] = 0;
  __syncthreads();
  const uint32_t off = load_off(off_ptr);   // a multiple of 32 elements: 128-bit loads stay aligned
  const uint32_t* __restrict__ keys = keys_base + off;
  const uint32_t n = load_n(n_ptr, n_max, off);
  const uint32_t len = seg_len(n, gridDim.x);
  const uint64_t begin64 = (uint64_t)blockIdx.x * len;
  const uint32_t begin = begin64 < n ? (uint32_t)begin64 : n;
  const uint32_t end = (begin64 + len) < n ? (uint32_t)(begin64 + len) : n;
  // Segments start on a multiple of the tile size, so 128-bit loads are aligned.
  for (uint32_t tile = begin + warp * (32 * SORT_ITEMS); tile < end; tile += COUNT_TILE) {   // warp-uniform trip count
    uint32_t k[SORT_ITEMS];
    if (tile + 32 * SORT_ITEMS <= end) {
#pragma unroll
      for (int v = 0; v < SORT_ITEMS / 4; v++) {
        const uint4 q = *reinterpret_cast<const uint4*>(keys + tile + v * 128 + lane * 4);
        k[v * 4] = q.x; k[v * 4 + 1] = q.y; k[v * 4 + 2] = q.z; k[v * 4 + 3] = q.w;
      }
#pragma unroll
      for (int j = 0; j < SORT_ITEMS; j++) atomicAdd(&s_hist[warp][(k[j] >> shift) & mask], 1u);
    } else {
#pragma unroll
      for (int j = 0; j < SORT_ITEMS; j++) { const uint32_t i = tile + j * 32 + lane; k[j] = i < end ? keys[i] : 0u; }
#pragma unroll
      for (int j = 0; j < SORT_ITEMS; j++)
        if (tile + j * 32 + lane < end) atomicAdd(&s_hist[warp][(k[j] >> shift) & mask], 1u);
    }
  }
  __syncthreads();
  for (int d = threadIdx.x; d < RADIX; d += SORT_THREADS) {
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; w++) t += s_hist[w][d];
    hist[(size_t)d * gridDim.x + blockIdx.x] = t;
  }
}

// Pass kernel 2: one block per digit turns its row of per-block counts into exclusive offsets and records the row
// total. blocks <= 1024.
__global__ void __launch_bounds__(1024) radix_rows_kernel(uint32_t* __restrict__ hist, int blocks, uint32_t* __restrict__ totals) {
  __shared__ uint32_t s_warp[32];
  const int d = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t v = t < blocks ? hist[(size_t)d * blocks + t] : 0u;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { uint32_t u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = s_warp[lane], wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { uint32_t u = __shfl_up_sync(0xffffffffu, wi, o); if (lane >= o) wi += u; }
    s_warp[lane] = wi - w;
    if (lane == 31) totals[d] = wi;
  }
  __syncthreads();
  if (t < blocks) hist[(size_t)d * blocks + t] = s_warp[warp] + incl - v;
}

// Pass kernel 3: ranked, stable scatter of each block's segment. 512 threads x 8 pairs per tile; the next tile's keys
// and this tile's values are in flight while the current tile is ranked, so memory and ranking phases overlap.
constexpr int SCAT_THREADS = 512;
constexpr int SCAT_ITEMS = SORT_TILE / SCAT_THREADS;   // 8
constexpr int SCAT_WARPS = SCAT_THREADS / 32;
constexpr size_t SCAT_SMEM = 2 * SORT_TILE * sizeof(uint32_t);

template <int BITS>
__global__ void __launch_bounds__(SCAT_THREADS, SCAT_THREADS <= 512 ? 2 : 1) radix_scatter_kernel(
    const uint32_t* __restrict__ keys_in_base, const uint32_t* __restrict__ vals_in_base, uint32_t* __restrict__ keys_out_base,
    uint32_t* __restrict__ vals_out_base, const uint32_t* __restrict__ n_ptr, uint32_t n_max, int shift, uint32_t mask,
    const uint32_t* __restrict__ hist, const uint32_t* __restrict__ totals, const uint32_t* __restrict__ off_ptr) {
  const uint32_t off = load_off(off_ptr);
  const uint32_t* __restrict__ keys_in = keys_in_base + off;
  const uint32_t* __restrict__ vals_in = vals_in_base + off;
  uint32_t* __restrict__ keys_out = keys_out_base + off;
  uint32_t* __restrict__ vals_out = vals_out_base + off;
  constexpr int RADIX = 1 << BITS;
  static_assert(RADIX <= SCAT_THREADS, "one thread per digit in the scans below");
  __shared__ uint32_t s_cnt[SCAT_WARPS][RADIX];   // per-warp digit counts, then per-warp offsets inside the digit
  __shared__ uint32_t s_gbase[RADIX];             // running global slot of the digit for this block
  __shared__ uint32_t s_delta[RADIX];             // global slot = s_delta[digit] + local slot (mod 2^32)
  __shared__ uint32_t s_scan[RADIX / 32];
  extern __shared__ uint32_t s_stage[];           // [2][SORT_TILE]: the tile's keys and values in digit order
  uint32_t* s_keys = s_stage;
  uint32_t* s_vals = s_stage + SORT_TILE;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t lane_lt = (1u << lane) - 1u;
  // Global base of (digit, block): exclusive scan of the digit totals + the block's offset inside the digit.
  {
    uint32_t tot = 0, incl = 0;
    if (tid < RADIX) {
      tot = totals[tid]; incl = tot;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { uint32_t u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
      if (lane == 31) s_scan[warp] = incl;
    }
    __syncthreads();
    if (tid < RADIX) {
      uint32_t pre = 0;
      for (int w = 0; w < warp; w++) pre += s_scan[w];
      s_gbase[tid] = pre + incl - tot + hist[(size_t)tid * gridDim.x + blockIdx.x];
    }
    __syncthreads();
  }
  const uint32_t n = load_n(n_ptr, n_max, off);
  const uint32_t len = seg_len(n, gridDim.x);
  const uint64_t begin64 = (uint64_t)blockIdx.x * len;
  const uint32_t begin = begin64 < n ? (uint32_t)begin64 : n;
  const uint32_t end = (begin64 + len) < n ? (uint32_t)(begin64 + len) : n;
  // Each warp owns 256 consecutive pairs of the tile; item j of lane l is pair j*32 + l of them, so (j, lane) order is
  // input order.
  const uint32_t wbase = warp * (32 * SCAT_ITEMS);
  uint32_t key[SCAT_ITEMS];
#pragma unroll
  for (int j = 0; j < SCAT_ITEMS; j++) { const uint32_t i = begin + wbase + j * 32 + lane; key[j] = i < end ? keys_in[i] : 0xFFFFFFFFu; }
  for (uint32_t tile = begin; tile < end; tile += SORT_TILE) {
    const uint32_t tile_n = end - tile < SORT_TILE ? end - tile : SORT_TILE;
    const bool full = tile_n == SORT_TILE;
    uint32_t val[SCAT_ITEMS], rank[SCAT_ITEMS];
    if (full) {
#pragma unroll
      for (int j = 0; j < SCAT_ITEMS; j++) val[j] = vals_in[tile + wbase + j * 32 + lane];
    } else {
#pragma unroll
      for (int j = 0; j < SCAT_ITEMS; j++) { const uint32_t li = wbase + j * 32 + lane; val[j] = li < tile_n ? vals_in[tile + li] : 0u; }
    }
    for (int i = tid; i < SCAT_WARPS * RADIX; i += SCAT_THREADS) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    // Rank of every pair among the warp's pairs with the same digit: the lowest lane holding the digit bumps the warp's counter for the digit (one shared-memory atomic) and hands the old value out.
#pragma unroll
    for (int j = 0; j < SCAT_ITEMS; j++) {
      const bool valid = full || wbase + j * 32 + lane < tile_n;
      const uint32_t d = (key[j] >> shift) & mask;
      uint32_t peers = full ? 0xffffffffu : __ballot_sync(0xffffffffu, valid);   // lanes holding the same digit: one vote per digit bit
#pragma unroll                                                                   // (measured 3x cheaper here than match.any)
      for (int b = 0; b < BITS; b++) {
        const bool bit = (d >> b) & 1u;
        const uint32_t vote = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? vote : ~vote;
      }
      const int leader = __ffs(peers) - 1;
      uint32_t old = 0;
      if (valid && lane == leader) old = atomicAdd(&s_cnt[warp][d], (uint32_t)__popc(peers));
      rank[j] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers & lane_lt);
    }
    __syncthreads();
    // Digit `tid`: the digit's first slot in the tile, and for every warp its first slot inside the digit.
    uint32_t total = 0, incl = 0;
    if (tid < RADIX) {
#pragma unroll
      for (int w = 0; w < SCAT_WARPS; w++) total += s_cnt[w][tid];
      incl = total;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) { uint32_t u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
      if (lane == 31) s_scan[warp] = incl;
    }
    __syncthreads();
    if (tid < RADIX) {
      uint32_t pre = 0;
      for (int w = 0; w < warp; w++) pre += s_scan[w];
      uint32_t at = pre + incl - total;       // first slot of the digit
      s_delta[tid] = s_gbase[tid] - at;
      s_gbase[tid] += total;
#pragma unroll
      for (int w = 0; w < SCAT_WARPS; w++) { const uint32_t c = s_cnt[w][tid]; s_cnt[w][tid] = at; at += c; }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SCAT_ITEMS; j++) {
      if (full || wbase + j * 32 + lane < tile_n) {
        const uint32_t slot = s_cnt[warp][(key[j] >> shift) & mask] + rank[j];
        s_keys[slot] = key[j];
        s_vals[slot] = val[j];
      }
    }
    // Prefetch the next tile's keys; they land while this tile is written out.
    {
      const uint32_t next = tile + SORT_TILE;
#pragma unroll
      for (int j = 0; j < SCAT_ITEMS; j++) { const uint64_t i = (uint64_t)next + wbase + j * 32 + lane; key[j] = i < end ? keys_in[i] : 0xFFFFFFFFu; }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SCAT_ITEMS; j++) {
      const uint32_t slot = j * SCAT_THREADS + tid;
      if (full || slot < tile_n) {
        const uint32_t k = s_keys[slot];
        const uint32_t dst = s_delta[(k >> shift) & mask] + slot;
        keys_out[dst] = k;
        vals_out[dst] = s_vals[slot];
      }
    }
    __syncthreads();
  }
}

__global__ void set_word_kernel(uint32_t* p, uint32_t v) { *p = v; }

struct SortScratch { uint32_t* hist; uint32_t* totals; uint32_t* n_word; };

int sort_blocks() { int b = sm_count() * BLOCKS_PER_SM; return b > 1024 ? 1024 : b; }

SortScratch carve(uint32_t* tables, int blocks) {
  SortScratch s;
  s.hist = tables;
  s.totals = s.hist + (size_t)RADIX_MAX * blocks;
  s.n_word = s.totals + RADIX_MAX;
  return s;
}
static_assert((size_t)RADIX_MAX * 1024 <= BINS_TABLE_WORDS, "the sort and the binning share one table");

// Optional timing marks for b2k_bin_sort_profile: when armed, an event is recorded on the stream at each mark.
struct Marks { cudaEvent_t ev[32]; int n = 0; bool armed = false; };
thread_local Marks g_marks;
void mark(cudaStream_t s) { if (g_marks.armed && g_marks.n < 32) cudaEventRecord(g_marks.ev[g_marks.n++], s); }

// Digit width of a sort over `bits` key bits: 8, except where 9 saves a whole pass (17 or 18 bits, the tile ids of a 4K
// image: two passes instead of three).
int sort_digit_bits(int bits) { return (bits > 16 && bits <= 18) ? 9 : 8; }
int sort_passes(int bits) { const int d = sort_digit_bits(bits); return (bits + d - 1) / d; }

template <int BITS>
int radix_pass(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, const uint32_t* n_ptr, uint32_t n_max, int shift, uint32_t mask, const SortScratch& sc,
               int blocks, cudaStream_t s, const uint32_t* off_ptr) {
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(radix_scatter_kernel<BITS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCAT_SMEM) != cudaSuccess) return check_launch();
    attr_set[dev] = true;
  }
  radix_count_kernel<BITS><<<blocks, SORT_THREADS, 0, s>>>(k0, n_ptr, n_max, shift, mask, sc.hist, off_ptr);
  radix_rows_kernel<<<1 << BITS, 1024, 0, s>>>(sc.hist, blocks, sc.totals);
  mark(s);
  radix_scatter_kernel<BITS><<<blocks, SCAT_THREADS, SCAT_SMEM, s>>>(k0, v0, k1, v1, n_ptr, n_max, shift, mask, sc.hist, sc.totals, off_ptr);
  mark(s);
  return B2K_OK;
}

// LSD radix sort of (key, value) pairs over bits [0, bits). The element count is read from *n_ptr on the device and
// clamped to n_max. Buffers (k0, v0) hold the input; the result lands in (k0, v0) when sort_passes(bits) is even and in
// (k1, v1) when it is odd.
int radix_sort(uint32_t* k0, uint32_t* v0, uint32_t* k1, uint32_t* v1, const uint32_t* n_ptr, uint32_t n_max, int bits, const SortScratch& sc,
               int blocks, cudaStream_t s, const uint32_t* off_ptr = nullptr) {
  const int digit = sort_digit_bits(bits), passes = sort_passes(bits);
  for (int p = 0; p < passes; p++) {
    const int shift = p * digit;
    const int pb = bits - shift < digit ? bits - shift : digit;
    const uint32_t mask = (1u << pb) - 1u;
    const int st = digit == 9 ? radix_pass<9>(k0, v0, k1, v1, n_ptr, n_max, shift, mask, sc, blocks, s, off_ptr)
                              : radix_pass<8>(k0, v0, k1, v1, n_ptr, n_max, shift, mask, sc, blocks, s, off_ptr);
    if (st) return st;
    uint32_t* t = k0; k0 = k1; k1 = t;
    t = v0; v0 = v1; v1 = t;
  }
  return check_launch();
}


int depth_sort(const B2kCtx* c, int n, uint32_t* tables, cudaStream_t s) {
  const int blocks = sort_blocks();
  const SortScratch sc = carve(tables, blocks);
  set_word_kernel<<<1, 1, 0, s>>>(sc.n_word, (uint32_t)n);
  return radix_sort(c->depth_keys_sorted, c->order, c->depth_keys, c->order_in, sc.n_word, (uint32_t)n, 32, sc, blocks, s);
}

// ---- front-to-back rendering in depth chunks ------------------------------------------------------------------------
// The view's splats are taken in a few chunks of increasing depth rank. A chunk is binned (its hits distributed to the
// tiles, bins.cu) and composited before the next one is touched, and a tile whose pixels have all reached the
// transmittance cutoff takes nothing from then on: in a dense scene most intersections lie behind saturated pixels and
// are never composited, so they need not be binned either. Chunk c covers the ranks [V b(c-1), V b(c)) of the V
// splats with a tile box, with b = 1/4^(C-1), ..., 1/16, 1/4, 1 (small chunks first: the nearest splats decide most
// pixels, and every chunk costs eight launches whatever its size). The projection of this path leaves tile boxes,
// not hit masks: the ellipse-tile tests run per chunk, against live tiles only. Every chunk's pairs occupy their own window
// of vals_sorted, and a tile has one range per chunk.
constexpr int MAX_CHUNKS = 5;

// V = number of depth-sorted keys that are not the culled marker (they sort last); every tile is alive.
__global__ void __launch_bounds__(256) chunk_prepare_kernel(const uint32_t* __restrict__ keys_sorted, int n, uint32_t* __restrict__ words, unsigned long long* __restrict__ alive,
                                                            int bins) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < bins) alive[i] = ~0ull;
  if (i >= 32) return;
  // First culled key in [lo, hi): the warp probes 32 places at a time (five dependent loads for six million keys, not 23).
  int lo = 0, hi = n;
  while (lo < hi) {
    const int step = (hi - lo + 32) / 33, at = lo + (i + 1) * step - 1;   // probes at the ends of the first 32 of 33 parts
    const uint32_t kept = __ballot_sync(0xffffffffu, at < hi && keys_sorted[at] != 0xFFFFFFFFu);
    const int passed = __popc(kept);                                       // keys are sorted: the kept probes come first
    const int next = lo + passed * step;
    if (passed < 32) hi = min(hi, next + step - 1);
    lo = min(next, hi);
  }
  if (i != 0) return;
  words[CW_V] = (uint32_t)lo;
  words[CW_BASE] = 0u;
}

}  // namespace
}  // namespace b2k

using namespace b2k;

namespace b2k {
namespace {
constexpr uint64_t sort_tmp_words(uint64_t n_cap) { return BIG_HEADER_WORDS + n_cap + BINS_TABLE_WORDS + BINS_EXTRA_WORDS; }
}  // namespace
}  // namespace b2k

extern "C" uint64_t b2k_sort_tmp_bytes(int32_t n, uint64_t isect_cap) {
  (void)isect_cap;
  return sizeof(uint32_t) * sort_tmp_words(n > 0 ? (uint64_t)n : 0);
}

extern "C" int b2k_bin_sort(const B2kCtx* c, int32_t n, b2k_stream_t stream) {
  B2K_REQUIRE(c && n >= 0);
  B2K_REQUIRE(c->tile_ranges && c->num_isect && c->n_tiles == c->tiles_x * c->tiles_y && c->tile_bits >= 1 && c->tile_bits <= 24);
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    B2K_CUDA(cudaMemsetAsync(c->tile_ranges, 0, sizeof(uint32_t) * 2 * (size_t)c->n_tiles, s));
    B2K_CUDA(cudaMemsetAsync(c->num_isect, 0, sizeof(uint32_t), s));
    return B2K_OK;
  }
  B2K_REQUIRE(c->proj0 && c->proj1 && c->tile_count && c->hit_info && c->depth_keys && c->depth_keys_sorted && c->order_in && c->order && c->tile_off);
  B2K_REQUIRE(c->keys && c->vals && c->keys_sorted && c->vals_sorted && c->sort_tmp);
  if (c->n_cap < n) return B2K_ERR_CAPACITY;
  if (c->sort_tmp_bytes < b2k_sort_tmp_bytes(c->n_cap, c->isect_cap) || c->isect_cap == 0 || c->isect_cap > 0xFFFFFFF0ull) return B2K_ERR_CAPACITY;
  uint32_t* tables = sort_tables_ptr(c);
  // 1. Splats by depth: key = bits of view z (culled splats carry 0xFFFFFFFF and land last), value = index. The
  //    projection left its keys and indices in the (depth_keys_sorted, order) pair: with four passes (an even count)
  //    the ping-pong returns to the pair it started from, so the sorted result lands where callers expect it and
  //    (depth_keys, order_in) is the scratch pair.
  mark(s);
  int st = depth_sort(c, n, tables, s);
  if (st) return st;
  mark(s);
  // 2. Hits to the tiles' lists, depth order surviving inside each tile; 3. the tile ids of the list.
  st = launch_bins(c, n, nullptr, 0, 0, 256, nullptr, tables, s);
  if (st) return st;
  mark(s);
  st = launch_fill_keys(c, s);
  mark(s);
  return st;
}

extern "C" int b2k_render_chunked(const B2kModel* m, const B2kCamera* cam, const B2kRenderOpts* o, const B2kCtx* c, b2k_stream_t stream) {
  B2K_REQUIRE(m && cam && o && c);
  const int C = c->n_chunks;
  B2K_REQUIRE(C >= 2 && C <= MAX_CHUNKS && c->chunk_words && c->last_idx && c->tile_off && c->depth_keys);
  B2K_REQUIRE(!o->bwd_info || c->bwd_scratch);
  if (o->bwd_info && c->bwd_scratch_bytes < b2k_bwd_scratch_bytes(c->W, c->H, C, c->isect_cap)) return B2K_ERR_CAPACITY;
  if (o->feat_mode != 0) {   // out_feat.xyz carries the colour sums between chunks: the feature sums ride in the backward's scratch
    if (o->bwd_info) return B2K_ERR_UNSUPPORTED;
    B2K_REQUIRE(o->feat_mode >= 1 && o->feat_mode <= 2 && c->proj3 && c->bwd_scratch && (o->feat_mode != 2 || o->feat_buffer));
    if (c->bwd_scratch_bytes < sizeof(float4) * (uint64_t)c->W * (uint64_t)c->H) return B2K_ERR_CAPACITY;
  }
  B2K_REQUIRE(c->tile_ranges && c->num_isect && c->n_tiles == c->tiles_x * c->tiles_y && c->tile_bits >= 1 && c->tile_bits <= 24);
  B2K_REQUIRE(c->out_rgba && c->out_feat && c->keys && c->vals && c->keys_sorted && c->vals_sorted && c->sort_tmp);
  cudaStream_t s = (cudaStream_t)stream;
  const int n = m->n;
  B2K_REQUIRE(n >= 0 && m->cap >= n && m->degree >= 0 && m->degree <= 4 && c->proj0 && c->proj1 && c->proj2 && c->tile_count && c->hit_info);
  B2K_REQUIRE(c->depth_keys_sorted && c->order && c->order_in);
  B2K_REQUIRE(cam->W == c->W && cam->H == c->H && c->tiles_x == div_up(c->W, RT_W) && c->tiles_y == div_up(c->H, RT_W));
  int st = B2K_OK;
  if (n > 0) {
    B2K_REQUIRE(m->pos_op && m->quat && m->lscale && m->sh_dc && (m->degree == 0 || m->sh_hi));
    if (c->n_cap < n) return B2K_ERR_CAPACITY;
    st = launch_project_lite(m, cam, o, c, s);
    if (st) return st;
  }
  uint32_t* words = c->chunk_words;
  unsigned long long* alive = (unsigned long long*)(words + CW_WORDS);
  if (n == 0) {
    B2K_CUDA(cudaMemsetAsync(c->tile_ranges, 0, sizeof(uint32_t) * 2 * (size_t)c->n_tiles * C, s));
    B2K_CUDA(cudaMemsetAsync(c->num_isect, 0, sizeof(uint32_t), s));
    for (int ch = 0; ch < C; ch++) { st = launch_raster_fwd(c, o, ch, C, alive, s); if (st) return st; }
    return B2K_OK;
  }
  if (c->sort_tmp_bytes < b2k_sort_tmp_bytes(c->n_cap, c->isect_cap) || c->isect_cap == 0 || c->isect_cap > 0x7FFFFFF0ull) return B2K_ERR_CAPACITY;
  uint32_t* tables = sort_tables_ptr(c);
  st = depth_sort(c, n, tables, s);   // exactly as in b2k_bin_sort
  if (st) return st;
  const int bins = div_up(c->tiles_x, 8) * div_up(c->tiles_y, 8);
  chunk_prepare_kernel<<<div_up(bins, 256), 256, 0, s>>>(c->depth_keys_sorted, n, words, alive, bins);
  for (int ch = 0; ch < C; ch++) {
    const int lo = ch == 0 ? 0 : 256 >> (2 * (C - ch)), hi = 256 >> (2 * (C - 1 - ch));
    st = launch_bins(c, n, words, ch, lo, hi, ch == 0 ? nullptr : alive, tables, s);   // the first chunk meets only live tiles
    if (st) return st;
    st = launch_raster_fwd(c, o, ch, C, alive, s);
    if (st) return st;
  }
  return B2K_OK;
}

extern "C" int b2k_bin_sort_profile(const B2kCtx* c, int32_t n, b2k_stream_t stream, float* ms) {
  B2K_REQUIRE(c && ms);
  Marks& mk = g_marks;
  for (int i = 0; i < 32; i++) B2K_CUDA(cudaEventCreate(&mk.ev[i]));
  mk.n = 0; mk.armed = true;
  const int st = b2k_bin_sort(c, n, stream);
  mk.armed = false;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  // Marks: start, then a pair per depth pass (after count + rows, after scatter), depth sort done, lists done, keys done.
  const int expect = 1 + 2 * sort_passes(32) + 3;
  for (int i = 0; i < 10; i++) ms[i] = 0.f;
  if (st == B2K_OK && e == cudaSuccess && mk.n == expect && n > 0) {
    auto dt = [&](int a, int b) { float t = 0.f; cudaEventElapsedTime(&t, mk.ev[a], mk.ev[b]); return t; };
    ms[0] = dt(0, expect - 3); ms[1] = dt(expect - 3, expect - 2); ms[8] = dt(expect - 2, expect - 1); ms[9] = dt(0, expect - 1);
  }
  for (int i = 0; i < 32; i++) cudaEventDestroy(mk.ev[i]);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return B2K_ERR_CUDA; }
  return st;
}

// The radix sort above for callers outside the binning (the refinement pass): stable, ascending, 32-bit keys, four
// passes, so the result returns to the pair it started from.
extern "C" int32_t b2k_sort_passes(int32_t bits) { return bits >= 1 && bits <= 32 ? sort_passes(bits) : 0; }

extern "C" uint64_t b2k_sort_pairs_tmp_bytes(void) { return (uint64_t)sizeof(uint32_t) * ((uint64_t)RADIX_MAX * 1024 + RADIX_MAX + 1024 + 16); }

extern "C" int b2k_sort_pairs_u32(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t n, void* tmp, uint64_t tmp_bytes, b2k_stream_t stream) {
  B2K_REQUIRE(n == 0 || (keys && vals && keys_alt && vals_alt && tmp));
  if (n == 0) return B2K_OK;
  if (tmp_bytes < b2k_sort_pairs_tmp_bytes() || n > 0xFFFFFFF0u) return B2K_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  const int blocks = sort_blocks();
  const SortScratch sc = carve((uint32_t*)tmp, blocks);
  set_word_kernel<<<1, 1, 0, s>>>(sc.n_word, n);
  return radix_sort(keys, vals, keys_alt, vals_alt, sc.n_word, n, 32, sc, blocks, s);
}

extern "C" int b2k_read_num_isect(const B2kCtx* c, b2k_stream_t stream, uint32_t* total) {
  B2K_REQUIRE(c && c->num_isect && total);
  cudaStream_t s = (cudaStream_t)stream;
  B2K_CUDA(cudaMemcpyAsync(total, c->num_isect, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  B2K_CUDA(cudaStreamSynchronize(s));
  return *total > c->isect_cap ? B2K_ERR_OVERFLOW : B2K_OK;
}

// ---------------------------------------------------------------------------------------------------------------
// Binning without any allocation on the caller's side.
//
// b2k_bin_sort needs a scratch buffer (ctx->sort_tmp) that somebody has to cudaMalloc. Some hosts of this library
// cannot: a plugin loaded into a process whose memory pool is owned and fully reserved by the host application, a
// render thread that must never take the allocator's lock, or a caller inside a region where the CUDA allocator is
// off limits. For them the same scratch lives here, inside the library image, as a fixed device array. It is sized
// for contexts of at most B2K_STATIC_MAX_SPLATS per-splat entries (about 3.2 MB, held by every GPU that loads the
// library, until the process exits).
// ---------------------------------------------------------------------------------------------------------------
namespace b2k {
namespace {
constexpr uint32_t STATIC_MAX_SPLATS = 262144;
constexpr size_t STATIC_WORDS = sort_tmp_words(STATIC_MAX_SPLATS);
static __device__ __align__(256) uint32_t g_static_sort_tmp[STATIC_WORDS];
// Device address of the array above, per device. In host code the array's name is only a handle for the runtime,
// never a pointer a kernel may be given; the address has to be asked for, once per device, with that device current.
void* g_static_addr[64] = {nullptr};
}  // namespace
}  // namespace b2k

extern "C" uint32_t b2k_static_max_splats(void) { return b2k::STATIC_MAX_SPLATS; }

extern "C" int b2k_bin_sort_static(const B2kCtx* c, int32_t n, b2k_stream_t stream) {
  B2K_REQUIRE(c && n >= 0);
  if (c->n_cap < 0 || (uint32_t)c->n_cap > STATIC_MAX_SPLATS || (uint32_t)n > STATIC_MAX_SPLATS) return B2K_ERR_CAPACITY;
  int dev = 0;
  B2K_CUDA(cudaGetDevice(&dev));
  B2K_REQUIRE(dev >= 0 && dev < 64);
  if (!g_static_addr[dev]) {   // first call on this device: resolve the array's device address
    void* p = nullptr;
    B2K_CUDA(cudaGetSymbolAddress(&p, g_static_sort_tmp));
    B2K_REQUIRE(p != nullptr);
    g_static_addr[dev] = p;
  }
  B2kCtx local = *c;            // same buffers, scratch redirected to the library's own array
  local.sort_tmp = g_static_addr[dev];
  local.sort_tmp_bytes = sizeof(uint32_t) * STATIC_WORDS;
  return b2k_bin_sort(&local, n, stream);
}
