// Stable sorts of 32-bit keys with 32-bit values: the splats by depth (the first library sort of bin_and_sort,
// src/gpu/binning.cu:109-116), and pairs for the refinement pass. Order = ascending (key, original position).
//
//  * Depth keys are float bits of positive depths, plus 0xFFFFFFFF for culled splats. They are sorted as (key - smallest key),
//    culled ones as largest + 1: the depths of a scene span 23 to 28 bits, so three digits of eight to ten bits do what four
//    passes over 32 bits did, whatever the range (three digits of eleven hold all 32 bits). The range is found on the device.
//  * Up to SMALL_N splats: one block sorts in its shared memory, one launch.
//  * Up to CLUSTER_N: one cluster of eight blocks, one launch. Whole sort, us, one block or ten launches / the cluster: 3,000 splats 17.7 /
//    15.9, 8,000 26.3 / 17.7, 16,000 30.3 / 20.1, 24,000 30.4 / 23.3, 32,000 31.0 / 27.5; 40,000 31.6 / 43.5 (and 2,000 13.0 / 15.1).
//    Sixteen blocks take 4 us more to launch and gain nothing.
//  * Above: three passes of the wait-free form (digit counts per block, scan over the blocks, ranked scatter); no block waits
//    for another. A block owns one contiguous run. Scatter is staged through shared memory so that global writes go out in
//    digit runs. Values that are the positions are not read.
// Bound by latency (launches, barriers) up to a few hundred thousand splats, by the scatter's issue and writes above. Against
// four passes of eight bits with tiles of 4,096 at every size, first launch to last: 2,000 splats 89 -> 12 us, 100,000 94 ->
// 52, 500,000 103 -> 64, three million 176 -> 132, six million 254 -> 204.
#include "bins.cuh"
#include <cooperative_groups.h>
#include <algorithm>

namespace b2k {
namespace {

constexpr uint32_t CULLED = 0xFFFFFFFFu;
constexpr int MAX_RADIX = 2048;             // eleven bits: any keys; depths that this library projected fit ten (see DEPTH_RADIX)
constexpr int DEPTH_RADIX = 1024;           // the projection keeps depths of 0.01 .. 1e10: 29 bits of range, three digits of ten

__device__ __forceinline__ uint32_t warp_incl(uint32_t v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(FULL, v, o); if (lane >= o) v += u; }
  return v;
}

// walk.cu's tile totals are zero when its kernels begin: a kernel of the sort clears them on the way (nullptr: no walk follows).
__device__ __forceinline__ void clear_totals(uint32_t* totals) {
  if (totals) for (int i = threadIdx.x; i < WALK_TILES; i += blockDim.x) totals[i] = 0u;
}

// How keys are cut into digits: `compress` from the range of the keys, else plain bytes.
struct Digits { uint32_t lo, span; int width; };   // sorted as key - lo; culled ones as span
__device__ __forceinline__ uint32_t compressed(uint32_t key, const Digits& d) { return key == CULLED ? d.span : key - d.lo; }
// lo <= hi: range of the keys that are not culled; lo > hi: there are none.
__device__ __forceinline__ Digits digits_of(uint32_t lo, uint32_t hi, int passes) {
  Digits d;
  d.lo = lo <= hi ? lo : 0u; d.span = lo <= hi ? hi - lo + 1u : 0u;   // hi < CULLED, so the span fits
  const int bits = 32 - __clz((int)d.span);
  d.width = max(8, (bits + passes - 1) / passes);
  return d;
}

// ---- one block -----------------------------------------------------------------------------------------------------------
constexpr int SMALL_THREADS = 1024, SMALL_WARPS = 32, SMALL_ITEMS = 2, SMALL_N = SMALL_THREADS * SMALL_ITEMS;

// A warp owns a contiguous run of 32 * ITEMS pairs, held in registers from one pass to the write of the next; pair j * 32 + l
// of the run is lane l's j-th.
__global__ void __launch_bounds__(SMALL_THREADS) small_sort_kernel(const uint32_t* keys, const uint32_t* vals, int n, uint32_t* keys_out, uint32_t* vals_out, uint32_t* totals) {   // may work in place
  after_previous();
  constexpr int ITEMS = SMALL_ITEMS;
  __shared__ uint32_t s_key[SMALL_N], s_val[SMALL_N], s_base[256];                 // s_base: first place of each digit
  __shared__ __align__(4) uint16_t s_cnt[SMALL_WARPS * 256];                       // [warp][256]: digit counts, then offsets inside the digit
  __shared__ uint32_t s_red[2][SMALL_WARPS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int first = warp * (32 * ITEMS) + lane;
  clear_totals(totals);
  uint32_t key[ITEMS], val[ITEMS], lo = CULLED, hi = 0u;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const int i = first + j * 32;
    key[j] = i < n ? keys[i] : CULLED;      // the fill sorts behind everything: culled, and later in the input
    val[j] = vals && i < n ? vals[i] : (uint32_t)i;
    if (key[j] != CULLED) { lo = min(lo, key[j]); hi = max(hi, key[j]); }
  }
  lo = __reduce_min_sync(FULL, lo); hi = __reduce_max_sync(FULL, hi);
  if (lane == 0) { s_red[0][warp] = lo; s_red[1][warp] = hi; }
  __syncthreads();
  lo = __reduce_min_sync(FULL, s_red[0][lane]); hi = __reduce_max_sync(FULL, s_red[1][lane]);
  const Digits d = digits_of(lo, hi, 4);
  const int bits = max(1, 32 - __clz((int)d.span));
  for (int shift = 0; shift < bits; shift += 8) {
    uint32_t* my_cnt = reinterpret_cast<uint32_t*>(s_cnt + warp * 256);
#pragma unroll
    for (int k = 0; k < 4; k++) my_cnt[lane + k * 32] = 0u;
    __syncwarp();
    uint32_t rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const uint32_t g = (compressed(key[j], d) >> shift) & 255u;
      uint32_t peers = FULL;   // lanes with the same digit: one vote per digit bit
#pragma unroll
      for (int b = 0; b < 8; b++) { const bool bit = (g >> b) & 1u; const uint32_t vote = __ballot_sync(FULL, bit); peers &= bit ? vote : ~vote; }
      const uint32_t before = s_cnt[warp * 256 + g];
      rank[j] = before + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (lane == __ffs(peers) - 1) s_cnt[warp * 256 + g] = (uint16_t)(before + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // Digit t's counts over the warps become offsets inside the digit; the digits' totals become first places.
    if (tid < 256) {
      uint32_t sum = 0;
#pragma unroll 8
      for (int w = 0; w < SMALL_WARPS; w++) { const uint32_t c = s_cnt[w * 256 + tid]; s_cnt[w * 256 + tid] = (uint16_t)sum; sum += c; }
      const uint32_t incl = warp_incl(sum);
      if (lane == 31) s_red[0][warp] = incl;
      s_base[tid] = incl - sum;
    }
    __syncthreads();
    if (tid < 256) { uint32_t pre = 0; for (int w = 0; w < warp; w++) pre += s_red[0][w]; s_base[tid] += pre; }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const uint32_t g = (compressed(key[j], d) >> shift) & 255u;
      const uint32_t at = s_base[g] + s_cnt[warp * 256 + g] + rank[j];
      s_key[at] = key[j]; s_val[at] = val[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) { key[j] = s_key[first + j * 32]; val[j] = s_val[first + j * 32]; }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < ITEMS; j++) { const int i = first + j * 32; if (i < n) { keys_out[i] = key[j]; vals_out[i] = val[j]; } }
}

// ---- one cluster ---------------------------------------------------------------------------------------------------------
// Eight blocks of a cluster hold the pairs in their registers and shared memory from the first pass to the last: digit totals and the
// pairs themselves cross between them in distributed shared memory, two barriers of the cluster a pass. Block b owns the places
// b * THREADS * ITEMS .. of the sorted order.
constexpr int CLUSTER = 8, CLUSTER_N = CLUSTER * SMALL_THREADS * 4;
constexpr size_t cluster_smem(int items) { return (size_t)SMALL_THREADS * items * 8 + SMALL_WARPS * 256 * 2; }

template <int ITEMS>
__global__ void __launch_bounds__(SMALL_THREADS) cluster_sort_kernel(const uint32_t* keys, const uint32_t* vals, int n, uint32_t* keys_out, uint32_t* vals_out, uint32_t* totals) {   // may work in place
  after_previous();
  namespace cg = cooperative_groups;
  constexpr uint32_t SHARE = SMALL_THREADS * ITEMS;
  extern __shared__ __align__(16) uint32_t s_mem[];
  uint2* s_pair = reinterpret_cast<uint2*>(s_mem);
  uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_pair + SHARE);   // [warp][256]: digit counts, then offsets inside the block's digit
  __shared__ uint32_t s_tot[256], s_base[256], s_red[2][SMALL_WARPS], s_range[2];
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t me = cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t first = warp * (32 * ITEMS) + lane, lane_lt = (1u << lane) - 1u;
  if (me == CLUSTER - 1u) clear_totals(totals);
  uint32_t key[ITEMS], val[ITEMS], lo = CULLED, hi = 0u;
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const uint32_t i = me * SHARE + first + j * 32;
    key[j] = i < (uint32_t)n ? keys[i] : CULLED;      // the fill sorts behind everything: culled, and later in the input
    val[j] = vals && i < (uint32_t)n ? vals[i] : i;
    if (key[j] != CULLED) { lo = min(lo, key[j]); hi = max(hi, key[j]); }
  }
  lo = __reduce_min_sync(FULL, lo); hi = __reduce_max_sync(FULL, hi);
  if (lane == 0) { s_red[0][warp] = lo; s_red[1][warp] = hi; }
  __syncthreads();
  if (warp == 0) {
    lo = __reduce_min_sync(FULL, s_red[0][lane]); hi = __reduce_max_sync(FULL, s_red[1][lane]);
    if (lane == 0) { s_range[0] = lo; s_range[1] = hi; }
  }
  cluster.sync();
  {
    const uint32_t* of = cluster.map_shared_rank(s_range, lane & (CLUSTER - 1));
    lo = __reduce_min_sync(FULL, of[0]); hi = __reduce_max_sync(FULL, of[1]);
  }
  const Digits d = digits_of(lo, hi, 4);
  const int bits = max(1, 32 - __clz((int)d.span));
  uint16_t* my_cnt = s_cnt + warp * 256;
  for (int shift = 0; shift < bits; shift += 8) {
#pragma unroll
    for (int k = 0; k < 4; k++) reinterpret_cast<uint32_t*>(my_cnt)[lane + k * 32] = 0u;
    __syncwarp();
    uint32_t rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const uint32_t g = (compressed(key[j], d) >> shift) & 255u;
      uint32_t peers = FULL;   // lanes with the same digit: one vote per digit bit
#pragma unroll
      for (int b = 0; b < 8; b++) { const bool bit = (g >> b) & 1u; const uint32_t vote = __ballot_sync(FULL, bit); peers &= bit ? vote : ~vote; }
      const uint32_t before = my_cnt[g];
      rank[j] = before + __popc(peers & lane_lt);
      __syncwarp();
      if (lane == __ffs(peers) - 1) my_cnt[g] = (uint16_t)(before + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // The warps' counts of a digit become offsets inside the block's; the block's totals are there for the others to read.
    if (tid < 256) {
      uint32_t sum = 0;
#pragma unroll 8
      for (int w = 0; w < SMALL_WARPS; w++) { const uint32_t c = s_cnt[w * 256 + tid]; s_cnt[w * 256 + tid] = (uint16_t)sum; sum += c; }
      s_tot[tid] = sum;
    }
    cluster.sync();            // (and the pairs of the pass before have been read)
    uint32_t base = 0;
    if (tid < 256) {
      uint32_t all = 0, before = 0;
#pragma unroll
      for (int c = 0; c < CLUSTER; c++) { const uint32_t t = cluster.map_shared_rank(s_tot, c)[tid]; before += (uint32_t)c < me ? t : 0u; all += t; }
      const uint32_t incl = warp_incl(all);
      if (lane == 31) s_red[0][warp] = incl;
      base = incl - all + before;
    }
    __syncthreads();
    if (tid < 256) { for (int w = 0; w < warp; w++) base += s_red[0][w]; s_base[tid] = base; }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const uint32_t g = (compressed(key[j], d) >> shift) & 255u, at = s_base[g] + my_cnt[g] + rank[j];
      cluster.map_shared_rank(s_pair, at / SHARE)[at % SHARE] = make_uint2(key[j], val[j]);
    }
    cluster.sync();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) { const uint2 p = s_pair[first + j * 32]; key[j] = p.x; val[j] = p.y; }
  }
#pragma unroll
  for (int j = 0; j < ITEMS; j++) { const uint32_t i = me * SHARE + first + j * 32; if (i < (uint32_t)n) { keys_out[i] = key[j]; vals_out[i] = val[j]; } }
}

// ---- many blocks ---------------------------------------------------------------------------------------------------------
constexpr int CNT_THREADS = 256;
constexpr int MAX_BLOCKS = 320;                 // MAX_RADIX * MAX_BLOCKS words of table
static_assert((size_t)MAX_RADIX * MAX_BLOCKS <= BINS_TABLE_WORDS, "the sort and the binning share one table");

struct Range { uint32_t lo[MAX_BLOCKS], hi[MAX_BLOCKS]; Digits digits; };   // per block of key_range_kernel; then what follows from them
// Elements a block owns: whole tiles of `tile` pairs.
__device__ __forceinline__ uint32_t run_of(uint32_t n, uint32_t blocks, uint32_t tile) { return ((n + blocks - 1) / blocks + tile - 1) / tile * tile; }

// Keys are read four at a time where the caller's array allows it.
__device__ __forceinline__ bool by_quads(const uint32_t* keys) { return ((uintptr_t)keys & 15u) == 0u; }

__global__ void __launch_bounds__(CNT_THREADS) key_range_kernel(const uint32_t* __restrict__ keys, uint32_t n, Range* __restrict__ range, uint32_t* __restrict__ totals) {
  after_previous();
  if (blockIdx.x == gridDim.x - 1) clear_totals(totals);
  __shared__ uint32_t s_lo[CNT_THREADS / 32], s_hi[CNT_THREADS / 32];
  uint32_t lo = CULLED, hi = 0u;
  auto see = [&](uint32_t k) { if (k != CULLED) { lo = min(lo, k); hi = max(hi, k); } };
  const uint32_t quads = by_quads(keys) ? n / 4 : 0u, stride = gridDim.x * CNT_THREADS;
#pragma unroll 8
  for (uint32_t q = blockIdx.x * CNT_THREADS + threadIdx.x; q < quads; q += stride) { const uint4 k = reinterpret_cast<const uint4*>(keys)[q]; see(k.x); see(k.y); see(k.z); see(k.w); }
  for (uint32_t i = quads * 4 + blockIdx.x * CNT_THREADS + threadIdx.x; i < n; i += stride) see(keys[i]);
  lo = __reduce_min_sync(FULL, lo); hi = __reduce_max_sync(FULL, hi);
  if ((threadIdx.x & 31) == 0) { s_lo[threadIdx.x >> 5] = lo; s_hi[threadIdx.x >> 5] = hi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < CNT_THREADS / 32; w++) { lo = min(lo, s_lo[w]); hi = max(hi, s_hi[w]); }
    range->lo[blockIdx.x] = lo; range->hi[blockIdx.x] = hi;
  }
}

// The digits of a sort: plain bytes, or from the range that the blocks of key_range_kernel found. The first pass's count works
// it out and leaves it for the kernels behind it. All threads of the block call this.
template <bool COMPRESS>
__device__ __forceinline__ Digits load_digits(Range* __restrict__ range, int range_blocks, int passes, bool work_out) {
  if (!COMPRESS) return Digits{0u, CULLED, 8};
  if (!work_out) return range->digits;
  __shared__ uint32_t s_lo, s_hi;
  if (threadIdx.x < 32) {
    uint32_t lo = CULLED, hi = 0u;
#pragma unroll
    for (int u = 0; u < MAX_BLOCKS / 32; u++) { const int b = u * 32 + threadIdx.x; if (b < range_blocks) { lo = min(lo, range->lo[b]); hi = max(hi, range->hi[b]); } }
    lo = __reduce_min_sync(FULL, lo); hi = __reduce_max_sync(FULL, hi);
    if (threadIdx.x == 0) { s_lo = lo; s_hi = hi; }
  }
  __syncthreads();
  const Digits d = digits_of(s_lo, s_hi, passes);
  if (blockIdx.x == 0 && threadIdx.x == 0) range->digits = d;
  return d;
}
template <bool COMPRESS>
__device__ __forceinline__ uint32_t digit_at(uint32_t key, const Digits& d, int pass) {
  const int shift = pass * d.width;   // the last digit of 32 bits may be cut short by the end of the word
  return (COMPRESS ? compressed(key, d) : key) >> shift & ((1u << d.width) - 1u);
}

// Digit counts of each block's run: table[digit][block]. Narrow digits are counted in several copies, a warp to each, against
// conflicts where few digits occur.
template <bool COMPRESS>
__global__ void __launch_bounds__(CNT_THREADS) digit_count_kernel(const uint32_t* __restrict__ keys, uint32_t n, uint32_t tile, int pass, int passes, Range* __restrict__ range,
                                                                  int range_blocks, uint32_t* __restrict__ table) {
  after_previous();
  __shared__ uint32_t s_hist[MAX_RADIX];
  const Digits d = load_digits<COMPRESS>(range, range_blocks, passes, pass == 0);
  const uint32_t radix = 1u << d.width, copies = min((uint32_t)(CNT_THREADS / 32), MAX_RADIX / radix);
  for (int i = threadIdx.x; i < MAX_RADIX; i += CNT_THREADS) s_hist[i] = 0u;
  __syncthreads();
  uint32_t* hist = s_hist + ((threadIdx.x >> 5) % copies) * radix;
  const uint32_t len = run_of(n, gridDim.x, tile);
  const uint64_t begin64 = (uint64_t)blockIdx.x * len;
  const uint32_t begin = begin64 < n ? (uint32_t)begin64 : n, end = begin64 + len < n ? (uint32_t)(begin64 + len) : n;   // a multiple of four
  const uint32_t whole = by_quads(keys) ? begin + ((end - begin) & ~3u) : begin;
#pragma unroll 4
  for (uint32_t i = begin + threadIdx.x * 4; i < whole; i += CNT_THREADS * 4) {
    const uint4 k = *reinterpret_cast<const uint4*>(keys + i);
    atomicAdd(&hist[digit_at<COMPRESS>(k.x, d, pass)], 1u); atomicAdd(&hist[digit_at<COMPRESS>(k.y, d, pass)], 1u);
    atomicAdd(&hist[digit_at<COMPRESS>(k.z, d, pass)], 1u); atomicAdd(&hist[digit_at<COMPRESS>(k.w, d, pass)], 1u);
  }
  for (uint64_t i = (uint64_t)whole + threadIdx.x; i < end; i += CNT_THREADS) atomicAdd(&hist[digit_at<COMPRESS>(keys[i], d, pass)], 1u);
  __syncthreads();
  for (uint32_t g = threadIdx.x; g < radix; g += CNT_THREADS) {
    uint32_t t = 0;
    for (uint32_t c = 0; c < copies; c++) t += s_hist[c * radix + g];
    table[(size_t)g * gridDim.x + blockIdx.x] = t;
  }
}

// A warp per digit: the blocks' counts become offsets inside the digit; the digit's total is recorded.
constexpr int ROW_WARPS = 16;
template <bool COMPRESS>
__global__ void __launch_bounds__(ROW_WARPS * 32) digit_rows_kernel(uint32_t* __restrict__ table, int blocks, Range* __restrict__ range, uint32_t* __restrict__ totals) {
  after_previous();
  const Digits d = load_digits<COMPRESS>(range, 0, 0, false);
  const int g = blockIdx.x * ROW_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (g >= 1 << d.width) return;
  uint32_t* row = table + (size_t)g * blocks;
  uint32_t c[MAX_BLOCKS / 32], at = 0;
#pragma unroll
  for (int u = 0; u < MAX_BLOCKS / 32; u++) c[u] = u * 32 + lane < blocks ? row[u * 32 + lane] : 0u;
#pragma unroll
  for (int u = 0; u < MAX_BLOCKS / 32; u++) {
    if (u * 32 >= blocks) break;
    const uint32_t incl = warp_incl(c[u]);
    if (u * 32 + lane < blocks) row[u * 32 + lane] = at + incl - c[u];
    at += __shfl_sync(FULL, incl, 31);
  }
  if (lane == 0) totals[g] = at;
}

// Ranked, stable scatter of each block's run, a tile of THREADS * ITEMS pairs at a time. A warp owns 32 * ITEMS consecutive pairs of
// the tile. The next tile's keys are in flight while this one is written out. vals_in == nullptr: the value is the position.
constexpr size_t scat_smem(int most, int threads, int items) { return most * 8 + (size_t)(threads / 32) * most * 2 + (size_t)threads * items * 8; }
template <bool COMPRESS, int MOST, int SCAT_THREADS, int ITEMS>
__global__ void __launch_bounds__(SCAT_THREADS, 2) digit_scatter_kernel(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
                                                                        uint32_t* __restrict__ vals_out, uint32_t n, int pass, Range* __restrict__ range,
                                                                        const uint32_t* __restrict__ table, const uint32_t* __restrict__ totals) {
  after_previous();
  constexpr int SCAT_WARPS = SCAT_THREADS / 32, PER = MOST > SCAT_THREADS ? MOST / SCAT_THREADS : 1;
  constexpr uint32_t TILE = SCAT_THREADS * ITEMS;
  extern __shared__ __align__(16) uint32_t s_mem[];
  uint32_t* s_gbase = s_mem;                      // [radix] running global place of the digit for this block
  uint32_t* s_delta = s_gbase + MOST;        // [radix] global place = s_delta[digit] + place in the tile (mod 2^32)
  uint16_t* s_cnt = reinterpret_cast<uint16_t*>(s_delta + MOST);   // [warp][radix] digit counts, then first places in the tile
  uint32_t* s_keys = reinterpret_cast<uint32_t*>(s_cnt + SCAT_WARPS * MOST);
  uint32_t* s_vals = s_keys + TILE;
  __shared__ uint32_t s_scan[SCAT_WARPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t lane_lt = (1u << lane) - 1u;
  const Digits d = load_digits<COMPRESS>(range, 0, 0, false);
  const int radix = 1 << d.width, per = radix > SCAT_THREADS ? radix / SCAT_THREADS : 1;   // digits per thread: the first radix / per threads hold them
  // Exclusive scan of one value per digit, `per` consecutive digits a thread.
  auto scan_digits = [&](const uint32_t (&v)[PER], uint32_t (&out)[PER]) {
    uint32_t sum = 0;
#pragma unroll
    for (int u = 0; u < PER; u++) { out[u] = sum; sum += u < per ? v[u] : 0u; }
    const uint32_t incl = warp_incl(sum);
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    uint32_t pre = incl - sum;
    for (int w = 0; w < warp; w++) pre += s_scan[w];
#pragma unroll
    for (int u = 0; u < PER; u++) out[u] += pre;
    __syncthreads();
  };
  const bool holder = tid * per < radix;
  {
    uint32_t tot[PER], base[PER];
#pragma unroll
    for (int u = 0; u < PER; u++) tot[u] = holder && u < per ? totals[tid * per + u] : 0u;
    scan_digits(tot, base);
#pragma unroll
    for (int u = 0; u < PER; u++)
      if (holder && u < per) s_gbase[tid * per + u] = base[u] + table[(size_t)(tid * per + u) * gridDim.x + blockIdx.x];
  }
  const uint32_t len = run_of(n, gridDim.x, TILE);
  const uint64_t begin64 = (uint64_t)blockIdx.x * len;
  const uint32_t begin = begin64 < n ? (uint32_t)begin64 : n, end = begin64 + len < n ? (uint32_t)(begin64 + len) : n;
  const uint32_t wbase = warp * (32 * ITEMS);
  uint32_t key[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; j++) { const uint32_t i = begin + wbase + j * 32 + lane; key[j] = i < end ? keys_in[i] : CULLED; }
  for (uint32_t tile = begin; tile < end; tile += TILE) {
    const uint32_t tile_n = min(end - tile, TILE);
    uint32_t val[ITEMS], rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; j++) { const uint32_t i = tile + wbase + j * 32 + lane; val[j] = vals_in ? (i < end ? vals_in[i] : 0u) : i; }
    uint16_t* my_cnt = s_cnt + warp * radix;
    for (int i = lane; i < radix / 2; i += 32) reinterpret_cast<uint32_t*>(my_cnt)[i] = 0u;
    __syncwarp();
    // Rank of every pair among the warp's pairs with the same digit. Pairs beyond the end count too: they come last.
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const uint32_t g = digit_at<COMPRESS>(key[j], d, pass);
      const uint32_t valid = __ballot_sync(FULL, wbase + j * 32 + lane < tile_n);
      uint32_t peers = valid;   // lanes with the same digit: one vote per digit bit
#pragma unroll
      for (int b = 0; b < 8; b++) { const bool bit = (g >> b) & 1u; const uint32_t vote = __ballot_sync(FULL, bit); peers &= bit ? vote : ~vote; }
      if (COMPRESS)
        for (int b = 8; b < d.width; b++) { const bool bit = (g >> b) & 1u; const uint32_t vote = __ballot_sync(FULL, bit); peers &= bit ? vote : ~vote; }
      const uint32_t before = my_cnt[g];
      rank[j] = before + __popc(peers & lane_lt);
      __syncwarp();
      if (lane == __ffs(peers) - 1) my_cnt[g] = (uint16_t)(before + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    {
      uint32_t total[PER], first[PER];
#pragma unroll
      for (int u = 0; u < PER; u++) {
        total[u] = 0u;
        if (holder && u < per)
#pragma unroll
          for (int w = 0; w < SCAT_WARPS; w++) total[u] += s_cnt[w * radix + tid * per + u];
      }
      scan_digits(total, first);
#pragma unroll
      for (int u = 0; u < PER; u++)
        if (holder && u < per) {
          const int g = tid * per + u;
          s_delta[g] = s_gbase[g] - first[u]; s_gbase[g] += total[u];
          uint32_t at = first[u];
#pragma unroll
          for (int w = 0; w < SCAT_WARPS; w++) { const uint32_t c = s_cnt[w * radix + g]; s_cnt[w * radix + g] = (uint16_t)at; at += c; }
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      if (wbase + j * 32 + lane < tile_n) {
        const uint32_t slot = my_cnt[digit_at<COMPRESS>(key[j], d, pass)] + rank[j];
        s_keys[slot] = key[j]; s_vals[slot] = val[j];
      }
    }
#pragma unroll
    for (int j = 0; j < ITEMS; j++) { const uint64_t i = (uint64_t)tile + TILE + wbase + j * 32 + lane; key[j] = i < end ? keys_in[i] : CULLED; }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; j++) {
      const uint32_t slot = j * SCAT_THREADS + tid;
      if (slot < tile_n) {
        const uint32_t k = s_keys[slot], dst = s_delta[digit_at<COMPRESS>(k, d, pass)] + slot;
        keys_out[dst] = k; vals_out[dst] = s_vals[slot];
      }
    }
    __syncthreads();
  }
}

}  // namespace

// Blocks and tile of the multi-block sort. Large inputs: two blocks of 512 threads per SM, tiles of 4,096, so that digit runs
// are long enough to write well. Below what fills those, smaller blocks; and where even they would leave SMs idle, small tiles.
enum Tile { SMALL_TILE = 256 * 2, MIDDLE_TILE = 256 * 8, LARGE_TILE = 512 * 8 };
struct Shape { int blocks, tile; };
Shape shape_of(uint32_t n) {
  const uint32_t most = std::min(2 * sm_count(), MAX_BLOCKS);
  const int tile = n >= most * LARGE_TILE ? LARGE_TILE : n >= most * SMALL_TILE ? MIDDLE_TILE : SMALL_TILE;
  return {(int)std::min<uint32_t>(most, (n + tile - 1) / tile), tile};
}

template <bool COMPRESS, int MOST, int THREADS, int ITEMS>
int scatter(const uint32_t* ki, const uint32_t* vi, uint32_t* ko, uint32_t* vo, uint32_t n, int blocks, int pass, Range* range, const uint32_t* table, const uint32_t* totals,
            cudaStream_t s) {
  static bool attr_set[64] = {false};
  int dev = 0;
  constexpr size_t smem = scat_smem(MOST, THREADS, ITEMS);
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
    B2K_CUDA(cudaFuncSetAttribute(digit_scatter_kernel<COMPRESS, MOST, THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[dev] = true;
  }
  launch_next(digit_scatter_kernel<COMPRESS, MOST, THREADS, ITEMS>, blocks, THREADS, smem, s, ki, vi, ko, vo, n, pass, range, table, totals);
  return check_launch();
}
template <bool COMPRESS, int MOST>
int one_pass(const Shape& sh, const uint32_t* ki, const uint32_t* vi, uint32_t* ko, uint32_t* vo, uint32_t n, int pass, int passes, Range* range, int range_blocks, uint32_t* table,
             uint32_t* totals, cudaStream_t s) {
  launch_next(digit_count_kernel<COMPRESS>, sh.blocks, CNT_THREADS, 0, s, ki, n, (uint32_t)sh.tile, pass, passes, range, range_blocks, table);
  launch_next(digit_rows_kernel<COMPRESS>, MOST / ROW_WARPS, ROW_WARPS * 32, 0, s, table, sh.blocks, range, totals);
  switch (sh.tile) {
    case LARGE_TILE: return scatter<COMPRESS, MOST, 512, 8>(ki, vi, ko, vo, n, sh.blocks, pass, range, table, totals, s);
    case MIDDLE_TILE: return scatter<COMPRESS, MOST, 256, 8>(ki, vi, ko, vo, n, sh.blocks, pass, range, table, totals, s);
    default: return scatter<COMPRESS, MOST, 256, 2>(ki, vi, ko, vo, n, sh.blocks, pass, range, table, totals, s);
  }
}

int small_sort(const uint32_t* keys, const uint32_t* vals, int n, uint32_t* ko, uint32_t* vo, uint32_t* totals, cudaStream_t s) {
  launch_next(small_sort_kernel, 1, SMALL_THREADS, 0, s, keys, vals, n, ko, vo, totals);
  return check_launch();
}

template <int ITEMS>
int cluster_sort(const uint32_t* keys, const uint32_t* vals, int n, uint32_t* ko, uint32_t* vo, uint32_t* totals, cudaStream_t s) {
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
    B2K_CUDA(cudaFuncSetAttribute(cluster_sort_kernel<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cluster_smem(ITEMS)));
    attr_set[dev] = true;
  }
  launch_clustered(CLUSTER, cluster_sort_kernel<ITEMS>, CLUSTER, SMALL_THREADS, cluster_smem(ITEMS), s, keys, vals, n, ko, vo, totals);
  return check_launch();
}

int depth_sort(const B2kCtx* c, int n, bool identity, bool for_walk, uint32_t* tables, cudaStream_t s) {
  const uint32_t* in = c->depth_keys_sorted;
  const uint32_t* index = identity ? nullptr : c->order;
  uint32_t* cleared = for_walk ? bins_tables(tables, nullptr).tile_totals : nullptr;
  uint32_t *k = c->depth_keys_sorted, *v = c->order;   // one block, or one cluster, reads everything before it writes: in place
  if (n <= SMALL_N) return small_sort(in, index, n, k, v, cleared, s);
  if (n <= CLUSTER_N) {
    const int items = div_up(n, CLUSTER * SMALL_THREADS);
    return items <= 1 ? cluster_sort<1>(in, index, n, k, v, cleared, s) : items <= 2 ? cluster_sort<2>(in, index, n, k, v, cleared, s)
           : items <= 3 ? cluster_sort<3>(in, index, n, k, v, cleared, s) : cluster_sort<4>(in, index, n, k, v, cleared, s);
  }
  uint32_t *table = tables, *totals = table + BINS_TABLE_WORDS;
  Range* range = (Range*)(totals + MAX_RADIX);
  static_assert(MAX_RADIX + sizeof(Range) / sizeof(uint32_t) <= MAX_BINS + 2 * (MAX_BINS + 1), "scratch: in front of the counters that outlive the sort");
  const Shape sh = shape_of((uint32_t)n);
  const int range_blocks = std::min<int>(std::min(2 * sm_count(), MAX_BLOCKS), div_up(n, CNT_THREADS * 16));
  launch_next(key_range_kernel, range_blocks, CNT_THREADS, 0, s, in, (uint32_t)n, range, cleared);
  // Three passes by way of two scratch pairs (the second: tile_off and the words per splat, both free here).
  uint32_t* list = splat_words_ptr(c);
  const uint32_t* ki[3] = {in, c->depth_keys, c->tile_off};
  const uint32_t* vi[3] = {index, c->order_in, list};
  uint32_t* ko[3] = {c->depth_keys, c->tile_off, c->depth_keys_sorted};
  uint32_t* vo[3] = {c->order_in, list, c->order};
  for (int p = 0; p < 3; p++) {
    const int st = identity ? one_pass<true, DEPTH_RADIX>(sh, ki[p], vi[p], ko[p], vo[p], (uint32_t)n, p, 3, range, range_blocks, table, totals, s)
                            : one_pass<true, MAX_RADIX>(sh, ki[p], vi[p], ko[p], vo[p], (uint32_t)n, p, 3, range, range_blocks, table, totals, s);   // keys may be a caller's own
    if (st) return st;
  }
  return B2K_OK;
}

}  // namespace b2k

using namespace b2k;

extern "C" int32_t b2k_sort_passes(int32_t bits) {
  if (bits < 1 || bits > 32) return 0;
  const int digit = bits > 16 && bits <= 18 ? 9 : 8;
  return (bits + digit - 1) / digit;
}

extern "C" uint64_t b2k_sort_pairs_tmp_bytes(void) { return (uint64_t)sizeof(uint32_t) * (BINS_TABLE_WORDS + MAX_RADIX); }

// The same passes for callers outside the binning (the refinement pass): plain bytes, four passes, so the result returns to the
// pair it started from.
extern "C" int b2k_sort_pairs_u32(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t n, void* tmp, uint64_t tmp_bytes, b2k_stream_t stream) {
  B2K_REQUIRE(n == 0 || (keys && vals && keys_alt && vals_alt && tmp));
  if (n == 0) return B2K_OK;
  if (tmp_bytes < b2k_sort_pairs_tmp_bytes() || n > 0xFFFFFFF0u) return B2K_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  uint32_t *table = (uint32_t*)tmp, *totals = table + BINS_TABLE_WORDS;
  const Shape sh = shape_of(n);
  for (int p = 0; p < 4; p++) {
    const int st = one_pass<false, 256>(sh, keys, vals, keys_alt, vals_alt, n, p, 4, nullptr, 0, table, totals, s);
    if (st) return st;
    std::swap(keys, keys_alt); std::swap(vals, vals_alt);
  }
  return B2K_OK;
}
