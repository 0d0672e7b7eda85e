// Entry points of the binning stage and of the front-to-back chunked renderer. Reference semantics: bin_and_sort
// (src/gpu/binning.cu:109-145). Depth order: sort.cu; from depth order to the tiles' lists: bins.cu, in small whole views walk.cu. No host round
// trip: every count stays on the device, so a view is one asynchronous chain.
#include "common.cuh"
#include <algorithm>

namespace b2k {
namespace {

// Optional timing marks for b2k_bin_sort_profile: when armed, an event is recorded on the stream at each mark.
constexpr int MARKS = 4;   // start, depth sort done, lists done, keys done
struct Marks { cudaEvent_t ev[MARKS]; int n = 0; bool armed = false; };
thread_local Marks g_marks;
void mark(cudaStream_t s) { if (g_marks.armed && g_marks.n < MARKS) cudaEventRecord(g_marks.ev[g_marks.n++], s); }

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
  after_previous();
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
  for (int k = CW_LONGEST; k < CW_COUNT; k++) words[k] = 0u;
  for (int k = CW_LONG; k < CW_WORDS; k++) words[k] = 0u;
}

}  // namespace
}  // namespace b2k

using namespace b2k;

namespace b2k {
namespace {
constexpr uint64_t sort_tmp_words(uint64_t n_cap) { return TMP_HEADER_WORDS + n_cap + BINS_TABLE_WORDS + BINS_EXTRA_WORDS; }
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
    B2K_CUDA(cudaMemsetAsync(c->num_isect + NI_LONGEST, 0, sizeof(uint32_t), s));
    return B2K_OK;
  }
  B2K_REQUIRE(c->proj0 && c->proj1 && c->tile_count && c->hit_info && c->depth_keys && c->depth_keys_sorted && c->order_in && c->order && c->tile_off);
  B2K_REQUIRE(c->keys && c->vals && c->keys_sorted && c->vals_sorted && c->sort_tmp);
  if (c->n_cap < n) return B2K_ERR_CAPACITY;
  if (c->sort_tmp_bytes < b2k_sort_tmp_bytes(c->n_cap, c->isect_cap) || c->isect_cap == 0 || c->isect_cap > 0xFFFFFFF0ull) return B2K_ERR_CAPACITY;
  uint32_t* tables = sort_tables_ptr(c);
  // 1. Splats by depth: key = bits of view z (culled splats carry 0xFFFFFFFF and land last), value = index.
  mark(s);
  int st = depth_sort(c, n, false, walks(c, n), tables, s);   // a view is binned again after its buffers have grown
  if (st) return st;
  mark(s);
  // 2. Hits to the tiles' lists, depth order surviving inside each tile; 3. the tile ids of the list.
  st = launch_bins(c, n, nullptr, 0, 0, 256, nullptr, nullptr, tables, s);
  if (st) return st;
  mark(s);
  if (!walks(c, n)) st = launch_fill_keys(c, s);
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
  unsigned long long* alive = (unsigned long long*)(((uintptr_t)(words + CW_WORDS) + 7) & ~(uintptr_t)7);   // the caller's array may start at any word
  const int bins = div_up(c->tiles_x, 8) * div_up(c->tiles_y, 8);
  uint32_t* tiles = (uint32_t*)(alive + bins);
  if (n == 0) {
    B2K_CUDA(cudaMemsetAsync(c->tile_ranges, 0, sizeof(uint32_t) * 2 * (size_t)c->n_tiles * C, s));
    B2K_CUDA(cudaMemsetAsync(c->num_isect, 0, sizeof(uint32_t), s));
    B2K_CUDA(cudaMemsetAsync(words, 0, sizeof(uint32_t) * CW_WORDS, s));   // no tile of any chunk has a list
    for (int ch = 0; ch < C; ch++) { st = launch_raster_fwd(c, o, ch, C, alive, lists_tiles(c, ch) ? tiles : nullptr, s); if (st) return st; }
    return B2K_OK;
  }
  if (c->sort_tmp_bytes < b2k_sort_tmp_bytes(c->n_cap, c->isect_cap) || c->isect_cap == 0 || c->isect_cap > 0x7FFFFFF0ull) return B2K_ERR_CAPACITY;
  uint32_t* tables = sort_tables_ptr(c);
  st = depth_sort(c, n, true, false, tables, s);
  if (st) return st;
  launch_next(chunk_prepare_kernel, div_up(bins, 256), 256, 0, s, c->depth_keys_sorted, n, words, alive, bins);
  for (int ch = 0; ch < C; ch++) {
    const int lo = ch == 0 ? 0 : 256 >> (2 * (C - ch)), hi = 256 >> (2 * (C - 1 - ch));
    st = launch_bins(c, n, words, ch, lo, hi, ch == 0 ? nullptr : alive, lists_tiles(c, ch) ? tiles : nullptr, tables, s);   // the first chunk meets only live tiles
    if (st) return st;
    st = launch_raster_fwd(c, o, ch, C, alive, lists_tiles(c, ch) ? tiles : nullptr, s);
    if (st) return st;
  }
  return B2K_OK;
}

extern "C" int b2k_bin_sort_profile(const B2kCtx* c, int32_t n, b2k_stream_t stream, float* ms) {
  B2K_REQUIRE(c && ms);
  Marks& mk = g_marks;
  for (int i = 0; i < MARKS; i++) B2K_CUDA(cudaEventCreate(&mk.ev[i]));
  mk.n = 0; mk.armed = true;
  const int st = b2k_bin_sort(c, n, stream);
  mk.armed = false;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  for (int i = 0; i < 10; i++) ms[i] = 0.f;
  if (st == B2K_OK && e == cudaSuccess && mk.n == MARKS && n > 0) {
    auto dt = [&](int a, int b) { float t = 0.f; cudaEventElapsedTime(&t, mk.ev[a], mk.ev[b]); return t; };
    ms[0] = dt(0, 1); ms[1] = dt(1, 2); ms[8] = dt(2, 3); ms[9] = dt(0, 3);
  }
  for (int i = 0; i < MARKS; i++) cudaEventDestroy(mk.ev[i]);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return B2K_ERR_CUDA; }
  return st;
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
// for contexts of at most B2K_STATIC_MAX_SPLATS per-splat entries (about 3.8 MB, held by every GPU that loads the
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
