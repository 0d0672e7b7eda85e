// Forward compositing: each 8x8 tile's depth-ordered fragment list is walked front to back. Reference semantics:
// raster_fwd_kernel (src/gpu/raster_fwd.cu:9-71); the optional expected-depth output follows the mean-depth mode of
// probe_kernel (src/gpu/probe.cu:30-46).
//
// Bound by instruction issue where tiles fill the GPU and by the latency of one list where they do not; memory traffic is the
// gather of 48 B per staged fragment, served mostly by L2. Fragments are gathered one batch ahead and staged in shared memory
// as operands of packed arithmetic (fp32x2); the hit test is one comparison; a pixel that does not see a fragment takes it with
// weight zero instead of branching around it (a vote and a branch per fragment cost more than the ten operations they saved).
// Transmittances are multiplied up for a group of fragments first, and fragments are compared and selected one by one only where a
// pixel of the warp closes inside the group (none_closes): 1024x1024 over 1M in four chunks 184 -> 172 us, 4K over 6M in five 681 -> 652.
// Three kernels with the same arithmetic, bit for bit:
//   raster_fwd_team_kernel  eight warps to a tile: some find alphas, two composite, two gather. For whole views of few tiles and the second of two
//                           chunks, where the time is that of the longest list (team_pays).
//   raster_fwd_half_kernel  two warps to a tile, a lane one pixel, two consecutive fragments to a packed operation: the chain of
//                           one list is half as long. For whole views and two chunks, where a visit to a tile is a long list.
//   raster_fwd_kernel       one warp to a tile, a lane two pixels that share packed operations: twice as many tiles in flight.
//                           For three and more depth chunks, whose visits are many and short.
// Measured, us (scalar pixels with a vote / one warp / two warps): 64x64 50 / 38 / 23, 333x217 54 / 42 / 28, 1001x751 with
// features 85 / 69 / 54, 1237x822 in two chunks 117 / 92 / 76, 1920x1080 in two 143 / 123 / 118; 1024x1024 over 1M in four
// 231 / 187 / 206, 4K over 6M with depth in five 847 / 740 / 953, sixteen views of 3M in four on eight streams 20.6 / 21.6 ms.
// Two warps / the team, us: 64x64 over 2k splats 21.3 / 15.1, 200x150 over 1k 11.7 / 9.9, 333x217 over 1k 11.8 / 10.0, over 20k 24.7 /
// 18.7, over 150k 78 / 50 (1,176 tiles, a block each); 400x300 over 4k 12.9 / 16.1, over 40k 25.3 / 26.3 (1,900 tiles),
// 512x512 over 10k 17.8 / 31.7, 1280x720 over 100k 40.7 / 70.7.
#include "common.cuh"

namespace b2k {
namespace {

constexpr int FWD_WARPS = 4;
constexpr int FWD_TILES = FWD_WARPS / 2;                 // of a block of raster_fwd_half_kernel
constexpr int FWD_BATCH = 64, FWD_SEG = 32;              // fragments staged at a time; between possible checkpoints
static_assert(FWD_SEG == 1 << SEG_SHIFT_MIN, "checkpoints");
constexpr int FWD_GROUP = 4;                             // fragments (one warp) or pairs of fragments (two) whose state-independent math is issued together

// CHUNKED: the view is composited in depth chunks (chunk `chunk` of `n_chunks`, one launch each, nearest first). Between
// launches a pixel's state lives in the output buffers: the colour sums in out_feat.xyz, the transmittance in
// out_feat.w, and last_idx with bit 31 set once the pixel has reached the cutoff; out_rgba holds the finished pixel
// after every chunk, so a launch only touches tiles that received fragments. With DEPTH the depth sum travels in
// out_depth, and the last chunk divides it out in every pixel, which is all it does in a tile that it leaves nothing in (the last of five
// visits to a 4K view 183 -> 130 us). The tile's bit in `alive` tells the binning of the next
// chunk whether any pixel of the tile can still take a fragment.
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Barrier of the 64 threads of a tile; whether `p` holds for any of them.
__device__ __forceinline__ bool pair_any(int id, bool p) {
  uint32_t r;
  asm volatile("{ .reg .pred p, q; setp.ne.u32 p, %1, 0; barrier.cta.red.or.pred q, %2, 64, p; selp.u32 %0, 1, 0, q; }" : "=r"(r) : "r"((uint32_t)p), "r"(id) : "memory");
  return r != 0u;
}

// Expected depth from the depth sum of a pixel and its transmittance.
__device__ __forceinline__ float finished_depth(float zs, float T) { return (1.f - T) > 0.05f ? zs / (1.f - T) : INFINITY; }

constexpr uint32_t DONE_BIT = 0x80000000u;

// A pixel carries its transmittance while it is open and zero once it has closed (the last value then waits in a variable of its own).
// So a group of fragments multiplies up the transmittances first, one operation a fragment, and only if some pixel of the warp closes
// inside the group (the product passes the cut-off: it never rises again) are fragments compared and selected one by one. Whether none does,
// from the transmittances before and behind a group of N: what an open pixel has left behind eight fragments is at least 1e-4 * (1 - 0.999)^8, far from
// zero, so that zero says "closed before". Behind sixteen fragments at the clamp it is below the smallest float, and the pixel itself is asked
// (the team: 64x64 over 2k splats 15.0 us with either test, 333x217 over 20k 18.8 and 18.7).
template <int N>
__device__ __forceinline__ bool none_closes(float before, float behind) {
  if constexpr (N <= 8) return __float_as_uint(behind) - 1u >= __float_as_uint(T_CUTOFF);   // zero, or above the cut-off
  else return before == 0.f || behind > T_CUTOFF;
}

// Two fragments that follow each other in a list, the nearer in the first of each pair of lanes.
constexpr int STAGED = 5;   // (-x, -y), (c00 / 2, c01), (c11 / 2, opacity), (power, r), (g, b); then (z, feature 0), (feature 1, 2)
// Alpha of the two at the lane's pixel, zero where it does not see one.
__device__ __forceinline__ float2 pair_alpha(const float4& q0, const float4& q1, const float4& q2, float2 power, float2 pcx, float2 pcy) {
  const float2 dx = __fadd2_rn(pcx, lo2(q0)), dy = __fadd2_rn(pcy, hi2(q0));
  const float2 sigma = __ffma2_rn(dx, __ffma2_rn(dx, lo2(q1), __fmul2_rn(hi2(q1), dy)), __fmul2_rn(__fmul2_rn(lo2(q2), dy), dy));
  const float2 e = __fmul2_rn(sigma, make_float2(-1.4426950408889634f, -1.4426950408889634f));
  const float2 al = __fmul2_rn(hi2(q2), make_float2(fast_ex2(e.x), fast_ex2(e.y)));
  // alpha >= 1/255 is 0 <= sigma <= power: one comparison of bit patterns (neither is ever -0). The exponent is at most
  // log2(255) in size there, so that flushing denormals changes nothing.
  return make_float2(__float_as_uint(sigma.x) <= __float_as_uint(power.x) ? fminf(ALPHA_MAX, al.x) : 0.f,
                     __float_as_uint(sigma.y) <= __float_as_uint(power.y) ? fminf(ALPHA_MAX, al.y) : 0.f);
}

// The tiles of a chunk that have a list (tile_scan has written them down, see lists_tiles): those with long lists first.
struct TileList {
  const uint32_t* list; uint32_t longs, count; int n_tiles;
  __device__ __forceinline__ int at(uint32_t w) const { return list ? (int)list[w < longs ? w : (uint32_t)n_tiles - 1u - (w - longs)] : (int)w; }
};
__device__ __forceinline__ TileList tile_list(const uint32_t* words, const uint32_t* list, int chunk, int n_tiles) {
  const uint32_t longs = words[CW_LONG + chunk];
  return {list, longs, longs + words[CW_SHORT + chunk], n_tiles};
}

// What the forward leaves for the backward (common.cuh): nothing, checkpoints of the running sums, or of each segment's sums.
enum Checkpoints { NONE = 0, RUNNING = 1, PER_SEGMENT = 2 };

// What the kernels that give a lane one pixel keep of it.
template <int CKPT, bool DEPTH, bool FEAT, bool TRACKED>
struct Pixel {
  float r = 0.f, g = 0.f, b = 0.f, zs = 0.f, f0 = 0.f, f1 = 0.f, f2 = 0.f;   // f: composited feature lanes (raster_fwd.cu:52)
  float sr = 0.f, sg = 0.f, sb = 0.f;   // PER_SEGMENT: colour sums of the segment at hand
  float T = 0.f, T_closed = 1.f;        // transmittance of a pixel that can take another fragment; else zero, and the transmittance it closed with
  uint32_t last = 0u;                   // TRACKED: behind the last fragment the pixel took
  // Adds a fragment that the pixel sees with blend weight `vis` (zero where it does not see it).
  __device__ __forceinline__ void add(float vis, float cr, float cg, float cb, float z, float e0, float e1, float e2, uint32_t end) {
    r += cr * vis; g += cg * vis; b += cb * vis;
    if constexpr (CKPT == PER_SEGMENT) { sr += cr * vis; sg += cg * vis; sb += cb * vis; }
    if constexpr (DEPTH) zs += vis * z;
    if constexpr (FEAT) { f0 += e0 * vis; f1 += e1 * vis; f2 += e2 * vis; }
    if constexpr (TRACKED) last = vis != 0.f ? end : last;
  }
  // The blend weight of a fragment of weight `al` and transmittance `through`, and the pixel's transmittance moved on: the fragment that
  // would saturate a pixel closes it and is not taken.
  __device__ __forceinline__ float weigh(float al, float through) {
    const float next_T = T * through;
    const bool stays = next_T > T_CUTOFF;
    const float vis = stays ? al * T : 0.f;
    T_closed = !stays && T != 0.f ? T : T_closed;
    T = stays ? next_T : 0.f;
    return vis;
  }
  __device__ __forceinline__ float now() const { return T != 0.f ? T : T_closed; }
  // The state before a boundary, for the backward.
  __device__ __forceinline__ void checkpoint(float4* dst) {
    if constexpr (CKPT == PER_SEGMENT) { *dst = make_float4(sr, sg, sb, now()); sr = sg = sb = 0.f; }   // the sums of the segment before the boundary
    else *dst = make_float4(r, g, b, now());
  }
  // 2 * PAIRS fragments in list order; `end`: behind the first. A pixel that does not see a fragment has its transmittance multiplied by
  // one, and its sums take zeros.
  template <int PAIRS, int RECORDS>
  __device__ __forceinline__ void take_pairs(const float2 (&alpha)[PAIRS], const float4 (*staged)[RECORDS], uint32_t end) {
    float2 vis[PAIRS], through[PAIRS];
    float ahead = T;
#pragma unroll
    for (int u = 0; u < PAIRS; u++) {
      through[u] = __fadd2_rn(make_float2(1.f, 1.f), make_float2(-alpha[u].x, -alpha[u].y));
      vis[u].x = alpha[u].x * ahead; ahead *= through[u].x; vis[u].y = alpha[u].y * ahead; ahead *= through[u].y;
    }
    if (__all_sync(0xffffffffu, none_closes<2 * PAIRS>(T, ahead))) T = ahead;
    else {
#pragma unroll
      for (int u = 0; u < PAIRS; u++) { vis[u].x = weigh(alpha[u].x, through[u].x); vis[u].y = weigh(alpha[u].y, through[u].y); }
    }
#pragma unroll
    for (int u = 0; u < PAIRS; u++) {
      const float4* f = staged[u];
      const float2 red = hi2(f[3]);
      const float4 q4 = f[4], q5 = DEPTH || FEAT ? f[RECORDS > 5 ? 5 : 0] : make_float4(0.f, 0.f, 0.f, 0.f), q6 = FEAT ? f[RECORDS > 6 ? 6 : 0] : q5;
      add(vis[u].x, red.x, q4.x, q4.z, q5.x, q5.z, q6.x, q6.z, end + 2 * u);
      add(vis[u].y, red.y, q4.y, q4.w, q5.y, q5.w, q6.y, q6.w, end + 2 * u + 1);
    }
  }
  // The same one by one, for colours or features that are not finite, which may not be added with weight zero. al: the fragment's alpha.
  template <int RECORDS>
  __device__ __forceinline__ void take_odd(float al, const float4* f, int k, uint32_t end) {
    if (al == 0.f || T == 0.f) return;
    const float* c = reinterpret_cast<const float*>(f) + k;
    const float z = DEPTH ? c[RECORDS > 5 ? 20 : 0] : 0.f, e0 = FEAT ? c[RECORDS > 6 ? 22 : 0] : 0.f, e1 = FEAT ? c[RECORDS > 6 ? 24 : 0] : 0.f, e2 = FEAT ? c[RECORDS > 6 ? 26 : 0] : 0.f;
    const float vis = weigh(al, 1.f - al);
    if (vis != 0.f) add(vis, c[14], c[16], c[18], z, e0, e1, e2, end);
  }
};

// A record's place in its staged pair (k: the pair's first or second); whether its colour or a feature is not finite.
template <bool DEPTH, bool FEAT>
__device__ __forceinline__ bool stage_record(float4* pair, int k, const float4& n0, const float4& n1, const float4& n2, const float2& n3) {
  float* s = reinterpret_cast<float*>(pair) + k;
  const float cr = fmaxf(n2.x, 0.f), cg = fmaxf(n2.y, 0.f), cb = fmaxf(n2.z, 0.f);
  s[0] = -n0.x; s[2] = -n0.y; s[4] = 0.5f * n0.z; s[6] = n0.w; s[8] = 0.5f * n1.x; s[10] = n1.y; s[12] = n1.w; s[14] = cr; s[16] = cg; s[18] = cb;
  bool strange = fmaxf(cr, fmaxf(cg, cb)) == INFINITY;
  if constexpr (DEPTH || FEAT) { s[20] = n1.z; s[22] = n2.w; }
  if constexpr (FEAT) { s[24] = n3.x; s[26] = n3.y; strange = strange || !(isfinite(n2.w) && isfinite(n3.x) && isfinite(n3.y)); }
  return strange;
}

// The pixels of the tiles without a list, by blocks of their own behind those that composite: a warp looks at 32 tiles at a time. In the
// first chunk they get the background (a tile with a list that the backward's end has moved back to (0, 0) holds just these values);
// in the last one their depths are finished, which a forward for a backward leaves to the compositing (it moves ranges).
template <bool DEPTH>
__device__ __forceinline__ void visit_unlisted(int block, int blocks, const uint2* __restrict__ tile_ranges, int n_tiles, int tiles_x, int W, int H, float3 bg, bool first,
                                               float4* __restrict__ out_rgba, float4* __restrict__ out_feat, float* __restrict__ out_depth, uint32_t* __restrict__ last_idx) {
  const int lane = threadIdx.x & 31, warps = blocks * FWD_WARPS;
  for (int t0 = (block * FWD_WARPS + (threadIdx.x >> 5)) * 32; t0 < n_tiles; t0 += warps * 32) {
    uint2 range = make_uint2(0u, 1u);
    if (t0 + lane < n_tiles) range = tile_ranges[t0 + lane];
    for (uint32_t todo = __ballot_sync(0xffffffffu, (range.x | range.y) == 0u); todo; todo &= todo - 1u) {
      const int tile = t0 + __ffs(todo) - 1, tx = tile % tiles_x, ty = tile / tiles_x;
      int pix[2];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int px = tx * RT_W + (lane & 7), py = ty * RT_W + (lane >> 3) + h * 4;
        pix[h] = px < W && py < H ? py * W + px : -1;
      }
      if (first) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          if (pix[h] < 0) continue;
          out_rgba[pix[h]] = make_float4(bg.x, bg.y, bg.z, 0.f);
          out_feat[pix[h]] = make_float4(0.f, 0.f, 0.f, 1.f);
          if constexpr (DEPTH) out_depth[pix[h]] = 0.f;   // a sum yet
          last_idx[pix[h]] = 0u;                          // an empty range starts at 0
        }
      } else if constexpr (DEPTH) {
        float zs[2], T[2];
#pragma unroll
        for (int h = 0; h < 2; h++) { zs[h] = pix[h] < 0 ? 0.f : out_depth[pix[h]]; T[h] = pix[h] < 0 ? 1.f : out_feat[pix[h]].w; }
#pragma unroll
        for (int h = 0; h < 2; h++) if (pix[h] >= 0) out_depth[pix[h]] = finished_depth(zs[h], T[h]);
      }
    }
  }
}

// Two warps to a tile, for a block of TILES pairs of warps: the pair of this thread takes every `step`-th tile from `begin` on.
template <int CKPT, bool DEPTH, bool CHUNKED, bool FEAT, bool LISTED, int TILES, int RECORDS>
__device__ __forceinline__ void composite_halves(
    uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ vals_sorted, const float4* __restrict__ proj0, const float4* __restrict__ proj1,
    const float4* __restrict__ proj2, int W, int H, int tiles_x, int n_tiles, float3 bg, float4* __restrict__ out_rgba, float4* __restrict__ out_feat,
    float* __restrict__ out_depth, uint32_t* __restrict__ last_idx, int chunk, int n_chunks, unsigned long long* __restrict__ alive,
    const float2* __restrict__ proj3, float4* __restrict__ ckpt, int seg_shift, float4* __restrict__ feat_acc, uint32_t* __restrict__ bwd_work,
    const TileList& tiles, uint32_t begin, uint32_t step,
    float4 (&s_staged)[TILES][2][FWD_BATCH / 2][RECORDS], uint32_t (&s_last)[TILES * 2], uint32_t (&s_odd)[TILES * 2][2]) {
  constexpr bool BWD = CKPT != NONE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = warp & 1;
  const bool first = !CHUNKED || chunk == 0, final = !CHUNKED || chunk == n_chunks - 1;
  for (uint32_t w = begin; w < tiles.count; w += step) {   // (once, unless LISTED)
  const int tile = tiles.at(w);
  const int tx = tile % tiles_x, ty = tile / tiles_x, in_tile = half * 32 + lane;   // the lane's pixel in its tile
  const int px = tx * RT_W + (in_tile & 7), py = ty * RT_W + (in_tile >> 3), pix = py * W + px;
  const bool inside = px < W && py < H;
  const float2 pcx = make_float2((float)px + 0.5f, (float)px + 0.5f), pcy = make_float2((float)py + 0.5f, (float)py + 0.5f);
  const uint2 range = tile_ranges[tile];
  if (CKPT == PER_SEGMENT && !LISTED && first && w == 0u && in_tile == 0) bwd_work[BWD_SUMMED] = 0u;
  if (CHUNKED && !LISTED && !first && range.y <= range.x && !(final && FEAT)) {   // nothing of this chunk lands here: pixels, state and flag stay
    if (DEPTH && final && inside) out_depth[pix] = finished_depth(out_depth[pix], out_feat[pix].w);
    return;
  }
  Pixel<CKPT, DEPTH, FEAT, BWD || CHUNKED> P;
  P.T = inside ? 1.f : 0.f;
  P.last = range.x;
  if (CHUNKED && !first && inside) {
    const float4 acc = out_feat[pix];
    P.r = acc.x; P.g = acc.y; P.b = acc.z;
    if constexpr (DEPTH) P.zs = out_depth[pix];
    if constexpr (FEAT) { const float4 fa = feat_acc[pix]; P.f0 = fa.x; P.f1 = fa.y; P.f2 = fa.z; }
    const uint32_t l = last_idx[pix];
    P.T = (l & DONE_BIT) == 0u ? acc.w : 0.f; P.T_closed = acc.w;
    P.last = l & ~DONE_BIT;
  }
  // Checkpoints for the backward's segmented replay (see common.cuh): the state a later chunk starts a tile with, and
  // the state before every (1 << seg_shift)-th fragment of the list.
  const int q = CHUNKED ? chunk * n_tiles + tile : tile;
  uint32_t seg_now = 0;
  auto checkpoint = [&](uint32_t seg) { P.checkpoint(ckpt + (size_t)ckpt_slot(range.x, q, seg, seg_shift) * RT_PX + in_tile); seg_now = seg; };
  if (BWD && CHUNKED && !first && range.y > range.x) checkpoint(0u);
  // The records of a batch are gathered one batch ahead, into registers, half by each warp: the two dependent loads (list
  // entry, then the splat's records) are in flight while the batch before them is composited.
  float4 n0, n1, n2;
  float2 n3;
  auto gather = [&](uint32_t from) {
    n0 = n1 = n2 = make_float4(0.f, 0.f, 0.f, 0.f); n3 = make_float2(0.f, 0.f);   // beyond the list: opacity zero
    if (from < range.y && (uint32_t)in_tile < range.y - from) {
      const uint32_t gid = vals_sorted[from + in_tile];
      n0 = proj0[gid]; n1 = proj1[gid]; n2 = proj2[gid];
      if constexpr (FEAT) n3 = proj3[gid];
    }
  };
  gather(range.x);
  int buf = 0;
  bool any_open = true;
  for (uint32_t start = range.x;; start += FWD_BATCH, buf ^= 1) {
    float4 (*staged)[RECORDS] = s_staged[warp >> 1][buf];
    {
      const bool strange = stage_record<DEPTH, FEAT>(staged[in_tile >> 1], lane & 1, n0, n1, n2, n3);
      const uint32_t any_strange = __any_sync(0xffffffffu, strange);
      if (lane == 0) s_odd[warp][buf] = any_strange;
    }
    // One barrier of the tile's two warps per batch: the batch is staged, the one before it is done with (it lies in the other
    // buffer), and whether any pixel is still open.
    any_open = pair_any(1 + (warp >> 1), P.T != 0.f);
    if (start >= range.y || !any_open) break;
    gather(start + FWD_BATCH);
    const bool odd = (s_odd[warp][buf] | s_odd[warp ^ 1][buf]) != 0u;
    // Pairs are taken FWD_GROUP at a time: first everything that does not depend on the pixel's running state (sigma, the hit test,
    // alpha with its exponential) for the whole group, so that those chains overlap, then the transmittances, then the sums, fragment by
    // fragment in list order.
    for (uint32_t t_begin = 0; t_begin < FWD_BATCH && t_begin < range.y - start; t_begin += FWD_SEG) {   // a segment of the backward is a whole number of these
      const uint32_t at = start + t_begin - range.x, t_end = min(t_begin + FWD_SEG, range.y - start);
      if (BWD && at != 0u && (at & ((1u << seg_shift) - 1u)) == 0u) checkpoint(at >> seg_shift);
      if (!__any_sync(0xffffffffu, P.T != 0.f)) continue;   // only the other half is still at it
      if (odd) {
#pragma unroll 1
        for (uint32_t t = t_begin; t < t_end; t++) {
          const float4* f = staged[t >> 1];
          const float2 al = pair_alpha(f[0], f[1], f[2], lo2(f[3]), pcx, pcy);
          P.template take_odd<RECORDS>(t & 1 ? al.y : al.x, f, t & 1, start + t + 1);
        }
        continue;
      }
      for (uint32_t t0 = t_begin; t0 < t_end; t0 += 2 * FWD_GROUP) {
        float2 alpha[FWD_GROUP];
#pragma unroll
        for (int u = 0; u < FWD_GROUP; u++) {
          const float4* f = staged[t0 / 2 + u];
          alpha[u] = pair_alpha(f[0], f[1], f[2], lo2(f[3]), pcx, pcy);
        }
        P.take_pairs(alpha, staged + t0 / 2, start + t0 + 1);
      }
    }
  }
  const bool open = P.T != 0.f;
  const float T = P.now();
  if (inside) {
    out_rgba[pix] = make_float4(P.r + T * bg.x, P.g + T * bg.y, P.b + T * bg.z, 1.f - T);
    if constexpr (CHUNKED) {
      if (FEAT && final) out_feat[pix] = make_float4(P.f0, P.f1, P.f2, T);
      else out_feat[pix] = make_float4(P.r, P.g, P.b, T);
      if constexpr (FEAT) { if (!final) feat_acc[pix] = make_float4(P.f0, P.f1, P.f2, 0.f); }
      if constexpr (DEPTH) out_depth[pix] = !final ? P.zs : finished_depth(P.zs, T);
      last_idx[pix] = P.last | (open ? 0u : DONE_BIT);
    } else {
      out_feat[pix] = make_float4(P.f0, P.f1, P.f2, T);
      if constexpr (DEPTH) out_depth[pix] = finished_depth(P.zs, T);
      if constexpr (BWD) last_idx[pix] = P.last;
    }
  }
  if constexpr (BWD || CHUNKED) {
  // What the tile's two warps settle together: whether any pixel is still open, and the last fragment any pixel used.
  const uint32_t mine = __reduce_max_sync(0xffffffffu, P.last);
  if (lane == 0) s_last[warp] = mine;
  any_open = pair_any(1 + (warp >> 1), open);
  if (CHUNKED && !final && in_tile == 0 && !any_open)
    atomicAnd(alive + (size_t)(ty >> 3) * ((tiles_x + 7) >> 3) + (tx >> 3), ~(1ull << ((ty & 7) * 8 + (tx & 7))));
  if constexpr (BWD) {
    // The backward never needs to look past the last fragment any pixel used. (A pixel whose last fragment lies in an
    // earlier chunk contributes this chunk's start: an empty range.)
    uint32_t m = max(s_last[warp], s_last[warp ^ 1]);
    if constexpr (CHUNKED) m = min(max(m, range.x), range.y);
    if (in_tile == 0) tile_ranges[tile].y = m;
    if (m > range.x) {
      const uint32_t segs = (m - range.x + (1u << seg_shift) - 1u) >> seg_shift;
      if constexpr (CKPT == PER_SEGMENT) {
        // Slot 0 has no segment before it: its colour takes the sums of the range's last segment (which is the one at hand
        // unless nothing after its boundary was seen).
        float* dst = reinterpret_cast<float*>(ckpt + (size_t)ckpt_slot(range.x, q, 0u, seg_shift) * RT_PX + in_tile);
        const float4 v = segs - 1u == seg_now ? make_float4(P.sr, P.sg, P.sb, 0.f) : ckpt[(size_t)ckpt_slot(range.x, q, segs, seg_shift) * RT_PX + in_tile];
        dst[0] = v.x; dst[1] = v.y; dst[2] = v.z;
      }
    }
  }
  }
  if (!LISTED) return;
  }
}

template <int CKPT, bool DEPTH, bool CHUNKED, bool FEAT, bool LISTED>
__global__ void __launch_bounds__(FWD_WARPS * 32) raster_fwd_half_kernel(
    uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ vals_sorted, const float4* __restrict__ proj0, const float4* __restrict__ proj1,
    const float4* __restrict__ proj2, int W, int H, int tiles_x, int n_tiles, float3 bg, float4* __restrict__ out_rgba, float4* __restrict__ out_feat,
    float* __restrict__ out_depth, uint32_t* __restrict__ last_idx, int chunk, int n_chunks, unsigned long long* __restrict__ alive,
    const float2* __restrict__ proj3, float4* __restrict__ ckpt, int seg_shift, float4* __restrict__ feat_acc, uint32_t* __restrict__ bwd_work,
    const uint32_t* __restrict__ words, const uint32_t* __restrict__ list, int fill_blocks) {
  after_previous();
  // CHUNKED with FEAT (forward only): between chunks out_feat.xyz carries the colour sums, so the feature sums of a
  // pixel travel in feat_acc and move into out_feat.xyz when the last chunk, which then visits every pixel, is done.
  static_assert(!(FEAT && CHUNKED && CKPT != NONE), "the chunked backward reads the colour sums from out_feat.xyz");
  constexpr int RECORDS = FEAT ? STAGED + 2 : DEPTH ? STAGED + 1 : STAGED;
  __shared__ float4 s_staged[FWD_TILES][2][FWD_BATCH / 2][RECORDS];   // [tile][buffer][pair]
  __shared__ uint32_t s_last[FWD_WARPS], s_odd[FWD_WARPS][2];
  const bool first = !CHUNKED || chunk == 0;
  const int blocks = (int)gridDim.x - (LISTED ? fill_blocks : 0);
  if (LISTED && (int)blockIdx.x >= blocks) {
    if (CKPT == PER_SEGMENT && first && (int)blockIdx.x == blocks && threadIdx.x == 0) bwd_work[BWD_SUMMED] = 0u;
    visit_unlisted<DEPTH>(blockIdx.x - blocks, fill_blocks, tile_ranges, n_tiles, tiles_x, W, H, bg, first, out_rgba, out_feat, out_depth, last_idx);
    return;
  }
  const TileList tiles = LISTED ? tile_list(words, list, chunk, n_tiles) : TileList{nullptr, 0u, (uint32_t)n_tiles, n_tiles};
  composite_halves<CKPT, DEPTH, CHUNKED, FEAT, LISTED>(
      tile_ranges, vals_sorted, proj0, proj1, proj2, W, H, tiles_x, n_tiles, bg, out_rgba, out_feat, out_depth, last_idx, chunk, n_chunks, alive, proj3, ckpt,
      seg_shift, feat_acc, bwd_work, tiles, blockIdx.x * FWD_TILES + (threadIdx.x >> 6), blocks * FWD_TILES, s_staged, s_last, s_odd);
}

// Eight warps to a tile, for views of so few tiles that the GPU is idle but for the longest lists: four warps
// find the alphas of a batch, two warps (a pixel per lane) carry the transmittances and the sums, two warps take turns to gather and stage
// the records of the batches ahead. A batch passes from one to the next with one barrier of the block.
constexpr int TEAM_BATCH = FWD_SEG, TEAM_PAIRS = TEAM_BATCH / 2, TEAM_PRODUCERS = 4, TEAM_THREADS = (2 + TEAM_PRODUCERS + 2) * 32, TEAM_PER_SM = 8;
// Up to TEAM_ALWAYS tiles to an SM there is a block for every tile at once. Above that (whole views of up to TEAM_PER_SM to an SM, and the
// second of two chunks) the team pays where the time is that of the longest list, and loses where all tiles have much the same to do: its
// blocks fill the GPU with fewer tiles. The binning leaves the number of hits and the longest list on the device, and the block asks them; where the
// team does not pay, the same blocks take four tiles at two warps each. Forward, us, at two warps / the team, against hits over (SMs * longest list):
//   whole views   200x150 over 20k splats 0.33: 28.5 / 19.1; 333x217 over 20k 0.66: 22.7 / 18.8; 256x192 over 8k 0.58: 30.1 / 23.0, over 20k 2.0: 13.1 /
//                 15.6; 333x217 over 8k 2.2: 25.7 / 33.5, over 2k faint 3.9: 27.8 / 41.1, over 300 wide ones 6.7: 9.7 / 16.1; lists below 100: 2.8 / 4.5
//   second chunk  1280x720 over 500k 0.50: 63.7 / 39.2, 1.07: 28.4 / 20.2; over 300k faint 2.35: 68.9 / 62.2, 4.1: 66.1 / 69.6; 1920x1080 over 500k 2.0: 24.1 /
//                 27.2, 4.6: 22.6 / 38.9, faint and close (19,035 tiles with a list) 370 / 490. More than CHUNK_TEAM_PER_SM listed tiles to an SM do
//                 not go to the team whatever their lists: 1,578 of up to 80 7.7 / 13.0, 1,970 of up to 745 24.1 / 27.2
constexpr int TEAM_ALWAYS = 2, CHUNK_TEAM_PER_SM = 10, TEAM_BLOCKS = 2, CHUNK_BLOCKS = 3, TEAM_TILES = TEAM_THREADS / 64;   // blocks of whole views and of chunks that fit on an SM
__device__ __forceinline__ bool team_pays(uint32_t hits, uint32_t longest, uint32_t sms, uint32_t blocks) {
  return longest >= LONG_LIST && 2ull * hits <= (2ull * blocks - 1ull) * sms * longest;
}

template <int CKPT, bool DEPTH, bool CHUNKED, bool FEAT>
__global__ void __launch_bounds__(TEAM_THREADS, CHUNKED ? CHUNK_BLOCKS : TEAM_BLOCKS) raster_fwd_team_kernel(
    uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ vals_sorted, const float4* __restrict__ proj0, const float4* __restrict__ proj1,
    const float4* __restrict__ proj2, int W, int H, int tiles_x, int n_tiles, float3 bg, float4* __restrict__ out_rgba, float4* __restrict__ out_feat,
    float* __restrict__ out_depth, uint32_t* __restrict__ last_idx, int chunk, int n_chunks, unsigned long long* __restrict__ alive,
    const float2* __restrict__ proj3, float4* __restrict__ ckpt, int seg_shift, uint32_t* __restrict__ bwd_work, const uint32_t* __restrict__ words, const uint32_t* __restrict__ list,
    const uint32_t* __restrict__ hits, const uint32_t* __restrict__ longest, uint32_t sms) {
  after_previous();
  constexpr bool BWD = CKPT != NONE;
  constexpr int RECORDS = FEAT ? STAGED + 2 : DEPTH ? STAGED + 1 : STAGED;
  union Shared {
    struct {
      float4 staged[3][TEAM_PAIRS][RECORDS];   // of the batches that are staged, weighed and composited
      float2 alpha[2][TEAM_PAIRS][RT_PX];
      uint32_t odd[3], last[2];
    } team;
    struct {
      float4 staged[TEAM_TILES][2][FWD_BATCH / 2][RECORDS];
      uint32_t last[TEAM_TILES * 2], odd[TEAM_TILES * 2][2];
    } halves;
  };
  __shared__ __align__(16) unsigned char s_mem[sizeof(Shared)];
  Shared& sh = *reinterpret_cast<Shared*>(s_mem);
  auto &s_staged = sh.team.staged;
  auto &s_alpha = sh.team.alpha;
  auto &s_odd = sh.team.odd;
  auto &s_last = sh.team.last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int TEAM_GROUP = CHUNKED ? 4 : 8;   // pairs whose sums are taken together: eight want registers for two blocks an SM, which is enough where tiles are few
  static_assert(!(CHUNKED && (DEPTH || FEAT)), "the last chunk finishes depths and features in every tile");
  const bool composites = warp < 2, weighs = !composites && warp < 2 + TEAM_PRODUCERS, final = !CHUNKED || chunk == n_chunks - 1;
  if (CKPT == PER_SEGMENT && !CHUNKED && blockIdx.x == 0 && threadIdx.x == 0) bwd_work[BWD_SUMMED] = 0u;
  const TileList tiles = CHUNKED ? tile_list(words, list, chunk, n_tiles) : TileList{nullptr, 0u, (uint32_t)n_tiles, n_tiles};
  constexpr int BLOCKS = CHUNKED ? CHUNK_BLOCKS : TEAM_BLOCKS;
  if (hits && ((CHUNKED && tiles.count > CHUNK_TEAM_PER_SM * sms) || !team_pays(*hits, *longest, sms, BLOCKS))) {
    // Two neighbours, which share splats, to two pairs of warps and two far from them to the others, over as many blocks as fit at once or are
    // needed (the 1,475 tiles of a faint scene, us: four neighbours to a block 122, none 108, this 99).
    const uint32_t pair = threadIdx.x >> 6, used = min(max((uint32_t)BLOCKS * sms, (tiles.count + TEAM_TILES - 1u) / TEAM_TILES), gridDim.x);
    if (blockIdx.x >= used) return;
    const uint32_t begin = ((pair >> 1) * used + blockIdx.x) * 2u + (pair & 1u), step = used * TEAM_TILES;
    composite_halves<CKPT, DEPTH, CHUNKED, FEAT, CHUNKED>(tile_ranges, vals_sorted, proj0, proj1, proj2, W, H, tiles_x, n_tiles, bg, out_rgba, out_feat, out_depth, last_idx, chunk, n_chunks,
                                                          alive, proj3, ckpt, seg_shift, nullptr, bwd_work, tiles, begin, step, sh.halves.staged, sh.halves.last, sh.halves.odd);
    return;
  }
  for (uint32_t w = blockIdx.x; w < tiles.count; w += gridDim.x) {
  if (w != blockIdx.x) __syncthreads();   // the last tile's batches have been read
  const int tile = tiles.at(w), tx = tile % tiles_x, ty = tile / tiles_x;
  const uint2 range = tile_ranges[tile];
  const uint32_t batches = range.y > range.x ? (range.y - range.x + TEAM_BATCH - 1) / TEAM_BATCH : 0u;
  // The lane's pixel, of a producer its first of two.
  const int in_tile = (composites ? warp * 32 : 0) + lane, px = tx * RT_W + (in_tile & 7), py = ty * RT_W + (in_tile >> 3), pix = py * W + px;
  const bool inside = composites && px < W && py < H;
  const float2 pcx = make_float2((float)px + 0.5f, (float)px + 0.5f), pcy = make_float2((float)py + 0.5f, (float)py + 0.5f);
  Pixel<CKPT, DEPTH, FEAT, BWD || CHUNKED> P;
  P.T = inside ? 1.f : 0.f;
  P.last = range.x;
  if (CHUNKED && inside) {
    const float4 acc = out_feat[pix];
    P.r = acc.x; P.g = acc.y; P.b = acc.z;
    const uint32_t l = last_idx[pix];
    P.T = (l & DONE_BIT) == 0u ? acc.w : 0.f; P.T_closed = acc.w;
    P.last = l & ~DONE_BIT;
  }
  const int q = CHUNKED ? chunk * n_tiles + tile : tile;
  uint32_t seg_now = 0;
  auto checkpoint = [&](uint32_t seg) { P.checkpoint(ckpt + (size_t)ckpt_slot(range.x, q, seg, seg_shift) * RT_PX + in_tile); seg_now = seg; };
  if (BWD && CHUNKED && composites) checkpoint(0u);   // the state this chunk starts the tile with
  // A gathering warp's next batch is in its registers, and the list entries of the one after that.
  const uint32_t turn = (uint32_t)warp & 1u;
  float4 n0, n1, n2;
  float2 n3;
  uint32_t gid = 0u;
  auto entries = [&](uint32_t b) { const uint32_t at = range.x + b * TEAM_BATCH + lane; gid = b < batches && at < range.y ? vals_sorted[at] : 0xFFFFFFFFu; };
  auto gather = [&]() {
    n0 = n1 = n2 = make_float4(0.f, 0.f, 0.f, 0.f); n3 = make_float2(0.f, 0.f);   // beyond the list: opacity zero
    if (gid != 0xFFFFFFFFu) {
      n0 = proj0[gid]; n1 = proj1[gid]; n2 = proj2[gid];
      if constexpr (FEAT) n3 = proj3[gid];
    }
  };
  if (!composites && !weighs) { entries(turn); gather(); entries(turn + 2u); }
  for (uint32_t t = 0; batches && t < batches + 2u; t++) {
    if (!__syncthreads_or(P.T != 0.f)) break;   // (only the pixels' own warps hold a transmittance)
    if (composites) {
      if (t < 2u) continue;
      const uint32_t at = (t - 2u) * TEAM_BATCH, start = range.x + at, count = min((uint32_t)TEAM_BATCH, range.y - start);
      const float4 (*staged)[RECORDS] = s_staged[(t - 2u) % 3u];
      const float2 (*alphas)[RT_PX] = s_alpha[t & 1u];
      if (BWD && at != 0u && (at & ((1u << seg_shift) - 1u)) == 0u) checkpoint(at >> seg_shift);
      if (!__any_sync(0xffffffffu, P.T != 0.f)) continue;   // only the other half is still at it
      if (s_odd[(t - 2u) % 3u]) {
#pragma unroll 1
        for (uint32_t k = 0; k < count; k++) {
          const float2 al = alphas[k >> 1][in_tile];
          P.template take_odd<RECORDS>(k & 1u ? al.y : al.x, staged[k >> 1], (int)(k & 1u), start + k + 1u);
        }
        continue;
      }
      for (uint32_t k = 0; k < count; k += 2 * TEAM_GROUP) {
        float2 alpha[TEAM_GROUP];
#pragma unroll
        for (int u = 0; u < TEAM_GROUP; u++) alpha[u] = alphas[k / 2 + u][in_tile];
        P.take_pairs(alpha, staged + k / 2, start + k + 1u);
      }
    } else if (weighs) {
      if (t == 0u || t > batches) continue;
      const uint32_t start = range.x + (t - 1u) * TEAM_BATCH, count = min((uint32_t)TEAM_BATCH, range.y - start);
      const uint32_t pairs = (count + 2 * TEAM_GROUP - 1) / (2 * TEAM_GROUP) * TEAM_GROUP;   // the sums take whole groups
      const float4 (*staged)[RECORDS] = s_staged[(t - 1u) % 3u];
      float2 (*alphas)[RT_PX] = s_alpha[(t - 1u) & 1u];
      const float2 pcy1 = make_float2(pcy.x + 4.f, pcy.y + 4.f);   // exact
#pragma unroll
      for (uint32_t k = 0; k < TEAM_PAIRS / TEAM_PRODUCERS; k++) {
        const uint32_t pair = k * TEAM_PRODUCERS + (uint32_t)warp - 2u;
        if (pair >= pairs) break;
        const float4* f = staged[pair];
        const float4 q0 = f[0], q1 = f[1], q2 = f[2];
        const float2 power = lo2(f[3]);
        alphas[pair][lane] = pair_alpha(q0, q1, q2, power, pcx, pcy);
        alphas[pair][lane + 32] = pair_alpha(q0, q1, q2, power, pcx, pcy1);
      }
    } else if (t < batches && (t & 1u) == turn) {
      const bool strange = stage_record<DEPTH, FEAT>(s_staged[t % 3u][lane >> 1], lane & 1, n0, n1, n2, n3);
      const uint32_t any_strange = __any_sync(0xffffffffu, strange);
      if (lane == 0) s_odd[t % 3u] = any_strange;
      gather();
      entries(t + 4u);
    }
  }
  if (!composites) continue;
  const bool open = P.T != 0.f;
  const float T = P.now();
  if (inside) {
    out_rgba[pix] = make_float4(P.r + T * bg.x, P.g + T * bg.y, P.b + T * bg.z, 1.f - T);
    if constexpr (CHUNKED) {
      out_feat[pix] = make_float4(P.r, P.g, P.b, T);
      last_idx[pix] = P.last | (open ? 0u : DONE_BIT);
    } else {
      out_feat[pix] = make_float4(P.f0, P.f1, P.f2, T);
      if constexpr (DEPTH) out_depth[pix] = finished_depth(P.zs, T);
      if constexpr (BWD) last_idx[pix] = P.last;
    }
  }
  if constexpr (BWD || CHUNKED) {
    // What the two warps settle together: whether any pixel is still open, and the last fragment any pixel used, which the backward never
    // needs to look past.
    const uint32_t mine = __reduce_max_sync(0xffffffffu, P.last);
    if (lane == 0) s_last[warp] = mine;
    const bool any_open = pair_any(1, open);
    if (CHUNKED && !final && in_tile == 0 && !any_open)
      atomicAnd(alive + (size_t)(ty >> 3) * ((tiles_x + 7) >> 3) + (tx >> 3), ~(1ull << ((ty & 7) * 8 + (tx & 7))));
    uint32_t m = max(s_last[0], s_last[1]);
    if constexpr (CHUNKED) m = min(max(m, range.x), range.y);
    if (BWD && in_tile == 0) tile_ranges[tile].y = m;
    if (CKPT == PER_SEGMENT && m > range.x) {
      // Slot 0 has no segment before it (see raster_fwd_half_kernel).
      const uint32_t segs = (m - range.x + (1u << seg_shift) - 1u) >> seg_shift;
      float* dst = reinterpret_cast<float*>(ckpt + (size_t)ckpt_slot(range.x, q, 0u, seg_shift) * RT_PX + in_tile);
      const float4 v = segs - 1u == seg_now ? make_float4(P.sr, P.sg, P.sb, 0.f) : ckpt[(size_t)ckpt_slot(range.x, q, segs, seg_shift) * RT_PX + in_tile];
      dst[0] = v.x; dst[1] = v.y; dst[2] = v.z;
    }
  }
  }
}

// One warp to a tile, for views in depth chunks.
template <int CKPT, bool DEPTH, bool FEAT, bool LISTED>
__global__ void __launch_bounds__(FWD_WARPS * 32) raster_fwd_kernel(
    uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ vals_sorted, const float4* __restrict__ proj0, const float4* __restrict__ proj1,
    const float4* __restrict__ proj2, int W, int H, int tiles_x, int n_tiles, float3 bg, float4* __restrict__ out_rgba, float4* __restrict__ out_feat,
    float* __restrict__ out_depth, uint32_t* __restrict__ last_idx, int chunk, int n_chunks, unsigned long long* __restrict__ alive,
    const float2* __restrict__ proj3, float4* __restrict__ ckpt, int seg_shift, float4* __restrict__ feat_acc, uint32_t* __restrict__ bwd_work,
    const uint32_t* __restrict__ words, const uint32_t* __restrict__ list, int fill_blocks) {
  after_previous();
  constexpr bool BWD = CKPT != NONE;
  // FEAT (forward only): between chunks out_feat.xyz carries the colour sums, so the feature sums of a
  // pixel travel in feat_acc and move into out_feat.xyz when the last chunk, which then visits every pixel, is done.
  static_assert(!(FEAT && BWD), "the chunked backward reads the colour sums from out_feat.xyz");
  __shared__ float4 s_staged[FWD_WARPS][FWD_SEG][FEAT ? 6 : 5];   // a fragment's constants, most of them twice, as operands of packed arithmetic
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool first = chunk == 0, final = chunk == n_chunks - 1;
  const int blocks = (int)gridDim.x - (LISTED ? fill_blocks : 0);
  if (LISTED && (int)blockIdx.x >= blocks) {
    if (CKPT == PER_SEGMENT && first && (int)blockIdx.x == blocks && threadIdx.x == 0) bwd_work[BWD_SUMMED] = 0u;
    visit_unlisted<DEPTH>(blockIdx.x - blocks, fill_blocks, tile_ranges, n_tiles, tiles_x, W, H, bg, first, out_rgba, out_feat, out_depth, last_idx);
    return;
  }
  const TileList tiles = LISTED ? tile_list(words, list, chunk, n_tiles) : TileList{nullptr, 0u, (uint32_t)n_tiles, n_tiles};
  for (uint32_t w = blockIdx.x * FWD_WARPS + warp; w < tiles.count; w += blocks * FWD_WARPS) {   // (once, unless LISTED)
  const int tile = tiles.at(w);
  float2 f0 = splat2(0.f), f1 = f0, f2 = f0;   // composited feature lanes (raster_fwd.cu:52)
  const int tx = tile % tiles_x, ty = tile / tiles_x;
  const int px0 = tx * RT_W + (lane & 3) * 2, py = ty * RT_W + (lane >> 2);
  const bool in0 = px0 < W && py < H, in1 = px0 + 1 < W && py < H;
  const float2 pcx = make_float2((float)px0 + 0.5f, (float)px0 + 1.5f), pcy = splat2((float)py + 0.5f);
  const uint2 range = tile_ranges[tile];
  if (CKPT == PER_SEGMENT && !LISTED && first && w == 0u && lane == 0) bwd_work[BWD_SUMMED] = 0u;
  if (!LISTED && !first && range.y <= range.x && !(final && FEAT)) {   // nothing of this chunk lands here: pixels, state and flag stay
    if (DEPTH && final) {
#pragma unroll
      for (int p = 0; p < 2; p++)
        if (p == 0 ? in0 : in1) { const int pix = py * W + px0 + p; out_depth[pix] = finished_depth(out_depth[pix], out_feat[pix].w); }
    }
    return;
  }
  float2 r = splat2(0.f), g = r, b = r, zs = r;   // of the two pixels
  float2 T = make_float2(in0 ? 1.f : 0.f, in1 ? 1.f : 0.f), T_closed = splat2(1.f);   // transmittance of a pixel that can take another fragment, else zero and the one it closed with
  uint32_t last[2] = {range.x, range.x};
  if (!first) {
#pragma unroll
    for (int p = 0; p < 2; p++) {
      if (p == 0 ? in0 : in1) {
        const int pix = py * W + px0 + p;
        const float4 acc = out_feat[pix];
        at(r, p) = acc.x; at(g, p) = acc.y; at(b, p) = acc.z; at(T_closed, p) = acc.w;
        if constexpr (DEPTH) at(zs, p) = out_depth[pix];
        if constexpr (FEAT) { const float4 fa = feat_acc[pix]; at(f0, p) = fa.x; at(f1, p) = fa.y; at(f2, p) = fa.z; }
        const uint32_t l = last_idx[pix];
        at(T, p) = (l & DONE_BIT) == 0u ? acc.w : 0.f;
        last[p] = l & ~DONE_BIT;
      }
    }
  }
  // Checkpoints for the backward's segmented replay (see common.cuh): the state a later chunk starts a tile with, and
  // the state before every (1 << seg_shift)-th fragment of the list.
  const int q = chunk * n_tiles + tile;
  float2 sr = splat2(0.f), sg = sr, sb = sr;   // PER_SEGMENT: colour sums of the segment at hand
  uint32_t seg_now = 0;
  auto checkpoint = [&](uint32_t seg) {
    float4* dst = ckpt + (size_t)ckpt_slot(range.x, q, seg, seg_shift) * RT_PX + lane * 2;
    const float2 now = make_float2(T.x != 0.f ? T.x : T_closed.x, T.y != 0.f ? T.y : T_closed.y);
    if constexpr (CKPT == PER_SEGMENT) {   // the sums of the segment before the boundary
      dst[0] = make_float4(sr.x, sg.x, sb.x, now.x); dst[1] = make_float4(sr.y, sg.y, sb.y, now.y);
      sr = sg = sb = splat2(0.f);
      seg_now = seg;
    } else {
      dst[0] = make_float4(r.x, g.x, b.x, now.x); dst[1] = make_float4(r.y, g.y, b.y, now.y);
    }
  };
  if (BWD && !first && range.y > range.x) checkpoint(0u);
  // The records of a batch are gathered one batch ahead, into registers: the two dependent loads (list entry, then the
  // splat's records) are in flight while the batch before them is composited.
  float4 n0 = make_float4(0.f, 0.f, 0.f, 0.f), n1 = n0, n2 = n0;
  float2 n3 = make_float2(0.f, 0.f);
  auto gather = [&](uint32_t from) {
    n0 = n1 = n2 = make_float4(0.f, 0.f, 0.f, 0.f); n3 = make_float2(0.f, 0.f);   // beyond the list: opacity zero
    if (from < range.y && (uint32_t)lane < range.y - from) {
      const uint32_t gid = vals_sorted[from + lane];
      n0 = proj0[gid]; n1 = proj1[gid]; n2 = proj2[gid];
      if constexpr (FEAT) n3 = proj3[gid];
    }
  };
  gather(range.x);
  for (uint32_t start = range.x; start < range.y; start += FWD_SEG) {
    if (!__any_sync(0xffffffffu, T.x != 0.f || T.y != 0.f)) break;
    if (BWD && start != range.x && ((start - range.x) & ((1u << seg_shift) - 1u)) == 0u) checkpoint((start - range.x) >> seg_shift);
    __syncwarp();
    uint32_t odd;   // fragments whose colour or feature is not finite: they may not be added with weight zero
    {
      float4* q = s_staged[warp][lane];
      q[0] = make_float4(-n0.x, -n0.x, -n0.y, -n0.y);
      q[1] = make_float4(0.5f * n0.z, 0.5f * n0.z, n0.w, n0.w);
      q[2] = make_float4(0.5f * n1.x, 0.5f * n1.x, n1.y, n1.w);
      const float cr = fmaxf(n2.x, 0.f), cg = fmaxf(n2.y, 0.f), cb = fmaxf(n2.z, 0.f);
      q[3] = make_float4(cr, cr, cg, cg);
      q[4] = make_float4(cb, cb, n1.z, n1.z);
      bool strange = fmaxf(cr, fmaxf(cg, cb)) == INFINITY;
      if constexpr (FEAT) {
        q[5] = make_float4(n2.w, n3.x, n3.y, 0.f);
        strange = strange || !(isfinite(n2.w) && isfinite(n3.x) && isfinite(n3.y));
      }
      odd = __ballot_sync(0xffffffffu, strange);
    }
    __syncwarp();
    gather(start + FWD_SEG);
    // Fragments are taken FWD_GROUP at a time: first everything that does not depend on the pixels' running state (sigma,
    // the hit test, alpha with its exponential) for the whole group, so that those chains overlap, then the transmittances, then the
    // sums, fragment by fragment in list order. A pixel that does not see a fragment has its transmittance multiplied by one, and its
    // sums take zeros.
    // The blend weight of a fragment, and the pixel's transmittance moved on: the fragment that would saturate a pixel closes it and is
    // not taken.
    auto weigh = [&](int p, float al, float through) {
      const float now = at(T, p), next_T = now * through;
      const bool stays = next_T > T_CUTOFF;
      at(T_closed, p) = !stays && now != 0.f ? now : at(T_closed, p);
      at(T, p) = stays ? next_T : 0.f;
      return stays ? al * now : 0.f;
    };
    const float4 (*staged)[FEAT ? 6 : 5] = s_staged[warp];
    const uint32_t remaining = min((uint32_t)FWD_SEG, range.y - start);
    if (odd) {
#pragma unroll 1
      for (uint32_t t = 0; t < remaining; t++) {
        const float2 alpha = fragment_alpha(staged[t][0], staged[t][1], staged[t][2], pcx, pcy);
        const float4 q3 = staged[t][3], q4 = staged[t][4];
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const float al = p == 0 ? alpha.x : alpha.y;
          if (al == 0.f || at(T, p) == 0.f) continue;
          const float vis = weigh(p, al, 1.f - al);
          if (vis == 0.f) continue;
          at(r, p) += q3.x * vis; at(g, p) += q3.z * vis; at(b, p) += q4.x * vis;
          if constexpr (CKPT == PER_SEGMENT) { at(sr, p) += q3.x * vis; at(sg, p) += q3.z * vis; at(sb, p) += q4.x * vis; }
          if constexpr (DEPTH) at(zs, p) += vis * q4.z;
          if constexpr (FEAT) { const float4 q5 = staged[t][5]; at(f0, p) += q5.x * vis; at(f1, p) += q5.y * vis; at(f2, p) += q5.z * vis; }
          last[p] = start + t + 1;
        }
      }
      continue;
    }
    for (uint32_t t0 = 0; t0 < remaining; t0 += FWD_GROUP) {
      float2 alpha[FWD_GROUP], through[FWD_GROUP];   // alpha: zero where the pixel does not see the fragment; 1 - alpha
#pragma unroll
      for (int u = 0; u < FWD_GROUP; u++) {
        const uint32_t t = t0 + (uint32_t)u;
        const float4 q0 = staged[t][0], q1 = staged[t][1], q2 = staged[t][2];
        alpha[u] = fragment_alpha(q0, q1, q2, pcx, pcy);
        through[u] = __fadd2_rn(splat2(1.f), make_float2(-alpha[u].x, -alpha[u].y));
      }
      float2 vis[FWD_GROUP];
      {
        float2 ahead = T;
#pragma unroll
        for (int u = 0; u < FWD_GROUP; u++) { vis[u] = __fmul2_rn(alpha[u], ahead); ahead = __fmul2_rn(ahead, through[u]); }
        if (__all_sync(0xffffffffu, none_closes<FWD_GROUP>(T.x, ahead.x) && none_closes<FWD_GROUP>(T.y, ahead.y))) T = ahead;
        else {
#pragma unroll
          for (int u = 0; u < FWD_GROUP; u++) vis[u] = make_float2(weigh(0, alpha[u].x, through[u].x), weigh(1, alpha[u].y, through[u].y));
        }
      }
#pragma unroll
      for (int u = 0; u < FWD_GROUP; u++) {
        const uint32_t t = t0 + (uint32_t)u;
        const float4 q3 = staged[t][3], q4 = staged[t][4];
        const float2 cr = make_float2(q3.x, q3.y), cg = make_float2(q3.z, q3.w), cb = make_float2(q4.x, q4.y);
        r = __ffma2_rn(cr, vis[u], r); g = __ffma2_rn(cg, vis[u], g); b = __ffma2_rn(cb, vis[u], b);
        if constexpr (CKPT == PER_SEGMENT) { sr = __ffma2_rn(cr, vis[u], sr); sg = __ffma2_rn(cg, vis[u], sg); sb = __ffma2_rn(cb, vis[u], sb); }
        if constexpr (DEPTH) zs = __ffma2_rn(vis[u], make_float2(q4.z, q4.w), zs);
        if constexpr (FEAT) {
          const float4 q5 = staged[t][5];
          f0 = __ffma2_rn(splat2(q5.x), vis[u], f0); f1 = __ffma2_rn(splat2(q5.y), vis[u], f1); f2 = __ffma2_rn(splat2(q5.z), vis[u], f2);
        }
        last[0] = vis[u].x != 0.f ? start + t + 1 : last[0]; last[1] = vis[u].y != 0.f ? start + t + 1 : last[1];
      }
    }
  }
  const bool open[2] = {T.x != 0.f, T.y != 0.f};
  T = make_float2(open[0] ? T.x : T_closed.x, open[1] ? T.y : T_closed.y);
#pragma unroll
  for (int p = 0; p < 2; p++) {
    if (p == 0 ? in0 : in1) {
      const int pix = py * W + px0 + p;
      out_rgba[pix] = make_float4(at(r, p) + at(T, p) * bg.x, at(g, p) + at(T, p) * bg.y, at(b, p) + at(T, p) * bg.z, 1.f - at(T, p));
      if (FEAT && final) out_feat[pix] = make_float4(at(f0, p), at(f1, p), at(f2, p), at(T, p));
      else out_feat[pix] = make_float4(at(r, p), at(g, p), at(b, p), at(T, p));
      if constexpr (FEAT) { if (!final) feat_acc[pix] = make_float4(at(f0, p), at(f1, p), at(f2, p), 0.f); }
      if constexpr (DEPTH) out_depth[pix] = !final ? at(zs, p) : finished_depth(at(zs, p), at(T, p));
      last_idx[pix] = last[p] | (open[p] ? 0u : DONE_BIT);
    }
  }
  if (!final) {
    const bool more = __any_sync(0xffffffffu, open[0] || open[1]);
    if (lane == 0 && !more) atomicAnd(alive + (size_t)(ty >> 3) * ((tiles_x + 7) >> 3) + (tx >> 3), ~(1ull << ((ty & 7) * 8 + (tx & 7))));
  }
  if constexpr (BWD) {
    // The backward never needs to look past the last fragment any pixel used. (A pixel whose last fragment lies in an
    // earlier chunk contributes this chunk's start: an empty range.)
    uint32_t m = max(last[0], last[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    m = min(max(m, range.x), range.y);
    if (lane == 0) tile_ranges[tile].y = m;
    if (CKPT == PER_SEGMENT && m > range.x) {
      // Slot 0 has no segment before it: its colour takes the sums of the range's last segment (which is the one at hand
      // unless nothing after its boundary was seen).
      const uint32_t segs = (m - range.x + (1u << seg_shift) - 1u) >> seg_shift;
      float* dst = reinterpret_cast<float*>(ckpt + (size_t)ckpt_slot(range.x, q, 0u, seg_shift) * RT_PX + lane * 2);
      const float4* src = ckpt + (size_t)ckpt_slot(range.x, q, segs, seg_shift) * RT_PX + lane * 2;
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const float4 v = segs - 1u == seg_now ? make_float4(at(sr, p), at(sg, p), at(sb, p), 0.f) : src[p];
        dst[p * 4] = v.x; dst[p * 4 + 1] = v.y; dst[p * 4 + 2] = v.z;
      }
    }
  }
  if (!LISTED) return;
  }
}

}  // namespace
}  // namespace b2k

using namespace b2k;

namespace b2k {
// One chunk of a chunked view (n_chunks > 1), or the whole view (n_chunks <= 1).
int launch_raster_fwd(const B2kCtx* c, const B2kRenderOpts* o, int chunk, int n_chunks, unsigned long long* alive, const uint32_t* tiles, cudaStream_t s) {
  const float3 bg = make_float3(o->bg[0], o->bg[1], o->bg[2]);
  uint2* ranges = (uint2*)c->tile_ranges + (n_chunks > 1 ? (size_t)chunk * c->n_tiles : 0);
  const bool chunked = n_chunks > 1, halves = n_chunks <= 2;   // (measured above)
  // Only the tiles with a list are composited; the others are filled by the first chunk, and by the last one finished where depths are
  // wanted. Features travel by way of every pixel, and so do depths in a forward for a backward.
  const bool depths = chunk == n_chunks - 1 && c->out_depth;
  const uint32_t* list = chunked && o->feat_mode == 0 && !(depths && o->bwd_info) ? tiles : nullptr;
  const int fill_blocks = list && (chunk == 0 || depths) ? min(div_up(c->n_tiles, 32 * FWD_WARPS), 8 * sm_count()) : 0, most = 24 * sm_count();   // (a few times what is resident: tiles differ)
#define ARGS s, ranges, c->vals_sorted, (const float4*)c->proj0, (const float4*)c->proj1, (const float4*)c->proj2, c->W, c->H, c->tiles_x, c->n_tiles, bg, \
    (float4*)c->out_rgba, (float4*)c->out_feat, c->out_depth, c->last_idx, chunk, n_chunks, alive, (const float2*)c->proj3, o->bwd_info ? bwd_ckpt_ptr(c) : nullptr, \
    seg_shift_of(short_segments(c)), (chunked && o->feat_mode != 0) ? (float4*)c->bwd_scratch : nullptr, bwd_work_ptr(c)
#define HALF(B, D, C, F, LISTED) launch_next(raster_fwd_half_kernel<B, D, C, F, LISTED>, (LISTED ? min(div_up(c->n_tiles, FWD_TILES), most) : div_up(c->n_tiles, FWD_TILES)) + fill_blocks, FWD_WARPS * 32, 0, ARGS, \
    c->chunk_words, list, fill_blocks)
#define TEAM(B, D, C, F, HITS, LONGEST) launch_next(raster_fwd_team_kernel<B, D, C, F>, C ? min(c->n_tiles, TEAM_PER_SM * sm_count()) : c->n_tiles, TEAM_THREADS, 0, s, ranges, c->vals_sorted, (const float4*)c->proj0, (const float4*)c->proj1, \
    (const float4*)c->proj2, c->W, c->H, c->tiles_x, c->n_tiles, bg, (float4*)c->out_rgba, (float4*)c->out_feat, c->out_depth, c->last_idx, chunk, n_chunks, alive, \
    (const float2*)c->proj3, o->bwd_info ? bwd_ckpt_ptr(c) : nullptr, seg_shift_of(short_segments(c)), bwd_work_ptr(c), c->chunk_words, list, HITS, LONGEST, (uint32_t)sm_count())
#define WARP(B, D, F) do { if (list) launch_next(raster_fwd_kernel<B, D, false, true>, min(div_up(c->n_tiles, FWD_WARPS), most) + fill_blocks, FWD_WARPS * 32, 0, ARGS, c->chunk_words, list, fill_blocks); \
    else launch_next(raster_fwd_kernel<B, D, F, false>, div_up(c->n_tiles, FWD_WARPS), FWD_WARPS * 32, 0, ARGS, c->chunk_words, list, 0); } while (0)
#define L(B, D, F) do { if (!chunked) { if (c->n_tiles <= TEAM_ALWAYS * sm_count()) TEAM(B, D, false, F, nullptr, nullptr); \
    else if (c->n_tiles <= TEAM_PER_SM * sm_count() && c->num_isect) TEAM(B, D, false, F, c->num_isect, c->num_isect + NI_LONGEST); else HALF(B, D, false, F, false); } \
    else if (halves && list && chunk > 0 && !c->out_depth) TEAM(B, false, true, false, c->chunk_words + CW_COUNT + chunk, c->chunk_words + CW_LONGEST + chunk); \
    else if (halves && list) HALF(B, D, true, false, true); else if (halves) HALF(B, D, true, (F) && (B) == NONE, false); \
    else WARP(B, D, (F) && (B) == NONE); } while (0)
#define LD(B, D) do { if (o->feat_mode != 0) L(B, D, true); else L(B, D, false); } while (0)   // a chunked view with features is forward only (checked by the caller)
#define LB(B) do { if (c->out_depth) LD(B, true); else LD(B, false); } while (0)
  if (!o->bwd_info) LB(NONE);
  else if (short_segments(c)) LB(PER_SEGMENT);
  else LB(RUNNING);
#undef LB
#undef LD
#undef L
#undef HALF
#undef TEAM
#undef WARP
#undef ARGS
  return check_launch();
}
}  // namespace b2k

extern "C" int b2k_raster_fwd(const B2kCtx* c, const B2kRenderOpts* o, b2k_stream_t stream) {
  B2K_REQUIRE(c && o && c->tile_ranges && c->vals_sorted && c->proj0 && c->proj1 && c->proj2 && c->out_rgba && c->out_feat);
  B2K_REQUIRE(!o->bwd_info || (c->last_idx && c->bwd_scratch));
  B2K_REQUIRE(c->W > 0 && c->H > 0 && c->n_tiles == c->tiles_x * c->tiles_y);
  if (o->bwd_info && c->bwd_scratch_bytes < b2k_bwd_scratch_bytes(c->W, c->H, c->n_chunks, c->isect_cap)) return B2K_ERR_CAPACITY;
  B2K_REQUIRE(o->feat_mode >= 0 && o->feat_mode <= 2 && (o->feat_mode == 0 || c->proj3));
  return launch_raster_fwd(c, o, 0, 1, nullptr, nullptr, (cudaStream_t)stream);
}
