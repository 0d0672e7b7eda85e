// Forward compositing: one warp per 8x8 tile walks the tile's depth-ordered fragment list front to back, each lane
// carrying two horizontally adjacent pixels. Reference semantics: raster_fwd_kernel (src/gpu/raster_fwd.cu:9-71); the
// optional expected-depth output follows the mean-depth mode of probe_kernel (src/gpu/probe.cu:30-46).
//
// Bound by instruction issue where tiles fill the GPU and by the latency of one list where they do not; memory traffic is the
// gather of 48 B per staged fragment, served mostly by L2. Fragments are gathered one batch of 32 ahead and staged per warp in
// shared memory; warps never synchronise with each other. A lane's two pixels share packed operations (fp32x2), whose constant
// operands are staged in pairs; the hit test is one comparison; a pixel that does not see a fragment takes it with weight zero
// instead of branching around it (a vote and a branch per fragment cost more than the ten operations they saved). Measured
// against scalar pixels with a vote: 1920x1080 view of 500k splats 143 -> 123 us, 4K with depth 847 -> 740, 1001x751 with
// features 85 -> 69, 1237x822 117 -> 92, 64x64 (one list at a time) 50 -> 38. Images are the same bit for bit.
#include "common.cuh"

namespace b2k {
namespace {

constexpr int FWD_WARPS = 4;
constexpr int FWD_BATCH = 32;
static_assert(FWD_BATCH == 1 << SEG_SHIFT_MIN, "a segment of the backward is a whole number of batches");
constexpr int FWD_GROUP = 4;                             // fragments whose state-independent math is issued together (8: the same within 3 %, more registers)

// CHUNKED: the view is composited in depth chunks (chunk `chunk` of `n_chunks`, one launch each, nearest first). Between
// launches a pixel's state lives in the output buffers: the colour sums in out_feat.xyz, the transmittance in
// out_feat.w, and last_idx with bit 31 set once the pixel has reached the cutoff; out_rgba holds the finished pixel
// after every chunk, so a launch only touches tiles that received fragments. With DEPTH the depth sum travels in
// out_depth and the last chunk visits every pixel to divide it out. The tile's bit in `alive` tells the binning of the next
// chunk whether any pixel of the tile can still take a fragment.
__device__ __forceinline__ float2 splat2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float& at(float2& v, int p) { return p == 0 ? v.x : v.y; }
__device__ __forceinline__ float fast_ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }

constexpr uint32_t DONE_BIT = 0x80000000u;

// Alpha of a staged fragment at the two pixels, zero where a pixel does not see it.
__device__ __forceinline__ float2 fragment_alpha(const float4& q0, const float4& q1, const float4& q2, const float2& pcx, const float2& pcy) {
  const float2 dy = __fadd2_rn(pcy, make_float2(q0.z, q0.w)), dx = __fadd2_rn(pcx, make_float2(q0.x, q0.y));
  const float2 sigma = __ffma2_rn(dx, __ffma2_rn(dx, make_float2(q1.x, q1.y), __fmul2_rn(make_float2(q1.z, q1.w), dy)),
                                  __fmul2_rn(__fmul2_rn(make_float2(q2.x, q2.y), dy), dy));
  const float2 e = __fmul2_rn(sigma, splat2(-1.4426950408889634f));
  // alpha >= 1/255 is 0 <= sigma <= power: one comparison of bit patterns (neither is ever -0). The exponent is at most
  // log2(255) in size there, so that flushing denormals changes nothing.
  const float a0 = __float_as_uint(sigma.x) <= __float_as_uint(q2.w) ? fminf(ALPHA_MAX, q2.z * fast_ex2(e.x)) : 0.f;
  const float a1 = __float_as_uint(sigma.y) <= __float_as_uint(q2.w) ? fminf(ALPHA_MAX, q2.z * fast_ex2(e.y)) : 0.f;
  return make_float2(a0, a1);
}

// What the forward leaves for the backward (common.cuh): nothing, checkpoints of the running sums, or of each segment's sums.
enum Checkpoints { NONE = 0, RUNNING = 1, PER_SEGMENT = 2 };

template <int CKPT, bool DEPTH, bool CHUNKED, bool FEAT>
__global__ void __launch_bounds__(FWD_WARPS * 32) raster_fwd_kernel(
    uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ vals_sorted, const float4* __restrict__ proj0, const float4* __restrict__ proj1,
    const float4* __restrict__ proj2, int W, int H, int tiles_x, int n_tiles, float3 bg, float4* __restrict__ out_rgba, float4* __restrict__ out_feat,
    float* __restrict__ out_depth, uint32_t* __restrict__ last_idx, int chunk, int n_chunks, unsigned long long* __restrict__ alive,
    const float2* __restrict__ proj3, float4* __restrict__ ckpt, int seg_shift, float4* __restrict__ feat_acc) {
  after_previous();
  constexpr bool BWD = CKPT != NONE;
  // CHUNKED with FEAT (forward only): between chunks out_feat.xyz carries the colour sums, so the feature sums of a
  // pixel travel in feat_acc and move into out_feat.xyz when the last chunk, which then visits every pixel, is done.
  static_assert(!(FEAT && CHUNKED && BWD), "the chunked backward reads the colour sums from out_feat.xyz");
  __shared__ float4 s_staged[FWD_WARPS][FWD_BATCH][FEAT ? 6 : 5];   // a fragment's constants, most of them twice, as operands of packed arithmetic
  float2 f0 = splat2(0.f), f1 = f0, f2 = f0;   // composited feature lanes (raster_fwd.cu:52)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x * FWD_WARPS + warp;
  if (tile >= n_tiles) return;
  const int tx = tile % tiles_x, ty = tile / tiles_x;
  const int px0 = tx * RT_W + (lane & 3) * 2, py = ty * RT_W + (lane >> 2);
  const bool in0 = px0 < W && py < H, in1 = px0 + 1 < W && py < H;
  const float2 pcx = make_float2((float)px0 + 0.5f, (float)px0 + 1.5f), pcy = splat2((float)py + 0.5f);
  const uint2 range = tile_ranges[tile];
  const bool first = !CHUNKED || chunk == 0, final = !CHUNKED || chunk == n_chunks - 1;
  if (CHUNKED && !first && range.y <= range.x && !(final && (DEPTH || FEAT))) return;   // nothing of this chunk lands here: pixels, state and flag stay
  float2 T = splat2(1.f), r = splat2(0.f), g = r, b = r, zs = r;   // of the two pixels
  bool open[2] = {in0, in1};   // the pixel can take another fragment
  uint32_t last[2] = {range.x, range.x};
  if (CHUNKED && !first) {
#pragma unroll
    for (int p = 0; p < 2; p++) {
      if (p == 0 ? in0 : in1) {
        const int pix = py * W + px0 + p;
        const float4 acc = out_feat[pix];
        at(r, p) = acc.x; at(g, p) = acc.y; at(b, p) = acc.z; at(T, p) = acc.w;
        if constexpr (DEPTH) at(zs, p) = out_depth[pix];
        if constexpr (FEAT) { const float4 fa = feat_acc[pix]; at(f0, p) = fa.x; at(f1, p) = fa.y; at(f2, p) = fa.z; }
        const uint32_t l = last_idx[pix];
        open[p] = (l & DONE_BIT) == 0u;
        last[p] = l & ~DONE_BIT;
      }
    }
  }
  // Checkpoints for the backward's segmented replay (see common.cuh): the state a later chunk starts a tile with, and
  // the state before every (1 << seg_shift)-th fragment of the list.
  const int q = CHUNKED ? chunk * n_tiles + tile : tile;
  float2 sr = splat2(0.f), sg = sr, sb = sr;   // PER_SEGMENT: colour sums of the segment at hand
  uint32_t seg_now = 0;
  auto checkpoint = [&](uint32_t seg) {
    float4* dst = ckpt + (size_t)ckpt_slot(range.x, q, seg, seg_shift) * RT_PX + lane * 2;
    if constexpr (CKPT == PER_SEGMENT) {   // the sums of the segment before the boundary
      dst[0] = make_float4(sr.x, sg.x, sb.x, T.x); dst[1] = make_float4(sr.y, sg.y, sb.y, T.y);
      sr = sg = sb = splat2(0.f);
      seg_now = seg;
    } else {
      dst[0] = make_float4(r.x, g.x, b.x, T.x); dst[1] = make_float4(r.y, g.y, b.y, T.y);
    }
  };
  if (BWD && CHUNKED && !first && range.y > range.x) checkpoint(0u);
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
  for (uint32_t start = range.x; start < range.y; start += FWD_BATCH) {
    if (!__any_sync(0xffffffffu, open[0] || open[1])) break;
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
    gather(start + FWD_BATCH);
    // Fragments are taken FWD_GROUP at a time: first everything that does not depend on the pixels' running state (sigma,
    // the hit test, alpha with its exponential) for the whole group, so that those chains overlap, then the short serial
    // part (transmittance and colour sums) fragment by fragment in list order.
    const float4 (*staged)[FEAT ? 6 : 5] = s_staged[warp];
    const uint32_t remaining = min((uint32_t)FWD_BATCH, range.y - start);
    if (odd) {
#pragma unroll 1
      for (uint32_t t = 0; t < remaining; t++) {
        const float2 alpha = fragment_alpha(staged[t][0], staged[t][1], staged[t][2], pcx, pcy);
        const float4 q3 = staged[t][3], q4 = staged[t][4];
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const float al = p == 0 ? alpha.x : alpha.y, next_T = at(T, p) * (1.f - al);
          open[p] = open[p] && next_T > T_CUTOFF;
          if (!open[p] || al == 0.f) continue;
          const float vis = al * at(T, p);
          at(r, p) += q3.x * vis; at(g, p) += q3.z * vis; at(b, p) += q4.x * vis;
          if constexpr (CKPT == PER_SEGMENT) { at(sr, p) += q3.x * vis; at(sg, p) += q3.z * vis; at(sb, p) += q4.x * vis; }
          if constexpr (DEPTH) at(zs, p) += vis * q4.z;
          if constexpr (FEAT) { const float4 q5 = staged[t][5]; at(f0, p) += q5.x * vis; at(f1, p) += q5.y * vis; at(f2, p) += q5.z * vis; }
          at(T, p) = next_T;
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
#pragma unroll
      for (int u = 0; u < FWD_GROUP; u++) {
        const uint32_t t = t0 + (uint32_t)u;
        // The fragment that would saturate a pixel closes it, and is not taken. A pixel that does not see the fragment has its
        // transmittance multiplied by one, and its sums take zeros.
        const float2 next_T = __fmul2_rn(T, through[u]);
        open[0] = open[0] && next_T.x > T_CUTOFF; open[1] = open[1] && next_T.y > T_CUTOFF;
        const float2 a = make_float2(open[0] ? alpha[u].x : 0.f, open[1] ? alpha[u].y : 0.f);
        const float4 q3 = staged[t][3], q4 = staged[t][4];
        const float2 vis = __fmul2_rn(a, T), cr = make_float2(q3.x, q3.y), cg = make_float2(q3.z, q3.w), cb = make_float2(q4.x, q4.y);
        r = __ffma2_rn(cr, vis, r); g = __ffma2_rn(cg, vis, g); b = __ffma2_rn(cb, vis, b);
        if constexpr (CKPT == PER_SEGMENT) { sr = __ffma2_rn(cr, vis, sr); sg = __ffma2_rn(cg, vis, sg); sb = __ffma2_rn(cb, vis, sb); }
        if constexpr (DEPTH) zs = __ffma2_rn(vis, make_float2(q4.z, q4.w), zs);
        if constexpr (FEAT) {
          const float4 q5 = staged[t][5];
          f0 = __ffma2_rn(splat2(q5.x), vis, f0); f1 = __ffma2_rn(splat2(q5.y), vis, f1); f2 = __ffma2_rn(splat2(q5.z), vis, f2);
        }
        T.x = open[0] ? next_T.x : T.x; T.y = open[1] ? next_T.y : T.y;
        last[0] = a.x != 0.f ? start + t + 1 : last[0]; last[1] = a.y != 0.f ? start + t + 1 : last[1];
      }
    }
  }
#pragma unroll
  for (int p = 0; p < 2; p++) {
    if (p == 0 ? in0 : in1) {
      const int pix = py * W + px0 + p;
      out_rgba[pix] = make_float4(at(r, p) + at(T, p) * bg.x, at(g, p) + at(T, p) * bg.y, at(b, p) + at(T, p) * bg.z, 1.f - at(T, p));
      if constexpr (CHUNKED) {
        if (FEAT && final) out_feat[pix] = make_float4(at(f0, p), at(f1, p), at(f2, p), at(T, p));
        else out_feat[pix] = make_float4(at(r, p), at(g, p), at(b, p), at(T, p));
        if constexpr (FEAT) { if (!final) feat_acc[pix] = make_float4(at(f0, p), at(f1, p), at(f2, p), 0.f); }
        if constexpr (DEPTH) out_depth[pix] = !final ? at(zs, p) : ((1.f - at(T, p)) > 0.05f ? at(zs, p) / (1.f - at(T, p)) : INFINITY);
        last_idx[pix] = last[p] | (open[p] ? 0u : DONE_BIT);
      } else {
        out_feat[pix] = make_float4(at(f0, p), at(f1, p), at(f2, p), at(T, p));
        if constexpr (DEPTH) out_depth[pix] = (1.f - at(T, p)) > 0.05f ? at(zs, p) / (1.f - at(T, p)) : INFINITY;
        if constexpr (BWD) last_idx[pix] = last[p];
      }
    }
  }
  if (CHUNKED && !final) {
    const bool more = __any_sync(0xffffffffu, open[0] || open[1]);
    if (lane == 0 && !more) atomicAnd(alive + (size_t)(ty >> 3) * ((tiles_x + 7) >> 3) + (tx >> 3), ~(1ull << ((ty & 7) * 8 + (tx & 7))));
  }
  if constexpr (BWD) {
    // The backward never needs to look past the last fragment any pixel used. (A pixel whose last fragment lies in an
    // earlier chunk contributes this chunk's start: an empty range.)
    uint32_t m = max(last[0], last[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if constexpr (CHUNKED) m = min(max(m, range.x), range.y);
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
}

}  // namespace
}  // namespace b2k

using namespace b2k;

namespace b2k {
// One chunk of a chunked view (n_chunks > 1), or the whole view (n_chunks <= 1).
int launch_raster_fwd(const B2kCtx* c, const B2kRenderOpts* o, int chunk, int n_chunks, unsigned long long* alive, cudaStream_t s) {
  const float3 bg = make_float3(o->bg[0], o->bg[1], o->bg[2]);
  uint2* ranges = (uint2*)c->tile_ranges + (n_chunks > 1 ? (size_t)chunk * c->n_tiles : 0);
#define L(B, D, C, F) launch_next(raster_fwd_kernel<B, D, C, F>, div_up(c->n_tiles, FWD_WARPS), FWD_WARPS * 32, 0, s, ranges, c->vals_sorted, (const float4*)c->proj0, \
    (const float4*)c->proj1, (const float4*)c->proj2, c->W, c->H, c->tiles_x, c->n_tiles, bg, (float4*)c->out_rgba, (float4*)c->out_feat, c->out_depth, c->last_idx, \
    chunk, n_chunks, alive, (const float2*)c->proj3, o->bwd_info ? bwd_ckpt_ptr(c) : nullptr, seg_shift_of(c->n_tiles), (n_chunks > 1 && o->feat_mode != 0) ? (float4*)c->bwd_scratch : nullptr)
#define LB(B) do { if (n_chunks > 1) { if (c->out_depth) L(B, true, true, false); else L(B, false, true, false); } \
    else if (o->feat_mode != 0) { if (c->out_depth) L(B, true, false, true); else L(B, false, false, true); } \
    else { if (c->out_depth) L(B, true, false, false); else L(B, false, false, false); } } while (0)
  if (n_chunks > 1 && o->feat_mode != 0) {   // forward only (checked by the caller): the scratch of the backward carries the feature sums
    if (c->out_depth) L(NONE, true, true, true); else L(NONE, false, true, true);
  } else if (!o->bwd_info) LB(NONE);
  else if (short_segments(c->n_tiles)) LB(PER_SEGMENT);
  else LB(RUNNING);
#undef LB
#undef L
  return check_launch();
}
}  // namespace b2k

extern "C" int b2k_raster_fwd(const B2kCtx* c, const B2kRenderOpts* o, b2k_stream_t stream) {
  B2K_REQUIRE(c && o && c->tile_ranges && c->vals_sorted && c->proj0 && c->proj1 && c->proj2 && c->out_rgba && c->out_feat);
  B2K_REQUIRE(!o->bwd_info || (c->last_idx && c->bwd_scratch));
  B2K_REQUIRE(c->W > 0 && c->H > 0 && c->n_tiles == c->tiles_x * c->tiles_y);
  if (o->bwd_info && c->bwd_scratch_bytes < b2k_bwd_scratch_bytes(c->W, c->H, c->n_chunks, c->isect_cap)) return B2K_ERR_CAPACITY;
  B2K_REQUIRE(o->feat_mode >= 0 && o->feat_mode <= 2 && (o->feat_mode == 0 || c->proj3));
  return launch_raster_fwd(c, o, 0, 1, nullptr, (cudaStream_t)stream);
}
