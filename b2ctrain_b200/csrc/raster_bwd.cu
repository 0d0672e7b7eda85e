// Backward through compositing: per-pixel reverse replay of the forward, per-fragment gradients reduced across the
// tile and accumulated per splat. Reference semantics: raster_bwd_kernel (src/gpu/raster_bwd.cu:11-143).
//
// Work decomposition (differs from the reference on purpose):
//   * A tile's fragment list is cut into SEGMENTS (128 fragments; 32 in a small image). The forward leaves the per-pixel state (colour
//     sums, transmittance) at every segment boundary (and where a depth chunk of a chunked view hands over to the next),
//     so each segment can be replayed on its own (common.cuh: lengths, and how the colour behind a boundary is found).
//     A small kernel lists the (range, segment) items; a persistent grid of independent warps pulls them from a
//     counter. The longest list of a view no longer decides the kernel's duration, and no warp slot idles while another
//     warp still has a thousand fragments to go.
//   * One WARP owns an item; each lane replays two horizontally adjacent pixels, two fragments at a time. Packed fp32x2
//     operations run over the two FRAGMENTS of a pair: their constants lie side by side in shared memory and the pixels'
//     constants are held doubled in registers, so no operand has to be assembled (packed over the two pixels, every
//     fragment constant needed a copy: 139 instead of 115 warp instructions per fragment). Only the short chain that carries the
//     transmittance and the colour behind runs one fragment after the other. A pair that no pixel of the tile sees is
//     rejected after the sigma test; otherwise the math is branch-free (a pixel that does not see a fragment has alpha = 0
//     and adds exact zeros).
//   * The colour behind a pixel is only ever needed through its product with the pixel's gradient, so the replay carries
//     that one scalar, not three colour sums.
//   * Reduction across the tile. All eleven lanes of a fragment are sums over the pixels of m and vis times factors
//     that need no more than the pixel's place: with m = -dL/dsigma and (X, Y) the pixel's offset from the splat's centre, the
//     position and conic lanes follow from the six moments of m (1, X, Y, XX, XY, YY), the colour lanes from vis times the
//     pixel's gradient.
//     So a lane leaves only (m, vis) of its pixels and its share of the refine lane in shared memory, and once RED_P pairs
//     are pending the warp turns round: each lane takes a pair and a row of the tile; shuffles join the
//     rows, and the lanes of a fragment share out its global reductions.
//
// Bound by instruction issue (59 % of the slots busy with 20 warps per SM; 75 fp32 operations, an ex2, an rcp and a square
// root per fragment-pixel), not by memory. Against the form before (eleven products per pixel pair summed in columns, 128
// fragments to a segment in every image), warm: 1920x1080, 500k splats, 0.75M fragments 187 -> 132 us; 1024x1024, 1M heavy-tailed splats,
// 2.1M fragments 486 -> 310 us; 64x64, 2k splats 53 -> 17 us.
#include "common.cuh"

namespace b2k {
namespace {

constexpr int BWD_WARPS = 4;                 // warps per CTA (independent: the CTA shape only sets the residency granularity)
constexpr int BWD_CTAS_PER_SM = 5;            // 96 registers: 131 us on the view below; 138 with 4 CTAs, 140 with 5.5, 139 with 6
constexpr int BWD_BATCH = 32;                 // fragments staged per warp and batch
constexpr int RED_P = 4;                      // fragment pairs pending before a reduction (8 save shuffles, but cost the memory of a third of the warps: 136 us)
constexpr int RED_STRIDE = 33;                // 16-byte words per pending pair, one of skew: conflict-free reads
constexpr int REF_STRIDE = 17;                // the same for eight bytes per lane
constexpr int V_STRIDE = 13;                  // 16-byte words per tile row of doubled pixel gradients (twelve, and one of skew)
constexpr unsigned FULL = 0xffffffffu;
static_assert(RT_W * RED_P == 32, "in a reduction a lane takes one row of one pair");

// Two staged fragments, the later one (nearer the end of the list) in .x. Constants of the packed math are folded once per
// fragment, not once per pixel; halving and negating are exact.
struct __align__(16) StagedPair {
  float2 nmx, nmy;    // -centre
  float2 h00, c01;    // c00 / 2, c01
  float2 h11, nop;    // c11 / 2, -opacity
  float2 power, r;    // cut-off (its bits are compared as integers: never negative); colour, clamped at zero
  float2 g, b;
};

// A warp's shared memory.
struct WarpMem {
  float4 nm[RED_P * RED_STRIDE];      // [pair][lane]: -m of (fragment x, y) at the lane's first pixel, then at its second
  float4 nvis[RED_P * RED_STRIDE];    // the same of -vis
  float4 ref[RED_P * REF_STRIDE];     // [pair][lane]: refine lane of (fragment x, y), summed over the lane's two pixels
  float4 v[RT_W * V_STRIDE];          // [row][column pair]: gradients of the two pixels, doubled: rr gg bb rr gg bb
  StagedPair frag[BWD_BATCH / 2];
  uint32_t gid[BWD_BATCH];            // [pair][x, y]
  uint32_t flags[BWD_BATCH];          // bits 0..2: colour clamped at zero
  uint32_t pending[RED_P];            // staged pair of each pending one
};
static_assert(sizeof(StagedPair) == 80 && sizeof(WarpMem) % 16 == 0, "layout");

constexpr size_t BWD_SMEM = BWD_WARPS * sizeof(WarpMem);

__device__ __forceinline__ float fast_sqrt(float x) { float r; asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float fast_rcp(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float2 f2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// Work list of the replay: one item (range index = chunk * n_tiles + tile, segment) per segment of every
// non-empty range the forward left. Order is irrelevant (items are independent); work[0] receives the count.
__global__ void __launch_bounds__(256) bwd_items_kernel(const uint2* __restrict__ tile_ranges, int n_ranges, int seg_shift, uint2* __restrict__ items, uint32_t* __restrict__ work) {
  after_previous();
  const int lane = threadIdx.x & 31;
  for (int q0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31; q0 < n_ranges; q0 += gridDim.x * blockDim.x) {
    const int q = q0 + lane;
    uint32_t segs = 0;
    if (q < n_ranges) { const uint2 rg = tile_ranges[q]; segs = rg.y > rg.x ? (rg.y - rg.x + (1u << seg_shift) - 1u) >> seg_shift : 0u; }
    uint32_t incl = segs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const uint32_t u = __shfl_up_sync(FULL, incl, o); if (lane >= o) incl += u; }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    if (total == 0u) continue;
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(work, total);
    base = __shfl_sync(FULL, base, 31) + incl - segs;
    for (uint32_t s = 0; s < segs; s++) items[base + s] = make_uint2((uint32_t)q, s);
  }
}

// Short segments: the same list, and the segments' colour sums that the forward left turned into the colour behind each
// boundary. One warp per tile walks its checkpoints from the far end: slot j of a range holds the sums of segment j - 1,
// slot 0 those of the last one; afterwards slot j holds the colour from boundary j on. A second backward on the same forward
// finds them so (BWD_SUMMED, which the forward clears and the replay sets) and lists the items only.
__global__ void __launch_bounds__(128) bwd_suffix_kernel(const uint2* __restrict__ tile_ranges, int n_tiles, int n_chunks, int seg_shift, uint2* __restrict__ items,
                                                         uint32_t* __restrict__ work, float4* __restrict__ ckpt) {
  after_previous();
  const int lane = threadIdx.x & 31, tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (tile >= n_tiles) return;
  const bool summed = work[BWD_SUMMED] != 0u;
  float3 acc[2] = {make_float3(0.f, 0.f, 0.f), make_float3(0.f, 0.f, 0.f)};
  for (int c = n_chunks - 1; c >= 0; c--) {
    const int q = c * n_tiles + tile;
    const uint2 range = tile_ranges[q];
    if (range.y <= range.x) continue;
    const uint32_t segs = (range.y - range.x + (1u << seg_shift) - 1u) >> seg_shift;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(work, segs);
    base = __shfl_sync(FULL, base, 0);
    for (uint32_t s = lane; s < segs; s += 32) items[base + s] = make_uint2((uint32_t)q, s);
    if (summed) continue;
    float4* at = ckpt + (size_t)ckpt_slot(range.x, q, 0u, seg_shift) * RT_PX + lane * 2;
    float4 own[2] = {at[0], at[1]};   // the sums of the segment behind the boundary that comes next
    for (uint32_t hi = segs; hi > 0u;) {   // boundaries hi - 1 .. hi - count, four in flight
      constexpr uint32_t U = 4;
      const uint32_t count = hi < U ? hi : U;
      float4 v[U][2];
#pragma unroll
      for (uint32_t u = 0; u < U; u++)
        if (u < count && hi - 1u - u > 0u) { v[u][0] = at[(size_t)(hi - 1u - u) * RT_PX]; v[u][1] = at[(size_t)(hi - 1u - u) * RT_PX + 1]; }
#pragma unroll
      for (uint32_t u = 0; u < U; u++) {
        if (u >= count) break;
        const uint32_t j = hi - 1u - u;
#pragma unroll
        for (int p = 0; p < 2; p++) {
          acc[p].x += own[p].x; acc[p].y += own[p].y; acc[p].z += own[p].z;
          float* dst = reinterpret_cast<float*>(at + (size_t)j * RT_PX + p);
          dst[0] = acc[p].x; dst[1] = acc[p].y; dst[2] = acc[p].z;
          own[p] = v[u][p];
        }
      }
      hi -= count;
    }
  }
}

enum Form { WHOLE = 0, CHUNKED = 1, SHORT = 2 };   // where the colour behind a boundary comes from

template <int FORM>
__global__ void __launch_bounds__(BWD_WARPS * 32, BWD_CTAS_PER_SM) raster_bwd_kernel(
    const uint2* __restrict__ tile_ranges, const uint32_t* __restrict__ vals_sorted, const float4* __restrict__ proj0, const float4* __restrict__ proj1,
    const float4* __restrict__ proj2, const float4* __restrict__ out_rgba, const float4* __restrict__ out_feat, const uint32_t* __restrict__ last_idx,
    const float4* __restrict__ v_out, int W, int H, int tiles_x, int n_tiles, float3 bg, float* __restrict__ v_splat, uint32_t* __restrict__ vis_flag,
    float* __restrict__ vis_weight, int n_chunks, const uint2* __restrict__ items, uint32_t* __restrict__ work, const float4* __restrict__ ckpt,
    int seg_shift, float out_scale) {
  after_previous();
  extern __shared__ __align__(16) unsigned char s_bytes[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WarpMem& sm = reinterpret_cast<WarpMem*>(s_bytes)[warp];
  const float aspect = (float)H / (float)W;
  const int red_p = lane % RED_P, red_row = lane / RED_P;   // in a reduction: this lane's pair and tile row
  const float2 aspect2 = f2(aspect);
  const uint32_t n_items = work[0];
  if (FORM == SHORT && blockIdx.x == 0 && threadIdx.x == 0) work[BWD_SUMMED] = 1u;

  for (;;) {
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(work + 1, 1u);   // (drawn ahead, while the last item is replayed, it costs balance: 131 -> 146 us)
    it = __shfl_sync(FULL, it, 0);
    if (it >= n_items) break;
    const uint2 item = items[it];
    const int q = (int)item.x, chunk = q / n_tiles, tile = q - chunk * n_tiles;
    const uint2 range = tile_ranges[q];
    const uint32_t seg_lo = range.x + (item.y << seg_shift);
    const uint32_t seg_hi = min(seg_lo + (1u << seg_shift), range.y);
    // The records of a batch are gathered one batch ahead, into registers: the two dependent loads (list entry, then the
    // splat's records) are in flight while the batch behind them is replayed.
    uint32_t n_gid = 0u;
    float4 n_a = make_float4(0.f, 0.f, 0.f, 0.f), n_c = n_a, n_col = n_a;
    auto gather = [&](uint32_t end) {   // the batch that ends at `end`
      if (end <= seg_lo) return;
      const uint32_t cnt = min(end - seg_lo, (uint32_t)BWD_BATCH);
      if ((uint32_t)lane < cnt) {
        n_gid = vals_sorted[end - cnt + lane];
        n_a = proj0[n_gid]; n_c = proj1[n_gid]; n_col = proj2[n_gid];
      }
    };
    gather(seg_hi);
    // The state behind this segment: the forward's checkpoint at its far boundary; for the last segment of a range,
    // the state with which the next non-empty range of the tile (a later depth chunk) started; else the final state.
    long long slot = -1;
    if (seg_hi < range.y) {
      slot = (long long)ckpt_slot(range.x, q, item.y + 1u, seg_shift);
    } else {
      for (int c2 = chunk + 1; c2 < n_chunks; c2++) {
        const uint2 r2 = tile_ranges[(size_t)c2 * n_tiles + tile];
        if (r2.y > r2.x) { slot = (long long)ckpt_slot(r2.x, c2 * n_tiles + tile, 0u, seg_shift); break; }
      }
    }
    const int tx = tile % tiles_x, ty = tile / tiles_x;
    const int px0 = tx * RT_W + (lane & 3) * 2, py = ty * RT_W + (lane >> 2);   // this lane's pixel pair (px0, px0 + 1) on row py
    // Per pixel: transmittance behind the fragments still ahead; dL/dalpha's part common to all of them less the colour behind.
    float T_[2] = {0.f, 0.f}, Q_[2] = {0.f, 0.f}, v_[2][3] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}}, k_[2] = {0.f, 0.f};
    uint32_t last0 = 0u, last1 = 0u;   // outside the image: sees no fragment
    {
      uint32_t last[2] = {0u, 0u};
#pragma unroll
      for (int p = 0; p < 2; p++) {
        const int px = px0 + p;
        if (px < W && py < H) {
          const int pix = py * W + px;
          const float4 vo = v_out[pix], fin = out_feat[pix], img = out_rgba[pix];
          const float T_fin = fin.w;
          T_[p] = T_fin;
          v_[p][0] = vo.x; v_[p][1] = vo.y; v_[p][2] = vo.z;
          Q_[p] = (vo.w - (bg.x * vo.x + bg.y * vo.y + bg.z * vo.z)) * T_fin;
          k_[p] = (float)W / fmaxf(img.w, 1e-5f);
          last[p] = last_idx[pix] & 0x7FFFFFFFu;   // a chunked forward keeps its saturation flag in bit 31
          if (slot >= 0 && last[p] > seg_hi) {     // the pixel went on past this segment: fragments behind it hold colour
            const float4 ck = ckpt[(size_t)slot * RT_PX + lane * 2 + p];
            float3 behind = make_float3(ck.x, ck.y, ck.z);
            if constexpr (FORM != SHORT) {   // final sums (a chunked forward keeps them in out_feat; otherwise the image minus the background term) less the checkpoint's
              const float3 sum = FORM == CHUNKED ? make_float3(fin.x, fin.y, fin.z) : make_float3(img.x - T_fin * bg.x, img.y - T_fin * bg.y, img.z - T_fin * bg.z);
              behind = make_float3(sum.x - ck.x, sum.y - ck.y, sum.z - ck.z);
            }
            T_[p] = ck.w;
            Q_[p] -= behind.x * vo.x + behind.y * vo.y + behind.z * vo.z;
          }
        }
      }
      last0 = last[0]; last1 = last[1];
    }
    const float2 v2[2][3] = {{f2(v_[0][0]), f2(v_[0][1]), f2(v_[0][2])}, {f2(v_[1][0]), f2(v_[1][1]), f2(v_[1][2])}};
    const float2 k2[2] = {f2(k_[0]), f2(k_[1])};
    __syncwarp();   // the last item's reduction has read these
    {
      float4* dst = sm.v + (lane >> 2) * V_STRIDE + (lane & 3) * 3;
      dst[0] = make_float4(v_[0][0], v_[0][0], v_[0][1], v_[0][1]);
      dst[1] = make_float4(v_[0][2], v_[0][2], v_[1][0], v_[1][0]);
      dst[2] = make_float4(v_[1][1], v_[1][1], v_[1][2], v_[1][2]);
    }
    const float2 pcy2 = f2((float)py + 0.5f);
    const float2 pcx2[2] = {f2((float)px0 + 0.5f), f2((float)px0 + 0.5f + 1.f)};
    const float tile_x = (float)(tx * RT_W) + 0.5f, tile_y = (float)(ty * RT_W) + 0.5f;   // centre of the tile's first pixel
    int n_pending = 0;

    // Sums over the tile of what the pending pairs left, then the splats' gradient lanes.
    auto flush = [&]() {
      __syncwarp();
      const StagedPair& fr2 = sm.frag[red_p < n_pending ? sm.pending[red_p] : 0u];
      const float2 nmx = fr2.nmx;
      float2 cr = f2(0.f), cg = f2(0.f), cb = f2(0.f), vis = f2(0.f), M0 = f2(0.f), Sx = f2(0.f), Sxx = f2(0.f);
      const int row_at = red_p * RED_STRIDE + red_row * 4;
      const float4 *pm = sm.nm + row_at, *pv = sm.nvis + row_at, *pr = sm.ref + red_p * REF_STRIDE + red_row * 2, *pg = sm.v + red_row * V_STRIDE;
      auto moments = [&](float2 m, float px) {   // about the splat's centre
        const float2 dx = __fadd2_rn(f2(px), nmx), md = __fmul2_rn(m, dx);
        M0 = __fadd2_rn(M0, m); Sx = __fadd2_rn(Sx, md); Sxx = __ffma2_rn(md, dx, Sxx);
      };
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float4 m4 = pm[c], n4 = pv[c], g0 = pg[c * 3], g1 = pg[c * 3 + 1], g2 = pg[c * 3 + 2];
        moments(lo2(m4), tile_x + (float)(2 * c)); moments(hi2(m4), tile_x + (float)(2 * c + 1));
        cr = __ffma2_rn(lo2(n4), lo2(g0), cr); cg = __ffma2_rn(lo2(n4), hi2(g0), cg); cb = __ffma2_rn(lo2(n4), lo2(g1), cb);
        cr = __ffma2_rn(hi2(n4), hi2(g1), cr); cg = __ffma2_rn(hi2(n4), lo2(g2), cg); cb = __ffma2_rn(hi2(n4), hi2(g2), cb);
        vis = __fadd2_rn(vis, __fadd2_rn(lo2(n4), hi2(n4)));
      }
      const float2 ref = __fadd2_rn(__fadd2_rn(lo2(pr[0]), hi2(pr[0])), __fadd2_rn(lo2(pr[1]), hi2(pr[1])));
      const float2 dy = __fadd2_rn(f2(tile_y + (float)red_row), fr2.nmy), Sy = __fmul2_rn(dy, M0), Sxy = __fmul2_rn(dy, Sx), Syy = __fmul2_rn(dy, Sy);
      // The rows' lanes joined: the first step leaves fragment x with the lower half of the warp and y with the upper.
      const bool upper = (lane & 16) != 0;
      float t[11];
      {
        const float2 q[11] = {M0, Sx, Sy, Sxx, Sxy, Syy, cr, cg, cb, vis, ref};
#pragma unroll
        for (int k = 0; k < 11; k++) t[k] = (upper ? q[k].y : q[k].x) + __shfl_xor_sync(FULL, upper ? q[k].x : q[k].y, 16);
      }
#pragma unroll
      for (int o = 8; o >= RED_P; o >>= 1)
#pragma unroll
        for (int k = 0; k < 11; k++) t[k] += __shfl_xor_sync(FULL, t[k], o);
      if (red_p < n_pending && t[9] != 0.f) {   // some pixel sees the fragment: its blend weight is not zero
        const uint32_t k = sm.pending[red_p], e = 2u * k + (upper ? 1u : 0u), gid = sm.gid[e], flags = sm.flags[e];
        const float* fr = reinterpret_cast<const float*>(&sm.frag[k]) + (upper ? 1 : 0);
        // The stored m and vis carry a minus sign.
        const float c00 = 2.f * fr[4], c01 = fr[6], c11 = 2.f * fr[8];
        // Gradient lanes: xy 2, conic 3, rgb 3, opacity, refine, shared out over the four lanes that hold the
        // fragment's sums. out_scale undoes a scale the caller put on the pixel gradients (1 unless asked
        // for); the blend weight is no gradient.
        float* o = v_splat + (size_t)gid * GRAD_LANES;
        auto add = [&](int at, float v) { v *= out_scale; if (v != 0.f) atomicAdd(o + at, v); };
        const int part = red_row & 3;
        float o0, o1 = 0.f, o2 = 0.f;
        if (part == 0) { o0 = -(c00 * t[1] + c01 * t[2]); o1 = -(c01 * t[1] + c11 * t[2]); o2 = 0.5f * t[3]; }
        else if (part == 1) { o0 = t[4]; o1 = 0.5f * t[5]; o2 = (flags & 1u) ? 0.f : -t[6]; }
        else if (part == 2) { o0 = (flags & 2u) ? 0.f : -t[7]; o1 = (flags & 4u) ? 0.f : -t[8]; o2 = __fdividef(t[0], fr[10]); }
        else o0 = t[10];
        add(part * 3, o0); add(part * 3 + 1, o1); add(part * 3 + 2, o2);
        if (part == 3) { vis_flag[gid] = 1u; if (vis_weight) atomicAdd(vis_weight + gid, -t[9]); }
      }
      __syncwarp();
      n_pending = 0;
    };

    for (uint32_t batch_end = seg_hi; batch_end > seg_lo;) {
      const uint32_t remaining = batch_end - seg_lo;
      const uint32_t count = remaining < (uint32_t)BWD_BATCH ? remaining : (uint32_t)BWD_BATCH;
      const uint32_t batch_start = batch_end - count;
      {
        // Fragments are numbered from the batch's end: e = 0 is replayed first; an odd batch ends with one nobody can see.
        const int e = (int)count - 1 - lane;
        const bool real = e >= 0, filler = e == -1 && (count & 1u) != 0u;
        if (real || filler) {
          const int at = real ? e : (int)count;
          float* d = reinterpret_cast<float*>(&sm.frag[at >> 1]) + (at & 1);
          const bool drawn = real && n_c.w >= 0.f;   // a negative cut-off hits nothing: opacity zero keeps it that way
          d[0] = real ? -n_a.x : 0.f; d[2] = real ? -n_a.y : 1e6f; d[4] = real ? 0.5f * n_a.z : 0.f; d[6] = real ? n_a.w : 0.f;
          d[8] = real ? 0.5f * n_c.x : 1.f; d[10] = drawn ? -n_c.y : 0.f; d[12] = drawn ? n_c.w : 0.f;
          d[14] = fmaxf(n_col.x, 0.f); d[16] = fmaxf(n_col.y, 0.f); d[18] = fmaxf(n_col.z, 0.f);
          sm.gid[at] = n_gid;
          sm.flags[at] = (n_col.x < 0.f ? 1u : 0u) | (n_col.y < 0.f ? 2u : 0u) | (n_col.z < 0.f ? 4u : 0u);
        }
      }
      // The clamp of alpha can only act on a splat this opaque (bit e: fragment e of the batch). Whether a pixel stopped
      // inside the batch decides if its last fragment has to be looked at.
      const uint32_t clamps = __brev(__ballot_sync(FULL, (uint32_t)lane < count && n_c.y > ALPHA_MAX)) >> (BWD_BATCH - count);
      const int stop0 = last0 > batch_start ? (int)min(last0 - batch_start, (uint32_t)BWD_BATCH) : 0;   // of the batch's fragments, from its start, each pixel took this many
      const int stop1 = last1 > batch_start ? (int)min(last1 - batch_start, (uint32_t)BWD_BATCH) : 0;
      const bool all_through = __all_sync(FULL, stop0 >= (int)count && stop1 >= (int)count);
      __syncwarp();
      gather(batch_start);
      const int pairs = (int)(count + 1) >> 1;
      for (int k = 0; k < pairs; k++) {
        // What does not depend on the pixels' running state: sigma, the visibility test, the exponential, alpha, 1 / (1 - alpha).
        const float4* rec = reinterpret_cast<const float4*>(&sm.frag[k]);
        const float4 q0 = rec[0], q1 = rec[1], q2 = rec[2], q3 = rec[3], q4 = rec[4];
        const float2 nmx = lo2(q0), h00 = lo2(q1), c01 = hi2(q1), nop = hi2(q2), power = lo2(q3);
        const float2 dy = __fadd2_rn(pcy2, hi2(q0)), hy = __fmul2_rn(lo2(q2), dy), wdy = __fmul2_rn(c01, dy), hyy = __fmul2_rn(hy, dy);
        float2 dx[2], inner[2], nal[2], live[2], ra[2];
        bool on[2][2];
#pragma unroll
        for (int p = 0; p < 2; p++) {   // sigma in the forward's operations
          dx[p] = __fadd2_rn(pcx2[p], nmx);
          inner[p] = __ffma2_rn(dx[p], h00, wdy);
          const float2 sigma = __ffma2_rn(dx[p], inner[p], hyy);
          // 0 <= sigma <= power as one comparison of bit patterns: neither is ever -0
          on[p][0] = __float_as_uint(sigma.x) <= __float_as_uint(power.x);
          on[p][1] = __float_as_uint(sigma.y) <= __float_as_uint(power.y);
          const float2 e2 = __fmul2_rn(sigma, f2(-1.4426950408889634f));
          live[p] = __fmul2_rn(nop, make_float2(fast_ex2(e2.x), fast_ex2(e2.y)));
        }
        if (!all_through) {
          const int i0 = (int)count - 1 - 2 * k, i1 = i0 - 1;
          on[0][0] = on[0][0] && i0 < stop0; on[0][1] = on[0][1] && i1 < stop0;
          on[1][0] = on[1][0] && i0 < stop1; on[1][1] = on[1][1] && i1 < stop1;
        }
        if (!__any_sync(FULL, on[0][0] || on[0][1] || on[1][0] || on[1][1])) continue;   // nobody in the tile sees either
#pragma unroll
        for (int p = 0; p < 2; p++) {   // -alpha; a pixel that does not see the fragment has alpha = 0 and adds exact zeros below
          live[p].x = on[p][0] ? live[p].x : 0.f; live[p].y = on[p][1] ? live[p].y : 0.f;
          nal[p] = live[p];
        }
        if ((clamps >> (2 * k)) & 3u) {   // the clamp has zero slope: m vanishes where it is active
#pragma unroll
          for (int p = 0; p < 2; p++) {
            nal[p] = make_float2(fmaxf(live[p].x, -ALPHA_MAX), fmaxf(live[p].y, -ALPHA_MAX));
            live[p] = make_float2(live[p].x < -ALPHA_MAX ? 0.f : live[p].x, live[p].y < -ALPHA_MAX ? 0.f : live[p].y);
          }
        }
        const float2 col_r = hi2(q3), col_g = lo2(q4), col_b = hi2(q4), hy2 = __fadd2_rn(hy, hy);
        float2 nm[2], nv[2], sf[2];
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const float2 oma = __fadd2_rn(f2(1.f), nal[p]);
          ra[p] = make_float2(fast_rcp(oma.x), fast_rcp(oma.y));
          const float2 d = __ffma2_rn(col_b, v2[p][2], __ffma2_rn(col_g, v2[p][1], __fmul2_rn(col_r, v2[p][0])));   // colour . pixel gradient
          float2 va;   // dL/dalpha, the later fragment first
          va.x = ra[p].x * fmaf(T_[p], d.x, Q_[p]);
          T_[p] *= ra[p].x; nv[p].x = nal[p].x * T_[p]; Q_[p] = fmaf(nv[p].x, d.x, Q_[p]);
          va.y = ra[p].y * fmaf(T_[p], d.y, Q_[p]);
          T_[p] *= ra[p].y; nv[p].y = nal[p].y * T_[p]; Q_[p] = fmaf(nv[p].y, d.y, Q_[p]);
          nm[p] = __fmul2_rn(live[p], va);         // dL/dsigma
          // Length of the screen-space position gradient per unit of |m|, in image widths.
          const float2 t1 = __ffma2_rn(dx[p], h00, inner[p]), t2 = __fmul2_rn(aspect2, __ffma2_rn(dx[p], c01, hy2));
          const float2 qq = __ffma2_rn(t1, t1, __fmul2_rn(t2, t2));
          sf[p] = __fmul2_rn(k2[p], make_float2(fast_sqrt(qq.x), fast_sqrt(qq.y)));
        }
        const int at = n_pending * RED_STRIDE + lane;
        sm.nm[at] = make_float4(nm[0].x, nm[0].y, nm[1].x, nm[1].y);
        sm.nvis[at] = make_float4(nv[0].x, nv[0].y, nv[1].x, nv[1].y);
        reinterpret_cast<float2*>(sm.ref)[n_pending * (2 * REF_STRIDE) + lane] =
            make_float2(fmaf(fabsf(nm[1].x), sf[1].x, fabsf(nm[0].x) * sf[0].x), fmaf(fabsf(nm[1].y), sf[1].y, fabsf(nm[0].y) * sf[0].y));
        if (lane == 0) sm.pending[n_pending] = (uint32_t)k;
        if (++n_pending == RED_P) flush();
      }
      if (n_pending) flush();   // the pending fragments' records are about to be replaced
      else __syncwarp();
      batch_end = batch_start;
    }
  }
}

}  // namespace
}  // namespace b2k

using namespace b2k;

extern "C" uint64_t b2k_bwd_scratch_bytes(int32_t W, int32_t H, int32_t n_chunks, uint64_t isect_cap) {
  if (W <= 0 || H <= 0) return 0;
  const uint64_t tiles = (uint64_t)div_up(W, RT_W) * div_up(H, RT_W), chunks = n_chunks > 1 ? (uint64_t)n_chunks : 1u;
  const uint64_t slots = bwd_slots(isect_cap, tiles * chunks, seg_shift_of(short_segments(tiles, isect_cap)));
  return sizeof(uint32_t) * BWD_HEADER_WORDS + sizeof(uint2) * slots + sizeof(float4) * RT_PX * slots;
}

extern "C" int b2k_raster_bwd(const B2kCtx* c, const B2kModel* m, const B2kRenderOpts* o, b2k_stream_t stream) {
  return b2k_raster_bwd_scaled(c, m, o, 1.f, stream);
}

extern "C" int b2k_raster_bwd_scaled(const B2kCtx* c, const B2kModel* m, const B2kRenderOpts* o, float grad_scale, b2k_stream_t stream) {
  B2K_REQUIRE(grad_scale > 0.f && isfinite(grad_scale));
  B2K_REQUIRE(c && m && o && c->tile_ranges && c->vals_sorted && c->proj0 && c->proj1 && c->proj2);
  B2K_REQUIRE(c->out_rgba && c->out_feat && c->last_idx && c->v_out && c->v_splat && c->vis_flag);
  B2K_REQUIRE(c->W > 0 && c->H > 0 && c->n_tiles == c->tiles_x * c->tiles_y && c->bwd_scratch);
  if (c->bwd_scratch_bytes < b2k_bwd_scratch_bytes(c->W, c->H, c->n_chunks, c->isect_cap)) return B2K_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  const float3 bg = make_float3(o->bg[0], o->bg[1], o->bg[2]);
  const int chunks = c->n_chunks > 1 ? c->n_chunks : 1;
  uint32_t* work = bwd_work_ptr(c);
  uint2* items = bwd_items_ptr(c);
  launch_clear(work, 2, nullptr, 0, s);
  const int n_ranges = chunks * c->n_tiles;
  const bool brief = short_segments(c);
  const int seg_shift = seg_shift_of(brief);
  if (brief) launch_next(bwd_suffix_kernel, div_up(c->n_tiles, 4), 128, 0, s, (const uint2*)c->tile_ranges, c->n_tiles, chunks, seg_shift, items, work, bwd_ckpt_ptr(c));
  else launch_next(bwd_items_kernel, min(div_up(n_ranges, 256), sm_count() * 4), 256, 0, s, (const uint2*)c->tile_ranges, n_ranges, seg_shift, items, work);
  // Persistent grid: as many CTAs as an SM holds.
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
    B2K_CUDA(cudaFuncSetAttribute(raster_bwd_kernel<WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BWD_SMEM));
    B2K_CUDA(cudaFuncSetAttribute(raster_bwd_kernel<CHUNKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BWD_SMEM));
    B2K_CUDA(cudaFuncSetAttribute(raster_bwd_kernel<SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BWD_SMEM));
    attr_set[dev] = true;
  }
  const int ctas = sm_count() * BWD_CTAS_PER_SM;
#define L(CH) launch_next(raster_bwd_kernel<CH>, ctas, BWD_WARPS * 32, BWD_SMEM, s,  \
      (const uint2*)c->tile_ranges, c->vals_sorted, (const float4*)c->proj0, (const float4*)c->proj1, (const float4*)c->proj2, (const float4*)c->out_rgba, \
      (const float4*)c->out_feat, c->last_idx, (const float4*)c->v_out, c->W, c->H, c->tiles_x, c->n_tiles, bg, c->v_splat, c->vis_flag, m->vis_weight, chunks, \
      items, work, bwd_ckpt_ptr(c), seg_shift, 1.f / grad_scale)
  if (brief) L(SHORT); else if (chunks > 1) L(CHUNKED); else L(WHOLE);
#undef L
  return check_launch();
}
