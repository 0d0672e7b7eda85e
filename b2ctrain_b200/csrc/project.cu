// Projection stage: EWA projection with the 3D-filter floor, SH colour, exact tile count and the depth sort key, one
// pass over the splats. Reference semantics: project_kernel (src/gpu/project.cu:9-84) and depth_keys_kernel
// (src/gpu/binning.cu:10-15), fused.
//
// HBM-bound stream: per splat 48 B of float4 parameters + 12 K B of planar SH in, 48 B of records + 12 B of
// count / key / index out. One thread per splat; the three float4 loads are 128-bit and coalesced, the planar SH
// lanes are coalesced across the warp.
#include "common.cuh"
#include "sh.cuh"

namespace b2k {

int g_last_cuda_error = 0;
std::atomic<uint64_t> g_launches_repeated{0};
int check_launch() {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return B2K_ERR_CUDA; }
  return B2K_OK;
}
int sm_count() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return NUM_SMS_HINT;
  if (!cached[dev]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = NUM_SMS_HINT;
    cached[dev] = n;
  }
  return cached[dev];
}

namespace {

constexpr int PROJ_BLOCK = 256;

// Tile boxes of at most MASK_TILES tiles are remembered as a bit mask of the tiles hit. Their tests are shared out over the splats' warp, and so
// are those of boxes of up to WARP_TILES where there are many splats, or where all such boxes of the warp make WARP_FEW tiles; the others are counted by
// a kernel of their own, a warp to each. Few splats are few warps, which wait for the one with the most tests; project_kernel and count_big_kernel
// together, us, WARP_FEW of 256 / 512 / 1,024: 256x192 over 2k splats over most of it 10.7 / 13.7 / 16.0, 333x217 over 45k wide ones 36.3 / 37.9 / 39.8; and
// every box of up to 128 tiles in the warp 200x150 over 2k 26.3 against 15.8. Many splats fill the GPU, and the large boxes' kernel is then the
// more costly one: 1001x751 over 200k 46 us up to 1,024, 45 up to 512, 47 up to 256, 54 up to 64; where a tenth are wide (801x603 over 90k) 114, 99, 95, 93.
constexpr int MASK_TILES = 64, WARP_TILES = 512, WARP_FEW = 256, WARP_MANY_SPLATS = 49152, DIRECT_TILES = 16;

// The tile tests of a warp's 32 splats, shared out in units of up to eight tiles of one row: boxes hold one to a thousand tiles, and with
// a splat per lane most lanes wait for the largest.
struct TileShare { float4 rec[64]; uint32_t corner[32], width[32], end[32], mask[64], count[32]; };
// box: the lane's tile box (empty: none); returns the tiles hit, and for boxes of at most MASK_TILES tiles their mask. All lanes call this.
__device__ __forceinline__ uint32_t shared_hits(TileShare& ts, const TileRec& rec, const TileBox& b, int area, uint32_t& mask_lo, uint32_t& mask_hi) {
  constexpr unsigned ALL = 0xffffffffu;
  const int lane = threadIdx.x & 31, bw = b.max_x - b.min_x;
  mask_lo = mask_hi = 0u;
  if (__reduce_max_sync(ALL, area) <= DIRECT_TILES) {   // each lane its own: 1920x1080 over 3M splats of one or two tiles 160 -> 144 us
    for (int k = 0, tx = b.min_x, ty = b.min_y; k < area; k++) {
      if (tile_hit(tx, ty, rec)) mask_lo |= 1u << k;
      if (++tx == b.max_x) { tx = b.min_x; ty++; }
    }
    return (uint32_t)__popc(mask_lo);
  }
  const int units = area > 0 ? (b.max_y - b.min_y) * ((bw + 7) >> 3) : 0;
  int end = units;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(ALL, end, o); if (lane >= o) end += u; }
  const int total = __shfl_sync(ALL, end, 31);
  ts.rec[lane * 2] = make_float4(rec.mx, rec.my, rec.c00, rec.c01);
  ts.rec[lane * 2 + 1] = make_float4(rec.c11, rec.power, rec.ia, rec.ib);
  ts.corner[lane] = (uint32_t)b.min_x | (uint32_t)b.min_y << 16; ts.width[lane] = (uint32_t)bw | (area <= MASK_TILES ? 0x80000000u : 0u); ts.end[lane] = (uint32_t)end;
  ts.mask[lane * 2] = ts.mask[lane * 2 + 1] = 0u; ts.count[lane] = 0u;
  __syncwarp();
  for (int u = lane; u < total; u += 32) {
    int owner = 0;   // the first lane whose units end behind u
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) owner += (int)ts.end[owner + step - 1] <= u ? step : 0;
    const uint32_t corner = ts.corner[owner], wide = ts.width[owner], w = wide & 0xFFFFu, per_row = (w + 7u) >> 3;
    const uint32_t at = (uint32_t)u - (owner ? ts.end[owner - 1] : 0u), row_in_box = per_row == 1u ? at : at / per_row, x0 = (at - row_in_box * per_row) * 8u;
    const float4 a = ts.rec[owner * 2], c = ts.rec[owner * 2 + 1];
    const TileRec r{a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
    const TileRow row = tile_row((int)((corner >> 16) + row_in_box), r);
    const uint32_t tiles = min(w - x0, 8u);
    uint32_t out = 0u;
    for (uint32_t k = 0; k < tiles; k++) out |= tile_hit((int)((corner & 0xFFFFu) + x0 + k), row, r) ? 1u << k : 0u;
    if (out == 0u) continue;
    atomicAdd(&ts.count[owner], (uint32_t)__popc(out));
    if (wide >> 31) {
      const uint32_t bit = row_in_box * w + x0;
      const unsigned long long word = (unsigned long long)out << (bit & 31u);
      atomicOr(&ts.mask[owner * 2 + (bit >> 5)], (uint32_t)word);
      if (word >> 32) atomicOr(&ts.mask[owner * 2 + 1], (uint32_t)(word >> 32));
    }
  }
  __syncwarp();
  mask_lo = ts.mask[lane * 2]; mask_hi = ts.mask[lane * 2 + 1];
  return ts.count[lane];
}

// What a splat's record says about its tiles: tiles hit, the words of hit_info, whether its box is left to count_big_kernel. All lanes of
// the warp call this; `drawn`: the splat has a record and its box is on the image.
struct TileHits { uint32_t hits, w0, w1, box, height; bool big; };
__device__ __forceinline__ TileHits decide_tiles(TileShare& ts, const TileRec& rec, const TileBox& b, bool drawn, int n) {
  const int bw = drawn ? b.max_x - b.min_x : 0, bh = drawn ? b.max_y - b.min_y : 0, area = bw > 0 && bh > 0 ? bw * bh : 0;
  const int limit = n > WARP_MANY_SPLATS || __reduce_add_sync(0xffffffffu, area > MASK_TILES && area <= WARP_TILES ? area : 0) <= WARP_FEW ? WARP_TILES : MASK_TILES;
  TileHits t{0u, 0u, 0u, 0u, drawn ? (uint32_t)bh : 0u, area > limit};
  t.hits = shared_hits(ts, rec, b, t.big ? 0 : area, t.w0, t.w1);
  if (area > MASK_TILES) {   // no mask: the box itself
    t.box = 0xFFFFFFFFu;
    t.w0 = (uint32_t)b.min_x | ((uint32_t)b.min_y << 16); t.w1 = (uint32_t)bw | ((uint32_t)bh << 16);
  } else if (area > 0) t.box = (uint32_t)b.min_x | ((uint32_t)b.min_y << 12) | ((uint32_t)bw << 24);
  return t;
}

// One bit a splat for count_big_kernel. All lanes call this.
__device__ __forceinline__ void flag_big(uint32_t* __restrict__ big, int i, int n, bool is) {
  const uint32_t word = __ballot_sync(0xffffffffu, is);
  if ((i & 31) == 0 && i < n) big[i >> 5] = word;
}

// Feature lanes of a splat (src/gpu/project.cu:62-77). Mode 1: pseudo-normal = the local axis of the shortest scale,
// turned to face the camera, in camera space. Mode 2: the caller's per-splat buffer, clamped to +-100, non-finite -> 0.
__device__ __forceinline__ float3 splat_feature(int mode, int i, const float4 po, const float4 ls, const float* Rq, const CamDev& cam,
                                                const float* __restrict__ feat_in) {
  if (mode == 1) {
    const int axis = (ls.x <= ls.y && ls.x <= ls.z) ? 0 : (ls.y <= ls.z ? 1 : 2);
    const float3 a = make_float3(Rq[axis], Rq[3 + axis], Rq[6 + axis]);
    const float inv = 1.f / fmaxf(sqrtf(a.x * a.x + a.y * a.y + a.z * a.z), 1e-12f);
    const float3 u = make_float3(a.x * inv, a.y * inv, a.z * inv);
    const float face = ((cam.pos[0] - po.x) * u.x + (cam.pos[1] - po.y) * u.y + (cam.pos[2] - po.z) * u.z) >= 0.f ? 1.f : -1.f;
    const float3 w = make_float3(u.x * face, u.y * face, u.z * face);
    const float* R = cam.R;
    return make_float3(R[0] * w.x + R[1] * w.y + R[2] * w.z, R[3] * w.x + R[4] * w.y + R[5] * w.z, R[6] * w.x + R[7] * w.y + R[8] * w.z);
  }
  float3 f = make_float3(feat_in[(size_t)i * 3], feat_in[(size_t)i * 3 + 1], feat_in[(size_t)i * 3 + 2]);
  f.x = isfinite(f.x) ? fminf(fmaxf(f.x, -100.f), 100.f) : 0.f;
  f.y = isfinite(f.y) ? fminf(fmaxf(f.y, -100.f), 100.f) : 0.f;
  f.z = isfinite(f.z) ? fminf(fmaxf(f.z, -100.f), 100.f) : 0.f;
  return f;
}

// The SH lanes of the warp's 32 splats on their way to the L2 while their geometry is worked out: a lane asks for 128 bytes of
// each of its lanes' arrays, if any of the splats is in front of the camera inside the guard band (the others may still be seen,
// and are then simply not ahead). Only where the rows are 16-byte aligned. The kernel is bound by the latency of its two rounds of loads
// (1M splats 73 -> 65 us, 6M of degree 4 627 -> 568, which is 3.8 TB/s); project_kernel, which tests tiles in between, gains nothing.
template <int DEG>
__device__ __forceinline__ void prefetch_colour(int i, int n, size_t cap, const float4& po, const CamDev& cam, int active, const float* sh_dc, const float* sh_hi) {
  const int lane = threadIdx.x & 31, first = i - lane, lanes = 3 * (active + 1) * (active + 1);
  if (first + 32 > n || (cap & 3) || (((uintptr_t)sh_dc | (uintptr_t)sh_hi) & 15)) return;
  const float3 c = to_camera(cam, po);
  const bool ahead = c.z >= 0.01f && c.x >= cam.lim_neg_x * c.z && c.x <= cam.lim_pos_x * c.z && c.y >= cam.lim_neg_y * c.z && c.y <= cam.lim_pos_y * c.z;
  if (!__any_sync(0xffffffffu, ahead)) return;
  for (int l = lane; l < lanes; l += 32) {
    const float* p = (l < 3 ? sh_dc + (size_t)l * cap : sh_hi + (size_t)(l - 3) * cap) + first;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], 128;" ::"l"(p) : "memory");
  }
}

template <int DEG>
__global__ void __launch_bounds__(PROJ_BLOCK) project_kernel(
    int n, size_t cap, const float4* __restrict__ pos_op, const float4* __restrict__ quat, const float4* __restrict__ lscale,
    const float* __restrict__ sh_dc, const float* __restrict__ sh_hi, CamDev cam, int active, int tiles_x, int tiles_y,
    float4* __restrict__ proj0, float4* __restrict__ proj1, float4* __restrict__ proj2, uint32_t* __restrict__ tile_count,
    uint4* __restrict__ hit_info, uint32_t* __restrict__ depth_keys, uint32_t* __restrict__ order_in, float* __restrict__ max_screen,
    int feat_mode, const float* __restrict__ feat_in, float2* __restrict__ proj3, uint32_t* __restrict__ big) {
  after_previous();
  __shared__ TileShare s_share[PROJ_BLOCK / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n;
  float4 po = make_float4(0.f, 0.f, 0.f, 0.f), q = po, ls = po;
  if (valid) { po = pos_op[i]; q = quat[i]; ls = lscale[i]; }
  Proj pr;
  TileRec rec{};
  TileBox bb{0, 0, 0, 0};
  bool drawn = false;
  if (valid) {
    if (project_one(po, q, ls, cam, pr)) {
      rec = make_tile_rec(pr.mx, pr.my, pr.c00, pr.c01, pr.c11, pr.power);
      drawn = tile_box(rec, cam.W, cam.H, tiles_x, tiles_y, bb);
      proj0[i] = make_float4(pr.mx, pr.my, pr.c00, pr.c01);
      proj1[i] = make_float4(pr.c11, pr.opac, pr.mean_c.z, pr.power);
    } else {
      proj1[i] = make_float4(0.f, 0.f, 0.f, -1.f);   // no record
    }
  }
  const TileHits t = decide_tiles(s_share[threadIdx.x >> 5], rec, bb, drawn, n);
  flag_big(big, i, n, t.big);
  if (!valid) return;
  if (drawn && max_screen) {
    const float detc = pr.c00 * pr.c11 - pr.c01 * pr.c01;
    const float ex = sqrtf(2.f * pr.power * pr.c11 / detc), ey = sqrtf(2.f * pr.power * pr.c00 / detc);
    const float ms = fmaxf(ex / (float)cam.W, ey / (float)cam.H);
    if (ms > max_screen[i]) atomic_max_nonneg(max_screen + i, ms);
  }
  if (t.hits || t.big) {
    float4 col = splat_colour<DEG>(i, cap, make_float3(po.x, po.y, po.z), cam.pos, active, sh_dc, sh_hi);
    if (feat_mode != 0) {
      const float3 f = splat_feature(feat_mode, i, po, ls, pr.Rq, cam, feat_in);
      col.w = f.x;
      proj3[i] = make_float2(f.y, f.z);
    }
    proj2[i] = col;
  }
  hit_info[i] = make_uint4(t.w0, t.w1, t.box, t.height);
  order_in[i] = (uint32_t)i;
  if (!t.big) {   // the others get their count and key from count_big_kernel
    tile_count[i] = t.hits;
    depth_keys[i] = t.hits ? __float_as_uint(pr.mean_c.z) : 0xFFFFFFFFu;
  }
}

// The projection of the chunked renderer, which decides tiles later and only for the splats whose tile box still holds
// a live tile: records, colours, the tile box, the depth key, the screen-size statistic.
// hit_info = (0, 0, box, height) with box = min_x | min_y << 12 | width << 24 for boxes of at most 64 tiles, and
// (min_x | min_y << 16, width | height << 16, 0xFFFFFFFF, height) above that; height = 0 marks an empty box.
// tile_count holds the box area, an upper bound of the tiles hit (zero exactly when the box is empty).
template <int DEG>
__global__ void __launch_bounds__(PROJ_BLOCK, 4) project_lite_kernel(
    int n, size_t cap, const float4* __restrict__ pos_op, const float4* __restrict__ quat, const float4* __restrict__ lscale,
    const float* __restrict__ sh_dc, const float* __restrict__ sh_hi, int active, CamDev cam, int tiles_x, int tiles_y,
    float4* __restrict__ proj0, float4* __restrict__ proj1, float4* __restrict__ proj2, uint32_t* __restrict__ tile_count, uint4* __restrict__ hit_info,
    uint32_t* __restrict__ depth_keys, float* __restrict__ max_screen, int feat_mode, const float* __restrict__ feat_in,
    float2* __restrict__ proj3) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 po = pos_op[i], q = quat[i], ls = lscale[i];
  prefetch_colour<DEG>(i, n, cap, po, cam, active, sh_dc, sh_hi);
  Proj pr;
  uint32_t area = 0, box = 0, bh_out = 0, w0 = 0, w1 = 0;
  if (project_one(po, q, ls, cam, pr)) {
    const TileRec rec = make_tile_rec(pr.mx, pr.my, pr.c00, pr.c01, pr.c11, pr.power);
    TileBox bb;
    if (tile_box(rec, cam.W, cam.H, tiles_x, tiles_y, bb)) {
      const int bw = bb.max_x - bb.min_x, bh = bb.max_y - bb.min_y;
      if (bw > 0 && bh > 0) {
        area = (uint32_t)(bw * bh);
        bh_out = (uint32_t)bh;
        if (area > (uint32_t)MASK_TILES) {
          box = 0xFFFFFFFFu;
          w0 = (uint32_t)bb.min_x | ((uint32_t)bb.min_y << 16); w1 = (uint32_t)bw | ((uint32_t)bh << 16);
        } else {
          box = (uint32_t)bb.min_x | ((uint32_t)bb.min_y << 12) | ((uint32_t)bw << 24);
        }
      }
      const float detc = pr.c00 * pr.c11 - pr.c01 * pr.c01;
      const float ex = sqrtf(2.f * pr.power * pr.c11 / detc), ey = sqrtf(2.f * pr.power * pr.c00 / detc);
      if (max_screen) { const float ms = fmaxf(ex / (float)cam.W, ey / (float)cam.H); if (ms > max_screen[i]) atomic_max_nonneg(max_screen + i, ms); }
    }
    proj0[i] = make_float4(pr.mx, pr.my, pr.c00, pr.c01);
    proj1[i] = make_float4(pr.c11, pr.opac, pr.mean_c.z, pr.power);
    // The colour is evaluated here for every splat with a tile box: this kernel reads the planar SH lanes coalesced,
    // while a colour evaluated later, for the emitting splats only and in depth order, costs one 32-byte sector per
    // lane and splat (it measured slower although it shades a tenth of the splats).
    if (area) {
      float4 col = splat_colour<DEG>(i, cap, make_float3(po.x, po.y, po.z), cam.pos, active, sh_dc, sh_hi);
      if (feat_mode != 0) {
        const float3 f = splat_feature(feat_mode, i, po, ls, pr.Rq, cam, feat_in);
        col.w = f.x;
        proj3[i] = make_float2(f.y, f.z);
      }
      proj2[i] = col;
    }
  } else {
    proj1[i] = make_float4(0.f, 0.f, 0.f, -1.f);   // no record
  }
  hit_info[i] = make_uint4(w0, w1, box, bh_out);
  tile_count[i] = area;
  depth_keys[i] = area ? __float_as_uint(pr.mean_c.z) : 0xFFFFFFFFu;
}

// Boxes that were not tested in their own warp: a warp to each, whose lanes take units of up to eight tiles of a row (562x569 over 4,303 wide splats: a tile
// a lane, which divides for each, 33.7 us, units 19.9). The projection leaves a bit a splat; a warp's lanes look at 1 << shift neighbours each,
// far from each other, so that large splats that follow each other go to different warps. (A list of them needs a counter that is
// cleared, which took a launch of its own, 64x64 over 2k splats 80.2 -> 78.9 us a step; finding them in hit_info reads 16 bytes a splat, 3M
// splats 16 us.)
constexpr int BIG_WARPS = 8;             // of a block
inline int big_shift(int n) { return n <= 32768 ? 0 : n <= 262144 ? 1 : 2; }
// A warp for every unit of few, for two of more (blocks without a large box cost as much as the launch: 8k splats 1.9 us in 500 blocks, 2.6 in 1,000;
// 256x192 over 1k splats over all of it 10.7 us with a warp to each, 13.8 with one to two).
inline int big_blocks(int n) {
  const int units = div_up(n, 1 << big_shift(n));
  return min(max(min(div_up(units, BIG_WARPS), 512), div_up(units, 2 * BIG_WARPS)), sm_count() * 8);
}
__global__ void __launch_bounds__(BIG_WARPS * 32) count_big_kernel(int n, int shift, const uint32_t* __restrict__ big, const float4* __restrict__ proj0, const float4* __restrict__ proj1, int W, int H,
                                                                   int tiles_x, int tiles_y, uint32_t* __restrict__ tile_count, uint32_t* __restrict__ depth_keys) {
  after_previous();
  const int lane = threadIdx.x & 31, warps = gridDim.x * BIG_WARPS;
  const long long units = ((long long)n + (1 << shift) - 1) >> shift;
  for (long long u0 = blockIdx.x * BIG_WARPS + (threadIdx.x >> 5); u0 < units; u0 += 32ll * warps) {
    const long long mine = (u0 + (long long)lane * warps) << shift;
    const uint32_t flags = mine < n ? (big[mine >> 5] >> (mine & 31)) & ((1u << (1 << shift)) - 1u) : 0u;
    for (uint32_t todo = __ballot_sync(0xffffffffu, flags != 0u); todo; todo &= todo - 1u) {
      const int owner = __ffs(todo) - 1;
      for (uint32_t left = __shfl_sync(0xffffffffu, flags, owner); left; left &= left - 1u) {
        const long long i = ((u0 + (long long)owner * warps) << shift) + __ffs(left) - 1;
        const float4 a = proj0[i], b = proj1[i];
        const TileRec rec = make_tile_rec(a.x, a.y, a.z, a.w, b.x, b.w);
        TileBox bb;
        uint32_t hits = 0;
        if (tile_box(rec, W, H, tiles_x, tiles_y, bb)) {
          // units of up to eight tiles of one row, as in shared_hits
          const int bw = bb.max_x - bb.min_x, per_row = (bw + 7) >> 3, units = (bb.max_y - bb.min_y) * per_row;
          for (int u = lane; u < units; u += 32) {
            const int y = u / per_row, x0 = (u - y * per_row) * 8;
            const TileRow row = tile_row(bb.min_y + y, rec);
#pragma unroll
            for (int k = 0; k < 8; k++) hits += x0 + k < bw && tile_hit(bb.min_x + x0 + k, row, rec) ? 1u : 0u;
          }
        }
        hits = __reduce_add_sync(0xffffffffu, hits);
        if (lane == 0) { tile_count[i] = hits; depth_keys[i] = hits ? __float_as_uint(b.z) : 0xFFFFFFFFu; }
      }
    }
  }
}

// The decision half of the projection on its own: tile counts, hit masks and depth keys recomputed from the records
// already in proj0 / proj1 (power < -0.5 marks "no record").
__global__ void __launch_bounds__(PROJ_BLOCK) count_tiles_kernel(int n, const float4* __restrict__ proj0, const float4* __restrict__ proj1, int W, int H,
                                                                 int tiles_x, int tiles_y, uint32_t* __restrict__ tile_count, uint4* __restrict__ hit_info,
                                                                 uint32_t* __restrict__ depth_keys, uint32_t* __restrict__ order_in, uint32_t* __restrict__ big) {
  after_previous();
  __shared__ TileShare s_share[PROJ_BLOCK / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < n;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = make_float4(0.f, 0.f, 0.f, -1.f);
  if (valid) { a = proj0[i]; b = proj1[i]; }
  TileRec rec{};
  TileBox bb{0, 0, 0, 0};
  bool drawn = false;
  if (b.w > -0.5f) {
    rec = make_tile_rec(a.x, a.y, a.z, a.w, b.x, b.w);
    drawn = tile_box(rec, W, H, tiles_x, tiles_y, bb);
  }
  const TileHits t = decide_tiles(s_share[threadIdx.x >> 5], rec, bb, drawn, n);
  flag_big(big, i, n, t.big);
  if (!valid) return;
  hit_info[i] = make_uint4(t.w0, t.w1, t.box, t.height);
  order_in[i] = (uint32_t)i;
  if (!t.big) { tile_count[i] = t.hits; depth_keys[i] = t.hits ? __float_as_uint(b.z) : 0xFFFFFFFFu; }
}

// A few words to zero. (A memset node would break the chain of overlapped launches on both sides.)
__global__ void clear_kernel(uint32_t* a, int words_a, uint32_t* b, int words_b) {
  after_previous();
  for (int i = threadIdx.x; i < words_a; i += 32) a[i] = 0u;
  for (int i = threadIdx.x; i < words_b; i += 32) b[i] = 0u;
}

template <int DEG>
int launch(const B2kModel* m, const CamDev& cam, const B2kRenderOpts* o, const B2kCtx* c, cudaStream_t s) {
  const float4* pos = (const float4*)(o->pos_override ? o->pos_override : m->pos_op);
  const float4* quat = (const float4*)(o->quat_override ? o->quat_override : m->quat);
  const float4* lscale = (const float4*)(o->lscale_override ? o->lscale_override : m->lscale);
  const int active = o->sh_degree < m->degree ? o->sh_degree : m->degree;
  launch_next(project_kernel<DEG>, div_up(m->n, PROJ_BLOCK), PROJ_BLOCK, 0, s, 
      m->n, (size_t)m->cap, pos, quat, lscale, m->sh_dc, m->sh_hi, cam, active < 0 ? 0 : active, c->tiles_x, c->tiles_y,
      (float4*)c->proj0, (float4*)c->proj1, (float4*)c->proj2, c->tile_count, (uint4*)c->hit_info, c->depth_keys_sorted, c->order, m->max_screen,
      o->feat_mode, o->feat_buffer, (float2*)c->proj3, splat_words_ptr(c));
  launch_next(count_big_kernel, big_blocks(m->n), BIG_WARPS * 32, 0, s, m->n, big_shift(m->n), splat_words_ptr(c), (const float4*)c->proj0, (const float4*)c->proj1, cam.W, cam.H, c->tiles_x,
                                                  c->tiles_y, c->tile_count, c->depth_keys_sorted);
  return check_launch();
}

}  // namespace

void launch_clear(void* a, int words_a, void* b, int words_b, cudaStream_t s) { launch_next(clear_kernel, 1, 32, 0, s, (uint32_t*)a, words_a, (uint32_t*)b, words_b); }

int launch_project_lite(const B2kModel* m, const B2kCamera* cam, const B2kRenderOpts* o, const B2kCtx* c, cudaStream_t s) {
  const float4* pos = (const float4*)(o->pos_override ? o->pos_override : m->pos_op);
  const float4* quat = (const float4*)(o->quat_override ? o->quat_override : m->quat);
  const float4* lscale = (const float4*)(o->lscale_override ? o->lscale_override : m->lscale);
  const int active = o->sh_degree < m->degree ? (o->sh_degree < 0 ? 0 : o->sh_degree) : m->degree;
  const CamDev cd = to_camdev(*cam);
#define L(D) launch_next(project_lite_kernel<D>, div_up(m->n, PROJ_BLOCK), PROJ_BLOCK, 0, s, m->n, (size_t)m->cap, pos, quat, lscale, m->sh_dc, m->sh_hi, active, cd, \
      c->tiles_x, c->tiles_y, (float4*)c->proj0, (float4*)c->proj1, (float4*)c->proj2, c->tile_count, (uint4*)c->hit_info, c->depth_keys_sorted, m->max_screen, \
      o->feat_mode, o->feat_buffer, (float2*)c->proj3)
  switch (m->degree) { case 0: L(0); break; case 1: L(1); break; case 2: L(2); break; case 3: L(3); break; default: L(4); break; }
#undef L
  return check_launch();
}
}  // namespace b2k

using namespace b2k;

extern "C" int b2k_project(const B2kModel* m, const B2kCamera* cam, const B2kRenderOpts* opts, const B2kCtx* ctx, b2k_stream_t s) {
  B2K_REQUIRE(m && cam && opts && ctx);
  if (m->n == 0) return B2K_OK;
  B2K_REQUIRE(m->n > 0 && m->cap >= m->n && m->pos_op && m->quat && m->lscale && m->sh_dc);
  B2K_REQUIRE(m->degree >= 0 && m->degree <= 4 && (m->degree == 0 || m->sh_hi));
  B2K_REQUIRE(ctx->proj0 && ctx->proj1 && ctx->proj2 && ctx->tile_count && ctx->hit_info && ctx->depth_keys_sorted && ctx->order && ctx->sort_tmp);
  if (ctx->sort_tmp_bytes < b2k_sort_tmp_bytes(ctx->n_cap, ctx->isect_cap)) return B2K_ERR_CAPACITY;
  B2K_REQUIRE(cam->W == ctx->W && cam->H == ctx->H && ctx->tiles_x == div_up(ctx->W, RT_W) && ctx->tiles_y == div_up(ctx->H, RT_W));
  B2K_REQUIRE(opts->feat_mode >= 0 && opts->feat_mode <= 2 && (opts->feat_mode == 0 || ctx->proj3) && (opts->feat_mode != 2 || opts->feat_buffer));
  if (ctx->n_cap < m->n) return B2K_ERR_CAPACITY;
  const CamDev cd = to_camdev(*cam);
  cudaStream_t st = (cudaStream_t)s;
  switch (m->degree) {
    case 0: return launch<0>(m, cd, opts, ctx, st);
    case 1: return launch<1>(m, cd, opts, ctx, st);
    case 2: return launch<2>(m, cd, opts, ctx, st);
    case 3: return launch<3>(m, cd, opts, ctx, st);
    default: return launch<4>(m, cd, opts, ctx, st);
  }
}

extern "C" int b2k_count_tiles(const B2kCtx* c, int32_t n, b2k_stream_t stream) {
  B2K_REQUIRE(c && n >= 0);
  if (n == 0) return B2K_OK;
  B2K_REQUIRE(c->proj0 && c->proj1 && c->tile_count && c->hit_info && c->depth_keys_sorted && c->order && c->sort_tmp);
  B2K_REQUIRE(c->W > 0 && c->H > 0 && c->tiles_x == div_up(c->W, RT_W) && c->tiles_y == div_up(c->H, RT_W));
  if (c->n_cap < n || c->sort_tmp_bytes < b2k_sort_tmp_bytes(c->n_cap, c->isect_cap)) return B2K_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  launch_next(count_tiles_kernel, div_up(n, 256), 256, 0, s, n, (const float4*)c->proj0, (const float4*)c->proj1, c->W, c->H, c->tiles_x, c->tiles_y, c->tile_count,
                                                   (uint4*)c->hit_info, c->depth_keys_sorted, c->order, splat_words_ptr(c));
  launch_next(count_big_kernel, big_blocks(n), BIG_WARPS * 32, 0, s, n, big_shift(n), splat_words_ptr(c), (const float4*)c->proj0, (const float4*)c->proj1, c->W, c->H, c->tiles_x, c->tiles_y,
                                                  c->tile_count, c->depth_keys_sorted);
  return check_launch();
}

static const char* kErrors[] = {"ok", "bad argument", "buffer capacity exceeded", "unsupported lane", "CUDA error",
                                "intersection buffers overflowed"};
extern "C" const char* b2k_error_string(int status) { return status >= 0 && status <= 5 ? kErrors[status] : "unknown status"; }
extern "C" int b2k_last_cuda_error(void) { return g_last_cuda_error; }
extern "C" uint64_t b2k_launches_repeated(void) { return g_launches_repeated.load(std::memory_order_relaxed); }
extern "C" const char* b2k_version(void) { return "b2k 0.1 (sm_100a)"; }
