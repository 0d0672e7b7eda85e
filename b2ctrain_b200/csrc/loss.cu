// Fused photometric loss: L1 + 11-tap Gaussian SSIM (sigma 1.5, zero padding) + alpha-match lane, value and
// per-pixel gradient in one kernel. Reference semantics: photometric_kernel (src/gpu/loss.cu:18-195),
// accumulate_kernel (loss.cu:317), eval_kernel (loss.cu:241-293).
//
// The work is a stencil: a separable blur of five moments, SSIM and its partial derivatives, the same blur applied
// backwards. It is bound by FP32 issue and shared-memory reads, not by HBM (36 bytes per pixel), so what counts is how
// many blur taps are spent per output. The loss kernel streams down column strips and pays for a halo in one direction
// only; every blur is register-tiled (a thread makes four consecutive outputs from a fourteen-wide sliding window).
#include "common.cuh"
#include <algorithm>

namespace b2k {
namespace {

constexpr int HALO = 5;
constexpr float C1 = 0.01f * 0.01f, C2 = 0.03f * 0.03f;

struct Gauss2 { float2 w[11]; };   // every weight twice, as an operand of packed arithmetic

Gauss2 make_gauss() {
  float w[11], sum = 0.f;
  for (int i = 0; i < 11; i++) { const float x = (float)i - 5.f; w[i] = expf(-x * x / (2.f * 1.5f * 1.5f)); sum += w[i]; }
  Gauss2 g;
  for (int i = 0; i < 11; i++) g.w[i] = make_float2(w[i] / sum, w[i] / sum);
  return g;
}

__device__ __forceinline__ float unpack(uint32_t p, int c) { return (float)((p >> (8 * c)) & 0xffu) * (1.f / 255.f); }

struct LossArgs {
  float l1_w, ssim_w, bg[3]; int composite, mask, alpha_lane; float match_alpha_weight, scale, grad_scale;
};

// ---- The loss kernel --------------------------------------------------------------------------------------------------
// One CTA owns a strip of STRIP_W output columns and a segment of rows, all three channels (or one, in a small image), and walks the segment four rows at
// a time. Both blurs are separable, so only the horizontal direction pays for a halo: the row-blurred moments and the
// derivative maps of the last RING rows live in shared-memory rings, and the four stages of the chain run side by side as a
// pipeline, each on its own warps (six to a channel) and on its own rows, with one barrier per four rows:
//   A (1 warp)   rows a..a+3      : prediction and effective target -> five moments blurred along the row
//   B (2 warps)  rows a-9..a-6    : blurred down the column -> SSIM -> derivative maps (three: the two that the chain
//                                   rule multiplies by p and by the target, and the sum of the three it does not)
//   C (1 warp)   rows a-18..a-15  : derivative maps blurred down the column
//   D (2 warps)  rows a-22..a-19  : blurred along the row, chain rule, L1 term
// While they work, all threads fetch the next four input rows, a whole pixel each, and write the gradient rows of the step
// before, a whole pixel each: with a CTA per channel every 32-byte sector crossed the L2 three times in both directions. A
// pixel's values also wait in a ring for stage D, so that no stage waits for global memory.
//
// Bound by instruction issue: 176 multiply-adds per pixel and channel in the four blurs. They run two to an instruction
// (fp32x2) with operands that lie in pairs as they are stored: prediction and target side by side, and so their means, their
// squares, and the two maps with a per-pixel factor; the product moment and the third map are paired over two rows (A) or two
// columns (C). A thread makes four or eight outputs from one window, so that a value read from shared memory feeds eleven to
// forty-four multiply-adds. Measured against the same pipeline with scalar multiply-adds and a CTA per channel: 187 -> 124 us on
// a 1920x1080 view, 101 -> 96 us on a masked 1024x1024 one, 26 -> 21 us on 333x217. Other arrangements on 1920x1080: packed,
// a CTA per channel 133 to 147; channels of one CTA with a barrier each 130; the pairs in plain order (two-way bank conflicts in
// stages A and D) 139; two columns per thread in stage B 142.
constexpr int STRIP_W = 54;                   // output columns of a strip
constexpr int STRIP_ST = STRIP_W + 2 * HALO;  // 64 statistics columns
constexpr int STRIP_IN = 80;                  // input columns staged: STRIP_W + 4 * HALO = 74, padded to whole groups of eight 16-byte chunks
constexpr int STRIP_ROWS = 4;                 // rows per pipeline step
constexpr int RING = 18;                      // rows of a ring: the 14 a column window of four outputs reads + the 4 being written
constexpr int BV_S = STRIP_ST + 16;           // row stride of stage C's output: the last row window overruns into zero padding
constexpr int PX_RING = 32;                   // rows of the ring that keeps pixels for stage D: a + 7 down to a - 22 are in use
constexpr int PX_S = 64;                      // its columns: STRIP_W, padded likewise
constexpr int CH_WARPS = 6, CH_THREADS = CH_WARPS * 32;
static_assert(STRIP_ST == 64 && STRIP_IN >= STRIP_W + 4 * HALO && STRIP_IN % 4 == 0, "strip geometry");

// One ring row of row-blurred moments, and one of derivative maps: everything of a row behind one address.
struct MomentRow { float2 mean[STRIP_ST], square[STRIP_ST]; float cross[STRIP_ST]; };   // (prediction, target) twice; their product
struct MapRow { float2 e12[STRIP_ST]; float e0[STRIP_ST]; };                            // the maps multiplied by p and by the target; the sum of the others
// Rows of pairs are kept as 16-byte chunks of two columns in a slightly permuted order: threads that read or write every other
// chunk (four columns each) then meet all banks, and runs of chunks still do.
__device__ __forceinline__ int chunk_at(int chunk) { return chunk ^ ((chunk >> 3) & 1); }
__device__ __forceinline__ int pair_at(int col) { return chunk_at(col >> 1) * 2 + (col & 1); }   // place of one column's pair

struct ChannelShare {
  float2 in[2][STRIP_ROWS][STRIP_IN];     // [buffer][row][column]: prediction, effective target
  float2 px[PX_RING][PX_S];               // the strip's own columns of the same, until stage D has used them
  MomentRow moments[RING];
  MapRow maps[RING];
  float2 b12[2][STRIP_ROWS][BV_S];        // [buffer] the maps blurred down the column
  float b0[2][STRIP_ROWS][BV_S];
};
template <int CHANNELS>
struct StripShare {
  ChannelShare ch[CHANNELS];
  float out[2][STRIP_ROWS][PX_S][4];      // [buffer] gradient of the step's pixels
  float red[20];
};
static_assert(sizeof(StripShare<3>) % 16 == 0 && sizeof(StripShare<1>) % 16 == 0 && sizeof(StripShare<3>) <= 227 * 1024, "one CTA per SM");

__device__ __forceinline__ int ring_slot(int row) { return (row + RING * 256) % RING; }
template <class ROW>
__device__ __forceinline__ ROW* ring_next(ROW* row, ROW* ring) { return row == ring + (RING - 1) ? ring : row + 1; }
__device__ __forceinline__ float fast_rcp(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// Byte c of a packed pixel as 0 .. 1: the byte under the exponent of 2^23, less 2^23 (an integer conversion runs at a quarter
// of the rate of these).
__device__ __forceinline__ float byte_unit(uint32_t p, int c) { return (__uint_as_float(__byte_perm(p, 0x4B000000u, 0x7440u | (uint32_t)c)) - 8388608.f) * (1.f / 255.f); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// MASKED: per-pixel weights or the target's alpha scale the loss, or there is an alpha lane.
// CHANNELS: 3, or 1 with a CTA per channel, which a small image has SMs to spare for.
template <bool MASKED, int CHANNELS>
__global__ void __launch_bounds__(CHANNELS * CH_THREADS, 1) photometric_strip_kernel(const float4* __restrict__ pred, const uint32_t* __restrict__ gt,
                                                                          const uint8_t* __restrict__ weights, int W, int H, int seg_rows, LossArgs lp,
                                                                          Gauss2 gauss, float4* __restrict__ v_out, float* __restrict__ loss_accum) {
  extern __shared__ __align__(16) unsigned char s_bytes[];
  constexpr int THREADS = CHANNELS * CH_THREADS;
  StripShare<CHANNELS>& all = *reinterpret_cast<StripShare<CHANNELS>*>(s_bytes);
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) % CH_WARPS;   // warp: role
  const int held = CHANNELS == 1 ? 0 : (tid >> 5) / CH_WARPS, c = CHANNELS == 1 ? (int)blockIdx.z : held;   // the CTA's channel, the image's
  ChannelShare& sh = all.ch[held];
  const int x0 = blockIdx.x * STRIP_W, y0 = blockIdx.y * seg_rows, y1 = min(y0 + seg_rows, H);
  const int x_end = min(x0 + STRIP_W, W);
  const float norm = lp.scale / (3.f * (float)W * (float)H);
  const float alpha_norm = lp.match_alpha_weight * lp.scale / ((float)W * (float)H);

  for (int i = tid; i < (int)(sizeof(all) / 16); i += THREADS) reinterpret_cast<float4*>(s_bytes)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  after_previous();
  __syncthreads();
  // The input pixels a thread fetches (zero outside the image and in the row pad): which, and whether their columns are inside
  // the image, does not change from step to step.
  constexpr int FETCH = (STRIP_ROWS * STRIP_IN + THREADS - 1) / THREADS;
  float3 f_p[FETCH];
  uint32_t f_t[FETCH];
  auto fetch = [&](int row0) {
#pragma unroll
    for (int u = 0; u < FETCH; u++) {
      const int e = tid + u * THREADS, row = e / STRIP_IN, col = e - row * STRIP_IN, x = x0 - 2 * HALO + col, y = row0 + row;
      f_p[u] = make_float3(0.f, 0.f, 0.f); f_t[u] = 0xFF000000u;   // an opaque black target is zero with any background
      if (e < STRIP_ROWS * STRIP_IN && col < STRIP_W + 4 * HALO && (unsigned)x < (unsigned)W && (unsigned)y < (unsigned)H) {
        const size_t q = (size_t)y * W + x;
        f_t[u] = gt[q];
        if constexpr (CHANNELS == 1) f_p[u].x = reinterpret_cast<const float*>(pred)[q * 4 + c];
        else { const float4 v = pred[q]; f_p[u] = make_float3(v.x, v.y, v.z); }
      }
    }
  };
  auto store = [&](int buf, int row0) {
#pragma unroll
    for (int u = 0; u < FETCH; u++) {
      const int e = tid + u * THREADS, row = e / STRIP_IN, col = e - row * STRIP_IN, px = col - 2 * HALO, slot = (row0 + row) & (PX_RING - 1);
      if (e >= STRIP_ROWS * STRIP_IN) break;
      const float p[3] = {f_p[u].x, f_p[u].y, f_p[u].z};
      const float behind = lp.composite ? 1.f - byte_unit(f_t[u], 3) : 0.f;
#pragma unroll
      for (int k = 0; k < CHANNELS; k++) {
        const int channel = CHANNELS == 1 ? c : k;
        const float2 v = make_float2(p[k], byte_unit(f_t[u], channel) + behind * lp.bg[channel]);
        all.ch[k].in[buf][row][pair_at(col)] = v;
        if (px >= 0 && px < PX_S) all.ch[k].px[slot][pair_at(px)] = v;
      }
    }
  };
  fetch(y0 - 2 * HALO);
  store(0, y0 - 2 * HALO);
  __syncthreads();

  float loss_local = 0.f;
  const int steps = 8 + (y1 - y0 + STRIP_ROWS - 1) / STRIP_ROWS;
  for (int it = 0; it <= steps; it++) {   // the last round only writes what stage D left in the one before
    const int a = y0 - 2 * HALO + STRIP_ROWS * it, b = a - 9, cr = b - 9, d = cr - STRIP_ROWS;
    const int buf = it & 1;
    const bool more = a + STRIP_ROWS <= y1 - 1 + 2 * HALO;   // stage A has rows to blur in the next step
    if (more) fetch(a + STRIP_ROWS);
    if (warp == 0) {
      // A: rows a .. a+3; a thread takes two rows and four statistics columns.
      if (a <= y1 - 1 + 2 * HALO) {
        const int r2 = (lane >> 4) * 2, g4 = (lane & 15) * 4;
        MomentRow *row_a = sh.moments + ring_slot(a + r2), *row_b = ring_next(row_a, sh.moments);
        float2 cross_in[14], cross[4];
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const float4* src = reinterpret_cast<const float4*>(sh.in[buf][r2 + r]);
          float2 mean[4], square[4];
#pragma unroll
          for (int o = 0; o < 4; o++) { mean[o] = make_float2(0.f, 0.f); square[o] = make_float2(0.f, 0.f); }
#pragma unroll
          for (int k2 = 0; k2 < 7; k2++) {
            const float4 v4 = src[chunk_at(g4 / 2 + k2)];
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int k = k2 * 2 + h;
              const float2 v = h ? hi2(v4) : lo2(v4), vv = __fmul2_rn(v, v);
              if (r == 0) cross_in[k].x = v.x * v.y; else cross_in[k].y = v.x * v.y;
#pragma unroll
              for (int o = 0; o < 4; o++)
                if (k - o >= 0 && k - o < 11) { mean[o] = __ffma2_rn(gauss.w[k - o], v, mean[o]); square[o] = __ffma2_rn(gauss.w[k - o], vv, square[o]); }
            }
          }
          MomentRow* row = r == 0 ? row_a : row_b;
          float4 *dm = reinterpret_cast<float4*>(row->mean), *dq = reinterpret_cast<float4*>(row->square);
          const int c0 = chunk_at(g4 / 2), c1 = chunk_at(g4 / 2 + 1);
          dm[c0] = make_float4(mean[0].x, mean[0].y, mean[1].x, mean[1].y); dm[c1] = make_float4(mean[2].x, mean[2].y, mean[3].x, mean[3].y);
          dq[c0] = make_float4(square[0].x, square[0].y, square[1].x, square[1].y); dq[c1] = make_float4(square[2].x, square[2].y, square[3].x, square[3].y);
        }
#pragma unroll
        for (int o = 0; o < 4; o++) {
          cross[o] = make_float2(0.f, 0.f);
#pragma unroll
          for (int k = 0; k < 11; k++) cross[o] = __ffma2_rn(gauss.w[k], cross_in[o + k], cross[o]);
        }
        *reinterpret_cast<float4*>(&row_a->cross[g4]) = make_float4(cross[0].x, cross[1].x, cross[2].x, cross[3].x);
        *reinterpret_cast<float4*>(&row_b->cross[g4]) = make_float4(cross[0].y, cross[1].y, cross[2].y, cross[3].y);
      }
    } else if (warp < 3) {
      // B: statistics rows b .. b+3; a thread takes one column.
      if (b + STRIP_ROWS - 1 >= y0 - HALO && b <= y1 - 1 + HALO) {
        const int col = (warp - 1) * 32 + lane, at = pair_at(col);
        const MomentRow* row = sh.moments + ring_slot(b - HALO);
        float2 mean[4], square[4];   // (prediction, target)
        float cross[4];
#pragma unroll
        for (int o = 0; o < 4; o++) { mean[o] = square[o] = make_float2(0.f, 0.f); cross[o] = 0.f; }
#pragma unroll
        for (int k = 0; k < 14; k++) {
          const float2 m2 = row->mean[at], q2 = row->square[at];
          const float x = row->cross[col];
          row = ring_next(row, const_cast<const MomentRow*>(sh.moments));
#pragma unroll
          for (int o = 0; o < 4; o++)
            if (k - o >= 0 && k - o < 11) {
              mean[o] = __ffma2_rn(gauss.w[k - o], m2, mean[o]); square[o] = __ffma2_rn(gauss.w[k - o], q2, square[o]);
              cross[o] = fmaf(gauss.w[k - o].x, x, cross[o]);
            }
        }
        const int xg = x0 - HALO + col;
        const bool col_in = xg >= 0 && xg < W, col_own = xg >= x0 && xg < x_end;
        MapRow* out = sh.maps + ring_slot(b);
#pragma unroll
        for (int o = 0; o < 4; o += 2) {   // two rows to a packed operation
          // Outside the image the weight is zero; the expressions below stay finite there (both images are zero).
          const int y = b + o;
          bool in[2], own[2];
          float2 M;
#pragma unroll
          for (int u = 0; u < 2; u++) {
            in[u] = col_in && y + u >= 0 && y + u < H; own[u] = col_own && y + u >= y0 && y + u < y1;
            float m = in[u] ? norm * lp.ssim_w : 0.f;
            if constexpr (MASKED) {
              if (in[u]) {
                const size_t q = (size_t)(y + u) * W + xg;
                if (weights) m *= (float)weights[q] * (1.f / 255.f);
                if (lp.mask) m *= byte_unit(gt[q], 3);
              }
            }
            (u ? M.y : M.x) = m;
          }
          const float2 mu1 = make_float2(mean[o].x, mean[o + 1].x), mu2 = make_float2(mean[o].y, mean[o + 1].y), mu1_sq = __fmul2_rn(mu1, mu1), two = make_float2(2.f, 2.f);
          const float2 neg1 = make_float2(-mu1.x, -mu1.y), neg2 = make_float2(-mu2.x, -mu2.y), dbl1 = __fadd2_rn(mu1, mu1), dbl2 = __fadd2_rn(mu2, mu2);
          const float2 c1 = make_float2(C1, C1), c2 = make_float2(C2, C2);
          // The expressions round as they always have (where a product is fused into a sum matters here: variances are small
          // differences, and so is the gradient below).
          const float2 s1_raw = __ffma2_rn(make_float2(-1.f, -1.f), mu1_sq, make_float2(square[o].x, square[o + 1].x));
          const float2 s2_raw = __ffma2_rn(neg2, mu2, make_float2(square[o].y, square[o + 1].y));
          const float2 sigma12 = __ffma2_rn(neg1, mu2, make_float2(cross[o], cross[o + 1]));
          const float2 A1 = __ffma2_rn(dbl1, mu2, c1), A2 = __ffma2_rn(two, sigma12, c2), B1 = __fadd2_rn(__ffma2_rn(mu2, mu2, mu1_sq), c1);
          const float2 B2 = __fadd2_rn(__fadd2_rn(make_float2(fmaxf(0.f, s1_raw.x), fmaxf(0.f, s1_raw.y)), make_float2(fmaxf(0.f, s2_raw.x), fmaxf(0.f, s2_raw.y))), c2);
          const float2 BB = __fmul2_rn(B1, B2);
          // approximate divisions, as in the reference's fast-math build
          const float2 inv_BB = make_float2(fast_rcp(BB.x), fast_rcp(BB.y)), inv_B1 = make_float2(fast_rcp(B1.x), fast_rcp(B1.y)), inv_B2 = make_float2(fast_rcp(B2.x), fast_rcp(B2.y));
          const float2 raw = __fmul2_rn(__fmul2_rn(A1, A2), inv_BB);
          const float2 ssim = make_float2(fminf(fmaxf(raw.x, -1.f), 1.f), fminf(fmaxf(raw.y, -1.f), 1.f));
          loss_local += (own[0] ? M.x * ssim.x : 0.f) + (own[1] ? M.y * ssim.y : 0.f);
          const float2 k = make_float2(raw.x > -1.f && raw.x < 1.f ? M.x : 0.f, raw.y > -1.f && raw.y < 1.f ? M.y : 0.f);   // the clamp has zero slope
          const float2 held = __fmul2_rn(__fmul2_rn(dbl1, ssim), inv_B1), d_mu1 = __ffma2_rn(__fmul2_rn(dbl2, A2), inv_BB, make_float2(-held.x, -held.y));
          const float2 share = __fmul2_rn(ssim, inv_B2), d_s1 = make_float2(s1_raw.x > 0.f ? -share.x : 0.f, s1_raw.y > 0.f ? -share.y : 0.f);
          const float2 Bv = __fmul2_rn(k, d_s1), Cc = __fmul2_rn(k, __fmul2_rn(__fadd2_rn(A1, A1), inv_BB)), pull = __fmul2_rn(Bv, mu1);
          // gradient = blur(Am) + 2 p blur(Bv) - 2 blur(Bv mu1) + target blur(Cc) - blur(Cc mu2): the three maps
          // without a per-pixel factor are blurred as one.
          const float2 e0 = __ffma2_rn(Cc, neg2, __ffma2_rn(k, d_mu1, __fmul2_rn(make_float2(-2.f, -2.f), pull)));
          out->e12[at] = make_float2(Bv.x, Cc.x); out->e0[col] = e0.x;
          out = ring_next(out, sh.maps);
          out->e12[at] = make_float2(Bv.y, Cc.y); out->e0[col] = e0.y;
          out = ring_next(out, sh.maps);
        }
      }
    } else if (warp == 3) {
      // C: rows cr .. cr+3 of the derivative maps blurred down the column, two columns per thread.
      if (cr + STRIP_ROWS - 1 >= y0 && cr < y1) {
        const int col = lane * 2, chunk = chunk_at(lane);
        const MapRow* row = sh.maps + ring_slot(cr - HALO);
        float2 b12[4][2], b0[4];
#pragma unroll
        for (int o = 0; o < 4; o++) b12[o][0] = b12[o][1] = b0[o] = make_float2(0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 14; k++) {
          const float4 e4 = reinterpret_cast<const float4*>(row->e12)[chunk];
          const float2 z2 = *reinterpret_cast<const float2*>(&row->e0[col]);
          row = ring_next(row, const_cast<const MapRow*>(sh.maps));
#pragma unroll
          for (int o = 0; o < 4; o++)
            if (k - o >= 0 && k - o < 11) {
              const float2 w = gauss.w[k - o];
              b12[o][0] = __ffma2_rn(w, lo2(e4), b12[o][0]); b12[o][1] = __ffma2_rn(w, hi2(e4), b12[o][1]); b0[o] = __ffma2_rn(w, z2, b0[o]);
            }
        }
#pragma unroll
        for (int o = 0; o < 4; o++) {
          reinterpret_cast<float4*>(sh.b12[buf][o])[chunk] = make_float4(b12[o][0].x, b12[o][0].y, b12[o][1].x, b12[o][1].y);
          *reinterpret_cast<float2*>(&sh.b0[buf][o][col]) = b0[o];
        }
      }
    } else {
      // D: rows d .. d+3 (stage C wrote them in the step before), fourteen groups of four output columns.
      const int row = (warp - 4) * 2 + (lane >> 4), g4 = (lane & 15) * 4, y = d + row;
      if (g4 < STRIP_W && y >= y0 && y < y1) {
        float2 b12[4];
        float b0[4];
#pragma unroll
        for (int o = 0; o < 4; o++) { b12[o] = make_float2(0.f, 0.f); b0[o] = 0.f; }
        const float4* s12 = reinterpret_cast<const float4*>(sh.b12[buf ^ 1][row]);
        const float4* s0 = reinterpret_cast<const float4*>(&sh.b0[buf ^ 1][row][g4]);
#pragma unroll
        for (int k2 = 0; k2 < 7; k2++) {
          const float4 v4 = s12[chunk_at(g4 / 2 + k2)];
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int o = 0; o < 4; o++) { const int k = k2 * 2 + h - o; if (k >= 0 && k < 11) b12[o] = __ffma2_rn(gauss.w[k], h ? hi2(v4) : lo2(v4), b12[o]); }
        }
#pragma unroll
        for (int k4 = 0; k4 < 4; k4++) {
          const float4 v4 = s0[k4];
          const float v[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
          for (int h = 0; h < 4; h++)
#pragma unroll
            for (int o = 0; o < 4; o++) { const int k = k4 * 4 + h - o; if (k >= 0 && k < 11) b0[o] = fmaf(gauss.w[k].x, v[h], b0[o]); }
        }
        const float4* own_row = reinterpret_cast<const float4*>(sh.px[y & (PX_RING - 1)]);
        const float4 own[2] = {own_row[chunk_at(g4 / 2)], own_row[chunk_at(g4 / 2 + 1)]};
#pragma unroll
        for (int o = 0; o < 4; o++) {
          const int x = x0 + g4 + o;
          if (x < x_end) {
            const float2 pg = o & 1 ? hi2(own[o >> 1]) : lo2(own[o >> 1]);
            float M = norm * lp.l1_w;
            if constexpr (MASKED) {
              const size_t q = (size_t)y * W + x;
              const float wp = weights ? (float)weights[q] * (1.f / 255.f) : 1.f, ga = byte_unit(gt[q], 3);
              M *= wp * (lp.mask ? ga : 1.f);
              if (c == 0 && lp.alpha_lane) {   // the alpha lane travels with the first channel
                const float da = pred[q].w - ga, Ma = wp * alpha_norm;
                all.out[buf][row][g4 + o][3] = (da > 0.f ? Ma : (da < 0.f ? -Ma : 0.f)) * lp.grad_scale;
                loss_local += Ma * fabsf(da);
              }
            }
            const float diff = pg.x - pg.y;
            loss_local += M * fabsf(diff);
            const float l1 = diff > 0.f ? M : (diff < 0.f ? -M : 0.f);
            all.out[buf][row][g4 + o][c] = (l1 + b0[o] + 2.f * pg.x * b12[o].x + pg.y * b12[o].y) * lp.grad_scale;
          }
        }
      }
    }
    {
      // The gradient rows that stage D left in the step before.
      constexpr int DRAIN = (STRIP_ROWS * PX_S + THREADS - 1) / THREADS;
#pragma unroll
      for (int u = 0; u < DRAIN; u++) {
        const int e = tid + u * THREADS, row = e / PX_S, col = e - row * PX_S, y = d - STRIP_ROWS + row, x = x0 + col;
        if (row >= STRIP_ROWS || col >= STRIP_W || x >= x_end || y < y0 || y >= y1) continue;
        const float4 v = *reinterpret_cast<const float4*>(all.out[buf ^ 1][row][col]);
        if constexpr (CHANNELS == 1) {
          float* out = reinterpret_cast<float*>(v_out + (size_t)y * W + x);
          out[c] = c == 0 ? v.x : (c == 1 ? v.y : v.z);
          if (c == 0) out[3] = v.w;
        } else v_out[(size_t)y * W + x] = v;
      }
    }
    if (more) store(buf ^ 1, a + STRIP_ROWS);   // consumed by stage A in the next step
    __syncthreads();
  }
  const float s = warp_sum(loss_local);
  if (lane == 0) all.red[tid >> 5] = s;
  __syncthreads();
  if (tid == 0) {
    float t = 0.f;
    for (int i = 0; i < THREADS / 32; i++) t += all.red[i];
    if (t != 0.f) atomicAdd(loss_accum, t);
  }
}

// Evaluation metrics (eval_metrics, src/gpu/loss.cu:241-293): squared error and SSIM sums of the 8-bit-quantised
// prediction against the target on a black background, optionally weighted by the target's alpha.
//
// One CTA takes a tile of 32x32 pixels of one channel: the quantised prediction and the target of its 42x42 footprint are staged
// side by side, both blur passes run on packed pairs of them (fp32x2) and make four outputs from one fourteen-wide window, rows
// in the order that avoids bank conflicts (chunk_at), and the vertical pass goes straight on to the metrics. Bound by instruction issue.
// Against 16x16 tiles that ran the channels one after the other on a quarter to a half of their threads: 1237x822 65 -> 41 us.
constexpr int EV_T = 32, EV_F = EV_T + 2 * HALO, EV_S = 48;   // tile, footprint, pairs of a staged row (padded to whole groups of chunks)
constexpr int EV_THREADS = 256;
struct EvalShare {
  float2 in[EV_F][EV_S];                       // (quantised prediction, target)
  float2 mean[EV_F][EV_T], square[EV_F][EV_T]; // blurred along the row
  float cross[EV_F][EV_T];
};
static_assert(EV_T * EV_T / 4 == EV_THREADS, "one column of four outputs per thread");

__global__ void __launch_bounds__(EV_THREADS, 4) eval_kernel(const float4* __restrict__ pred, const uint32_t* __restrict__ gt, int W, int H, int mask_w, Gauss2 gauss,
                                                          float* __restrict__ accum) {
  after_previous();
  __shared__ __align__(16) EvalShare sh;
  __shared__ float s_part[2][EV_THREADS / 32];
  const int tid = threadIdx.x, c = blockIdx.z;
  const int x0 = blockIdx.x * EV_T, y0 = blockIdx.y * EV_T;
  const float* pred_c = reinterpret_cast<const float*>(pred) + c;
  for (int fy = tid / EV_S, fx = tid % EV_S; fy < EV_F;) {
    const int y = y0 + fy - HALO, x = x0 + fx - HALO;
    float2 v = make_float2(0.f, 0.f);   // zero padding outside the image and in the row pad
    if (fx < EV_F && (unsigned)y < (unsigned)H && (unsigned)x < (unsigned)W) {
      const size_t q = (size_t)(y * W + x);
      // level / 255, correctly rounded (checked for all 256 levels), without a division
      const float level = rintf(fminf(fmaxf(pred_c[q * 4], 0.f), 1.f) * 255.f), near = level * (1.f / 255.f);
      v = make_float2(fmaf(fmaf(-255.f, near, level), 1.f / 255.f, near), byte_unit(gt[q], c));
    }
    sh.in[fy][pair_at(fx)] = v;
    fx += EV_THREADS % EV_S; fy += EV_THREADS / EV_S;   // EV_THREADS elements on
    if (fx >= EV_S) { fx -= EV_S; fy++; }
  }
  __syncthreads();
  // Along the rows: eight groups of four output columns each.
  for (int t = tid; t < EV_F * (EV_T / 4); t += EV_THREADS) {
    const int row = t / (EV_T / 4), g4 = (t % (EV_T / 4)) * 4;
    const float4* src = reinterpret_cast<const float4*>(sh.in[row]);
    float2 mean[4], square[4];
    float cross[4];
#pragma unroll
    for (int o = 0; o < 4; o++) { mean[o] = square[o] = make_float2(0.f, 0.f); cross[o] = 0.f; }
#pragma unroll
    for (int k2 = 0; k2 < 7; k2++) {
      const float4 v4 = src[chunk_at(g4 / 2 + k2)];
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int k = k2 * 2 + h;
        const float2 v = h ? hi2(v4) : lo2(v4), vv = __fmul2_rn(v, v);
        const float x = v.x * v.y;
#pragma unroll
        for (int o = 0; o < 4; o++)
          if (k - o >= 0 && k - o < 11) {
            mean[o] = __ffma2_rn(gauss.w[k - o], v, mean[o]); square[o] = __ffma2_rn(gauss.w[k - o], vv, square[o]); cross[o] = fmaf(gauss.w[k - o].x, x, cross[o]);
          }
      }
    }
    float4 *dm = reinterpret_cast<float4*>(sh.mean[row]), *dq = reinterpret_cast<float4*>(sh.square[row]);
    const int c0 = chunk_at(g4 / 2), c1 = chunk_at(g4 / 2 + 1);
    dm[c0] = make_float4(mean[0].x, mean[0].y, mean[1].x, mean[1].y); dm[c1] = make_float4(mean[2].x, mean[2].y, mean[3].x, mean[3].y);
    dq[c0] = make_float4(square[0].x, square[0].y, square[1].x, square[1].y); dq[c1] = make_float4(square[2].x, square[2].y, square[3].x, square[3].y);
    *reinterpret_cast<float4*>(&sh.cross[row][g4]) = make_float4(cross[0], cross[1], cross[2], cross[3]);
  }
  __syncthreads();
  // Down the columns, and the metrics: a column of four outputs per thread.
  float se_sum = 0.f, ssim_sum = 0.f;
  {
    const int col = tid & (EV_T - 1), r4 = (tid / EV_T) * 4, at = pair_at(col);
    float2 mean[4], square[4];
    float cross[4];
#pragma unroll
    for (int o = 0; o < 4; o++) { mean[o] = square[o] = make_float2(0.f, 0.f); cross[o] = 0.f; }
#pragma unroll
    for (int k = 0; k < 14; k++) {
      const float2 m2 = sh.mean[r4 + k][at], q2 = sh.square[r4 + k][at];
      const float x = sh.cross[r4 + k][col];
#pragma unroll
      for (int o = 0; o < 4; o++)
        if (k - o >= 0 && k - o < 11) {
          mean[o] = __ffma2_rn(gauss.w[k - o], m2, mean[o]); square[o] = __ffma2_rn(gauss.w[k - o], q2, square[o]); cross[o] = fmaf(gauss.w[k - o].x, x, cross[o]);
        }
    }
#pragma unroll
    for (int o = 0; o < 4; o++) {
      const int y = y0 + r4 + o, x = x0 + col;
      if (y < H && x < W) {
        const float mu_p = mean[o].x, mu_t = mean[o].y;
        const float var_p = fmaxf(0.f, square[o].x - mu_p * mu_p), var_t = fmaxf(0.f, square[o].y - mu_t * mu_t), cov = cross[o] - mu_p * mu_t;
        const float raw = ((2.f * mu_p * mu_t + C1) * (2.f * cov + C2)) / ((mu_p * mu_p + mu_t * mu_t + C1) * (var_p + var_t + C2));
        const float2 centre = sh.in[r4 + o + HALO][pair_at(col + HALO)];
        const float wgt = mask_w ? unpack(gt[(size_t)y * W + x], 3) : 1.f;
        const float err = fabsf(centre.x - centre.y) * wgt;
        se_sum += err * err;
        ssim_sum += fminf(fmaxf(raw, -1.f), 1.f) * wgt;
      }
    }
  }
  const float a = warp_sum(se_sum), b = warp_sum(ssim_sum);
  if ((tid & 31) == 0) { s_part[0][tid >> 5] = a; s_part[1][tid >> 5] = b; }
  __syncthreads();
  if (tid < 2) {
    float total = 0.f;
    for (int i = 0; i < EV_THREADS / 32; i++) total += s_part[tid][i];
    atomicAdd(accum + 4 + tid, total);
  }
}

// Running loss sum and view count; also keeps the largest intersection total any view of the step produced, so that
// one readback per step (instead of one per view) tells the host whether a view overflowed its buffers.
__global__ void accumulate_kernel(float* a, uint32_t* num_isect) {
  after_previous();
  a[2] += a[0] + a[1]; a[3] += 1.f;
  if (num_isect) num_isect[2] = max(num_isect[2], num_isect[0]);
}
// dst[2] += src[2], dst[3] += src[3]: folds the running loss of a second context (a view in flight on another stream).
__global__ void fold_loss_kernel(float* dst, const float* src) { after_previous(); dst[2] += src[2]; dst[3] += src[3]; }

}  // namespace
}  // namespace b2k

using namespace b2k;

extern "C" int b2k_loss_photometric(const B2kCtx* c, const B2kLoss* lp, b2k_stream_t stream) {
  B2K_REQUIRE(c && lp && lp->rgba && c->out_rgba && c->v_out && c->loss_accum && c->W > 0 && c->H > 0);
  LossArgs a;
  a.l1_w = lp->l1_w; a.ssim_w = lp->ssim_w; a.bg[0] = lp->bg[0]; a.bg[1] = lp->bg[1]; a.bg[2] = lp->bg[2];
  a.composite = lp->composite; a.mask = lp->mask; a.alpha_lane = lp->alpha_lane;
  a.match_alpha_weight = lp->match_alpha_weight; a.scale = lp->scale; a.grad_scale = lp->grad_scale;
  static const Gauss2 g2 = make_gauss();
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64 && !attr_set[dev]) {
    B2K_CUDA(cudaFuncSetAttribute(photometric_strip_kernel<false, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StripShare<3>)));
    B2K_CUDA(cudaFuncSetAttribute(photometric_strip_kernel<true, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StripShare<3>)));
    B2K_CUDA(cudaFuncSetAttribute(photometric_strip_kernel<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StripShare<1>)));
    B2K_CUDA(cudaFuncSetAttribute(photometric_strip_kernel<true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StripShare<1>)));
    attr_set[dev] = true;
  }
  // Rows per segment: as many segments as there are SMs (a second, partial wave costs more than the eight pipeline-fill
  // steps a longer segment amortises), in whole steps of four rows.
  const int strips = div_up(c->W, STRIP_W);
  auto rows_for = [&](int columns) {   // CTAs side by side
    const int segs = std::max(1, sm_count() / columns);
    return std::max(8, div_up(div_up(c->H, segs), STRIP_ROWS) * STRIP_ROWS);
  };
  auto steps_of = [](int rows) { return 8 + rows / STRIP_ROWS; };
  // A CTA per channel steps faster than one of three channels (64x64 0.96 against 1.46 us a step, 333x217 with mask 1.7 against
  // 2.0) but leaves a third of the SMs to cut the rows for: taken where its segments are at most a fifth longer in steps (64x64
  // 14.6 -> 9.6 us, 200x150 14.9 -> 11.8; 333x217 would go from 22.4 to 27.2).
  const int rows3 = rows_for(strips), rows1 = rows_for(strips * 3);
  // It is also the one that writes the gradient by single floats: taken where the caller's array is not aligned for whole pixels.
  const bool whole_pixels = (((uintptr_t)c->out_rgba | (uintptr_t)c->v_out) & 15) == 0;
  const bool apart = !whole_pixels || (steps_of(rows1) * 5 <= steps_of(rows3) * 6 && strips * 3 <= sm_count());
  const int seg_rows = apart ? rows1 : rows3;
  const dim3 grid(strips, div_up(c->H, seg_rows), apart ? 3 : 1);
#define L(MASKED, CHANNELS) launch_next(photometric_strip_kernel<MASKED, CHANNELS>, grid, CHANNELS * CH_THREADS, sizeof(StripShare<CHANNELS>), (cudaStream_t)stream, \
    (const float4*)c->out_rgba, lp->rgba, lp->weights, c->W, c->H, seg_rows, a, g2, (float4*)c->v_out, c->loss_accum)
  const bool masked = lp->weights || lp->mask || lp->alpha_lane;
  if (apart) { if (masked) L(true, 1); else L(false, 1); }
  else { if (masked) L(true, 3); else L(false, 3); }
#undef L
  return check_launch();
}

extern "C" int b2k_loss_accumulate(const B2kCtx* c, b2k_stream_t stream) {
  B2K_REQUIRE(c && c->loss_accum);
  launch_next(accumulate_kernel, 1, 1, 0, (cudaStream_t)stream, c->loss_accum, c->num_isect);
  return check_launch();
}

extern "C" int b2k_loss_zero(const B2kCtx* c, int32_t first, int32_t count, b2k_stream_t stream) {
  B2K_REQUIRE(c && c->loss_accum && first >= 0 && count >= 0 && first + count <= 16);
  if (count) launch_clear(c->loss_accum + first, count, nullptr, 0, (cudaStream_t)stream);
  return check_launch();
}

extern "C" int b2k_step_begin(const B2kCtx* c, b2k_stream_t stream) {
  B2K_REQUIRE(c && c->loss_accum);
  launch_clear(c->loss_accum, 16, c->num_isect ? c->num_isect + 2 : nullptr, c->num_isect ? 1 : 0, (cudaStream_t)stream);
  return check_launch();
}

extern "C" int b2k_loss_fold(const B2kCtx* dst, const B2kCtx* src, b2k_stream_t stream) {
  B2K_REQUIRE(dst && src && dst->loss_accum && src->loss_accum && dst->loss_accum != src->loss_accum);
  launch_next(fold_loss_kernel, 1, 1, 0, (cudaStream_t)stream, dst->loss_accum, src->loss_accum);
  return check_launch();
}

extern "C" int b2k_eval_metrics(const B2kCtx* c, const uint32_t* rgba, int32_t mask_weighted, b2k_stream_t stream) {
  B2K_REQUIRE(c && rgba && c->out_rgba && c->loss_accum && c->W > 0 && c->H > 0);
  static const Gauss2 g = make_gauss();
  launch_next(eval_kernel, dim3(div_up(c->W, EV_T), div_up(c->H, EV_T), 3), EV_THREADS, 0, (cudaStream_t)stream, (const float4*)c->out_rgba, rgba, c->W, c->H, mask_weighted, g,
              c->loss_accum);
  return check_launch();
}
