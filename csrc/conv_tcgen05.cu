// K13: causal 3x3x3 convolutions of the video tokenizer as an implicit GEMM on tcgen05, on channels-last bf16 volumes
// [frames, H + 2, W + 2, C] with a zero border. The two frames before the first one are a tensor of their own (absent: zero, and
// their products are left out), and so may be a volume's last two frames, which are the next chunk's: what a chunk hands on is
// neither copied nor holds the whole volume.
//
// A CTA pair (cta_group::2) computes R x 256 rows (positions of a frame) by up to 256 output channels. A plain implicit GEMM
// fetches a fresh 128-row tile of activations for each of the 27 taps, more than L2 delivers into shared memory under the
// products (60 - 80 B per clock and SM). Here
//   * the three taps of one row of the filter read one staged tile of 128 R + 8 rows at row offsets 0, 1 and 2: the matrix
//     descriptor starts in the middle of a swizzle atom (the swizzle is a function of the shared-memory address), so a tile
//     crosses L2 -> shared memory 9 times and not 27;
//   * with 128 output channels or fewer R = 2 row tiles share each weight tile, in tensor memory as two accumulators of 128
//     columns, double-buffered against the epilogue;
//   * activations and weights have rings of their own, so that a weight tile holds its slot for one product and an
//     activation tile for three.
// Per 64 channels, tap and 128 rows a CTA of the pair stages 5.6 KB of activations and 4 of weights at 128 output channels, where
// a tile for each tap would take 16 and 8. Wide layers are bound by the products at the power limit (figures below), narrow ones by
// the epilogue (64 channels and less, conv_time_kernel), the first and the last by memory.
//
// A strided convolution reads its input split into the four parities of (row, column) ("s2d": [frames, 4, (H + 2) / 2,
// (W + 2) / 2, C]), which the layer before it writes; each tap is then again a row offset, taps of equal column parity share
// a tile, and only the kept positions and frames are computed.
//
// The epilogue adds bias and residual, writes zeros on the border, and can write: the volume, the s2d form, the nearest
// upsampling by two in space, and in time, that the next convolution reads, and / or silu(rmsnorm(.)) over the channels (a thread holds a
// whole row); or, for the 3 output channels of the decoder, uint8 pixels.
//
// Measured (480p, chunks of 8 frames at full resolution): 128 -> 128 channels with skip projection 1.95 ms = 1.47 PFLOP/s,
// 256 -> 256 at half resolution 1.9 ms = 1.5, 256 -> 128 0.93 ms = 1.52, 64 -> 128 with norm 1.2 ms = 1.2: at these rates the GPU runs at
// its power limit (1.45 GHz, tensor pipe busy 83 % of the clocks). The one-tile-per-tap form with its separate passes took 48 ms a
// chunk of the encoder's convolutions and norms where this takes 8.7.
// Order of the sum: filter taps, then channel blocks of 64 (of up to 256 channels at a time). Waits are bounded as
// everywhere (common.cuh).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace cb {
using namespace cosmos;   // ConvOut

// Rows of a tile: those of its row tiles and the 2 that shifted taps need, in boxes of whole swizzle atoms (8 rows).
__host__ __device__ constexpr int cv_box_rows(int r) { return r == 2 ? 88 : 136; }
__host__ __device__ constexpr int cv_boxes(int r) { return r == 2 ? 3 : 1; }
constexpr int CV_MAX_GROUPS = 18;
constexpr int CV_CHUNK = 4;                    // channel blocks of 64 whose tiles are staged together
constexpr int CV_SMEM_MAX = 227 * 1024;
constexpr int CV_BARS = 512;                   // bytes for barriers, tensor-memory slot and abort flag
constexpr int CV_SUMS = 8192;                  // row sums of the norm: [2 tiles][2 row tiles][2 column halves][128 rows][2] floats
constexpr int CV_GAMMA = 1024;                 // the norm's weights as fp32; behind them the bias (up to 256 channels)
constexpr int CV_TAIL = CV_BARS + CV_SUMS + 2 * CV_GAMMA;

// Taps that read one staged tile: row offset of the tile, and per tap its shift inside the tile and its index in the weights.
struct ConvGroup {
  int kt;                // tap of time: input frame = output frame (kept frame's place) + kt - 2
  int off;               // rows, inside the input frame
  int n_taps;
  short shift[3], tap[3];
};

// Frames 0 .. split - 1 in one tensor, the others in a second.
template <typename P>
struct Split {
  P body, tail;          // `tail`: where frame 0 of the second tensor's frames would be
  int split;
  __device__ __forceinline__ P at(int frame) const { return frame < split ? body : tail; }
};

struct ConvParams {
  ConvGroup g[CV_MAX_GROUPS];
  int n_groups;          // over the input volume; the skip projection (second input) has one group of one tap, offset 0
  int cblocks, skip_cblocks, skip_kcol;
  int n_out, mma_n, n_tiles;
  int na, nb;            // ring slots
  // rows: n_seg segments (frames of a strided convolution, else one) of seg_rows rows
  int n_seg, seg_rows, tiles_per_seg;
  int frame_rows;        // rows of an input frame
  int has_ctx;           // else the products with its two frames are left out
  int v_first, v_step;   // segment s begins at input frame v_first + s v_step (counted from the first context frame)
  int x_split, skip_split;
  int pw, plane;         // width and size of the plane that a segment's rows walk through
  int hp, wp;            // padded size of that plane (strided: kept rows + 1, kept columns + 1)
  const float* bias;
  Split<const bf16*> resid;   // layout of the volume; null body and tail: none
  Split<bf16*> out;           // raw result
  Split<bf16*> out_norm;      // silu(rmsnorm(result))
  int has_resid, has_out, has_norm;
  const bf16* gamma;
  float eps;
  uint8_t* rgb;
  int mode;              // CONV_OUT_*
  int keep_border;       // CONV_OUT_SAME: the border's cells are not written
  int f_out;             // frames computed
  int seg_frames;        // conv_time_kernel: output frames of a time segment (n_seg of them)
  int kt_taps;           // taps of a frame in the weights: 9, or 1 (taps in time only)
  int nt;                // conv_time_kernel: accumulator columns of a frame, 16, 32 or 64
  int up_t, up_first;    // CONV_OUT_UP: temporal doubling, first chunk (its first frame is not doubled)
  int* status;
};

template <int R>
struct ConvCfg {
  static constexpr int BOX = cv_box_rows(R), BOXES = cv_boxes(R), A_ROWS = BOX * BOXES;
  static constexpr int A_SLOT = A_ROWS * 128;
  static constexpr int ACC_COLS = 256 / R;     // tensor-memory columns of one accumulator
  static constexpr int THREADS = 96 + 256 * R; // producer, MMA issuer, eight epilogue warps per row tile, second producer
};

// The 16 columns of a row are 32 bytes, one sector, held by one thread. Stored by it as two vectors they reach L2 as half sectors,
// two requests for each, and L2 reads the sector from memory to complete it: the first layer of the encoder (64 channels, two outputs)
// read 1.23 GB where its input has 0.41. So neighbouring lanes swap halves, and a store instruction writes whole sectors of every
// other row: first those of the even lanes' rows (`even`), then those of the odd lanes' (`odd`), lane parity = half of the sector.
__device__ __forceinline__ void cv_swap_halves(const uint32_t (&pk)[8], int lane, uint4& even, uint4& odd) {
  const bool o = lane & 1;
  uint32_t r[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = __shfl_xor_sync(0xffffffffu, o ? pk[k] : pk[4 + k], 1);
  even = o ? make_uint4(r[0], r[1], r[2], r[3]) : make_uint4(pk[0], pk[1], pk[2], pk[3]);
  odd = o ? make_uint4(pk[4], pk[5], pk[6], pk[7]) : make_uint4(r[0], r[1], r[2], r[3]);
}

// silu(z) = z / (1 + exp(-z)) of two values given as their negatives: z times an approximate reciprocal, with one step of iterative
// refinement by the residual (silu16 in common.cuh takes two); negatives of value and reciprocal let every step be a packed
// instruction. For magnitudes below 80. Of all 2^32 values two differ from the division's result, in their last bit, and none
// once it is rounded to bf16 (conv_silu_selftest).
__device__ __forceinline__ float2 cv_silu2(uint64_t zn) {
  const float2 t = unpack2(mul2(zn, pack2(1.4426950408889634f, 1.4426950408889634f)));
  const uint64_t den = add2(pack2(ex2(t.x), ex2(t.y)), pack2(1.f, 1.f));
  const float2 d = unpack2(den);
  float r0, r1;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-d.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-d.y));
  const uint64_t rn = pack2(r0, r1), q = mul2(zn, rn);
  return unpack2(fma2(fma2(q, den, zn), rn, q));
}
// 16 of them rounded to bf16. Beyond 80, where the exponential leaves its range, and for infinities the division itself.
__device__ __forceinline__ void cv_silu16(const uint64_t (&zn)[8], uint32_t (&out)[8]) {
  float top = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float2 z = unpack2(zn[k]);
    top = fmaxf(top, fmaxf(fabsf(z.x), fabsf(z.y)));
    const float2 y = cv_silu2(zn[k]);
    out[k] = pack_bf16(y.x, y.y);
  }
  if (top >= 80.f) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float2 z = unpack2(zn[k]);
      out[k] = pack_bf16(-z.x / (1.f + __expf(z.x)), -z.y / (1.f + __expf(z.y)));
    }
  }
}

// Meeting of the two warps that share the rows of a quadrant. Both come to every one of them: a warp whose wait for an accumulator
// gave up goes on without storing (the later waits give up at once).
__device__ __forceinline__ void cv_meet(int id) { asm volatile("barrier.cta.sync %0, 64;" ::"r"(id) : "memory"); }

// Input frame v, counted from the first context frame: the tensor that holds it and its first row there.
struct ConvSource {
  const CUtensorMap* map;
  int row;
};
__device__ __forceinline__ ConvSource conv_source(const ConvParams& p, int v, const CUtensorMap* ctx, const CUtensorMap* body,
                                                  const CUtensorMap* tail) {
  if (v < 2) return {ctx, v * p.frame_rows};
  if (v - 2 < p.x_split) return {body, (v - 2) * p.frame_rows};
  return {tail, (v - 2 - p.x_split) * p.frame_rows};
}

// Where a row of the result goes: `n_t` x `n_y` x `n_x` rows starting at `row` (one row except for the upsampled form).
struct ConvDest {
  long long row, st, sy;
  int frame;             // the first of the frames
  int n_t, n_y, n_x;
};

__device__ __forceinline__ ConvDest conv_dest(const ConvParams& p, int f, int y, int x) {
  ConvDest d{0, 0, 0, f, 1, 1, 1};
  if (p.mode == CONV_OUT_SAME) {
    d.row = (long long)f * p.plane + y * p.pw + x;
  } else if (p.mode == CONV_OUT_S2D) {
    const int q = (p.hp >> 1) * (p.wp >> 1);
    d.row = ((long long)f * 4 + (y & 1) * 2 + (x & 1)) * q + (y >> 1) * (p.wp >> 1) + (x >> 1);
  } else if (p.mode == CONV_OUT_DOWN) {
    d.row = ((long long)f * (p.hp + 1) + y + 1) * (p.wp + 1) + x + 1;
  } else {  // CONV_OUT_UP: interior position (y, x) -> rows 2y - 1, 2y and columns 2x - 1, 2x; the border stays one wide
    const int hd = 2 * (p.hp - 2) + 2, wd = 2 * (p.wp - 2) + 2;
    const int y0 = y == 0 ? 0 : 2 * y - 1, x0 = x == 0 ? 0 : 2 * x - 1;
    int t0 = f;
    if (p.up_t) {
      t0 = p.up_first ? max(0, 2 * f - 1) : 2 * f;
      d.n_t = p.up_first && f == 0 ? 1 : 2;
    }
    d.n_y = (y == 0 || y == p.hp - 1) ? 1 : 2;
    d.n_x = (x == 0 || x == p.wp - 1) ? 1 : 2;
    d.sy = wd;
    d.st = (long long)hd * wd;
    d.frame = t0;
    d.row = t0 * d.st + (long long)y0 * wd + x0;   // both frames of a doubled one are in one tensor: the last two share a pair
  }
  return d;
}

// One accumulator's row per thread, at tensor-memory address `ta` (the quadrant's lanes): row (y, x) of the plane, `rem` in it, of
// frame `f`; output channels from `n_base` on. The two warps of a quadrant take every other group of 16 columns (`half`) and
// meet at named barrier `pair_id`; sums: where this row's sum of squares goes, [2 halves][128]. ZERO: the accumulator is left
// zero for the next frame's products.
// `release` hands the accumulator back and is called once the last of it is read.
template <int NC, bool RGB, bool ZERO, int U, typename Release>
__device__ __forceinline__ void conv_emit(const ConvParams& p, uint32_t ta, int f, int rem, int y, int x, bool row_ok, int n_base,
                                          int half, int pair_id, float2* sums, const float* gamma, const float* bias, Release release) {
  const bool down = p.mode == CONV_OUT_DOWN;
  const bool inside = row_ok && (down ? (y < p.hp - 1 && x < p.wp - 1) : (y >= 1 && y <= p.hp - 2 && x >= 1 && x <= p.wp - 2));
  const uint32_t zero16[16] = {};
  if constexpr (RGB) {
    uint32_t v[16];
    tmem_ld16(ta, v);
    tmem_wait_ld();
    if constexpr (ZERO) {
      if (half == 0) tmem_st16(ta, zero16);
      tmem_wait_st();
    }
    release();
    if (inside && half == 0) {
      uint8_t* o = p.rgb + (((long long)f * (p.hp - 2) + y - 1) * (p.wp - 2) + x - 1) * 3;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        // columns 3 .. 8: the low parts of fp32 weights, exact in three bf16 terms
        const float a = ((__uint_as_float(v[6 + c]) + __uint_as_float(v[3 + c])) + __uint_as_float(v[c])) + bias[c];
        o[c] = (uint8_t)__float2int_rn((fminf(fmaxf(a, -1.f), 1.f) + 1.f) * 127.5f);
      }
    }
  } else {
    const ConvDest dst = conv_dest(p, f, y, x);
    const int n_end = min(256, p.n_out - n_base);
    const long long ld = p.n_out;
    if (down && row_ok && half == 0 && (x == 0 || y == 0)) {
      // border cells that no position of the plane maps to: left column, top row
      for (int k = 0; k < 3; ++k) {
        if ((k == 0 && x != 0) || (k == 1 && y != 0) || (k == 2 && (x != 0 || y != 0))) continue;
        const long long cell = dst.row - (k == 1 ? 0 : 1) - (k == 0 ? 0 : p.wp + 1);
        for (int c = 0; c < n_end; c += 8) {
          if (p.has_out) *reinterpret_cast<uint4*>(p.out.at(f) + cell * ld + n_base + c) = make_uint4(0, 0, 0, 0);
          if (p.has_norm) *reinterpret_cast<uint4*>(p.out_norm.at(f) + cell * ld + n_base + c) = make_uint4(0, 0, 0, 0);
        }
      }
    }
    __syncwarp();
    // the rows that this lane stores: its pair's even and odd one (bits of `to`: copies in time, y and x; result
    // stored, norm stored, frame in the second tensor)
    const int lane = threadIdx.x & 31;
    const int info = dst.n_t | dst.n_y << 2 | dst.n_x << 4 | (row_ok && (inside || !p.keep_border) ? 64 : 0) | (row_ok ? 128 : 0) |
                     (dst.frame < p.out.split ? 0 : 256);
    const long long row0 = __shfl_sync(0xffffffffu, dst.row, lane & ~1), row1 = __shfl_sync(0xffffffffu, dst.row, lane | 1);
    const int to0 = __shfl_sync(0xffffffffu, info, lane & ~1), to1 = __shfl_sync(0xffffffffu, info, lane | 1);
    auto store = [&](bf16* o, const uint4& v, int to) {
      if (p.mode != CONV_OUT_UP) {
        *reinterpret_cast<uint4*>(o) = v;
      } else {
        for (int tt = 0; tt < (to & 3); ++tt)
          for (int yy = 0; yy < (to >> 2 & 3); ++yy)
            for (int xx = 0; xx < (to >> 4 & 3); ++xx) *reinterpret_cast<uint4*>(o + (tt * dst.st + yy * dst.sy + xx) * ld) = v;
      }
    };
    const bf16* res = p.has_resid ? p.resid.at(f) + ((long long)f * p.plane + rem) * ld + n_base : nullptr;
    static_assert(U == 2 || (U == 1 && NC != 64), "columns at a time");
    constexpr bool KEEP = NC == 64;   // the rounded values stay in registers until the row's norm is known; else in tensor memory
    // Squares are added per 8 channels (two such chains side by side) and these sums in the order of a warp's butterfly: groups
    // in bit-reversed order, summed like a binary counter.
    uint64_t lvl[3] = {0, 0, 0}, sum = 0;
    uint32_t pk[U][8];
    const int groups = (NC > 0 ? NC : n_end) >> 5;   // of 16 columns, of this warp; U at a time
#pragma unroll 1
    for (int i = 0; i < groups; i += U) {
      int c[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = i + u;
        c[u] = 32 * (NC == 256 ? ((j & 1) << 2 | (j & 2) | j >> 2) : NC == 128 ? ((j & 1) << 1 | j >> 1) : j) + 16 * half;
      }
      const bool two = U == 2 && (NC > 0 || i + 1 < groups);
      uint32_t v[U][16];
      uint4 ru[U][2];
      tmem_ld16(ta + c[0], v[0]);
      if (two) tmem_ld16(ta + c[U - 1], v[U - 1]);
      if (res && inside) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u == 0 || two) {
            ru[u][0] = reinterpret_cast<const uint4*>(res + c[u])[0];
            ru[u][1] = reinterpret_cast<const uint4*>(res + c[u])[1];
          }
      }
      tmem_wait_ld();
      if constexpr (ZERO) {
        tmem_st16(ta + c[0], zero16);
        if (two) tmem_st16(ta + c[U - 1], zero16);
      }
      if ((NC == 0 || KEEP) && i + U >= groups) {
        if constexpr (ZERO) tmem_wait_st();
        release();
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (u == 1 && !two) break;
        uint64_t a[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] = pack2(__uint_as_float(v[u][2 * k]), __uint_as_float(v[u][2 * k + 1]));
        if (bias) {
          const float4* b4 = reinterpret_cast<const float4*>(bias + n_base + c[u]);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 b = b4[k];
            a[2 * k] = add2(a[2 * k], pack2(b.x, b.y));
            a[2 * k + 1] = add2(a[2 * k + 1], pack2(b.z, b.w));
          }
        }
        if (res) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t w[4] = {ru[u][k].x, ru[u][k].y, ru[u][k].z, ru[u][k].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) a[4 * k + e] = add2(a[4 * k + e], pack2(bf16lo(w[e]), bf16hi(w[e])));
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float2 y2 = unpack2(a[k]);
          pk[u][k] = inside ? pack_bf16(y2.x, y2.y) : 0u;
        }
        if (p.has_out) {
          uint4 v0, v1;
          cv_swap_halves(pk[u], lane, v0, v1);
          const int col = n_base + c[u] + 8 * (lane & 1);
          if (to0 & 64) store((to0 & 256 ? p.out.tail : p.out.body) + row0 * ld + col, v0, to0);
          if (to1 & 64) store((to1 & 256 ? p.out.tail : p.out.body) + row1 * ld + col, v1, to1);
          __syncwarp();
        }
      }
      if constexpr (NC > 0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
          uint64_t q = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t lo = pack2(bf16lo(pk[u][k]), bf16lo(pk[u][4 + k])), hi = pack2(bf16hi(pk[u][k]), bf16hi(pk[u][4 + k]));
            q = fma2(lo, lo, q);
            q = fma2(hi, hi, q);
          }
          const int j = i + u;
          if (j & 1) {
            q = add2(lvl[0], q);
            if (j & 2) {
              q = add2(lvl[1], q);
              if (j & 4) q = add2(lvl[2], q); else lvl[2] = q;
            } else {
              lvl[1] = q;
            }
          } else {
            lvl[0] = q;
          }
          sum = q;
        }
        if constexpr (!KEEP) {
#pragma unroll
          for (int u = 0; u < U; ++u) tmem_st8(ta + c[u], pk[u]);   // in place of their accumulators
        }
      }
    }
    if constexpr (NC > 0) {
      // the other half's sums (two buffers: a warp is at most one meeting ahead of its partner)
      const float2 own = unpack2(sum);
      sums[half * 128] = own;
      if constexpr (!KEEP) tmem_wait_st();
      cv_meet(pair_id);
      const float2 other = sums[(half ^ 1) * 128];
      const float s0 = own.x + other.x, s1 = own.y + other.y;
      const float rneg = -rsqrtf((s0 + s1) / (float)NC + p.eps);
      const uint64_t rneg2 = pack2(rneg, rneg);
      bf16* const o0 = (to0 & 256 ? p.out_norm.tail : p.out_norm.body) + row0 * ld + 8 * (lane & 1);
      bf16* const o1 = (to1 & 256 ? p.out_norm.tail : p.out_norm.body) + row1 * ld + 8 * (lane & 1);
#pragma unroll 1
      for (int c = 16 * half; c < NC; c += 32 * U) {
        if constexpr (!KEEP) {
#pragma unroll
          for (int u = 0; u < U; ++u) tmem_ld8(ta + c + 32 * u, pk[u]);
          tmem_wait_ld();
          if (c + 32 * U >= NC) release();
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          uint32_t on[8];
          uint64_t zn[8];
          const float4* g4 = reinterpret_cast<const float4*>(gamma + c + 32 * u);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float4 g = g4[k];
            zn[2 * k] = mul2(mul2(pack2(bf16lo(pk[u][2 * k]), bf16hi(pk[u][2 * k])), rneg2), pack2(g.x, g.y));
            zn[2 * k + 1] = mul2(mul2(pack2(bf16lo(pk[u][2 * k + 1]), bf16hi(pk[u][2 * k + 1])), rneg2), pack2(g.z, g.w));
          }
          cv_silu16(zn, on);   // zero on the border
          uint4 v0, v1;
          cv_swap_halves(on, lane, v0, v1);
          if (to0 & 128) *reinterpret_cast<uint4*>(o0 + c + 32 * u) = v0;
          if (to1 & 128) *reinterpret_cast<uint4*>(o1 + c + 32 * u) = v1;
          __syncwarp();
        }
      }
    }
  }
}

// R row tiles per CTA; NC = channels of the fused norm (64, 128, 256) or 0.
template <int R, int NC>
__global__ void __launch_bounds__(ConvCfg<R>::THREADS, 1)
conv_kernel(const __grid_constant__ CUtensorMap tmCtx, const __grid_constant__ CUtensorMap tmBody,
            const __grid_constant__ CUtensorMap tmTail, const __grid_constant__ CUtensorMap tmSkip,
            const __grid_constant__ CUtensorMap tmSkipTail, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ ConvParams p) {
  using Cfg = ConvCfg<R>;
  constexpr int TILE_M = 256 * R;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int NA = p.na, NB = p.nb;
  const int b_slot = p.mma_n * 64;   // (mma_n / 2 rows) x 128 bytes
  const uint32_t b_base = smem_base + NA * Cfg::A_SLOT;
  const uint32_t bar_base = b_base + NB * b_slot;
  auto full_a = [&](int s) { return bar_base + 8u * s; };
  auto empty_a = [&](int s) { return bar_base + 8u * (NA + s); };
  auto full_b = [&](int s) { return bar_base + 8u * (2 * NA + s); };
  auto empty_b = [&](int s) { return bar_base + 8u * (2 * NA + NB + s); };
  const uint32_t t_base = bar_base + 16u * (NA + NB);
  auto tfull = [&](int b) { return t_base + 8u * b; };
  auto tempty = [&](int b) { return t_base + 16u + 8u * b; };
  const uint32_t tmem_slot = t_base + 32u;
  uint8_t* gen = smem_raw + (tmem_slot - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gen);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + 8);
  float2* row_sums = reinterpret_cast<float2*>(smem_raw + (bar_base + CV_BARS - smem_u32(smem_raw)));
  float* gamma = reinterpret_cast<float*>(row_sums) + CV_SUMS / 4;

  const uint32_t rank = cluster_ctarank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int total = p.n_seg * p.tiles_per_seg * p.n_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NA; ++s) { mbar_init(full_a(s), 1); mbar_init(empty_a(s), 1); }
    for (int s = 0; s < NB; ++s) { mbar_init(full_b(s), 1); mbar_init(empty_b(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(tfull(b), 1); mbar_init(tempty(b), 16 * R); }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmBody);
    prefetch_tmap(&tmB);
  }
  if constexpr (NC > 0) {
    for (int c = threadIdx.x; c < NC; c += Cfg::THREADS) gamma[c] = __bfloat162float(p.gamma[c]);
  }
  if (p.n_tiles == 1)
    for (int c = threadIdx.x; c < p.n_out; c += Cfg::THREADS) gamma[CV_GAMMA / 4 + c] = p.bias ? p.bias[c] : 0.f;
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  if (warp == 0) {
    // ---------------- TMA producer of the activations, in the order in which the products consume them (the last warp brings
    // the weights: a thread's instructions for both take longer than a tap's products of 64 columns)
    const bool issuer = elect_one();
    int ia = 0;
    uint32_t pha = 0;
    bool ok = true;
    for (int t = first_tile; t < total && ok; t += tile_step) {
      const int mt = t / p.n_tiles;
      const int seg = mt / p.tiles_per_seg, tile = mt - seg * p.tiles_per_seg;
      const int local = tile * TILE_M + int(rank) * (128 * R), v0 = p.v_first + seg * p.v_step;
      for (int ph = 0; ph < 2 && ok; ++ph) {
        const int cblocks = ph ? p.skip_cblocks : p.cblocks;
        for (int c0 = 0; c0 < cblocks && ok; c0 += CV_CHUNK) {
          const int nc = min(CV_CHUNK, cblocks - c0);
          const int n_groups = ph ? 1 : p.n_groups;
          for (int g = 0; g < n_groups && ok; ++g) {
            ConvSource src;
            if (ph) {
              src = seg < p.skip_split ? ConvSource{&tmSkip, seg * p.frame_rows} : ConvSource{&tmSkipTail, (seg - p.skip_split) * p.frame_rows};
            } else {
              const int v = v0 + p.g[g].kt;
              if (v < 2 && !p.has_ctx) continue;
              src = conv_source(p, v, &tmCtx, &tmBody, &tmTail);
              src.row += p.g[g].off;
            }
            const int y = src.row + local;
            for (int c = 0; c < nc; ++c) {
              if (!__all_sync(0xffffffffu, mbar_wait(empty_a(ia), pha ^ 1, abort_flag, p.status, ST_TIMEOUT_TMA))) { ok = false; break; }
              if (issuer) {
                if (rank == 0) mbar_arrive_expect_tx(full_a(ia), 2 * Cfg::A_SLOT);
                const uint32_t fb = mapa(full_a(ia), 0);
                const uint32_t dst = smem_base + ia * Cfg::A_SLOT;
#pragma unroll
                for (int r = 0; r < Cfg::BOXES; ++r)
                  tma_load_2d_pair(dst + r * Cfg::BOX * 128, src.map, fb, (c0 + c) * 64, y + r * Cfg::BOX);
              }
              __syncwarp();
              if (++ia == NA) { ia = 0; pha ^= 1; }
            }
          }
        }
      }
    }
    if (!ok && issuer) {
      // copies in flight are counted on the leader's barriers: give them a fixed time, far beyond a copy's latency
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000ll) {}
    }
    __syncwarp();
  } else if (warp == Cfg::THREADS / 32 - 1) {
    // ---------------- TMA producer of the weights
    const bool issuer = elect_one();
    int ib = 0;
    uint32_t phb = 0;
    bool ok = true;
    for (int t = first_tile; t < total && ok; t += tile_step) {
      const int y = (t % p.n_tiles) * 256 + int(rank) * (p.mma_n >> 1);
      const int v0 = p.v_first + t / p.n_tiles / p.tiles_per_seg * p.v_step;
      for (int ph = 0; ph < 2 && ok; ++ph) {
        const int cblocks = ph ? p.skip_cblocks : p.cblocks;
        for (int c0 = 0; c0 < cblocks && ok; c0 += CV_CHUNK) {
          const int nc = min(CV_CHUNK, cblocks - c0);
          const int n_groups = ph ? 1 : p.n_groups;
          for (int g = 0; g < n_groups && ok; ++g) {
            if (!ph && v0 + p.g[g].kt < 2 && !p.has_ctx) continue;
            const int n_taps = ph ? 1 : p.g[g].n_taps;
            for (int i = 0; i < n_taps && ok; ++i) {
              const int x = (ph ? p.skip_kcol : p.g[g].tap[i] * cblocks * 64) + c0 * 64;
              for (int c = 0; c < nc; ++c) {
                if (!__all_sync(0xffffffffu, mbar_wait(empty_b(ib), phb ^ 1, abort_flag, p.status, ST_TIMEOUT_TMA))) { ok = false; break; }
                if (issuer) {
                  if (rank == 0) mbar_arrive_expect_tx(full_b(ib), 2 * b_slot);
                  tma_load_2d_pair(b_base + ib * b_slot, &tmB, mapa(full_b(ib), 0), x + c * 64, y);
                }
                __syncwarp();
                if (++ib == NB) { ib = 0; phb ^= 1; }
              }
            }
          }
        }
      }
    }
    if (!ok && issuer) {
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000ll) {}
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      // ---------------- MMA issuer (the whole warp walks the loop, one elected lane issues)
      const uint32_t idesc = make_idesc_bf16(256, p.mma_n, 0, 0);
      int ia0 = 0, ib = 0, tcount = 0;
      uint32_t pha0 = 0, phb = 0;
      bool ok = true;
      for (int t = first_tile; t < total && ok; t += tile_step, ++tcount) {
        const int buf = tcount & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(tempty(buf), ((tcount >> 1) & 1) ^ 1, abort_flag, p.status, ST_TIMEOUT_MMA))) break;
        tc_fence_after();
        const uint32_t d = tmem_base + buf * 256;
        const int v0 = p.v_first + t / p.n_tiles / p.tiles_per_seg * p.v_step;
        uint32_t acc = 0;
        for (int ph = 0; ph < 2 && ok; ++ph) {
          const int cblocks = ph ? p.skip_cblocks : p.cblocks;
          for (int c0 = 0; c0 < cblocks && ok; c0 += CV_CHUNK) {
            const int nc = min(CV_CHUNK, cblocks - c0);
            const int n_groups = ph ? 1 : p.n_groups;
            for (int g = 0; g < n_groups && ok; ++g) {
              if (!ph && v0 + p.g[g].kt < 2 && !p.has_ctx) continue;
              const int n_taps = ph ? 1 : p.g[g].n_taps;
              int ia = ia0;
              uint32_t pha = pha0;
              for (int i = 0; i < n_taps && ok; ++i) {
                const int shift = ph ? 0 : p.g[g].shift[i];
                ia = ia0;
                pha = pha0;
                for (int c = 0; c < nc; ++c) {
                  if (i == 0 && !__all_sync(0xffffffffu, mbar_wait(full_a(ia), pha, abort_flag, p.status, ST_TIMEOUT_MMA))) { ok = false; break; }
                  if (!__all_sync(0xffffffffu, mbar_wait(full_b(ib), phb, abort_flag, p.status, ST_TIMEOUT_MMA))) { ok = false; break; }
                  tc_fence_after();
                  const uint64_t bdesc = make_smem_desc_sw128(b_base + ib * b_slot, 16, 1024);
                  const uint32_t sa = smem_base + ia * Cfg::A_SLOT + shift * 128;
                  if (elect_one()) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                      const uint64_t adesc = make_smem_desc_sw128(sa + r * 16384, 16, 1024);
#pragma unroll
                      for (int k = 0; k < 4; ++k)
                        mma_ss_pair(d + r * Cfg::ACC_COLS, adesc + 2 * k, bdesc + 2 * k, idesc, (acc | k) ? 1u : 0u);
                    }
                    tc_commit_pair(empty_b(ib));
                    tc_commit_pair(mapa(empty_b(ib), 1));
                    if (i == n_taps - 1) {
                      tc_commit_pair(empty_a(ia));
                      tc_commit_pair(mapa(empty_a(ia), 1));
                    }
                  }
                  __syncwarp();
                  acc = 1;
                  if (++ib == NB) { ib = 0; phb ^= 1; }
                  if (++ia == NA) { ia = 0; pha ^= 1; }
                }
              }
              ia0 = ia;
              pha0 = pha;
            }
          }
        }
        if (ok) {
          if (elect_one()) {
            tc_commit_pair(tfull(buf));
            tc_commit_pair(mapa(tfull(buf), 1));
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ---------------- epilogue: eight warps per row tile; tensor-memory lane quadrant = warp % 4, and the two warps of a
    // quadrant take every other group of 16 columns. The loops over these groups stay rolled: unrolled over 256 columns the
    // code left the instruction cache and a tile took 67 us. Latency bounds what is left (the chain of the SiLU most of all,
    // though its quotient takes no division, cv_silu2), hence the number of warps.
    const int quad = warp & 3, half = ((warp - 2) >> 2) & 1, r = (warp - 2) >> 3;
    const int pair_id = 1 + r * 4 + quad;
    const float* bias = p.n_tiles == 1 ? gamma + CV_GAMMA / 4 : p.bias;
    int tcount = 0;
    bool alive = true;
    for (int t = first_tile; t < total; t += tile_step, ++tcount) {
      const int buf = tcount & 1;
      const int nt = t % p.n_tiles, mt = t / p.n_tiles;
      const int seg = mt / p.tiles_per_seg, tile = mt - seg * p.tiles_per_seg;
      const int q = tile * TILE_M + int(rank) * (128 * R) + r * 128 + quad * 32 + lane;
      const uint32_t ta = tmem_base + (uint32_t(quad * 32) << 16) + buf * 256 + r * Cfg::ACC_COLS;
      const bool row_ok = q < p.seg_rows;
      const int y = q / p.pw, x = q - y * p.pw;
      alive = mbar_wait(tfull(buf), (tcount >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_EPI) && alive;
      __syncwarp();
      tc_fence_after();
      conv_emit<NC, false, false, R == 1 || NC == 64 ? 2 : 1>(p, ta, seg, q, y, x, row_ok && alive, nt * 256, half, pair_id,
                                  row_sums + (buf * 2 + r) * 256 + quad * 32 + lane, gamma, bias, [&] {
                                    tc_fence_before();
                                    __syncwarp();
                                    if (lane == 0) {
                                      if (rank != 0) mbar_arrive_peer(mapa(tempty(buf), 0));
                                      else mbar_arrive(tempty(buf));
                                    }
                                  });
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Convolutions with at most 64 output channels: a CTA pair walks its 512 positions through time, and one product of up to
// 3 x 64 columns adds an input frame's tap to the three output frames that the frame belongs to (temporal taps side by side along
// N). With 64 columns a product is bound by the reads of its A operand from shared memory (32 clocks for 32 of MMA, and a
// fresh A three times), and a frame's activations crossed L2 -> shared memory for each temporal tap; here every activation tile
// crosses 3 times and not 9, and its reads are shared by 192 columns (96 clocks).
// A ring of four accumulators per row tile: three frames being summed, one being drained. The epilogue leaves a drained
// accumulator zero, so that every product accumulates. Where the ring wraps, the frames' columns are not contiguous and a
// tap takes two products.
// 480p, 8 frames, us, against the flattened walk of conv_kernel on one box: 128 -> 64 channels 1648 -> 908 (1.55 PFLOP/s), pixels
// 1000 -> 300, first layer (epilogue-bound) 555 -> 397. One thread's instructions for both operands and a barrier for every tap took
// 850 clocks a tap, whatever the products (pixels 455 us with the same walk); hence two producer threads and one stage for the three
// taps of a filter row (249 us).
constexpr int CT_SLOTS = 4;
constexpr int CT_THREADS = ConvCfg<2>::THREADS;
__host__ __device__ constexpr int ct_stage(int nt) { return ConvCfg<2>::A_SLOT + 9 * nt * 64; }
template <int NC, bool RGB>
__global__ void __launch_bounds__(CT_THREADS, 1)
conv_time_kernel(const __grid_constant__ CUtensorMap tmCtx, const __grid_constant__ CUtensorMap tmBody,
                 const __grid_constant__ CUtensorMap tmTail, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ ConvParams p) {
  using Cfg = ConvCfg<2>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int NS = p.na;
  const int piece = p.nt * 64;        // half of a frame's columns: (nt / 2 rows) x 128 bytes
  const int stage = ct_stage(p.nt);   // activations, and a CTA's half of the weights of three taps for three frames
  const uint32_t bar_base = smem_base + NS * stage;
  auto full = [&](int s) { return bar_base + 8u * s; };
  auto empty = [&](int s) { return bar_base + 8u * (NS + s); };
  const uint32_t t_base = bar_base + 16u * NS;
  auto tfull = [&](int b) { return t_base + 8u * b; };
  auto tempty = [&](int b) { return t_base + 8u * (CT_SLOTS + b); };
  const uint32_t tmem_slot = t_base + 16u * CT_SLOTS;
  uint8_t* gen = smem_raw + (tmem_slot - smem_u32(smem_raw));
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(gen);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + 8);
  float2* row_sums = reinterpret_cast<float2*>(smem_raw + (bar_base + CV_BARS - smem_u32(smem_raw)));
  float* gamma = reinterpret_cast<float*>(row_sums) + CV_SUMS / 4;

  const uint32_t rank = cluster_ctarank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
  const int total = p.n_seg * p.tiles_per_seg;
  const int n_taps = p.g[0].n_taps;   // of every group: the three columns of a filter row, or one

  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(full(s), 2); mbar_init(empty(s), 1); }   // two producers
    for (int b = 0; b < CT_SLOTS; ++b) { mbar_init(tfull(b), 1); mbar_init(tempty(b), 32); }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmBody);
    prefetch_tmap(&tmB);
  }
  if constexpr (NC > 0) {
    for (int c = threadIdx.x; c < NC; c += CT_THREADS) gamma[c] = __bfloat162float(p.gamma[c]);
  }
  for (int c = threadIdx.x; c < min(p.n_out, 64); c += CT_THREADS) gamma[CV_GAMMA / 4 + c] = p.bias && (!RGB || c < 3) ? p.bias[c] : 0.f;
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;

  // Output frames lo .. lo + n - 1 take part in the products of input frame `i`, counted from the first context frame (output frame
  // i - k by tap k of time);
  // n1 of them up to the end of the ring. `base`: frames that this pair has begun in earlier tiles.
  struct Step { int lo, n, n1, slot; };
  auto step_of = [&](int i, int j0, int j1, int base) {
    Step st;
    st.lo = max(j0, i - 2);
    st.n = min(j1 - 1, i) - st.lo + 1;
    st.slot = (base + st.lo - j0) & (CT_SLOTS - 1);
    st.n1 = min(st.n, CT_SLOTS - st.slot);
    return st;
  };

  if (warp == 0) {
    // ---------------- TMA producer of the activations (the last warp brings the weights: one thread's instructions for both took
    // about 850 clocks a tap, more than its products)
    const bool issuer = elect_one();
    int ia = 0;
    uint32_t pha = 0;
    bool ok = true;
    for (int t = first_tile; t < total && ok; t += tile_step) {
      const int seg = t / p.tiles_per_seg, tile = t - seg * p.tiles_per_seg;
      const int j0 = seg * p.seg_frames, j1 = min(j0 + p.seg_frames, p.f_out);
      const int local = tile * 512 + int(rank) * 256;
      for (int i = p.has_ctx ? j0 : max(j0, 2); i < j1 + 2 && ok; ++i) {
        const ConvSource src = conv_source(p, i, &tmCtx, &tmBody, &tmTail);
        for (int g = 0; g < p.n_groups && ok; ++g) {
          const int y = src.row + local + p.g[0].off + g * p.pw;
          for (int c = 0; c < p.cblocks; ++c) {
            if (!__all_sync(0xffffffffu, mbar_wait(empty(ia), pha ^ 1, abort_flag, p.status, ST_TIMEOUT_TMA))) { ok = false; break; }
            if (issuer) {
              if (rank == 0) mbar_arrive_expect_tx(full(ia), 2 * Cfg::A_SLOT);
              const uint32_t fa = mapa(full(ia), 0);
              const uint32_t dst = smem_base + ia * stage;
#pragma unroll
              for (int r = 0; r < Cfg::BOXES; ++r)
                tma_load_2d_pair(dst + r * Cfg::BOX * 128, src.map, fa, c * 64, y + r * Cfg::BOX);
            }
            __syncwarp();
            if (++ia == NS) { ia = 0; pha ^= 1; }
          }
        }
      }
    }
    if (!ok && issuer) {
      // copies in flight are counted on the leader's barriers: give them a fixed time, far beyond a copy's latency
      const long long t0 = clock64();
      while (clock64() - t0 < 2000000ll) {}
    }
    __syncwarp();
  } else if (warp == CT_THREADS / 32 - 1) {
    if (lane == 0) {
      // ---------------- TMA producer of the weights
      int ib = 0, base = 0;
      uint32_t phb = 0;
      bool ok = true;
      const int c_in = p.cblocks * 64;
      for (int t = first_tile; t < total && ok; t += tile_step) {
        const int seg = t / p.tiles_per_seg;
        const int j0 = seg * p.seg_frames, j1 = min(j0 + p.seg_frames, p.f_out);
        for (int i = p.has_ctx ? j0 : max(j0, 2); i < j1 + 2 && ok; ++i) {
          const Step st = step_of(i, j0, j1, base);
          // a product of n frames has 2 n pieces along N, of which the even CTA holds the first n
          int x[3], y[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const int first = k < st.n1 ? 0 : st.n1, len = k < st.n1 ? st.n1 : st.n - st.n1;
            const int q = (k - first) + int(rank) * len;           // piece of this product
            const int kt = i - (st.lo + first + (q >> 1));         // tap of time of the piece's frame: i = frame + kt
            x[k] = kt * p.kt_taps * c_in;
            y[k] = (q & 1) * (p.nt >> 1);
          }
          for (int g = 0; g < p.n_groups && ok; ++g) {
            for (int c = 0; c < p.cblocks && ok; ++c) {
              if (!mbar_wait(empty(ib), phb ^ 1, abort_flag, p.status, ST_TIMEOUT_TMA)) { ok = false; break; }
              if (rank == 0) mbar_arrive_expect_tx(full(ib), 2 * n_taps * st.n * piece);
              const uint32_t fb = mapa(full(ib), 0);
              uint32_t to = smem_base + ib * stage + Cfg::A_SLOT;
              int col = g * n_taps * c_in + c * 64;
              for (int w = 0; w < n_taps; ++w, col += c_in, to += 3 * piece) {
                tma_load_2d_pair(to, &tmB, fb, x[0] + col, y[0]);
                if (st.n > 1) tma_load_2d_pair(to + piece, &tmB, fb, x[1] + col, y[1]);
                if (st.n > 2) tma_load_2d_pair(to + 2 * piece, &tmB, fb, x[2] + col, y[2]);
              }
              if (++ib == NS) { ib = 0; phb ^= 1; }
            }
          }
        }
        base += j1 - j0;
      }
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) {}
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---------------- MMA issuer (the whole warp walks the loop, one elected lane issues)
      int ia = 0, base = 0;
      uint32_t pha = 0;
      bool ok = true;
      for (int t = first_tile; t < total && ok; t += tile_step) {
        const int seg = t / p.tiles_per_seg;
        const int j0 = seg * p.seg_frames, j1 = min(j0 + p.seg_frames, p.f_out);
        for (int i = j0; i < j1 + 2 && ok; ++i) {
          const Step st = step_of(i, j0, j1, base);
          if (i < j1) {   // a new frame: its accumulator is drained and zero
            const int n = base + i - j0;
            if (!__all_sync(0xffffffffu, mbar_wait(tempty(n & (CT_SLOTS - 1)), (n / CT_SLOTS) & 1, abort_flag, p.status, ST_TIMEOUT_MMA))) {
              ok = false;
              break;
            }
            tc_fence_after();
          }
          const int n2 = st.n - st.n1;
          const uint32_t idesc1 = make_idesc_bf16(256, st.n1 * p.nt, 0, 0), idesc2 = make_idesc_bf16(256, n2 * p.nt, 0, 0);
          const int n_groups = i < 2 && !p.has_ctx ? 0 : p.n_groups;   // no frame there
          for (int g = 0; g < n_groups && ok; ++g) {
            for (int c = 0; c < p.cblocks && ok; ++c) {
              if (!__all_sync(0xffffffffu, mbar_wait(full(ia), pha, abort_flag, p.status, ST_TIMEOUT_MMA))) { ok = false; break; }
              tc_fence_after();
              if (elect_one()) {
                const uint32_t sa = smem_base + ia * stage;
                uint64_t a = make_smem_desc_sw128(sa, 16, 1024), b1 = make_smem_desc_sw128(sa + Cfg::A_SLOT, 16, 1024);
                for (int w = 0; w < n_taps; ++w) {   // a tap further: a row of the activations, three pieces of the weights
#pragma unroll
                  for (int r = 0; r < 2; ++r) {
                    const uint32_t d = tmem_base + r * CT_SLOTS * p.nt;
#pragma unroll
                    for (int k = 0; k < 4; ++k) mma_ss_pair(d + st.slot * p.nt, a + r * 1024 + 2 * k, b1 + 2 * k, idesc1, 1u);
                    if (n2 > 0) {
                      const uint64_t b2 = b1 + (st.n1 * piece >> 4);
#pragma unroll
                      for (int k = 0; k < 4; ++k) mma_ss_pair(d, a + r * 1024 + 2 * k, b2 + 2 * k, idesc2, 1u);
                    }
                  }
                  a += 8;
                  b1 += 3 * piece >> 4;
                }
                tc_commit_both(empty(ia));
              }
              __syncwarp();
              if (++ia == NS) { ia = 0; pha ^= 1; }
            }
          }
          if (ok && i - 2 >= j0) {
            if (elect_one()) tc_commit_both(tfull((base + i - 2 - j0) & (CT_SLOTS - 1)));
            __syncwarp();
          }
        }
        base += j1 - j0;
      }
    }
  } else {
    // ---------------- epilogue (as in conv_kernel)
    const int quad = warp & 3, half = ((warp - 2) >> 2) & 1, r = (warp - 2) >> 3;
    const int pair_id = 1 + r * 4 + quad;
    const uint32_t mine = tmem_base + (uint32_t(quad * 32) << 16) + r * CT_SLOTS * p.nt;
    auto hand_back = [&](int slot) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (rank != 0) mbar_arrive_peer(mapa(tempty(slot), 0));
        else mbar_arrive(tempty(slot));
      }
    };
    {
      const uint32_t zero16[16] = {};
      for (int c = 16 * half; c < CT_SLOTS * p.nt; c += 32) tmem_st16(mine + c, zero16);
      tmem_wait_st();
      for (int slot = 0; slot < CT_SLOTS; ++slot) hand_back(slot);
    }
    int n = 0;
    bool alive = true;
    for (int t = first_tile; t < total; t += tile_step) {
      const int seg = t / p.tiles_per_seg, tile = t - seg * p.tiles_per_seg;
      const int rem = tile * 512 + int(rank) * 256 + r * 128 + quad * 32 + lane;
      const bool row_ok = rem < p.plane;
      const int y = rem / p.pw, x = rem - y * p.pw;
      const int j0 = seg * p.seg_frames, j1 = min(j0 + p.seg_frames, p.f_out);
      for (int j = j0; j < j1; ++j, ++n) {
        const int slot = n & (CT_SLOTS - 1);
        alive = mbar_wait(tfull(slot), (n / CT_SLOTS) & 1, abort_flag, p.status, ST_TIMEOUT_EPI) && alive;
        __syncwarp();
        tc_fence_after();
        conv_emit<NC, RGB, true, 2>(p, mine + slot * p.nt, j, rem, y, x, row_ok && alive, 0, half, pair_id,
                                 row_sums + ((n & 1) * 2 + r) * 256 + quad * 32 + lane, gamma, gamma + CV_GAMMA / 4,
                                 [&] { hand_back(slot); });
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// First layer of the encoder: 3 channels would fill 3 of 64 columns of every operand row. dst[f, y, x, (kh * 3 + kw) * 3 + c] =
// src[c, f, y + kh - 1, x + kw - 1] (zero outside) for interior positions, channels 27 .. 63 zero: the spatial taps become
// channels and three taps in time are left. Bound by its writes (128 B a position).
template <typename T>
__global__ void __launch_bounds__(256)
conv_pack_rgb_kernel(const T* __restrict__ src, long long c_stride, uint4* __restrict__ dst, int n, int h, int w) {
  const long long total = (long long)n * (h + 2) * (w + 2);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int x = (int)(i % (w + 2));
    const int y = (int)(i / (w + 2) % (h + 2));
    const int f = (int)(i / ((long long)(w + 2) * (h + 2)));
    float v[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = 0.f;
    if (x >= 1 && x <= w && y >= 1 && y <= h) {
#pragma unroll
      for (int kh = 0; kh < 3; ++kh)
#pragma unroll
        for (int kw = 0; kw < 3; ++kw) {
          const int yy = y + kh - 2, xx = x + kw - 2;   // unpadded coordinates
          if (yy >= 0 && yy < h && xx >= 0 && xx < w)
#pragma unroll
            for (int c = 0; c < 3; ++c)
              v[(kh * 3 + kw) * 3 + c] = (float)src[c * c_stride + ((long long)f * h + yy) * w + xx];
        }
    }
    uint4* o = dst + i * 8;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      o[k] = make_uint4(pack_bf16(v[8 * k], v[8 * k + 1]), pack_bf16(v[8 * k + 2], v[8 * k + 3]),
                        pack_bf16(v[8 * k + 4], v[8 * k + 5]), pack_bf16(v[8 * k + 6], v[8 * k + 7]));
#pragma unroll
    for (int k = 4; k < 8; ++k) o[k] = make_uint4(0, 0, 0, 0);
  }
}

// Values with the bit patterns first .. first + 16 n - 1 against the division: [0] how many results differ in bf16, [1] in fp32 where
// no value of 80 or more takes the division, [2] by how many spacings of fp32 at most.
__global__ void __launch_bounds__(256)
conv_silu_selftest_kernel(uint32_t first, long long n, unsigned long long* differ) {
  unsigned long long bad16 = 0, bad32 = 0, far = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    uint64_t zn[8];
    uint32_t o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t g = first + (uint32_t)(i * 16) + 2 * k;
      zn[k] = pack2(-__uint_as_float(g), -__uint_as_float(g + 1));
    }
    cv_silu16(zn, o);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float2 z = unpack2(zn[k]), y = cv_silu2(zn[k]);
      const float got[2] = {y.x, y.y}, neg[2] = {z.x, z.y};
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float want = -neg[e] / (1.f + __expf(neg[e])), stored = e ? bf16hi(o[k]) : bf16lo(o[k]);
        const float rounded = bf16lo(pack_bf16(want, 0.f));
        bad16 += stored != rounded && !(isnan(stored) && isnan(rounded));
        if (fabsf(neg[e]) < 80.f && got[e] != want) {
          ++bad32;
          const long long d = llabs((long long)__float_as_int(got[e]) - __float_as_int(want));
          far = max(far, (unsigned long long)d);
        }
      }
    }
  }
  if (bad16) atomicAdd(differ, bad16);
  if (bad32) {
    atomicAdd(differ + 1, bad32);
    atomicMax(differ + 2, far);
  }
}

}  // namespace cb

// ====================================================================== host
namespace cosmos {

namespace {

CUtensorMap rows_map(const void* base, long long rows, int c, int box_rows) {
  const uint64_t dims[2] = {(uint64_t)c, (uint64_t)rows};
  const uint64_t str[1] = {(uint64_t)c * 2};
  const uint32_t box[2] = {64, (uint32_t)box_rows};
  return cbh::make_tmap_bf16(base, 2, dims, str, box, true);
}

// CTA pairs of `kern` that the GPU holds at once, with one CTA an SM; the kernel's shared-memory limit is raised on the way.
template <typename K>
int conv_pairs(K kern, cudaLaunchConfig_t cfg) {
  int dev = 0, sms = 148, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cb::CV_SMEM_MAX);
  cfg.gridDim = dim3(sms & ~1);
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = sms / 2;
  }
  return std::min(n, sms / 2);
}

struct ConvLaunch {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  ConvLaunch(int threads, cudaStream_t s) {
    cfg.blockDim = dim3(threads);
    // always the whole shared memory: a second CTA on the SM would wait for tensor memory that the first one holds
    cfg.dynamicSmemBytes = cb::CV_SMEM_MAX;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cfg.stream = s;
  }
  ConvLaunch(const ConvLaunch&) = delete;
};

int pairs_allowed(int pairs) {
  const int limit = gemm_grid_limit();
  return limit > 0 ? std::min(pairs, std::max(1, limit / 2)) : pairs;
}

void conv_check(cudaError_t e) {
  if (e != cudaSuccess) throw std::runtime_error(std::string("conv: launch failed: ") + cudaGetErrorString(e));
}

template <int R, int NC>
void conv_launch(const CUtensorMap (&maps)[6], const cb::ConvParams& p, cudaStream_t s) {
  auto kern = cb::conv_kernel<R, NC>;
  static int pairs = 0;   // of this kernel
  ConvLaunch l(cb::ConvCfg<R>::THREADS, s);
  if (pairs == 0) pairs = conv_pairs(kern, l.cfg);
  l.cfg.gridDim = dim3(2 * std::min(pairs_allowed(pairs), p.n_seg * p.tiles_per_seg * p.n_tiles));
  conv_check(cudaLaunchKernelEx(&l.cfg, kern, maps[0], maps[1], maps[2], maps[3], maps[4], maps[5], p));
}

// The chunk's frames are cut into time segments where whole columns of frames would leave pairs idle: each cut costs two input
// frames more. Clocks of a segment: products (40 is what the reads of A take), or the epilogue's about 4000 a frame.
void pick_segments(cb::ConvParams& p, int pairs) {
  long long best = 0;
  for (int n_seg = 1; n_seg <= p.f_out; ++n_seg) {
    const int frames = (p.f_out + n_seg - 1) / n_seg;
    if (n_seg > 1 && frames == p.seg_frames) continue;
    long long mma = 0;
    for (int i = 0; i < frames + 2; ++i) {
      const int act = std::min(frames - 1, i) - std::max(0, i - 2) + 1;
      mma += std::max(40, act * p.nt / 2) * 8ll * p.n_groups * p.g[0].n_taps * p.cblocks;
    }
    const int segs = (p.f_out + frames - 1) / frames;
    const long long rounds = ((long long)segs * p.tiles_per_seg + pairs - 1) / pairs;
    const long long cost = rounds * std::max(mma, frames * 4000ll);
    if (n_seg == 1 || cost < best) {
      best = cost;
      p.n_seg = segs;
      p.seg_frames = frames;
    }
  }
}

template <int NC, bool RGB>
void conv_time_launch(const CUtensorMap (&maps)[6], cb::ConvParams p, cudaStream_t s) {
  auto kern = cb::conv_time_kernel<NC, RGB>;
  static int pairs = 0;
  ConvLaunch l(cb::CT_THREADS, s);
  if (pairs == 0) pairs = conv_pairs(kern, l.cfg);
  const int at_once = pairs_allowed(pairs);
  pick_segments(p, at_once);
  l.cfg.gridDim = dim3(2 * std::min(at_once, p.n_seg * p.tiles_per_seg));
  conv_check(cudaLaunchKernelEx(&l.cfg, kern, maps[0], maps[1], maps[2], maps[5], p));
}

template <int R>
void conv_dispatch(const CUtensorMap (&maps)[6], const cb::ConvParams& p, cudaStream_t s) {
  if (!p.has_norm) return conv_launch<R, 0>(maps, p, s);
  if constexpr (R == 2) {
    if (p.n_out == 64) return conv_launch<2, 64>(maps, p, s);
    if (p.n_out == 128) return conv_launch<2, 128>(maps, p, s);
  } else {
    if (p.n_out == 256) return conv_launch<1, 256>(maps, p, s);
  }
  throw std::runtime_error("conv: the fused norm takes 64, 128 or 256 channels");
}

}  // namespace

namespace {

// A volume of `frames` frames of `elems` elements: all of them at `body`, or the last two (one of one, then the second) at `tail`.
template <typename P>
cb::Split<P> split_of(const void* body, const void* tail, int frames, long long elems) {
  cb::Split<P> r;
  r.split = tail ? frames - 2 : frames;
  r.body = reinterpret_cast<P>(reinterpret_cast<uintptr_t>(body));
  r.tail = reinterpret_cast<P>(reinterpret_cast<uintptr_t>(tail) - (uintptr_t)(2 * elems * r.split));
  return r;
}

}  // namespace

void conv3d_fused(const ConvArgs& a, cudaStream_t s) {
  const bool strided = a.mode == CONV_OUT_DOWN, rgb = a.rgb != nullptr;
  const bool has_out = a.out || a.out_tail, has_norm = a.out_norm || a.out_norm_tail, has_skip = a.skip || a.skip_tail;
  const bool has_resid = a.resid || a.resid_tail;
  if (a.c <= 0 || a.c % 64 || a.skip_c % 64 || a.hp < 3 || a.wp < 3 || (!rgb && (a.n_out <= 0 || a.n_out % 32)))
    throw std::runtime_error("conv: needs input channels % 64 == 0, output channels % 32 == 0 and a padded volume");
  if ((strided || a.mode == CONV_OUT_S2D) && (a.hp % 2 || a.wp % 2)) throw std::runtime_error("conv: stride 2 needs even padded sizes");
  if (rgb ? a.n_out != 9 : (!has_out && !has_norm)) throw std::runtime_error("conv: nothing to write");
  if ((has_skip && (strided || a.mode == CONV_OUT_UP)) || (has_resid && (strided || rgb)))
    throw std::runtime_error("conv: no residual or skip input in this form");
  if (has_norm && (a.mode == CONV_OUT_S2D || a.mode == CONV_OUT_UP)) throw std::runtime_error("conv: no norm in this form");
  if (a.keep_border && (a.mode != CONV_OUT_SAME || has_norm || rgb)) throw std::runtime_error("conv: this form writes its border");
  if (a.f_out < 1) return;
  cb::ConvParams p{};
  p.cblocks = a.c / 64;
  p.n_out = a.n_out;
  p.n_tiles = (a.n_out + 255) / 256;
  p.mma_n = p.n_tiles > 1 ? 256 : (a.n_out + 15) / 16 * 16;
  p.bias = a.bias;
  const long long plane = (long long)a.hp * a.wp, sub = (long long)(a.hp / 2) * (a.wp / 2);
  if ((a.frames + 1) * plane > 0x7fffffffll) throw std::runtime_error("conv: volume too large for 32-bit row indices; use shorter chunks");
  int f_dst = a.f_out;
  long long dst_rows = plane;
  if (a.mode == CONV_OUT_UP) {
    f_dst = a.up_temporal ? 2 * a.f_out - (a.up_first ? 1 : 0) : a.f_out;
    dst_rows = (2ll * (a.hp - 2) + 2) * (2ll * (a.wp - 2) + 2);
  } else if (strided) {
    dst_rows = (a.hp / 2 + 1ll) * (a.wp / 2 + 1ll);
  }
  p.has_out = has_out;
  p.has_norm = has_norm;
  p.has_resid = has_resid;
  p.resid = split_of<const bf16*>(a.resid, a.resid_tail, a.frames, plane * a.n_out);
  p.out = split_of<bf16*>(a.out, a.out_tail, f_dst, dst_rows * a.n_out);
  p.out_norm = split_of<bf16*>(a.out_norm, a.out_norm_tail, f_dst, dst_rows * a.n_out);
  // one frame index decides for both outputs
  if (has_out && has_norm && p.out.split != p.out_norm.split) throw std::runtime_error("conv: outputs split in different ways");
  if (!has_out) p.out.split = p.out_norm.split;
  p.gamma = reinterpret_cast<const bf16*>(a.gamma);
  p.eps = a.eps;
  p.rgb = reinterpret_cast<uint8_t*>(a.rgb);
  p.mode = a.mode;
  p.keep_border = a.keep_border;
  p.f_out = a.f_out;
  p.up_t = a.up_temporal;
  p.up_first = a.up_first;
  p.status = a.status;
  p.frame_rows = (int)plane;
  p.has_ctx = a.ctx != nullptr;
  p.x_split = a.x_tail ? a.frames - 2 : a.frames;
  p.skip_split = a.skip_tail ? a.frames - 2 : a.frames;
  p.n_seg = a.f_out;
  p.v_step = 1;
  const int k_cols = (a.taps_t_only ? 3 : 27) * a.c + a.skip_c;
  // two row tiles share a weight tile where tensor memory holds two double-buffered accumulators
  const int R = p.mma_n <= 128 ? 2 : 1, box = cb::cv_box_rows(R);
  CUtensorMap maps[6];
  // a volume whose frames are all in one of its tensors has that one's map twice
  auto volume = [&](CUtensorMap& body, CUtensorMap& tail, const void* x, const void* t, int c) {
    const int n = t ? a.frames - 2 : a.frames;
    if (t) tail = rows_map(t, 2 * plane, c, box);
    body = n > 0 ? rows_map(x, n * plane, c, box) : tail;
    if (!t) tail = body;
  };
  volume(maps[1], maps[2], a.x, a.x_tail, a.c);
  maps[0] = a.ctx ? rows_map(a.ctx, 2 * plane, a.c, box) : maps[1];
  if (has_skip) volume(maps[3], maps[4], a.skip, a.skip_tail, a.skip_c);
  else maps[3] = maps[4] = maps[1];
  const int stage_max = cb::CV_SMEM_MAX - 1024 - cb::CV_TAIL;
  if (!strided) {
    p.seg_rows = (int)plane;
    p.plane = (int)plane;
    p.pw = a.wp; p.hp = a.hp; p.wp = a.wp;
  } else {
    // segment = kept frame; the kept position (j, i) of a frame sits at padded (2 j + kh, 2 i + kw) for tap (kh, kw)
    p.v_first = a.t_first;
    p.v_step = a.t_step;
    p.seg_rows = (int)sub;
    p.plane = (int)sub;
    p.pw = a.wp / 2; p.hp = a.hp / 2; p.wp = a.wp / 2;
  }
  if (!strided && !has_skip && a.n_out <= 64) {
    // one group per filter row, for all taps of time (strided convolutions and skip inputs would take columns of their own)
    p.nt = rgb ? 16 : a.n_out;
    p.kt_taps = a.taps_t_only ? 1 : 9;
    p.n_groups = a.taps_t_only ? 1 : 3;
    p.g[0] = {0, a.taps_t_only ? 0 : -a.wp - 1, a.taps_t_only ? 1 : 3, {0, 1, 2}, {0, 0, 0}};
    p.tiles_per_seg = (int)((plane + 511) / 512);
    p.na = stage_max / cb::ct_stage(p.nt);   // 3, 4 or 5 stages
    maps[5] = rows_map(a.w, a.n_out, k_cols, p.nt / 2);
    if (rgb) return conv_time_launch<0, true>(maps, p, s);
    if (!has_norm) return conv_time_launch<0, false>(maps, p, s);
    if (a.n_out == 64) return conv_time_launch<64, false>(maps, p, s);
    throw std::runtime_error("conv: the fused norm takes 64, 128 or 256 channels");
  }
  if (!strided) {
    if (a.taps_t_only) {
      for (int kt = 0; kt < 3; ++kt) p.g[p.n_groups++] = {kt, 0, 1, {0, 0, 0}, {(short)kt, 0, 0}};
    } else {
      for (int kt = 0; kt < 3; ++kt)
        for (int kh = 0; kh < 3; ++kh) {
          const short t0 = (short)((kt * 3 + kh) * 3);
          p.g[p.n_groups++] = {kt, (kh - 1) * a.wp - 1, 3, {0, 1, 2}, {t0, (short)(t0 + 1), (short)(t0 + 2)}};
        }
    }
  } else {
    for (int kt = 0; kt < 3; ++kt)
      for (int kh = 0; kh < 3; ++kh) {
        const int base = (int)((kh & 1) * 2 * sub + (kh >> 1) * (a.wp / 2));
        const short t0 = (short)((kt * 3 + kh) * 3);
        p.g[p.n_groups++] = {kt, base, 2, {0, 1, 0}, {t0, (short)(t0 + 2), 0}};
        p.g[p.n_groups++] = {kt, base + (int)sub, 1, {0, 0, 0}, {(short)(t0 + 1), 0, 0}};
      }
  }
  if (has_skip) {
    p.skip_cblocks = a.skip_c / 64;
    p.skip_kcol = 27 * a.c;
  }
  p.tiles_per_seg = (p.seg_rows + 256 * R - 1) / (256 * R);
  const int a_slot = box * cb::cv_boxes(R) * 128, b_slot = p.mma_n * 64;
  const int chunk = std::min(cb::CV_CHUNK, std::max(p.cblocks, p.skip_cblocks));
  // activations: one group's tiles and as many of the next one as fit beside the weight tiles: eight of those, or six where
  // four channel blocks meet 256 output channels
  p.nb = 8;
  if ((stage_max - p.nb * b_slot) / a_slot < chunk + 2) p.nb = 6;
  p.na = std::min(2 * chunk + (chunk == 1 ? 1 : 0), (stage_max - p.nb * b_slot) / a_slot);
  if (p.na < chunk + 1) throw std::runtime_error("conv: no room for the operand rings");
  maps[5] = rows_map(a.w, a.n_out, k_cols, p.mma_n / 2);
  if (R == 2) conv_dispatch<2>(maps, p, s);
  else conv_dispatch<1>(maps, p, s);
}

void conv_silu_selftest(uint32_t first, long long n, unsigned long long* differ, cudaStream_t s) {
  if (n > 0) cb::conv_silu_selftest_kernel<<<(int)std::min<long long>((n + 255) / 256, 148 * 8), 256, 0, s>>>(first, n, differ);
}

void conv_pack_rgb(const void* src, int is_f32, long long c_stride, void* dst, int n, int h, int w, cudaStream_t s) {
  const long long total = (long long)n * (h + 2) * (w + 2);
  if (total == 0) return;
  const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
  if (is_f32)
    cb::conv_pack_rgb_kernel<float><<<blocks, 256, 0, s>>>((const float*)src, c_stride, (uint4*)dst, n, h, w);
  else
    cb::conv_pack_rgb_kernel<bf16><<<blocks, 256, 0, s>>>((const bf16*)src, c_stride, (uint4*)dst, n, h, w);
}

}  // namespace cosmos
