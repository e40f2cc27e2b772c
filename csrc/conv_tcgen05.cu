// K13: causal 3x3x3 convolutions of the video tokenizer as an implicit GEMM on tcgen05, on channels-last bf16 volumes
// [frames, H + 2, W + 2, C] with a zero border and two context frames in front.
//
// A CTA pair (cta_group::2) computes R x 256 rows (positions of the flattened volume) by up to 256 output channels. What
// bounds such a kernel is the delivery of the operands from L2 into shared memory (about 45 B per clock and SM): a plain
// implicit GEMM fetches a fresh 128-row tile of activations for each of the 27 taps. Here
//   * the three taps of one row of the filter read one staged tile of 128 R + 8 rows at row offsets 0, 1 and 2: the matrix
//     descriptor starts in the middle of a swizzle atom (the swizzle is a function of the shared-memory address), so a tile
//     crosses L2 -> shared memory 9 times and not 27;
//   * with 128 output channels or fewer R = 2 row tiles share each weight tile, in tensor memory as two accumulators of 128
//     columns, double-buffered against the epilogue;
//   * activations and weights have rings of their own, so that a weight tile holds its slot for one product and an
//     activation tile for three.
// Per 64 channels, tap and 128 rows a CTA of the pair stages 5.6 KB of activations and 4 of weights at 128 output channels, where
// a tile for each tap would take 16 and 8.
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
// 256 -> 256 at half resolution 1.74 ms = 1.62, 128 -> 64 upsampled 1.57 ms = 0.90 (at 64 columns the reads of A from shared
// memory bound the product). The one-tile-per-tap form with its separate passes took 48 ms a chunk of the encoder's
// convolutions and norms where this takes 9.5.
// Order of the sum: filter taps, then channel blocks of 64 (of up to 256 channels at a time). Waits are bounded as
// everywhere (common.cuh).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace cb {
using namespace cosmos;   // ConvOut

constexpr int CV_HALO_ROWS = 136;              // rows of the first box of a tile: 128 and the 2 rows that shifted taps need
constexpr int CV_MAX_GROUPS = 18;
constexpr int CV_CHUNK = 4;                    // channel blocks of 64 whose tiles are staged together
constexpr int CV_SMEM_MAX = 227 * 1024;
constexpr int CV_BARS = 512;                   // bytes for barriers, tensor-memory slot and abort flag
constexpr int CV_SUMS = 4096;                  // row sums of the norm: [2 tiles][2 row tiles][2 column halves][128 rows] floats
constexpr int CV_GAMMA = 1024;                 // the norm's weights as fp32

// Taps that read one staged tile: row offset of the tile, and per tap its shift inside the tile and its index in the weights.
struct ConvGroup {
  int off;
  int n_taps;
  short shift[3], tap[3];
};

struct ConvParams {
  ConvGroup g[CV_MAX_GROUPS];
  int n_groups;          // over the input volume; the skip projection (second input) has one group of one tap, offset 0
  int cblocks, skip_cblocks, skip_kcol;
  int n_out, mma_n, n_tiles;
  int na, nb;            // ring slots
  // rows: n_seg segments (frames of a strided convolution, else one) of seg_rows rows
  int n_seg, seg_rows, tiles_per_seg;
  int a_row0, a_seg_stride, skip_row0;
  int pw, plane;         // width and size of the plane that a segment's rows walk through
  int hp, wp;            // padded size of that plane (strided: kept rows + 1, kept columns + 1)
  const float* bias;
  const bf16* resid;     // layout of the volume
  bf16* out;             // raw result or null
  bf16* out_norm;        // silu(rmsnorm(result)) or null
  const bf16* gamma;
  float eps;
  uint8_t* rgb;
  int mode;              // CONV_OUT_*
  int keep_border;       // CONV_OUT_SAME: the border's cells are not written
  int tpad;              // context frames in front of every output volume
  int f_out;             // frames computed
  int up_t, up_first;    // CONV_OUT_UP: temporal doubling, first chunk (its first frame is not doubled)
  int* status;
};

template <int R>
struct ConvCfg {
  static constexpr int A_ROWS = 128 * R + 8;
  static constexpr int A_SLOT = A_ROWS * 128;
  static constexpr int ACC_COLS = 256 / R;     // tensor-memory columns of one accumulator
  static constexpr int THREADS = 64 + 256 * R; // producer, MMA issuer, eight epilogue warps per row tile
};

__device__ __forceinline__ void cv_store16(bf16* dst, const uint32_t (&pk)[8]) {
  reinterpret_cast<uint4*>(dst)[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
  reinterpret_cast<uint4*>(dst)[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
}

// silu(z) = z / (1 + exp(-z)) of 16 values given as their negatives, rounded to bf16. The quotient is z times an approximate
// reciprocal, refined once by its residual (of all 2^32 fp32 values, two then differ from the division's, in their last bit);
// negatives of value and reciprocal let every step be a packed instruction. Beyond 80, where the exponential leaves its range,
// and for infinities the division itself.
__device__ __forceinline__ void cv_silu16(const uint64_t (&zn)[8], uint32_t (&out)[8]) {
  const uint64_t log2e = pack2(1.4426950408889634f, 1.4426950408889634f), one = pack2(1.f, 1.f);
  float top = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float2 z = unpack2(zn[k]);
    top = fmaxf(top, fmaxf(fabsf(z.x), fabsf(z.y)));
    const float2 t = unpack2(mul2(zn[k], log2e));
    const uint64_t den = add2(pack2(ex2(t.x), ex2(t.y)), one);
    const float2 d = unpack2(den);
    float r0, r1;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(-d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(-d.y));
    const uint64_t rn = pack2(r0, r1), q = mul2(zn[k], rn);
    const float2 y = unpack2(fma2(fma2(q, den, zn[k]), rn, q));
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

// Meeting of the two warps that share the rows of a quadrant; true when both say so.
__device__ __forceinline__ bool cv_pair_and(int id, bool ok) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 q, %1, 0;\n\t"
      "barrier.cta.red.and.pred p, %2, 64, q;\n\t"
      "selp.s32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1 : 0), "r"(id)
      : "memory");
  return r != 0;
}

// Where a row of the result goes: `n_t` x `n_y` x `n_x` rows starting at `row` (one row except for the upsampled form).
struct ConvDest {
  long long row, st, sy;
  int n_t, n_y, n_x;
};

__device__ __forceinline__ ConvDest conv_dest(const ConvParams& p, int f, int y, int x) {
  ConvDest d{0, 0, 0, 1, 1, 1};
  if (p.mode == CONV_OUT_SAME) {
    d.row = (long long)(f + p.tpad) * p.plane + y * p.pw + x;
  } else if (p.mode == CONV_OUT_S2D) {
    const int q = (p.hp >> 1) * (p.wp >> 1);
    d.row = ((long long)(f + p.tpad) * 4 + (y & 1) * 2 + (x & 1)) * q + (y >> 1) * (p.wp >> 1) + (x >> 1);
  } else if (p.mode == CONV_OUT_DOWN) {
    d.row = ((long long)(f + p.tpad) * (p.hp + 1) + y + 1) * (p.wp + 1) + x + 1;
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
    d.row = (t0 + p.tpad) * d.st + (long long)y0 * wd + x0;
  }
  return d;
}

// R row tiles per CTA; NC = channels of the fused norm (64, 128, 256) or 0; RGB: pixels.
template <int R, int NC, bool RGB>
__global__ void __launch_bounds__(ConvCfg<R>::THREADS, 1)
conv_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmA2,
            const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmX2,
            const __grid_constant__ CUtensorMap tmB, const __grid_constant__ ConvParams p) {
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
  float* row_sums = reinterpret_cast<float*>(smem_raw + (bar_base + CV_BARS - smem_u32(smem_raw)));
  float* gamma = row_sums + CV_SUMS / 4;

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
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if constexpr (NC > 0) {
    for (int c = threadIdx.x; c < NC; c += Cfg::THREADS) gamma[c] = __bfloat162float(p.gamma[c]);
  }
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
    if (lane == 0) {
      // ---------------- TMA producer: both rings, in the order in which the products consume them
      int ia = 0, ib = 0;
      uint32_t pha = 0, phb = 0;   // phase parities of the rings
      bool ok = true;
      for (int t = first_tile; t < total && ok; t += tile_step) {
        const int nt = t % p.n_tiles, mt = t / p.n_tiles;
        const int seg = mt / p.tiles_per_seg, tile = mt - seg * p.tiles_per_seg;
        const int local = tile * TILE_M + int(rank) * (128 * R);
        for (int ph = 0; ph < 2 && ok; ++ph) {
          const int cblocks = ph ? p.skip_cblocks : p.cblocks;
          const int row = (ph ? p.skip_row0 : p.a_row0 + seg * p.a_seg_stride) + local;
          const CUtensorMap* m0 = ph ? &tmX : &tmA;
          const CUtensorMap* m1 = ph ? &tmX2 : &tmA2;
          for (int c0 = 0; c0 < cblocks && ok; c0 += CV_CHUNK) {
            const int nc = min(CV_CHUNK, cblocks - c0);
            const int n_groups = ph ? 1 : p.n_groups;
            for (int g = 0; g < n_groups && ok; ++g) {
              const int n_taps = ph ? 1 : p.g[g].n_taps;
              const int y = row + (ph ? 0 : p.g[g].off);
              for (int i = 0; i < n_taps && ok; ++i) {
                const int kcol = ph ? p.skip_kcol : p.g[g].tap[i] * cblocks * 64;
                for (int c = 0; c < nc; ++c) {
                  if (i == 0) {
                    if (!mbar_wait(empty_a(ia), pha ^ 1, abort_flag, p.status, ST_TIMEOUT_TMA)) { ok = false; break; }
                    if (rank == 0) mbar_arrive_expect_tx(full_a(ia), 2 * Cfg::A_SLOT);
                    const uint32_t fb = mapa(full_a(ia), 0);
                    const uint32_t dst = smem_base + ia * Cfg::A_SLOT;
                    tma_load_2d_pair(dst, m0, fb, (c0 + c) * 64, y);
#pragma unroll
                    for (int r = 1; r < R; ++r)
                      tma_load_2d_pair(dst + (CV_HALO_ROWS + (r - 1) * 128) * 128, m1, fb, (c0 + c) * 64,
                                       y + CV_HALO_ROWS + (r - 1) * 128);
                    if (++ia == NA) { ia = 0; pha ^= 1; }
                  }
                  if (!mbar_wait(empty_b(ib), phb ^ 1, abort_flag, p.status, ST_TIMEOUT_TMA)) { ok = false; break; }
                  if (rank == 0) mbar_arrive_expect_tx(full_b(ib), 2 * b_slot);
                  tma_load_2d_pair(b_base + ib * b_slot, &tmB, mapa(full_b(ib), 0), kcol + (c0 + c) * 64,
                                   nt * 256 + int(rank) * (p.mma_n >> 1));
                  if (++ib == NB) { ib = 0; phb ^= 1; }
                }
              }
            }
          }
        }
      }
      if (!ok) {
        // copies in flight are counted on the leader's barriers: give them a fixed time, far beyond a copy's latency
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) {}
      }
    }
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
        uint32_t acc = 0;
        for (int ph = 0; ph < 2 && ok; ++ph) {
          const int cblocks = ph ? p.skip_cblocks : p.cblocks;
          for (int c0 = 0; c0 < cblocks && ok; c0 += CV_CHUNK) {
            const int nc = min(CV_CHUNK, cblocks - c0);
            const int n_groups = ph ? 1 : p.n_groups;
            for (int g = 0; g < n_groups && ok; ++g) {
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
    // code left the instruction cache and a tile took 67 us. Latency bounds what is left (the divisions of the SiLU most of
    // all, which are exact so that the result is the separate norm kernel's), hence the number of warps.
    const int quad = warp & 3, half = ((warp - 2) >> 2) & 1, r = (warp - 2) >> 3;
    const int pair_id = 1 + r * 4 + quad;
    int tcount = 0;
    for (int t = first_tile; t < total; t += tile_step, ++tcount) {
      const int buf = tcount & 1;
      const int nt = t % p.n_tiles, mt = t / p.n_tiles;
      const int seg = mt / p.tiles_per_seg, tile = mt - seg * p.tiles_per_seg;
      const int q = tile * TILE_M + int(rank) * (128 * R) + r * 128 + quad * 32 + lane;
      const uint32_t ta = tmem_base + (uint32_t(quad * 32) << 16) + buf * 256 + r * Cfg::ACC_COLS;
      const bool row_ok = q < p.seg_rows;
      const int f0 = q / p.plane, rem = q - f0 * p.plane;
      const int f = f0 + seg, y = rem / p.pw, x = rem - y * p.pw;   // several segments: one frame each
      const bool down = p.mode == CONV_OUT_DOWN;
      const bool inside = row_ok && (down ? (y < p.hp - 1 && x < p.wp - 1) : (y >= 1 && y <= p.hp - 2 && x >= 1 && x <= p.wp - 2));
      bool go = mbar_wait(tfull(buf), (tcount >> 1) & 1, abort_flag, p.status, ST_TIMEOUT_EPI);
      // warps that meet below leave together: a wait that one of them gave up is given up by both
      go = NC > 0 ? cv_pair_and(pair_id, go) : __all_sync(0xffffffffu, go);
      if (!go) break;
      tc_fence_after();
      if constexpr (RGB) {
        uint32_t v[16];
        tmem_ld16(ta, v);
        tmem_wait_ld();
        if (inside && half == 0) {
          uint8_t* o = p.rgb + (((long long)f * (p.hp - 2) + y - 1) * (p.wp - 2) + x - 1) * 3;
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            // columns 3 .. 8: the low parts of fp32 weights, exact in three bf16 terms
            const float a = ((__uint_as_float(v[6 + c]) + __uint_as_float(v[3 + c])) + __uint_as_float(v[c])) + p.bias[c];
            o[c] = (uint8_t)__float2int_rn((fminf(fmaxf(a, -1.f), 1.f) + 1.f) * 127.5f);
          }
        }
      } else {
        const ConvDest dst = conv_dest(p, f, y, x);
        const int n_base = nt * 256, n_end = min(256, p.n_out - n_base);
        const long long ld = p.n_out;
        if (down && row_ok && half == 0 && (x == 0 || y == 0)) {
          // border cells that no position of the plane maps to: left column, top row
          for (int k = 0; k < 3; ++k) {
            if ((k == 0 && x != 0) || (k == 1 && y != 0) || (k == 2 && (x != 0 || y != 0))) continue;
            const long long cell = dst.row - (k == 1 ? 0 : 1) - (k == 0 ? 0 : p.wp + 1);
            for (int c = 0; c < n_end; c += 8) {
              if (p.out) *reinterpret_cast<uint4*>(p.out + cell * ld + n_base + c) = make_uint4(0, 0, 0, 0);
              if (p.out_norm) *reinterpret_cast<uint4*>(p.out_norm + cell * ld + n_base + c) = make_uint4(0, 0, 0, 0);
            }
          }
        }
        __syncwarp();
        const bf16* res = p.resid ? p.resid + ((long long)(f + p.tpad) * p.plane + rem) * ld + n_base : nullptr;
        uint64_t sq[2] = {0, 0};                         // sums of squares, two pairs
        const int groups = (NC > 0 ? NC : n_end) >> 5;   // of this warp
#pragma unroll 1
        for (int i = 0; i < groups; ++i) {
          const int c = 32 * i + 16 * half;
          uint32_t v[16], pk[8];
          tmem_ld16(ta + c, v);
          uint4 ru[2];
          if (res && inside) {
            ru[0] = reinterpret_cast<const uint4*>(res + c)[0];
            ru[1] = reinterpret_cast<const uint4*>(res + c)[1];
          }
          tmem_wait_ld();
          if (inside) {
            uint64_t a[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = pack2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
            if (p.bias) {
              const float4* b4 = reinterpret_cast<const float4*>(p.bias + n_base + c);
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
                const uint32_t w[4] = {ru[k].x, ru[k].y, ru[k].z, ru[k].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) a[4 * k + e] = add2(a[4 * k + e], pack2(bf16lo(w[e]), bf16hi(w[e])));
              }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              float lo, hi;
              unpack2(a[k], lo, hi);
              pk[k] = pack_bf16(lo, hi);
            }
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) pk[k] = 0u;
          }
          if (p.out && (inside || (row_ok && !p.keep_border))) {
            bf16* o = p.out + dst.row * ld + n_base + c;
            if (p.mode != CONV_OUT_UP) {
              cv_store16(o, pk);
            } else {
              for (int tt = 0; tt < dst.n_t; ++tt)
                for (int yy = 0; yy < dst.n_y; ++yy)
                  for (int xx = 0; xx < dst.n_x; ++xx) cv_store16(o + (tt * dst.st + yy * dst.sy + xx) * ld, pk);
            }
          }
          if constexpr (NC > 0) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const uint64_t x = pack2(bf16lo(pk[k]), bf16hi(pk[k]));
              sq[k & 1] = fma2(x, x, sq[k & 1]);
            }
            __syncwarp();
            tmem_st8(ta + c, pk);   // the rounded values wait in place of their accumulators
          }
          __syncwarp();
        }
        if constexpr (NC > 0) {
          // the other half's sum (two buffers: a warp is at most one meeting ahead of its partner)
          const float2 s2 = unpack2(add2(sq[0], sq[1]));
          const float sum = s2.x + s2.y;
          row_sums[((buf * 2 + r) * 2 + half) * 128 + quad * 32 + lane] = sum;
          tmem_wait_st();
          cv_pair_and(pair_id, true);
          const float other = row_sums[((buf * 2 + r) * 2 + (half ^ 1)) * 128 + quad * 32 + lane];
          const float rneg = -rsqrtf((sum + other) / (float)NC + p.eps);
          const uint64_t rneg2 = pack2(rneg, rneg);
          bf16* o = p.out_norm + dst.row * ld;
#pragma unroll 1
          for (int c = 16 * half; c < NC; c += 32) {
            uint32_t pk[8], on[8];
            uint64_t zn[8];
            tmem_ld8(ta + c, pk);
            const float4* g4 = reinterpret_cast<const float4*>(gamma + c);
            float4 g[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) g[k] = g4[k];
            tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 8; ++k)
              zn[k] = mul2(mul2(pack2(bf16lo(pk[k]), bf16hi(pk[k])), rneg2),
                           k & 1 ? pack2(g[k >> 1].z, g[k >> 1].w) : pack2(g[k >> 1].x, g[k >> 1].y));
            cv_silu16(zn, on);   // zero on the border
            if (row_ok) cv_store16(o + c, on);
            __syncwarp();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (rank != 0) mbar_arrive_cluster(mapa(tempty(buf), 0));
        else mbar_arrive(tempty(buf));
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
conv_pack_rgb_kernel(const T* __restrict__ src, long long c_stride, uint4* __restrict__ dst, int n, int h, int w, int tpad) {
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
    uint4* o = dst + (i + (long long)tpad * (h + 2) * (w + 2)) * 8;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      o[k] = make_uint4(pack_bf16(v[8 * k], v[8 * k + 1]), pack_bf16(v[8 * k + 2], v[8 * k + 3]),
                        pack_bf16(v[8 * k + 4], v[8 * k + 5]), pack_bf16(v[8 * k + 6], v[8 * k + 7]));
#pragma unroll
    for (int k = 4; k < 8; ++k) o[k] = make_uint4(0, 0, 0, 0);
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

template <int R, int NC, bool RGB>
void conv_launch(const CUtensorMap (&maps)[5], const cb::ConvParams& p, int smem, cudaStream_t s) {
  auto kern = cb::conv_kernel<R, NC, RGB>;
  static int pairs = 0;   // of this kernel, at its largest shared-memory size
  cudaLaunchConfig_t cfg{};
  cfg.blockDim = dim3(cb::ConvCfg<R>::THREADS);
  cfg.dynamicSmemBytes = cb::CV_SMEM_MAX;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  if (pairs == 0) {
    int dev = 0, sms = 148, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cb::CV_SMEM_MAX);
    cfg.gridDim = dim3(sms & ~1);
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = sms / 2;
    }
    pairs = std::min(n, sms / 2);
  }
  const int total = p.n_seg * p.tiles_per_seg * p.n_tiles;
  const int limit = gemm_grid_limit(), at_once = limit > 0 ? std::min(pairs, std::max(1, limit / 2)) : pairs;
  cfg.gridDim = dim3(2 * std::min(at_once, total));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, maps[0], maps[1], maps[2], maps[3], maps[4], p);
  if (e != cudaSuccess) throw std::runtime_error(std::string("conv: launch failed: ") + cudaGetErrorString(e));
}

template <int R>
void conv_dispatch(const CUtensorMap (&maps)[5], const cb::ConvParams& p, int smem, cudaStream_t s) {
  if (p.rgb) return conv_launch<2, 0, true>(maps, p, smem, s);
  if (!p.out_norm) return conv_launch<R, 0, false>(maps, p, smem, s);
  if constexpr (R == 2) {
    if (p.n_out == 64) return conv_launch<2, 64, false>(maps, p, smem, s);
    if (p.n_out == 128) return conv_launch<2, 128, false>(maps, p, smem, s);
  } else {
    if (p.n_out == 256) return conv_launch<1, 256, false>(maps, p, smem, s);
  }
  throw std::runtime_error("conv: the fused norm takes 64, 128 or 256 channels");
}

}  // namespace

void conv3d_fused(const ConvArgs& a, cudaStream_t s) {
  const bool strided = a.mode == CONV_OUT_DOWN, rgb = a.rgb != nullptr;
  if (a.c <= 0 || a.c % 64 || a.skip_c % 64 || a.hp < 3 || a.wp < 3 || (!rgb && (a.n_out <= 0 || a.n_out % 32)))
    throw std::runtime_error("conv: needs input channels % 64 == 0, output channels % 32 == 0 and a padded volume");
  if ((strided || a.mode == CONV_OUT_S2D) && (a.hp % 2 || a.wp % 2)) throw std::runtime_error("conv: stride 2 needs even padded sizes");
  if (rgb ? a.n_out != 9 : (!a.out && !a.out_norm)) throw std::runtime_error("conv: nothing to write");
  if ((a.skip && (strided || a.mode == CONV_OUT_UP)) || (a.resid && (strided || rgb)))
    throw std::runtime_error("conv: no residual or skip input in this form");
  if (a.out_norm && (a.mode == CONV_OUT_S2D || a.mode == CONV_OUT_UP)) throw std::runtime_error("conv: no norm in this form");
  if (a.keep_border && (a.mode != CONV_OUT_SAME || a.out_norm || rgb)) throw std::runtime_error("conv: this form writes its border");
  if (a.f_out < 1) return;
  cb::ConvParams p{};
  p.cblocks = a.c / 64;
  p.n_out = a.n_out;
  p.n_tiles = (a.n_out + 255) / 256;
  p.mma_n = p.n_tiles > 1 ? 256 : (a.n_out + 15) / 16 * 16;
  p.bias = a.bias;
  p.resid = reinterpret_cast<const bf16*>(a.resid);
  p.out = reinterpret_cast<bf16*>(a.out);
  p.out_norm = reinterpret_cast<bf16*>(a.out_norm);
  p.gamma = reinterpret_cast<const bf16*>(a.gamma);
  p.eps = a.eps;
  p.rgb = reinterpret_cast<uint8_t*>(a.rgb);
  p.mode = a.mode;
  p.keep_border = a.keep_border;
  p.tpad = a.tpad;
  p.f_out = a.f_out;
  p.up_t = a.up_temporal;
  p.up_first = a.up_first;
  p.status = a.status;
  const int plane = a.hp * a.wp, sub = (a.hp / 2) * (a.wp / 2);
  const long long rows = (long long)a.frames_in * plane;
  if (rows + plane > 0x7fffffffll) throw std::runtime_error("conv: volume too large for 32-bit row indices; use shorter chunks");
  if (!strided) {
    p.n_seg = 1;
    p.seg_rows = a.f_out * plane;
    p.a_row0 = a.tpad * plane;
    p.plane = plane;
    p.pw = a.wp; p.hp = a.hp; p.wp = a.wp;
    if (a.taps_t_only) {
      for (int kt = 0; kt < 3; ++kt) p.g[p.n_groups++] = {(kt - 2) * plane, 1, {0, 0, 0}, {(short)kt, 0, 0}};
    } else {
      for (int kt = 0; kt < 3; ++kt)
        for (int kh = 0; kh < 3; ++kh) {
          const short t0 = (short)((kt * 3 + kh) * 3);
          p.g[p.n_groups++] = {(kt - 2) * plane + (kh - 1) * a.wp - 1, 3, {0, 1, 2}, {t0, (short)(t0 + 1), (short)(t0 + 2)}};
        }
    }
  } else {
    // segment = kept frame; the kept position (j, i) of a frame sits at padded (2 j + kh, 2 i + kw) for tap (kh, kw)
    p.n_seg = a.f_out;
    p.seg_rows = sub;
    p.a_row0 = a.t_first * 4 * sub;
    p.a_seg_stride = a.t_step * 4 * sub;
    p.plane = sub;
    p.pw = a.wp / 2; p.hp = a.hp / 2; p.wp = a.wp / 2;
    for (int kt = 0; kt < 3; ++kt)
      for (int kh = 0; kh < 3; ++kh) {
        const int base = (kt * 4 + (kh & 1) * 2) * sub + (kh >> 1) * (a.wp / 2);
        const short t0 = (short)((kt * 3 + kh) * 3);
        p.g[p.n_groups++] = {base, 2, {0, 1, 0}, {t0, (short)(t0 + 2), 0}};
        p.g[p.n_groups++] = {base + sub, 1, {0, 0, 0}, {(short)(t0 + 1), 0, 0}};
      }
  }
  if (a.skip) {
    p.skip_cblocks = a.skip_c / 64;
    p.skip_kcol = 27 * a.c;
    p.skip_row0 = p.a_row0;
  }
  // two row tiles share a weight tile where tensor memory holds two double-buffered accumulators
  const int R = p.mma_n <= 128 ? 2 : 1;
  p.tiles_per_seg = (p.seg_rows + 256 * R - 1) / (256 * R);
  const int a_slot = (128 * R + 8) * 128, b_slot = p.mma_n * 64;
  const int stage_max = cb::CV_SMEM_MAX - 1024 - cb::CV_BARS - cb::CV_SUMS - cb::CV_GAMMA;
  const int chunk = std::min(cb::CV_CHUNK, std::max(p.cblocks, p.skip_cblocks));
  // activations: one group's tiles and as many of the next one as fit beside the weight tiles: eight of those, or six where
  // four channel blocks meet 256 output channels
  p.nb = 8;
  if ((stage_max - p.nb * b_slot) / a_slot < chunk + 2) p.nb = 6;
  p.na = std::min(2 * chunk + (chunk == 1 ? 1 : 0), (stage_max - p.nb * b_slot) / a_slot);
  if (p.na < chunk + 1) throw std::runtime_error("conv: no room for the operand rings");
  // always the whole shared memory: a second CTA on the SM would wait for tensor memory that the first one holds
  const int smem = cb::CV_SMEM_MAX;
  const int k_cols = (a.taps_t_only ? 3 : 27) * a.c + a.skip_c;
  CUtensorMap maps[5];
  maps[0] = rows_map(a.x, rows, a.c, cb::CV_HALO_ROWS);
  maps[1] = rows_map(a.x, rows, a.c, 128);
  maps[2] = a.skip ? rows_map(a.skip, rows, a.skip_c, cb::CV_HALO_ROWS) : maps[0];
  maps[3] = a.skip ? rows_map(a.skip, rows, a.skip_c, 128) : maps[1];
  maps[4] = rows_map(a.w, a.n_out, k_cols, p.mma_n / 2);
  if (R == 2) conv_dispatch<2>(maps, p, smem, s);
  else conv_dispatch<1>(maps, p, smem, s);
}

void conv_pack_rgb(const void* src, int is_f32, long long c_stride, void* dst, int n, int h, int w, cudaStream_t s) {
  const long long total = (long long)n * (h + 2) * (w + 2);
  if (total == 0) return;
  const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
  if (is_f32)
    cb::conv_pack_rgb_kernel<float><<<blocks, 256, 0, s>>>((const float*)src, c_stride, (uint4*)dst, n, h, w, 2);
  else
    cb::conv_pack_rgb_kernel<bf16><<<blocks, 256, 0, s>>>((const bf16*)src, c_stride, (uint4*)dst, n, h, w, 2);
}

}  // namespace cosmos
