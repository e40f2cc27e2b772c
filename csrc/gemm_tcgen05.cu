// K1: persistent bf16 GEMM  C[M,N] = A[M,K] * B[N,K]^T  on tcgen05 tensor cores.
//
// Layout of one CTA (320 threads):
//   warp 0      TMA producer  (A 128x64 and B 256x64 tiles, 128-byte swizzle, 4-stage ring)
//   warp 1      MMA issuer    (tcgen05.mma M=128 N=256 K=16, fp32 accumulators in TMEM,
//                              two 256-column accumulator buffers so the epilogue of tile i
//                              overlaps the main loop of tile i+1)
//   warps 2..9  epilogue      (tcgen05.ld -> registers -> fused epilogue -> global / peer stores)
//
// Fused epilogues (template parameter EPI):
//   EPI_PLAIN        C = acc (+ bias)
//   EPI_GELU         C = gelu(acc (+ bias)), the exact (erf) form
//   EPI_SWIGLU       B holds [gate ; up] stacked along N; C[m, j] = silu(gate_j) * up_j  (N/2 wide)
//   EPI_GATED_RESID  C = R + gate[m / rows_per_batch, n] * (acc + bias)   (AdaLN gated residual)
//   EPI_QKV_ROPE     columns are heads of 128: per-head RMSNorm (q/k) + rotary embedding, and
//                    each 128-column chunk is written through a routing table, so a chunk
//                    can land in another GPU's buffer (sequence->head all-to-all of Ulysses
//                    context parallelism done by the epilogue's stores).
//
// Grouped by a tile map (GemmParams::tile_map, mixture-of-experts layers): the rows of A are sorted by group, the map
// names the group and the row range of every m-tile, and the group picks its N rows of B (the groups' weights stacked
// along N). Segments are neither padded nor aligned: a tile's rows beyond its range are other groups' rows, computed
// and not stored. The number of m-tiles lives on the device, so a captured graph follows the routing of each replay.
//
// All mbarrier waits are bounded; on expiry the kernel records a status code and exits
// through the common tail (TMEM is freed).
#include "common.cuh"
#include "kernels.h"
#include "launch.cuh"
#include <algorithm>
#include <cstdlib>

namespace cb {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_BYTES = BM * BK * 2;      // 16 KB
// NC = 1: one CTA per 128x256 tile, 4 stages of A 16 KB + B 32 KB.
// NC = 2: a CTA pair per 256x256 tile (tcgen05 cta_group::2, M = 256): each CTA stages its own 128 rows
// of A and its own 128 of the tile's 256 B rows, so a stage is 32 KB per CTA and the B operand crosses
// shared memory once per pair instead of once per CTA; 6 stages.
// NW = 2 (pairs only): a pair computes 256 x 512, two neighbouring 256-column tiles of one A tile, with 48 KB of operands per CTA
// and 1024 clocks of products where a 256x256 tile has 32 KB and 512. The two accumulators fill tensor memory, so they are not
// double-buffered: the first and last k-blocks of a tile are issued accumulator by accumulator, so that one is drained while the
// other is computed. 4 stages.
constexpr int EPI_WARPS = 8;   // two per quadrant of accumulator rows, each with half of the columns
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;
constexpr int gamma_smem(int epi) { return epi == EPI_QKV_ROPE ? 1024 : 0; }  // both norms' weights as fp32, behind the barriers
template <int NC, int NW = 1> struct GemmCfg {
  static constexpr int STAGES = NW == 2 ? 4 : NC == 2 ? 6 : 4;
  static constexpr int B_BYTES = NW * (BN / NC) * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SLABS = EPI_WARPS * 4096;  // one per epilogue warp (see Slab)
  static constexpr int SMEM = STAGES * STAGE_BYTES + SLABS + 1024 /*align*/ + 256 /*barriers*/;
};

struct GemmParams {
  int M, N, K;
  int b_row1;            // row offset in B of the second 128-row half of the tile
  int n_tiles, m_tiles;  // tile counts (n_tiles counts tiles of 256 * NW columns, 128 * NW for SWIGLU)
  bf16* C;
  long long ldc;
  const bf16* bias;      // [N] or null
  const bf16* R;         // residual [M, ldr]
  long long ldr;
  const bf16* gate;      // [batches, N]
  int rows_per_batch;
  // EPI_QKV_ROPE
  const long long* route_ptr;  // per 128-col chunk: destination base address (bf16*)
  const long long* route_ld;   // per chunk: row stride in elements
  int route_rows;              // rows per routing table: row m goes through table m / route_rows, as its row m % route_rows
  const float* cos_tab;        // [rope_rows, 64]
  const float* sin_tab;
  int rope_rows;
  const bf16* gamma_q;         // [128]
  const bf16* gamma_k;
  int n_q_heads, n_k_heads;
  float eps;
  int* status;
  // split-K (skinny problems, e.g. decode): the K range is divided among k_splits CTAs per output
  // tile; each writes its raw fp32 accumulators to partial[ks][M][N] and a second kernel reduces
  // them and applies the epilogue.
  int k_splits;
  float* partial;
  const float* rowvec;   // EPI_ATTN_P: lse[M]; EPI_ATTN_DS: D[M]
  float attn_scale;
  int attn_mask, attn_n_ar;
  // operand majors: 0 = K-major ([rows, K] storage), 1 = MN-major ([K, rows] storage, i.e. the
  // transposed operand is read in place; used by the backward GEMMs dX = dY W and dW = dY^T X)
  int a_mn, b_mn;
  // Rows of A that a single CTA's stage receives: 128, or 8 or 16 in a decode step of so few sequences. The rows behind them
  // keep what was there before: products of theirs land in accumulator rows that nobody reads. Zero-filling them took a
  // third of the bytes that reach a CTA, and these launches are bound by that, not by HBM: with the weights resident in L2
  // they took as long. M 1, with the reduction, us: 24576 x 4096 SwiGLU 42.3 -> 38.2, 6144 x 4096 15.9 -> 14.3, 151936 x 4096
  // 229 -> 212. With 32 rows nothing is gained (43.0 -> 43.1): there the fp32 partial sums weigh more.
  int a_rows;
  // grouped by a tile map (see the file comment): {group, first row, rows, unused} per m-tile; tile rows = TILE_M
  const int4* tile_map;
  const int* n_tiles_m;  // number of m-tiles of this launch (device)
  int early_b;           // B may be read before the kernels ahead of this one have finished
  int debug;             // timing experiments (wrong results): 1 = every tile loads operand tile (0, 0); 2 = no loads at all
};

// Up to two independent problems served by one persistent launch (grouped GEMM): tiles
// [0, tiles0) belong to problem 0, the rest to problem 1. Used for the per-modality weight
// routing of the Mixture-of-Transformers layers (AR tokens x AR weights, DM tokens x DM weights).
struct GemmGroup {
  GemmParams p[2];
  int tiles0;
  int total;
};

__device__ __forceinline__ void tile_coords(int t, int m_tiles, int n_tiles, int& tm, int& tn) {
  // Rasterise in bands of 16 m-tiles so that CTAs running together share A and B tiles in L2.
  constexpr int GM = 16;
  const int band = t / (GM * n_tiles);
  const int first_m = band * GM;
  const int band_m = min(GM, m_tiles - first_m);
  const int r = t - band * GM * n_tiles;
  tm = first_m + r % band_m;
  tn = r / band_m;
}

// Row ranges of an m-tile: first row of A, end of the rows it owns, first row of its group's weights in B.
struct TileRows {
  int m0, m_end, b_row;
};
template <int TILE_M>
__device__ __forceinline__ TileRows tile_rows(const GemmParams& p, int tm) {
  if (p.tile_map) {
    const int4 e = p.tile_map[tm];
    return {e.y, e.y + e.z, e.x * p.N};
  }
  return {tm * TILE_M, p.M, 0};
}

// A warp's staging area: 32 rows of 128 bytes, the 16-byte chunk c of row r at position c ^ (r & 7). In the accumulator's
// layout a lane holds a row, so a direct access of global memory touches 32 lines per instruction, and those wavefronts
// compete with the operand copies and the tensor core's reads for the shared memory's bandwidth; through the slab an
// instruction touches 4 whole lines.
struct Slab {
  uint32_t base;
  int lane;
  __device__ __forceinline__ uint32_t at(int r, int c) const { return base + r * 128 + ((c ^ (r & 7)) << 4); }
  __device__ __forceinline__ void put(int r, int c, uint4 v) const {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at(r, c)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
  }
  __device__ __forceinline__ uint4 get(int r, int c) const {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at(r, c)) : "memory");
    return v;
  }
  // 8 columns f[0..7] of this lane's row
  __device__ __forceinline__ void put_bf16(int c, const float* f) const {
    put(lane, c, make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7])));
  }
  // Whether rows of `ld` elements from `p` on take 16-byte accesses: callers may pass views that start at any element.
  template <class T>
  static __device__ __forceinline__ bool aligned(const T* p, long long ld) {
    return ((reinterpret_cast<uintptr_t>(p) | (uintptr_t)(ld * (long long)sizeof(T))) & 15) == 0;
  }
  // Coalesced order: lane's i-th chunk is chunk (lane & 7) of row 4 i + lane / 8. rows x 64 columns of `src` (row stride
  // ld) in that order; what lies beyond is zero.
  __device__ __forceinline__ void fetch(uint4 (&v)[8], const bf16* src, long long ld, int rows, int cols) const {
    const int c = (lane & 7) * 8;
    const int vec_cols = aligned(src, ld) ? cols : 0;   // the rest goes by element
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + (lane >> 3);
      v[i] = make_uint4(0, 0, 0, 0);
      if (r < rows && c < cols) {
        const bf16* s = src + r * ld + c;
        if (c + 8 <= vec_cols) {
          v[i] = *reinterpret_cast<const uint4*>(s);
        } else {
          uint32_t u[4] = {0, 0, 0, 0};
          const unsigned short* h = reinterpret_cast<const unsigned short*>(s);
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (c + e < cols) u[e >> 1] |= uint32_t(h[e]) << (16 * (e & 1));
          v[i] = make_uint4(u[0], u[1], u[2], u[3]);
        }
      }
    }
  }
  __device__ __forceinline__ void fill(const uint4 (&v)[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) put(i * 4 + (lane >> 3), lane & 7, v[i]);
    __syncwarp();
  }
  // slab -> rows x 64 columns of `dst` (bf16) or rows x 32 (fp32)
  template <class T>
  __device__ __forceinline__ void store(T* dst, long long ld, int rows, int cols) const {
    constexpr int PER = 16 / sizeof(T);
    __syncwarp();
    const int c = (lane & 7) * PER;
    const int vec_cols = aligned(dst, ld) ? cols : 0;
    if (c < cols) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3);
        if (r < rows) {
          const uint4 v = get(r, lane & 7);
          T* d = dst + r * ld + c;
          if (c + PER <= vec_cols) {
            *reinterpret_cast<uint4*>(d) = v;
          } else {
            const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
            for (int j = 0; j < PER; ++j)
              if (c + j < cols) d[j] = e[j];
          }
        }
      }
    }
    __syncwarp();
  }
};

// Epilogue of a warp: its 32 rows m0 .. (those below m_end) and one half of the 256 columns of accumulator tile tn. `wait`
// waits for the accumulator, `release` hands it back once it has been read. The loops over columns stay rolled: unrolled,
// the code of one tile does not fit the instruction cache and fetching it takes longer than the work.
template <int EPI, class Wait, class Release>
__device__ __forceinline__ bool finish_half(const GemmParams& p, const Slab& slab, uint32_t t_addr, int half, int m0, int m_end,
                                            int tn, int ks, const float* sgamma, Wait wait, Release release) {
  const int lane = slab.lane, m = min(m0 + lane, m_end - 1), rows = m_end - m0;
  const int n0 = EPI == EPI_SWIGLU ? tn * 128 + half * 64 : tn * BN + half * 128;   // first output column
  const int n_out = EPI == EPI_SWIGLU ? p.N / 2 : p.N;
  if (rows <= 0 || n0 >= n_out) {   // nothing to store
    if (!wait()) return false;
    release();
    return true;
  }
  if (p.partial) {   // raw fp32 sums of a K range, the columns of B
    if (!wait()) return false;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      const int at = EPI == EPI_SWIGLU ? (c >> 1) * 128 + half * 64 + (c & 1) * 32 : half * 128 + c * 32;
      tmem_ld32(t_addr + at, v);
      tmem_wait_ld();
      if (c == 3) release();
      const int n = EPI == EPI_SWIGLU ? n0 + (c & 1) * 32 : n0 + c * 32;
      if (rows <= 8 && n + 32 <= n_out) {   // few rows (decode): a lane's own stores touch no more lines, and need no staging
        if (lane < rows) {
          uint4* d = reinterpret_cast<uint4*>(p.partial + ((long long)ks * p.M + m) * p.N + n + (EPI == EPI_SWIGLU && c >= 2 ? n_out : 0));
#pragma unroll
          for (int q = 0; q < 8; ++q) d[q] = make_uint4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
        }
        __syncwarp();
        continue;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) slab.put(lane, q, make_uint4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]));
      float* dst = p.partial + ((long long)ks * p.M + m0) * p.N + n + (EPI == EPI_SWIGLU && c >= 2 ? n_out : 0);
      slab.store(dst, p.N, rows, n_out - n);
    }
    return true;
  }
  if constexpr (EPI == EPI_SWIGLU) {
    if (!wait()) return false;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t g[16], u[16];
      tmem_ld16(t_addr + half * 64 + c * 16, g);
      tmem_ld16(t_addr + 128 + half * 64 + c * 16, u);
      tmem_wait_ld();
      if (c == 3) release();
      float o[16];
      silu16(g, o);
#pragma unroll
      for (int i = 0; i < 16; ++i) o[i] *= __uint_as_float(u[i]);
      slab.put_bf16(c * 2, o);
      slab.put_bf16(c * 2 + 1, o + 8);
    }
    slab.store(p.C + (long long)m0 * p.ldc + n0, p.ldc, rows, n_out - n0);
    return true;
  }
  if constexpr (EPI == EPI_QKV_ROPE) {
    const int chunk = tn * 2 + half;
    // This warp's rows lie in one routing table or, from row `next` on, in the one after it (any, with short tables).
    const int t_rows = p.route_rows, tab0 = p.route_ptr ? m0 / t_rows : 0, next = p.route_ptr ? (tab0 + 1) * t_rows - m0 : 32;
    const int chunks = p.N >> 7;
    const bool crosses = p.route_ptr && next < min(rows, 32);
    long long ld = p.ldc, ld1 = 0;
    bf16 *dst = p.C + n0, *dst1 = nullptr;   // where row m0 = 0 of either table would lie
    if (p.route_ptr) {
      ld = p.route_ld[tab0 * chunks + chunk];
      dst = reinterpret_cast<bf16*>(p.route_ptr[tab0 * chunks + chunk]) - (long long)tab0 * t_rows * ld;
    }
    if (crosses) {
      ld1 = p.route_ld[(tab0 + 1) * chunks + chunk];
      dst1 = reinterpret_cast<bf16*>(p.route_ptr[(tab0 + 1) * chunks + chunk]) - (long long)(tab0 + 1) * t_rows * ld1;
    }
    auto row_at = [&](int r) -> bf16* {
      if (!crosses || r < next) return dst + (m0 + r) * ld;
      if (r < next + t_rows) return dst1 + (m0 + r) * ld1;
      const int t = (m0 + r) / t_rows;
      return reinterpret_cast<bf16*>(p.route_ptr[t * chunks + chunk]) + (long long)(m0 + r - t * t_rows) * p.route_ld[t * chunks + chunk];
    };
    if (chunk < p.n_q_heads + p.n_k_heads && (p.gamma_q || p.gamma_k || p.cos_tab)) {
      // Norm and rotary embedding of one head. 16 columns of both tables at a time go through the slab (chunks 0-3 of a row
      // cosines, 4-7 sines), requested two steps ahead: their latency would otherwise hold the accumulator. The norm's
      // weights are in shared memory for the same reason.
      const bool is_q = chunk < p.n_q_heads;
      const bool normed = (is_q ? p.gamma_q : p.gamma_k) != nullptr, rope = p.cos_tab != nullptr;
      const float* gam = sgamma + (is_q ? 0 : 128);
      const bf16* bias = p.bias ? p.bias + n0 : nullptr;
      const float* tab = (lane & 4 ? p.sin_tab : p.cos_tab) + (lane & 3) * 4;
      const int rr = p.rope_rows, row0 = m0 % rr;
      uint4 t0[8], t1[8];
      auto fetch_tab = [&](uint4 (&t)[8], int q) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          t[i] = make_uint4(0, 0, 0, 0);
          int row = row0 + r;
          if (row >= rr) row = rr >= 32 ? row - rr : row % rr;
          if (r < rows) t[i] = *reinterpret_cast<const uint4*>(tab + (long long)row * 64 + q * 16);
        }
      };
      if (rope) {
        fetch_tab(t0, 0);
        fetch_tab(t1, 1);
      }
      if (!wait()) return false;
      t_addr += half * 128;
      float rinv = 1.f;
      if (normed) {
        float ss = 0.f;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t v[32];
          tmem_ld32(t_addr + c * 32, v);
          tmem_wait_ld();
          if (bias) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __bfloat162float(bias[c * 32 + i]));
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) ss += __uint_as_float(v[i]) * __uint_as_float(v[i]);
        }
        rinv = rsqrtf(ss * (1.f / 128.f) + p.eps);
      }
      auto step = [&](uint4 (&t)[8], int q) {
        uint32_t va[16], vb[16];
        tmem_ld16(t_addr + q * 16, va);
        tmem_ld16(t_addr + 64 + q * 16, vb);
        tmem_wait_ld();
        if (q == 3) release();
        float a[16], b[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          a[i] = __uint_as_float(va[i]);
          b[i] = __uint_as_float(vb[i]);
        }
        if (bias) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            a[i] += __bfloat162float(bias[q * 16 + i]);
            b[i] += __bfloat162float(bias[64 + q * 16 + i]);
          }
        }
        if (normed) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            a[i] = a[i] * rinv * gam[q * 16 + i];
            b[i] = b[i] * rinv * gam[64 + q * 16 + i];
          }
        }
        if (rope) {
          slab.fill(t);
          if (q < 2) fetch_tab(t, q + 2);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint4 cu = slab.get(lane, j), su = slab.get(lane, 4 + j);
            const uint32_t c4[4] = {cu.x, cu.y, cu.z, cu.w}, s4[4] = {su.x, su.y, su.z, su.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float x = a[j * 4 + e], y = b[j * 4 + e], cc = __uint_as_float(c4[e]), sn = __uint_as_float(s4[e]);
              a[j * 4 + e] = fmaf(x, cc, -__fmul_rn(y, sn));
              b[j * 4 + e] = fmaf(x, sn, __fmul_rn(y, cc));
            }
          }
          __syncwarp();
        }
        slab.put_bf16(0, a);
        slab.put_bf16(1, a + 8);
        slab.put_bf16(2, b);
        slab.put_bf16(3, b + 8);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // 8 rows of 2 x 32 bytes per instruction
          const int r = i * 8 + (lane >> 2), c = lane & 3;
          const uint4 v = slab.get(r, c);
          if (r < rows) *reinterpret_cast<uint4*>(row_at(r) + (c >> 1) * 64 + q * 16 + (c & 1) * 8) = v;
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int q = 0; q < 4; q += 2) {
        step(t0, q);
        step(t1, q + 1);
      }
      return true;
    }
    if (!wait()) return false;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      tmem_ld32(t_addr + half * 128 + c * 32, v);
      tmem_wait_ld();
      if (c == 3) release();
      float f[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        f[i] = __uint_as_float(v[i]);
        if (p.bias) f[i] += __bfloat162float(p.bias[n0 + c * 32 + i]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) slab.put_bf16((c & 1) * 4 + q, f + q * 8);
      if (c & 1) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3);
          const uint4 o = slab.get(r, lane & 7);
          if (r < rows) *reinterpret_cast<uint4*>(row_at(r) + (c >> 1) * 64 + (lane & 7) * 8) = o;
        }
        __syncwarp();
      }
    }
    return true;
  }
  if constexpr (EPI == EPI_PLAIN || EPI == EPI_GELU || EPI == EPI_GATED_RESID) {
    // the residual of both 64-column steps is on its way before the accumulator is waited for
    uint4 r1[8];
    if constexpr (EPI == EPI_GATED_RESID) {
      const bf16* r = p.R + (long long)m0 * p.ldr + n0;
      slab.fetch(r1, r, p.ldr, rows, p.N - n0);
      slab.fill(r1);
      slab.fetch(r1, r + 64, p.ldr, rows, p.N - n0 - 64);
    }
    if (!wait()) return false;
    const bf16* gate = EPI == EPI_GATED_RESID && p.gate ? p.gate + (long long)(m / p.rows_per_batch) * p.N : nullptr;
    const bool gate_vec = (p.N & 7) == 0 && (reinterpret_cast<uintptr_t>(p.gate) & 15) == 0;   // rows of whole 16-byte vectors
#pragma unroll 1
    for (int c = 0; c < 8; ++c) {   // 16 columns at a time
      const int n = n0 + c * 16;
      uint32_t v[16];
      tmem_ld16(t_addr + half * 128 + c * 16, v);
      tmem_wait_ld();
      if (c == 7) release();
      if (c == 4) {
        slab.store(p.C + (long long)m0 * p.ldc + n0, p.ldc, rows, p.N - n0);
        if constexpr (EPI == EPI_GATED_RESID) slab.fill(r1);
      }
      float f[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (n + i < p.N) f[i] += __bfloat162float(p.bias[n + i]);
      }
      if constexpr (EPI == EPI_GELU) {
#pragma unroll
        for (int i = 0; i < 16; ++i) f[i] = gelu_erf(f[i]);
      }
      if constexpr (EPI == EPI_GATED_RESID) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint4 rv = slab.get(lane, (c & 3) * 2 + q);
          const uint32_t ru[4] = {rv.x, rv.y, rv.z, rv.w};
          uint32_t gu[4] = {0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u};
          if (gate && gate_vec) {
            if (n + q * 8 < p.N) {
              const uint4 gv = *reinterpret_cast<const uint4*>(gate + n + q * 8);
              gu[0] = gv.x; gu[1] = gv.y; gu[2] = gv.z; gu[3] = gv.w;
            }
          } else if (gate) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (n + q * 8 + e < p.N)
                gu[e >> 1] = (gu[e >> 1] & (e & 1 ? 0x0000ffffu : 0xffff0000u)) |
                             (uint32_t(reinterpret_cast<const unsigned short*>(gate)[n + q * 8 + e]) << (16 * (e & 1)));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            f[q * 8 + e * 2] = bf16lo(ru[e]) + bf16lo(gu[e]) * f[q * 8 + e * 2];
            f[q * 8 + e * 2 + 1] = bf16hi(ru[e]) + bf16hi(gu[e]) * f[q * 8 + e * 2 + 1];
          }
        }
      }
      slab.put_bf16((c & 3) * 2, f);
      slab.put_bf16((c & 3) * 2 + 1, f + 8);
    }
    slab.store(p.C + (long long)m0 * p.ldc + n0 + 64, p.ldc, rows, p.N - n0 - 64);
    return true;
  }
  if constexpr (EPI == EPI_ATTN_P || EPI == EPI_ATTN_DS) {
    if (!wait()) return false;
    const bool row_ok = lane < rows;
    const float rv = p.rowvec[m];
    int lim = p.N;
    if (p.attn_mask == MASK_CAUSAL) lim = min(p.N, m + 1 + (p.N - p.M));
    if (p.attn_mask == MASK_MOT) lim = m < p.attn_n_ar ? m + 1 : p.N;
    const float sl2 = p.attn_scale * 1.4426950408889634f;
    const float rv2 = rv * 1.4426950408889634f;
#pragma unroll 1
    for (int c = 0; c < 128; c += 32) {
      const int n = n0 + c;
      if (n >= p.N) break;
      uint32_t v[32];
      tmem_ld32(t_addr + half * 128 + c, v);
      tmem_wait_ld();
      if (row_ok) {
        float f[32];
        const bool full32 = (n + 32 <= p.N);
        if constexpr (EPI == EPI_ATTN_P) {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            f[i] = (n + i < lim) ? exp2f(fmaf(__uint_as_float(v[i]), sl2, -rv2)) : 0.f;
        } else {
          const bf16* pr = p.R + (long long)m * p.ldr + n;
          if (full32) {
            const uint4* r4 = reinterpret_cast<const uint4*>(pr);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 rr = r4[q];
              const uint32_t ru[4] = {rr.x, rr.y, rr.z, rr.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                f[q * 8 + 2 * e] = bf16lo(ru[e]) * (__uint_as_float(v[q * 8 + 2 * e]) - rv) * p.attn_scale;
                f[q * 8 + 2 * e + 1] = bf16hi(ru[e]) * (__uint_as_float(v[q * 8 + 2 * e + 1]) - rv) * p.attn_scale;
              }
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              f[i] = (n + i < p.N) ? __bfloat162float(pr[i]) * (__uint_as_float(v[i]) - rv) * p.attn_scale : 0.f;
          }
        }
        bf16* dst = p.C + (long long)m * p.ldc + n;
        if (full32) {
          uint4* d4 = reinterpret_cast<uint4*>(dst);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 o;
            o.x = pack_bf16(f[q * 8 + 0], f[q * 8 + 1]);
            o.y = pack_bf16(f[q * 8 + 2], f[q * 8 + 3]);
            o.z = pack_bf16(f[q * 8 + 4], f[q * 8 + 5]);
            o.w = pack_bf16(f[q * 8 + 6], f[q * 8 + 7]);
            d4[q] = o;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (n + i < p.N) dst[i] = __float2bfloat16(f[i]);
        }
      }
    }
    release();
    return true;
  }
  return false;
}

template <int EPI, int NC, int NW>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmA1, const __grid_constant__ CUtensorMap tmB1,
                 const __grid_constant__ GemmGroup g) {
  static_assert(NW == 1 || NC == 2, "two column tiles per item need a CTA pair");
  using Cfg = GemmCfg<NC, NW>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr int B_BYTES = Cfg::B_BYTES;
  constexpr int STAGE_BYTES = Cfg::STAGE_BYTES;
  constexpr int TN = BN / NC * BK * 2;  // bytes of one column tile's B in this CTA
  constexpr int BARS = STAGES * STAGE_BYTES + Cfg::SLABS;  // offset of the barriers
  constexpr int TILE_M = BM * NC;  // rows of one output tile (of the CTA pair when NC == 2)
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t bar_base = smem_base + BARS;
  // CTA pair: rank 0 (the leader) issues the MMAs and owns the `full` and `tempty` barriers that
  // both CTAs signal; `empty` and `tfull` exist in both CTAs and the leader's commits reach both.
  const uint32_t cta_rank = NC == 2 ? cluster_ctarank() : 0u;
  const int first_tile = NC == 2 ? int(blockIdx.x >> 1) : int(blockIdx.x);
  const int tile_step = NC == 2 ? int(gridDim.x >> 1) : int(gridDim.x);
  // barriers: full[STAGES], empty[STAGES], tfull[2], tempty[2]; then tmem slot, abort flag
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + 2 + b); };
  const uint32_t tmem_slot = bar_base + 8u * (2 * STAGES + 4);
  uint8_t* gen_base = smem_raw + (smem_base - smem_u32(smem_raw));
  volatile int* abort_flag =
      reinterpret_cast<volatile int*>(gen_base + BARS + 8 * (2 * STAGES + 4) + 8);
  volatile uint32_t* tmem_slot_ptr =
      reinterpret_cast<volatile uint32_t*>(gen_base + BARS + 8 * (2 * STAGES + 4));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // the tile map's length is read before any programmatic-dependency wait: such launches are never programmatic
  const int m_tiles0 = g.p[0].tile_map ? *g.p[0].n_tiles_m : g.p[0].m_tiles;
  const int total_tiles = g.p[0].tile_map ? m_tiles0 * g.p[0].n_tiles * g.p[0].k_splits : g.total;
  const int tiles0 = g.p[0].tile_map ? total_tiles : g.tiles0;

  int prefetched = 0;  // stages whose B half thread 0 has requested ahead of the producer loop
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), EPI_WARPS * NC);
    }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
    if (g.total > g.tiles0) {
      prefetch_tmap(&tmA1);
      prefetch_tmap(&tmB1);
    }
    // Weight prefetch (single-CTA tiles, B in its [N, K] layout): the B halves of the first tile's first stages are
    // requested here, while warp 1 still allocates tensor memory and before the dependency wait, where B is known to be a weight
    // that no kernel before this one writes (early_b); their A halves follow in the producer loop. A stage's full barrier
    // completes when both have landed.
    if (NC == 1 && g.p[0].early_b && first_tile < total_tiles && first_tile < tiles0 && !g.p[0].b_mn &&
        !g.p[0].debug && !g.p[0].tile_map) {
      const GemmParams& p = g.p[0];
      const int k_blocks = (p.K + BK - 1) / BK;
      const int ks = first_tile % p.k_splits;
      const int kb0 = ks * k_blocks / p.k_splits, kb1 = (ks + 1) * k_blocks / p.k_splits;
      int tm, tn;
      tile_coords(first_tile / p.k_splits, p.m_tiles, p.n_tiles, tm, tn);
      const int n0 = (EPI == EPI_SWIGLU) ? tn * 128 : tn * BN;
      for (int kb = kb0; kb < kb1 && prefetched < STAGES; ++kb, ++prefetched) {
        const uint32_t sa = smem_base + prefetched * STAGE_BYTES;
        mbar_arrive_expect_tx(full_bar(prefetched), B_BYTES + p.a_rows * BK * 2);
        tma_load_2d(sa + A_BYTES, &tmB, full_bar(prefetched), kb * BK, n0);
        tma_load_2d(sa + A_BYTES + B_BYTES / 2, &tmB, full_bar(prefetched), kb * BK, n0 + p.b_row1);
      }
    }
  }
  if (warp == 1) {
    if constexpr (NC == 2) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (NC == 2) cluster_sync_all();  // the peer's barriers are initialised before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // The set-up above overlapped the previous kernel's tail (every launch but a grouped one is its programmatic dependent); the
  // successor may begin its own set-up now. Everybody waits for the previous kernel's results.
  pdl_launch_dependents();
  if (warp != 0) pdl_wait();

  if (warp == 0) {
    // ---------------- TMA producer. The whole warp walks the loop, so that barrier phases, addresses and coordinates are
    // warp-uniform values, and one elected lane issues the copies. With one lane alone in the loop, every operand of a copy went
    // through a vector register, and that thread's instructions, not the copies, bounded the delivery of operands to 41 B per
    // clock and SM: 880 x 4096 x 12288 95 us (with the products but no copies 68), now 76; 1920 x 6144 x 4096 with norm and
    // rotary embedding 105 -> 84.
    pdl_wait();
    prefetched = __shfl_sync(0xffffffffu, prefetched, 0);
    const bool issuer = elect_one();
    const uint32_t full0 = NC == 2 ? mapa(full_bar(0), 0) : full_bar(0);  // the pair's bytes are counted on the leader's barriers
    int it = 0, s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int t = first_tile; t < total_tiles && ok; t += tile_step) {
      const int second = t >= tiles0;
      const GemmParams& p = g.p[second];
      const CUtensorMap* mA = second ? &tmA1 : &tmA;
      const CUtensorMap* mB = second ? &tmB1 : &tmB;
      const int k_blocks = (p.K + BK - 1) / BK;
      const int tl = second ? t - tiles0 : t;
      const int ks = tl % p.k_splits;
      const int kb0 = ks * k_blocks / p.k_splits, kb1 = (ks + 1) * k_blocks / p.k_splits;
      int tm, tn;
      tile_coords(tl / p.k_splits, second ? p.m_tiles : m_tiles0, p.n_tiles, tm, tn);
      const TileRows tr = tile_rows<TILE_M>(p, tm);
      const int m0 = (p.debug & 1) ? 0 : tr.m0 + int(cta_rank) * BM;
      const int n0 = ((p.debug & 1) ? 0 : tr.b_row + ((EPI == EPI_SWIGLU) ? tn * NW * 128 : tn * NW * BN)) + int(cta_rank) * p.b_row1;
      if (p.debug & 2) continue;
      const bool a_mn = p.a_mn, b_mn = p.b_mn;
      const int b_row1 = p.b_row1;
      const uint32_t bytes = NC == 2 ? 2 * STAGE_BYTES : B_BYTES + p.a_rows * BK * 2;
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const uint32_t sa = smem_base + s * STAGE_BYTES, fb = full0 + 8u * s;
        // a prefetched stage is armed already and its B half in flight: only the A half is left
        const bool fresh = it >= prefetched;
        if (fresh && !__all_sync(0xffffffffu, mbar_wait(empty_bar(s), ph, abort_flag, p.status, ST_TIMEOUT_TMA))) {
          ok = false;
          break;
        }
        if (issuer) {
          const int k0 = kb * BK;
          if (fresh && (NC == 1 || cta_rank == 0)) mbar_arrive_expect_tx(full_bar(s), bytes);
          auto load = [&](uint32_t dst, const CUtensorMap* m, int x, int y) {
            if constexpr (NC == 2) tma_load_2d_pair(dst, m, fb, x, y);
            else tma_load_2d(dst, m, fb, x, y);
          };
          if (a_mn) {
            load(sa, mA, m0, k0);
            load(sa + A_BYTES / 2, mA, m0 + 64, k0);
          } else {
            load(sa, mA, k0, m0);
          }
          if constexpr (NC == 2) {
#pragma unroll
            for (int w = 0; w < NW; ++w) {
              // this CTA's 128 B rows (N columns) of each column tile
              const int nb = n0 + w * (EPI == EPI_SWIGLU ? 128 : BN);
              const uint32_t sb = sa + A_BYTES + w * TN;
              if (b_mn) {
                load(sb, mB, nb, k0);
                load(sb + TN / 2, mB, nb + 64, k0);
              } else {
                load(sb, mB, k0, nb);
              }
            }
          } else if (fresh) {
            if (b_mn) {
#pragma unroll
              for (int h = 0; h < 4; ++h) load(sa + A_BYTES + h * (B_BYTES / 4), mB, n0 + (h & 1) * 64 + (h >> 1) * b_row1, k0);
            } else {
              load(sa + A_BYTES, mB, k0, n0);
              load(sa + A_BYTES + B_BYTES / 2, mB, k0, n0 + b_row1);
            }
          }
        }
        __syncwarp();
        if (++s == STAGES) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    if (!ok && issuer) {
      // Drain our own copies in flight (bounded) before the CTA leaves.
      if (NC == 2 && cta_rank != 0) {
        // this CTA's copies are counted on the leader's barrier, which only the leader can wait
        // on: give them a fixed time (far beyond a copy's latency) to land instead
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) {}
      } else {
        volatile int no_abort = 0;
        const int first = it > STAGES ? it - STAGES : 0;
        for (int j = first; j < it; ++j)
          mbar_wait(full_bar(j % STAGES), (j / STAGES) & 1, &no_abort, nullptr, 0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (cta_rank == 0) {
      // ---------------- MMA issuer. The whole warp walks the loop, so barrier phases, descriptors and
      // addresses are warp-uniform values; one elected lane issues the tcgen05 instructions.
      // (instruction descriptor is built per tile: the operand majors are per-problem)
      int it = 0, tcount = 0;
      bool ok = true;
      for (int t = first_tile; t < total_tiles && ok; t += tile_step, ++tcount) {
        const int second = t >= tiles0;
        const GemmParams& p = g.p[second];
        const int k_blocks = (p.K + BK - 1) / BK;
        const int ks = (second ? t - tiles0 : t) % p.k_splits;
        const int kb0 = ks * k_blocks / p.k_splits, kb1 = (ks + 1) * k_blocks / p.k_splits;
        const int b = NW == 2 ? 0 : tcount & 1;
        const uint32_t bph = NW == 2 ? tcount & 1 : (tcount >> 1) & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(tempty_bar(b), bph ^ 1, abort_flag, p.status, ST_TIMEOUT_MMA))) break;
        tc_fence_after();
        const uint32_t a_step = p.a_mn ? 128u : 2u, b_step = p.b_mn ? 128u : 2u;
        const uint32_t idesc = make_idesc_bf16(TILE_M, BN, p.a_mn, p.b_mn);
        // the products of one stage with one column tile
        auto issue = [&](uint32_t sa, int w, bool first) {
          // K-major: 128-byte rows along K, +32 B per k-step. MN-major: 64-element chunks along M/N
          // 8 KB apart (LBO), k advances by rows of 128 B, +2048 B per k-step of 16.
          const uint32_t d_tmem = tmem_base + (NW == 2 ? w : b) * BN, sb = sa + A_BYTES + w * TN;
          const uint64_t adesc = p.a_mn ? make_smem_desc_sw128(sa, 8192, 1024) : make_smem_desc_sw128(sa, 16, 1024);
          const uint64_t bdesc = p.b_mn ? make_smem_desc_sw128(sb, 8192, 1024) : make_smem_desc_sw128(sb, 16, 1024);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            // advance 32 bytes (16 bf16) along K inside the 128-byte swizzle row: +2 in >>4 units
            if constexpr (NC == 2)
              mma_ss_pair(d_tmem, adesc + a_step * k, bdesc + b_step * k, idesc, (!first || k > 0) ? 1u : 0u);
            else
              mma_ss(d_tmem, adesc + a_step * k, bdesc + b_step * k, idesc, (!first || k > 0) ? 1u : 0u);
          }
        };
        for (int kb = kb0; kb < kb1;) {
          // k-blocks issued together: at the two ends of a 256x512 tile EDGE of them, first for one accumulator and then
          // for the other, so that a drain has EDGE x 512 clocks of the other accumulator's products to hide behind
          constexpr int EDGE = 2;
          const int nk = (NW == 2 && (kb == kb0 || kb + EDGE >= kb1)) ? min(EDGE, kb1 - kb) : 1;
          for (int j = 0; j < nk; ++j) {
            const int s = (it + j) % STAGES;
            const uint32_t ph = ((it + j) / STAGES) & 1;
            if (!(p.debug & 2) &&
                !__all_sync(0xffffffffu, mbar_wait(full_bar(s), ph, abort_flag, p.status, ST_TIMEOUT_MMA))) {
              ok = false;
              break;
            }
            tc_fence_after();
            if (elect_one()) {
              issue(smem_base + s * STAGE_BYTES, 0, kb + j == kb0);
              if constexpr (NW == 1) {
                if constexpr (NC == 2) tc_commit_both(empty_bar(s));  // frees the stage in both CTAs
                else tc_commit(empty_bar(s));
              }
            }
            __syncwarp();
          }
          if (!ok) break;
          if constexpr (NW == 2) {
            if (kb + nk == kb1) {
              if (elect_one()) tc_commit_both(tfull_bar(0));
              __syncwarp();
            }
            if (kb == kb0) {
              if (!__all_sync(0xffffffffu, mbar_wait(tempty_bar(1), bph ^ 1, abort_flag, p.status, ST_TIMEOUT_MMA))) {
                ok = false;
                break;
              }
              tc_fence_after();
            }
            if (elect_one()) {
              for (int j = 0; j < nk; ++j) {
                const int s = (it + j) % STAGES;
                issue(smem_base + s * STAGE_BYTES, 1, kb + j == kb0);
                tc_commit_both(empty_bar(s));
              }
            }
            __syncwarp();
          }
          kb += nk;
          it += nk;
        }
        if (ok) {
          if (elect_one()) {
            if constexpr (NC == 2) tc_commit_both(tfull_bar(NW == 2 ? 1 : b));
            else tc_commit(tfull_bar(b));
          }
          __syncwarp();
        }
      }
    }
  } else {
    // ---------------- epilogue warps (2..9); TMEM lane quadrant = warp % 4
    const int quad = warp & 3;
    const Slab slab{smem_base + STAGES * STAGE_BYTES + uint32_t(warp - 2) * 4096u, lane};
    float* sgamma = reinterpret_cast<float*>(gen_base + BARS + 256);
    if constexpr (EPI == EPI_QKV_ROPE) {   // one problem per launch (checked on the host)
      for (int i = threadIdx.x - 64; i < 256; i += EPI_WARPS * 32) {
        const bf16* gam = i < 128 ? g.p[0].gamma_q : g.p[0].gamma_k;
        sgamma[i] = gam ? __bfloat162float(gam[i & 127]) : 1.f;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_WARPS * 32) : "memory");
    }
    int tcount = 0;
    for (int t = first_tile; t < total_tiles; t += tile_step, ++tcount) {
      const int second = t >= tiles0;
      const GemmParams& p = g.p[second];
      const int tl = second ? t - tiles0 : t;
      int tm, tn;
      tile_coords(tl / p.k_splits, second ? p.m_tiles : m_tiles0, p.n_tiles, tm, tn);
      const TileRows tr = tile_rows<TILE_M>(p, tm);
      const int m0 = tr.m0 + int(cta_rank) * BM + quad * 32;
      bool ok = true;
#pragma unroll 1
      for (int w = 0; w < NW && ok; ++w) {
        const int half = (warp - 2) >> 2;
        const int b = NW == 2 ? w : tcount & 1;
        const uint32_t bph = NW == 2 ? tcount & 1 : (tcount >> 1) & 1;
        ok = finish_half<EPI>(
            p, slab, tmem_base + (uint32_t(quad * 32) << 16) + b * BN, half, m0, tr.m_end, tn * NW + w,
            tl % p.k_splits, sgamma,
            [&] {
              const bool up = __all_sync(0xffffffffu, mbar_wait(tfull_bar(b), bph, abort_flag, p.status, ST_TIMEOUT_EPI));
              tc_fence_after();
              return up;
            },
            [&] {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) {
                // the leader's MMA warp waits for both CTAs' epilogues
                if (NC == 2 && cta_rank != 0) mbar_arrive_cluster(mapa(tempty_bar(b), 0));
                else mbar_arrive(tempty_bar(b));
              }
            });
      }
      if (!ok) break;
    }
  }

  // ---------------- common tail
  tc_fence_before();
  __syncthreads();
  // neither CTA of a pair leaves (or frees tensor memory) while the other may still signal its
  // barriers or have MMAs in flight that read its shared memory
  if constexpr (NC == 2) cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if constexpr (NC == 2)
      tmem_dealloc_pair(tmem_base, 512);
    else
      tmem_dealloc(tmem_base, 512);
  }
}

// Second pass of split-K fused with the residual add and the RMS-norm that follow an output projection in a
// decode step: x = R + sum_ks partial[ks]; X[m] = x; H[m] = x * rsqrt(mean(x^2) + eps) * gamma. One CTA per row.
constexpr int RN_THREADS = 1024;
// One CTA of 1024 threads per row: a row of 4096 columns is one float4 per thread and split, and the loads of four
// splits are in flight together (with 256 threads and one split at a time the kernel took 13 us for 147 KB).
__global__ void __launch_bounds__(RN_THREADS)
splitk_reduce_rmsnorm_kernel(const float* __restrict__ partial, int k_splits, int M, int N, const bf16* __restrict__ R,
                             long long ldr, const bf16* __restrict__ gamma, float eps, bf16* __restrict__ X,
                             bf16* __restrict__ H, long long ldc) {
  __shared__ float red[RN_THREADS / 32];
  pdl_launch_dependents();
  pdl_wait();
  const int m = blockIdx.x, tid = threadIdx.x;
  const int nvec = N >> 2;
  constexpr int MAXJ = 2;  // N <= 8192
  float4 v[MAXJ];
  float ss = 0.f;
  const long long split_stride = (long long)M * N;
#pragma unroll
  for (int j = 0; j < MAXJ; ++j) {
    const int vi = tid + j * RN_THREADS;
    if (vi < nvec) {
      float4 a = make_float4(0, 0, 0, 0);
      const float* src = partial + (long long)m * N + vi * 4;
      int ks = 0;
      for (; ks + 4 <= k_splits; ks += 4) {
        const float4 x0 = *reinterpret_cast<const float4*>(src + (ks + 0) * split_stride);
        const float4 x1 = *reinterpret_cast<const float4*>(src + (ks + 1) * split_stride);
        const float4 x2 = *reinterpret_cast<const float4*>(src + (ks + 2) * split_stride);
        const float4 x3 = *reinterpret_cast<const float4*>(src + (ks + 3) * split_stride);
        a.x += (x0.x + x1.x) + (x2.x + x3.x); a.y += (x0.y + x1.y) + (x2.y + x3.y);
        a.z += (x0.z + x1.z) + (x2.z + x3.z); a.w += (x0.w + x1.w) + (x2.w + x3.w);
      }
      for (; ks < k_splits; ++ks) {
        const float4 x = *reinterpret_cast<const float4*>(src + ks * split_stride);
        a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
      }
      if (R) {
        const uint2 r = *reinterpret_cast<const uint2*>(R + (long long)m * ldr + vi * 4);
        a.x += bf16lo(r.x); a.y += bf16hi(r.x); a.z += bf16lo(r.y); a.w += bf16hi(r.y);
      }
      v[j] = a;
      ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int w = 0; w < RN_THREADS / 32; ++w) tot += red[w];
  const float rinv = rsqrtf(tot / N + eps);
#pragma unroll
  for (int j = 0; j < MAXJ; ++j) {
    const int vi = tid + j * RN_THREADS;
    if (vi < nvec) {
      const float4 a = v[j];
      uint2 xo, ho;
      xo.x = pack_bf16(a.x, a.y); xo.y = pack_bf16(a.z, a.w);
      float g0 = 1.f, g1 = 1.f, g2 = 1.f, g3 = 1.f;
      if (gamma) {
        const uint2 g = *reinterpret_cast<const uint2*>(gamma + vi * 4);
        g0 = bf16lo(g.x); g1 = bf16hi(g.x); g2 = bf16lo(g.y); g3 = bf16hi(g.y);
      }
      ho.x = pack_bf16(a.x * rinv * g0, a.y * rinv * g1);
      ho.y = pack_bf16(a.z * rinv * g2, a.w * rinv * g3);
      *reinterpret_cast<uint2*>(X + (long long)m * ldc + vi * 4) = xo;
      *reinterpret_cast<uint2*>(H + (long long)m * ldc + vi * 4) = ho;
    }
  }
}

// Second pass of split-K: out = epilogue(sum_ks partial[ks]). One thread per 4 output columns.
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ partial, int k_splits, int M, int N, int epi, bf16* __restrict__ C,
                     long long ldc, const bf16* __restrict__ bias, const bf16* __restrict__ R, long long ldr,
                     const bf16* __restrict__ gate, int rows_per_batch) {
  pdl_launch_dependents();
  pdl_wait();
  const int n_out = epi == EPI_SWIGLU ? N / 2 : N;
  const int vec_per_row = n_out / 4;
  const long long total = (long long)M * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int m = (int)(i / vec_per_row);
    const int n = (int)(i - (long long)m * vec_per_row) * 4;
    float4 a = make_float4(0, 0, 0, 0), u = make_float4(0, 0, 0, 0);
#pragma unroll 4
    for (int ks = 0; ks < k_splits; ++ks) {
      const float* row = partial + ((long long)ks * M + m) * N;
      const float4 x = *reinterpret_cast<const float4*>(row + n);
      a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
      if (epi == EPI_SWIGLU) {
        const float4 y = *reinterpret_cast<const float4*>(row + N / 2 + n);
        u.x += y.x; u.y += y.y; u.z += y.z; u.w += y.w;
      }
    }
    float f[4] = {a.x, a.y, a.z, a.w};
    if (epi == EPI_SWIGLU) {
      const float uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) f[e] = f[e] / (1.f + __expf(-f[e])) * uu[e];
    } else {
      if (bias) {
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] += __bfloat162float(bias[n + e]);
      }
      if (epi == EPI_GELU) {
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = gelu_erf(f[e]);
      }
      if (epi == EPI_GATED_RESID) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float gg = gate ? __bfloat162float(gate[(long long)(m / rows_per_batch) * N + n + e]) : 1.f;
          f[e] = __bfloat162float(R[(long long)m * ldr + n + e]) + gg * f[e];
        }
      }
    }
    uint2 o;
    o.x = pack_bf16(f[0], f[1]);
    o.y = pack_bf16(f[2], f[3]);
    *reinterpret_cast<uint2*>(C + (long long)m * ldc + n) = o;
  }
}

// Gates with the bit patterns first .. first + 16 n - 1: how many results of silu16 differ from the division's.
__global__ void __launch_bounds__(256)
silu_selftest_kernel(uint32_t first, long long n, unsigned long long* differ) {
  unsigned long long bad = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    uint32_t g[16];
    float o[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) g[e] = first + (uint32_t)(i * 16) + e;
    silu16(g, o);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float gv = __uint_as_float(g[e]), want = gv / (1.f + __expf(-gv));
      bad += __float_as_uint(o[e]) != __float_as_uint(want) && !(isnan(o[e]) && isnan(want));
    }
  }
  if (bad) atomicAdd(differ, bad);
}

}  // namespace cb

// ====================================================================== host
namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !ptr)
      throw std::runtime_error("cuTensorMapEncodeTiled entry point not found");
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}
}  // namespace

namespace cbh {
CUtensorMap make_tmap_bf16(const void* base, int rank, const uint64_t* dims,
                           const uint64_t* strides_bytes, const uint32_t* box, bool swizzle128) {
  CUtensorMap m;
  cuuint64_t gdim[5], gstr[5];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i + 1 < rank) gstr[i] = strides_bytes[i];
  }
  // The driver-API encode needs a current context in the calling thread; autograd's backward
  // threads may not have one bound yet, so bind the runtime's primary context once per thread.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaSetDevice(dev);
    cudaFree(nullptr);
    ctx_bound = true;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0)
    throw std::runtime_error("TMA base address must be 16-byte aligned");
  for (int i = 0; i + 1 < rank; ++i)
    if (gstr[i] % 16 != 0) throw std::runtime_error("TMA strides must be multiples of 16 bytes");
  CUresult r = get_encode()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base),
                            gdim, gstr, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw std::runtime_error("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return m;
}
const char* status_str(int st) {
  switch (st & 0xff) {  // the upper bits say which wait gave up
    case cb::ST_OK: return "ok";
    case cb::ST_TIMEOUT_TMA: return "timeout: TMA producer waiting for a free stage";
    case cb::ST_TIMEOUT_MMA: return "timeout: MMA issuer waiting for data";
    case cb::ST_TIMEOUT_EPI: return "timeout: epilogue waiting for accumulators";
    case cb::ST_TIMEOUT_SOFTMAX: return "timeout: softmax waiting for scores";
    case cb::ST_TIMEOUT_PEER: return "timeout: waiting for a peer signal";
    case cb::ST_BAD_ARG: return "bad argument";
  }
  return "unknown";
}
}  // namespace cbh

namespace cosmos {

// Debug knob (gemm_set_grid_limit): caps the number of persistent CTAs, which changes which CTA computes
// which tile and how many tiles share one CTA's pipeline state. Results must not depend on it.
static int g_grid_limit = 0;

static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = 148;  // no device visible (host-side use of the heuristics): a B200's count
    }
  }
  return n;
}

// Whether problems with more than one 128-row tile run on CTA pairs (COSMOS_GEMM_CTA_PAIR=0 keeps
// every launch on single CTAs, for A/B timing).
static int g_debug = 0;
static int g_tile_ctas = 0, g_tile_cols = 0;   // gemm_set_tile
static int g_pair = -1;
static bool pair_enabled() {
  if (g_pair < 0) {
    const char* e = std::getenv("COSMOS_GEMM_CTA_PAIR");
    g_pair = (e && e[0] == '0') ? 0 : 1;
  }
  return g_pair == 1;
}

template <int EPI, int NC, int NW>
static int max_grid() {
  // NC == 1: one CTA per SM. NC == 2: as many CTA pairs as the device can hold at once.
  static int n = 0;
  if (n) return n;
  cudaFuncSetAttribute(cb::gemm_bf16_kernel<EPI, NC, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (cb::GemmCfg<NC, NW>::SMEM + cb::gamma_smem(EPI)));
  if (NC == 1) {
    n = sm_count();
    return n;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sm_count() & ~1, 1, 1);
  cfg.blockDim = dim3(cb::GEMM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = (cb::GemmCfg<NC, NW>::SMEM + cb::gamma_smem(EPI));
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, cb::gemm_bf16_kernel<EPI, NC, NW>, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    clusters = sm_count() / 2;
  }
  if (clusters > sm_count() / 2) clusters = sm_count() / 2;
  n = 2 * clusters;
  return n;
}

// `units` = number of tiles (of CTA pairs when NC == 2); `limit` caps the number of CTAs (0 = none).
template <int EPI, int NC, int NW = 1>
static void launch(const CUtensorMap* maps, const cb::GemmGroup& g, int units, int limit, cudaStream_t stream) {
  int grid = max_grid<EPI, NC, NW>();
  if (limit > 0 && grid > limit) grid = limit;
  if (NC == 2) {
    grid &= ~1;
    if (grid < 2) grid = 2;
    if (grid > 2 * units) grid = 2 * units;
  } else if (grid > units) {
    grid = units;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(cb::GEMM_THREADS, 1, 1);
  cfg.dynamicSmemBytes = (cb::GemmCfg<NC, NW>::SMEM + cb::gamma_smem(EPI));
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = NC; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = g.p[0].tile_map || !early_on() ? 1 : 2;
  cudaLaunchKernelEx(&cfg, cb::gemm_bf16_kernel<EPI, NC, NW>, maps[0], maps[1], maps[2], maps[3], g);
}

template <int NC>
static void launch_epi(int epi, const CUtensorMap* maps, const cb::GemmGroup& g, int units, int limit,
                       cudaStream_t stream) {
  switch (epi) {
    case EPI_PLAIN: launch<EPI_PLAIN, NC>(maps, g, units, limit, stream); break;
    case EPI_GELU: launch<EPI_GELU, NC>(maps, g, units, limit, stream); break;
    case EPI_SWIGLU: launch<EPI_SWIGLU, NC>(maps, g, units, limit, stream); break;
    case EPI_GATED_RESID: launch<EPI_GATED_RESID, NC>(maps, g, units, limit, stream); break;
    case EPI_QKV_ROPE: launch<EPI_QKV_ROPE, NC>(maps, g, units, limit, stream); break;
    case EPI_ATTN_P: launch<EPI_ATTN_P, NC>(maps, g, units, limit, stream); break;
    case EPI_ATTN_DS: launch<EPI_ATTN_DS, NC>(maps, g, units, limit, stream); break;
    default: throw std::runtime_error("gemm_bf16: unknown epilogue");
  }
}

// Epilogues that exist for the 256x512 tile.
static void launch_wide(int epi, const CUtensorMap* maps, const cb::GemmGroup& g, int units, int limit, cudaStream_t stream) {
  switch (epi) {
    case EPI_PLAIN: launch<EPI_PLAIN, 2, 2>(maps, g, units, limit, stream); break;
    case EPI_GELU: launch<EPI_GELU, 2, 2>(maps, g, units, limit, stream); break;
    case EPI_SWIGLU: launch<EPI_SWIGLU, 2, 2>(maps, g, units, limit, stream); break;
    case EPI_GATED_RESID: launch<EPI_GATED_RESID, 2, 2>(maps, g, units, limit, stream); break;
    case EPI_QKV_ROPE: launch<EPI_QKV_ROPE, 2, 2>(maps, g, units, limit, stream); break;
    default: throw std::runtime_error("gemm_bf16: unknown epilogue");
  }
}
static bool wide_epi(int epi) {
  return epi == EPI_PLAIN || epi == EPI_GELU || epi == EPI_SWIGLU || epi == EPI_GATED_RESID || epi == EPI_QKV_ROPE;
}

static void fill_problem(const GemmArgs& a, cb::GemmParams& p, CUtensorMap& ta, CUtensorMap& tb, int nc = 1, int nw = 1) {
  // TMA needs 16-byte row strides; a ragged K is fine (out-of-range columns are zero-filled)
  if (a.lda % 8 != 0 || a.ldb % 8 != 0)
    throw std::runtime_error("gemm_bf16: leading dimensions must be multiples of 8");
  if (a.epi == EPI_SWIGLU && (a.N % 2 != 0 || (a.N / 2) % 8 != 0))
    throw std::runtime_error("gemm_bf16: SwiGLU epilogue needs N/2 to be a multiple of 8");
  if (a.epi == EPI_QKV_ROPE && a.N % 128 != 0)
    throw std::runtime_error("gemm_bf16: QKV epilogue needs N to be a multiple of 128");
  if ((a.epi == EPI_PLAIN || a.epi == EPI_GELU || a.epi == EPI_GATED_RESID) && (a.ldc % 8 != 0))
    throw std::runtime_error("gemm_bf16: ldc must be a multiple of 8");
  const uint64_t dimsA[2] = {(uint64_t)a.K, (uint64_t)a.M};
  const uint64_t strA[1] = {(uint64_t)a.lda * 2};
  const int a_rows = nc == 1 && a.M <= 16 && !a.a_mn && !a.tile_map ? (a.M + 7) / 8 * 8 : cb::BM;
  const uint32_t boxA[2] = {cb::BK, (uint32_t)a_rows};
  const uint64_t dimsB[2] = {(uint64_t)a.K, (uint64_t)a.N * (uint64_t)(a.tile_map ? a.n_groups : 1)};
  const uint64_t strB[1] = {(uint64_t)a.ldb * 2};
  const uint32_t boxB[2] = {cb::BK, 128};
  if (a.a_mn) {
    const uint64_t d[2] = {(uint64_t)a.M, (uint64_t)a.K};
    const uint32_t bx[2] = {64, cb::BK};
    ta = cbh::make_tmap_bf16(a.A, 2, d, strA, bx, true);
  } else {
    ta = cbh::make_tmap_bf16(a.A, 2, dimsA, strA, boxA, true);
  }
  if (a.b_mn) {
    const uint64_t d[2] = {(uint64_t)a.N, (uint64_t)a.K};
    const uint32_t bx[2] = {64, cb::BK};
    tb = cbh::make_tmap_bf16(a.B, 2, d, strB, bx, true);
  } else {
    tb = cbh::make_tmap_bf16(a.B, 2, dimsB, strB, boxB, true);
  }
  p = cb::GemmParams{};
  p.rowvec = a.rowvec; p.attn_scale = a.attn_scale; p.attn_mask = a.attn_mask; p.attn_n_ar = a.attn_n_ar;
  if ((a.epi == EPI_ATTN_P || a.epi == EPI_ATTN_DS) && (!a.rowvec || a.ldc % 8 != 0))
    throw std::runtime_error("gemm_bf16: attention-backward epilogues need a row vector and ldc % 8 == 0");
  if (a.epi == EPI_ATTN_DS && (!a.R || a.ldr % 8 != 0))
    throw std::runtime_error("gemm_bf16: the dS epilogue needs P as the residual operand");
  p.a_rows = a_rows;
  p.a_mn = a.a_mn ? 1 : 0;
  p.b_mn = a.b_mn ? 1 : 0;
  p.M = a.M; p.N = a.N; p.K = a.K;
  p.m_tiles = (a.M + cb::BM * nc - 1) / (cb::BM * nc);
  if (a.epi == EPI_SWIGLU) {
    p.n_tiles = (a.N / 2 + 128 * nw - 1) / (128 * nw);
    p.b_row1 = a.N / 2;
  } else {
    p.n_tiles = (a.N + cb::BN * nw - 1) / (cb::BN * nw);
    p.b_row1 = 128;
  }
  p.C = reinterpret_cast<bf16*>(a.C); p.ldc = a.ldc;
  p.bias = reinterpret_cast<const bf16*>(a.bias);
  p.R = reinterpret_cast<const bf16*>(a.R); p.ldr = a.ldr;
  p.gate = reinterpret_cast<const bf16*>(a.gate);
  p.rows_per_batch = a.rows_per_batch > 0 ? a.rows_per_batch : (a.M > 0 ? a.M : 1);
  p.route_ptr = a.route_ptr; p.route_ld = a.route_ld;
  p.route_rows = a.route_rows > 0 ? a.route_rows : (a.M > 0 ? a.M : 1);
  p.cos_tab = a.cos_tab; p.sin_tab = a.sin_tab; p.rope_rows = a.rope_rows > 0 ? a.rope_rows : 1;
  p.gamma_q = reinterpret_cast<const bf16*>(a.gamma_q);
  p.gamma_k = reinterpret_cast<const bf16*>(a.gamma_k);
  p.n_q_heads = a.n_q_heads; p.n_k_heads = a.n_k_heads; p.eps = a.eps;
  p.status = a.status;
  p.k_splits = 1;
  p.partial = nullptr;
  p.early_b = pdl_on() ? 1 : 0;
  p.debug = g_debug;
  p.tile_map = reinterpret_cast<const int4*>(a.tile_map);
  p.n_tiles_m = a.n_tiles_m;
  if (a.tile_map) {
    if (a.a_mn || a.b_mn || !a.n_tiles_m || a.n_groups < 1 || a.max_tiles_m < 1 || a.tile_m != cb::BM * nc ||
        (a.epi != EPI_PLAIN && a.epi != EPI_GELU) || (long long)a.N * a.n_groups > 0x7fffffffll)
      throw std::runtime_error("gemm_bf16: bad tile-map launch");
    p.m_tiles = a.max_tiles_m;   // upper bound for the grid; the kernel reads the count
  }
}

void gemm_set_grid_limit(int max_ctas) { g_grid_limit = max_ctas > 0 ? max_ctas : 0; }
int gemm_grid_limit() { return g_grid_limit; }
void gemm_set_tile(int ctas, int col_tiles) {
  if (!(ctas == 0 && col_tiles == 0) && !(ctas == 1 && col_tiles == 1) && !(ctas == 2 && (col_tiles == 1 || col_tiles == 2)))
    throw std::runtime_error("gemm_set_tile: (1, 1), (2, 1), (2, 2) or (0, 0)");
  g_tile_ctas = ctas;
  g_tile_cols = col_tiles;
}
void gemm_set_cta_pair(bool on) { g_pair = on ? 1 : 0; }
void gemm_set_debug(int bits) { g_debug = bits; }

void silu_selftest(uint32_t first, long long n, unsigned long long* differ, cudaStream_t stream) {
  if (n > 0) cb::silu_selftest_kernel<<<(int)std::min<long long>((n + 255) / 256, 148 * 8), 256, 0, stream>>>(first, n, differ);
}

int gemm_pick_k_splits(int M, int N, int K, int epi) {
  if (epi != EPI_PLAIN && epi != EPI_SWIGLU && epi != EPI_GATED_RESID && epi != EPI_GELU) return 1;
  const int m_tiles = (M + cb::BM - 1) / cb::BM;
  const int n_tiles = epi == EPI_SWIGLU ? (N / 2 + 127) / 128 : (N + cb::BN - 1) / cb::BN;
  const int tiles = m_tiles * n_tiles;
  const int k_blocks = (K + cb::BK - 1) / cb::BK;
  const int sms = sm_count();
  if (tiles >= sms || k_blocks < 8 || N % 8 != 0) return 1;
  if (tiles * 2 <= sms) {
    int ks = sms / tiles;                      // one wave: tiles * ks <= number of SMs
    if (ks > k_blocks / 4) ks = k_blocks / 4;  // at least 4 k-blocks (256 columns of K) per split
    if (ks > 32) ks = 32;
    return ks < 2 ? 1 : ks;
  }
  // Between half a wave and a full one (the 96 tiles of a 24576-wide SwiGLU projection leave 52 SMs idle and took
  // 59 us for 201 MB of weights): split so that the work items fill whole rounds of the persistent CTAs. Cost of a
  // choice = rounds x k-blocks per item; the smallest split count within 3 % of the best wins. Only for skinny
  // problems (at most two 128-row tiles), where the weights dominate the traffic; taller ones would pay more for
  // the fp32 partial sums than they gain.
  if (m_tiles > 2) return 1;
  int best = 1;
  double best_cost = (double)k_blocks;
  for (int ks = 2; ks <= 8 && ks <= k_blocks / 4; ++ks) {
    const int rounds = (tiles * ks + sms - 1) / sms;
    const double cost = rounds * (double)((k_blocks + ks - 1) / ks);
    if (cost < 0.97 * best_cost) {
      best = ks;
      best_cost = cost;
    }
  }
  return best;
}

// Tile of a problem taller than 128 rows: 128x256 on single CTAs (only for SwiGLU), 256x256 or 256x512 on CTA pairs. Cost of a
// launch: its rounds of the persistent CTAs times the time of a tile, in k-blocks of 256x256 (0.35 us: bound by the products). A
// 256x512 tile has twice the products, which take 1.85 times as long (48 KB of operands for 1024 clocks of products instead of
// 64 KB, and less power), but its accumulators are not double-buffered: its drain costs about 20 k-blocks, 10 more with norm and
// rotary embedding, against 2. A 128x256 tile is bound by its 48 KB of operands a k-block: 1.4. A last round that is not full
// costs about half of what it leaves idle (under the power cap the others clock higher). So wide tiles pay where K is long, and
// single CTAs where they fill two rounds that pairs fill to 2.6.
// Measured back to back, 256x256 and 256x512, us: N x K = 24576 x 4096 SwiGLU M 14080 2009 / 2117, M 1920 311 / 343; 4096 x 12288
// M 57600 4841 / 4656, M 14080 1076 / 1058, M 8448 (transposed weights) 679 / 649, M 2560 231 / 269; 4096 x 4096 M 3600 109 / 116; 6144 x 4096
// with norm and rotary embedding M 14080 565 / 669, M 1920 91 / 126. SwiGLU M 333 on single CTAs 76, on pairs 82, M 480 100 / 82.
static void pick_tile(const GemmArgs* args, int n, int limit, int& nc, int& nw) {
  nc = nw = 1;
  if (!pair_enabled() || (args[0].M <= cb::BM && (n < 2 || args[1].M <= cb::BM))) return;
  if (g_tile_ctas) {
    nc = g_tile_ctas;
    nw = wide_epi(args[0].epi) ? g_tile_cols : 1;
    return;
  }
  const int ctas = limit > 0 && limit < sm_count() ? limit : sm_count();
  const int epi = args[0].epi, k_blocks = (args[0].K + cb::BK - 1) / cb::BK;
  auto cost = [&](int c, int w, double per_kb, double per_tile) {
    long long tiles = 0;
    for (int i = 0; i < n; ++i) {
      const int cols = epi == EPI_SWIGLU ? args[i].N / 2 : args[i].N;
      const int tile_n = (epi == EPI_SWIGLU ? 128 : cb::BN) * w;
      tiles += (long long)((args[i].M + cb::BM * c - 1) / (cb::BM * c)) * ((cols + tile_n - 1) / tile_n);
    }
    const int at_once = ctas / c > 0 ? ctas / c : 1;
    const long long rounds = (tiles + at_once - 1) / at_once;
    return 0.5 * (rounds + double(tiles) / at_once) * (k_blocks * per_kb + per_tile);
  };
  nc = 2;
  nw = 1;
  double best = cost(2, 1, 1.0, 2.0);
  if (wide_epi(epi)) {
    const double wide = cost(2, 2, 1.85, epi == EPI_QKV_ROPE ? 30.0 : 20.0);
    if (wide < best) {
      nw = 2;
      best = wide;
    }
  }
  if (epi == EPI_SWIGLU && cost(1, 1, 1.4, 2.0) < best) nc = nw = 1;
}

void gemm_pick_tile(int M, int N, int K, int epi, int& ctas, int& col_tiles) {
  GemmArgs a;
  a.M = M; a.N = N; a.K = K; a.epi = epi;
  pick_tile(&a, 1, g_grid_limit, ctas, col_tiles);
}

// One launch for one or two problems that share the epilogue kind.
void gemm_bf16_grouped(const GemmArgs* args, int n, cudaStream_t stream) {
  if (n < 1 || n > 2) throw std::runtime_error("gemm_bf16_grouped: 1 or 2 problems per launch");
  if (n == 2 && args[0].epi != args[1].epi)
    throw std::runtime_error("gemm_bf16_grouped: both problems must use the same epilogue");
  const bool two = n == 2 && args[1].M > 0;
  if (args[0].epi == EPI_QKV_ROPE && two) throw std::runtime_error("gemm_bf16_grouped: the QKV epilogue takes one problem");
  if (args[0].tile_map && two) throw std::runtime_error("gemm_bf16_grouped: a tile map takes one problem");
  int limit = args[0].max_ctas > 0 ? args[0].max_ctas : 0;
  if (g_grid_limit > 0 && (limit == 0 || limit > g_grid_limit)) limit = g_grid_limit;
  int nc = args[0].tile_map ? args[0].tile_m / cb::BM : 1, nw = 1;
  if (!args[0].tile_map) pick_tile(args, two ? 2 : 1, limit, nc, nw);
  if (nc != 1 && nc != 2) throw std::runtime_error("gemm_bf16_grouped: tile rows must be 128 or 256");
  cb::GemmGroup g{};
  CUtensorMap maps[4];
  fill_problem(args[0], g.p[0], maps[0], maps[1], nc, nw);
  g.tiles0 = g.p[0].m_tiles * g.p[0].n_tiles;
  g.total = g.tiles0;
  if (two) {
    fill_problem(args[1], g.p[1], maps[2], maps[3], nc, nw);
    g.total += g.p[1].m_tiles * g.p[1].n_tiles;
  } else {
    maps[2] = maps[0];
    maps[3] = maps[1];
  }
  if (g.total == 0) return;
  if (nw == 2)
    launch_wide(args[0].epi, maps, g, g.total, limit, stream);
  else if (nc == 2)
    launch_epi<2>(args[0].epi, maps, g, g.total, limit, stream);
  else
    launch_epi<1>(args[0].epi, maps, g, g.total, limit, stream);
}

// CTAs of a split-K launch's tiles. More than one 128-row tile (a serving batch of 256): CTA pairs, so that each CTA stages half of the
// weight tile. The split count was chosen for single CTAs, so pairs can need a second, mostly empty round where those have one:
// 257 - 384 rows of a 4096-wide projection in three splits are 96 items on 74 pairs, or 144 on 148 CTAs whose k-block takes 1.4 times
// as long (see pick_tile). 333 x 4096 x 4096 with the reduction 36 us on pairs, 30 on single CTAs; 333 x 4096 x 12288 67 and 54.
static int split_ctas(int M, int N, int k_splits, int epi) {
  if (!pair_enabled() || epi == EPI_SWIGLU || M <= cb::BM) return 1;
  if (g_tile_ctas) return g_tile_ctas;
  auto rounds = [&](int c) {
    const long long items = (long long)((M + cb::BM * c - 1) / (cb::BM * c)) * ((N + cb::BN - 1) / cb::BN) * k_splits;
    return (items + sm_count() / c - 1) / (sm_count() / c);
  };
  return rounds(2) * 1.0 <= rounds(1) * 1.4 ? 2 : 1;
}
int gemm_pick_split_ctas(int M, int N, int K, int epi) { return split_ctas(M, N, gemm_pick_k_splits(M, N, K, epi), epi); }

void gemm_bf16(const GemmArgs& a, cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0) return;
  if (a.k_splits <= 1 && !a.partial_only) {
    gemm_bf16_grouped(&a, 1, stream);
    return;
  }
  // split-K: pass 1 writes fp32 partials, pass 2 reduces and applies the epilogue
  if (a.epi == EPI_QKV_ROPE) throw std::runtime_error("gemm_bf16: split-K does not support the QKV epilogue");
  if (!a.partial || a.N % 8 != 0) throw std::runtime_error("gemm_bf16: split-K needs a partial buffer and N % 8 == 0");
  cb::GemmGroup g{};
  CUtensorMap maps[4];
  const int nc = a.tile_map ? a.tile_m / cb::BM : split_ctas(a.M, a.N, a.k_splits, a.epi);
  if (nc != 1 && nc != 2) throw std::runtime_error("gemm_bf16: tile rows must be 128 or 256");
  fill_problem(a, g.p[0], maps[0], maps[1], nc);
  const int k_blocks = (a.K + cb::BK - 1) / cb::BK;
  const int ks = a.k_splits < 1 ? 1 : a.k_splits < k_blocks ? a.k_splits : k_blocks;
  g.p[0].k_splits = ks;
  g.p[0].partial = a.partial;
  g.tiles0 = g.total = g.p[0].m_tiles * g.p[0].n_tiles * ks;
  maps[2] = maps[0];
  maps[3] = maps[1];
  if (nc == 2) {
    switch (a.epi) {
      case EPI_PLAIN: launch<EPI_PLAIN, 2>(maps, g, g.total, 0, stream); break;
      case EPI_GELU: launch<EPI_GELU, 2>(maps, g, g.total, 0, stream); break;
      case EPI_GATED_RESID: launch<EPI_GATED_RESID, 2>(maps, g, g.total, 0, stream); break;
      default: throw std::runtime_error("gemm_bf16: unknown epilogue");
    }
  } else {
    switch (a.epi) {
      case EPI_PLAIN: launch<EPI_PLAIN, 1>(maps, g, g.total, 0, stream); break;
      case EPI_GELU: launch<EPI_GELU, 1>(maps, g, g.total, 0, stream); break;
      case EPI_SWIGLU: launch<EPI_SWIGLU, 1>(maps, g, g.total, 0, stream); break;
      case EPI_GATED_RESID: launch<EPI_GATED_RESID, 1>(maps, g, g.total, 0, stream); break;
      default: throw std::runtime_error("gemm_bf16: unknown epilogue");
    }
  }
  if (a.partial_only) return;
  if (a.norm_out) {
    if (a.epi != EPI_PLAIN || a.N > 8192 || a.N % 4 != 0 || a.ldc % 4 != 0 || (a.R && a.ldr % 4 != 0))
      throw std::runtime_error("gemm_bf16: the fused reduce + RMS-norm pass needs a plain epilogue and N <= 8192");
    launch_early(cb::splitk_reduce_rmsnorm_kernel, dim3(a.M), dim3(cb::RN_THREADS), 0, stream,
        a.partial, ks, a.M, a.N, reinterpret_cast<const bf16*>(a.R), a.ldr, reinterpret_cast<const bf16*>(a.norm_gamma),
        a.norm_eps, reinterpret_cast<bf16*>(a.C), reinterpret_cast<bf16*>(a.norm_out), a.ldc);
    return;
  }
  const int n_out = a.epi == EPI_SWIGLU ? a.N / 2 : a.N;
  const long long vecs = (long long)a.M * (n_out / 4);
  const int blocks = (int)std::min<long long>((vecs + 255) / 256, 148 * 8);
  launch_early(cb::splitk_reduce_kernel, dim3(blocks), dim3(256), 0, stream,
      a.partial, ks, a.M, a.N, a.epi, reinterpret_cast<bf16*>(a.C), a.ldc,
      reinterpret_cast<const bf16*>(a.bias), reinterpret_cast<const bf16*>(a.R), a.ldr,
      reinterpret_cast<const bf16*>(a.gate), a.rows_per_batch > 0 ? a.rows_per_batch : (a.M > 0 ? a.M : 1));
}

}  // namespace cosmos
