// Flash attention backward (head_dim 128, bf16, GQA) on tcgen05 tensor cores, as two kernels that
// need no atomics and no O(S^2) memory:
//
//   dK/dV kernel: one CTA owns a 128-row K/V tile (stationary in shared memory) and streams the
//   Q / dO tiles of every query head of its GQA group. Per tile pair
//       S^T  = K Q^T          (SS MMA)          dP^T = V dO^T             (SS MMA)
//       P^T  = exp2(S^T * scale*log2e - lse)    dS^T = P^T (dP^T - D) scale   (registers -> TMEM, bf16)
//       dV  += P^T dO         (TS MMA)          dK  += dS^T Q             (TS MMA)
//   The transposed products put the K/V rows on the TMEM lanes, so P^T and dS^T can feed the
//   accumulating MMAs straight from tensor memory (they alias S^T and dP^T), and dK / dV
//   accumulate in TMEM over the whole loop: 4 x 128 columns = the full 512.
//
//   dQ kernel: one CTA owns a 128-row Q / dO tile and streams K/V tiles:
//       S = Q K^T, dP = dO V^T (SS), dS = P (dP - D) scale -> TMEM (bf16), dQ += dS K (TS).
//
// A handoff between the tensor core and the element-wise warps takes 0.3 - 0.5 us, as long as the products of half a tile. So
// scores and score gradients are handed over separately, and neither waits for the other:
//   dK/dV: P^T written -> dV += P^T dO, next S^T; dS^T written -> dK += dS^T Q, next dP^T. The element-wise warps work on dS^T
//          while the next S^T is made and on the next P^T while the next dP^T is, in two 64-query halves of a warpgroup each.
//   dQ:    S and dP are free for the next tile as soon as they are in registers, because dS has tensor memory of its own
//          (two buffers), so both are a tile ahead of the element-wise warps.
// Q and dO (K and V) therefore live for different spans, and each has its own ring: three slots for the one that the last
// product of a tile pair reads, two for the other.
// 14080 queries x 14336 keys, 32 / 8 heads, against one handoff for both: dK/dV 6.82 -> 5.59 ms, dQ 4.21 -> 3.61 ms. The
// latter is 1.38 PFLOP/s of its three products, what cuBLAS sustains under the power cap (1.39); the former loses 1/7 to a
// last wave of 8 CTAs. Four element-wise warpgroups of 32 columns each in place of two of 64: 5.72 and 3.62 ms.
//
// Warp roles (384 threads): warp 0 TMA producer, warp 1 MMA issuer, warps 4..11 element-wise math
// and epilogue: two warpgroups, each thread owns one TMEM lane (a K/V row resp. a Q row) and one
// 64-column half of the score tile; in the dK/dV kernel a warpgroup writes its bf16 P / dS into the first half of its
// own fp32 score columns, so the two never touch each other's inputs.
// D = rowsum(dO * O) and the log-sum-exp of the forward pass come in as [B, Hq, Sq] fp32.
// Masks as in the forward kernel (full, causal, Mixture-of-Transformers block mask).
// Every wait is bounded; on expiry the kernel records a status code and unwinds.
#include "common.cuh"
#include "kernels.h"

namespace cb {

constexpr int BWD_THREADS = 384;
constexpr int BT = 128;                         // tile rows (queries and keys), = head_dim
constexpr int BTILE_BYTES = BT * 128 * 2;       // 32 KB
constexpr int BHALF_BYTES = BTILE_BYTES / 2;    // one 64-column half
constexpr int BWD_NA = 3, BWD_NB = 2;           // ring slots: tiles that the gradient product reads again, and the others
constexpr int BWD_TILES = 2 + BWD_NA + BWD_NB;  // two stationary tiles first
// 226 KB: no room to align the tiles by hand, so the kernels check that the runtime did (1024 bytes, the swizzle's period)
constexpr int BWD_SMEM = BWD_TILES * BTILE_BYTES + 4 * BT * 4 + 256;

struct AttnBwdParams {
  int Sq, Skv, Hq, Hkv, group;
  int mask, n_ar;
  float scale, scale_log2;
  const float* lse;    // [B, Hq, Sq] natural log
  const float* delta;  // [B, Hq, Sq]
  bf16* dQ;            // [B, Sq, Hq, 128] contiguous
  bf16* dK;            // [B, Skv, Hkv, 128] contiguous
  bf16* dV;
  int* status;
};

__device__ __forceinline__ bool bwd_masked(int kv, int q, const AttnBwdParams& p) {
  if (kv >= p.Skv) return true;
  if (p.mask == MASK_CAUSAL) return kv > q + (p.Skv - p.Sq);
  if (p.mask == MASK_MOT) return q < p.n_ar && kv > q;
  return false;
}

// True when some (kv, q) pair of the 128 x 128 tile pair is masked.
__device__ __forceinline__ bool bwd_tile_needs_mask(int kv0, int q0, const AttnBwdParams& p) {
  if (kv0 + BT > p.Skv) return true;
  if (p.mask == MASK_CAUSAL) return kv0 + BT - 1 > q0 + (p.Skv - p.Sq);
  if (p.mask == MASK_MOT) return q0 < p.n_ar && kv0 + BT - 1 > q0;
  return false;
}

__device__ __forceinline__ void named_bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

struct BwdSmem {
  uint32_t base;         // 1024-aligned shared address of the tile area
  uint32_t bar;          // first barrier
  __device__ uint32_t fixed(int t) const { return base + t * BTILE_BYTES; }                 // two stationary tiles
  __device__ uint32_t ring_a(int s) const { return base + (2 + s) * BTILE_BYTES; }
  __device__ uint32_t ring_b(int s) const { return base + (2 + BWD_NA + s) * BTILE_BYTES; }
  __device__ uint32_t at(int i) const { return bar + 8u * i; }
};

// barrier indices
constexpr int BB_FIXED = 0;                   // stationary tiles landed
constexpr int BB_FULL_A = 1;                  // + slot
constexpr int BB_EMPTY_A = BB_FULL_A + BWD_NA;
constexpr int BB_FULL_B = BB_EMPTY_A + BWD_NA;
constexpr int BB_EMPTY_B = BB_FULL_B + BWD_NB;
constexpr int BB_S = BB_EMPTY_B + BWD_NB;     // + half (dK/dV): scores ready (tcgen05.commit)
constexpr int BB_DP = BB_S + 2;               // + half (dK/dV): score gradients ready
constexpr int BB_P = BB_DP + 2;               // dK/dV, + half: P written. dQ: S read (0), dP read (1)
constexpr int BB_DS = BB_P + 2;               // dK/dV, + half: dS written. dQ: + buffer
constexpr int BB_DONE = BB_DS + 2;            // accumulators final
constexpr int BB_COUNT = BB_DONE + 1;
static_assert(8 * BB_COUNT + 16 <= 256, "barriers, tensor-memory slot and abort flag");
constexpr uint32_t HALF_ROWS_DESC = (64 * 128) >> 4;  // descriptor offset of rows 64.. of a K-major tile

// `arrivals`: threads behind each of the barriers BB_P and BB_DS
__device__ __forceinline__ void bwd_init_barriers(const BwdSmem& sm, volatile int* abort_flag, int arrivals) {
  for (int i = 0; i < BB_COUNT; ++i) mbar_init(sm.at(i), i >= BB_P && i < BB_DONE ? arrivals : 1);
  *abort_flag = 0;
  fence_barrier_init();
}

// Loads one 128 x 128 tile (two 64-column halves) of a [B, S, H, 128] tensor.
__device__ __forceinline__ void bwd_load_tile(uint32_t dst, const CUtensorMap* tm, uint32_t bar, int head, int row0,
                                              int batch) {
  tma_load_4d(dst, tm, bar, 0, head, row0, batch);
  tma_load_4d(dst + BHALF_BYTES, tm, bar, 64, head, row0, batch);
}

// The producer: the stationary tiles, then tile i of both streams, i = 0 .. n - 1; `coords(i, head, row)` says where it is.
// After a failed wait its own copies in flight must land before the CTA's shared memory is released.
template <class Coords>
__device__ __forceinline__ void bwd_produce(const BwdSmem& sm, const CUtensorMap* f0, const CUtensorMap* f1, int f_head, int f_row,
                                            const CUtensorMap* a, const CUtensorMap* b, int batch, int n, volatile int* abort_flag,
                                            int* status, Coords coords) {
  if (n <= 0) return;
  mbar_arrive_expect_tx(sm.at(BB_FIXED), 2 * BTILE_BYTES);
  bwd_load_tile(sm.fixed(0), f0, sm.at(BB_FIXED), f_head, f_row, batch);
  bwd_load_tile(sm.fixed(1), f1, sm.at(BB_FIXED), f_head, f_row, batch);
  int na = 0, nb = 0;
  for (; nb < n; ++nb) {
    int head, row;
    coords(nb, head, row);
    const int sa = na % BWD_NA, sb = nb % BWD_NB;
    if (!mbar_wait(sm.at(BB_EMPTY_A + sa), ((na / BWD_NA) & 1) ^ 1, abort_flag, status, ST_TIMEOUT_TMA)) break;
    mbar_arrive_expect_tx(sm.at(BB_FULL_A + sa), BTILE_BYTES);
    bwd_load_tile(sm.ring_a(sa), a, sm.at(BB_FULL_A + sa), head, row, batch);
    ++na;
    if (!mbar_wait(sm.at(BB_EMPTY_B + sb), ((nb / BWD_NB) & 1) ^ 1, abort_flag, status, ST_TIMEOUT_TMA)) break;
    mbar_arrive_expect_tx(sm.at(BB_FULL_B + sb), BTILE_BYTES);
    bwd_load_tile(sm.ring_b(sb), b, sm.at(BB_FULL_B + sb), head, row, batch);
  }
  if (nb == n) return;
  volatile int no_abort = 0;
  mbar_wait(sm.at(BB_FIXED), 0, &no_abort, nullptr, 0);
  for (int i = max(0, na - BWD_NA); i < na; ++i) mbar_wait(sm.at(BB_FULL_A + i % BWD_NA), (i / BWD_NA) & 1, &no_abort, nullptr, 0);
  for (int i = max(0, nb - BWD_NB); i < nb; ++i) mbar_wait(sm.at(BB_FULL_B + i % BWD_NB), (i / BWD_NB) & 1, &no_abort, nullptr, 0);
}

// fp32 accumulator row (this thread's TMEM lane, columns [c_begin, c_end) at `taddr`) -> bf16 at dst.
__device__ __forceinline__ void bwd_store_row(uint32_t taddr, bf16* dst, bool row_ok, int c_begin, int c_end) {
#pragma unroll 1
  for (int c = c_begin; c < c_end; c += 32) {
    uint32_t o[32];
    tmem_ld32(taddr + c, o);
    tmem_wait_ld();
    if (row_ok) {
      uint4* d4 = reinterpret_cast<uint4*>(dst + c);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 v;
        v.x = pack_bf16(__uint_as_float(o[q * 8 + 0]), __uint_as_float(o[q * 8 + 1]));
        v.y = pack_bf16(__uint_as_float(o[q * 8 + 2]), __uint_as_float(o[q * 8 + 3]));
        v.z = pack_bf16(__uint_as_float(o[q * 8 + 4]), __uint_as_float(o[q * 8 + 5]));
        v.w = pack_bf16(__uint_as_float(o[q * 8 + 6]), __uint_as_float(o[q * 8 + 7]));
        d4[q] = v;
      }
    }
  }
}

// ====================================================================== dK / dV
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                           const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                           const AttnBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const BwdSmem sm{smem_u32(smem_raw), smem_u32(smem_raw) + BWD_TILES * BTILE_BYTES + 4 * BT * 4};
  if (sm.base & 1023u) {   // the same for every thread
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_BAD_ARG);
    return;
  }
  float* lse_s = reinterpret_cast<float*>(smem_raw + BWD_TILES * BTILE_BYTES);  // [2][128], negated
  float* dlt_s = lse_s + 2 * BT;                                                // [2][128], negated
  const uint32_t tmem_slot = sm.at(BB_COUNT);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - sm.base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot_ptr + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kv0 = blockIdx.x * BT, kvh = blockIdx.y, batch = blockIdx.z;
  const int n_qt_all = (p.Sq + BT - 1) / BT;
  // leading query tiles that the mask removes completely for this K/V tile
  int i0 = 0;
  if (p.mask == MASK_CAUSAL) i0 = max(0, kv0 - (p.Skv - p.Sq)) / BT;
  if (p.mask == MASK_MOT) i0 = min(p.n_ar, kv0) / BT;
  i0 = min(i0, n_qt_all);
  const int n_qt = n_qt_all - i0;
  const int n_it = n_qt * p.group;

  if (threadIdx.x == 0) {
    bwd_init_barriers(sm, abort_flag, 128);
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmdO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  const uint32_t T_ST = tmem_base, T_DPT = tmem_base + 128, T_DV = tmem_base + 256, T_DK = tmem_base + 384;

  if (warp == 0 && lane == 0) {
    bwd_produce(sm, &tmK, &tmV, kvh, kv0, &tmQ, &tmdO, batch, n_it, abort_flag, p.status, [&](int it, int& head, int& row) {
      head = kvh * p.group + it / n_qt;
      row = (i0 + it % n_qt) * BT;
    });
  } else if (warp == 1) {
    // ---------------- MMA issuer: the whole warp walks the loop (barrier phases and descriptors are warp-uniform
    // values), one elected lane issues the tcgen05 instructions
    const bool issuer = elect_one();
    auto wait_all = [&](int bar, uint32_t phase) {
      const bool up = __all_sync(0xffffffffu, mbar_wait(sm.at(bar), phase, abort_flag, p.status, ST_TIMEOUT_MMA)) != 0;
      tc_fence_after();
      return up;
    };
    constexpr uint32_t idesc_ss = make_idesc_bf16(BT, 64, 0, 0);   // one 64-column half of the score tile
    constexpr uint32_t idesc_ts = make_idesc_bf16(BT, 128, 0, 1);
    // D[:, 64 h ..] = (stationary tile t) x (64 rows of the tile at `tile`)^T
    auto scores = [&](uint32_t d, int t, uint32_t tile, int h, int bar) {
      const uint64_t a = make_smem_desc_sw128(sm.fixed(t), 16, 1024);
      const uint64_t b = make_smem_desc_sw128(tile, 16, 1024) + uint64_t(h * HALF_ROWS_DESC);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const uint32_t off = (kk >> 2) * (BHALF_BYTES >> 4) + 2 * (kk & 3);
        mma_ss(d + 64 * h, a + off, b + off, idesc_ss, kk > 0 ? 1u : 0u);
      }
      tc_commit(sm.at(bar + h));
    };
    // D += (bf16 at 32-bit columns [64 h, 64 h + 32) of `a`) x (rows 64 h .. of the tile)
    auto grads = [&](uint32_t d, uint32_t a, uint32_t tile, int h, bool first) {
      const uint64_t b = make_smem_desc_sw128(tile, BHALF_BYTES, 1024);
#pragma unroll
      for (int k4 = 0; k4 < 4; ++k4)
        mma_ts(d, a + h * 64 + k4 * 8, b + uint64_t((4 * h + k4) * (2048 >> 4)), idesc_ts, (first && h == 0 && k4 == 0) ? 0u : 1u);
    };
    bool ok = n_it > 0 && wait_all(BB_FIXED, 0) && wait_all(BB_FULL_A, 0);
    if (ok && issuer) {
      scores(T_ST, 0, sm.ring_a(0), 0, BB_S);
      scores(T_ST, 0, sm.ring_a(0), 1, BB_S);
    }
    __syncwarp();
    ok = ok && wait_all(BB_FULL_B, 0);
    if (ok && issuer) {
      scores(T_DPT, 1, sm.ring_b(0), 0, BB_DP);
      scores(T_DPT, 1, sm.ring_b(0), 1, BB_DP);
    }
    __syncwarp();
    for (int it = 0; it < n_it && ok; ++it) {
      const int a = it % BWD_NA, b = it % BWD_NB, an = (it + 1) % BWD_NA, bn = (it + 1) % BWD_NB;
      const bool more = it + 1 < n_it;
      // Q and dO of the next tile pair are waited for where its first product is issued. In issue order, the next scores
      // stand behind the product that reads this half's P^T (dS^T) from the columns that they overwrite.
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ok = ok && wait_all(BB_P + h, it & 1);
        if (ok && issuer) {
          grads(T_DV, T_ST, sm.ring_b(b), h, it == 0);
          if (h == 1) tc_commit(sm.at(BB_EMPTY_B + b));
        }
        if (more && h == 0) ok = ok && wait_all(BB_FULL_A + an, ((it + 1) / BWD_NA) & 1);
        if (more && ok && issuer) scores(T_ST, 0, sm.ring_a(an), h, BB_S);
        __syncwarp();
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ok = ok && wait_all(BB_DS + h, it & 1);
        if (ok && issuer) {
          grads(T_DK, T_DPT, sm.ring_a(a), h, it == 0);
          if (h == 1) tc_commit(sm.at(BB_EMPTY_A + a));
        }
        if (more && h == 0) ok = ok && wait_all(BB_FULL_B + bn, ((it + 1) / BWD_NB) & 1);
        if (more && ok && issuer) scores(T_DPT, 1, sm.ring_b(bn), h, BB_DP);
        __syncwarp();
      }
    }
    if (ok && issuer) tc_commit(sm.at(BB_DONE));
    __syncwarp();
  } else if (warp >= 4) {
    // ---------------- element-wise math: this thread owns K/V row kv0 + r (TMEM lane r)
    const int quad = warp & 3;
    const int wg = (warp - 4) >> 2;  // which 64-column half of the score tile
    const int r = quad * 32 + lane;
    const int kv = kv0 + r;
    const uint32_t half_addr = (uint32_t(quad * 32) << 16) + 64 * wg;
    const uint32_t lane_addr = uint32_t(quad * 32) << 16;
    const uint64_t scale_log2 = pack2(p.scale_log2, p.scale_log2), scale = pack2(p.scale, p.scale);
    auto query0 = [&](int it) { return (i0 + it % n_qt) * BT; };
    // log-sum-exp and D of this warpgroup's 64 query columns, fetched an iteration ahead by its first 64 threads
    float l_next = 0.f, d_next = 0.f;
    auto fetch = [&](int it) {
      const int qi = query0(it) + 64 * wg + r;
      const long long off = ((long long)batch * p.Hq + kvh * p.group + it / n_qt) * p.Sq + qi;
      l_next = qi < p.Sq ? p.lse[off] * -1.4426950408889634f : -INFINITY;
      d_next = qi < p.Sq ? -p.delta[off] : 0.f;
    };
    auto put = [&](int it) {
      lse_s[(it & 1) * BT + 64 * wg + r] = l_next;
      dlt_s[(it & 1) * BT + 64 * wg + r] = d_next;
    };
    if (r < 64 && n_it > 0) {
      fetch(0);
      put(0);
    }
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int q0 = query0(it);
      // this iteration's rows are in place, and nobody still reads the buffer that the next iteration's go to
      named_bar_sync(1 + wg, 128);
      if (r < 64 && it + 1 < n_it) fetch(it + 1);
      const float4* ls = reinterpret_cast<const float4*>(lse_s + (it & 1) * BT + 64 * wg);
      const float4* dl = reinterpret_cast<const float4*>(dlt_s + (it & 1) * BT + 64 * wg);
      ok = ok && mbar_wait(sm.at(BB_S + wg), it & 1, abort_flag, p.status, ST_TIMEOUT_SOFTMAX);
      ok = __all_sync(0xffffffffu, ok);   // a warp that gave up keeps to the barriers of its warpgroup
      float pr[64];
      if (ok) {
        tc_fence_after();
        const bool need_mask = bwd_tile_needs_mask(kv0, q0, p);
        uint32_t pk[32];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t s[32];
          tmem_ld32(T_ST + half_addr + hh * 32, s);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 l4 = ls[hh * 8 + i / 4];
            const float2 x = unpack2(fma2(pack2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), scale_log2, pack2(l4.x, l4.y)));
            const float2 y = unpack2(fma2(pack2(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])), scale_log2, pack2(l4.z, l4.w)));
            pr[hh * 32 + i] = ex2(x.x);
            pr[hh * 32 + i + 1] = ex2(x.y);
            pr[hh * 32 + i + 2] = ex2(y.x);
            pr[hh * 32 + i + 3] = ex2(y.y);
          }
        }
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (bwd_masked(kv, q0 + 64 * wg + i, p)) pr[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = pack_bf16(pr[2 * i], pr[2 * i + 1]);
        // bf16 P^T aliases the fp32 scores: the 64 columns of this warpgroup become the first 32 of them, which only covers
        // scores that this thread already holds. dS^T does the same below.
        tmem_st32(T_ST + half_addr, pk);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(sm.at(BB_P + wg));
      }
      ok = ok && mbar_wait(sm.at(BB_DP + wg), it & 1, abort_flag, p.status, ST_TIMEOUT_SOFTMAX);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
        uint32_t dsk[32];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          uint32_t dp[32];
          tmem_ld32(T_DPT + half_addr + hh * 32, dp);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 d4 = dl[hh * 8 + i / 4];
            const int c = hh * 32 + i;
            const uint64_t x = add2(pack2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), pack2(d4.x, d4.y));
            const uint64_t y = add2(pack2(__uint_as_float(dp[i + 2]), __uint_as_float(dp[i + 3])), pack2(d4.z, d4.w));
            const float2 u = unpack2(mul2(mul2(pack2(pr[c], pr[c + 1]), x), scale));
            const float2 v = unpack2(mul2(mul2(pack2(pr[c + 2], pr[c + 3]), y), scale));
            dsk[c / 2] = pack_bf16(u.x, u.y);
            dsk[c / 2 + 1] = pack_bf16(v.x, v.y);
          }
        }
        tmem_st32(T_DPT + half_addr, dsk);
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(sm.at(BB_DS + wg));
      }
      if (r < 64 && it + 1 < n_it) put(it + 1);
    }
    const bool row_ok = kv < p.Skv;
    bf16* dk_row = p.dK + (((long long)batch * p.Skv + kv) * p.Hkv + kvh) * 128;
    bf16* dv_row = p.dV + (((long long)batch * p.Skv + kv) * p.Hkv + kvh) * 128;
    if (n_it == 0) {
      if (row_ok) {
        for (int c = 0; c < 16; ++c) reinterpret_cast<uint4*>(wg == 0 ? dv_row : dk_row)[c] = make_uint4(0, 0, 0, 0);
      }
    } else {
      ok = ok && mbar_wait(sm.at(BB_DONE), 0, abort_flag, p.status, ST_TIMEOUT_SOFTMAX);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after();
        // one accumulator per warpgroup
        if (wg == 0) bwd_store_row(T_DV + lane_addr, dv_row, row_ok, 0, 128);
        else bwd_store_row(T_DK + lane_addr, dk_row, row_ok, 0, 128);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ====================================================================== dQ
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                         const AttnBwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const BwdSmem sm{smem_u32(smem_raw), smem_u32(smem_raw) + BWD_TILES * BTILE_BYTES + 4 * BT * 4};
  if (sm.base & 1023u) {   // the same for every thread
    if (threadIdx.x == 0) atomicCAS(p.status, 0, ST_BAD_ARG);
    return;
  }
  const uint32_t tmem_slot = sm.at(BB_COUNT);
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(smem_raw + (tmem_slot - sm.base));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot_ptr + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q0 = blockIdx.x * BT, head = blockIdx.y, batch = blockIdx.z;
  const int kvh = head / p.group;
  int n_blocks;
  {
    const int last_row = min(p.Sq - 1, q0 + BT - 1);
    int lim = p.Skv;
    if (p.mask == MASK_CAUSAL) lim = min(p.Skv, last_row + 1 + (p.Skv - p.Sq));
    if (p.mask == MASK_MOT) lim = (last_row >= p.n_ar) ? p.Skv : last_row + 1;
    n_blocks = (max(lim, 1) + BT - 1) / BT;
  }

  if (threadIdx.x == 0) {
    bwd_init_barriers(sm, abort_flag, 256);
    prefetch_tmap(&tmQ);
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmdO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  const uint32_t T_S = tmem_base, T_DP = tmem_base + 128, T_DQ = tmem_base + 256, T_DS = tmem_base + 384;

  if (warp == 0 && lane == 0) {
    bwd_produce(sm, &tmQ, &tmdO, head, q0, &tmK, &tmV, batch, n_blocks, abort_flag, p.status, [&](int j, int& h, int& row) {
      h = kvh;
      row = j * BT;
    });
  } else if (warp == 1) {
    // ---------------- MMA issuer (whole warp walks the loop, one elected lane issues)
    const bool issuer = elect_one();
    auto wait_all = [&](int bar, uint32_t phase) {
      const bool up = __all_sync(0xffffffffu, mbar_wait(sm.at(bar), phase, abort_flag, p.status, ST_TIMEOUT_MMA)) != 0;
      tc_fence_after();
      return up;
    };
    constexpr uint32_t idesc_ss = make_idesc_bf16(BT, 128, 0, 0);
    constexpr uint32_t idesc_ts = make_idesc_bf16(BT, 128, 0, 1);
    // D = (stationary tile t) x (tile)^T
    auto scores = [&](uint32_t d, int t, uint32_t tile, int bar) {
      const uint64_t a = make_smem_desc_sw128(sm.fixed(t), 16, 1024), b = make_smem_desc_sw128(tile, 16, 1024);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const uint32_t off = (kk >> 2) * (BHALF_BYTES >> 4) + 2 * (kk & 3);
        mma_ss(d, a + off, b + off, idesc_ss, kk > 0 ? 1u : 0u);
      }
      tc_commit(sm.at(bar));
    };
    bool ok = wait_all(BB_FIXED, 0) && wait_all(BB_FULL_A, 0);
    if (ok && issuer) scores(T_S, 0, sm.ring_a(0), BB_S);
    __syncwarp();
    ok = ok && wait_all(BB_FULL_B, 0);
    if (ok && issuer) {
      scores(T_DP, 1, sm.ring_b(0), BB_DP);
      tc_commit(sm.at(BB_EMPTY_B));
    }
    __syncwarp();
    for (int j = 0; j < n_blocks && ok; ++j) {
      const int a = j % BWD_NA, an = (j + 1) % BWD_NA, bn = (j + 1) % BWD_NB;
      if (j + 1 < n_blocks) {   // both products of the next tile, once this tile's are in registers
        ok = wait_all(BB_FULL_A + an, ((j + 1) / BWD_NA) & 1) && wait_all(BB_P, j & 1);
        if (ok && issuer) scores(T_S, 0, sm.ring_a(an), BB_S);
        __syncwarp();
        ok = ok && wait_all(BB_FULL_B + bn, ((j + 1) / BWD_NB) & 1) && wait_all(BB_P + 1, j & 1);
        if (ok && issuer) {
          scores(T_DP, 1, sm.ring_b(bn), BB_DP);
          tc_commit(sm.at(BB_EMPTY_B + bn));
        }
        __syncwarp();
      }
      // dQ += dS K. The commit of a later dP also says that this product has read its dS buffer: the element-wise warps write
      // the buffer again only after dP of tile j + 2, which is issued behind it.
      ok = ok && wait_all(BB_DS + (j & 1), (j >> 1) & 1);
      if (ok && issuer) {
        const uint64_t k_mn = make_smem_desc_sw128(sm.ring_a(a), BHALF_BYTES, 1024);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          mma_ts(T_DQ, T_DS + (j & 1) * 64 + kk * 8, k_mn + uint64_t(kk * (2048 >> 4)), idesc_ts, (j == 0 && kk == 0) ? 0u : 1u);
        tc_commit(sm.at(BB_EMPTY_A + a));
      }
      __syncwarp();
    }
    if (ok && issuer) tc_commit(sm.at(BB_DONE));
    __syncwarp();
  } else if (warp >= 4) {
    // ---------------- element-wise math: this thread owns query row q0 + r (TMEM lane r)
    const int quad = warp & 3;
    const int wg = (warp - 4) >> 2;  // which 64-column half of the score tile
    const int r = quad * 32 + lane;
    const int qi = q0 + r;
    const uint32_t lane_addr = uint32_t(quad * 32) << 16;
    const bool row_ok = qi < p.Sq;
    const long long off = ((long long)batch * p.Hq + head) * p.Sq + qi;
    const float lse2 = row_ok ? p.lse[off] * -1.4426950408889634f : -INFINITY;
    const float dlt = row_ok ? -p.delta[off] : 0.f;
    const uint64_t lse_2 = pack2(lse2, lse2), dlt_2 = pack2(dlt, dlt);
    const uint64_t scale_log2 = pack2(p.scale_log2, p.scale_log2), scale = pack2(p.scale, p.scale);
    bool ok = true;
    for (int j = 0; j < n_blocks; ++j) {
      ok = mbar_wait(sm.at(BB_S), j & 1, abort_flag, p.status, ST_TIMEOUT_SOFTMAX);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int kv0 = j * BT;
      float pr[64];
      {
        uint32_t s[2][32];
        tmem_ld32(T_S + lane_addr + 64 * wg, s[0]);
        tmem_ld32(T_S + lane_addr + 64 * wg + 32, s[1]);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(sm.at(BB_P));
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
          const uint64_t x = pack2(__uint_as_float(s[i >> 5][i & 31]), __uint_as_float(s[i >> 5][(i & 31) + 1]));
          const float2 e = unpack2(fma2(x, scale_log2, lse_2));
          pr[i] = ex2(e.x);
          pr[i + 1] = ex2(e.y);
        }
      }
      if (bwd_tile_needs_mask(kv0, q0, p)) {
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (bwd_masked(kv0 + 64 * wg + i, qi, p)) pr[i] = 0.f;
      }
      ok = mbar_wait(sm.at(BB_DP), j & 1, abort_flag, p.status, ST_TIMEOUT_SOFTMAX);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t dsk[32];
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        uint32_t dp[32];
        tmem_ld32(T_DP + lane_addr + 64 * wg + hh * 32, dp);
        tmem_wait_ld();
        if (hh == 1) {
          tc_fence_before();
          mbar_arrive(sm.at(BB_P + 1));
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const uint64_t x = add2(pack2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), dlt_2);
          const float2 u = unpack2(mul2(mul2(pack2(pr[hh * 32 + i], pr[hh * 32 + i + 1]), x), scale));
          dsk[(hh * 32 + i) / 2] = pack_bf16(u.x, u.y);
        }
      }
      tmem_st32(T_DS + lane_addr + 64 * (j & 1) + 32 * wg, dsk);
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(sm.at(BB_DS + (j & 1)));
    }
    ok = ok && mbar_wait(sm.at(BB_DONE), 0, abort_flag, p.status, ST_TIMEOUT_SOFTMAX);
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      tc_fence_after();
      bf16* dq_row = p.dQ + (((long long)batch * p.Sq + qi) * p.Hq + head) * 128;
      bwd_store_row(T_DQ + lane_addr, dq_row, row_ok, 64 * wg, 64 * wg + 64);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace cb

namespace cosmos {

static CUtensorMap bwd_map(const void* base, int B, int S, int H, long long sb, long long ss, long long sh) {
  const uint64_t dims[4] = {128, (uint64_t)H, (uint64_t)S, (uint64_t)B};
  const uint64_t strides[3] = {(uint64_t)sh * 2, (uint64_t)ss * 2, (uint64_t)(sb > 0 ? sb : ss * S) * 2};
  const uint32_t box[4] = {64, 1, 128, 1};
  return cbh::make_tmap_bf16(base, 4, dims, strides, box, true);
}

void flash_attn_bwd(const AttnBwdArgs& a, cudaStream_t stream) {
  if (a.Hkv <= 0 || a.Hq % a.Hkv != 0) throw std::runtime_error("flash_attn_bwd: Hq % Hkv != 0");
  if (a.Sq <= 0 || a.Skv <= 0 || a.B <= 0) return;
  if (a.mask == MASK_CAUSAL && a.Skv < a.Sq) throw std::runtime_error("flash_attn_bwd: causal mask needs Skv >= Sq");
  if (a.mask == MASK_MOT && a.Skv != a.Sq) throw std::runtime_error("flash_attn_bwd: MoT mask needs Skv == Sq");
  static thread_local bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(cb::flash_attn_bwd_dkdv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cb::BWD_SMEM);
    cudaFuncSetAttribute(cb::flash_attn_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cb::BWD_SMEM);
    configured = true;
  }
  CUtensorMap tq = bwd_map(a.Q, a.B, a.Sq, a.Hq, a.q_stride_b, a.q_stride_s, a.q_stride_h);
  CUtensorMap tk = bwd_map(a.K, a.B, a.Skv, a.Hkv, a.k_stride_b, a.k_stride_s, a.k_stride_h);
  CUtensorMap tv = bwd_map(a.V, a.B, a.Skv, a.Hkv, a.v_stride_b, a.v_stride_s, a.v_stride_h);
  CUtensorMap tdo = bwd_map(a.dO, a.B, a.Sq, a.Hq, a.do_stride_b, a.do_stride_s, a.do_stride_h);
  cb::AttnBwdParams p{};
  p.Sq = a.Sq; p.Skv = a.Skv; p.Hq = a.Hq; p.Hkv = a.Hkv; p.group = a.Hq / a.Hkv;
  p.mask = a.mask; p.n_ar = a.n_ar;
  p.scale = a.scale; p.scale_log2 = a.scale * 1.4426950408889634f;
  p.lse = a.lse; p.delta = a.delta;
  p.dQ = reinterpret_cast<bf16*>(a.dQ); p.dK = reinterpret_cast<bf16*>(a.dK); p.dV = reinterpret_cast<bf16*>(a.dV);
  p.status = a.status;
  dim3 grid_kv((a.Skv + cb::BT - 1) / cb::BT, a.Hkv, a.B);
  cb::flash_attn_bwd_dkdv_kernel<<<grid_kv, cb::BWD_THREADS, cb::BWD_SMEM, stream>>>(tq, tk, tv, tdo, p);
  dim3 grid_q((a.Sq + cb::BT - 1) / cb::BT, a.Hq, a.B);
  cb::flash_attn_bwd_dq_kernel<<<grid_q, cb::BWD_THREADS, cb::BWD_SMEM, stream>>>(tq, tk, tv, tdo, p);
}

}  // namespace cosmos
