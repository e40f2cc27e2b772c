// The small kernels at both ends of a step: rotary tables, what a decode step needs before its layers, and its greedy choice.
// Each was a chain of ten or so torch kernels of 1 - 4 us on a few kilobytes, with a gap behind every one; launches count there, not
// bytes. All start behind the end of the kernel before them (launch.cuh).
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"
#include "launch.cuh"

namespace cb {

// cos, sin [S, half] of pos[axis(i)][s] * theta^(-2 i / head_dim), the angle in fp64 as the positions of long videos need. Axis of
// frequency i: T, H, W, T, H, W, ... while H (below h3) and W (below w3) last, then T. The frequencies are worked out once
// per block, before the positions are waited for. It was 14 kernels of 1 - 4 us; with it a prefill of 333 tokens takes 1066 us, without 1134.
constexpr int ROPE_HALF_MAX = 256;

__global__ void __launch_bounds__(256)
rope_tables_kernel(const long long* __restrict__ pos, int S, int half, double theta, int head_dim, int h3, int w3,
                   float* __restrict__ cos_t, float* __restrict__ sin_t) {
  __shared__ double inv[ROPE_HALF_MAX];
  pdl_launch_dependents();
  for (int i = threadIdx.x; i < half; i += 256) inv[i] = 1.0 / pow(theta, (double)i * 2.0 / (double)head_dim);
  __syncthreads();
  pdl_wait();
  const long long total = (long long)S * half;
  for (long long e = (long long)blockIdx.x * 256 + threadIdx.x; e < total; e += (long long)gridDim.x * 256) {
    const int i = int(e % half);
    const long long s = e / half;
    const int axis = i % 3 == 1 && i < h3 ? 1 : i % 3 == 2 && i < w3 ? 2 : 0;
    const double ang = (double)pos[axis * (long long)S + s] * inv[i];
    cos_t[e] = (float)cos(ang);
    sin_t[e] = (float)sin(ang);
  }
}

// One block per sequence: rotary tables of its position, the cache slot of the new token, its embedding, and the length moved on.
// Ids are compared with their limits before they become addresses, and a bad one is reported. Row 0 stands in for a bad token. A
// position past the table's row, and a page that is none of the cache's (unused entries are -1), give slot -1, for which the
// layers store nothing, and the length stays where it is, inside the row, so that attention reads no further either.
// The kernels behind may start only once this one's wait is over: the layers' GEMMs request weights ahead of their own waits, so
// everything that ran before the step (which may have written these weights) must be complete when the first of them starts. In a
// captured step the later trigger costs nothing that shows: batch 1 over 1500 tokens 993 us either way, batch 32 over 8448 2321 and 2322.
__global__ void __launch_bounds__(256) decode_begin_kernel(const cosmos::DecodeBeginArgs a) {
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.x, tid = threadIdx.x;
  const long long pos = a.lens[b];
  const float rpos = (float)(a.pos_delta ? pos + a.pos_delta[b] : pos);
  for (int i = tid; i < a.half; i += 256) {
    const float ang = rpos * a.inv_freq[i];
    a.cos_t[(long long)b * a.half + i] = cosf(ang);
    a.sin_t[(long long)b * a.half + i] = sinf(ang);
  }
  long long tok = a.tokens[b];
  if (tok < 0) tok += a.vocab;   // as an index of torch: -1 is the last row
  if (tok < 0 || tok >= a.vocab) {
    if (tid == 0) atomicCAS(a.status, 0, ST_BAD_INDEX | (SITE_STACK_TOKEN << 8));
    tok = 0;
  }
  const uint4* src = reinterpret_cast<const uint4*>((const bf16*)a.embed + tok * a.embed_stride);
  uint4* dst = reinterpret_cast<uint4*>((bf16*)a.x + (long long)b * a.d);
  for (int i = tid; i < a.d / 8; i += 256) dst[i] = src[i];
  __syncthreads();   // everybody has read the length
  if (tid == 0) {
    const long long room = (long long)a.pages * a.page_size;
    long long slot = -1;
    if (pos >= 0 && pos < room) {
      const int page = a.table[b * a.table_stride + pos / a.page_size];
      if (page >= 0 && (a.num_pages <= 0 || page < a.num_pages)) slot = (long long)page * a.page_size + pos % a.page_size;
    }
    if (slot < 0) atomicCAS(a.status, 0, ST_BAD_INDEX | (SITE_DECODE_POST_SLOT << 8));
    a.slots[b] = slot;
    a.lens[b] = (int)(slot < 0 ? min(max(pos, 0ll), room) : pos + (a.inc ? a.inc[b] : 1));
  }
}

// next[b] = the smallest index of the row's largest logit (NaN counts as the largest), plus `first`, at most `limit`. A cluster of eight
// blocks per row, so that one sequence's 152 k logits are read by eight SMs.
struct Best {
  float v;
  int i;
  __device__ __forceinline__ void take(float w, int j) {
    const bool better = isnan(w) ? (!isnan(v) || j < i) : (!isnan(v) && (w > v || (w == v && j < i)));
    if (better) {
      v = w;
      i = j;
    }
  }
};
constexpr int PICK_CTAS = 8, PICK_THREADS = 512;

__global__ void __cluster_dims__(PICK_CTAS, 1, 1) __launch_bounds__(PICK_THREADS)
greedy_pick_kernel(const bf16* __restrict__ logits, long long ld, int V, bool vec, long long first, long long limit, long long* __restrict__ next) {
  namespace cg = cooperative_groups;
  __shared__ Best red[PICK_THREADS / 32];
  __shared__ Best mine;
  pdl_launch_dependents();
  pdl_wait();
  auto cluster = cg::this_cluster();
  const int rank = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const bf16* row = logits + b * ld;
  Best best{-INFINITY, INT_MAX};
  const int nvec = vec ? V / 8 : 0;
  for (int j = rank * PICK_THREADS + tid; j < nvec; j += PICK_CTAS * PICK_THREADS) {
    const uint4 u = reinterpret_cast<const uint4*>(row)[j];
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      best.take(bf16lo(w[e]), j * 8 + 2 * e);
      best.take(bf16hi(w[e]), j * 8 + 2 * e + 1);
    }
  }
  for (int j = nvec * 8 + rank * PICK_THREADS + tid; j < V; j += PICK_CTAS * PICK_THREADS) best.take(__bfloat162float(row[j]), j);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) best.take(__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o));
  if ((tid & 31) == 0) red[tid >> 5] = best;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < PICK_THREADS / 32; ++w) best.take(red[w].v, red[w].i);
    mine = best;
  }
  cluster.sync();
  if (rank == 0 && tid == 0) {
    for (int r = 1; r < PICK_CTAS; ++r) {
      const Best* o = cluster.map_shared_rank(&mine, r);
      best.take(o->v, o->i);
    }
    next[b] = min((long long)best.i + first, limit);
  }
  cluster.sync();   // nobody leaves while its best may still be read
}

}  // namespace cb

namespace cosmos {

void rope_tables(const long long* pos, int S, int half, double theta, int head_dim, int h3, int w3, float* cos_t, float* sin_t, cudaStream_t s) {
  if (S <= 0 || half <= 0) return;
  if (half > cb::ROPE_HALF_MAX) throw std::runtime_error("rope_tables: at most 256 frequencies");
  const long long blocks = ((long long)S * half + 255) / 256;
  launch_early(cb::rope_tables_kernel, dim3((unsigned)(blocks < 148 * 4 ? blocks : 148 * 4)), dim3(256), 0, s, pos, S, half, theta, head_dim, h3, w3,
               cos_t, sin_t);
}

void decode_begin(const DecodeBeginArgs& a, cudaStream_t s) {
  if (a.B <= 0) return;
  launch_early(cb::decode_begin_kernel, dim3((unsigned)a.B), dim3(256), 0, s, a);
}

void greedy_pick(const void* logits, long long ld, int B, int V, long long first, long long limit, long long* next, cudaStream_t s) {
  if (B <= 0 || V <= 0) return;
  const bool vec = ld % 8 == 0 && reinterpret_cast<uintptr_t>(logits) % 16 == 0;
  launch_early(cb::greedy_pick_kernel, dim3(cb::PICK_CTAS, (unsigned)B), dim3(cb::PICK_THREADS), 0, s, (const bf16*)logits, ld, V, vec, first, limit, next);
}

}  // namespace cosmos
