// Optimizer kernels over lists of tensors: global gradient norm and AdamW with clipping, one launch for a whole model.
//
// What bounds both is memory: the norm reads 2 bytes a parameter; the update reads 14 (bf16 gradient, fp32 weight and two
// moments) and writes 14 (the state again, and the bf16 weight). A tensor is cut into chunks of 8192 elements and the
// chunks of all tensors form one grid-stride loop, so that a list of many small tensors costs one launch and a large one
// fills the chip. The clip factor is worked out from the device-side norm, so no host round trip stands between the two.
// Measured on the 543 M parameters of a two-layer Nano generator (2 layers of 193 M, 17 tensors outside them, the largest
// 100 M): update 2.33 ms = 6.5 TB/s, norm 0.17 ms = 6.4 TB/s. Before, the layers took a launch each (2.6 ms together) and the
// tensors outside them a chain of about 14 elementwise launches each, 5.1 ms more.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.h"

namespace cb {

constexpr int OPT_CHUNK = 8192;    // elements: 256 threads x 4 elements x 8 trips, four of them in flight
constexpr int OPT_THREADS = 256;
constexpr int OPT_TRIPS = 4;

struct OptList {
  cosmos::OptTensor t[cosmos::OPT_MAX];
  long long first_chunk[cosmos::OPT_MAX + 1];
  int n;
};

__device__ __forceinline__ int opt_find(const OptList& l, long long chunk) {
  int lo = 0, hi = l.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (l.first_chunk[mid] <= chunk) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8]) {
  f[0] = bf16lo(u.x); f[1] = bf16hi(u.x); f[2] = bf16lo(u.y); f[3] = bf16hi(u.y);
  f[4] = bf16lo(u.z); f[5] = bf16hi(u.z); f[6] = bf16lo(u.w); f[7] = bf16hi(u.w);
}

// Sum over the block in a fixed order; valid in thread 0.
__device__ __forceinline__ double block_sum(double sum) {
  __shared__ double red[OPT_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < OPT_THREADS / 32; ++w) sum += red[w];
  }
  return sum;
}

// sums[block] = sum of squares of the block's chunks: a thread's few hundred squares in fp32, the threads' sums in fp64.
__global__ void __launch_bounds__(OPT_THREADS)
grad_sq_kernel(const __grid_constant__ OptList l, double* sums) {
  double sum = 0.0;
  for (long long ch = blockIdx.x; ch < l.first_chunk[l.n]; ch += gridDim.x) {
    const int k = opt_find(l, ch);
    const cosmos::OptTensor& t = l.t[k];
    const long long e0 = (ch - l.first_chunk[k]) * OPT_CHUNK;
    const int len = (int)min((long long)OPT_CHUNK, t.n - e0);
    const bf16* g = reinterpret_cast<const bf16*>(t.grad) + e0;
    float s = 0.f;
    if (t.vec && len == OPT_CHUNK) {
      uint4 u[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) u[j] = reinterpret_cast<const uint4*>(g)[j * OPT_THREADS + threadIdx.x];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float f[8];
        unpack8(u[j], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(f[e], f[e], s);
      }
    } else {
      for (int i = threadIdx.x; i < len; i += OPT_THREADS) {
        const float f = __bfloat162float(g[i]);
        s = fmaf(f, f, s);
      }
    }
    sum += (double)s;
  }
  sum = block_sum(sum);
  if (threadIdx.x == 0) sums[blockIdx.x] = sum;
}

// sq += scale^2 * the blocks' sums, in a fixed order: the ranks of a data-parallel step add up the squares of replicated gradients
// each by itself, and their clip factors, and with them the replicated weights, stay the same bits. (Blocks that added to
// sq by themselves gave 11 results in 40 runs.) One block, about 3 us behind a norm of 170.
__global__ void __launch_bounds__(OPT_THREADS)
add_sums_kernel(const double* sums, int n, float scale, double* sq) {
  double sum = 0.0;
  for (int i = threadIdx.x; i < n; i += OPT_THREADS) sum += sums[i];
  sum = block_sum(sum);
  if (threadIdx.x == 0) *sq += sum * (double)scale * (double)scale;
}

// omb1, omb2: 1 - b1 and 1 - b2, worked out in fp64 as bc1 and bc2 are (1.f - 0.999f is 1.3e-5 off, and so would be every v).
struct AdamWStep {
  float lr, b1, b2, omb1, omb2, eps, wd, bc1, bc2;
  __device__ __forceinline__ void operator()(float g, float& m, float& v, float& w) const {
    m = b1 * m + omb1 * g;
    v = b2 * v + omb2 * g * g;
    w -= lr * ((m / bc1) / (sqrtf(v / bc2) + eps) + wd * w);
  }
};

// g = grad * scale * clip with clip = min(1, max_norm / (norm + 1e-6)) from the device-side `sq`; max_norm < 0: no clipping.
__global__ void __launch_bounds__(OPT_THREADS)
adamw_list_kernel(const __grid_constant__ OptList l, const __grid_constant__ AdamWStep opt, float scale, const double* sq,
                  float max_norm) {
  float gs = scale;
  if (max_norm >= 0.f) {
    const double norm = sqrt(*sq);
    if (norm > (double)max_norm) gs *= (float)((double)max_norm / (norm + 1e-6));
  }
  for (long long ch = blockIdx.x; ch < l.first_chunk[l.n]; ch += gridDim.x) {
    const int k = opt_find(l, ch);
    const cosmos::OptTensor& t = l.t[k];
    const long long e0 = (ch - l.first_chunk[k]) * OPT_CHUNK;
    const int len = (int)min((long long)OPT_CHUNK, t.n - e0);
    const bf16* g = reinterpret_cast<const bf16*>(t.grad) + e0;
    float *w = t.master + e0, *m = t.m + e0, *v = t.v + e0;
    bf16* p = reinterpret_cast<bf16*>(t.param) + e0;
    if (t.vec && len == OPT_CHUNK) {
      // Four elements a lane, so that a warp's access covers whole lines (with eight, every access took half of each 32-byte
      // sector: 5.4 TB/s), four trips' loads in flight together, and many short blocks, which spread the end of the launch.
      // 386 M parameters, TB/s: two trips and 8 blocks an SM 5.9, four trips 6.2, 64 blocks an SM 6.5 (two trips 6.4).
#pragma unroll 1
      for (int j = 0; j < OPT_CHUNK / (4 * OPT_THREADS); j += OPT_TRIPS) {
        uint2 gu[OPT_TRIPS];
        float4 mu[OPT_TRIPS], vu[OPT_TRIPS], wu[OPT_TRIPS];
#pragma unroll
        for (int k = 0; k < OPT_TRIPS; ++k) {
          const int i = ((j + k) * OPT_THREADS + threadIdx.x) * 4;
          gu[k] = *reinterpret_cast<const uint2*>(g + i);
          mu[k] = *reinterpret_cast<const float4*>(m + i);
          vu[k] = *reinterpret_cast<const float4*>(v + i);
          wu[k] = *reinterpret_cast<const float4*>(w + i);
        }
#pragma unroll
        for (int k = 0; k < OPT_TRIPS; ++k) {
          const int i = ((j + k) * OPT_THREADS + threadIdx.x) * 4;
          opt(bf16lo(gu[k].x) * gs, mu[k].x, vu[k].x, wu[k].x);
          opt(bf16hi(gu[k].x) * gs, mu[k].y, vu[k].y, wu[k].y);
          opt(bf16lo(gu[k].y) * gs, mu[k].z, vu[k].z, wu[k].z);
          opt(bf16hi(gu[k].y) * gs, mu[k].w, vu[k].w, wu[k].w);
          *reinterpret_cast<float4*>(m + i) = mu[k];
          *reinterpret_cast<float4*>(v + i) = vu[k];
          *reinterpret_cast<float4*>(w + i) = wu[k];
          *reinterpret_cast<uint2*>(p + i) = make_uint2(pack_bf16(wu[k].x, wu[k].y), pack_bf16(wu[k].z, wu[k].w));
        }
      }
    } else {
      for (int i = threadIdx.x; i < len; i += OPT_THREADS) {
        float mi = m[i], vi = v[i], wi = w[i];
        opt(__bfloat162float(g[i]) * gs, mi, vi, wi);
        m[i] = mi;
        v[i] = vi;
        w[i] = wi;
        p[i] = __float2bfloat16(wi);
      }
    }
  }
}

static long long fill_list(const cosmos::OptTensor* t, int n, OptList& l) {
  if (n < 1 || n > cosmos::OPT_MAX) throw std::runtime_error("optimizer list: 1 to 64 tensors per launch");
  l.n = n;
  l.first_chunk[0] = 0;
  for (int i = 0; i < n; ++i) {
    l.t[i] = t[i];
    const auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
    // 16-byte loads where every address allows them; the chunks keep that alignment
    l.t[i].vec = al(t[i].grad) && al(t[i].master) && al(t[i].m) && al(t[i].v) && al(t[i].param);
    l.first_chunk[i + 1] = l.first_chunk[i] + (t[i].n + OPT_CHUNK - 1) / OPT_CHUNK;
  }
  return l.first_chunk[n];
}

}  // namespace cb

namespace cosmos {

void grad_sq_list(const OptTensor* t, int n, float scale, double* sums, double* sq, cudaStream_t s) {
  cb::OptList l;
  const long long chunks = cb::fill_list(t, n, l);
  if (chunks == 0) return;
  const int blocks = (int)std::min<long long>(chunks, OPT_SUMS);
  cb::grad_sq_kernel<<<blocks, cb::OPT_THREADS, 0, s>>>(l, sums);
  cb::add_sums_kernel<<<1, cb::OPT_THREADS, 0, s>>>(sums, blocks, scale, sq);
}

void adamw_list(const OptTensor* t, int n, float scale, const double* sq, float max_norm, float lr, double b1, double b2, float eps,
                float wd, int step, cudaStream_t s) {
  cb::OptList l;
  const long long chunks = cb::fill_list(t, n, l);
  if (chunks == 0) return;
  const cb::AdamWStep opt{lr, (float)b1, (float)b2, (float)(1.0 - b1), (float)(1.0 - b2), eps, wd,
                          (float)(1.0 - std::pow(b1, step)), (float)(1.0 - std::pow(b2, step))};
  cb::adamw_list_kernel<<<(int)std::min<long long>(chunks, 148 * 64), cb::OPT_THREADS, 0, s>>>(l, opt, scale, sq, max_norm);
}

}  // namespace cosmos
