// Global-norm gradient clipping fused with the Adam update over flat fp32
// parameter / gradient / moment buffers.
//
//   sb_grad_sumsq   two-stage deterministic sum of squares -> norm (device scalar)
//   sb_adam_step    g' = g * min(1, max_norm / (norm + 1e-6)) * inv_scale, then the
//                   Adam update of torch.optim.Adam (no weight decay, no amsgrad);
//                   the clip coefficient is read on the device, so the step needs
//                   no host synchronisation.
//
// Role of the reference: clip_grad_norm_(1.0) + fused Adam in
// ScaFFold/utils/trainer.py:678-694.
#include "common.cuh"
#include "host_api.h"

namespace sb {

constexpr int OPT_THREADS = 256;

__global__ void __launch_bounds__(OPT_THREADS) sumsq_partial_kernel(const float* __restrict__ g, long long n,
                                                                    float* __restrict__ partials) {
  __shared__ float red[OPT_THREADS / 32];
  float acc = 0.f;
  const long long n4 = n / 4;
  const float4* g4 = reinterpret_cast<const float4*>(g);
  for (long long i = (long long)blockIdx.x * OPT_THREADS + threadIdx.x; i < n4; i += (long long)gridDim.x * OPT_THREADS) {
    const float4 v = __ldg(g4 + i);
    acc += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  if (blockIdx.x == 0 && threadIdx.x < (int)(n - n4 * 4)) {
    const float v = g[n4 * 4 + threadIdx.x];
    acc += v * v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float r = 0.f;
#pragma unroll
    for (int w = 0; w < OPT_THREADS / 32; ++w) r += red[w];
    partials[blockIdx.x] = r;
  }
}

// One block, a fixed order: thread t adds the partials t, t + 256, ... (all loads in flight at once), then a shuffle
// tree and the eight warps in order. (One thread walking up to 1184 partials took 23-28 us: one L2 latency each.)
__global__ void __launch_bounds__(OPT_THREADS) sumsq_finalize_kernel(const float* __restrict__ partials, int nblocks,
                                                                     float* __restrict__ out) {
  __shared__ double red[OPT_THREADS / 32];
  double acc = 0.0;
#pragma unroll 8
  for (int i = threadIdx.x; i < nblocks; i += OPT_THREADS) acc += (double)partials[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = 0.0;
#pragma unroll
    for (int w = 0; w < OPT_THREADS / 32; ++w) r += red[w];
    out[0] = (float)sqrt(r);
  }
}

struct AdamCoef {
  float lr_step, b1, b2, eps, bc2_sqrt, coef;
};
__device__ __forceinline__ void adam_one(float& p, float g, float& m, float& v, const AdamCoef& k) {
  const float gi = g * k.coef;
  m = m + (gi - m) * (1.f - k.b1);  // lerp, as torch does
  v = v * k.b2 + gi * gi * (1.f - k.b2);
  p -= k.lr_step * m / (sqrtf(v) / k.bc2_sqrt + k.eps);
}

// Bound: memory (28 bytes per parameter). 16-byte accesses and eight of them in flight per thread; the moments are not
// read again before the next step, so they bypass L2's retention (streaming hints) and leave it to p, which the weight
// packing reads next. 90.3 M parameters, whole optimizer step (norm, update, packing): 619 us with 4-byte accesses and
// the serial norm, 476 us now (5.3 TB/s over the step's 2.5 GB).
__global__ void __launch_bounds__(OPT_THREADS) adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                                                           float* __restrict__ m, float* __restrict__ v, long long n,
                                                           int vec, float lr, float b1, float b2, float eps, float bc1,
                                                           float bc2_sqrt, float max_norm,
                                                           const float* __restrict__ norm, float grad_scale) {
  float coef = grad_scale;
  if (max_norm > 0.f && norm != nullptr) {
    const float c = max_norm / (norm[0] * grad_scale + 1e-6f);
    coef *= c < 1.f ? c : 1.f;
  }
  const AdamCoef k{lr / bc1, b1, b2, eps, bc2_sqrt, coef};
  const long long n4 = vec ? n / 4 : 0, stride = (long long)gridDim.x * OPT_THREADS;
  float4* p4 = reinterpret_cast<float4*>(p);
  const float4* g4 = reinterpret_cast<const float4*>(g);
  float4* m4 = reinterpret_cast<float4*>(m);
  float4* v4 = reinterpret_cast<float4*>(v);
  for (long long i = (long long)blockIdx.x * OPT_THREADS + threadIdx.x; i < n4; i += 2 * stride) {
    const bool two = i + stride < n4;
    float4 pp[2], gg[2], mm[2], vv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 0 || two) {
        const long long j = i + u * stride;
        gg[u] = __ldcs(g4 + j);
        mm[u] = __ldcs(m4 + j);
        vv[u] = __ldcs(v4 + j);
        pp[u] = p4[j];
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 0 || two) {
        const long long j = i + u * stride;
        adam_one(pp[u].x, gg[u].x, mm[u].x, vv[u].x, k);
        adam_one(pp[u].y, gg[u].y, mm[u].y, vv[u].y, k);
        adam_one(pp[u].z, gg[u].z, mm[u].z, vv[u].z, k);
        adam_one(pp[u].w, gg[u].w, mm[u].w, vv[u].w, k);
        __stcs(m4 + j, mm[u]);
        __stcs(v4 + j, vv[u]);
        p4[j] = pp[u];
      }
    }
  }
  // what the vectors leave over: up to three elements, or all of them when a buffer does not start on 16 bytes
  for (long long j = n4 * 4 + (long long)blockIdx.x * OPT_THREADS + threadIdx.x; j < n; j += stride) {
    float pj = p[j], mj = m[j], vj = v[j];
    adam_one(pj, g[j], mj, vj, k);
    p[j] = pj; m[j] = mj; v[j] = vj;
  }
}

}  // namespace sb

using namespace sb;

extern "C" int sb_opt_blocks(long long n) {
  long long b = (n / 4 + OPT_THREADS - 1) / OPT_THREADS;
  const long long cap = 148LL * 8;
  return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

extern "C" int sb_grad_norm(const float* g, long long n, float* partials, float* norm_out, cudaStream_t stream) {
  if ((reinterpret_cast<uintptr_t>(g) & 15) != 0) return SB_ERR_ALIGN;
  const int blocks = sb_opt_blocks(n);
  sumsq_partial_kernel<<<blocks, OPT_THREADS, 0, stream>>>(g, n, partials);
  sb_count_launch(1);
  sumsq_finalize_kernel<<<1, OPT_THREADS, 0, stream>>>(partials, blocks, norm_out);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_adam_step(float* p, const float* g, float* m, float* v, long long n, float lr, float b1, float b2,
                            float eps, int step, float max_norm, const float* norm, float grad_scale,
                            cudaStream_t stream) {
  const int vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
                    reinterpret_cast<uintptr_t>(v)) & 15) == 0;
  const float bc1 = 1.f - powf(b1, (float)step);
  const float bc2_sqrt = sqrtf(1.f - powf(b2, (float)step));
  const int blocks = sb_opt_blocks(n);
  adam_kernel<<<blocks, OPT_THREADS, 0, stream>>>(p, g, m, v, n, vec, lr, b1, b2, eps, bc1, bc2_sqrt, max_norm, norm,
                                                  grad_scale);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}
