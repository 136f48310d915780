// Fused segmentation loss: softmax cross-entropy (class-weighted) + soft Dice
// sums in ONE pass over the logits, and the gradient w.r.t. the logits in one
// more pass; plus the hard-Dice (argmax) counts of the validation metric.
//
// Logits are voxel-major bf16 [N, S, CP] (CP = classes padded to a multiple of
// 8, at most 32), labels int16/int32/int64 [N, S]. No fp32 probability tensor,
// no one-hot tensor and no log-softmax tensor is ever written: every thread
// keeps one voxel's classes in registers.
//
// Pass 1 (loss_sums_kernel): per sample n and class c
//     P[n][c] = sum_v p_c(v)        Q[n][c] = sum_v [y(v) = c]
//     I[n][c] = sum_v p_c(v) [y(v) = c]
//   and CE numerator sum_v w[y] * (-log p_y), denominator sum_v w[y].
//   Block partials go to a workspace; loss_finalize_kernel adds them in a fixed
//   order (deterministic) into sums[N][3C+2]; loss_head_kernel turns the sums
//   (after the shards' all-reduce on a sharded volume) into Dice, loss and the
//   coefficients of pass 2.
// Pass 2 (loss_grad_kernel): with per-(n,c) coefficients alpha, beta of
//   dL/dp_c(v) = alpha[n][c] * [y(v)=c] + beta[n][c] and k_ce = g / denominator:
//     dlogit_j = k_ce * w[y] * (p_j - [y=j]) + p_j * (a_j - sum_c a_c p_c)
//
// A label outside [0, C) (a dataset with more categories than the model, an ignore
// value) is never used as an index: the voxel gets weight 0 in the cross entropy and
// belongs to no class in the Dice sums, and the kernels record ST_BAD_ARG (site 61 /
// 62, detail = label value) in the status word so that the host can raise.
//
// Role of the reference: ScaFFold/utils/trainer.py:635-664,
// ScaFFold/utils/losses.py:117-205, ScaFFold/utils/dice_score.py:101-136,
// ScaFFold/utils/evaluate.py:178-193.
#include "common.cuh"
#include "host_api.h"

namespace sb {

constexpr int LOSS_THREADS = 128;
constexpr int LOSS_MAXC = 32;
constexpr float LOSS_EPS = 1e-6f;  // of the Dice quotient

__device__ __forceinline__ long long load_label(const void* labels, int kind, long long i) {
  if (kind == 2) return reinterpret_cast<const short*>(labels)[i];
  if (kind == 4) return reinterpret_cast<const int*>(labels)[i];
  return reinterpret_cast<const long long*>(labels)[i];
}

// The first CN logits of a voxel; classes from C on become -inf, so they take no part in the softmax.
template <int CN>
__device__ __forceinline__ void load_logits(const __nv_bfloat16* p, float (&f)[CN], int C) {
#pragma unroll
  for (int i = 0; i < (CN + 7) / 8; ++i) {
    const uint4 raw = __ldg(reinterpret_cast<const uint4*>(p) + i);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = __bfloat1622float2(h[j]);
      const int c = i * 8 + 2 * j;
      if (c < CN) f[c] = c < C ? t.x : -INFINITY;
      if (c + 1 < CN) f[c + 1] = c + 1 < C ? t.y : -INFINITY;
    }
  }
}

// softmax over the CN entries (-inf entries become 0); returns log-sum-exp
template <int CN>
__device__ __forceinline__ float softmax_regs(float (&f)[CN]) {
  float m = f[0];
#pragma unroll
  for (int c = 1; c < CN; ++c) m = fmaxf(m, f[c]);
  float s = 0.f;
#pragma unroll
  for (int c = 0; c < CN; ++c) {
    f[c] = __expf(f[c] - m);
    s += f[c];
  }
  const float inv = 1.f / s;
#pragma unroll
  for (int c = 0; c < CN; ++c) f[c] *= inv;
  return m + __logf(s);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// workspace layout per (n, block): [3*C + 2] floats: P[c], Q[c], I[c], ce_num, ce_den
//
// Bound: issue rate and latency, not memory (16 exponentials and about 150 instructions for 34 bytes). Q and I change
// for ONE class per voxel, so every thread keeps its own column of (I, Q) pairs in shared memory, indexed by the label:
// one 8-byte read and write instead of 2 x CN predicated adds, and 2 x CN registers less, which is what lets 32 warps
// live on an SM. CN is the class count rounded up to 4, so 9 classes pay for 12 exponentials and not for 16.
// Call with its collapse, 2 x 128^3 voxels: 9 classes 145 -> 65 us, 17 classes 349 -> 95 us (before: all sums in
// registers, classes rounded up to 16).
template <int CN>
__global__ void __launch_bounds__(LOSS_THREADS) loss_sums_kernel(const __nv_bfloat16* __restrict__ logits,
                                                                 const void* __restrict__ labels, int label_kind,
                                                                 const float* __restrict__ cw, float* __restrict__ ws,
                                                                 int C, int CP, long long S, int argmax_mode,
                                                                 uint32_t* __restrict__ status) {
  __shared__ float2 s_iq[CN][LOSS_THREADS];
  __shared__ float s_ce[2][LOSS_THREADS / 32];
  const int n = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float P[CN];
#pragma unroll
  for (int c = 0; c < CN; ++c) {
    P[c] = 0.f;
    s_iq[c][tid] = make_float2(0.f, 0.f);
  }
  float ce_num = 0.f, ce_den = 0.f;
  auto voxel = [&](float (&f)[CN], const long long y_raw) {
    const bool y_ok = y_raw >= 0 && y_raw < C;
    const int y = y_ok ? (int)y_raw : 0;
    if (!y_ok) report(status, ST_BAD_ARG, 61, (uint32_t)y_raw, (uint32_t)n);
    float ly = 0.f, py = 0.f;
#pragma unroll
    for (int c = 0; c < CN; ++c) ly = c == y ? f[c] : ly;
    const float lse = softmax_regs<CN>(f);  // f now holds probabilities
    if (argmax_mode) {
      // hard prediction: one-hot of the first maximum
      int best = 0;
      float bv = f[0];
#pragma unroll
      for (int c = 1; c < CN; ++c)
        if (f[c] > bv) { bv = f[c]; best = c; }
#pragma unroll
      for (int c = 0; c < CN; ++c) f[c] = c == best ? 1.f : 0.f;
    }
#pragma unroll
    for (int c = 0; c < CN; ++c) {
      P[c] += f[c];
      py = c == y ? f[c] : py;
    }
    if (y_ok) {
      float2 iq = s_iq[y][tid];
      iq.x += py;
      iq.y += 1.f;
      s_iq[y][tid] = iq;
      const float wy = cw ? __ldg(cw + y) : 1.f;
      ce_num += wy * (lse - ly);
      ce_den += wy;
    }
  };
  // two voxels per iteration: both voxels' logits and labels are requested before either is used
  const long long stride = (long long)gridDim.x * LOSS_THREADS;
  long long v = (long long)blockIdx.x * LOSS_THREADS + tid;
  for (; v + stride < S; v += 2 * stride) {
    float f0[CN], f1[CN];
    load_logits<CN>(logits + ((long long)n * S + v) * CP, f0, C);
    load_logits<CN>(logits + ((long long)n * S + v + stride) * CP, f1, C);
    const long long y0 = load_label(labels, label_kind, (long long)n * S + v);
    const long long y1 = load_label(labels, label_kind, (long long)n * S + v + stride);
    voxel(f0, y0);
    voxel(f1, y1);
  }
  for (; v < S; v += stride) {
    float f0[CN];
    load_logits<CN>(logits + ((long long)n * S + v) * CP, f0, C);
    voxel(f0, load_label(labels, label_kind, (long long)n * S + v));
  }
  // block sums in a fixed order: a warp takes the classes warp, warp + 4, ... and adds the columns lane, lane + 32, ...
  float* dst = ws + ((long long)n * gridDim.x + blockIdx.x) * (3 * C + 2);
  __syncthreads();
  for (int c = warp; c < C; c += LOSS_THREADS / 32) {
    float i = 0.f, q = 0.f;
#pragma unroll
    for (int k = 0; k < LOSS_THREADS / 32; ++k) {
      const float2 iq = s_iq[c][k * 32 + lane];
      i += iq.x;
      q += iq.y;
    }
    i = warp_sum(i);
    q = warp_sum(q);
    if (lane == 0) {
      dst[C + c] = q;
      dst[2 * C + c] = i;
    }
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < CN; ++c) s_iq[c][tid].x = P[c];
  ce_num = warp_sum(ce_num);
  ce_den = warp_sum(ce_den);
  if (lane == 0) {
    s_ce[0][warp] = ce_num;
    s_ce[1][warp] = ce_den;
  }
  __syncthreads();
  for (int c = warp; c < C; c += LOSS_THREADS / 32) {
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < LOSS_THREADS / 32; ++k) a += s_iq[c][k * 32 + lane].x;
    a = warp_sum(a);
    if (lane == 0) dst[c] = a;
  }
  if (tid < 2) {
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < LOSS_THREADS / 32; ++k) a += s_ce[tid][k];
    dst[3 * C + tid] = a;
  }
}

// out[n][k] = sum_b ws[n][b][k], k < 3C+2, in double: one warp per output, lanes take the blocks lane, lane + 32, ...
// in order, eight loads in flight, then a fixed shuffle tree. (A thread per output walking every block in turn took
// 35 us: one L2 latency per block.)
__global__ void __launch_bounds__(256) loss_finalize_kernel(const float* __restrict__ ws, float* __restrict__ out,
                                                            int N, int nblocks, int K) {
  const int o = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (o >= N * K) return;
  const int n = o / K, k = o - n * K;
  const float* src = ws + (long long)n * nblocks * K + k;
  double acc = 0.0;
  int b = lane;
  for (; b + 7 * 32 < nblocks; b += 8 * 32) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = src[(long long)(b + u * 32) * K];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc += (double)v[u];
  }
  for (; b < nblocks; b += 32) acc += (double)src[(long long)b * K];
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (lane == 0) out[o] = (float)acc;
}

// From the sums of all shards: dice[N][C] and, when asked for, the loss and what its gradient needs.
//   loss[1] = ce + (1 - fg), ce[1], fg[1] (mean foreground Dice)
//   coef[N][2][C]: alpha, beta of d(-fg)/dp_c (zero for class 0 and for a class that is absent on both sides), den[1]
// One block: N * C is a few dozen values; in torch operations the same arithmetic is some thirty launches.
__global__ void __launch_bounds__(256) loss_head_kernel(const float* __restrict__ sums, int N, int C,
                                                        float* __restrict__ dice, float* __restrict__ loss,
                                                        float* __restrict__ ce_out, float* __restrict__ fg_out,
                                                        float* __restrict__ coef, float* __restrict__ den_out) {
  __shared__ float red[3][8];
  const int K = 3 * C + 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float m = (float)N * (float)(C - 1);
  float fg = 0.f, num = 0.f, den = 0.f;
  for (int i = threadIdx.x; i < N * C; i += 256) {
    const int n = i / C, c = i - n * C;
    const float* s = sums + (long long)n * K;
    const float inter2 = 2.f * s[2 * C + c], sets = s[c] + s[C + c];
    const bool empty = sets == 0.f;
    const float u = (empty ? inter2 : sets) + LOSS_EPS;
    const float d = (inter2 + LOSS_EPS) / u;
    if (dice) dice[i] = d;
    if (c > 0) fg += d;
    if (coef) {
      const bool on = c > 0 && !empty;
      coef[((long long)n * 2 + 0) * C + c] = on ? -2.f / (m * u) : 0.f;
      coef[((long long)n * 2 + 1) * C + c] = on ? (inter2 + LOSS_EPS) / (m * u * u) : 0.f;
    }
  }
  if (loss == nullptr) return;
  for (int n = threadIdx.x; n < N; n += 256) {
    num += sums[(long long)n * K + 3 * C];
    den += sums[(long long)n * K + 3 * C + 1];
  }
  fg = warp_sum(fg);
  num = warp_sum(num);
  den = warp_sum(den);
  if (lane == 0) { red[0][warp] = fg; red[1][warp] = num; red[2][warp] = den; }
  __syncthreads();
  if (threadIdx.x == 0) {
    fg = num = den = 0.f;
    for (int w = 0; w < 8; ++w) { fg += red[0][w]; num += red[1][w]; den += red[2][w]; }
    den = den < 1.1920929e-7f ? 1.1920929e-7f : den;  // the fp32 step above 1, as clamp_min(finfo.eps): a NaN stays one
    fg /= m;
    const float ce = num / den;
    loss[0] = ce + (1.f - fg);
    ce_out[0] = ce;
    fg_out[0] = fg;
    den_out[0] = den;
  }
}

// dlogit_j = p_j * (k_ce w_y + beta_j - dot) + [y = j] * (p_y alpha_y - k_ce w_y), dot = sum_c beta_c p_c + alpha_y p_y.
// Only the label's alpha is needed, so alpha is read from shared memory by the label and the label's class is one
// correction. Call, 2 x 128^3 voxels, 9 classes: 133 -> 80 us.
template <int CN>
__global__ void __launch_bounds__(LOSS_THREADS) loss_grad_kernel(const __nv_bfloat16* __restrict__ logits,
                                                                 const void* __restrict__ labels, int label_kind,
                                                                 const float* __restrict__ cw,
                                                                 const float* __restrict__ coef,  // [N][2][C]
                                                                 const float* __restrict__ g,     // [1] d / d loss
                                                                 const float* __restrict__ den,   // [1]
                                                                 __nv_bfloat16* __restrict__ dlogits, int C, int CP,
                                                                 long long S, uint32_t* __restrict__ status) {
  __shared__ float s_alpha[CN];
  const int n = blockIdx.y;
  const float gv = g[0], k_ce = gv / den[0];
  if (threadIdx.x < CN)
    s_alpha[threadIdx.x] = (int)threadIdx.x < C ? gv * coef[(long long)n * 2 * C + threadIdx.x] : 0.f;
  float beta[CN];
#pragma unroll
  for (int c = 0; c < CN; ++c) beta[c] = c < C ? gv * coef[((long long)n * 2 + 1) * C + c] : 0.f;
  __syncthreads();
  auto voxel = [&](float (&f)[CN], const long long y_raw, const long long off) {
    const bool y_ok = y_raw >= 0 && y_raw < C;
    const int y = y_ok ? (int)y_raw : -1;
    if (!y_ok) report(status, ST_BAD_ARG, 62, (uint32_t)y_raw, (uint32_t)n);
    softmax_regs<CN>(f);
    const float wy = y_ok ? (cw ? __ldg(cw + y) : 1.f) * k_ce : 0.f;
    const float ay = y_ok ? s_alpha[y] : 0.f;
    float dot = 0.f, py = 0.f;
#pragma unroll
    for (int c = 0; c < CN; ++c) {
      dot += beta[c] * f[c];
      py = c == y ? f[c] : py;
    }
    dot += ay * py;
    const float base = wy - dot, fix = y_ok ? py * ay - wy : 0.f;
#pragma unroll
    for (int c = 0; c < CN; ++c) {
      const float v = f[c] * (base + beta[c]);
      f[c] = c == y ? v + fix : v;
    }
    for (int i = 0; i < CP / 8; ++i) {
      uint4 o = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int k = 0; k < (CN + 7) / 8; ++k)
        if (k == i) {
          float t[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) t[j] = k * 8 + j < CN ? f[k * 8 + j < CN ? k * 8 + j : 0] : 0.f;
          o.x = pack_bf16x2(t[0], t[1]);
          o.y = pack_bf16x2(t[2], t[3]);
          o.z = pack_bf16x2(t[4], t[5]);
          o.w = pack_bf16x2(t[6], t[7]);
        }
      reinterpret_cast<uint4*>(dlogits + off)[i] = o;
    }
  };
  // two voxels per iteration: both voxels' logits and labels are requested before either is used
  const long long stride = (long long)gridDim.x * LOSS_THREADS;
  long long v = (long long)blockIdx.x * LOSS_THREADS + threadIdx.x;
  for (; v + stride < S; v += 2 * stride) {
    float f0[CN], f1[CN];
    const long long off0 = ((long long)n * S + v) * CP, off1 = ((long long)n * S + v + stride) * CP;
    load_logits<CN>(logits + off0, f0, C);
    load_logits<CN>(logits + off1, f1, C);
    const long long y0 = load_label(labels, label_kind, (long long)n * S + v);
    const long long y1 = load_label(labels, label_kind, (long long)n * S + v + stride);
    voxel(f0, y0, off0);
    voxel(f1, y1, off1);
  }
  for (; v < S; v += stride) {
    float f0[CN];
    const long long off0 = ((long long)n * S + v) * CP;
    load_logits<CN>(logits + off0, f0, C);
    voxel(f0, load_label(labels, label_kind, (long long)n * S + v), off0);
  }
}

}  // namespace sb

using namespace sb;

// 8 blocks of 4 warps per SM in one wave
extern "C" int sb_loss_blocks(long long S) {
  long long b = (S + LOSS_THREADS - 1) / LOSS_THREADS;
  const long long cap = 148LL * 8;
  return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

// largest class count of the fused kernels (callers route wider heads to the framework formula)
extern "C" int sb_loss_max_classes(void) { return LOSS_MAXC; }

static bool loss_args_ok(int C, int CP, int label_kind) {
  return C >= 1 && C <= CP && CP % 8 == 0 && CP <= LOSS_MAXC && (label_kind == 2 || label_kind == 4 || label_kind == 8);
}

// sums: [N][3C+2] floats; ws: [N][sb_loss_blocks(S)][3C+2]
extern "C" int sb_loss_sums(const void* logits, const void* labels, int label_kind, const float* cw, float* ws,
                            float* sums, int N, long long S, int C, int CP, int argmax_mode, uint32_t* status,
                            cudaStream_t stream) {
  if (!loss_args_ok(C, CP, label_kind)) return SB_ERR_SHAPE;
  const int blocks = sb_loss_blocks(S);
  dim3 grid(blocks, N);
  const __nv_bfloat16* lg = (const __nv_bfloat16*)logits;
#define SB_LOSS_SUMS(cn)                                                                                            \
  case cn / 4:                                                                                                      \
    loss_sums_kernel<cn><<<grid, LOSS_THREADS, 0, stream>>>(lg, labels, label_kind, cw, ws, C, CP, S, argmax_mode, status); \
    break;
  switch ((C + 3) / 4) {
    SB_LOSS_SUMS(4) SB_LOSS_SUMS(8) SB_LOSS_SUMS(12) SB_LOSS_SUMS(16)
    SB_LOSS_SUMS(20) SB_LOSS_SUMS(24) SB_LOSS_SUMS(28) SB_LOSS_SUMS(32)
    default: return SB_ERR_SHAPE;
  }
#undef SB_LOSS_SUMS
  const int outs = N * (3 * C + 2);
  loss_finalize_kernel<<<(outs + 7) / 8, 256, 0, stream>>>(ws, sums, N, blocks, 3 * C + 2);
  sb_count_launch(2);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

// dice[N][C]; loss[1], ce[1], fg[1], coef[N][2][C] and den[1] together, or all null
extern "C" int sb_loss_head(const float* sums, int N, int C, float* dice, float* loss, float* ce, float* fg, float* coef,
                            float* den, cudaStream_t stream) {
  if (N < 1 || C < 1) return SB_ERR_SHAPE;
  const void* all[5] = {loss, ce, fg, coef, den};
  for (const void* p : all)
    if ((p == nullptr) != (loss == nullptr)) return SB_ERR_SHAPE;
  loss_head_kernel<<<1, 256, 0, stream>>>(sums, N, C, dice, loss, ce, fg, coef, den);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_loss_grad(const void* logits, const void* labels, int label_kind, const float* cw,
                            const float* coef, const float* g, const float* den, void* dlogits, int N, long long S,
                            int C, int CP, uint32_t* status, cudaStream_t stream) {
  if (!loss_args_ok(C, CP, label_kind)) return SB_ERR_SHAPE;
  dim3 grid(sb_loss_blocks(S), N);
  const __nv_bfloat16* lg = (const __nv_bfloat16*)logits;
  __nv_bfloat16* dl = (__nv_bfloat16*)dlogits;
#define SB_LOSS_GRAD(cn)                                                                                            \
  case cn / 4:                                                                                                      \
    loss_grad_kernel<cn><<<grid, LOSS_THREADS, 0, stream>>>(lg, labels, label_kind, cw, coef, g, den, dl, C, CP, S, status); \
    break;
  switch ((C + 3) / 4) {
    SB_LOSS_GRAD(4) SB_LOSS_GRAD(8) SB_LOSS_GRAD(12) SB_LOSS_GRAD(16)
    SB_LOSS_GRAD(20) SB_LOSS_GRAD(24) SB_LOSS_GRAD(28) SB_LOSS_GRAD(32)
    default: return SB_ERR_SHAPE;
  }
#undef SB_LOSS_GRAD
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}
