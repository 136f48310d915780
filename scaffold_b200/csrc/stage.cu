// Input staging: a channel-major volume [N, C, S] (fp32 as the data loader delivers it, or bf16) with few
// channels becomes the voxel-major bf16 operand [N, S, 16 or 32] of the stem convolution in one pass: layout
// change, down-cast and zero padding of the channels, one 32-byte store per voxel.
//
// A stem of at most three channels gets its in-plane neighbourhood instead of padding: stage_stem_kernel writes the
// 3 x 3 (kh, kw) neighbours x C channels of every voxel into 32 channels, (kh * 3 + kw) * C + c, zeros outside the
// plane and behind 9 * C. The convolution and its weight gradient are then three taps deep instead of 27. The pass is
// bound by its 64-byte stores (the 27 reads of a voxel hit L1: neighbours in w are neighbouring lanes).
//
// Role of the reference: the `.to(device, dtype, memory_format=channels_last_3d)` of a batch
// (ScaFFold/utils/trainer.py:575-583).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "host_api.h"

namespace sb {

template <typename T>
__global__ void __launch_bounds__(256) stage_input_kernel(const T* __restrict__ x, int C, long long S,
                                                          __nv_bfloat16* __restrict__ y, long long total, int cpad) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long n = i / S, v = i - n * S;
    const T* src = x + n * C * S + v;
    __align__(16) __nv_bfloat16 out[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) out[c] = c < C ? __float2bfloat16((float)src[(long long)c * S]) : __float2bfloat16(0.f);
    uint4* dst = reinterpret_cast<uint4*>(y + i * cpad);
    dst[0] = reinterpret_cast<const uint4*>(out)[0];
    dst[1] = reinterpret_cast<const uint4*>(out)[1];
    if (cpad == 32) {  // channels 16..31 are padding
      dst[2] = make_uint4(0u, 0u, 0u, 0u);
      dst[3] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
}

template <typename T, int C>
__global__ void __launch_bounds__(256) stage_stem_kernel(const T* __restrict__ x, int D, int H, int W,
                                                         __nv_bfloat16* __restrict__ y, long long total) {
  const long long S = (long long)D * H * W;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long row = i / W;
    const int w = (int)(i - row * W);
    const int h = (int)(row % H);
    const long long n = row / ((long long)D * H);
    const T* src = x + n * C * S + (i - n * S);  // this voxel in channel 0
    __align__(16) __nv_bfloat16 out[32];
#pragma unroll
    for (int kh = 0; kh < 3; ++kh)
#pragma unroll
      for (int kw = 0; kw < 3; ++kw) {
        const bool in = (unsigned)(h + kh - 1) < (unsigned)H && (unsigned)(w + kw - 1) < (unsigned)W;
#pragma unroll
        for (int c = 0; c < C; ++c)
          out[(kh * 3 + kw) * C + c] =
              __float2bfloat16(in ? (float)src[(long long)c * S + (long long)(kh - 1) * W + (kw - 1)] : 0.f);
      }
#pragma unroll
    for (int k = 9 * C; k < 32; ++k) out[k] = __float2bfloat16(0.f);
    uint4* dst = reinterpret_cast<uint4*>(y + i * 32);
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[k] = reinterpret_cast<const uint4*>(out)[k];
  }
}

// w [cout][C][3][3][3] fp32 -> bf16 [2 - kd][cout_pad][32], column (kh * 3 + kw) * C + c
__global__ void __launch_bounds__(256) pack_stem_kernel(const float* __restrict__ w, int cout, int cout_pad, int C,
                                                        __nv_bfloat16* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 3 * cout_pad * 32) return;
  const int k = i % 32, co = (i / 32) % cout_pad, kd = 2 - i / (32 * cout_pad);
  const int c = k % C, khw = k / C;
  y[i] = __float2bfloat16(co < cout && khw < 9 ? w[((co * C + c) * 3 + kd) * 9 + khw] : 0.f);
}

template <typename T>
static void stage_stem(const void* x, int C, int D, int H, int W, void* y, long long total, int blocks,
                       cudaStream_t stream) {
  const T* src = (const T*)x;
  __nv_bfloat16* dst = (__nv_bfloat16*)y;
  if (C == 1) stage_stem_kernel<T, 1><<<blocks, 256, 0, stream>>>(src, D, H, W, dst, total);
  else if (C == 2) stage_stem_kernel<T, 2><<<blocks, 256, 0, stream>>>(src, D, H, W, dst, total);
  else stage_stem_kernel<T, 3><<<blocks, 256, 0, stream>>>(src, D, H, W, dst, total);
}

}  // namespace sb

// x: [N, C, D, H, W] contiguous, C <= 3; y: bf16 [N, D, H, W, 32]
extern "C" int sb_stage_stem(const void* x, int is_bf16, int N, int C, int D, int H, int W, void* y,
                             cudaStream_t stream) {
  if (C < 1 || C > 3 || N < 1 || D < 1 || H < 1 || W < 1) return SB_ERR_SHAPE;
  const long long total = (long long)N * D * H * W;
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  if (is_bf16) sb::stage_stem<__nv_bfloat16>(x, C, D, H, W, y, total, (int)blocks, stream);
  else sb::stage_stem<float>(x, C, D, H, W, y, total, (int)blocks, stream);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_pack_stem(const float* w, int cout, int cout_pad, int C, void* y, cudaStream_t stream) {
  if (C < 1 || C > 3 || cout < 1 || cout_pad < cout) return SB_ERR_SHAPE;
  sb::pack_stem_kernel<<<(3 * cout_pad * 32 + 255) / 256, 256, 0, stream>>>(w, cout, cout_pad, C, (__nv_bfloat16*)y);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

// x: [N, C, S] contiguous, C <= 16, is_bf16 selects the element type; y: bf16 [N, S, cpad], cpad 16 or 32
extern "C" int sb_stage_input(const void* x, int is_bf16, int N, int C, long long S, void* y, int cpad,
                              cudaStream_t stream) {
  if (C < 1 || C > 16 || N < 1 || S < 1 || (cpad != 16 && cpad != 32)) return SB_ERR_SHAPE;
  const long long total = (long long)N * S;
  long long blocks = (total + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (is_bf16)
    sb::stage_input_kernel<__nv_bfloat16><<<(int)blocks, 256, 0, stream>>>((const __nv_bfloat16*)x, C, S, (__nv_bfloat16*)y, total, cpad);
  else
    sb::stage_input_kernel<float><<<(int)blocks, 256, 0, stream>>>((const float*)x, C, S, (__nv_bfloat16*)y, total, cpad);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}
