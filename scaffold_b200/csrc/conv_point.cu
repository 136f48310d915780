// 1x1x1 convolution from few channels (16 or 32, the backward-data of a segmentation head) to 16 .. 128.
//
// The call is a stream: 32 (64) bytes in and up to 256 out per voxel, some 30 operations per byte. The tiled kernel
// (conv_igemm.cu) was bound by its operand loads, a TMA row per voxel and per weight row for 16 channels each: 257 us for
// 16 -> 64 channels at 2 x 128^3, 671 MB. Here nothing is staged: a warp takes 16 consecutive voxels, whose rows are the
// A fragment of mma.m16n8k16 as they lie in memory, the weights stay in registers as B fragments, and the columns are
// dealt to the fragments so that a lane's accumulators are NC / 4 consecutive channels of a voxel: the four lanes of a
// voxel store its row, a warp store covers eight whole rows. 16 -> 64 now takes 114 us (5.9 TB/s); 16 -> 32 243 / 72 us,
// 16 -> 128 323 / 237 us, 16 -> 16 169 / 47 us.
#include "common.cuh"
#include "host_api.h"

namespace sb {

struct PointParams {
  const __nv_bfloat16* x;
  const __nv_bfloat16* w;  // [rows][K]
  __nv_bfloat16* y;
  long long voxels;
  int rows;  // output channels, a multiple of NC
};

__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// KB: 16-channel blocks of the input; NC: output channels per warp (64, 32 or 16); blockIdx.y selects them.
template <int KB, int NC>
__global__ void __launch_bounds__(256) conv_point_kernel(const PointParams p) {
  constexpr int K = 16 * KB, NT = NC / 8, PER = NC / 4;  // fragments of 8 columns; channels per lane and voxel
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.y * NC;
  // column c of fragment j: lane t = c / 2 holds it, as its channel 2 j + c % 2
  uint32_t b[NT][KB][2];
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const __nv_bfloat16* row = p.w + (long long)(n0 + (g >> 1) * PER + 2 * j + (g & 1)) * K;
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      b[j][k][0] = *reinterpret_cast<const uint32_t*>(row + k * 16 + 2 * t);
      b[j][k][1] = *reinterpret_cast<const uint32_t*>(row + k * 16 + 8 + 2 * t);
    }
  }
  const long long tiles = (p.voxels + 15) / 16;
  const long long stride = (long long)gridDim.x * (blockDim.x / 32);
  const long long first = (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  constexpr int FLIGHT = KB == 1 ? 4 : 2;  // tiles whose loads are in flight
  for (long long tile = first; tile < tiles; tile += FLIGHT * stride) {
    uint32_t a[FLIGHT][KB][4];
#pragma unroll
    for (int u = 0; u < FLIGHT; ++u) {
      const long long v = (tile + u * stride) * 16 + g;
      const bool lo = v < p.voxels, hi = v + 8 < p.voxels;
      const uint32_t* r = reinterpret_cast<const uint32_t*>(p.x + v * K) + t;
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        a[u][k][0] = lo ? __ldg(r + k * 8) : 0u;
        a[u][k][2] = lo ? __ldg(r + k * 8 + 4) : 0u;
        a[u][k][1] = hi ? __ldg(r + k * 8 + 4 * K) : 0u;
        a[u][k][3] = hi ? __ldg(r + k * 8 + 4 * K + 4) : 0u;
      }
    }
#pragma unroll
    for (int u = 0; u < FLIGHT; ++u) {
      const long long v = (tile + u * stride) * 16 + g;
      uint32_t out[2][PER / 2];  // [voxel g / g + 8][pairs of channels]
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < KB; ++k) mma_16816(d, a[u][k], b[j][k]);
        out[0][j] = pack_bf16x2(d[0], d[1]);
        out[1][j] = pack_bf16x2(d[2], d[3]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (v + 8 * h >= p.voxels) continue;
        __nv_bfloat16* dst = p.y + (v + 8 * h) * p.rows + n0 + t * PER;
        if constexpr (PER == 16)
          st_global_v8(dst, make_uint4(out[h][0], out[h][1], out[h][2], out[h][3]),
                       make_uint4(out[h][4], out[h][5], out[h][6], out[h][7]));
        else if constexpr (PER == 8)
          *reinterpret_cast<uint4*>(dst) = make_uint4(out[h][0], out[h][1], out[h][2], out[h][3]);
        else
          *reinterpret_cast<uint2*>(dst) = make_uint2(out[h][0], out[h][1]);
      }
    }
  }
}

// -1: not this kernel's call. One dense source of 16 or 32 channels, one dense destination of at most 128 channels (each
// 64 of them read the source again, which costs more than the tiled kernel's loads beyond that), no bias.
int conv_point_launch(const SbConvArgs* a, cudaStream_t stream) {
  if (a->ksize != 1 || a->src_c[1] > 0 || a->dst[1] != nullptr || a->bias != nullptr || a->wpack == nullptr) return -1;
  if ((a->src_c[0] != 16 && a->src_c[0] != 32) || a->src_ld[0] != a->src_c[0]) return -1;
  if (a->cout_pad % 16 != 0 || a->cout_pad > 128 || a->dst_c[0] != a->cout_pad || a->dst_ld[0] != a->cout_pad) return -1;
  if (a->off_d || a->off_h || a->off_w || (a->in_d && a->in_d != a->D) || (a->in_h && a->in_h != a->H) ||
      (a->in_w && a->in_w != a->W))
    return -1;
  if (((uintptr_t)a->src[0] & 15) || ((uintptr_t)a->wpack & 3) || ((uintptr_t)a->dst[0] & 31)) return -1;
  PointParams p;
  p.x = (const __nv_bfloat16*)a->src[0];
  p.w = (const __nv_bfloat16*)a->wpack;
  p.y = (__nv_bfloat16*)a->dst[0];
  p.voxels = (long long)a->N * a->D * a->H * a->W;
  p.rows = a->cout_pad;
  const int nc = p.rows % 64 == 0 ? 64 : p.rows % 32 == 0 ? 32 : 16;
  long long blocks = (p.voxels + 127) / 128;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const dim3 grid((unsigned)blocks, p.rows / nc);
  const bool k2 = a->src_c[0] == 32;
  if (nc == 64) k2 ? conv_point_kernel<2, 64><<<grid, 256, 0, stream>>>(p) : conv_point_kernel<1, 64><<<grid, 256, 0, stream>>>(p);
  else if (nc == 32) k2 ? conv_point_kernel<2, 32><<<grid, 256, 0, stream>>>(p) : conv_point_kernel<1, 32><<<grid, 256, 0, stream>>>(p);
  else k2 ? conv_point_kernel<2, 16><<<grid, 256, 0, stream>>>(p) : conv_point_kernel<1, 16><<<grid, 256, 0, stream>>>(p);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

}  // namespace sb
