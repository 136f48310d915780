// GPU data generation: batched IFS chaos game and point-cloud rasterisation.
//
//   ifs_search_kernel   one thread per candidate: runs the float64 orbit and
//                       keeps only running statistics (min/max/mean/M2 per
//                       axis, runaway / non-finite flags) -> the acceptance
//                       test of the category search needs no point storage
//   ifs_points_kernel   one thread per instance, 32 steps at a time: writes the float32 cloud
//   voxel_bbox / voxel_paint   per-cloud bounding box (block reduction), then
//                       isotropic normalise + centre + floor + clip and paint
//                       the class colour / label straight into the shard-local
//                       (3,d,h,w) fp32 volume and uint16 mask
//
// Role of the reference: ScaFFold/datagen/generate_fractal_points.py:23-126,
// ScaFFold/datagen/category_search.py:114-201, ScaFFold/datagen/volumegen.py:103-160,259-294.
#include "common.cuh"
#include "host_api.h"
#include "ifs_common.h"

namespace sb {
using namespace sbifs;

__global__ void ifs_search_kernel(const double* __restrict__ params, const unsigned long long* __restrict__ seeds,
                                  int batch, long long n, double* __restrict__ out) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  double P[26];
  for (int i = 0; i < 26; ++i) P[i] = params[(size_t)b * 26 + i];
  Rng rng{seeds[b]};
  Stats st;
  stats_init(st);
  double x = 0, y = 0, z = 0;
  const double p0 = P[12];
  for (long long i = 0; i < n; ++i) {
    if (i > 0) step(P, p0, rng, x, y, z);
    stats_add(st, x, y, z);
  }
  double* o = out + (size_t)b * 16;
  for (int a = 0; a < 3; ++a) {
    o[a] = st.mn[a];
    o[3 + a] = st.mx[a];
    o[6 + a] = st.mean[a];
    o[9 + a] = st.count > 0 ? st.m2[a] / (double)st.count : 0.0;
  }
  o[12] = (double)st.count;
  o[13] = st.runaway;
  o[14] = st.nonfinite;
  o[15] = 0;
}

// One block per 32 orbits. What bounds it is the orbit itself: every point depends on the last (four dependent fp64
// operations), and a few hundred orbits are a few dozen warps on 148 SMs. So the first warp walks the orbits, one per
// lane, and does nothing else: it selects the step's map in registers (not from local memory at a dynamic index) and
// leaves the points in shared memory. Meanwhile the other three draw the choices of the next 32 steps (the stream's
// state is a counter, so a draw needs no earlier one) and store the last 32 steps, 32 consecutive floats of one orbit at
// a time instead of 12 bytes of 32 orbits. 725 orbits of 8192 points: one thread per orbit doing all of it 1515 us,
// now 867 us.
constexpr int IFS_TILE = 32;                 // steps between two barriers
constexpr int IFS_ROW = 3 * IFS_TILE + 1;    // floats per orbit of a tile; odd: the lanes of a step hit 32 banks

__global__ void __launch_bounds__(128) ifs_points_kernel(const double* __restrict__ params,
                                                         const unsigned long long* __restrict__ seeds, int batch,
                                                         long long n, float* __restrict__ pts,
                                                         int* __restrict__ flags) {
  __shared__ float tile[2][32 * IFS_ROW];
  __shared__ uint32_t choice[2][IFS_TILE];   // [step]: bit o set, orbit o takes the first map
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b0 = blockIdx.x * 32;
  const int b = b0 + lane < batch ? b0 + lane : batch - 1;  // idle lanes of the last block repeat its last orbit
  const int orbits = batch - b0 < 32 ? batch - b0 : 32;
  const double p0 = params[(size_t)b * 26 + 12];
  const unsigned long long seed = seeds[b];
  const long long tiles = (n + IFS_TILE - 1) / IFS_TILE;

  // Step k > 0 takes draw k - 1; draws of step 0 and of steps past the last point are never used.
  auto draw = [&](long long t, int first, int every) {
    for (int j = first; j < IFS_TILE; j += every) {
      Rng r{seed + (unsigned long long)(t * IFS_TILE + j - 1) * RNG_STEP};
      const uint32_t bits = __ballot_sync(0xffffffffu, next_unit(r) < p0);
      if (lane == 0) choice[t & 1][j] = bits;
    }
  };
  draw(0, warp, 4);
  __syncthreads();

  double A[12], B[12];
  for (int i = 0; i < 12; ++i) {
    A[i] = warp == 0 ? params[(size_t)b * 26 + i] : 0.0;
    B[i] = warp == 0 ? params[(size_t)b * 26 + 13 + i] : 0.0;
  }
  double x = 0, y = 0, z = 0;
  int bad = 0;
  for (long long t = 0; t <= tiles; ++t) {
    if (warp == 0) {
      if (t < tiles) {
        const long long base = t * IFS_TILE;
        const int steps = n - base < IFS_TILE ? (int)(n - base) : IFS_TILE;
        float* row = tile[t & 1] + lane * IFS_ROW;
#pragma unroll 4
        for (int j = 0; j < steps; ++j) {
          if (base + j > 0) {
            const bool pick = (choice[t & 1][j] >> lane) & 1u;
            double m[12];
#pragma unroll
            for (int i = 0; i < 12; ++i) m[i] = pick ? A[i] : B[i];
            const double nx = x * m[0] + y * m[1] + z * m[2] + m[9];
            const double ny = x * m[3] + y * m[4] + z * m[5] + m[10];
            const double nz = x * m[6] + y * m[7] + z * m[8] + m[11];
            x = nx; y = ny; z = nz;
          }
          if (!(fabs(x) <= 1e10 && fabs(y) <= 1e10 && fabs(z) <= 1e10)) {
            if (!(x == x) || !(y == y) || !(z == z)) bad |= 2;
            if (fabs(x) > 1e10 || fabs(y) > 1e10 || fabs(z) > 1e10) bad |= 1;
          }
          row[3 * j] = (float)x;
          row[3 * j + 1] = (float)y;
          row[3 * j + 2] = (float)z;
        }
      }
    } else {
      if (t + 1 < tiles) draw(t + 1, warp - 1, 3);
      if (t > 0) {
        const long long base = (t - 1) * IFS_TILE;
        const int vals = 3 * (n - base < IFS_TILE ? (int)(n - base) : IFS_TILE);
        const float* src = tile[(t - 1) & 1];
        for (int o = warp - 1; o < orbits; o += 3) {
          float* dst = pts + ((size_t)(b0 + o) * n + base) * 3;
          for (int i = lane; i < vals; i += 32) dst[i] = src[o * IFS_ROW + i];
        }
      }
    }
    __syncthreads();
  }
  if (warp == 0 && b0 + lane < batch) flags[b] = bad;
}

// bbox[cloud][6] = min xyz, max xyz ; one block per cloud
__global__ void __launch_bounds__(256) voxel_bbox_kernel(const float* __restrict__ pts, long long n,
                                                         float* __restrict__ bbox) {
  __shared__ float smin[3][256], smax[3][256];
  const float* p = pts + (size_t)blockIdx.x * n * 3;
  float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (long long i = threadIdx.x; i < n; i += 256)
    for (int a = 0; a < 3; ++a) {
      const float c = p[3 * i + a];
      mn[a] = fminf(mn[a], c);
      mx[a] = fmaxf(mx[a], c);
    }
  for (int a = 0; a < 3; ++a) { smin[a][threadIdx.x] = mn[a]; smax[a][threadIdx.x] = mx[a]; }
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int a = 0; a < 3; ++a) {
        smin[a][threadIdx.x] = fminf(smin[a][threadIdx.x], smin[a][threadIdx.x + s]);
        smax[a][threadIdx.x] = fmaxf(smax[a][threadIdx.x], smax[a][threadIdx.x + s]);
      }
    __syncthreads();
  }
  if (threadIdx.x < 3) {
    bbox[blockIdx.x * 6 + threadIdx.x] = smin[threadIdx.x][0];
    bbox[blockIdx.x * 6 + 3 + threadIdx.x] = smax[threadIdx.x][0];
  }
}

// Paints cloud `blockIdx.y` into the shard [lo, hi) of a G^3 grid. Later clouds overwrite earlier
// ones where they overlap only if launched later: callers paint the clouds of a volume one launch each.
__global__ void __launch_bounds__(256) voxel_paint_kernel(const float* __restrict__ pts, long long n,
                                                          const float* __restrict__ bbox, int G, int lo_d, int lo_h,
                                                          int lo_w, int sd, int sh, int sw, float r, float g,
                                                          float b, unsigned short label, float* __restrict__ vol,
                                                          unsigned short* __restrict__ mask) {
  const double mn[3] = {bbox[0], bbox[1], bbox[2]};
  const double ex[3] = {(double)bbox[3] - bbox[0], (double)bbox[4] - bbox[1], (double)bbox[5] - bbox[2]};
  const double ext = fmax(ex[0], fmax(ex[1], ex[2]));
  const double voxel = (ext + 1e-6) / G;
  const size_t plane = (size_t)sd * sh * sw;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    int idx[3];
    for (int a = 0; a < 3; ++a) {
      const double off = (G - ex[a] / voxel) / 2.0;
      long long v = (long long)floor(((double)pts[3 * i + a] - mn[a]) / voxel + off);
      idx[a] = (int)(v < 0 ? 0 : (v > G - 1 ? G - 1 : v));
    }
    const int d = idx[0] - lo_d, h = idx[1] - lo_h, w = idx[2] - lo_w;
    if (d < 0 || d >= sd || h < 0 || h >= sh || w < 0 || w >= sw) continue;
    const size_t o = ((size_t)d * sh + h) * sw + w;
    vol[o] = r;
    vol[plane + o] = g;
    vol[2 * plane + o] = b;
    mask[o] = label;
  }
}

}  // namespace sb

using namespace sb;

extern "C" int sb_ifs_search(const double* params, const unsigned long long* seeds, int batch, long long n,
                             double* out, cudaStream_t stream) {
  ifs_search_kernel<<<(batch + 63) / 64, 64, 0, stream>>>(params, seeds, batch, n, out);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_ifs_points(const double* params, const unsigned long long* seeds, int batch, long long n,
                             float* pts, int* flags, cudaStream_t stream) {
  ifs_points_kernel<<<(batch + 31) / 32, 128, 0, stream>>>(params, seeds, batch, n, pts, flags);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_voxel_bbox(const float* pts, int clouds, long long n, float* bbox, cudaStream_t stream) {
  voxel_bbox_kernel<<<clouds, 256, 0, stream>>>(pts, n, bbox);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_voxel_paint(const float* pts, long long n, const float* bbox, int G, const int* lo,
                              const int* shape, const float* rgb, int label, float* vol, unsigned short* mask,
                              cudaStream_t stream) {
  long long blocks = (n + 255) / 256;
  if (blocks > 1024) blocks = 1024;
  voxel_paint_kernel<<<(unsigned)blocks, 256, 0, stream>>>(pts, n, bbox, G, lo[0], lo[1], lo[2], shape[0], shape[1],
                                                          shape[2], rgb[0], rgb[1], rgb[2], (unsigned short)label,
                                                          vol, mask);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}
