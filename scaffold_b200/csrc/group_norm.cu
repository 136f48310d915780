// GroupNorm (+ fused ReLU) for channels-last bf16 activations, forward and
// backward, with statistics that can span several spatial shards.
//
// Forward, two streaming passes (3 tensor-volumes of traffic):
//   gn_stats_kernel     per (split, n) CTA: Welford-style (count, mean, M2)
//                       partials for all G groups over a contiguous voxel range
//   gn_apply_kernel     every CTA merges the partials of its sample in index
//                       order (Chan's formula; deterministic), then
//                       y = relu((x - mean) * rstd * w + b), stored in bf16
// Backward, two streaming passes (5 volumes):
//   gn_bwd_partial      per (split, n): per-channel sum(dy') and sum(dy' * xhat),
//                       dy' = dy gated by the recomputed ReLU mask
//   gn_bwd_dx           merges partials, dx = rstd * (dy' w - c1 - xhat c2);
//                       CTA (0,0) also reduces dweight / dbias over samples
//
// "Peer" partial blocks: both merge steps walk `n_parts` partial buffers (this
// rank's first, then its spatial neighbours' through peer pointers), which
// makes a sharded volume normalise exactly like the unsharded one.
//
// Every thread owns 8 consecutive channels (one 16-byte vector) of a voxel, so
// all global accesses are full coalesced 16-byte vectors.
//
// Role of the reference: ScaFFold/unet/triton_group_norm.py:594-1043.
#include <atomic>

#include "common.cuh"
#include "host_api.h"

namespace sb {

constexpr int GN_THREADS = 256;
constexpr int GN_MAX_PARTS = 8;

struct GnParams {
  const __nv_bfloat16* x;
  const __nv_bfloat16* dy;
  __nv_bfloat16* y;   // forward output / backward dx
  const float* w;
  const float* b;
  float* mean;   // [N, G]
  float* rstd;   // [N, G]
  float* part;   // this rank's partials
  float* fin;    // optional: the last block of a statistics / backward-sums launch also collapses the partials here
  unsigned int* ticket;  // block counter of that hand-over (zero before the launch, reset by the last block)
  const float* parts[GN_MAX_PARTS];  // partial buffers to merge (own first)
  int n_parts;
  float* dw;     // [C]
  float* db;     // [C]
  int N, C, G;
  long long S;   // voxels per sample (local shard)
  int nsplit;
  float eps;
  int relu;
  int accumulate;     // add to dw / db
  float group_elems;  // elements per (n, g) over ALL shards = S_total * C/G
  const uint32_t* wait_flags;  // optional: peers' "statistics landed" flags (local memory)
  uint32_t wait_epoch;
  long long wait_ticks;
  uint32_t* status;
};

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]);
  o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]);
  o.w = pack_bf16x2(f[6], f[7]);
  return o;
}

__device__ __forceinline__ void chan_merge(float& n_a, float& mean_a, float& m2_a, float n_b, float mean_b,
                                           float m2_b) {
  if (n_b == 0.f) return;
  const float n = n_a + n_b;
  const float delta = mean_b - mean_a;
  const float r = n_b / n;
  mean_a += delta * r;
  m2_a += m2_b + delta * delta * n_a * r;
  n_a = n;
}


// Pooled (count, mean, M2) of a set of partials as three plain sums in double: count, count * mean and
// M2 + count * mean^2. No division stands in the chain (Chan's merge has one per partial), the loads of a thread are
// independent, and double leaves nothing of the cancellation in M2 = S2 - S1^2 / count at fp32.
struct StatSums {
  double n, s1, s2;
};
__device__ __forceinline__ void stat_add(StatSums& a, float n, float mean, float m2) {
  const double nm = (double)n * (double)mean;
  a.n += (double)n;
  a.s1 += nm;
  a.s2 += (double)m2 + nm * (double)mean;
}
__device__ __forceinline__ void stat_store(float* dst, const StatSums& a) {
  const double mean = a.n > 0.0 ? a.s1 / a.n : 0.0;
  const double m2 = a.s2 - a.s1 * mean;
  dst[0] = (float)a.n;
  dst[1] = (float)mean;
  dst[2] = (float)(m2 < 0.0 ? 0.0 : m2);  // a NaN stays one: an overflow has to show in what follows
}
// The sums of partials first, first + step, ... of (n, g) (`base`: partial 0), FLIGHT partials in flight. Loads bypass
// L1 (the partials may have been written by other SMs during this launch).
template <int FLIGHT>
__device__ __forceinline__ StatSums stat_walk(const float* __restrict__ base, int G, int first, int step, int nsplit) {
  StatSums a{0.0, 0.0, 0.0};
  for (int s = first; s < nsplit; s += FLIGHT * step) {
    float e[FLIGHT][3];
#pragma unroll
    for (int u = 0; u < FLIGHT; ++u) {
      const float* q = base + (long long)(s + u * step) * G * 3;
      if (s + u * step < nsplit) { e[u][0] = __ldcg(q); e[u][1] = __ldcg(q + 1); e[u][2] = __ldcg(q + 2); }
    }
#pragma unroll
    for (int u = 0; u < FLIGHT; ++u)
      if (s + u * step < nsplit) stat_add(a, e[u][0], e[u][1], e[u][2]);
  }
  return a;
}
__device__ __forceinline__ StatSums stat_warp_sum(StatSums a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a.n += __shfl_xor_sync(0xffffffffu, a.n, o);
    a.s1 += __shfl_xor_sync(0xffffffffu, a.s1, o);
    a.s2 += __shfl_xor_sync(0xffffffffu, a.s2, o);
  }
  return a;
}

// One warp collapses the `nsplit` partials of (n, g): up to 32 of them one per lane, more as GN_FIN_WARPS strands (32
// lanes each, partials strand * 32 + lane, + 128, ...) whose sums it adds in order. The separate finalize launch gives
// each strand a warp of its own (gn_stats_finalize_block_kernel) and takes the same sums in the same order, so it and
// the last-block tail of the statistics kernel give the same bits.
// 592 partials, kernel time: 13 us as a chain of Chan merges (one L2 latency and one division each).
constexpr int GN_FIN_WARPS = 4;
__device__ __forceinline__ void stats_collapse_warp(const float* __restrict__ part, float* __restrict__ fin, int G,
                                                    int nsplit, int n, int g, int lane) {
  const float* base = part + ((long long)n * nsplit * G + g) * 3;
  StatSums t{0.0, 0.0, 0.0};
  const int strands = nsplit > 32 ? GN_FIN_WARPS : 1;
  for (int w = 0; w < strands; ++w) {
    // (five in flight: all of a lane's share of 592, and with eight the statistics kernel takes 80 registers instead of
    // 64, so one block per SM less: 75 us more for ten launches at 3 x 35x32x28 voxels of 16 channels)
    const StatSums a = stat_warp_sum(stat_walk<5>(base, G, w * 32 + lane, strands * 32, nsplit));
    t.n += a.n; t.s1 += a.s1; t.s2 += a.s2;
  }
  if (lane == 0) stat_store(fin + ((long long)n * G + g) * 3, t);
}

__device__ __forceinline__ void bwd_collapse_warp(const float* __restrict__ part, float* __restrict__ fin, int C,
                                                  int nsplit, int n, int c, int lane) {
  float a = 0.f, b = 0.f;
  for (int s = lane; s < nsplit; s += 8 * 32) {
    float2 e[8];  // eight in flight, the last ones too
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (s + u * 32 < nsplit)
        e[u] = __ldcg(reinterpret_cast<const float2*>(part + (((long long)n * nsplit + s + u * 32) * C + c) * 2));
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (s + u * 32 < nsplit) { a += e[u].x; b += e[u].y; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    float* dst = fin + ((long long)n * C + c) * 2;
    dst[0] = a; dst[1] = b;
  }
}

// True in every thread of the block that finished last (all blocks' global writes are then visible to it).
__device__ __forceinline__ bool last_block_done(unsigned int* ticket) {
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned int total = gridDim.x * gridDim.y;
    s_last = atomicAdd(ticket, 1u) == total - 1u ? 1 : 0;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last != 0;
}

// ----------------------------------------------------------------------------
// forward: statistics
// ----------------------------------------------------------------------------
__global__ void __launch_bounds__(GN_THREADS) gn_stats_kernel(const GnParams p) {
  __shared__ float s_n[GN_THREADS * 4], s_mean[GN_THREADS * 4], s_m2[GN_THREADS * 4];
  const int split = blockIdx.x, n = blockIdx.y;
  const int tpv = p.C / 8;            // threads per voxel
  const int vpb = GN_THREADS / tpv;   // voxels per block iteration
  const int oct = threadIdx.x % tpv;
  const int vl = threadIdx.x / tpv;
  const int cg = p.C / p.G;
  const long long chunk = (p.S + p.nsplit - 1) / p.nsplit;
  const long long v0 = (long long)split * chunk;
  const long long v1 = v0 + chunk < p.S ? v0 + chunk : p.S;
  const __nv_bfloat16* xb = p.x + (long long)n * p.S * p.C + oct * 8;

  float s[8], q[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) { s[i] = 0.f; q[i] = 0.f; }
  float cnt = 0.f;
  // first value of the thread is the shift: sums of (x - shift) stay small
  float shift[8];
  bool have_shift = false;
  if (vl < vpb) {
    auto body = [&](const uint4 raw) {
      float f[8];
      unpack8(raw, f);
      if (!have_shift) {
#pragma unroll
        for (int i = 0; i < 8; ++i) shift[i] = f[i];
        have_shift = true;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float d = f[i] - shift[i];
        s[i] += d;
        q[i] += d * d;
      }
      cnt += 1.f;
    };
    for (long long v = v0 + vl; v < v1; v += vpb) body(__ldg(reinterpret_cast<const uint4*>(xb + v * p.C)));
  }
  // per-thread (count, mean, M2) for each group it touches (ngt = max(1, 8/cg) groups)
  const int ngt = cg >= 8 ? 1 : 8 / cg;
  const int cpg = 8 / ngt;  // channels of this thread per group
  for (int gi = 0; gi < ngt; ++gi) {
    float gn = 0.f, gm = 0.f, g2 = 0.f;
    if (cnt > 0.f) {
      for (int j = 0; j < cpg; ++j) {
        const int i = gi * cpg + j;
        const float m = s[i] / cnt;
        const float m2 = fmaxf(q[i] - s[i] * m, 0.f);
        chan_merge(gn, gm, g2, cnt, m + shift[i], m2);
      }
    }
    s_n[threadIdx.x * 4 + gi] = gn;
    s_mean[threadIdx.x * 4 + gi] = gm;
    s_m2[threadIdx.x * 4 + gi] = g2;
  }
  __syncthreads();
  // one thread per group merges that group's entries in thread order
  if (threadIdx.x < p.G) {
    const int g = threadIdx.x;
    float gn = 0.f, gm = 0.f, g2 = 0.f;
    // channels of group g: [g*cg, (g+1)*cg) -> octs [g*cg/8, ...]
    const int oct0 = (g * cg) / 8;
    const int octs = cg >= 8 ? cg / 8 : 1;
    const int gi = cg >= 8 ? 0 : (g * cg % 8) / cg;
    for (int v = 0; v < vpb; ++v)
      for (int o = 0; o < octs; ++o) {
        const int t = v * tpv + oct0 + o;
        chan_merge(gn, gm, g2, s_n[t * 4 + gi], s_mean[t * 4 + gi], s_m2[t * 4 + gi]);
      }
    float* dst = p.part + (((long long)n * p.nsplit + split) * p.G + g) * 3;
    dst[0] = gn;
    dst[1] = gm;
    dst[2] = g2;
  }
  if (p.fin != nullptr && last_block_done(p.ticket)) {
    // the last block to finish collapses every (n, g): no separate finalize launch
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int o = warp; o < p.N * p.G; o += GN_THREADS / 32)
      stats_collapse_warp(p.part, p.fin, p.G, p.nsplit, o / p.G, o % p.G, lane);
    if (threadIdx.x == 0) *p.ticket = 0u;
  }
}

// Bounded wait until every peer's statistics landed; returns false (after reporting) on timeout.
__device__ __forceinline__ bool gn_wait_peers(const GnParams& p, uint32_t site) {
  if (p.wait_flags == nullptr) return true;
  int ok = 1;
  if (threadIdx.x < p.n_parts) {
    const long long t0 = clock64();
    while (true) {
      uint32_t v;
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p.wait_flags + threadIdx.x) : "memory");
      if ((int)(v - p.wait_epoch) >= 0) break;
      if (clock64() - t0 > p.wait_ticks) {
        report(p.status, ST_FLAG_TIMEOUT, site, threadIdx.x, p.wait_epoch);
        ok = 0;
        break;
      }
      __nanosleep(32);
    }
  }
  return __syncthreads_and(ok) != 0;
}

// merges every partial of sample n, group g, in (part buffer, split) order
__device__ __forceinline__ void merge_group(const GnParams& p, int n, int g, float& mean, float& rstd) {
  float gn = 0.f, gm = 0.f, g2 = 0.f;
  for (int pi = 0; pi < p.n_parts; ++pi) {
    const float* base = p.parts[pi] + ((long long)n * p.nsplit * p.G + g) * 3;
    for (int s = 0; s < p.nsplit; ++s) {
      const float* e = base + (long long)s * p.G * 3;
      chan_merge(gn, gm, g2, e[0], e[1], e[2]);
    }
  }
  mean = gm;
  rstd = rsqrtf(g2 / gn + p.eps);
}

// ----------------------------------------------------------------------------
// The three streaming kernels are bound by memory and need some 45 KB of loads in flight per SM. They run in ONE wave
// of GN_WAVE (the sums: GN_WAVE_SUMS) blocks per SM at 64 (85) registers a thread, each thread with as many 16-byte
// loads in flight as fit. What made room: an octet of channels covers GP groups (1 for the usual eight or more channels
// per group), so means and the like are GP registers instead of 8; the ReLU's mask is the sign of the forward's own
// x * a + c, whose `a` is also dx's factor of dy; and xhat is never formed: dx is linear in x - mean, and
// sum(dy xhat) = rstd * sum(dy (x - mean)). With 97 / 92 registers two blocks fitted per SM, and four blocks' worth of
// them came in two waves. 64 channels at 2 x 128^3, before / after: sums 225 / 176 us (6.1 TB/s), dx 295 / 248 us
// (6.5 TB/s), forward 186 / 181 us (5.9 TB/s).
// ----------------------------------------------------------------------------
constexpr int GN_WAVE = 4;
constexpr int GN_WAVE_SUMS = 3;  // the backward sums: 16 more registers of accumulators

// ----------------------------------------------------------------------------
// forward: normalise + affine + ReLU
// ----------------------------------------------------------------------------
__global__ void __launch_bounds__(GN_THREADS, GN_WAVE) gn_apply_kernel(const GnParams p) {
  __shared__ float s_mean[256], s_rstd[256];
  const int n = blockIdx.y;
  if (!gn_wait_peers(p, 61)) return;
  for (int g = threadIdx.x; g < p.G; g += GN_THREADS) {
    float m, r;
    merge_group(p, n, g, m, r);
    s_mean[g] = m;
    s_rstd[g] = r;
    if (blockIdx.x == 0) {
      p.mean[n * p.G + g] = m;
      p.rstd[n * p.G + g] = r;
    }
  }
  __syncthreads();
  const int tpv = p.C / 8;
  const int vpb = GN_THREADS / tpv;
  const int oct = threadIdx.x % tpv;
  const int vl = threadIdx.x / tpv;
  if (vl >= vpb) return;
  const int cg = p.C / p.G;
  float a[8], c[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int ch = oct * 8 + i;
    const int g = ch / cg;
    a[i] = s_rstd[g] * p.w[ch];
    c[i] = p.b[ch] - s_mean[g] * a[i];
  }
  const long long base = (long long)n * p.S * p.C + oct * 8;
  auto body = [&](const uint4 raw, long long v) {
    float f[8];
    unpack8(raw, f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float yv = fmaf(f[i], a[i], c[i]);
      if (p.relu) yv = yv <= 0.f ? 0.f : yv;  // NaN propagates
      f[i] = yv;
    }
    *reinterpret_cast<uint4*>(p.y + base + v * p.C) = pack8(f);
  };
  // four voxels (four 16-byte loads) in flight per thread
  const long long stride = (long long)gridDim.x * vpb;
  long long v = (long long)blockIdx.x * vpb + vl;
  for (; v + 3 * stride < p.S; v += 4 * stride) {
    uint4 r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = __ldg(reinterpret_cast<const uint4*>(p.x + base + (v + u * stride) * p.C));
#pragma unroll
    for (int u = 0; u < 4; ++u) body(r[u], v + u * stride);
  }
  for (; v < p.S; v += stride) body(__ldg(reinterpret_cast<const uint4*>(p.x + base + v * p.C)), v);
}

// ----------------------------------------------------------------------------
// backward: per-channel partial sums
// ----------------------------------------------------------------------------
template <int GP>
__global__ void __launch_bounds__(GN_THREADS, GN_WAVE_SUMS) gn_bwd_partial_kernel(const GnParams p) {
  __shared__ float s_a[GN_THREADS * 8], s_b[GN_THREADS * 8];
  const int split = blockIdx.x, n = blockIdx.y;
  const int tpv = p.C / 8;
  const int vpb = GN_THREADS / tpv;
  const int oct = threadIdx.x % tpv;
  const int vl = threadIdx.x / tpv;
  const int cg = p.C / p.G;
  const long long chunk = (p.S + p.nsplit - 1) / p.nsplit;
  const long long v0 = (long long)split * chunk;
  const long long v1 = v0 + chunk < p.S ? v0 + chunk : p.S;
  float a[8], c[8], A[8], B[8], mu[GP];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int ch = oct * 8 + i;
    const int g = ch / cg;
    a[i] = p.rstd[n * p.G + g] * p.w[ch];
    c[i] = p.b[ch] - p.mean[n * p.G + g] * a[i];
    if (i % (8 / GP) == 0) mu[i / (8 / GP)] = p.mean[n * p.G + g];
    A[i] = 0.f;
    B[i] = 0.f;
  }
  const long long base = (long long)n * p.S * p.C + oct * 8;
  if (vl < vpb) {
    auto body = [&](const uint4 rx, const uint4 rd) {
      float fx[8], fd[8];
      unpack8(rx, fx);
      unpack8(rd, fd);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float d = fd[i];
        if (p.relu && fmaf(fx[i], a[i], c[i]) <= 0.f) d = 0.f;
        A[i] += d;
        B[i] = fmaf(d, fx[i] - mu[i / (8 / GP)], B[i]);
      }
    };
    // two voxels (four 16-byte loads) in flight per thread; the summation order per thread is unchanged
    const __nv_bfloat16* px = p.x + base + (v0 + vl) * p.C;
    const __nv_bfloat16* pd = p.dy + base + (v0 + vl) * p.C;
    const long long row = (long long)vpb * p.C;
    long long v = v0 + vl;
    for (; v + vpb < v1; v += 2 * vpb, px += 2 * row, pd += 2 * row) {
      const uint4 rx0 = __ldg(reinterpret_cast<const uint4*>(px));
      const uint4 rd0 = __ldg(reinterpret_cast<const uint4*>(pd));
      const uint4 rx1 = __ldg(reinterpret_cast<const uint4*>(px + row));
      const uint4 rd1 = __ldg(reinterpret_cast<const uint4*>(pd + row));
      body(rx0, rd0);
      body(rx1, rd1);
    }
    for (; v < v1; v += vpb, px += row, pd += row)
      body(__ldg(reinterpret_cast<const uint4*>(px)), __ldg(reinterpret_cast<const uint4*>(pd)));
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) B[i] *= p.rstd[n * p.G + (oct * 8 + i) / cg];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    s_a[threadIdx.x * 8 + i] = A[i];
    s_b[threadIdx.x * 8 + i] = B[i];
  }
  __syncthreads();
  for (int ch = threadIdx.x; ch < p.C; ch += GN_THREADS) {
    const int o = ch / 8, j = ch % 8;
    float sa = 0.f, sbv = 0.f;
    for (int v = 0; v < vpb; ++v) {
      const int t = v * tpv + o;
      sa += s_a[t * 8 + j];
      sbv += s_b[t * 8 + j];
    }
    float* dst = p.part + (((long long)n * p.nsplit + split) * p.C + ch) * 2;
    dst[0] = sa;
    dst[1] = sbv;
  }
  if (p.fin != nullptr && last_block_done(p.ticket)) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int o = warp; o < p.N * p.C; o += GN_THREADS / 32)
      bwd_collapse_warp(p.part, p.fin, p.C, p.nsplit, o / p.C, o % p.C, lane);
    if (threadIdx.x == 0) *p.ticket = 0u;
  }
}

// ----------------------------------------------------------------------------
// backward: dx (+ dweight / dbias)
// ----------------------------------------------------------------------------
template <int GP>
__global__ void __launch_bounds__(GN_THREADS, GN_WAVE) gn_bwd_dx_kernel(const GnParams p) {
  extern __shared__ float sm[];
  float* s_A = sm;              // [C] this rank's sum(dy')
  float* s_B = sm + p.C;        // [C] this rank's sum(dy' xhat)
  float* s_c1 = sm + 2 * p.C;   // [G]
  float* s_c2 = s_c1 + p.G;     // [G]
  float* s_At = s_c2 + p.G;     // [C] all shards, times the weight
  float* s_Bt = s_At + p.C;
  const int n = blockIdx.y;
  const int cg = p.C / p.G;
  if (!gn_wait_peers(p, 62)) return;
  // What a thread needs of its own channels is read ahead of the collapse below: on a small tensor this prologue is most
  // of the launch, and its phases are one L2 latency each.
  const int tpv = p.C / 8;
  const int vpb = GN_THREADS / tpv;
  const int oct = threadIdx.x % tpv;
  const int vl = threadIdx.x / tpv;
  float a[8], c[8], mu[GP], rs[GP];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int ch = oct * 8 + i;
    const int g = ch / cg;
    const float m = p.mean[n * p.G + g], r = p.rstd[n * p.G + g];
    a[i] = r * p.w[ch];
    c[i] = p.b[ch] - m * a[i];
    if (i % (8 / GP) == 0) {
      mu[i / (8 / GP)] = m;
      rs[i / (8 / GP)] = r;
    }
  }
  for (int ch = threadIdx.x; ch < p.C; ch += GN_THREADS) {
    const float wc = p.w[ch];
    float At = 0.f, Bt = 0.f, A0 = 0.f, B0 = 0.f;
    for (int pi = 0; pi < p.n_parts; ++pi) {
      const float* base = p.parts[pi] + ((long long)n * p.nsplit * p.C + ch) * 2;
      float a = 0.f, b = 0.f;
      for (int s = 0; s < p.nsplit; ++s) {
        a += base[(long long)s * p.C * 2];
        b += base[(long long)s * p.C * 2 + 1];
      }
      if (pi == 0) { A0 = a; B0 = b; }
      At += a;
      Bt += b;
    }
    s_A[ch] = A0; s_B[ch] = B0; s_At[ch] = wc * At; s_Bt[ch] = wc * Bt;
  }
  __syncthreads();
  for (int g = threadIdx.x; g < p.G; g += GN_THREADS) {
    float c1 = 0.f, c2 = 0.f;
    for (int j = 0; j < cg; ++j) {
      const int ch = g * cg + j;
      c1 += s_At[ch];
      c2 += s_Bt[ch];
    }
    s_c1[g] = c1 / p.group_elems;
    s_c2[g] = c2 / p.group_elems;
  }
  __syncthreads();
  // dweight / dbias: this rank's share, summed over samples in index order
  if (blockIdx.x == 0 && blockIdx.y == 0 && p.dw != nullptr) {
    for (int ch = threadIdx.x; ch < p.C; ch += GN_THREADS) {
      float a = s_A[ch], b = s_B[ch];  // sample 0 is this block's
      for (int nn = 1; nn < p.N; ++nn) {
        const float* base = p.parts[0] + ((long long)nn * p.nsplit * p.C + ch) * 2;
        for (int s = 0; s < p.nsplit; ++s) {
          a += base[(long long)s * p.C * 2];
          b += base[(long long)s * p.C * 2 + 1];
        }
      }
      p.db[ch] = p.accumulate ? p.db[ch] + a : a;
      p.dw[ch] = p.accumulate ? p.dw[ch] + b : b;
    }
  }
  if (vl >= vpb) return;
  // dx = rstd (d w - c1 - xhat c2) = d a + (x - mean) q + r
  float q[GP], r[GP];
#pragma unroll
  for (int i = 0; i < GP; ++i) {
    const int g = (oct * 8 + i * (8 / GP)) / cg;
    q[i] = -rs[i] * rs[i] * s_c2[g];
    r[i] = -rs[i] * s_c1[g];
  }
  const long long base = (long long)n * p.S * p.C + oct * 8;
  auto body = [&](const uint4 rx, const uint4 rd, long long at) {
    float fx[8], fd[8];
    unpack8(rx, fx);
    unpack8(rd, fd);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float d = fd[i];
      if (p.relu && fmaf(fx[i], a[i], c[i]) <= 0.f) d = 0.f;
      fx[i] = fmaf(d, a[i], fmaf(fx[i] - mu[i / (8 / GP)], q[i / (8 / GP)], r[i / (8 / GP)]));
    }
    *reinterpret_cast<uint4*>(p.y + at) = pack8(fx);
  };
  // two voxels (four 16-byte loads) in flight per thread
  const long long stride = (long long)gridDim.x * vpb;
  const long long row = stride * p.C;
  long long v = (long long)blockIdx.x * vpb + vl;
  long long at = base + v * p.C;
  for (; v + stride < p.S; v += 2 * stride, at += 2 * row) {
    const uint4 rx0 = __ldg(reinterpret_cast<const uint4*>(p.x + at));
    const uint4 rd0 = __ldg(reinterpret_cast<const uint4*>(p.dy + at));
    const uint4 rx1 = __ldg(reinterpret_cast<const uint4*>(p.x + at + row));
    const uint4 rd1 = __ldg(reinterpret_cast<const uint4*>(p.dy + at + row));
    body(rx0, rd0, at);
    body(rx1, rd1, at + row);
  }
  for (; v < p.S; v += stride, at += row)
    body(__ldg(reinterpret_cast<const uint4*>(p.x + at)), __ldg(reinterpret_cast<const uint4*>(p.dy + at)), at);
}

// ----------------------------------------------------------------------------
// finalize: collapse the per-split partials of one rank into a single entry per
// (n, g) / (n, c), in parallel and in a fixed order, so the
// streaming kernels start from O(1) statistics instead of walking every split.
// ----------------------------------------------------------------------------
__global__ void __launch_bounds__(GN_THREADS) gn_stats_finalize_kernel(const float* __restrict__ part,
                                                                       float* __restrict__ fin, int N, int G,
                                                                       int nsplit) {
  const int warp = (blockIdx.x * GN_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= N * G) return;
  stats_collapse_warp(part, fin, G, nsplit, warp / G, warp % G, lane);
}

// The same collapse with a block per (n, g), a warp per strand, beyond 32 partials: a lane's 16 partials were two trips
// to L2 and 16 dependent double additions, a thread's 4 are one trip (512 partials 4.9 us a launch, now 2.7).
constexpr int GN_FIN_THREADS = 32 * GN_FIN_WARPS;
__global__ void __launch_bounds__(GN_FIN_THREADS) gn_stats_finalize_block_kernel(const float* __restrict__ part,
                                                                                 float* __restrict__ fin, int G,
                                                                                 int nsplit) {
  __shared__ double s_w[GN_FIN_WARPS][3];
  const int n = blockIdx.x / G, g = blockIdx.x % G, warp = threadIdx.x >> 5;
  const StatSums a = stat_warp_sum(stat_walk<8>(part + ((long long)n * nsplit * G + g) * 3, G, threadIdx.x, GN_FIN_THREADS,
                                             nsplit));
  if ((threadIdx.x & 31) == 0) { s_w[warp][0] = a.n; s_w[warp][1] = a.s1; s_w[warp][2] = a.s2; }
  __syncthreads();
  if (threadIdx.x == 0) {
    StatSums t{0.0, 0.0, 0.0};
    for (int w = 0; w < GN_FIN_WARPS; ++w) { t.n += s_w[w][0]; t.s1 += s_w[w][1]; t.s2 += s_w[w][2]; }
    stat_store(fin + ((long long)n * G + g) * 3, t);
  }
}

// The same collapse for MANY partials per (n, g) (the per-warp partials a convolution's epilogue leaves: up to
// 16K per sample). Bound: L2 latency and the sectors around 12-byte entries, so a cluster of eight CTAs shares one
// (n, g): thread t of CTA r adds the partials r * 256 + t, + 2048, ..., each CTA adds its warps in order, and CTA 0
// reads the eight sums over distributed shared memory in rank order. 16K partials of 2 x 8 groups, call: 17.9 us with
// one CTA per (n, g), 10.4 us (the cost of the call itself) with the cluster.
constexpr int GN_WIDE_CLUSTER = 8;
__global__ void __cluster_dims__(GN_WIDE_CLUSTER, 1, 1) __launch_bounds__(GN_THREADS)
    gn_stats_finalize_wide_kernel(const float* __restrict__ part, float* __restrict__ fin, int N, int G, int nsplit) {
  __shared__ double s_w[GN_THREADS / 32][3];
  __shared__ double s_cta[3];
  const int out = blockIdx.x / GN_WIDE_CLUSTER, rank = blockIdx.x % GN_WIDE_CLUSTER;
  const int n = out / G, g = out % G, warp = threadIdx.x >> 5;
  const StatSums a = stat_warp_sum(stat_walk<8>(part + ((long long)n * nsplit * G + g) * 3, G,
                                             rank * GN_THREADS + threadIdx.x, GN_WIDE_CLUSTER * GN_THREADS, nsplit));
  if ((threadIdx.x & 31) == 0) { s_w[warp][0] = a.n; s_w[warp][1] = a.s1; s_w[warp][2] = a.s2; }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < GN_THREADS / 32; ++w) t += s_w[w][threadIdx.x];
    s_cta[threadIdx.x] = t;
  }
  __syncthreads();
  cluster_sync_all();
  if (rank == 0 && threadIdx.x == 0) {
    StatSums t{0.0, 0.0, 0.0};
    for (int r = 0; r < GN_WIDE_CLUSTER; ++r) {
      t.n += ld_cluster_f64(&s_cta[0], r);
      t.s1 += ld_cluster_f64(&s_cta[1], r);
      t.s2 += ld_cluster_f64(&s_cta[2], r);
    }
    stat_store(fin + ((long long)n * G + g) * 3, t);
  }
  __syncthreads();
  cluster_sync_all();  // no CTA leaves while its shared memory is still being read
}

__global__ void __launch_bounds__(GN_THREADS) gn_bwd_finalize_kernel(const float* __restrict__ part,
                                                                     float* __restrict__ fin, int N, int C,
                                                                     int nsplit) {
  const int warp = (blockIdx.x * GN_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= N * C) return;
  bwd_collapse_warp(part, fin, C, nsplit, warp / C, warp % C, lane);
}

// Channel / group counts the kernels cover: C a multiple of 8 in [8, 2048] (one thread per channel
// octet, at most GN_THREADS octets), G dividing C, and a group either a whole number of octets or a
// divisor of one octet holding at most four groups.
static bool gn_channels_ok(int C, int G) {
  if (C < 8 || C % 8 != 0 || C > 8 * GN_THREADS || G < 1 || G > 256 || C % G != 0) return false;
  const int cg = C / G;
  if (cg < 8 ? (8 % cg != 0) : (cg % 8 != 0)) return false;
  return !(cg < 8 && 8 / cg > 4);
}

static int gn_fill(const SbGnArgs* a, GnParams& p) {
  if (!gn_channels_ok(a->C, a->G) || a->N < 1 || a->S < 1) return SB_ERR_SHAPE;
  if (a->x == nullptr || a->w == nullptr || a->b == nullptr) return SB_ERR_SHAPE;
  const int cg = a->C / a->G;
  if (a->n_parts < 1 || a->n_parts > GN_MAX_PARTS) return SB_ERR_SHAPE;
  memset(&p, 0, sizeof(p));
  p.x = (const __nv_bfloat16*)a->x;
  p.dy = (const __nv_bfloat16*)a->dy;
  p.y = (__nv_bfloat16*)a->y;
  p.w = a->w; p.b = a->b; p.mean = a->mean; p.rstd = a->rstd;
  p.part = a->part;
  p.fin = a->fin;
  for (int i = 0; i < a->n_parts; ++i) p.parts[i] = a->parts[i];
  p.n_parts = a->n_parts;
  p.dw = a->dw; p.db = a->db;
  p.N = a->N; p.C = a->C; p.G = a->G; p.S = a->S;
  p.nsplit = a->nsplit;
  p.eps = a->eps;
  p.relu = a->relu;
  p.accumulate = a->accumulate;
  p.group_elems = (float)((double)a->S_total * cg);
  p.wait_flags = a->wait_flags;
  p.wait_epoch = a->wait_epoch;
  p.wait_ticks = (long long)((a->wait_s > 0 ? a->wait_s : 2.0) * 1.8e9);
  p.status = a->status;
  return 0;
}

// Block counters of the fused finalize: launches on one stream run one after another and each leaves its counter
// at zero, so a small rotating pool is plenty. The NAME is only a handle for cudaGetSymbolAddress in host code.
static __device__ unsigned int g_gn_tickets[256];
constexpr int GN_TICKET_DEVICES = 64;
static unsigned int* g_gn_ticket_ptr[GN_TICKET_DEVICES] = {nullptr};
static std::atomic<unsigned int> g_gn_ticket_seq{0};
static unsigned int* gn_ticket() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= GN_TICKET_DEVICES) return nullptr;
  if (g_gn_ticket_ptr[dev] == nullptr) {
    unsigned int* q = nullptr;
    if (cudaGetSymbolAddress((void**)&q, g_gn_tickets) != cudaSuccess || q == nullptr) return nullptr;
    g_gn_ticket_ptr[dev] = q;
  }
  return g_gn_ticket_ptr[dev] + (g_gn_ticket_seq.fetch_add(1u) % 256u);
}

// groups that eight consecutive channels cover: 1, 2 or 4 (gn_channels_ok)
static int groups_per_octet(const GnParams& p) { return p.C / p.G >= 8 ? 1 : 8 / (p.C / p.G); }

static int apply_blocks(const GnParams& p) {
  const int vpb = GN_THREADS / (p.C / 8);
  long long need = (p.S + vpb - 1) / vpb;
  long long cap = 148LL * GN_WAVE / p.N;  // one wave; more samples than its slots: one block each
  long long b = need < cap ? need : cap;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace sb

using namespace sb;

// 1 when the kernels cover GroupNorm over C channels in G groups, else 0 (callers then take another path)
extern "C" int sb_gn_supported(int C, int G) { return gn_channels_ok(C, G) ? 1 : 0; }

// Splits of a sample's voxels, at least `rows` rows of voxels (one per thread) in each.
static int gn_nsplit(int N, long long S, int C, int rows, int wave) {
  if (N < 1 || S < 1 || C < 8 || C / 8 > GN_THREADS) return 1;  // unsupported shapes are refused by the launchers
  const long long step = (long long)rows * (GN_THREADS / (C / 8));
  const long long maxs = (S + step - 1) / step;
  long long want = 148LL * wave / N;  // all samples' splits in one wave
  long long s = want < maxs ? want : maxs;
  if (s > 1024) s = 1024;
  return (int)(s < 1 ? 1 : s);
}

extern "C" int sb_gn_nsplit(int N, long long S, int C) { return gn_nsplit(N, S, C, 1, GN_WAVE); }

// Splits of the backward sums (never more than sb_gn_nsplit). Their partials have 2 C floats per split, so with one
// row of voxels per split a small wide tensor (512 voxels of 1024 channels) would write and read back twice its own
// bytes; four rows keep them below a quarter of the two tensors that the pass reads.
extern "C" int sb_gn_bwd_nsplit(int N, long long S, int C) { return gn_nsplit(N, S, C, 4, GN_WAVE_SUMS); }

extern "C" int sb_gn_stats(const SbGnArgs* a, cudaStream_t stream) {
  GnParams p;
  int rc = gn_fill(a, p);
  if (rc) return rc;
  if (p.fin != nullptr && (p.ticket = gn_ticket()) == nullptr) return SB_ERR_DRIVER;
  gn_stats_kernel<<<dim3(p.nsplit, p.N), GN_THREADS, 0, stream>>>(p);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_gn_apply(const SbGnArgs* a, cudaStream_t stream) {
  GnParams p;
  int rc = gn_fill(a, p);
  if (rc) return rc;
  gn_apply_kernel<<<dim3(apply_blocks(p), p.N), GN_THREADS, 0, stream>>>(p);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_gn_bwd_partial(const SbGnArgs* a, cudaStream_t stream) {
  GnParams p;
  int rc = gn_fill(a, p);
  if (rc) return rc;
  if (p.fin != nullptr && (p.ticket = gn_ticket()) == nullptr) return SB_ERR_DRIVER;
  const dim3 grid(p.nsplit, p.N);
  switch (groups_per_octet(p)) {
    case 1: gn_bwd_partial_kernel<1><<<grid, GN_THREADS, 0, stream>>>(p); break;
    case 2: gn_bwd_partial_kernel<2><<<grid, GN_THREADS, 0, stream>>>(p); break;
    default: gn_bwd_partial_kernel<4><<<grid, GN_THREADS, 0, stream>>>(p);
  }
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_gn_bwd_dx(const SbGnArgs* a, cudaStream_t stream) {
  GnParams p;
  int rc = gn_fill(a, p);
  if (rc) return rc;
  const size_t smem = (size_t)(4 * p.C + 2 * p.G) * sizeof(float);
  const dim3 grid(apply_blocks(p), p.N);
  switch (groups_per_octet(p)) {
    case 1: gn_bwd_dx_kernel<1><<<grid, GN_THREADS, smem, stream>>>(p); break;
    case 2: gn_bwd_dx_kernel<2><<<grid, GN_THREADS, smem, stream>>>(p); break;
    default: gn_bwd_dx_kernel<4><<<grid, GN_THREADS, smem, stream>>>(p);
  }
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}


namespace sb {
struct ShareParams {
  const float* fin;
  long long count;
  float* dst[8];
  uint32_t* flags[8];
  int world;
  uint32_t epoch;
};
// one CTA: copy the (tiny) statistics block into every rank's landing slot, then raise the flags
__global__ void __launch_bounds__(GN_THREADS) gn_share_kernel(const ShareParams p) {
  for (int r = 0; r < p.world; ++r)
    for (long long i = threadIdx.x; i < p.count; i += GN_THREADS) p.dst[r][i] = p.fin[i];
  __threadfence_system();
  __syncthreads();
  if (threadIdx.x < p.world)
    asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.flags[threadIdx.x]), "r"(p.epoch) : "memory");
}
}  // namespace sb

extern "C" int sb_gn_share(const float* fin, long long count, void* const* dst, void* const* flags, int world,
                           unsigned epoch, cudaStream_t stream) {
  if (world < 1 || world > 8) return SB_ERR_SHAPE;
  ShareParams p;
  memset(&p, 0, sizeof(p));
  p.fin = fin; p.count = count; p.world = world; p.epoch = epoch;
  for (int r = 0; r < world; ++r) { p.dst[r] = (float*)dst[r]; p.flags[r] = (uint32_t*)flags[r]; }
  gn_share_kernel<<<1, GN_THREADS, 0, stream>>>(p);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

// fin: [N][G][3] (stats) / [N][C][2] (bwd) -- the single-split form the apply / dx kernels merge
extern "C" int sb_gn_stats_finalize(const float* part, float* fin, int N, int G, int nsplit, cudaStream_t stream) {
  const int warps = N * G;
  // a warp per output up to 32 partials, a block of four up to 1024 (8 per thread, all in flight), a cluster beyond
  if (nsplit > 1024) {
    gn_stats_finalize_wide_kernel<<<warps * GN_WIDE_CLUSTER, GN_THREADS, 0, stream>>>(part, fin, N, G, nsplit);
    sb_count_launch(1);
    return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
  }
  if (nsplit > 32)
    gn_stats_finalize_block_kernel<<<warps, GN_FIN_THREADS, 0, stream>>>(part, fin, G, nsplit);
  else
    gn_stats_finalize_kernel<<<(warps * 32 + GN_THREADS - 1) / GN_THREADS, GN_THREADS, 0, stream>>>(part, fin, N, G, nsplit);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

extern "C" int sb_gn_bwd_finalize(const float* part, float* fin, int N, int C, int nsplit, cudaStream_t stream) {
  const int warps = N * C;
  gn_bwd_finalize_kernel<<<(warps * 32 + GN_THREADS - 1) / GN_THREADS, GN_THREADS, 0, stream>>>(part, fin, N, C, nsplit);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

// ----------------------------------------------------------------------------
// Allocation-free forward (declared in no_alloc.h)
// ----------------------------------------------------------------------------
#include "no_alloc.h"

namespace sb {
// Scratch of the allocation-free entry point: partial statistics, then the per-sample
// finals, then (when the caller passes none) mean / rstd. In host code this NAME is only a
// handle for cudaGetSymbolAddress; kernels get the resolved device address.
static __device__ __align__(256) float g_gn_noalloc_scratch[SB_GN_NOALLOC_SCRATCH_FLOATS + 2 * 256 * 64];
constexpr int NOALLOC_MAX_DEVICES = 64;
static float* g_gn_noalloc_ptr[NOALLOC_MAX_DEVICES] = {nullptr};
}  // namespace sb

extern "C" int sb_gn_forward_noalloc(const void* x, void* y, const float* w, const float* b, float* mean,
                                     float* rstd, int N, long long S, int C, int G, float eps, int relu,
                                     cudaStream_t stream) {
  if (N < 1 || N > 64 || S < 1 || !gn_channels_ok(C, G)) return SB_ERR_SHAPE;
  if (x == nullptr || y == nullptr || w == nullptr || b == nullptr) return SB_ERR_SHAPE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return SB_ERR_DRIVER;
  if (g_gn_noalloc_ptr[dev] == nullptr) {
    // once per device, with that device current: the symbol's address on THIS device
    float* p = nullptr;
    if (cudaGetSymbolAddress((void**)&p, g_gn_noalloc_scratch) != cudaSuccess || p == nullptr) return SB_ERR_DRIVER;
    g_gn_noalloc_ptr[dev] = p;
  }
  float* scratch = g_gn_noalloc_ptr[dev];
  const int nsplit = sb_gn_nsplit(N, S, C);
  const long long part_floats = (long long)N * nsplit * G * 3;
  const long long fin_floats = (long long)N * G * 3;
  if (part_floats + fin_floats > SB_GN_NOALLOC_SCRATCH_FLOATS) return SB_ERR_TOO_LARGE;
  float* part = scratch;
  float* fin = scratch + part_floats;
  float* tail = scratch + SB_GN_NOALLOC_SCRATCH_FLOATS;  // room for mean / rstd when the caller wants neither
  SbGnArgs a;
  memset(&a, 0, sizeof(a));
  a.x = x; a.y = y; a.w = w; a.b = b;
  a.mean = mean ? mean : tail;
  a.rstd = rstd ? rstd : tail + 256 * 64;
  a.N = N; a.C = C; a.G = G; a.S = S; a.S_total = S;
  a.eps = eps; a.relu = relu;
  a.part = part;
  a.parts[0] = part;
  a.n_parts = 1;
  a.nsplit = nsplit;
  a.fin = fin;  // the statistics launch collapses its own partials (last block)
  int rc = sb_gn_stats(&a, stream);
  if (rc) return rc;
  a.fin = nullptr;
  a.parts[0] = fin;
  a.nsplit = 1;
  return sb_gn_apply(&a, stream);
}
