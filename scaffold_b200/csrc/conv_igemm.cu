// Implicit-GEMM 3-D convolution on Blackwell tensor cores (sm_100a).
//
//   Y[voxel, co] = sum_{tap, ci} X[voxel + off(tap), ci] * Wp[tap][co][ci]
//
// Activations are NDHWC bf16. One CTA tile is 128 output voxels (a small brick
// h x w x d x n; h fastest with the w-shift reuse below, else w fastest) by BN
// output channels. Per K step the producer warp issues ONE 5-D TMA box load of
// the (shifted) input brick and one 3-D box load of the packed weights; TMA
// out-of-bounds zero fill is the convolution's zero padding, so no im2col buffer
// and no padded copy of the activation exists.
// A single elected thread issues tcgen05.mma into a TMEM accumulator
// (double-buffered, so the epilogue of tile i overlaps the main loop of tile
// i+1); four epilogue warps read TMEM with tcgen05.ld and store bf16.
//
// Stores: a lane holds one voxel's channels, so stores from registers touch 32 lines per instruction, and the 1x1x1
// head, its backward-data and the transposed convolution, which do next to no arithmetic, were bound by them. Each
// epilogue warp therefore lays its 32 rows x up to 64 channels out in shared memory (two buffers, swizzled: no bank
// conflicts) and one lane hands the tile to the TMA store, which also clips it at the volume's edges. A 1x1x1 call
// walks the voxels as one row, so a tile's output is contiguous; a transposed convolution writes through four strided
// views of the fine grid, one per (kd, kh), where the two kw taps of a voxel are one run of 2*Cout channels.
// Calls that no TMA box covers (two destinations with a bias or split off the 16-channel grid, unaligned views) keep
// the stores from registers. At 2 x 128^3, before / after: transposed 128 -> 64 354 / 162 us (671 MB), head 64 -> 16
// 121 / 117 us, its backward-data 320 / 257 us (its 32-byte rows now bound by the TMA loads).
//
// Small volumes: a tile's reduction over 27 taps is one SM's serial work (L2 to one SM is about 60 bytes a clock: 81 us
// for 512 -> 512 channels at 6 x 5 x 7), so when the tiles leave SMs idle the taps x channel blocks are split over
// them; the slices leave fp32 partial sums that a second kernel adds in slice order (all such layers of a step at
// 2 x 44x60x76: 472 / 225 us).
//
// W-shift reuse: with rows ordered h-fastest and 8 rows per swizzle atom, a
// shift of the input by one voxel along w is a shift of the shared-memory start
// address by exactly one atom. One halo'd box (8 h x (TW+2) w) therefore serves
// the three kw taps of a 3x3x3 filter: 9 activation loads per channel block
// instead of 27.
//
// The same kernel serves forward, backward-data (weights packed transposed and
// tap-flipped by the caller), the k2s2 transposed convolution (forward: one
// tap, N = 8*Cout columns scattered to the 2x upsampled grid; backward-data:
// four strided views of the gradient, one per (kd,kh)), reading up to two
// channel-concatenated sources (the U-Net skip concat is never materialised)
// and writing up to two channel-split destinations.
//
// Role of the reference: triton_conv3d/gather_gemm.py:112-341 (forward),
// triton_conv3d/bwd_data.py:275-363, triton_conv3d/transposed.py:135-319.
#include "common.cuh"
#include "host_api.h"

namespace sb {

constexpr int MAX_STAGES = 8;
constexpr int MAX_OUTER = 32;

struct IgemmParams {
  CUtensorMap mapA[8];
  CUtensorMap mapB;
  int TH, TW, TD, TN;
  int KWS, KHS, n_outer, BK, BN;
  int stages, stage_bytes, a_bytes, b_bytes, tx_bytes;  // a_bytes: offset of B inside a stage
  int N, D, H, W;  // output voxel grid (== the grid the tile bricks walk)
  int tiles_h, tiles_w, tiles_d, tiles_n, tiles_co, num_tiles;
  int cblks, cblks0;  // channel blocks in total / in the first source
  int maps_per_tap;   // stride of the tap's map index (2 when two sources)
  signed char tap_map[MAX_OUTER];
  signed char tap_dh[MAX_OUTER], tap_dw[MAX_OUTER], tap_dd[MAX_OUTER];
  // epilogue
  __nv_bfloat16* out0;
  __nv_bfloat16* out1;
  int width0, width1;  // stored channels per destination
  int ld0, ld1;        // channel stride (elements per voxel) per destination
  const float* bias;
  int scatter;  // 1: columns are (tap8, co) of a k2s2 transposed conv
  int sc_cout;
  uint32_t inv_cout, inv_2cout;  // ceil(2^32 / n): __umulhi(col, inv) = col / n for the columns here (col * n < 2^32)
  // row order of the brick and of every box: w fastest (plain loads) or h fastest (w-shift reuse)
  int wfirst;
  // TMA stores: one map per destination (scatter: per (kd,kh) view); ocols channels x a 32-row sub-brick per store
  CUtensorMap mapO[4];
  int ocols;          // 64 / 32 / 16; 0: stores from registers
  int stg_off;        // staging buffers (4 warps x 2) and then the bias in dynamic shared memory
  int bias_off, bias_n;
  // split reduction
  int splits, k_per_split;
  float* ws;
  uint32_t* status;
};

// Position of a work item, (slice, column tile, w, h, d, n) with the slice fastest. A CTA's next item is gridDim.x
// further: adding that step digit by digit keeps some 2000 clocks of divisions per tile off the producer lane and the
// epilogue, more than a 1x1x1 tile's loads and stores take.
struct Walk { int sl, co, w, h, d, n; };
__device__ __forceinline__ Walk walk_at(const IgemmParams& p, int item) {
  Walk t;
  t.sl = item % p.splits; item /= p.splits;
  t.co = item % p.tiles_co; item /= p.tiles_co;
  t.w = item % p.tiles_w; item /= p.tiles_w;
  t.h = item % p.tiles_h; item /= p.tiles_h;
  t.d = item % p.tiles_d;
  t.n = item / p.tiles_d;
  return t;
}
__device__ __forceinline__ void walk_step(const IgemmParams& p, Walk& t, const Walk& by) {
  t.sl += by.sl; t.co += by.co; t.w += by.w; t.h += by.h; t.d += by.d; t.n += by.n;
  if (t.sl >= p.splits) { t.sl -= p.splits; ++t.co; }
  if (t.co >= p.tiles_co) { t.co -= p.tiles_co; ++t.w; }
  if (t.w >= p.tiles_w) { t.w -= p.tiles_w; ++t.h; }
  if (t.h >= p.tiles_h) { t.h -= p.tiles_h; ++t.d; }
  if (t.d >= p.tiles_d) { t.d -= p.tiles_d; ++t.n; }
}

// 8 accumulator columns (+ bias) -> 16 bytes of bf16
__device__ __forceinline__ uint4 pack_octet(const uint32_t* v, const float* bias) {
  float f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[j]);
  if (bias) {
    const float4 a = reinterpret_cast<const float4*>(bias)[0], b = reinterpret_cast<const float4*>(bias)[1];
    f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
    f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
  }
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
  return o;
}

__global__ void __launch_bounds__(192, 2) igemm_kernel(const __grid_constant__ IgemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[MAX_STAGES];
  __shared__ uint64_t empty_bar[MAX_STAGES];
  __shared__ uint64_t tfull_bar[2];
  __shared__ uint64_t tempty_bar[2];
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_s;
  volatile uint32_t* abort_flag = &abort_s;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int rowb = p.BK * 2;

  if (threadIdx.x == 0) {
    abort_s = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], 4);
    }
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&tmem_base_s, 256);
    tmem_relinquish();
  }
  float* bias_s = reinterpret_cast<float*>(smem + p.bias_off);
  for (int i = threadIdx.x; i < p.bias_n; i += blockDim.x) bias_s[i] = p.bias[i];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_s;

  const int kiters = p.n_outer * p.cblks;
  const int work = p.num_tiles * p.splits;  // (tile, slice of the reduction), slices fastest

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      for (int i = 0; i < 8; ++i) tma_prefetch_desc(&p.mapA[i]);
      tma_prefetch_desc(&p.mapB);
      bool ok = true;
      uint32_t s = 0, ph = 0;
      const Walk by = walk_at(p, gridDim.x);
      Walk t = walk_at(p, blockIdx.x);
      for (int item = blockIdx.x; item < work && ok; item += gridDim.x, walk_step(p, t, by)) {
        const int h0 = t.h * p.TH, w0 = t.w * p.TW, d0 = t.d * p.TD, n0 = t.n * p.TN;
        const int co0 = t.co * p.BN;
        const int k0 = t.sl * p.k_per_split;
        const int k1 = k0 + p.k_per_split < kiters ? k0 + p.k_per_split : kiters;
        int o = 0, cb = 0;
        if (k0 > 0) { o = k0 / p.cblks; cb = k0 - o * p.cblks; }
        for (int k = k0; k < k1; ++k) {
          if (!mbar_wait(&empty_bar[s], ph ^ 1u, abort_flag, p.status, 1)) { ok = false; break; }
          uint8_t* sa = smem + (size_t)s * p.stage_bytes;
          uint8_t* sbm = sa + p.a_bytes;
          mbar_expect_tx(&full_bar[s], (uint32_t)p.tx_bytes);
          const int second = cb >= p.cblks0 ? 1 : 0;
          const int mi = p.tap_map[o] + second;
          const int c = (second ? cb - p.cblks0 : cb) * p.BK;
          const int hc = h0 + p.tap_dh[o], wc = w0 + p.tap_dw[o];
          tma_load_5d(sa, &p.mapA[mi], &full_bar[s], c, p.wfirst ? wc : hc, p.wfirst ? hc : wc, d0 + p.tap_dd[o], n0);
          tma_load_3d(sbm, &p.mapB, &full_bar[s], cb * p.BK, co0, o * p.KWS * p.KHS);
          if (++cb == p.cblks) { cb = 0; ++o; }
          if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    // Warp-uniform control flow (wait results are voted on) keeps the descriptor arithmetic in
    // uniform registers; one elected lane issues. Descriptors are (lo, hi) words: a new operand
    // address is one add.
    {
      const bool leader = elect_one();
      const uint32_t idesc = make_idesc_bf16(128, p.BN, 0, 0);
      const uint32_t swz = swizzle_code_for(rowb);
      const int rh = p.TH + p.KHS - 1;             // rows per w column of the A box
      // 8-row groups are contiguous unless the box carries an h halo (then one w step apart)
      const uint32_t a_hi = desc_hi((uint32_t)(p.KHS > 1 ? rh : 8) * rowb, swz);
      const uint32_t b_hi = desc_hi(8u * rowb, swz);
      const uint32_t b_shift = ((uint32_t)p.BN * rowb) >> 4;
      const uint32_t a_wstep = ((uint32_t)(p.KHS > 1 ? rh : p.TH) * rowb) >> 4;
      const uint32_t a_hstep = (uint32_t)rowb >> 4;
      const int ksteps = p.BK / 16;
      const uint32_t s0 = smem_u32(smem);
      uint32_t stage = 0, sph = 0, tcount = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < work && ok; item += gridDim.x, ++tcount) {
        const int k0 = p.splits > 1 ? (item % p.splits) * p.k_per_split : 0;
        const int k1 = k0 + p.k_per_split < kiters ? k0 + p.k_per_split : kiters;
        const uint32_t buf = tcount & 1u;
        const uint32_t bph = (tcount >> 1) & 1u;
        if (!__all_sync(0xffffffffu, mbar_wait(&tempty_bar[buf], bph ^ 1u, abort_flag, p.status, 2))) { ok = false; break; }
        tc_fence_after();
        const uint32_t acc = tmem_base + buf * 128u;
        for (int ki = 0; ki < k1 - k0; ++ki) {
          if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], sph, abort_flag, p.status, 3))) { ok = false; break; }
          tc_fence_after();
          const uint32_t sa = s0 + stage * (uint32_t)p.stage_bytes;
          const uint32_t a_lo0 = desc_lo(sa, 16u);
          const uint32_t b_lo0 = desc_lo(sa + p.a_bytes, 16u);
          for (int kh = 0; kh < p.KHS; ++kh) {
            for (int kw = 0; kw < p.KWS; ++kw) {
              const uint32_t a_lo = a_lo0 + kw * a_wstep + kh * a_hstep;
              const uint32_t b_lo = b_lo0 + (uint32_t)(kh * p.KWS + kw) * b_shift;
              if (leader) {
                for (int k = 0; k < ksteps; ++k)
                  tc_mma_bf16_pred(acc, a_lo + 2u * k, a_hi, b_lo + 2u * k, b_hi, idesc,
                                   (ki | kh | kw | k) != 0 ? 1u : 0u);
              }
            }
          }
          if (leader) tc_commit(&empty_bar[stage]);
          __syncwarp();
          if (++stage == (uint32_t)p.stages) { stage = 0; sph ^= 1u; }
        }
        if (ok && leader) tc_commit(&tfull_bar[buf]);
      }
    }
  } else {
    // -------------------------------- epilogue --------------------------------
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int rh = p.wfirst ? (row / p.TW) % p.TH : row % p.TH;
    const int rw = p.wfirst ? row % p.TW : (row / p.TH) % p.TW;
    const int rd = (row / (p.TH * p.TW)) % p.TD;
    const int rn = row / (p.TH * p.TW * p.TD);
    uint32_t tcount = 0;
    bool ok = true;
    // TMA stores: this warp's two staging buffers; its rows start at the brick position of lane 0
    const int stg_bytes = 64 * p.ocols;
    uint8_t* stg = smem + p.stg_off + q * 2 * stg_bytes;
    const uint32_t row_off = (uint32_t)(lane * p.ocols * 2);
    const uint32_t swz = p.ocols == 64 ? (uint32_t)(lane & 7) << 4
                         : p.ocols == 32 ? (uint32_t)((lane >> 1) & 3) << 4 : (uint32_t)((lane >> 2) & 1) << 4;
    uint32_t nstore = 0;
    const Walk by = walk_at(p, gridDim.x);
    Walk t = walk_at(p, blockIdx.x);
    for (int item = blockIdx.x; item < work && ok; item += gridDim.x, ++tcount, walk_step(p, t, by)) {
      const uint32_t buf = tcount & 1u;
      const uint32_t bph = (tcount >> 1) & 1u;
      if (!mbar_wait(&tfull_bar[buf], bph, abort_flag, p.status, 4)) { ok = false; break; }
      tc_fence_after();
      const int h = t.h * p.TH + rh, w = t.w * p.TW + rw, d = t.d * p.TD + rd, n = t.n * p.TN + rn;
      const bool valid = (rn < p.TN) && h < p.H && w < p.W && d < p.D && n < p.N;
      const long long vox = (((long long)n * p.D + d) * p.H + h) * p.W + w;
      const int co0 = t.co * p.BN;
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + buf * 128u;
      if (p.splits > 1) {
        // fp32 partial sums [slice][voxel][column]; a second kernel adds the slices in order
        const long long rows_all = (long long)p.N * p.D * p.H * p.W;
        const int ld = p.tiles_co * p.BN;
        float* dst = p.ws + ((long long)t.sl * rows_all + vox) * ld + co0;
        for (int c = 0; c < p.BN; c += 16) {
          uint32_t v[16];
          tmem_ld_32x16(tbase + c, v);
          tmem_ld_wait();
          if (valid) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              reinterpret_cast<uint4*>(dst + c)[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[buf]);
        continue;
      }
      if (p.ocols > 0) {
        for (int c = 0; c < p.BN; c += p.ocols, ++nstore) {
          uint8_t* sbuf = stg + (nstore & 1u) * stg_bytes;
          // the store before the last one has read this buffer
          if (lane == 0) bulk_wait_read_but_one();
          __syncwarp();
          const int col = co0 + c;
          // bias: of the column, or of the column's channel within its tap
          int bcol = p.scatter ? col - (int)__umulhi((uint32_t)col, p.inv_cout) * p.sc_cout : col;
          if (p.ocols >= 32) {
            for (int hh = 0; hh < p.ocols; hh += 32) {
              uint32_t v[32];
              tmem_ld_32x32(tbase + c + hh, v);
              tmem_ld_wait();
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const uint4 o = pack_octet(v + 8 * g, p.bias_n ? bias_s + bcol : nullptr);
                bcol += 8;
                if (p.scatter && bcol >= p.sc_cout) bcol = 0;
                *reinterpret_cast<uint4*>(sbuf + row_off + ((uint32_t)(hh * 2 + g * 16) ^ swz)) = o;
              }
            }
          } else {
            uint32_t v[16];
            tmem_ld_32x16(tbase + c, v);
            tmem_ld_wait();
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              const uint4 o = pack_octet(v + 8 * g, p.bias_n ? bias_s + bcol : nullptr);
              bcol += 8;
              if (p.scatter && bcol >= p.sc_cout) bcol = 0;
              *reinterpret_cast<uint4*>(sbuf + row_off + ((uint32_t)(g * 16) ^ swz)) = o;
            }
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0 && valid) {  // lane 0's voxel is the sub-brick's first: nothing of a box that starts outside
            int mi = 0, oc = col;
            if (p.scatter) { mi = (int)__umulhi((uint32_t)col, p.inv_2cout); oc = col - mi * 2 * p.sc_cout; }
            else if (col >= p.width0) { mi = 1; oc = col - p.width0; }
            if (p.scatter || oc < (mi ? p.width1 : p.width0))
              tma_store_5d(&p.mapO[mi], sbuf, oc, p.wfirst ? w : h, p.wfirst ? h : w, d, n);
          }
          if (lane == 0) bulk_commit();
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[buf]);
        continue;
      }
      const int nchunk = (p.BN + 31) / 32;
      for (int ch = 0; ch < nchunk; ++ch) {
        uint32_t v[32];
        if (p.BN >= 32) {
          tmem_ld_32x32(tbase + ch * 32, v);
        } else {
          uint32_t v16[16];
          tmem_ld_32x16(tbase, v16);
#pragma unroll
          for (int j = 0; j < 16; ++j) { v[j] = v16[j]; v[16 + j] = 0u; }
        }
        tmem_ld_wait();
        if (valid) {
          const int ngroups = p.BN >= 32 ? 4 : 2;
#pragma unroll
          for (int g2 = 0; g2 < 2; ++g2) {
            if (g2 * 2 >= ngroups) break;
            // two groups of 8 channels; they share a destination row when the split points are multiples of 16
            uint4 o[2];
            __nv_bfloat16* dst[2] = {nullptr, nullptr};
#pragma unroll
            for (int gi = 0; gi < 2; ++gi) {
              const int g = g2 * 2 + gi;
              const int col = co0 + ch * 32 + g * 8;
              float f[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[g * 8 + j]);
              if (p.scatter) {
                const int tap = col / p.sc_cout;
                const int co = col - tap * p.sc_cout;
                if (tap < 8) {
                  const int kd = tap >> 2, kh = (tap >> 1) & 1, kw = tap & 1;
                  const long long ov =
                      (((long long)n * (2 * p.D) + (2 * d + kd)) * (2 * p.H) + (2 * h + kh)) * (2 * p.W) +
                      (2 * w + kw);
                  dst[gi] = p.out0 + ov * p.ld0 + co;
                  if (p.bias) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) f[j] += p.bias[co + j];
                  }
                }
              } else if (col < p.width0) {
                dst[gi] = p.out0 + vox * p.ld0 + col;
                if (p.bias) {
#pragma unroll
                  for (int j = 0; j < 8; ++j) f[j] += p.bias[col + j];
                }
              } else if (col - p.width0 < p.width1) {
                dst[gi] = p.out1 + vox * p.ld1 + (col - p.width0);
              }
              o[gi].x = pack_bf16x2(f[0], f[1]);
              o[gi].y = pack_bf16x2(f[2], f[3]);
              o[gi].z = pack_bf16x2(f[4], f[5]);
              o[gi].w = pack_bf16x2(f[6], f[7]);
            }
            if (dst[0] && dst[1] == dst[0] + 8 && (reinterpret_cast<uintptr_t>(dst[0]) & 31) == 0) {
              st_global_v8(dst[0], o[0], o[1]);
            } else {
              if (dst[0]) *reinterpret_cast<uint4*>(dst[0]) = o[0];
              if (dst[1]) *reinterpret_cast<uint4*>(dst[1]) = o[1];
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty_bar[buf]);
    }
    if (lane == 0) bulk_wait_all();  // none pending without TMA stores
  }

  // ------------------------------- teardown ---------------------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // copies may still be in flight towards this CTA's shared memory: give
    // them a bounded grace period before the CTA (and its TMEM) goes away
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// ---------------------------------------------------------------------------
// Host side: tensor maps and launch plans
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

static CUtensorMapSwizzle swz_enum(int rowb) {
  return rowb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                     : rowb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
}

// bf16 tensor map; dims/strides fastest first, strides in ELEMENTS (stride[0] is implicit 1)
int make_map_bf16(CUtensorMap* m, const void* base, int rank, const long long* dims, const long long* strides,
                  const int* box, int rowb) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return SB_ERR_DRIVER;
  cuuint64_t gdim[5];
  cuuint64_t gstr[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = (cuuint64_t)dims[i];
    bx[i] = (cuuint32_t)box[i];
    es[i] = 1;
    if (i > 0) gstr[i - 1] = (cuuint64_t)strides[i] * 2ull;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return SB_ERR_ALIGN;
  for (int i = 0; i + 1 < rank; ++i)
    if (gstr[i] % 16 != 0) return SB_ERR_ALIGN;
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr,
                   bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz_enum(rowb), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : SB_ERR_TENSORMAP;
}

static int pow2_floor(int v) {
  int p = 1;
  while (p * 2 <= v) p *= 2;
  return p;
}
static int cdiv(int a, int b) { return (a + b - 1) / b; }

static int g_smem_limit = 0;
static int g_sm_count = 0;
static int device_setup() {
  if (g_smem_limit) return 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return SB_ERR_DRIVER;
  int lim = 0, sms = 0;
  cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaFuncSetAttribute(igemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lim - 2048) != cudaSuccess)
    return SB_ERR_DRIVER;
  g_smem_limit = lim - 2048;
  g_sm_count = sms;
  return 0;
}

// Choose the voxel brick and finish the geometry common to all plans.
static void choose_brick(IgemmParams& p, bool shift) {
  p.KHS = 1;
  if (shift) {
    p.TH = 8; p.TW = 16; p.TD = 1; p.TN = 1; p.KWS = 3;
    p.wfirst = 0;
  } else {
    // w fastest; of all bricks of 128 voxels with power-of-two edges the one that covers the volume with the fewest
    // tiles, and of those the one with the longest runs along w
    p.KWS = 1;
    p.wfirst = 1;
    long long best = -1;
    for (int tw = 128; tw >= 1; tw /= 2)
      for (int th = 128 / tw; th >= 1; th /= 2)
        for (int td = 128 / (tw * th); td >= 1; td /= 2) {
          const int tn = 128 / (tw * th * td);
          const long long tiles = (long long)cdiv(p.W, tw) * cdiv(p.H, th) * cdiv(p.D, td) * cdiv(p.N, tn);
          if (best < 0 || tiles < best) {
            best = tiles;
            p.TW = tw; p.TH = th; p.TD = td; p.TN = tn;
          }
        }
  }
  p.tiles_h = cdiv(p.H, p.TH);
  p.tiles_w = cdiv(p.W, p.TW);
  p.tiles_d = cdiv(p.D, p.TD);
  p.tiles_n = cdiv(p.N, p.TN);
}

// Tensor map of an output (or of one strided view of it) for stores of p.ocols channels x the 32-row sub-brick of a
// warp. dims / strides in the order C, W, H, D, N.
static int out_map(const IgemmParams& p, CUtensorMap* m, const void* base, const long long* dims,
                   const long long* strides) {
  int left = 32;
  const int t[4] = {p.wfirst ? p.TW : p.TH, p.wfirst ? p.TH : p.TW, p.TD, p.TN};
  int box[5] = {p.ocols, 1, 1, 1, 1};
  for (int i = 0; i < 4; ++i) {
    box[1 + i] = t[i] < left ? t[i] : left;
    left /= box[1 + i];
  }
  long long dm[5], st[5];
  for (int i = 0; i < 5; ++i) {
    const int j = p.wfirst ? i : i == 1 ? 2 : i == 2 ? 1 : i;
    dm[i] = dims[j];
    st[i] = strides[j];
  }
  return make_map_bf16(m, base, 5, dm, st, box, p.ocols * 2);
}

// (C, H, W, ...) -> (C, W, H, ...)
static void w_first(long long* dims, long long* strides, int* box) {
  const long long d = dims[1], s = strides[1];
  const int b = box[1];
  dims[1] = dims[2]; strides[1] = strides[2]; box[1] = box[2];
  dims[2] = d; strides[2] = s; box[2] = b;
}

// Channels per TMA store: the widest of 64 / 32 / 16 that never crosses a tile or a destination's end (`run` channels).
static int store_columns(int bn, int run) {
  for (int c = 64; c >= 16; c /= 2)
    if (bn % c == 0 && run % c == 0) return c;
  return 0;
}

static int finish_and_launch(IgemmParams& p, int cout_rows, cudaStream_t stream) {
  const int rowb = p.BK * 2;
  const int rows_a = (p.TH + p.KHS - 1) * (p.TW + p.KWS - 1) * p.TD * p.TN;
  // the MMA always reads 128 rows starting at an offset of up to (KWS-1)*TH rows
  const int rows_alloc = rows_a > 128 + (p.KWS - 1) * p.TH ? rows_a : 128 + (p.KWS - 1) * p.TH;
  p.a_bytes = ((rows_alloc * rowb + 1023) / 1024) * 1024;
  p.b_bytes = p.KWS * p.KHS * p.BN * rowb;
  p.stage_bytes = ((p.a_bytes + p.b_bytes + 1023) / 1024) * 1024;
  p.tiles_co = cdiv(cout_rows, p.BN);
  p.num_tiles = p.tiles_co * p.tiles_w * p.tiles_h * p.tiles_d * p.tiles_n;
  const int kiters = p.n_outer * p.cblks;
  if (p.splits < 1) p.splits = 1;
  p.k_per_split = cdiv(kiters, p.splits);
  if (p.splits > 1) p.ocols = 0;
  // Two CTAs per SM when there are tiles for them and three stages fit in half the shared memory (two where the
  // staging buffers take their share and the whole reduction is at most two steps): the second CTA's MMAs and epilogue
  // fill the first one's waits (each CTA allocates 256 of the 512 TMEM columns).
  const int half = g_smem_limit / 2 - 2048;
  int extra = 0, st = 0;
  bool dual = false;
  for (;; p.ocols = 0) {
    // behind the stages: staging buffers (8 of 32 rows), and the bias as far as columns read it
    p.bias_n = p.ocols > 0 && p.bias ? (p.scatter ? p.sc_cout : p.width0) : 0;
    extra = 8 * 64 * p.ocols + (p.bias_n ? (((p.scatter ? p.sc_cout : cout_rows) * 4 + 127) / 128) * 128 : 0);
    const int need = p.ocols > 0 && kiters <= 2 ? 2 : 3;
    dual = p.num_tiles * p.splits > g_sm_count && (half - 1024 - extra) / p.stage_bytes >= need;
    st = ((dual ? half : g_smem_limit) - 1024 - extra) / p.stage_bytes;
    if (st >= 2) break;
    if (p.ocols == 0) return SB_ERR_SHAPE;  // with a bias too wide to stage: stores from registers
  }
  if (st > MAX_STAGES) st = MAX_STAGES;
  p.stages = st;
  p.stg_off = st * p.stage_bytes;
  p.bias_off = p.stg_off + 8 * 64 * p.ocols;
  // expected transaction bytes are what the two boxes really deliver
  p.tx_bytes = rows_a * rowb + p.b_bytes;
  const IgemmParams& q = p;
  const int slots = dual ? 2 * g_sm_count : g_sm_count;
  const int work = q.num_tiles * q.splits;
  int grid = work < slots ? work : slots;
  const size_t smem = (size_t)q.stages * q.stage_bytes + extra + 1024;
  igemm_kernel<<<grid, 192, smem, stream>>>(q);
  sb_count_launch(1);
  return cudaGetLastError() == cudaSuccess ? 0 : SB_ERR_LAUNCH;
}

}  // namespace sb

using namespace sb;

// Stride-1 "same" convolution, k in {1,3}; also backward-data when the caller
// packs the weights transposed and tap-flipped.
namespace sb {
int conv_plane_launch(const SbConvArgs* a, cudaStream_t stream);
int conv_plane2_launch(const SbConvArgs* a, cudaStream_t stream);
int conv_plane2_gn_splits(const SbConvArgs* a);
int conv_plane3_launch(const SbConvArgs* a, cudaStream_t stream);
int conv_plane3_gn_splits(const SbConvArgs* a);
int conv_small_launch(const SbConvArgs* a, cudaStream_t stream);
long long conv_small_workspace(const SbConvArgs* a);
int conv_point_launch(const SbConvArgs* a, cudaStream_t stream);
int conv_reduce_slices(const SbConvArgs* a, const float* ws, int splits, cudaStream_t stream);
}

// fp32 scratch elements sb_conv_fwd wants for this call (0: none)
static bool automatic(const SbConvArgs* a) { return a->force_plain == 0 || a->force_plain == 4; }

static int block_channels(const SbConvArgs* a) {
  const int tot = a->src_c[0] + a->src_c[1];
  int bk = 64;
  while (bk > 16 && (a->src_c[0] % bk != 0 || tot % bk != 0)) bk /= 2;
  return a->src_c[0] % bk != 0 || tot % bk != 0 ? 0 : bk;
}

// Slices of the reduction for a 3x3x3 call on a volume that is too small for the plane kernels (the only calls that
// reach the generic kernel by themselves). Worth it when at least half of the SMs would idle and a slice keeps eight
// steps.
static int generic_splits(const SbConvArgs* a) {
  if (!automatic(a) || a->ksize != 3 || (a->W >= 16 && a->H >= 8) || a->wpack == nullptr || a->cout_pad % 16) return 1;
  const int bk = block_channels(a);
  const int bn = a->cout_pad >= 128 ? 128 : a->cout_pad;
  if (bk == 0 || a->cout_pad % bn != 0 || device_setup()) return 1;
  IgemmParams p;
  p.N = a->N; p.D = a->D; p.H = a->H; p.W = a->W;
  choose_brick(p, false);
  const long long tiles = (long long)p.tiles_h * p.tiles_w * p.tiles_d * p.tiles_n * (a->cout_pad / bn);
  const int kiters = 27 * ((a->src_c[0] + a->src_c[1]) / bk);
  if (tiles * 2 > g_sm_count || kiters < 32) return 1;
  int splits = (int)(g_sm_count / tiles);
  if (splits > kiters / 8) splits = kiters / 8;
  if (splits > 32) splits = 32;
  return cdiv(kiters, cdiv(kiters, splits));  // no empty slice
}

static long long generic_workspace(const SbConvArgs* a, int splits) {
  return splits < 2 ? 0 : (long long)splits * a->N * a->D * a->H * a->W * a->cout_pad;
}

extern "C" long long sb_conv_fwd_workspace(const SbConvArgs* a) {
  if (!automatic(a)) return 0;
  const long long small = conv_small_workspace(a);
  return small > 0 ? small : generic_workspace(a, generic_splits(a));
}

static bool pair_first(const SbConvArgs* a) { return a->force_plain == 0 && a->wpack_kd == nullptr; }

extern "C" int sb_conv_gn_splits(const SbConvArgs* a) {
  if (!automatic(a)) return 0;
  if (pair_first(a)) {
    const int s2 = conv_plane2_gn_splits(a);
    if (s2 > 0) return s2;
  }
  return conv_plane3_gn_splits(a);
}

// force_plain: 0 = automatic (k = 1 from 16 or 32 channels; 8 x 8 plane kernel; the two-SM pair kernel for wide outputs
// given tap-ordered weights only; kd-fused or plane-walk kernel when the shape is eligible; else this file's generic
// kernel),
// 1 = generic kernel one tap per load, 2 = generic kernel with the w-shift reuse, 3 = generic kernel with the
// (h, w)-shift reuse, 4 = automatic without the pair kernel.
extern "C" int sb_conv_fwd(const SbConvArgs* a, cudaStream_t stream) {
  if (automatic(a)) {
    const int pt = conv_point_launch(a, stream);
    if (pt >= 0) return pt;
    const int sm = conv_small_launch(a, stream);
    if (sm >= 0) return sm;
    // with a partial-statistics buffer only when the pair kernel is the one that sized it (sb_conv_gn_splits)
    if (pair_first(a) && (a->gn_part == nullptr || conv_plane2_gn_splits(a) > 0)) {
      const int p2 = conv_plane2_launch(a, stream);
      if (p2 >= 0) return p2;
    }
    const int p3 = conv_plane3_launch(a, stream);
    if (p3 >= 0) return p3;
    if (a->gn_part != nullptr) return SB_ERR_SHAPE;  // statistics come from the kd-fused kernel only
    if (a->wpack == nullptr) return SB_ERR_SHAPE;  // only the kd-ordered weights were given
    const int prc = conv_plane_launch(a, stream);
    if (prc >= 0) return prc;
  }
  if (a->wpack == nullptr) return SB_ERR_SHAPE;
  if (a->halo_land[0][0] || a->halo_land[0][1] || a->slab_out[0]) return SB_ERR_SHAPE;  // plane-walk kernel only
  int rc = device_setup();
  if (rc) return rc;
  IgemmParams p;
  memset(&p, 0, sizeof(p));
  const int cin_tot = a->src_c[0] + a->src_c[1];
  const int nsrc = a->src_c[1] > 0 ? 2 : 1;
  const int bk = block_channels(a);
  if (bk == 0) return SB_ERR_SHAPE;
  p.BK = bk;
  p.BN = a->cout_pad >= 128 ? 128 : a->cout_pad;
  if (p.BN % 16 != 0 || a->cout_pad % p.BN != 0) return SB_ERR_SHAPE;
  if (a->ksize != 1 && a->ksize != 3) return SB_ERR_SHAPE;
  p.N = a->N; p.D = a->D; p.H = a->H; p.W = a->W;
  const bool can_shift = a->ksize == 3 && a->W >= 16 && a->H >= 8;
  const bool shift = can_shift && a->force_plain != 1;
  long long iD = a->in_d ? a->in_d : a->D, iH = a->in_h ? a->in_h : a->H, iW = a->in_w ? a->in_w : a->W;
  const long long voxels = (long long)a->N * a->D * a->H * a->W;
  if (a->ksize == 1 && !a->off_d && !a->off_h && !a->off_w && iD == a->D && iH == a->H && iW == a->W &&
      voxels < 0x7fffff00ll) {
    // no neighbours: the voxels are one row
    p.N = p.D = p.H = 1;
    p.W = (int)voxels;
    iD = iH = 1;
    iW = voxels;
  }
  choose_brick(p, shift);
  if (shift && a->force_plain == 3) p.KHS = 3;
  const int taps = a->ksize * a->ksize * a->ksize;
  p.n_outer = taps / (p.KWS * p.KHS);
  p.maps_per_tap = nsrc;
  const int half = a->ksize / 2;
  for (int o = 0; o < p.n_outer; ++o) {
    const int t0 = o * p.KWS * p.KHS;  // taps ordered (kd, kh, kw), kw fastest
    const int kd = t0 / (a->ksize * a->ksize), kh = (t0 / a->ksize) % a->ksize, kw = t0 % a->ksize;
    p.tap_map[o] = 0;
    p.tap_dd[o] = (signed char)(kd - half + a->off_d);
    p.tap_dh[o] = (signed char)(kh - half + a->off_h);
    p.tap_dw[o] = (signed char)(kw - half + a->off_w);  // shift mode: kw == 0 -> -1, the box is TW+2 wide
  }
  p.cblks0 = a->src_c[0] / bk;
  p.cblks = cin_tot / bk;
  const int rowb = bk * 2;
  for (int s = 0; s < nsrc; ++s) {
    const long long C = a->src_ld[s];
    long long dims[5] = {a->src_c[s], iH, iW, iD, p.N};
    long long str[5] = {1, iW * C, C, iH * iW * C, iD * iH * iW * C};
    int box[5] = {bk, p.TH + p.KHS - 1, p.TW + p.KWS - 1, p.TD, p.TN};
    if (p.wfirst) w_first(dims, str, box);
    rc = make_map_bf16(&p.mapA[s], a->src[s], 5, dims, str, box, rowb);
    if (rc) return rc;
  }
  for (int s = nsrc; s < 8; ++s) p.mapA[s] = p.mapA[0];
  {
    long long dims[3] = {cin_tot, a->cout_pad, taps};
    long long str[3] = {1, cin_tot, (long long)a->cout_pad * cin_tot};
    int box[3] = {bk, p.BN, p.KWS * p.KHS};
    rc = make_map_bf16(&p.mapB, a->wpack, 3, dims, str, box, rowb);
    if (rc) return rc;
  }
  p.out0 = (__nv_bfloat16*)a->dst[0];
  p.out1 = (__nv_bfloat16*)a->dst[1];
  p.width0 = a->dst_c[0];
  p.width1 = a->dst[1] ? a->dst_c[1] : 0;
  p.ld0 = a->dst_ld[0];
  p.ld1 = a->dst_ld[1];
  if (p.width0 % 8 || p.width1 % 8 || p.ld0 % 8 || p.ld1 % 8) return SB_ERR_SHAPE;
  p.bias = a->bias;
  p.scatter = 0;
  p.sc_cout = 1;
  p.status = a->status;
  const int splits = generic_splits(a);
  if (splits > 1 && a->workspace != nullptr && a->workspace_elems >= generic_workspace(a, splits)) {
    p.splits = splits;
    p.ws = a->workspace;
    rc = finish_and_launch(p, a->cout_pad, stream);
    return rc ? rc : conv_reduce_slices(a, p.ws, splits, stream);
  }
  // the bias belongs to the first destination; a destination narrower than its columns is clipped by its map
  p.ocols = p.out1 ? (p.bias ? 0 : store_columns(p.BN, p.width0)) : store_columns(p.BN, p.BN);
  if ((reinterpret_cast<uintptr_t>(p.out0) | reinterpret_cast<uintptr_t>(p.out1)) & 15) p.ocols = 0;
  for (int i = 0; p.ocols > 0 && i < (p.out1 ? 2 : 1); ++i) {
    const long long C = i ? p.ld1 : p.ld0;
    const long long dims[5] = {i ? p.width1 : p.width0, p.W, p.H, p.D, p.N};
    const long long str[5] = {1, C, p.W * C, (long long)p.H * p.W * C, (long long)p.D * p.H * p.W * C};
    rc = out_map(p, &p.mapO[i], i ? p.out1 : p.out0, dims, str);
    if (rc) return rc;
  }
  return finish_and_launch(p, a->cout_pad, stream);
}

// k=2, s=2 transposed convolution, forward: pointwise GEMM with N = 8*Cout
// columns (tap-major) scattered to the upsampled grid, bias fused.
extern "C" int sb_convT_fwd(const SbConvTArgs* a, cudaStream_t stream) {
  int rc = device_setup();
  if (rc) return rc;
  IgemmParams p;
  memset(&p, 0, sizeof(p));
  int bk = 64;
  while (bk > 16 && a->cin % bk != 0) bk /= 2;
  if (a->cin % bk != 0 || a->cout % 8 != 0) return SB_ERR_SHAPE;
  const int ncols = 8 * a->cout;
  p.BK = bk;
  p.BN = ncols >= 128 ? 128 : ncols;
  if (ncols % p.BN != 0) return SB_ERR_SHAPE;
  p.N = a->N; p.D = a->D; p.H = a->H; p.W = a->W;  // input grid
  choose_brick(p, false);
  p.n_outer = 1;
  p.maps_per_tap = 1;
  p.cblks0 = p.cblks = a->cin / bk;
  const int rowb = bk * 2;
  {
    const long long C = a->src_ld;
    long long dims[5] = {a->cin, a->H, a->W, a->D, a->N};
    long long str[5] = {1, (long long)a->W * C, C, (long long)a->H * a->W * C, (long long)a->D * a->H * a->W * C};
    int box[5] = {bk, p.TH, p.TW, p.TD, p.TN};
    w_first(dims, str, box);
    rc = make_map_bf16(&p.mapA[0], a->src, 5, dims, str, box, rowb);
    if (rc) return rc;
    for (int s = 1; s < 8; ++s) p.mapA[s] = p.mapA[0];
  }
  {
    long long dims[3] = {a->cin, ncols, 1};
    long long str[3] = {1, a->cin, (long long)ncols * a->cin};
    int box[3] = {bk, p.BN, 1};
    rc = make_map_bf16(&p.mapB, a->wpack, 3, dims, str, box, rowb);
    if (rc) return rc;
  }
  p.out0 = (__nv_bfloat16*)a->dst;
  p.width0 = a->cout;
  p.ld0 = a->dst_ld;
  p.bias = a->bias;
  p.scatter = 1;
  p.sc_cout = a->cout;
  p.inv_cout = (uint32_t)(0xffffffffu / (uint32_t)a->cout + 1u);
  p.inv_2cout = (uint32_t)(0xffffffffu / (2u * (uint32_t)a->cout) + 1u);
  p.status = a->status;
  // (inv_2cout divides exactly while column * 2 cout < 2^32)
  p.ocols = a->dst_ld == a->cout && (reinterpret_cast<uintptr_t>(a->dst) & 15) == 0 && a->cout < 16384
                ? store_columns(p.BN, 2 * a->cout) : 0;
  for (int o = 0; p.ocols > 0 && o < 4; ++o) {
    const long long C = a->cout, W2 = 2LL * a->W, H2 = 2LL * a->H, D2 = 2LL * a->D;
    const long long dims[5] = {2 * C, a->W, a->H, a->D, a->N};
    const long long str[5] = {1, 2 * C, 2 * W2 * C, 2 * H2 * W2 * C, D2 * H2 * W2 * C};
    rc = out_map(p, &p.mapO[o], p.out0 + ((o >> 1) * H2 + (o & 1)) * W2 * C, dims, str);
    if (rc) return rc;
  }
  return finish_and_launch(p, ncols, stream);
}

// k=2, s=2 transposed convolution, backward-data: gx[v, ci] = sum_{tap,co}
// gy[2v+tap, co] * W[ci, co, tap]. The gradient is read through four strided
// views (one per (kd,kh)); kw is folded into the channel axis (2*Cout wide).
extern "C" int sb_convT_dgrad(const SbConvTArgs* a, cudaStream_t stream) {
  int rc = device_setup();
  if (rc) return rc;
  IgemmParams p;
  memset(&p, 0, sizeof(p));
  // here: src = gy [N, 2D, 2H, 2W, cout], dst = gx [N, D, H, W, cin]; a->cout is the
  // channel count of gy, a->cin the channel count of gx; wpack = [4][cin_pad][2*cout]
  const int kc = 2 * a->cout;
  int bk = 64;
  while (bk > 16 && kc % bk != 0) bk /= 2;
  if (kc % bk != 0 || a->cin % 8 != 0) return SB_ERR_SHAPE;
  const int rows = a->wrows;
  p.BK = bk;
  p.BN = rows >= 128 ? 128 : rows;
  if (p.BN % 16 != 0 || rows % p.BN != 0) return SB_ERR_SHAPE;
  p.N = a->N; p.D = a->D; p.H = a->H; p.W = a->W;  // gx grid
  choose_brick(p, false);
  p.n_outer = 4;
  p.maps_per_tap = 1;
  p.cblks0 = p.cblks = kc / bk;
  const int rowb = bk * 2;
  const long long C = a->src_ld;  // channel stride of gy
  const long long W2 = 2LL * a->W, H2 = 2LL * a->H, D2 = 2LL * a->D;
  for (int o = 0; o < 4; ++o) {
    const int kd = o >> 1, kh = o & 1;
    const __nv_bfloat16* base = (const __nv_bfloat16*)a->src + ((long long)kd * H2 + kh) * W2 * C;
    // when ld == cout the pair (kw, co) is one contiguous run of 2*cout elements
    if (C != a->cout) return SB_ERR_SHAPE;
    long long dims[5] = {kc, a->H, a->W, a->D, a->N};
    long long str[5] = {1, 2 * W2 * C, 2 * C, 2 * H2 * W2 * C, D2 * H2 * W2 * C};
    int box[5] = {bk, p.TH, p.TW, p.TD, p.TN};
    w_first(dims, str, box);
    rc = make_map_bf16(&p.mapA[o], base, 5, dims, str, box, rowb);
    if (rc) return rc;
    p.tap_map[o] = (signed char)o;
  }
  for (int s = 4; s < 8; ++s) p.mapA[s] = p.mapA[0];
  {
    long long dims[3] = {kc, rows, 4};
    long long str[3] = {1, kc, (long long)rows * kc};
    int box[3] = {bk, p.BN, 1};
    rc = make_map_bf16(&p.mapB, a->wpack, 3, dims, str, box, rowb);
    if (rc) return rc;
  }
  p.out0 = (__nv_bfloat16*)a->dst;
  p.width0 = a->cin;
  p.ld0 = a->dst_ld;
  p.scatter = 0;
  p.sc_cout = 1;
  p.status = a->status;
  p.ocols = (reinterpret_cast<uintptr_t>(a->dst) & 15) == 0 && a->dst_ld % 8 == 0 ? store_columns(p.BN, p.BN) : 0;
  if (p.ocols > 0) {
    const long long L = a->dst_ld;
    const long long dims[5] = {a->cin, a->W, a->H, a->D, a->N};
    const long long str[5] = {1, L, a->W * L, (long long)a->H * a->W * L, (long long)a->D * a->H * a->W * L};
    rc = out_map(p, &p.mapO[0], a->dst, dims, str);
    if (rc) return rc;
  }
  return finish_and_launch(p, rows, stream);
}
