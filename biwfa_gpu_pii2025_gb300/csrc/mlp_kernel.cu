// Learned scheduling: per-pair sketch features and a small MLP that predicts each pair's
// alignment score. The prediction only orders and bins pairs and sizes scratch; it never
// changes a result (a mispredicted pair overflows into a larger-arena pass).
//
// Features (32 per pair, bf16):
//   f0  log2(|P|+1)/16          f1  log2(|T|+1)/16        f2  (|P|-|T|)/(|P|+|T|+1)
//   f3..f30  histogram of the 256 per-4-mer count differences |cP[k]-cT[k]| in 28 bins
//            (d = 0..15 one bin each, then one bin per power of two up to 2^15), / 256
//   f31 the 4-mer count L1 distance sum_k |cP[k]-cT[k]| / (|P|+|T|+1)
// Network: 32 -> 64 -> 64 -> 1, ReLU, bf16 weights and activations between layers, fp32
// accumulation (mma.sync m16n8k16 bf16 -> f32), target log(1 + |score|).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "wfg_internal.h"

namespace wfg {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kIn = 32, kHid = 64;

__device__ __forceinline__ int kmer_bin(int d) {
  if (d < 16) return d;
  const int lg = 31 - __clz(d);  // >= 4
  return min(27, 16 + (lg - 4));
}

// One warp per pair: 4-mer counts of both sequences in shared memory, then the features.
template <int WPB>
__global__ void __launch_bounds__(WPB * 32) kmer_features_kernel(int n, const uint8_t* __restrict__ ascii,
                                                                const PairDesc* __restrict__ pairs,
                                                                __nv_bfloat16* __restrict__ feats) {
  __shared__ int s_cnt[WPB][2][256];
  __shared__ int s_hist[WPB][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  for (long long i = (long long)blockIdx.x * WPB + wib; i < n; i += (long long)gridDim.x * WPB) {
    const PairDesc pd = pairs[i];
    for (int k = lane; k < 512; k += 32) (&s_cnt[wib][0][0])[k] = 0;
    s_hist[wib][lane] = 0;
    __syncwarp();
    for (int side = 0; side < 2; ++side) {
      const uint8_t* s = ascii + (side ? pd.t_off : pd.p_off);
      const int len = side ? pd.tlen : pd.plen;
      for (int j = lane; j + 3 < len; j += 32) {
        const int code = (((s[j] >> 1) & 3) << 6) | (((s[j + 1] >> 1) & 3) << 4) | (((s[j + 2] >> 1) & 3) << 2) |
                         ((s[j + 3] >> 1) & 3);
        atomicAdd(&s_cnt[wib][side][code], 1);
      }
    }
    __syncwarp();
    int l1 = 0;
    for (int k = lane; k < 256; k += 32) {
      const int d = abs(s_cnt[wib][0][k] - s_cnt[wib][1][k]);
      l1 += d;
      atomicAdd(&s_hist[wib][kmer_bin(d)], 1);
    }
    l1 = __reduce_add_sync(kFull, l1);
    __syncwarp();
    const float tot = (float)(pd.plen + pd.tlen + 1);
    float f;
    if (lane == 0) f = log2f((float)pd.plen + 1.f) * (1.f / 16.f);
    else if (lane == 1) f = log2f((float)pd.tlen + 1.f) * (1.f / 16.f);
    else if (lane == 2) f = (float)(pd.plen - pd.tlen) / tot;
    else if (lane < 31) f = (float)s_hist[wib][lane - 3] * (1.f / 256.f);
    else f = (float)l1 / tot;
    feats[i * kIn + lane] = __float2bfloat16(f);
    __syncwarp();
  }
}

// Parameters: fp32 master copy in one block {W1[32][64] (in-major), b1[64], W2[64][64], b2[64],
// w3[64], b3}; bf16 copies of the weight matrices transposed to [out][in] (mma B operands).
struct MlpParams {
  const float* master;            // kParamCount floats
  const __nv_bfloat16* w1t;       // [64][32]
  const __nv_bfloat16* w2t;       // [64][64]
};
constexpr int kOffW1 = 0, kOffB1 = kIn * kHid, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid;
constexpr int kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid, kParamCount = kOffB3 + 1;
// Train step: a block of 8 warps per 16-row tile. Row pitches of the staged matrices: W2's spreads
// eight rows' 16-byte reads over all banks.
constexpr int kTrainWarps = 8, kW2Pitch = kHid + 4, kHPitch = kHid + 4;

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Forward of one 16-row tile by one warp. Fragment layouts of m16n8k16 (g = lane/4, t = lane%4):
// A rows g / g+8, columns 2t..2t+1 and 2t+8..2t+9; B (col) rows 2t..2t+1 and 2t+8..2t+9 of
// column g; C rows g / g+8, columns 2t..2t+1. Layer outputs in C layout are re-packed in
// registers as the next layer's A fragments (two 8-column tiles form one 16-column k-step).
struct TileAct {
  float h1[8][4];   // layer-1 outputs after ReLU, as bf16-rounded floats (8 n-tiles)
  float h2[8][4];   // layer-2 outputs after ReLU
  float y[2];       // rows g and g+8 (valid in every lane of the group)
};

__device__ __forceinline__ void mlp_tile_forward(const __nv_bfloat16* __restrict__ x, int row0, int n,
                                                 const __nv_bfloat16* s_w1t, const __nv_bfloat16* s_w2t,
                                                 const float* s_b1, const float* s_b2, const float* s_w3,
                                                 float b3, int lane, TileAct& act) {
  const int g = lane >> 2, t = lane & 3;
  const int r0 = row0 + g, r1 = row0 + g + 8;
  // A fragments of the input tile (2 k-steps of 16 features)
  uint32_t a[2][4];
  for (int ks = 0; ks < 2; ++ks) {
    const int c0 = ks * 16 + 2 * t;
    auto ld = [&](int r, int c) -> uint32_t {
      if (r >= n) return 0u;
      return *reinterpret_cast<const uint32_t*>(x + (size_t)r * kIn + c);
    };
    a[ks][0] = ld(r0, c0);
    a[ks][1] = ld(r1, c0);
    a[ks][2] = ld(r0, c0 + 8);
    a[ks][3] = ld(r1, c0 + 8);
  }
  // Layer 1: 8 n-tiles of 8 outputs
  for (int j = 0; j < 8; ++j) {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    const int col = j * 8 + g;  // B column held by this lane
    for (int ks = 0; ks < 2; ++ks) {
      const __nv_bfloat16* wrow = s_w1t + col * kIn + ks * 16 + 2 * t;
      mma_bf16(d, a[ks], *reinterpret_cast<const uint32_t*>(wrow), *reinterpret_cast<const uint32_t*>(wrow + 8));
    }
    const int c = j * 8 + 2 * t;
    act.h1[j][0] = __bfloat162float(__float2bfloat16(fmaxf(d[0] + s_b1[c], 0.f)));
    act.h1[j][1] = __bfloat162float(__float2bfloat16(fmaxf(d[1] + s_b1[c + 1], 0.f)));
    act.h1[j][2] = __bfloat162float(__float2bfloat16(fmaxf(d[2] + s_b1[c], 0.f)));
    act.h1[j][3] = __bfloat162float(__float2bfloat16(fmaxf(d[3] + s_b1[c + 1], 0.f)));
  }
  // Layer 2: A from layer-1 tiles (2j, 2j+1) per k-step
  uint32_t a2[4][4];
  for (int ks = 0; ks < 4; ++ks) {
    a2[ks][0] = pack_bf16x2(act.h1[2 * ks][0], act.h1[2 * ks][1]);
    a2[ks][1] = pack_bf16x2(act.h1[2 * ks][2], act.h1[2 * ks][3]);
    a2[ks][2] = pack_bf16x2(act.h1[2 * ks + 1][0], act.h1[2 * ks + 1][1]);
    a2[ks][3] = pack_bf16x2(act.h1[2 * ks + 1][2], act.h1[2 * ks + 1][3]);
  }
  float y0 = 0.f, y1 = 0.f;
  for (int j = 0; j < 8; ++j) {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    const int col = j * 8 + g;
    for (int ks = 0; ks < 4; ++ks) {
      const __nv_bfloat16* wrow = s_w2t + col * kHid + ks * 16 + 2 * t;
      mma_bf16(d, a2[ks], *reinterpret_cast<const uint32_t*>(wrow), *reinterpret_cast<const uint32_t*>(wrow + 8));
    }
    const int c = j * 8 + 2 * t;
    act.h2[j][0] = fmaxf(d[0] + s_b2[c], 0.f);
    act.h2[j][1] = fmaxf(d[1] + s_b2[c + 1], 0.f);
    act.h2[j][2] = fmaxf(d[2] + s_b2[c], 0.f);
    act.h2[j][3] = fmaxf(d[3] + s_b2[c + 1], 0.f);
    y0 += act.h2[j][0] * s_w3[c] + act.h2[j][1] * s_w3[c + 1];
    y1 += act.h2[j][2] * s_w3[c] + act.h2[j][3] * s_w3[c + 1];
  }
  // Layer 3: reduce the 4 lanes of a group (columns 2t..2t+1 of every tile)
  y0 += __shfl_xor_sync(kFull, y0, 1); y0 += __shfl_xor_sync(kFull, y0, 2);
  y1 += __shfl_xor_sync(kFull, y1, 1); y1 += __shfl_xor_sync(kFull, y1, 2);
  act.y[0] = y0 + b3;
  act.y[1] = y1 + b3;
}

template <int WPB>
__device__ __forceinline__ void load_params_smem(const MlpParams& prm, __nv_bfloat16* s_w1t, __nv_bfloat16* s_w2t,
                                                 float* s_b1, float* s_b2, float* s_w3) {
  for (int i = threadIdx.x; i < kHid * kIn; i += WPB * 32) s_w1t[i] = prm.w1t[i];
  for (int i = threadIdx.x; i < kHid * kHid; i += WPB * 32) s_w2t[i] = prm.w2t[i];
  for (int i = threadIdx.x; i < kHid; i += WPB * 32) {
    s_b1[i] = prm.master[kOffB1 + i];
    s_b2[i] = prm.master[kOffB2 + i];
    s_w3[i] = prm.master[kOffW3 + i];
  }
  __syncthreads();
}

// Inference: y[i] = MLP(features[i]) (log-score), and the predicted score expm1(y) >= 0.
template <int WPB>
__global__ void __launch_bounds__(WPB * 32) mlp_forward_kernel(int n, const __nv_bfloat16* __restrict__ x,
                                                              MlpParams prm, float* __restrict__ y_out,
                                                              float* __restrict__ score_out) {
  __shared__ __align__(16) __nv_bfloat16 s_w1t[kHid * kIn];
  __shared__ __align__(16) __nv_bfloat16 s_w2t[kHid * kHid];
  __shared__ float s_b1[kHid], s_b2[kHid], s_w3[kHid];
  load_params_smem<WPB>(prm, s_w1t, s_w2t, s_b1, s_b2, s_w3);
  const float b3 = prm.master[kOffB3];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int tiles = (n + 15) / 16;
  for (int tile = blockIdx.x * WPB + wib; tile < tiles; tile += gridDim.x * WPB) {
    TileAct act;
    mlp_tile_forward(x, tile * 16, n, s_w1t, s_w2t, s_b1, s_b2, s_w3, b3, lane, act);
    if (t == 0) {
      const int r0 = tile * 16 + g, r1 = r0 + 8;
      if (r0 < n) { if (y_out) y_out[r0] = act.y[0]; if (score_out) score_out[r0] = fmaxf(expm1f(act.y[0]), 0.f); }
      if (r1 < n) { if (y_out) y_out[r1] = act.y[1]; if (score_out) score_out[r1] = fmaxf(expm1f(act.y[1]), 0.f); }
    }
  }
}

// Training step: forward (tensor cores) + backward (fp32) of the mean-squared error on a minibatch of
// `rows` rows (rows_idx); gradients and the squared error are added to grad and loss_sum. step_next,
// if given, is advanced by one (the Adam step that follows uses *step_next - 1).
//
// A minibatch of 2,048 rows is 128 tiles of 16 rows: a block of 8 warps takes a tile (more when there
// are more tiles than SMs), each warp an eighth of every layer's columns, and each thread keeps its
// 16 + 8 sums of dW2 and dW1 in registers over the block's tiles. With a warp per tile (four per block,
// 32 blocks on 152 SMs) and the sums in shared memory by atomics, a step took 58 us (ncu, caches
// flushed); now 25 us. What bounds it: latency, of the parameters' load into shared memory and of the
// chain of a tile's five products between barriers; then the 6,465 sums that each block adds to the
// gradient. Two epochs of 16,384 rows, end to end on a GB300: 1,221 -> 667 us.
__global__ void __launch_bounds__(kTrainWarps * 32) mlp_train_step_kernel(const __nv_bfloat16* __restrict__ x,
                                                                          const float* __restrict__ target,
                                                                          const int* __restrict__ rows_idx, int rows,
                                                                          MlpParams prm, float* __restrict__ grad,
                                                                          float* __restrict__ loss_sum,
                                                                          int* __restrict__ step_next) {
  __shared__ __align__(16) __nv_bfloat16 s_w1t[kHid * kIn];
  __shared__ __align__(16) __nv_bfloat16 s_w2t[kHid * kHid];
  __shared__ float s_b1[kHid], s_b2[kHid], s_w3[kHid];
  __shared__ __align__(16) float s_w2[kHid * kW2Pitch];                             // fp32 W2 [in][out]
  __shared__ __align__(16) float s_x[16 * kIn], s_h1[16 * kHPitch], s_dh2[16 * kHPitch], s_dh1[16 * kHPitch];
  __shared__ __align__(16) __nv_bfloat16 s_xb[16 * kIn];
  __shared__ float s_part[kTrainWarps][16], s_dy[16];
  const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5, g = lane >> 2, t = lane & 3;
  load_params_smem<kTrainWarps>(prm, s_w1t, s_w2t, s_b1, s_b2, s_w3);
  for (int i = tid; i < kHid * kHid; i += kTrainWarps * 32) s_w2[(i / kHid) * kW2Pitch + i % kHid] = prm.master[kOffW2 + i];
  const float b3 = prm.master[kOffB3], inv_rows = 1.f / (float)rows;
  // this thread's sums: dW2[i2 .. i2+15][j2], dW1[f1 .. f1+7][j2], db1/db2[tid], dW3 of columns c, c + 1
  const int j2 = tid & 63, i2 = (tid >> 6) * 16, f1 = (tid >> 6) * 8, c = wib * 8 + 2 * t;
  float dw2[16] = {}, dw1[8] = {}, db1 = 0.f, db2 = 0.f, dw3a = 0.f, dw3b = 0.f, db3 = 0.f, lsum = 0.f;
  const int tiles = (rows + 15) / 16;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    __syncthreads();
    for (int e = tid; e < 16 * kIn; e += kTrainWarps * 32) {
      const int rr = tile * 16 + e / kIn;
      const __nv_bfloat16 v = rr < rows ? x[(size_t)rows_idx[rr] * kIn + e % kIn] : __float2bfloat16(0.f);
      s_xb[e] = v;
      s_x[e] = __bfloat162float(v);
    }
    __syncthreads();
    // Layer 1, this warp's 8 columns (fragment layouts: mlp_tile_forward)
    {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      #pragma unroll
      for (int ks = 0; ks < 2; ++ks) {
        const int c0 = ks * 16 + 2 * t;
        uint32_t a[4];
        a[0] = *reinterpret_cast<const uint32_t*>(s_xb + g * kIn + c0);
        a[1] = *reinterpret_cast<const uint32_t*>(s_xb + (g + 8) * kIn + c0);
        a[2] = *reinterpret_cast<const uint32_t*>(s_xb + g * kIn + c0 + 8);
        a[3] = *reinterpret_cast<const uint32_t*>(s_xb + (g + 8) * kIn + c0 + 8);
        const __nv_bfloat16* w = s_w1t + (wib * 8 + g) * kIn + c0;
        mma_bf16(d, a, *reinterpret_cast<const uint32_t*>(w), *reinterpret_cast<const uint32_t*>(w + 8));
      }
      #pragma unroll
      for (int q = 0; q < 4; ++q)
        s_h1[(g + 8 * (q >> 1)) * kHPitch + c + (q & 1)] =
            __bfloat162float(__float2bfloat16(fmaxf(d[q] + s_b1[c + (q & 1)], 0.f)));
    }
    __syncthreads();
    // Layer 2 and this warp's part of the output
    float h2[4] = {0.f, 0.f, 0.f, 0.f};
    #pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const int c0 = ks * 16 + 2 * t;
      const float* r0 = s_h1 + g * kHPitch + c0;
      const float* r1 = r0 + 8 * kHPitch;
      uint32_t a[4] = {pack_bf16x2(r0[0], r0[1]), pack_bf16x2(r1[0], r1[1]), pack_bf16x2(r0[8], r0[9]),
                       pack_bf16x2(r1[8], r1[9])};
      const __nv_bfloat16* w = s_w2t + (wib * 8 + g) * kHid + c0;
      mma_bf16(h2, a, *reinterpret_cast<const uint32_t*>(w), *reinterpret_cast<const uint32_t*>(w + 8));
    }
    #pragma unroll
    for (int q = 0; q < 4; ++q) h2[q] = fmaxf(h2[q] + s_b2[c + (q & 1)], 0.f);
    float y0 = h2[0] * s_w3[c] + h2[1] * s_w3[c + 1], y1 = h2[2] * s_w3[c] + h2[3] * s_w3[c + 1];
    y0 += __shfl_xor_sync(kFull, y0, 1); y0 += __shfl_xor_sync(kFull, y0, 2);
    y1 += __shfl_xor_sync(kFull, y1, 1); y1 += __shfl_xor_sync(kFull, y1, 2);
    if (t == 0) { s_part[wib][g] = y0; s_part[wib][g + 8] = y1; }
    __syncthreads();
    if (tid < 16) {  // dL/dy = 2 (y - target) / rows
      const int rr = tile * 16 + tid;
      float dy = 0.f;
      if (rr < rows) {
        float y = 0.f;
        #pragma unroll
        for (int w = 0; w < kTrainWarps; ++w) y += s_part[w][tid];
        const float e = y + b3 - target[rows_idx[rr]];
        dy = 2.f * e * inv_rows;
        lsum += e * e;
        db3 += dy;
      }
      s_dy[tid] = dy;
    }
    __syncthreads();
    // dh2 = dy * w3 * (h2 > 0), dW3
    const float dy0 = s_dy[g], dy1 = s_dy[g + 8];
    #pragma unroll
    for (int q = 0; q < 4; ++q)
      s_dh2[(g + 8 * (q >> 1)) * kHPitch + c + (q & 1)] = h2[q] > 0.f ? (q < 2 ? dy0 : dy1) * s_w3[c + (q & 1)] : 0.f;
    dw3a += h2[0] * dy0 + h2[2] * dy1;
    dw3b += h2[1] * dy0 + h2[3] * dy1;
    __syncthreads();
    // dh1[r][i] = (h1 > 0) * sum_j dh2[r][j] W2[i][j]: row tid / 16, columns tid % 16 + 16 q
    {
      const int r = tid >> 4, i0 = tid & 15;
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      #pragma unroll 4
      for (int j = 0; j < kHid; j += 4) {
        const float4 v = *reinterpret_cast<const float4*>(s_dh2 + r * kHPitch + j);
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 w = *reinterpret_cast<const float4*>(s_w2 + (i0 + 16 * q) * kW2Pitch + j);
          acc[q] += v.x * w.x; acc[q] += v.y * w.y; acc[q] += v.z * w.z; acc[q] += v.w * w.w;
        }
      }
      #pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int at = r * kHPitch + i0 + 16 * q;
        s_dh1[at] = s_h1[at] > 0.f ? acc[q] : 0.f;
      }
    }
    // dW2[i][j] = sum_r h1[r][i] dh2[r][j], db2
    #pragma unroll 4
    for (int r = 0; r < 16; ++r) {
      const float dh = s_dh2[r * kHPitch + j2];
      #pragma unroll
      for (int q = 0; q < 16; q += 4) {
        const float4 h = *reinterpret_cast<const float4*>(s_h1 + r * kHPitch + i2 + q);
        dw2[q] += h.x * dh; dw2[q + 1] += h.y * dh; dw2[q + 2] += h.z * dh; dw2[q + 3] += h.w * dh;
      }
      if (tid < kHid) db2 += dh;
    }
    __syncthreads();
    // dW1[f][i] = sum_r x[r][f] dh1[r][i], db1
    #pragma unroll 4
    for (int r = 0; r < 16; ++r) {
      const float dh = s_dh1[r * kHPitch + j2];
      #pragma unroll
      for (int q = 0; q < 8; q += 4) {
        const float4 v = *reinterpret_cast<const float4*>(s_x + r * kIn + f1 + q);
        dw1[q] += v.x * dh; dw1[q + 1] += v.y * dh; dw1[q + 2] += v.z * dh; dw1[q + 3] += v.w * dh;
      }
      if (tid < kHid) db1 += dh;
    }
  }
  // The block's sums into the gradient.
  #pragma unroll
  for (int q = 0; q < 16; ++q) atomicAdd(&grad[kOffW2 + (i2 + q) * kHid + j2], dw2[q]);
  #pragma unroll
  for (int q = 0; q < 8; ++q) atomicAdd(&grad[kOffW1 + (f1 + q) * kHid + j2], dw1[q]);
  if (tid < kHid) { atomicAdd(&grad[kOffB1 + tid], db1); atomicAdd(&grad[kOffB2 + tid], db2); }
  #pragma unroll
  for (int off = 4; off < 32; off <<= 1) {  // over the rows (lanes with equal t)
    dw3a += __shfl_xor_sync(kFull, dw3a, off);
    dw3b += __shfl_xor_sync(kFull, dw3b, off);
  }
  if (g == 0) { atomicAdd(&grad[kOffW3 + c], dw3a); atomicAdd(&grad[kOffW3 + c + 1], dw3b); }
  if (wib == 0) {
    #pragma unroll
    for (int off = 8; off > 0; off >>= 1) {
      lsum += __shfl_xor_sync(kFull, lsum, off);
      db3 += __shfl_xor_sync(kFull, db3, off);
    }
    if (lane == 0) {
      atomicAdd(&grad[kOffB3], db3);
      if (loss_sum) atomicAdd(loss_sum, lsum);
      if (step_next && blockIdx.x == 0) *step_next += 1;
    }
  }
}

// Adam update of the fp32 master parameters, then the bf16 transposed weight copies.
// step_next points at the next 1-based Adam step in device memory (the train step has advanced it),
// so a captured training epoch replays with fresh bias corrections. The gradient is zeroed for the
// next train step.
__global__ void mlp_adam_kernel(float* __restrict__ master, float* __restrict__ grad, float* __restrict__ m,
                                float* __restrict__ v, float lr, float beta1, float beta2, float eps,
                                const int* __restrict__ step_next, __nv_bfloat16* __restrict__ w1t,
                                __nv_bfloat16* __restrict__ w2t) {
  const float t = (float)(*step_next - 1);
  const float bc1 = 1.f - powf(beta1, t), bc2 = 1.f - powf(beta2, t);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParamCount; i += gridDim.x * blockDim.x) {
    const float gi = grad[i];
    grad[i] = 0.f;
    const float mi = beta1 * m[i] + (1.f - beta1) * gi;
    const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float p = master[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    master[i] = p;
    if (i < kOffB1) { const int f = i / kHid, o = i % kHid; w1t[o * kIn + f] = __float2bfloat16(p); }
    else if (i >= kOffW2 && i < kOffB2) { const int a = (i - kOffW2) / kHid, o = (i - kOffW2) % kHid; w2t[o * kHid + a] = __float2bfloat16(p); }
  }
}

// bf16 transposed copies of the weight matrices from the fp32 master (after init or load).
__global__ void mlp_sync_bf16_kernel(const float* __restrict__ master, __nv_bfloat16* __restrict__ w1t,
                                     __nv_bfloat16* __restrict__ w2t) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kIn * kHid + kHid * kHid; i += gridDim.x * blockDim.x) {
    if (i < kIn * kHid) { const int f = i / kHid, o = i % kHid; w1t[o * kIn + f] = __float2bfloat16(master[kOffW1 + i]); }
    else { const int k = i - kIn * kHid; const int a = k / kHid, o = k % kHid; w2t[o * kHid + a] = __float2bfloat16(master[kOffW2 + k]); }
  }
}

}  // namespace

int mlp_param_count() { return kParamCount; }

cudaError_t launch_kmer_features(int n, const uint8_t* ascii, const PairDesc* pairs, void* feats_bf16, int num_sms,
                                 cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  constexpr int WPB = 8;
  long long blocks = ((long long)n + WPB - 1) / WPB;
  if (blocks > (long long)num_sms * 8) blocks = (long long)num_sms * 8;
  kmer_features_kernel<WPB><<<(int)blocks, WPB * 32, 0, stream>>>(n, ascii, pairs, (__nv_bfloat16*)feats_bf16);
  return cudaGetLastError();
}

cudaError_t launch_mlp_forward(int n, const void* feats_bf16, const float* master, const void* w1t, const void* w2t,
                               float* y_out, float* score_out, int num_sms, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  constexpr int WPB = 4;
  MlpParams prm{master, (const __nv_bfloat16*)w1t, (const __nv_bfloat16*)w2t};
  const int tiles = (n + 15) / 16;
  long long blocks = ((long long)tiles + WPB - 1) / WPB;
  if (blocks > (long long)num_sms * 8) blocks = (long long)num_sms * 8;
  mlp_forward_kernel<WPB><<<(int)blocks, WPB * 32, 0, stream>>>(n, (const __nv_bfloat16*)feats_bf16, prm, y_out,
                                                                score_out);
  return cudaGetLastError();
}

cudaError_t launch_mlp_train_step(const void* feats_bf16, const float* target, const int* rows_idx, int rows,
                                  const float* master, const void* w1t, const void* w2t, float* grad, float* loss_sum,
                                  int* step_next, int num_sms, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  MlpParams prm{master, (const __nv_bfloat16*)w1t, (const __nv_bfloat16*)w2t};
  const int blocks = std::min((rows + 15) / 16, num_sms);
  mlp_train_step_kernel<<<blocks, kTrainWarps * 32, 0, stream>>>((const __nv_bfloat16*)feats_bf16, target, rows_idx, rows,
                                                                 prm, grad, loss_sum, step_next);
  return cudaGetLastError();
}

cudaError_t launch_mlp_adam(float* master, float* grad, float* m, float* v, float lr, float beta1, float beta2,
                            float eps, const int* step_next, void* w1t, void* w2t, cudaStream_t stream) {
  mlp_adam_kernel<<<(kParamCount + 127) / 128, 128, 0, stream>>>(master, grad, m, v, lr, beta1, beta2, eps, step_next,
                                                                 (__nv_bfloat16*)w1t, (__nv_bfloat16*)w2t);
  return cudaGetLastError();
}

// Training targets log(1 + |score|), rounded from 64 bits.
__global__ void mlp_targets_kernel(int n, const int* __restrict__ scores, float* __restrict__ targets) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    targets[i] = (float)log1p(fabs((double)scores[i]));
}

cudaError_t launch_mlp_targets(int n, const int* scores, float* targets, cudaStream_t stream) {
  if (n <= 0) return cudaSuccess;
  mlp_targets_kernel<<<std::min((n + 255) / 256, 1024), 256, 0, stream>>>(n, scores, targets);
  return cudaGetLastError();
}

cudaError_t launch_mlp_sync_bf16(const float* master, void* w1t, void* w2t, cudaStream_t stream) {
  mlp_sync_bf16_kernel<<<(kIn * kHid + kHid * kHid + 255) / 256, 256, 0, stream>>>(master, (__nv_bfloat16*)w1t,
                                                                                    (__nv_bfloat16*)w2t);
  return cudaGetLastError();
}

}  // namespace wfg
