// w2d_nn_train.cu -- training steps of the cooling network on batches of more
// than one tile.  The network, its operand layouts and the quantities of a
// step (forward, loss, backward data and weight gradients, all BF16 MMAs with
// FP32 accumulation) are those of k_nn_train in w2d_nn.cu, which keeps batches
// of one tile and single gradients: programs train one tile at a time to get
// the same weights again, and the order in which that kernel adds its bias
// gradients carries, through BF16 rounding, into weights 1e-4 apart after a few
// hundred steps, while the kernels here add in another order.
//
// k_nn_train_multi: one CTA of 256 threads per 128-sample tile, threads r and
// 128 + r owning sample r of the tile (TMEM lane r), the first and the second
// 32 of its 64 hidden units.  Every CTA stores its gradient to a slot of its
// own, and the Adam kernel adds the slots in a fixed order: the same training
// repeats bit for bit.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/w2d.h"
#include "w2d_launch.h"
#include "w2d_nn.cuh"

using namespace w2d;

namespace {

// Operand [R][128 samples] of the K = samples MMAs: core matrices of 8 rows x
// 8 samples, 16 per 8 rows, 144 bytes apart: with the 16 bytes of padding the
// 32 samples of a warp fall in different banks (without, four by four in one).
constexpr uint32_t kCoreT = 144;
constexpr int kGroupT = 16 * (int)kCoreT / 2;   // halfwords per 8 rows
__device__ __forceinline__ uint32_t tct_at(int r, int s)   // halfword index of (r, s)
{
  return (uint32_t)(((r >> 3) * 16 + (s >> 3)) * (int)(kCoreT / 2) + (r & 7) * 8 + (s & 7));
}

struct __align__(128) NNMultiSmem {
  // A operands of the K = samples MMAs: rows 0..63 (0..1 for dot) hold the
  // data, rows up to 127 read whatever follows (those D rows are unused),
  // so each of these is followed by at least 36 KB - its size of buffers
  uint16_t dz2t[NN_H / 8 * kGroupT];
  uint16_t dz1t[NN_H / 8 * kGroupT];
  uint16_t dot[kGroupT];
  uint16_t h1t[NN_H / 8 * kGroupT];
  uint16_t h2t[NN_H / 8 * kGroupT];
  uint16_t xt[NN_KIN / 8 * kGroupT];
  NNFwdSmem f;
  uint16_t dout[128 * NN_NOUT];
  uint16_t dz2[128 * NN_H];
  uint16_t w2t[NN_H * NN_H];
  uint16_t w3t[NN_H * NN_NOUT];
  float gb[4][2 * NN_H];     // bias gradients of a warp's 32 samples (layers 1, 2)
  float g3[4][3];            // output biases and the loss
  uint64_t bar;
  uint32_t tmem;
};

// a CTA's gradient slot: P_N values and the loss, padded to 16 bytes
constexpr int NN_PART = (P_N + 1 + 3) / 4 * 4;

// MMAs with K = 128 samples into an accumulator: D += A[128 x 128] B[N x 128]^T
__device__ __forceinline__ void nn_kmma(uint32_t d, const uint16_t* a, const uint16_t* b, int N, bool acc)
{
  const uint32_t aa = smem_u32(a), bb = smem_u32(b);
  const uint32_t idesc = tc_idesc_bf16(128, N);
  for (int k = 0; k < 8; ++k)
    tc_mma(d, tc_desc(aa + 2u * kCoreT * k, kCoreT, 16u * kCoreT), tc_desc(bb + 2u * kCoreT * k, kCoreT, 16u * kCoreT),
           idesc, acc || k > 0);
}

// Sums of 32 columns over the warp's 32 lanes: column `lane` to each lane.  Every
// round halves the columns a lane carries (31 shuffles instead of 32 x 5); the
// sums pair the lanes as a shuffle tree per column does.  v is overwritten.
__device__ __forceinline__ float nn_colsum(float (&v)[32], int lane)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int k = 0; k < o; ++k) {
      const float keep = up ? v[k + o] : v[k], send = up ? v[k] : v[k + o];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// What bounds it: the latency of one tile, six dependent MMA rounds with their
// epilogues on a batch of 64 tiles for 148 SMs.  Two threads per sample halve
// the epilogues; the bias gradients' column sums exchange halves instead of
// reducing column by column (one thread per sample, 640 shuffles and 128
// shared atomics each, 300,000 global atomics a launch: 48 us; so 15 us under the same profiler).
__global__ void __launch_bounds__(256, 1) k_nn_train_multi(const float* __restrict__ feat, const float* __restrict__ targ,
                                                    int64_t ld, int64_t first, int64_t count, float inv_batch,
                                                    const NNImage* __restrict__ img, float* __restrict__ part,
                                                    int* __restrict__ err)
{
  extern __shared__ __align__(1024) uint8_t nn_smem[];
  NNMultiSmem& s = *reinterpret_cast<NNMultiSmem*>(nn_smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = tid & 127, lane0 = 32 * (warp & 3);   // sample of the tile, its warp's first TMEM lane
  const bool lo = tid < 128;
  const int c0 = lo ? 0 : NN_H / 2;                     // this thread's hidden units c0 .. c0 + 31
  for (int k = tid; k < 128 * NN_NOUT; k += 256) s.dout[k] = 0;
  if (tid == 0) mbar_init(&s.bar, 1);
  if (warp == 0) tc_alloc(&s.tmem, C_ALLOC);
  pdl_begin();
  nn_load_weights(s.f, img);
  for (int k = tid; k < (int)(sizeof(s.w2t) / 16); k += 256)
    reinterpret_cast<uint4*>(s.w2t)[k] = reinterpret_cast<const uint4*>(img->w2t)[k];
  for (int k = tid; k < (int)(sizeof(s.w3t) / 16); k += 256)
    reinterpret_cast<uint4*>(s.w3t)[k] = reinterpret_cast<const uint4*>(img->w3t)[k];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = s.tmem;
  uint32_t phase = 0;
  bool first_tile = true, ok = true;
  const int64_t ntiles = (count + 127) / 128;
  float lsum = 0.f, gb3a = 0.f, gb3b = 0.f, gb1 = 0.f, gb2 = 0.f;
  auto ld32 = [&](int col, float* v) {
    tc_ld16(tc_addr(tm, lane0, col + c0), v);
    tc_ld16(tc_addr(tm, lane0, col + c0 + 16), v + 16);
  };
  for (int64_t t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
    const int64_t i = first + t * 128 + row;
    const bool valid = t * 128 + row < count;
    float y[2] = {0.f, 0.f};
    if (lo) {
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      if (valid) {
#pragma unroll
        for (int q = 0; q < 4; ++q) f[q] = feat[q * ld + i];
        y[0] = targ[i];
        y[1] = targ[ld + i];
      }
      nn_put_x(s.f, row, f);
#pragma unroll
      for (int k = 0; k < NN_KIN; ++k) s.xt[tct_at(k, row)] = k < NN_IN ? f2bf(f[k]) : (uint16_t)0;
    }
    nn_sync();
    if (tid == 0) {
      nn_layer_mma(tm + C_Z1, 0, s.f.x, s.f.w1, NN_KIN, NN_H);
      tc_commit(&s.bar);
    }
    if (!(ok = nn_wait(&s.bar, phase, err))) break;
    float h1[32], h2[32], v[32];
    ld32(C_Z1, v);
    // h1 holds the clamped pre-activation y of layer 1 (its gradient needs y)
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      h1[k] = nn_clamp2(v[k] + s.f.b1[c0 + k]);
      v[k] = nn_cubic(h1[k]);
      s.h1t[tct_at(c0 + k, row)] = f2bf(v[k]);
    }
#pragma unroll
    for (int k = 0; k < 32; k += 8) nn_put8(s.f.h1, row, c0 + k, NN_H, v + k);
    nn_sync();
    if (tid == 0) {
      nn_layer_mma(tm + C_Z2, 0, s.f.h1, s.f.w2, NN_H, NN_H);
      tc_commit(&s.bar);
    }
    if (!(ok = nn_wait(&s.bar, phase, err))) break;
    ld32(C_Z2, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      h2[k] = nn_tanh(v[k] + s.f.b2[c0 + k]);
      s.h2t[tct_at(c0 + k, row)] = f2bf(h2[k]);
    }
#pragma unroll
    for (int k = 0; k < 32; k += 8) nn_put8(s.f.h2, row, c0 + k, NN_H, h2 + k);
    nn_sync();
    if (tid == 0) {
      nn_layer_mma(tm + C_O, 0, s.f.h2, s.f.w3, NN_H, NN_NOUT);
      tc_commit(&s.bar);
    }
    if (!(ok = nn_wait(&s.bar, phase, err))) break;
    if (lo) {
      tc_ld16(tc_addr(tm, lane0, C_O), v);
      const float o0 = v[0] + s.f.b3[0], o1 = v[1] + s.f.b3[1];
      const float e0 = valid ? o0 - y[0] : 0.f, e1 = valid ? o1 - y[1] : 0.f;
      lsum += e0 * e0 + NN_W1 * e1 * e1;
      const float d0 = 2.f * e0 * inv_batch, d1 = 2.f * NN_W1 * e1 * inv_batch;
      gb3a += d0;
      gb3b += d1;
      s.dout[tc_off(row, 0, NN_NOUT) >> 1] = f2bf(d0);
      s.dout[tc_off(row, 1, NN_NOUT) >> 1] = f2bf(d1);
      s.dot[tct_at(0, row)] = f2bf(d0);
      s.dot[tct_at(1, row)] = f2bf(d1);
    }
    nn_sync();
    if (tid == 0) {
      nn_layer_mma(tm + C_Z2, 0, s.dout, s.w3t, NN_NOUT, NN_H);      // dH2 over Z2
      nn_kmma(tm + C_G3, s.dot, s.h2t, NN_H, !first_tile);           // G3 += dO^T H2
      tc_commit(&s.bar);
    }
    if (!(ok = nn_wait(&s.bar, phase, err))) break;
    ld32(C_Z2, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      v[k] = v[k] * (1.f - h2[k] * h2[k]);
      s.dz2t[tct_at(c0 + k, row)] = f2bf(v[k]);
    }
#pragma unroll
    for (int k = 0; k < 32; k += 8) nn_put8(s.dz2, row, c0 + k, NN_H, v + k);
    nn_sync();
    if (tid == 0) {
      nn_layer_mma(tm + C_Z1, 0, s.dz2, s.w2t, NN_H, NN_H);          // dH1 over Z1
      nn_kmma(tm + C_G2, s.dz2t, s.h1t, NN_H, !first_tile);          // G2 += dZ2^T H1
      tc_commit(&s.bar);
    }
    gb2 += nn_colsum(v, lane);   // bias gradient of layer 2, while the MMAs run
    if (!(ok = nn_wait(&s.bar, phase, err))) break;
    ld32(C_Z1, v);
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      v[k] = v[k] * nn_cubic_grad(h1[k]);
      s.dz1t[tct_at(c0 + k, row)] = f2bf(v[k]);
    }
    nn_sync();
    if (tid == 0) {
      nn_kmma(tm + C_G1, s.dz1t, s.xt, NN_KIN, !first_tile);         // G1 += dZ1^T X
      tc_commit(&s.bar);
    }
    gb1 += nn_colsum(v, lane);
    if (!(ok = nn_wait(&s.bar, phase, err))) break;
    first_tile = false;
  }
  // bias gradients and the loss: warp sums, then the four sample warps' in a
  // fixed order
  s.gb[warp & 3][c0 + lane] = gb1;
  s.gb[warp & 3][NN_H + c0 + lane] = gb2;
  if (lo) {
    for (int o = 16; o > 0; o >>= 1) {
      gb3a += __shfl_xor_sync(0xffffffffu, gb3a, o);
      gb3b += __shfl_xor_sync(0xffffffffu, gb3b, o);
      lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    }
    if (lane == 0) {
      s.g3[warp][0] = gb3a;
      s.g3[warp][1] = gb3b;
      s.g3[warp][2] = lsum;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  float* out = part + (size_t)blockIdx.x * NN_PART;
  if (ok) {
    float v[32];
    if ((warp & 3) < 2) {   // rows 0..63 of G1 and G2 live in lanes 0..63
      ld32(C_G2, v);
#pragma unroll
      for (int k = 0; k < 32; k += 4)
        *reinterpret_cast<float4*>(out + P_W2 + row * NN_H + c0 + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
      if (lo) {
        tc_ld16(tc_addr(tm, lane0, C_G1), v);
        *reinterpret_cast<float4*>(out + P_W1 + row * NN_IN) = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
    if ((warp & 3) == 0) {
      ld32(C_G3, v);
      if (lane < NN_OUT)
#pragma unroll
        for (int k = 0; k < 32; ++k) out[P_W3 + lane * NN_H + c0 + k] = v[k];
    }
    if (tid < 2 * NN_H)
      out[(tid < NN_H ? P_B1 : P_B2 - NN_H) + tid] = ((s.gb[0][tid] + s.gb[1][tid]) + s.gb[2][tid]) + s.gb[3][tid];
    if (tid < 3) {
      const float x = ((s.g3[0][tid] + s.g3[1][tid]) + s.g3[2][tid]) + s.g3[3][tid];
      out[P_B3 + tid] = tid < 2 ? x : x * inv_batch;   // (the loss follows the biases)
    }
  } else {
    for (int k = tid; k < P_N + 1; k += 256) out[k] = 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tc_dealloc(tm, C_ALLOC);
}

// The gradient (with the loss behind it) from the CTAs' slots, in slot order
// per slice of eight and then the slices in order; Adam (fp32 master weights)
// and the bf16 operand image.  32 parameters per CTA, a warp per slice.
__global__ void __launch_bounds__(256) k_nn_adam_multi(const float* __restrict__ part, int nparts, float* __restrict__ p,
                                                 float* __restrict__ m, float* __restrict__ v, NNImage* __restrict__ img,
                                                 float* __restrict__ loss, float lr, float b1c, float b2c)
{
  __shared__ float red[8][32];
  const int slice = threadIdx.x >> 5, k = blockIdx.x * 32 + (threadIdx.x & 31);
  pdl_begin();
  float gr = 0.f;
  if (k <= P_N)
    for (int c = slice; c < nparts; c += 8) gr += part[(size_t)c * NN_PART + k];
  red[slice][threadIdx.x & 31] = gr;
  __syncthreads();
  if (slice > 0 || k > P_N) return;
  for (int q = 1; q < 8; ++q) gr += red[q][threadIdx.x & 31];
  if (k == P_N) {
    *loss = gr;
    return;
  }
  float w = p[k];
  const float mk = 0.9f * m[k] + 0.1f * gr;
  const float vk = 0.999f * v[k] + 0.001f * gr * gr;
  m[k] = mk;
  v[k] = vk;
  w -= lr * (mk / b1c) / (sqrtf(vk / b2c) + 1e-8f);
  p[k] = w;
  const uint16_t wb = f2bf(w);
  if (k < P_B1) {
    const int r = k / NN_IN, c = k % NN_IN;
    img->w1[tc_off(r, c, NN_KIN) >> 1] = wb;
  } else if (k < P_W2) {
    img->b1[k - P_B1] = w;
  } else if (k < P_B2) {
    const int r = (k - P_W2) / NN_H, c = (k - P_W2) % NN_H;
    img->w2[tc_off(r, c, NN_H) >> 1] = wb;
    img->w2t[tc_off(c, r, NN_H) >> 1] = wb;
  } else if (k < P_W3) {
    img->b2[k - P_B2] = w;
  } else if (k < P_B3) {
    const int r = (k - P_W3) / NN_H, c = (k - P_W3) % NN_H;
    img->w3[tc_off(r, c, NN_H) >> 1] = wb;
    img->w3t[tc_off(c, r, NN_NOUT) >> 1] = wb;
  } else {
    img->b3[k - P_B3] = w;
  }
}

}  // namespace

namespace w2d {

size_t nn_part_floats(int nsm) { return (size_t)NN_PART * (size_t)nsm + 4; }   // the slots, then the loss
const float* nn_train_loss(const NNTrainArgs& a) { return a.part + (size_t)NN_PART * (size_t)a.nsm; }

cudaError_t nn_train_step(const NNTrainArgs& a, const float* feat, const float* targ, int64_t ld, int64_t first,
                          int64_t count, float lr, float b1c, float b2c, cudaStream_t st)
{
  static bool opted = false;
  if (!opted) {
    cudaError_t e = cudaFuncSetAttribute(k_nn_train_multi, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(NNMultiSmem));
    if (e != cudaSuccess) return e;
    opted = true;
  }
  const int grid = (int)std::min<int64_t>((count + 127) / 128, a.nsm);
  cudaError_t e = launch_pdl(k_nn_train_multi, grid, 256, sizeof(NNMultiSmem), st, feat, targ, ld, first, count,
                             1.f / (float)count, a.img, a.part, a.err);
  if (e != cudaSuccess) return e;
  return launch_pdl(k_nn_adam_multi, (P_N + 1 + 31) / 32, 256, 0, st, a.part, grid, a.p, a.m, a.v, a.img,
                    a.part + (size_t)NN_PART * (size_t)a.nsm, lr, b1c, b2c);
}

}  // namespace w2d
