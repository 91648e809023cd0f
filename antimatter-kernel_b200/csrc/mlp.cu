// Learned far-field correction: a 35 -> 128 -> 128 -> 128 -> 3 MLP with GELU
// activations, BF16 weights and FP32 accumulation (no reference
// counterpart).
//
// Inference runs on the 5th-generation tensor cores: a persistent CTA keeps
// all weights in shared memory (BF16, the canonical K-major no-swizzle
// layout of 8-row x 16-byte core matrices), stages each 128-particle tile of
// features as BF16, and issues tcgen05.mma (M = 128, K = 16 per
// instruction) from one thread into an FP32 accumulator in tensor memory;
// the four warps read their 32 rows back with tcgen05.ld, add the bias,
// apply GELU and write the next layer's BF16 operand. Completion of each
// layer is tracked by tcgen05.commit on an mbarrier whose waits are
// bounded (a timeout sets an error flag and the kernel returns).
//
// Training runs in FP32 on the CUDA cores with the same BF16-rounded
// weights, two kernels per step: mlp_backprop_kernel (forward, loss, backward
// and weight gradients of a tile of samples, everything in shared memory)
// and mlp_update_kernel (the tiles' gradients summed in a fixed order, Adam).
// It is checked against an FP64 CPU implementation.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cuda_bf16.h>

#include "amk_internal.cuh"
#include "philox.cuh"
#include "tcgen05.cuh"

namespace amk {

constexpr int kMlpIn = 35;      // features
constexpr int kMlpInPad = 48;   // K of layer 1 (multiple of 16)
constexpr int kMlpHidden = 128;
constexpr int kMlpOut = 3;
constexpr int kMlpOutPad = 16;  // N of layer 4

// FP32 master parameters, flat: W1[128][35] b1[128] W2[128][128] b2 W3 b3 W4[3][128] b4[3]
constexpr int kOffW1 = 0;
constexpr int kOffB1 = kOffW1 + kMlpHidden * kMlpIn;
constexpr int kOffW2 = kOffB1 + kMlpHidden;
constexpr int kOffB2 = kOffW2 + kMlpHidden * kMlpHidden;
constexpr int kOffW3 = kOffB2 + kMlpHidden;
constexpr int kOffB3 = kOffW3 + kMlpHidden * kMlpHidden;
constexpr int kOffW4 = kOffB3 + kMlpHidden;
constexpr int kOffB4 = kOffW4 + kMlpOut * kMlpHidden;
constexpr int kMlpParams = kOffB4 + kMlpOut;

struct Mlp {
  DevBuf master, grad, adam_m, adam_v;  // FP32, kMlpParams each
  DevBuf packed;                         // BF16 weights in the tensor-core smem image + FP32 biases
  DevBuf train;                          // BF16 weights in the training kernels' layouts (TrainImg)
  DevBuf status;                         // int error flag
  long adam_step = 0;
  bool packed_valid = false, train_valid = false;
  bool initialized = false;
};

namespace {

// ---------------------------------------------------------------- layout
using namespace tc;  // op_offset: the K-major no-swizzle operand layout

// smem image of the weights (built once on the host side of every update)
constexpr uint32_t kImgW1 = 0;                                            // 128 x 48
constexpr uint32_t kImgW2 = kImgW1 + kMlpHidden * kMlpInPad * 2;          // 128 x 128
constexpr uint32_t kImgW3 = kImgW2 + kMlpHidden * kMlpHidden * 2;
constexpr uint32_t kImgW4 = kImgW3 + kMlpHidden * kMlpHidden * 2;         // 16 x 128
constexpr uint32_t kImgBias = kImgW4 + kMlpOutPad * kMlpHidden * 2;       // FP32: 128*3 + 16
constexpr uint32_t kImgBytes = kImgBias + (3 * kMlpHidden + kMlpOutPad) * 4;
constexpr uint32_t kActBytes = kMlpHidden * kMlpHidden * 2;               // 128 x 128 BF16 operand
constexpr uint32_t kSmemBytes = kImgBytes + kActBytes + 64;               // + mbarrier, TMEM slot

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
  return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) + x * 0.3989422804014327f * expf(-0.5f * x * x);
}

// 8 FP32 values -> 8 BF16 packed in 16 bytes
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 u;
  u.x = (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[1]))) << 16) |
        __bfloat16_as_ushort(__float2bfloat16_rn(v[0]));
  u.y = (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[3]))) << 16) |
        __bfloat16_as_ushort(__float2bfloat16_rn(v[2]));
  u.z = (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[5]))) << 16) |
        __bfloat16_as_ushort(__float2bfloat16_rn(v[4]));
  u.w = (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[7]))) << 16) |
        __bfloat16_as_ushort(__float2bfloat16_rn(v[6]));
  return u;
}

constexpr long kWaitLimit = 1L << 26;  // polls before an mbarrier wait gives up

// Tensor-core inference: y[n][3] = MLP(x[n][35]). One CTA of 128 threads per
// SM walks 128-row tiles. status[0] is set to 1 if a wait times out.
__global__ void __launch_bounds__(128, 1)
mlp_forward_tc_kernel(const unsigned char* __restrict__ img, const float* __restrict__ x, long n,
                      float* __restrict__ y, int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* w_img = sm;
  unsigned char* act = sm + kImgBytes;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kImgBytes + kActBytes);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kImgBytes + kActBytes + 16);
  const int tid = threadIdx.x, warp = tid >> 5;

  // weights + biases -> smem (16-byte copies)
  for (uint32_t o = tid * 16; o < kImgBytes; o += 128 * 16)
    *reinterpret_cast<uint4*>(w_img + o) = *reinterpret_cast<const uint4*>(img + o);
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(128));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  const float* bias = reinterpret_cast<const float*>(w_img + kImgBias);
  const uint32_t a_base = smem_u32(act), w_base = smem_u32(w_img);
  const uint32_t mbar_a = smem_u32(mbar);
  uint32_t phase = 0;
  bool failed = false;
  const long tiles = (n + 127) / 128;

  auto run_layer = [&](uint32_t w_off, int k_steps, int n_out, int w_rows) -> bool {
    // operands written by all threads are complete and visible to the async proxy
    fence_proxy_async();
    fence_before();
    __syncthreads();
    if (tid == 0) {
      fence_after();
      const uint32_t idesc = make_idesc(n_out);
      for (int s = 0; s < k_steps; ++s) {
        const uint64_t ad = make_sdesc(a_base + s * 128 * 32);
        const uint64_t bd = make_sdesc(w_base + w_off + s * w_rows * 32);
        mma_bf16(tmem, ad, bd, idesc, s > 0);
      }
      mma_commit(mbar_a);
    }
    long spins = 0;
    bool ok = true;
    while (!mbar_try_wait(mbar_a, phase)) {
      if (++spins > kWaitLimit) {
        ok = false;
        break;
      }
    }
    phase ^= 1u;
    fence_after();
    return __syncthreads_and(ok) != 0;  // every thread takes the same decision
  };

  for (long tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x) {
    const long row = tile * 128 + tid;
    // ---- features -> BF16 operand (K padded to 48 with zeros)
    {
      float f[kMlpInPad];
#pragma unroll
      for (int k = 0; k < kMlpInPad; ++k) f[k] = 0.f;
      if (row < n)
        for (int k = 0; k < kMlpIn; ++k) f[k] = x[row * kMlpIn + k];
#pragma unroll
      for (int c = 0; c < kMlpInPad / 8; ++c)
        *reinterpret_cast<uint4*>(act + op_offset(tid, c * 8, 128)) = pack8(f + c * 8);
    }
    // ---- three hidden layers
    const uint32_t w_offs[3] = {kImgW1, kImgW2, kImgW3};
    const int ksteps[3] = {kMlpInPad / 16, kMlpHidden / 16, kMlpHidden / 16};
    for (int l = 0; l < 3 && !failed; ++l) {
      if (!run_layer(w_offs[l], ksteps[l], kMlpHidden, kMlpHidden)) {
        failed = true;
        break;
      }
      const float* b = bias + l * kMlpHidden;
      for (int c0 = 0; c0 < kMlpHidden; c0 += 32) {
        float v[32];
        tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + c0, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = gelu(v[i] + b[c0 + i]);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(act + op_offset(tid, c0 + c * 8, 128)) = pack8(v + c * 8);
      }
    }
    if (failed) break;
    // ---- output layer (N = 16, first 3 used)
    if (!run_layer(kImgW4, kMlpHidden / 16, kMlpOutPad, kMlpOutPad)) {
      failed = true;
      break;
    }
    {
      float v[16];
      tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16), v);
      const float* b = bias + 3 * kMlpHidden;
      if (row < n)
        for (int o = 0; o < kMlpOut; ++o) y[row * kMlpOut + o] = v[o] + b[o];
    }
  }
  if (failed && tid == 0) atomicExch(status, 1);
  fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128));
}

// Packs FP32 masters into the BF16 shared-memory image + FP32 biases.
__global__ void mlp_pack_kernel(const float* __restrict__ p, unsigned char* __restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  auto put = [&](uint32_t base, int rows, int r, int k, float v) {
    *reinterpret_cast<__nv_bfloat16*>(img + base + op_offset(r, k, rows)) = __float2bfloat16_rn(v);
  };
  if (i < kMlpHidden * kMlpInPad) {  // W1 (K padded)
    const int r = i / kMlpInPad, k = i % kMlpInPad;
    put(kImgW1, kMlpHidden, r, k, k < kMlpIn ? p[kOffW1 + r * kMlpIn + k] : 0.f);
  }
  if (i < kMlpHidden * kMlpHidden) {
    const int r = i / kMlpHidden, k = i % kMlpHidden;
    put(kImgW2, kMlpHidden, r, k, p[kOffW2 + i]);
    put(kImgW3, kMlpHidden, r, k, p[kOffW3 + i]);
  }
  if (i < kMlpOutPad * kMlpHidden) {  // W4 (N padded)
    const int r = i / kMlpHidden, k = i % kMlpHidden;
    put(kImgW4, kMlpOutPad, r, k, r < kMlpOut ? p[kOffW4 + r * kMlpHidden + k] : 0.f);
  }
  float* bias = reinterpret_cast<float*>(img + kImgBias);
  if (i < kMlpHidden) {
    bias[i] = p[kOffB1 + i];
    bias[kMlpHidden + i] = p[kOffB2 + i];
    bias[2 * kMlpHidden + i] = p[kOffB3 + i];
  }
  if (i < kMlpOutPad) bias[3 * kMlpHidden + i] = i < kMlpOut ? p[kOffB4 + i] : 0.f;
}

// ---------------------------------------------------------------- training (FP32)
// BF16 weights for training, [contraction index][output]: W1..W3 transposed
// for the forward pass, W4 as it is (its rows are its three outputs), then W3
// and W2 as they are for the backward pass.
constexpr int kTrW1 = 0;                                     // [35][128]
constexpr int kTrW2 = kTrW1 + kMlpIn * kMlpHidden;           // [128][128]
constexpr int kTrW3 = kTrW2 + kMlpHidden * kMlpHidden;
constexpr int kTrW4 = kTrW3 + kMlpHidden * kMlpHidden;       // [3][128]
constexpr int kTrFwd = kTrW4 + kMlpOut * kMlpHidden;         // elements the forward pass stages
constexpr int kTrBack = kTrFwd;                              // W3, W2 [out][in]
constexpr int kTrElems = kTrBack + 2 * kMlpHidden * kMlpHidden;
static_assert(kTrW2 % 8 == 0 && kTrFwd % 8 == 0 && kTrElems % 8 == 0, "16-byte staging copies");

// Parameter i of the flat master vector into the training image (biases are
// read from the masters).
__device__ __forceinline__ void train_image_put(int i, float v, __nv_bfloat16* __restrict__ img) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  if (i < kOffB1) {
    img[kTrW1 + (i % kMlpIn) * kMlpHidden + i / kMlpIn] = b;
  } else if (i >= kOffW2 && i < kOffB2) {
    const int e = i - kOffW2, o = e / kMlpHidden, k = e % kMlpHidden;
    img[kTrW2 + k * kMlpHidden + o] = b;
    img[kTrBack + kMlpHidden * kMlpHidden + e] = b;
  } else if (i >= kOffW3 && i < kOffB3) {
    const int e = i - kOffW3, o = e / kMlpHidden, k = e % kMlpHidden;
    img[kTrW3 + k * kMlpHidden + o] = b;
    img[kTrBack + e] = b;
  } else if (i >= kOffW4 && i < kOffB4) {
    img[kTrW4 + i - kOffW4] = b;
  }
}

__global__ void mlp_train_pack_kernel(const float* __restrict__ p, __nv_bfloat16* __restrict__ img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kMlpParams) train_image_put(i, p[i], img);
}

// Forward, loss, backward and weight gradients of tiles of T samples, one
// tile per CTA (more tiles than SMs: a CTA walks them and adds to its own
// partial gradient). Everything of a tile lives in shared memory: activations
// h1-h3, the GELU derivatives (turned into the layer gradients dz in place)
// and the inputs, stored [unit][sample] with a row pitch of T + 4 floats, so
// that 16-byte reads of eight different rows or of eight sample groups touch
// 32 distinct banks; the weights as BF16 (exact: they are used rounded to
// BF16), re-staged in the other orientation for the backward pass.
//   layer products   a thread computes 4 samples x T/8 outputs, the
//                    contraction in ascending order as one FMA chain
//   weight gradients a thread owns 8 x 8 of the 128 x 128 (rows 16 apart),
//                    summed over the tile's samples in order
// A CTA writes its gradient to part[blockIdx.x]; mlp_update_kernel adds the
// CTAs' parts in order, so a step is deterministic.
// The previous form ran one thread per gradient element over the whole batch
// (64 CTAs of a 4,096-long serial chain per layer: 5.2 ms of the 5.8 ms that
// the step's kernels took one by one, 3.4 ms a step overlapped). A
// 4,096-sample step is 2 x 3 x 37,632 x 4,096 flop (0.92 GFLOP, 13 us at the
// FP32 rate); it takes 54 us with the update, bound by the latency of the
// layers' chains at 8 warps per SM.
constexpr int kBpThreads = 256;
template <int T>
struct BpSmem {
  static constexpr int kPitch = T + 4;
  static constexpr int kRow = kMlpHidden * kPitch;  // one [128][pitch] array
  static constexpr int kX = 6 * kRow;               // inputs [35][pitch]
  static constexpr int kDy = kX + kMlpIn * kPitch;  // dY [3][pitch]
  static constexpr int kRed = kDy + kMlpOut * kPitch;  // reduction words
  static constexpr int kFloats = kRed + 8;
  static constexpr size_t kBytes = kFloats * sizeof(float) + kTrFwd * sizeof(__nv_bfloat16);
  static_assert(kFloats % 4 == 0 && kBytes <= 227 * 1024, "training tile shared memory");
};

// acc[j][c] = sum_r in[r][4 sg + c] * w[r][out0 + j] over the rows r in order
template <int T, int kOutPer>
__device__ __forceinline__ void bp_product(const float* __restrict__ in, const __nv_bfloat16* __restrict__ w, int rows,
                                           int sg, int out0, float (&acc)[kOutPer][4]) {
  constexpr int kPitch = T + 4;
#pragma unroll
  for (int j = 0; j < kOutPer; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.f;
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    const float4 x = *reinterpret_cast<const float4*>(in + r * kPitch + 4 * sg);
    float wv[kOutPer];
    if constexpr (kOutPer == 4) {
      const uint2 u = *reinterpret_cast<const uint2*>(w + r * kMlpHidden + out0);
      wv[0] = __uint_as_float(u.x << 16);
      wv[1] = __uint_as_float(u.x & 0xffff0000u);
      wv[2] = __uint_as_float(u.y << 16);
      wv[3] = __uint_as_float(u.y & 0xffff0000u);
    } else if constexpr (kOutPer == 2) {
      const uint32_t u = *reinterpret_cast<const uint32_t*>(w + r * kMlpHidden + out0);
      wv[0] = __uint_as_float(u << 16);
      wv[1] = __uint_as_float(u & 0xffff0000u);
    } else {
#pragma unroll
      for (int j = 0; j < kOutPer; ++j) wv[j] = __bfloat162float(w[r * kMlpHidden + out0 + j]);
    }
#pragma unroll
    for (int j = 0; j < kOutPer; ++j) {
      acc[j][0] = fmaf(wv[j], x.x, acc[j][0]);
      acc[j][1] = fmaf(wv[j], x.y, acc[j][1]);
      acc[j][2] = fmaf(wv[j], x.z, acc[j][2]);
      acc[j][3] = fmaf(wv[j], x.w, acc[j][3]);
    }
  }
}

// g[w_off + o * in + k] (+)= sum_s dz[o][s] h[k][s] for the 128 x kIn matrix,
// g[b_off + o] (+)= sum_s dz[o][s]
template <int T, int kIn>
__device__ __forceinline__ void bp_weight_grad(const float* __restrict__ dz, const float* __restrict__ h, int w_off,
                                               int b_off, bool add, float* __restrict__ g) {
  constexpr int kPitch = T + 4, kJ = (kIn + 15) / 16;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[8][kJ];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < kJ; ++j) acc[i][j] = 0.f;
#pragma unroll 1
  for (int s = 0; s < T; s += 4) {
    float4 a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4*>(dz + (ty + 16 * i) * kPitch + s);
#pragma unroll
    for (int j = 0; j < kJ; ++j) {
      const int k = tx + 16 * j;
      const float4 b = k < kIn ? *reinterpret_cast<const float4*>(h + k * kPitch + s) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
        acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
        acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < kJ; ++j) {
      const int k = tx + 16 * j;
      if (k >= kIn) continue;
      float* dst = g + w_off + (ty + 16 * i) * kIn + k;
      *dst = add ? *dst + acc[i][j] : acc[i][j];
    }
  if (threadIdx.x < kMlpHidden) {
    float b = 0.f;
    for (int s = 0; s < T; s += 4) {
      const float4 v = *reinterpret_cast<const float4*>(dz + threadIdx.x * kPitch + s);
      b += v.x;
      b += v.y;
      b += v.z;
      b += v.w;
    }
    float* dst = g + b_off + threadIdx.x;
    *dst = add ? *dst + b : b;
  }
}

// loss_part[block] = sum over its samples and outputs of (y - target)^2;
// dY = 2 (y - target) / (3 batch); yhat (may be null) receives y.
template <int T>
__global__ void __launch_bounds__(kBpThreads, 1)
mlp_backprop_kernel(const float* __restrict__ p, const __nv_bfloat16* __restrict__ img, const float* __restrict__ xin,
                    const float* __restrict__ target, long batch, float* __restrict__ part,
                    float* __restrict__ loss_part, float* __restrict__ yhat) {
  using S = BpSmem<T>;
  constexpr int kPitch = S::kPitch, kSg = T / 4, kOutPer = kSg / 2;
  extern __shared__ __align__(16) float bp_smem[];
  float* h[3] = {bp_smem, bp_smem + S::kRow, bp_smem + 2 * S::kRow};
  float* dz[3] = {bp_smem + 3 * S::kRow, bp_smem + 4 * S::kRow, bp_smem + 5 * S::kRow};
  float* xs = bp_smem + S::kX;
  float* dy = bp_smem + S::kDy;
  __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(bp_smem + S::kFloats);
  const int tid = threadIdx.x, sg = tid % kSg, out0 = (tid / kSg) * kOutPer;
  float* g = part + static_cast<size_t>(blockIdx.x) * kMlpParams;
  const float dscale = static_cast<float>(batch * kMlpOut);
  const long tiles = (batch + T - 1) / T;
  float loss = 0.f;
  bool add = false;
  for (long tile = blockIdx.x; tile < tiles; tile += gridDim.x, add = true) {
    const long s0 = tile * T;
    const int ns = static_cast<int>(min(static_cast<long>(T), batch - s0));
    if (add) __syncthreads();  // the previous tile's gradients have read the arrays
    for (int e = tid; e < kTrFwd / 8; e += kBpThreads)
      reinterpret_cast<uint4*>(w)[e] = reinterpret_cast<const uint4*>(img)[e];
    for (int e = tid; e < T * kMlpIn; e += kBpThreads) {
      const int s = e / kMlpIn, k = e - s * kMlpIn;
      xs[k * kPitch + s] = s < ns ? xin[s0 * kMlpIn + e] : 0.f;
    }
    __syncthreads();
    // ---- forward: z = W in + b, h = gelu(z), dz = gelu'(z)
    const int w_off[3] = {kTrW1, kTrW2, kTrW3}, b_off[3] = {kOffB1, kOffB2, kOffB3};
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      float acc[kOutPer][4];
      bp_product<T, kOutPer>(l == 0 ? xs : h[l - 1], w + w_off[l], l == 0 ? kMlpIn : kMlpHidden, sg, out0, acc);
#pragma unroll
      for (int j = 0; j < kOutPer; ++j) {
        const float b = p[b_off[l] + out0 + j];
        float hv[4], gv[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float z = acc[j][c] + b;
          hv[c] = gelu(z);
          gv[c] = gelu_grad(z);
        }
        const int at = (out0 + j) * kPitch + 4 * sg;
        *reinterpret_cast<float4*>(h[l] + at) = make_float4(hv[0], hv[1], hv[2], hv[3]);
        *reinterpret_cast<float4*>(dz[l] + at) = make_float4(gv[0], gv[1], gv[2], gv[3]);
      }
      __syncthreads();
    }
    // ---- outputs, loss and dY (a thread per sample and output); the other
    // threads stage W3 and W2 for the backward pass over the forward copies
    if (tid < T * kMlpOut) {
      const int s = tid % T, o = tid / T;
      const __nv_bfloat16* w4 = w + kTrW4 + o * kMlpHidden;
      float acc = 0.f;
#pragma unroll 8
      for (int k = 0; k < kMlpHidden; ++k) acc = fmaf(__bfloat162float(w4[k]), h[2][k * kPitch + s], acc);
      acc += p[kOffB4 + o];
      float d = 0.f;
      if (s < ns) {
        const long at = (s0 + s) * kMlpOut + o;
        if (yhat) yhat[at] = acc;
        d = acc - target[at];
      }
      loss += d * d;
      dy[o * kPitch + s] = 2.f * d / dscale;
    } else {
      for (int e = tid - T * kMlpOut; e < 2 * kMlpHidden * kMlpHidden / 8; e += kBpThreads - T * kMlpOut)
        reinterpret_cast<uint4*>(w + kTrW2)[e] = reinterpret_cast<const uint4*>(img + kTrBack)[e];
    }
    __syncthreads();
    // ---- layer 4: dW4, db4, dz3 = (W4^T dY) gelu'(z3)
    for (int e = tid; e < kMlpOut * kMlpHidden + kMlpOut; e += kBpThreads) {
      const bool bias = e >= kMlpOut * kMlpHidden;
      const int o = bias ? e - kMlpOut * kMlpHidden : e / kMlpHidden, k = e % kMlpHidden;
      float acc = 0.f;
      for (int s = 0; s < T; ++s) acc = bias ? acc + dy[o * kPitch + s] : fmaf(dy[o * kPitch + s], h[2][k * kPitch + s], acc);
      float* dst = g + (bias ? kOffB4 + o : kOffW4 + e);
      *dst = add ? *dst + acc : acc;
    }
    for (int e = tid; e < kMlpHidden * kSg; e += kBpThreads) {
      const int k = e / kSg, c = 4 * (e % kSg);
      float4 v = *reinterpret_cast<float4*>(dz[2] + k * kPitch + c);
      float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int o = 0; o < kMlpOut; ++o) {
        const float wv = __bfloat162float(w[kTrW4 + o * kMlpHidden + k]);
        const float4 d = *reinterpret_cast<const float4*>(dy + o * kPitch + c);
        a[0] = fmaf(d.x, wv, a[0]);
        a[1] = fmaf(d.y, wv, a[1]);
        a[2] = fmaf(d.z, wv, a[2]);
        a[3] = fmaf(d.w, wv, a[3]);
      }
      *reinterpret_cast<float4*>(dz[2] + k * kPitch + c) = make_float4(a[0] * v.x, a[1] * v.y, a[2] * v.z, a[3] * v.w);
    }
    __syncthreads();
    // ---- layers 3 and 2: dz_(l-1) = (W_l^T dz_l) gelu'(z_(l-1)), dW_l, db_l
#pragma unroll
    for (int l = 2; l >= 1; --l) {
      float acc[kOutPer][4];
      bp_product<T, kOutPer>(dz[l], w + kTrW2 + (l == 2 ? 0 : kMlpHidden * kMlpHidden), kMlpHidden, sg, out0, acc);
#pragma unroll
      for (int j = 0; j < kOutPer; ++j) {
        float4* at = reinterpret_cast<float4*>(dz[l - 1] + (out0 + j) * kPitch + 4 * sg);
        const float4 v = *at;
        *at = make_float4(acc[j][0] * v.x, acc[j][1] * v.y, acc[j][2] * v.z, acc[j][3] * v.w);
      }
      bp_weight_grad<T, kMlpHidden>(dz[l], h[l - 1], l == 2 ? kOffW3 : kOffW2, l == 2 ? kOffB3 : kOffB2, add, g);
      __syncthreads();
    }
    bp_weight_grad<T, kMlpIn>(dz[0], xs, kOffW1, kOffB1, add, g);
  }
  // the block's loss: warp sums, then the warps in order
  for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  float* red = bp_smem + S::kRed;
  if ((tid & 31) == 0) red[tid >> 5] = loss;
  __syncthreads();
  if (tid == 0) {
    float l = 0.f;
    for (int k = 0; k < kBpThreads / 32; ++k) l += red[k];
    loss_part[blockIdx.x] = l;
  }
}

// The CTAs' gradients summed in order; with adam_m the Adam update of the
// masters and of their BF16 training image, else the gradient into grad.
__global__ void mlp_update_kernel(const float* __restrict__ part, int n_part, float* __restrict__ grad,
                                  float* __restrict__ p, float* __restrict__ adam_m, float* __restrict__ adam_v,
                                  __nv_bfloat16* __restrict__ img, float lr, float b1, float b2, float eps, float c1,
                                  float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMlpParams) return;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  int k = 0;
#pragma unroll 2
  for (; k + 4 <= n_part; k += 4)
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[u] += part[static_cast<size_t>(k + u) * kMlpParams + i];
  for (; k < n_part; ++k) acc[0] += part[static_cast<size_t>(k) * kMlpParams + i];
  const float gi = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  grad[i] = gi;
  if (adam_m == nullptr) return;
  const float mi = b1 * adam_m[i] + (1.f - b1) * gi;
  const float vi = b2 * adam_v[i] + (1.f - b2) * gi * gi;
  adam_m[i] = mi;
  adam_v[i] = vi;
  const float v = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = v;
  train_image_put(i, v, img);
}

__global__ void mlp_init_kernel(float* __restrict__ p, uint32_t seed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMlpParams) return;
  int fan_in = 0;
  bool bias = false;
  if (i < kOffB1) fan_in = kMlpIn;
  else if (i < kOffW2) bias = true;
  else if (i < kOffB2) fan_in = kMlpHidden;
  else if (i < kOffW3) bias = true;
  else if (i < kOffB3) fan_in = kMlpHidden;
  else if (i < kOffW4) bias = true;
  else if (i < kOffB4) fan_in = kMlpHidden;
  else bias = true;
  if (bias) {
    p[i] = 0.f;
    return;
  }
  const Philox4 w = philox4x32(seed, 0x3A71u, static_cast<uint32_t>(i), 0u, 0u, 0u);
  const float u = static_cast<float>(u01(w.w[0])) * 2.f - 1.f;  // U(-1, 1)
  p[i] = u * sqrtf(3.f / static_cast<float>(fan_in));           // variance 1 / fan_in
}

}  // namespace

// ---------------------------------------------------------------- host side
static int mlp_get(amk_ctx* c, Mlp** out) {
  if (!c->mlp) c->mlp = new Mlp();
  Mlp* m = c->mlp;
  if (!m->initialized) {
    const size_t pb = kMlpParams * sizeof(float);
    AMK_TRY(m->master.reserve(pb));
    AMK_TRY(m->grad.reserve(pb));
    AMK_TRY(m->adam_m.reserve(pb));
    AMK_TRY(m->adam_v.reserve(pb));
    AMK_TRY(m->packed.reserve(kImgBytes));
    AMK_TRY(m->train.reserve(kTrElems * sizeof(__nv_bfloat16)));
    AMK_TRY(m->status.reserve(16));
    AMK_CUDA_TRY(cudaMemsetAsync(m->adam_m.ptr, 0, pb, c->stream));
    AMK_CUDA_TRY(cudaMemsetAsync(m->adam_v.ptr, 0, pb, c->stream));
    AMK_CUDA_TRY(cudaMemsetAsync(m->packed.ptr, 0, kImgBytes, c->stream));
    mlp_init_kernel<<<(kMlpParams + 255) / 256, 256, 0, c->stream>>>(m->master.as<float>(), 12345u);
    AMK_TRY(check_launch(c, "mlp_init_kernel"));
    m->initialized = true;
    m->packed_valid = m->train_valid = false;
  }
  *out = m;
  return AMK_OK;
}

static int mlp_pack(amk_ctx* c, Mlp* m) {
  if (m->packed_valid) return AMK_OK;
  mlp_pack_kernel<<<(kMlpHidden * kMlpHidden + 255) / 256, 256, 0, c->stream>>>(m->master.as<float>(),
                                                                                 m->packed.as<unsigned char>());
  AMK_TRY(check_launch(c, "mlp_pack_kernel"));
  m->packed_valid = true;
  return AMK_OK;
}

// Device-side inference on device buffers (used by the learned FMM).
int mlp_forward_device(amk_ctx* c, const float* x, long n, float* y) {
  if (n <= 0) return AMK_OK;
  Mlp* m = nullptr;
  AMK_TRY(mlp_get(c, &m));
  AMK_TRY(mlp_pack(c, m));
  static bool attr_set = false;
  if (!attr_set) {
    AMK_CUDA_TRY(cudaFuncSetAttribute(mlp_forward_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kSmemBytes)));
    attr_set = true;
  }
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);
  const long tiles = (n + 127) / 128;
  const int grid = static_cast<int>(std::min<long>(tiles, sms));
  AMK_CUDA_TRY(cudaMemsetAsync(m->status.ptr, 0, sizeof(int), c->stream));
  AMK_TRY(phase_begin(c, AMK_PHASE_MLP));
  mlp_forward_tc_kernel<<<grid, 128, kSmemBytes, c->stream>>>(m->packed.as<unsigned char>(), x, n, y,
                                                              m->status.as<int>());
  AMK_TRY(check_launch(c, "mlp_forward_tc_kernel"));
  AMK_TRY(phase_end(c, AMK_PHASE_MLP));
  return AMK_OK;
}

int mlp_check_status(amk_ctx* c) {
  if (!c->mlp) return AMK_OK;
  int st = 0;
  AMK_CUDA_TRY(cudaMemcpyAsync(&st, c->mlp->status.ptr, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  if (st) return fail(AMK_ERR_TIMEOUT, "tensor-core MLP: an mbarrier wait timed out");
  return AMK_OK;
}

// Samples per tile of mlp_backprop_kernel: a tile's time falls more slowly
// than its samples, so the tiles are made smaller only while all of them run
// at once. us per training step with tiles of 8 / 16 / 32 samples (148 SMs):
// batch 256 33.7 / 39.6 / 48.4, 1,184 38.8 / 43.9 / 50.0, 1,500 61.7 / 46.0 /
// 52.1, 2,368 62.7 / 47.1 / 52.2, 3,000 85.2 / 76.4 / 54.3, 4,096 108 / 77.4 /
// 54.3.
static int mlp_tile_rows(long batch, int sms) {
  if (batch > 16L * sms) return 32;
  return batch > 8L * sms ? 16 : 8;
}

// Forward, backward and (lr given) one Adam step on a device batch; the
// summed gradient is left in m->grad. loss_host and yhat_out may be null.
static int mlp_step_device(amk_ctx* c, const float* x, const float* target, long batch, const float* lr,
                           float* loss_host, float* yhat_out) {
  Mlp* m = nullptr;
  AMK_TRY(mlp_get(c, &m));
  if (!m->train_valid) {
    mlp_train_pack_kernel<<<(kMlpParams + 255) / 256, 256, 0, c->stream>>>(m->master.as<float>(),
                                                                           m->train.as<__nv_bfloat16>());
    AMK_TRY(check_launch(c, "mlp_train_pack_kernel"));
    m->train_valid = true;
  }
  int rc = AMK_OK, sms = 0;
  AMK_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
  const int rows = mlp_tile_rows(batch, sms);
  const int grid = static_cast<int>(std::min<long>((batch + rows - 1) / rows, sms));
  float* part = slot<float>(c, kSlotMlp0, static_cast<size_t>(grid) * kMlpParams, &rc);
  AMK_TRY(rc);
  float* lp = slot<float>(c, kSlotMlp1, std::max(256, grid), &rc);
  AMK_TRY(rc);
  auto launch = [&](auto kernel, size_t smem) -> int {
    AMK_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    kernel<<<grid, kBpThreads, smem, c->stream>>>(m->master.as<float>(), m->train.as<__nv_bfloat16>(), x, target,
                                                  batch, part, lp, yhat_out);
    return check_launch(c, "mlp_backprop_kernel");
  };
  if (rows == 32)
    AMK_TRY(launch(mlp_backprop_kernel<32>, BpSmem<32>::kBytes));
  else if (rows == 16)
    AMK_TRY(launch(mlp_backprop_kernel<16>, BpSmem<16>::kBytes));
  else
    AMK_TRY(launch(mlp_backprop_kernel<8>, BpSmem<8>::kBytes));
  const float b1 = 0.9f, b2 = 0.999f;
  float c1 = 1.f, c2 = 1.f;
  if (lr) {
    m->adam_step++;
    c1 = 1.f - std::pow(b1, static_cast<float>(m->adam_step));
    c2 = 1.f - std::pow(b2, static_cast<float>(m->adam_step));
    m->packed_valid = false;
  }
  mlp_update_kernel<<<(kMlpParams + 127) / 128, 128, 0, c->stream>>>(
      part, grid, m->grad.as<float>(), m->master.as<float>(), lr ? m->adam_m.as<float>() : nullptr,
      lr ? m->adam_v.as<float>() : nullptr, m->train.as<__nv_bfloat16>(), lr ? *lr : 0.f, b1, b2, 1e-8f, c1, c2);
  AMK_TRY(check_launch(c, "mlp_update_kernel"));
  if (loss_host) {
    std::vector<float> h(grid);
    AMK_CUDA_TRY(cudaMemcpyAsync(h.data(), lp, grid * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
    AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
    double s = 0.0;
    for (float v : h) s += v;
    *loss_host = static_cast<float>(s / static_cast<double>(batch * kMlpOut));
  }
  return AMK_OK;
}

// Minibatch Adam over a device dataset: batches are consecutive windows of
// the data (wrapping), so a run is deterministic.
int mlp_train_device(amk_ctx* c, const float* x, const float* target, long n, int steps, long batch, float lr,
                     float* final_loss) {
  batch = std::min(batch, n);
  float loss = 0.f;
  for (int s = 0; s < steps; ++s) {
    const long start = (static_cast<long>(s) * batch) % std::max(1L, n - batch + 1);
    const bool last = s + 1 == steps;
    AMK_TRY(mlp_step_device(c, x + start * kMlpIn, target + start * kMlpOut, batch, &lr, last ? &loss : nullptr,
                            nullptr));
  }
  if (final_loss) *final_loss = loss;
  return AMK_OK;
}

}  // namespace amk

using namespace amk;

void mlp_destroy(amk_ctx* c) {
  delete c->mlp;
  c->mlp = nullptr;
}

extern "C" int amk_mlp_num_params(void) { return kMlpParams; }

extern "C" int amk_mlp_set_params(amk_ctx* c, const float* params, long n) {
  if (!c || !params || n != kMlpParams) return fail(AMK_ERR_INVALID, "amk_mlp_set_params: expected %d floats", kMlpParams);
  Mlp* m = nullptr;
  AMK_TRY(mlp_get(c, &m));
  AMK_CUDA_TRY(cudaMemcpyAsync(m->master.ptr, params, kMlpParams * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  AMK_CUDA_TRY(cudaMemsetAsync(m->adam_m.ptr, 0, kMlpParams * sizeof(float), c->stream));
  AMK_CUDA_TRY(cudaMemsetAsync(m->adam_v.ptr, 0, kMlpParams * sizeof(float), c->stream));
  m->adam_step = 0;
  m->packed_valid = m->train_valid = false;
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return AMK_OK;
}

extern "C" int amk_mlp_get_params(amk_ctx* c, float* params, long n) {
  if (!c || !params || n != kMlpParams) return fail(AMK_ERR_INVALID, "amk_mlp_get_params: expected %d floats", kMlpParams);
  Mlp* m = nullptr;
  AMK_TRY(mlp_get(c, &m));
  AMK_CUDA_TRY(cudaMemcpyAsync(params, m->master.ptr, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return AMK_OK;
}

extern "C" int amk_mlp_forward(amk_ctx* c, const float* x, long n, float* y) {
  if (!c || n < 0 || (n > 0 && (!x || !y))) return fail(AMK_ERR_INVALID, "amk_mlp_forward: bad argument");
  if (n == 0) return AMK_OK;
  int rc = AMK_OK;
  float* dx = slot<float>(c, kSlotMlp2, static_cast<size_t>(n) * kMlpIn, &rc);
  AMK_TRY(rc);
  float* dy = slot<float>(c, kSlotMlp3, static_cast<size_t>(n) * kMlpOut, &rc);
  AMK_TRY(rc);
  AMK_CUDA_TRY(cudaMemcpyAsync(dx, x, n * kMlpIn * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  AMK_TRY(mlp_forward_device(c, dx, n, dy));
  AMK_TRY(mlp_check_status(c));
  AMK_CUDA_TRY(cudaMemcpyAsync(y, dy, n * kMlpOut * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return AMK_OK;
}

extern "C" int amk_mlp_gradients(amk_ctx* c, const float* x, const float* target, long n, float* grad,
                                 float* loss, float* yhat) {
  if (!c || n <= 0 || !x || !target) return fail(AMK_ERR_INVALID, "amk_mlp_gradients: bad argument");
  int rc = AMK_OK;
  float* dx = slot<float>(c, kSlotMlp2, static_cast<size_t>(n) * kMlpIn, &rc);
  AMK_TRY(rc);
  float* dt = slot<float>(c, kSlotMlp3, static_cast<size_t>(n) * kMlpOut, &rc);
  AMK_TRY(rc);
  float* dyh = slot<float>(c, kSlotMlp4, static_cast<size_t>(n) * kMlpOut, &rc);
  AMK_TRY(rc);
  AMK_CUDA_TRY(cudaMemcpyAsync(dx, x, n * kMlpIn * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(dt, target, n * kMlpOut * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  float l = 0.f;
  AMK_TRY(mlp_step_device(c, dx, dt, n, nullptr, &l, dyh));
  if (loss) *loss = l;
  if (grad)
    AMK_CUDA_TRY(cudaMemcpyAsync(grad, c->mlp->grad.ptr, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  if (yhat) AMK_CUDA_TRY(cudaMemcpyAsync(yhat, dyh, n * kMlpOut * sizeof(float), cudaMemcpyDeviceToHost, c->stream));
  AMK_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return AMK_OK;
}

extern "C" int amk_mlp_train(amk_ctx* c, const float* x, const float* target, long n, int steps, long batch,
                             float lr, float* final_loss) {
  if (!c || n <= 0 || !x || !target || steps < 0 || batch <= 0)
    return fail(AMK_ERR_INVALID, "amk_mlp_train: bad argument");
  int rc = AMK_OK;
  float* dx = slot<float>(c, kSlotMlp2, static_cast<size_t>(n) * kMlpIn, &rc);
  AMK_TRY(rc);
  float* dt = slot<float>(c, kSlotMlp3, static_cast<size_t>(n) * kMlpOut, &rc);
  AMK_TRY(rc);
  AMK_CUDA_TRY(cudaMemcpyAsync(dx, x, n * kMlpIn * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  AMK_CUDA_TRY(cudaMemcpyAsync(dt, target, n * kMlpOut * sizeof(float), cudaMemcpyHostToDevice, c->stream));
  return mlp_train_device(c, dx, dt, n, steps, batch, lr, final_loss);
}

