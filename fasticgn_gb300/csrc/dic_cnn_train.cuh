// The proposal network layer by layer: forward, loss and backward of a mini-batch (training,
// and dic_cnn_forward).  Every product is an mma.sync.m16n8k16 in BF16 with FP32 accumulation;
// activations and their gradients are BF16 in NHWC.
//
// The layers are small (32 channels; K = 18, 288, 288, 288, 128, 256), so what costs is moving
// operands: a generic GEMM that staged every operand element by element, with the im2col
// division per element, took 7.2 ms of kernels for 4096 samples (0.3 % of the tensor rate).
// Here each layer's geometry is a template argument and operands come straight as fragments:
//   forward, data gradients   A fragments by 4-byte loads of the NHWC rows (a k16 step is half
//                             of a pixel's channels: four lanes read 16 consecutive bytes), B
//                             fragments from shared memory in fragment order, filled once per
//                             CTA.  B's columns are permuted so that a thread ends with eight
//                             consecutive channels: one 16-byte store per output row.
//   data gradients            the stride-2 scatter by output parity: pixel (2 y + a, 2 x + b)
//                             has 1, 2, 2 or 4 taps, so 9 of the 36 (pixel, tap) products of a
//                             2 x 2 block exist and only those are formed.
//   weight gradients          K is the pixels: both operands transposed by ldmatrix.trans from
//                             shared memory (pixel pitch 80 B, conflict-free), one warp per tap
//                             with its 32 x 32 block in registers for all its samples, one FP32
//                             partial per CTA; k_reduce_parts adds the partials in a fixed order.
// The k16 steps of forward and data gradients run in the order k = (ky, kx, channel).
// 4096 samples: 14 kernels of 5-45 us, 0.27 ms in all; the call 7.3 -> 0.34 ms.  conv2's forward and
// data gradient (45 and 44 us) wait for those 4-byte loads (long-scoreboard stalls 53 and 15 cycles
// an issue; tensor pipe a fifth busy, shared-memory pipe 18 %).
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace dic
{
namespace cnn
{

constexpr int kTrainThreads = 256;
constexpr int kMaxParts = 152;      // CTAs (and FP32 partials) of a convolution's weight gradient
constexpr int kMlpParts = 64;       // the same for the two dense layers together
constexpr int kConvPart = 32 * 288 + 32, kConv1Part = 32 * 18 + 32;
constexpr int kMlpPart = kHidden * 128 + kHidden + kOut * kHidden + kOut;
// partial sums of one backward pass: conv1, conv2..4, the dense layers
constexpr size_t kPartConv1 = 0, kPartConv = kPartConv1 + (size_t)kMaxParts * kConv1Part;
constexpr size_t kPartMlp = kPartConv + 3 * (size_t)kMaxParts * kConvPart;
constexpr size_t kPartFloats = kPartMlp + (size_t)kMlpParts * kMlpPart;

// channel of column c (0..7) of n-tile j under the permutation that gives thread t of a
// fragment row the channels 8 t .. 8 t + 7 (columns 2 t, 2 t + 1 of the four n-tiles)
__device__ __forceinline__ int perm_channel(int j, int c) { return (c >> 1) * 8 + j * 2 + (c & 1); }

__device__ __forceinline__ uint32_t pack_relu(float a, float b)
{
  return pack_bf16(__float2bfloat16(fmaxf(a, 0.f)), __float2bfloat16(fmaxf(b, 0.f)));
}
// v where the BF16 activations packed in act are positive, else 0
__device__ __forceinline__ uint32_t pack_masked(float a, float b, uint32_t act)
{
  const float lo = __uint_as_float(act << 16), hi = __uint_as_float(act & 0xFFFF0000u);
  return pack_bf16(__float2bfloat16(lo > 0.f ? a : 0.f), __float2bfloat16(hi > 0.f ? b : 0.f));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// 16 bytes global -> shared, zeros where !on (the address must be readable only when on)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool on)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, bool on)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(on ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void cp_wait()
{
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kLeft) : "memory");
}

// --------------------------------------------------------------------------------------
// Forward convolutions.  Rows m = (sample, oy, ox); one warp per 16-row tile at a time.
// --------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kTrainThreads) k_conv1_fwd(const uint32_t* __restrict__ x0,
                                                             const __nv_bfloat16* __restrict__ wb,
                                                             const float* __restrict__ params,
                                                             __nv_bfloat16* __restrict__ out, int64_t n)
{
  // a tile is one output row of a sample: pixels (2 ox + kx - 1, 2 oy + ky - 1), ox = 0..15
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint32_t b[2][4][2];
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      const __nv_bfloat16* w = wb + WeightLayout::c1 + perm_channel(j, g) * kC1K + s * 16 + 2 * t;
      b[s][j][0] = *reinterpret_cast<const uint32_t*>(w);
      b[s][j][1] = *reinterpret_cast<const uint32_t*>(w + 8);
    }
  float bias[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) bias[c] = params[ParamLayout::b1 + 8 * t + c];
  const int64_t tiles = n * 16, step = (int64_t)gridDim.x * (kTrainThreads / 32);
  for (int64_t tile = (int64_t)blockIdx.x * (kTrainThreads / 32) + (threadIdx.x >> 5); tile < tiles; tile += step)
  {
    const int64_t i = tile >> 4;
    const int oy = (int)(tile & 15);
    const uint32_t* img = x0 + i * (kWin * kWin);
    const auto px = [&](int tap, int ox) -> uint32_t {
      const int iy = 2 * oy + tap / 3 - 1, ix = 2 * ox + tap % 3 - 1;
      return (iy >= 0 && ix >= 0 && iy < kWin && ix < kWin) ? __ldg(img + iy * kWin + ix) : 0u;
    };
    // k = 2 tap + channel: step 0 holds taps 0..7, step 1 tap 8 (weights past it are zero)
    uint32_t a0[4] = {px(t, g), px(t, g + 8), px(t + 4, g), px(t + 4, g + 8)};
    uint32_t a1[4] = {t == 0 ? px(8, g) : 0u, t == 0 ? px(8, g + 8) : 0u, 0u, 0u};
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
      mma_bf16_16816(acc[j], a0, b[0][j]);
      mma_bf16_16816(acc[j], a1, b[1][j]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
      uint4 v;
      v.x = pack_relu(acc[0][2 * h] + bias[0], acc[0][2 * h + 1] + bias[1]);
      v.y = pack_relu(acc[1][2 * h] + bias[2], acc[1][2 * h + 1] + bias[3]);
      v.z = pack_relu(acc[2][2 * h] + bias[4], acc[2][2 * h + 1] + bias[5]);
      v.w = pack_relu(acc[3][2 * h] + bias[6], acc[3][2 * h + 1] + bias[7]);
      *reinterpret_cast<uint4*>(out + (tile * 16 + g + 8 * h) * 32 + 8 * t) = v;
    }
  }
}

// the 32 channels of one pixel as a row's share of two k16 steps' A fragments: words t, t + 4
// (step 0) and t + 8, t + 12 (step 1)
struct PixelWords
{
  uint32_t w[4];
};
__device__ __forceinline__ PixelWords pixel_words(const __nv_bfloat16* p, int t, bool on)
{
  PixelWords r;
#pragma unroll
  for (int k = 0; k < 4; ++k) r.w[k] = on ? __ldg(reinterpret_cast<const uint32_t*>(p) + t + 4 * k) : 0u;
  return r;
}
// acc += rows (lo: rows 0..7, hi: rows 8..15) x the tap's two k16 steps of fragment-ordered B
__device__ __forceinline__ void mma_pixel(float (&acc)[4][4], const PixelWords& lo, const PixelWords& hi, const uint4* tap,
                                          int lane)
{
#pragma unroll
  for (int h = 0; h < 2; ++h)
  {
    const uint32_t a[4] = {lo.w[2 * h], hi.w[2 * h], lo.w[2 * h + 1], hi.w[2 * h + 1]};
    const uint4 p = tap[(2 * h) * 32 + lane], q = tap[(2 * h + 1) * 32 + lane];
    const uint32_t b0[2] = {p.x, p.y}, b1[2] = {p.z, p.w}, b2[2] = {q.x, q.y}, b3[2] = {q.z, q.w};
    mma_bf16_16816(acc[0], a, b0);
    mma_bf16_16816(acc[1], a, b1);
    mma_bf16_16816(acc[2], a, b2);
    mma_bf16_16816(acc[3], a, b3);
  }
}

template <int SO>
__global__ void __launch_bounds__(kTrainThreads) k_conv_fwd(const __nv_bfloat16* __restrict__ in,
                                                            const __nv_bfloat16* __restrict__ w,
                                                            const float* __restrict__ bias_p,
                                                            __nv_bfloat16* __restrict__ out, int64_t n)
{
  constexpr int SI = 2 * SO;
  __shared__ uint4 sb[9 * 4 * 32];   // [tap][half][n-tile pair][lane]
  for (int e = threadIdx.x; e < 9 * 4 * 32; e += kTrainThreads)
  {
    const int l = e & 31, jj = (e >> 5) & 1, h = (e >> 6) & 1, tap = e >> 7, g = l >> 2, t = l & 3;
    uint32_t v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      v[q] = *reinterpret_cast<const uint32_t*>(w + perm_channel(2 * jj + (q >> 1), g) * 288 + tap * 32 + h * 16 + 2 * t +
                                                (q & 1) * 8);
    sb[e] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float bias[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) bias[c] = bias_p[8 * t + c];
  const int64_t M = n * SO * SO, tiles = (M + 15) / 16, step = (int64_t)gridDim.x * (kTrainThreads / 32);
  for (int64_t tile = (int64_t)blockIdx.x * (kTrainThreads / 32) + (threadIdx.x >> 5); tile < tiles; tile += step)
  {
    const __nv_bfloat16* base[2];
    int oy[2], ox[2];
    bool live[2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
    {
      const int64_t m = tile * 16 + g + 8 * r;
      live[r] = m < M;
      const int64_t i = m / (SO * SO);
      const int p = (int)(m % (SO * SO));
      oy[r] = p / SO;
      ox[r] = p % SO;
      base[r] = in + ((i * SI + 2 * oy[r]) * SI + 2 * ox[r]) * 32;
    }
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
    {
      const int dy = tap / 3 - 1, dx = tap % 3 - 1;   // only the first row's and column's taps leave the image
      PixelWords a[2];
#pragma unroll
      for (int r = 0; r < 2; ++r)
        a[r] = pixel_words(base[r] + (dy * SI + dx) * 32, t, live[r] && oy[r] * 2 + dy >= 0 && ox[r] * 2 + dx >= 0);
      mma_pixel(acc, a[0], a[1], sb + tap * 128, lane);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (live[r])
      {
        uint4 v;
        v.x = pack_relu(acc[0][2 * r] + bias[0], acc[0][2 * r + 1] + bias[1]);
        v.y = pack_relu(acc[1][2 * r] + bias[2], acc[1][2 * r + 1] + bias[3]);
        v.z = pack_relu(acc[2][2 * r] + bias[4], acc[2][2 * r + 1] + bias[5]);
        v.w = pack_relu(acc[3][2 * r] + bias[6], acc[3][2 * r + 1] + bias[7]);
        *reinterpret_cast<uint4*>(out + (tile * 16 + g + 8 * r) * 32 + 8 * t) = v;
      }
  }
}

// --------------------------------------------------------------------------------------
// Data gradient of a convolution with output side SO: a tile is 16 positions (sample, y, x) of
// the SO x SO grid, whose 2 x 2 input pixels (2 y + a, 2 x + b) read dz at (y, x), (y, x + 1),
// (y + 1, x), (y + 1, x + 1): tap ky = 1 for a = 0; ky = 0 (from y + 1), then ky = 2 (from y)
// for a = 1; kx likewise.  Masked by the input activation (ReLU) and stored BF16.
// --------------------------------------------------------------------------------------
template <int SO>
__global__ void __launch_bounds__(kTrainThreads) k_conv_dgrad(const __nv_bfloat16* __restrict__ dz,
                                                              const __nv_bfloat16* __restrict__ w,
                                                              const __nv_bfloat16* __restrict__ act,
                                                              __nv_bfloat16* __restrict__ dzin, int64_t n)
{
  constexpr int SI = 2 * SO;
  __shared__ uint4 sb[9 * 4 * 32];   // [tap][half of co][n-tile pair][lane]
  for (int e = threadIdx.x; e < 9 * 4 * 32; e += kTrainThreads)
  {
    const int l = e & 31, jj = (e >> 5) & 1, h = (e >> 6) & 1, tap = e >> 7, g = l >> 2, t = l & 3;
    uint32_t v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
      const __nv_bfloat16* p = w + (h * 16 + 2 * t + (q & 1) * 8) * 288 + tap * 32 + perm_channel(2 * jj + (q >> 1), g);
      v[q] = pack_bf16(p[0], p[288]);
    }
    sb[e] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int64_t M = n * SO * SO, tiles = (M + 15) / 16, step = (int64_t)gridDim.x * (kTrainThreads / 32);
  for (int64_t tile = (int64_t)blockIdx.x * (kTrainThreads / 32) + (threadIdx.x >> 5); tile < tiles; tile += step)
  {
    PixelWords a[2][2][2];   // [row half][y + dy][x + dx]
    int64_t o[2];
    bool live[2];
#pragma unroll
    for (int r = 0; r < 2; ++r)
    {
      const int64_t m = tile * 16 + g + 8 * r;
      live[r] = m < M;
      const int64_t i = m / (SO * SO);
      const int p = (int)(m % (SO * SO)), y = p / SO, x = p % SO;
      o[r] = ((i * SI + 2 * y) * SI + 2 * x) * 32 + 8 * t;
#pragma unroll
      for (int dy = 0; dy < 2; ++dy)
#pragma unroll
        for (int dx = 0; dx < 2; ++dx)
          a[r][dy][dx] = pixel_words(dz + (m + dy * SO + dx) * 32, t, live[r] && y + dy < SO && x + dx < SO);
    }
#pragma unroll
    for (int cls = 0; cls < 4; ++cls)
    {
      const int py = cls >> 1, pxl = cls & 1;
      float acc[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
      for (int sy = 0; sy <= py; ++sy)
#pragma unroll
        for (int sx = 0; sx <= pxl; ++sx)
        {
          const int ky = py ? 2 * sy : 1, kx = pxl ? 2 * sx : 1;
          const int dy = py ? 1 - sy : 0, dx = pxl ? 1 - sx : 0;
          mma_pixel(acc, a[0][dy][dx], a[1][dy][dx], sb + (ky * 3 + kx) * 128, lane);
        }
#pragma unroll
      for (int r = 0; r < 2; ++r)
        if (live[r])
        {
          const int64_t q = o[r] + (py * SI + pxl) * 32;
          const uint4 m = __ldg(reinterpret_cast<const uint4*>(act + q));
          uint4 v;
          v.x = pack_masked(acc[0][2 * r], acc[0][2 * r + 1], m.x);
          v.y = pack_masked(acc[1][2 * r], acc[1][2 * r + 1], m.y);
          v.z = pack_masked(acc[2][2 * r], acc[2][2 * r + 1], m.z);
          v.w = pack_masked(acc[3][2 * r], acc[3][2 * r + 1], m.w);
          *reinterpret_cast<uint4*>(dzin + q) = v;
        }
    }
  }
}

// --------------------------------------------------------------------------------------
// Dense layers of 16 samples per CTA: f1, f2 and, with a target, the loss gradient and the two
// data gradients.  W5 sits in shared memory once for both directions (rows padded to 272 B:
// fragment loads and ldmatrix rows fall in distinct banks).
// --------------------------------------------------------------------------------------
constexpr int kW5Row = 128 + 8, kMlpA4Row = 128 + 8, kMlpA5Row = 256 + 8;
struct MlpSmem
{
  __nv_bfloat16 w5[kHidden * kW5Row];
  __nv_bfloat16 a4[16 * kMlpA4Row];
  __nv_bfloat16 a5[16 * kMlpA5Row];
  __nv_bfloat16 d5[16 * kMlpA5Row];
  __nv_bfloat16 dout[16 * 16];   // columns 8..15 zero
  float out[16 * 8];
};

__global__ void __launch_bounds__(kTrainThreads) k_mlp(const __nv_bfloat16* __restrict__ a4, const __nv_bfloat16* __restrict__ wb,
                                                       const float* __restrict__ params, const float* __restrict__ target,
                                                       int64_t n, __nv_bfloat16* __restrict__ a5, float* __restrict__ out,
                                                       __nv_bfloat16* __restrict__ dout, float* __restrict__ row_loss,
                                                       __nv_bfloat16* __restrict__ d5, __nv_bfloat16* __restrict__ d4)
{
  extern __shared__ __align__(16) unsigned char mlp_raw[];
  MlpSmem& S = *reinterpret_cast<MlpSmem*>(mlp_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  using L = WeightLayout;
  using P = ParamLayout;
  for (int e = tid; e < kHidden * 16; e += kTrainThreads)
    *reinterpret_cast<uint4*>(S.w5 + (e >> 4) * kW5Row + (e & 15) * 8) =
        __ldg(reinterpret_cast<const uint4*>(wb + L::f1) + e);
  S.dout[tid] = bz();
  const int64_t tiles = (n + 15) / 16;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x)
  {
    const int64_t m0 = tile * 16;
    {
      const int r = tid >> 4, c = tid & 15;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (m0 + r < n) v = __ldg(reinterpret_cast<const uint4*>(a4 + (m0 + r) * 128) + c);
      *reinterpret_cast<uint4*>(S.a4 + r * kMlpA4Row + c * 8) = v;
    }
    __syncthreads();
    // f1: warp takes columns 32 warp .. + 31
    {
      float acc[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
      for (int s = 0; s < 8; ++s)
      {
        const __nv_bfloat16* ar = S.a4 + g * kMlpA4Row + s * 16 + 2 * t;
        const uint32_t a[4] = {*reinterpret_cast<const uint32_t*>(ar), *reinterpret_cast<const uint32_t*>(ar + 8 * kMlpA4Row),
                               *reinterpret_cast<const uint32_t*>(ar + 8),
                               *reinterpret_cast<const uint32_t*>(ar + 8 * kMlpA4Row + 8)};
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
          const __nv_bfloat16* br = S.w5 + (warp * 32 + j * 8 + g) * kW5Row + s * 16 + 2 * t;
          const uint32_t b[2] = {*reinterpret_cast<const uint32_t*>(br), *reinterpret_cast<const uint32_t*>(br + 8)};
          mma_bf16_16816(acc[j], a, b);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const int c = warp * 32 + j * 8 + 2 * t;
        const float b0 = params[P::b5 + c], b1 = params[P::b5 + c + 1];
#pragma unroll
        for (int r = 0; r < 2; ++r)
          *reinterpret_cast<uint32_t*>(S.a5 + (g + 8 * r) * kMlpA5Row + c) = pack_relu(acc[j][2 * r] + b0, acc[j][2 * r + 1] + b1);
      }
    }
    __syncthreads();
    for (int e = tid; e < 16 * 32; e += kTrainThreads)
      if (m0 + (e >> 5) < n)
        *reinterpret_cast<uint4*>(a5 + (m0 + (e >> 5)) * kHidden + (e & 31) * 8) =
            *reinterpret_cast<const uint4*>(S.a5 + (e >> 5) * kMlpA5Row + (e & 31) * 8);
    // f2 (8 columns, k in order on one warp), then the loss and dL/dout
    if (warp == 0)
    {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int s = 0; s < 16; ++s)
      {
        const __nv_bfloat16* ar = S.a5 + g * kMlpA5Row + s * 16 + 2 * t;
        const uint32_t a[4] = {*reinterpret_cast<const uint32_t*>(ar), *reinterpret_cast<const uint32_t*>(ar + 8 * kMlpA5Row),
                               *reinterpret_cast<const uint32_t*>(ar + 8),
                               *reinterpret_cast<const uint32_t*>(ar + 8 * kMlpA5Row + 8)};
        const __nv_bfloat16* br = wb + L::f2 + g * kHidden + s * 16 + 2 * t;
        const uint32_t b[2] = {__ldg(reinterpret_cast<const uint32_t*>(br)), __ldg(reinterpret_cast<const uint32_t*>(br + 8))};
        mma_bf16_16816(acc, a, b);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
      {
        const int r = g + 8 * (e >> 1), c = 2 * t + (e & 1);
        const float z = acc[e] + (c < kOut ? params[P::b6 + c] : 0.f);
        S.out[r * 8 + c] = z;
        if (c < kOut && m0 + r < n) out[(m0 + r) * kOutPad + c] = z;
      }
      __syncwarp();
      if (target && lane < 16 && m0 + lane < n)
      {
        const int64_t m = m0 + lane;
        const float scale = 2.f / (float)(n * kOut);
        float l = 0.f;
#pragma unroll
        for (int j = 0; j < kOutPad; ++j)
        {
          float gr = 0.f;
          if (j < kOut)
          {
            const float d = S.out[lane * 8 + j] - target[m * kOut + j] * out_scale(j);
            l += d * d;
            gr = d * scale;
          }
          const __nv_bfloat16 v = __float2bfloat16(gr);
          S.dout[lane * 16 + j] = v;
          dout[m * kOutPad + j] = v;
        }
        row_loss[m] = l;
      }
    }
    __syncthreads();
    if (target)
    {
      // d5 = dout x W6 (k = 6, one step), masked by a5
      const __nv_bfloat16* ar = S.dout + g * 16 + 2 * t;
      const uint32_t a[4] = {*reinterpret_cast<const uint32_t*>(ar), *reinterpret_cast<const uint32_t*>(ar + 8 * 16), 0u, 0u};
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const int nc = warp * 32 + j * 8 + g;
        const uint32_t b[2] = {t < kOut / 2 ? pack_bf16(wb[L::f2 + 2 * t * kHidden + nc], wb[L::f2 + (2 * t + 1) * kHidden + nc])
                                            : 0u,
                               0u};
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16_16816(acc, a, b);
        const int c = warp * 32 + j * 8 + 2 * t;
#pragma unroll
        for (int r = 0; r < 2; ++r)
        {
          const uint32_t m = *reinterpret_cast<const uint32_t*>(S.a5 + (g + 8 * r) * kMlpA5Row + c);
          *reinterpret_cast<uint32_t*>(S.d5 + (g + 8 * r) * kMlpA5Row + c) = pack_masked(acc[2 * r], acc[2 * r + 1], m);
        }
      }
      __syncthreads();
      for (int e = tid; e < 16 * 32; e += kTrainThreads)
        if (m0 + (e >> 5) < n)
          *reinterpret_cast<uint4*>(d5 + (m0 + (e >> 5)) * kHidden + (e & 31) * 8) =
              *reinterpret_cast<const uint4*>(S.d5 + (e >> 5) * kMlpA5Row + (e & 31) * 8);
      // d4 = d5 x W5 (k = 256): warp takes columns 16 warp .. + 15, masked by a4
      float acc[2][4];
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
      for (int s = 0; s < 16; ++s)
      {
        const __nv_bfloat16* dr = S.d5 + g * kMlpA5Row + s * 16 + 2 * t;
        const uint32_t da[4] = {*reinterpret_cast<const uint32_t*>(dr), *reinterpret_cast<const uint32_t*>(dr + 8 * kMlpA5Row),
                                *reinterpret_cast<const uint32_t*>(dr + 8),
                                *reinterpret_cast<const uint32_t*>(dr + 8 * kMlpA5Row + 8)};
        uint32_t b[4];
        ldsm_x4_trans(b, smem_u32(S.w5 + (s * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * kW5Row + warp * 16 + (lane >> 4) * 8));
        const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
        mma_bf16_16816(acc[0], da, b0);
        mma_bf16_16816(acc[1], da, b1);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 2; ++r)
        {
          const int c = warp * 16 + j * 8 + 2 * t;
          const uint32_t m = *reinterpret_cast<const uint32_t*>(S.a4 + (g + 8 * r) * kMlpA4Row + c);
          if (m0 + g + 8 * r < n)
            *reinterpret_cast<uint32_t*>(d4 + (m0 + g + 8 * r) * 128 + c) = pack_masked(acc[j][2 * r], acc[j][2 * r + 1], m);
        }
    }
    __syncthreads();   // the tile's buffers are free
  }
}

// --------------------------------------------------------------------------------------
// Weight gradients.  64 output pixels are in flight per stage: one sample of conv2, four of conv3,
// sixteen of conv4; stages double-buffered with cp.async.  Warps 0..8 take one tap
// each, warp 9 the bias.
// --------------------------------------------------------------------------------------
constexpr int kWgradThreads = 320;
template <int SO>
struct WgradStage
{
  static constexpr int SI = 2 * SO, G = 64 / (SO * SO), SP = SI + 1;   // one zero row and column before the image
  __nv_bfloat16 in[G * SP * SP * kPix];
  __nv_bfloat16 dz[64 * kPix];
};

template <int SO>
__global__ void __launch_bounds__(kWgradThreads) k_conv_wgrad(const __nv_bfloat16* __restrict__ dz,
                                                              const __nv_bfloat16* __restrict__ in, float* __restrict__ part,
                                                              int64_t n)
{
  using Stage = WgradStage<SO>;
  constexpr int SI = Stage::SI, G = Stage::G, SP = Stage::SP;
  extern __shared__ __align__(16) unsigned char wgrad_raw[];
  Stage* st = reinterpret_cast<Stage*>(wgrad_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  for (size_t e = tid; e < 2 * sizeof(Stage) / 4; e += kWgradThreads) reinterpret_cast<uint32_t*>(wgrad_raw)[e] = 0u;
  __syncthreads();
  const int64_t groups = (n + G - 1) / G;
  const auto load = [&](Stage& s, int64_t grp) {
    const int64_t i0 = grp * G;
    for (int e = tid; e < 1024 + 256; e += kWgradThreads)
    {
      if (e < 1024)
      {
        const int p = e >> 2, k = p / (SI * SI), q = p % (SI * SI), y = q / SI, x = q % SI;
        const bool on = i0 + k < n;
        cp_async16(smem_u32(s.in + ((k * SP + y + 1) * SP + x + 1) * kPix + (e & 3) * 8),
                   in + (on ? (i0 * SI * SI + p) * 32 + (e & 3) * 8 : 0), on);
      }
      else
      {
        const int p = (e - 1024) >> 2;
        const bool on = i0 + p / (SO * SO) < n;
        cp_async16(smem_u32(s.dz + p * kPix + (e & 3) * 8), dz + (on ? (i0 * SO * SO + p) * 32 + (e & 3) * 8 : 0), on);
      }
    }
    cp_commit();
  };
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  float bsum = 0.f;
  const int ky = warp / 3, kx = warp % 3;
  int buf = 0;
  if ((int64_t)blockIdx.x < groups) load(st[0], blockIdx.x);
  for (int64_t grp = blockIdx.x; grp < groups; grp += gridDim.x)
  {
    if (grp + gridDim.x < groups)
    {
      load(st[buf ^ 1], grp + gridDim.x);
      cp_wait<1>();
    }
    else
      cp_wait<0>();
    __syncthreads();
    const Stage& s = st[buf];
    if (warp < 9)
    {
#pragma unroll
      for (int q = 0; q < 4; ++q)
      {
        // A = dz^T: matrices (k 0-7, co 0-7), (k 0-7, co 8-15), (k 8-15, co 0-7), (k 8-15, co 8-15)
        const __nv_bfloat16* ap = s.dz + (16 * q + (lane & 7) + (lane >> 4) * 8) * kPix + ((lane >> 3) & 1) * 8;
        uint32_t a[2][4];
        ldsm_x4_trans(a[0], smem_u32(ap));
        ldsm_x4_trans(a[1], smem_u32(ap + 16));
        // B = the tap's input pixels: (k 0-7, ci 0-7), (k 8-15, ci 0-7), (k 0-7, ci 8-15), (k 8-15, ci 8-15)
        const int p = 16 * q + (lane & 7) + ((lane >> 3) & 1) * 8;
        const int k = p / (SO * SO), y = (p % (SO * SO)) / SO, x = p % SO;
        const __nv_bfloat16* bp = s.in + ((k * SP + 2 * y + ky) * SP + 2 * x + kx) * kPix + (lane >> 4) * 8;
        uint32_t b[2][4];
        ldsm_x4_trans(b[0], smem_u32(bp));
        ldsm_x4_trans(b[1], smem_u32(bp + 16));
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
          {
            const uint32_t bb[2] = {b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]};
            mma_bf16_16816(acc[i][j], a[i], bb);
          }
      }
    }
    else
    {
#pragma unroll 8
      for (int p = 0; p < 64; ++p) bsum += __bfloat162float(s.dz[p * kPix + lane]);
    }
    __syncthreads();   // before this stage's buffer is loaded again
    buf ^= 1;
  }
  float* dst = part + (size_t)blockIdx.x * kConvPart;
  if (warp < 9)
  {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float2*>(dst + (i * 16 + g + 8 * h) * 288 + warp * 32 + j * 8 + 2 * t) =
              make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  }
  else
    dst[32 * 288 + lane] = bsum;
}

// conv1: K = 256 pixels a sample, N = 18 (tap, channel).  A k16 step is one output row; the
// eight warps take rows warp and warp + 8 and add their sums at the end.
struct Wgrad1Stage
{
  __nv_bfloat16 dz[256 * kPix];
  uint32_t x[33 * 33];   // one zero pixel around the window
  uint32_t pad[3];
};
__global__ void __launch_bounds__(kTrainThreads) k_conv1_wgrad(const __nv_bfloat16* __restrict__ dz,
                                                               const uint32_t* __restrict__ x0, float* __restrict__ part,
                                                               int64_t n)
{
  extern __shared__ __align__(16) unsigned char wgrad_raw[];
  Wgrad1Stage* st = reinterpret_cast<Wgrad1Stage*>(wgrad_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  for (size_t e = tid; e < 2 * sizeof(Wgrad1Stage) / 4; e += kTrainThreads) reinterpret_cast<uint32_t*>(wgrad_raw)[e] = 0u;
  __syncthreads();
  const auto load = [&](Wgrad1Stage& s, int64_t i) {
    for (int e = tid; e < 1024; e += kTrainThreads)
      cp_async16(smem_u32(s.dz + (e >> 2) * kPix + (e & 3) * 8), dz + (i * 256 + (e >> 2)) * 32 + (e & 3) * 8, true);
    for (int e = tid; e < kWin * kWin; e += kTrainThreads)
      cp_async4(smem_u32(s.x + (e / kWin + 1) * 33 + e % kWin + 1), x0 + i * (kWin * kWin) + e, true);
    cp_commit();
  };
  float acc[2][3][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  float bsum = 0.f;
  int buf = 0;
  if ((int64_t)blockIdx.x < n) load(st[0], blockIdx.x);
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x)
  {
    if (i + gridDim.x < n)
    {
      load(st[buf ^ 1], i + gridDim.x);
      cp_wait<1>();
    }
    else
      cp_wait<0>();
    __syncthreads();
    const Wgrad1Stage& s = st[buf];
#pragma unroll
    for (int half = 0; half < 2; ++half)
    {
      const int q = warp + 8 * half;
      const __nv_bfloat16* ap = s.dz + (16 * q + (lane & 7) + (lane >> 4) * 8) * kPix + ((lane >> 3) & 1) * 8;
      uint32_t a[2][4];
      ldsm_x4_trans(a[0], smem_u32(ap));
      ldsm_x4_trans(a[1], smem_u32(ap + 16));
#pragma unroll
      for (int j = 0; j < 3; ++j)
      {
        const int col = j * 8 + g, tap = col >> 1, c = col & 1;   // columns 18..23 are zero
        uint32_t b[2] = {0u, 0u};
        if (col < 18)
        {
          const uint16_t* xp = reinterpret_cast<const uint16_t*>(s.x + (2 * q + tap / 3) * 33 + tap % 3) + c;
          // pixels ox = 2 t, 2 t + 1 (and + 8): padded column 2 ox
          b[0] = (uint32_t)xp[8 * t] | ((uint32_t)xp[8 * t + 4] << 16);
          b[1] = (uint32_t)xp[8 * t + 32] | ((uint32_t)xp[8 * t + 36] << 16);
        }
        mma_bf16_16816(acc[0][j], a[0], b);
        mma_bf16_16816(acc[1][j], a[1], b);
      }
#pragma unroll
      for (int p = 0; p < 16; ++p) bsum += __bfloat162float(s.dz[(16 * q + p) * kPix + lane]);
    }
    __syncthreads();
    buf ^= 1;
  }
  // the warps' sums, added in warp order
  float* red = reinterpret_cast<float*>(wgrad_raw);   // [8][32][24], then [8][32]
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        red[(warp * 32 + i * 16 + g + 8 * (e >> 1)) * 24 + j * 8 + 2 * t + (e & 1)] = acc[i][j][e];
  red[8 * 32 * 24 + warp * 32 + lane] = bsum;
  __syncthreads();
  float* dst = part + (size_t)blockIdx.x * kConv1Part;
  for (int e = tid; e < kConv1Part; e += kTrainThreads)
  {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k)
      v += e < 32 * 18 ? red[(k * 32 + e / 18) * 24 + e % 18] : red[8 * 32 * 24 + k * 32 + e - 32 * 18];
    dst[e] = v;
  }
}
static_assert(2 * sizeof(Wgrad1Stage) >= (8 * 32 * 24 + 8 * 32) * sizeof(float), "conv1's warp sums fit in its stages");

// Dense layers: dW5 [256][128] = sum d5^T a4, dW6 [6][256] = sum dout^T a5, and the biases, of
// the samples [split * rows, ...).  Warp w holds rows 32 w .. + 31 of dW5 and columns
// 32 w .. + 31 of dW6.
constexpr int kMlpStage = 64;
struct MlpWgradSmem
{
  __nv_bfloat16 d5[kMlpStage * kMlpA5Row];
  __nv_bfloat16 a5[kMlpStage * kMlpA5Row];
  __nv_bfloat16 a4[kMlpStage * kMlpA4Row];
  __nv_bfloat16 dout[kMlpStage * 8];
};
__global__ void __launch_bounds__(kTrainThreads, 1) k_mlp_wgrad(const __nv_bfloat16* __restrict__ dout,
                                                                const __nv_bfloat16* __restrict__ d5,
                                                                const __nv_bfloat16* __restrict__ a5,
                                                                const __nv_bfloat16* __restrict__ a4, float* __restrict__ part,
                                                                int64_t n)
{
  extern __shared__ __align__(16) unsigned char wgrad_raw[];
  MlpWgradSmem& S = *reinterpret_cast<MlpWgradSmem*>(wgrad_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  float acc[2][16][4], acc6[4][4];
#pragma unroll
  for (int e = 0; e < 4; ++e)
  {
#pragma unroll
    for (int j = 0; j < 16; ++j) acc[0][j][e] = acc[1][j][e] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc6[j][e] = 0.f;
  }
  float b5 = 0.f, b6 = 0.f;
  const int64_t stages = (n + kMlpStage - 1) / kMlpStage;
  for (int64_t sg = blockIdx.x; sg < stages; sg += gridDim.x)
  {
    const int64_t m0 = sg * kMlpStage;
    for (int e = tid; e < kMlpStage * 32; e += kTrainThreads)
    {
      const int r = e >> 5, c = e & 31;
      const bool on = m0 + r < n;
      const int64_t o = on ? (m0 + r) * kHidden + c * 8 : 0;
      cp_async16(smem_u32(S.d5 + r * kMlpA5Row + c * 8), d5 + o, on);
      cp_async16(smem_u32(S.a5 + r * kMlpA5Row + c * 8), a5 + o, on);
      if (c < 16) cp_async16(smem_u32(S.a4 + r * kMlpA4Row + c * 8), a4 + (on ? (m0 + r) * 128 + c * 8 : 0), on);
      if (c == 16) cp_async16(smem_u32(S.dout + r * 8), dout + (on ? (m0 + r) * kOutPad : 0), on);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kMlpStage / 16; ++q)
    {
      const int ka = 16 * q + (lane & 7) + (lane >> 4) * 8, ma = ((lane >> 3) & 1) * 8;
      const int kb = 16 * q + (lane & 7) + ((lane >> 3) & 1) * 8, nb = (lane >> 4) * 8;
      uint32_t a[2][4];
      ldsm_x4_trans(a[0], smem_u32(S.d5 + ka * kMlpA5Row + warp * 32 + ma));
      ldsm_x4_trans(a[1], smem_u32(S.d5 + ka * kMlpA5Row + warp * 32 + 16 + ma));
#pragma unroll
      for (int jj = 0; jj < 8; ++jj)
      {
        uint32_t b[4];
        ldsm_x4_trans(b, smem_u32(S.a4 + kb * kMlpA4Row + jj * 16 + nb));
        const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
#pragma unroll
        for (int i = 0; i < 2; ++i)
        {
          mma_bf16_16816(acc[i][2 * jj], a[i], b0);
          mma_bf16_16816(acc[i][2 * jj + 1], a[i], b1);
        }
      }
      // dW6: rows 0..7 of the m16 tile (dout's eight columns), the others zero
      uint32_t d[4];
      ldsm_x4_trans(d, smem_u32(S.dout + (16 * q + (lane & 15)) * 8));   // matrices 0, 1: k 0-7, k 8-15
      const uint32_t a6[4] = {d[0], 0u, d[1], 0u};
#pragma unroll
      for (int jj = 0; jj < 2; ++jj)
      {
        uint32_t b[4];
        ldsm_x4_trans(b, smem_u32(S.a5 + kb * kMlpA5Row + warp * 32 + jj * 16 + nb));
        const uint32_t b0[2] = {b[0], b[1]}, b1[2] = {b[2], b[3]};
        mma_bf16_16816(acc6[2 * jj], a6, b0);
        mma_bf16_16816(acc6[2 * jj + 1], a6, b1);
      }
    }
#pragma unroll 8
    for (int r = 0; r < kMlpStage; ++r) b5 += __bfloat162float(S.d5[r * kMlpA5Row + tid]);
    if (tid < kOut)
      for (int r = 0; r < kMlpStage; ++r) b6 += __bfloat162float(S.dout[r * 8 + tid]);
    __syncthreads();
  }
  float* dst = part + (size_t)blockIdx.x * kMlpPart;   // w5, b5, w6, b6: the parameters' order
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 16; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(dst + (warp * 32 + i * 16 + g + 8 * h) * 128 + j * 8 + 2 * t) =
            make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  dst[kHidden * 128 + tid] = b5;
  float* w6 = dst + kHidden * 128 + kHidden;
  if (g < kOut)
  {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float2*>(w6 + g * kHidden + warp * 32 + j * 8 + 2 * t) = make_float2(acc6[j][0], acc6[j][1]);
  }
  if (tid < kOut) w6[kOut * kHidden + tid] = b6;
}

// grads[i] = the sum of its layer's partials, in an order that does not depend on scheduling:
// eight threads take every eighth partial each, their sums are added in order.  The partials of
// a layer hold its weights, then its bias, as the parameters do.
struct PartLayout
{
  int parts[5];      // conv1, conv2, conv3, conv4, dense layers
};
__global__ void __launch_bounds__(256) k_reduce_parts(const float* __restrict__ part, PartLayout L, float* __restrict__ grads)
{
  using P = ParamLayout;
  __shared__ float red[8][32];
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), y = threadIdx.x >> 5;
  float s = 0.f;
  if (i < P::count)
  {
    const int layer = i < P::w2 ? 0 : i < P::w3 ? 1 : i < P::w4 ? 2 : i < P::w5 ? 3 : 4;
    const int first = layer == 0 ? P::w1 : layer == 1 ? P::w2 : layer == 2 ? P::w3 : layer == 3 ? P::w4 : P::w5;
    const int size = layer == 0 ? kConv1Part : layer < 4 ? kConvPart : kMlpPart;
    const float* p = part + (layer == 0 ? kPartConv1 : layer < 4 ? kPartConv + (size_t)(layer - 1) * kMaxParts * kConvPart
                                                                 : kPartMlp) + (i - first);
#pragma unroll 4
    for (int k = y; k < L.parts[layer]; k += 8) s += p[(size_t)k * size];
  }
  red[y][threadIdx.x & 31] = s;
  __syncthreads();
  if (y == 0 && i < P::count)
  {
    float v = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) v += red[k][threadIdx.x];
    grads[i] = v;
  }
}

}  // namespace cnn
}  // namespace dic
