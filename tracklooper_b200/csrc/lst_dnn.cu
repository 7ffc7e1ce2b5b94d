// Training kernels of the T5 classifier (SDL/NeuralNetwork.h: 38 inputs ->
// 32 ReLU -> 32 ReLU -> 1, sigmoid on the output).  The inference copy lives
// in the quintuplet kernels; these are the forward pass that keeps the hidden
// activations and the backward (adjoint) pass that turns the loss gradient
// w.r.t. the logits into the gradient w.r.t. all 2337 parameters.
//
// Parameter layout (as the weight file): W0[38][32], b0[32], W2[32][32],
// b2[32], w4[32], b4.  The weight gradients are sums over samples; they are
// formed in a fixed order (each block's tiles one after the other, then the
// blocks), so the result does not depend on scheduling.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "lst_b200.h"

namespace {

  constexpr int kIn = 38, kH = 32;
  constexpr int kW0 = 0, kB0 = kIn * kH, kW2 = kB0 + kH, kB2 = kW2 + kH * kH, kW4 = kB2 + kH, kB4 = kW4 + kH;
  constexpr int kParams = kB4 + 1;
  static_assert(kParams == 2337, "T5 DNN parameter count");
  static_assert(kW0 % 4 == 0 && kW2 % 4 == 0 && kB0 % 4 == 0 && kB2 % 4 == 0 && kW4 % 4 == 0, "16-byte rows");

  // The file is compiled without contraction.  The forward sums stay unfused, in
  // the order of the inputs and with the bias last: an activation within a
  // rounding of zero opens or closes its ReLU gate for the whole gradient of the
  // sample, and with fused sums other gates would open (262143 samples: one such
  // gate moved the gradient by 2e-6 of its norm, five times its error in 64 bits).
  // The gradient sums, which gate nothing, fuse explicitly.
  __device__ __forceinline__ void mulAdd4(float* acc, float a, const float4& w) {
    acc[0] += a * w.x;
    acc[1] += a * w.y;
    acc[2] += a * w.z;
    acc[3] += a * w.w;
  }
  __device__ __forceinline__ void fma4(float* acc, float a, const float4& w) {
    acc[0] = fmaf(a, w.x, acc[0]);
    acc[1] = fmaf(a, w.y, acc[1]);
    acc[2] = fmaf(a, w.z, acc[2]);
    acc[3] = fmaf(a, w.w, acc[3]);
  }

  // Rows [s0, s0 + rows) of a row-major (n x C) matrix into shared memory with
  // row stride `stride`, coalesced; the tile's rows past the end become zero.
  template <int C>
  __device__ __forceinline__ void loadRows(const float* __restrict__ src, int s0, int rows, int tile, float* dst,
                                           int stride) {
    const float* from = src + size_t(s0) * C;
    for (int i = threadIdx.x; i < tile * C; i += blockDim.x) {
      const int r = i / C;
      dst[r * stride + (i - r * C)] = r < rows ? from[i] : 0.f;
    }
  }

  // kSPT samples per thread: the inputs of the block's samples are staged in
  // shared memory (coalesced, odd row stride), a layer's 32 sums per sample stay
  // in registers, and a weight row is eight 16-byte broadcasts from shared memory
  // for 32 kSPT multiply-adds.  The activations go out through the warp's own
  // rows of the staging, whole lines at a time.  Bound by the unfused multiplies
  // and adds and the broadcasts, so large batches take two samples a thread; below
  // kFwdPairFrom samples, where one block per SM of that shape would leave SMs
  // idle, one a thread.  262143 samples: 389 us with strided reads and writes and
  // one sum at a time, now 151; 8192 samples: 35 us, now 25.
  constexpr int kFwdThreads = 64;
  constexpr int kFwdPairFrom = 1 << 16;
  template <int kSPT>
  __global__ void __launch_bounds__(kFwdThreads) kDnnForward(const float* __restrict__ W, const float* __restrict__ x,
                                                             int n, float* __restrict__ h1, float* __restrict__ h2,
                                                             float* __restrict__ logit) {
    constexpr int kRows = kFwdThreads * kSPT, kStride = kIn + 1;
    __shared__ __align__(16) float sW[kParams + 3];
    __shared__ float sX[kRows * kStride];
    const int lane = threadIdx.x & 31;
    // the warp's samples are rows [warpRow, warpRow + 32 kSPT) of the tile; this
    // thread's are warpRow + lane + 32 p
    const int warpRow = (threadIdx.x >> 5) * 32 * kSPT;
    for (int i = threadIdx.x; i < kParams; i += blockDim.x)
      sW[i] = W[i];
    // activations of part p (32 samples) from registers to row-major memory
    auto write = [&](const float* a, int p, int s0, float* to) {
      float* own = sX + (warpRow + 32 * p) * kStride;  // 32 x 33 floats fit these 32 rows
      __syncwarp();
#pragma unroll
      for (int c = 0; c < kH; ++c)
        own[lane * (kH + 1) + c] = a[c];
      __syncwarp();
      const int first = s0 + warpRow + 32 * p;
      for (int r = 0; r < 32 && first + r < n; ++r)
        to[size_t(first + r) * kH + lane] = own[r * (kH + 1) + lane];
    };
    for (int s0 = blockIdx.x * kRows; s0 < n; s0 += gridDim.x * kRows) {
      __syncthreads();
      loadRows<kIn>(x, s0, min(n - s0, kRows), kRows, sX, kStride);
      __syncthreads();
      float a1[kSPT][kH];
#pragma unroll
      for (int p = 0; p < kSPT; ++p)
#pragma unroll
        for (int c = 0; c < kH; ++c)
          a1[p][c] = 0.f;
#pragma unroll 2
      for (int k = 0; k < kIn; ++k) {
        float xk[kSPT];
#pragma unroll
        for (int p = 0; p < kSPT; ++p)
          xk[p] = sX[(warpRow + lane + 32 * p) * kStride + k];
        const float4* w = reinterpret_cast<const float4*>(sW + kW0 + k * kH);
#pragma unroll
        for (int c = 0; c < kH / 4; ++c) {
          const float4 wc = w[c];
#pragma unroll
          for (int p = 0; p < kSPT; ++p)
            mulAdd4(a1[p] + 4 * c, xk[p], wc);
        }
      }
#pragma unroll
      for (int p = 0; p < kSPT; ++p) {
#pragma unroll
        for (int c = 0; c < kH; ++c) {
          const float v = a1[p][c] + sW[kB0 + c];
          a1[p][c] = v > 0.f ? v : 0.f;
        }
        write(a1[p], p, s0, h1);
      }
      // the second layer in two halves of its columns, so that the sums and the
      // first layer's activations fit the registers
      float z[kSPT];
#pragma unroll
      for (int p = 0; p < kSPT; ++p)
        z[p] = 0.f;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        constexpr int kC = kH / 2;
        float a2[kSPT][kC];
#pragma unroll
        for (int p = 0; p < kSPT; ++p)
#pragma unroll
          for (int c = 0; c < kC; ++c)
            a2[p][c] = 0.f;
#pragma unroll
        for (int k = 0; k < kH; ++k) {
          const float4* w = reinterpret_cast<const float4*>(sW + kW2 + k * kH + half * kC);
#pragma unroll
          for (int c = 0; c < kC / 4; ++c) {
            const float4 wc = w[c];
#pragma unroll
            for (int p = 0; p < kSPT; ++p)
              mulAdd4(a2[p] + 4 * c, a1[p][k], wc);
          }
        }
#pragma unroll
        for (int p = 0; p < kSPT; ++p) {
          float* own = sX + (warpRow + 32 * p) * kStride;
          if (half == 0)
            __syncwarp();
#pragma unroll
          for (int c = 0; c < kC; ++c) {
            const float v = a2[p][c] + sW[kB2 + half * kC + c];
            const float a = v > 0.f ? v : 0.f;
            z[p] += a * sW[kW4 + half * kC + c];
            own[lane * (kH + 1) + half * kC + c] = a;
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int p = 0; p < kSPT; ++p) {
        const float* own = sX + (warpRow + 32 * p) * kStride;
        const int first = s0 + warpRow + 32 * p;
        for (int r = 0; r < 32 && first + r < n; ++r)
          h2[size_t(first + r) * kH + lane] = own[r * (kH + 1) + lane];
        if (first + lane < n)
          logit[first + lane] = z[p] + sW[kB4];
      }
    }
  }

  // The backward pass of a tile of 64 samples and its share of every weight
  // gradient, in one kernel.  Per sample: g2 = dz w4 (ReLU-gated), dh1 = W2 g2
  // (ReLU-gated), by two threads.  The gradients are the products
  //   [x | 1]^T dh1  (40 x 32, with b0 as the row of ones)  and
  //   [h1 | 1]^T g2  (36 x 32, with b2 as the row of ones),
  // of which each of 152 threads keeps a 4 x 4 tile in registers over all the
  // block's tiles (two 16-byte reads of shared memory for 16 multiply-adds), and
  // 8 threads the w4 and b4 sums.  A block writes its sums once.  Bound by the
  // multiply-adds (3.3 k per sample) and their shared-memory operands.
  // With dh1 and dh2 in memory and a thread per gradient element that read every
  // sample's two factors, 262143 samples took 1955 us, now 130; 8192: 146 and 26.
  constexpr int kTile = 64;
  constexpr int kBwdThreads = 160;
  constexpr int kXRow = 40, kHRow = 36;  // row strides: 16-byte rows, lanes on different banks
  struct BwdShared {
    float x[kTile * kXRow];    // 38 inputs, 1, 0
    float h1[kTile * kHRow];   // 32 activations, 1, 0, 0, 0
    float h2[kTile * kHRow];
    float g2[kTile * kHRow];
    float dh1[kTile * kHRow];
    float w2[kH * kH];
    float w4[kH];
    float dz[kTile];
  };
  __device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }

  __global__ void __launch_bounds__(kBwdThreads) kDnnBackward(const float* __restrict__ W, const float* __restrict__ x,
                                                              const float* __restrict__ h1,
                                                              const float* __restrict__ h2,
                                                              const float* __restrict__ dlogit, int n,
                                                              float* __restrict__ partial) {
    extern __shared__ __align__(16) unsigned char smem[];
    BwdShared& sm = *reinterpret_cast<BwdShared*>(smem);
    const int t = threadIdx.x;
    for (int i = t; i < kH * kH; i += kBwdThreads)
      sm.w2[i] = W[kW2 + i];
    if (t < kH)
      sm.w4[t] = W[kW4 + t];
    if (t < kTile) {
      sm.x[t * kXRow + kIn] = 1.f;
      sm.x[t * kXRow + kIn + 1] = 0.f;
      sm.h1[t * kHRow + kH] = 1.f;
      for (int k = 1; k < 4; ++k)
        sm.h1[t * kHRow + kH + k] = 0.f;
    }
    // this thread's tile of a product: rows 4 r .., columns 4 c ..
    const bool first = t < 80, second = !first && t < 152;
    const int u = first ? t : second ? t - 80 : t - 152;
    const int r = u / 8, c = u % 8;
    const float* rowsOf = first ? sm.x + 4 * r : sm.h1 + 4 * r;
    const int rowStride = first ? kXRow : kHRow;
    const float* colsOf = (first ? sm.dh1 : second ? sm.g2 : sm.h2) + 4 * c;
    float acc[16];
#pragma unroll
    for (int k = 0; k < 16; ++k)
      acc[k] = 0.f;
    float accDz = 0.f;
    for (int s0 = blockIdx.x * kTile; s0 < n; s0 += gridDim.x * kTile) {
      const int rows = min(n - s0, kTile);
      __syncthreads();
      loadRows<kIn>(x, s0, rows, kTile, sm.x, kXRow);
      loadRows<kH>(h1, s0, rows, kTile, sm.h1, kHRow);
      loadRows<kH>(h2, s0, rows, kTile, sm.h2, kHRow);
      if (t < kTile)
        sm.dz[t] = t < rows ? dlogit[s0 + t] : 0.f;
      __syncthreads();
      if (t < 2 * kTile) {
        const int s = t % kTile, i0 = (t / kTile) * (kH / 2);
        const float dz = sm.dz[s];
        float g[kH];
#pragma unroll
        for (int j = 0; j < kH; j += 4) {
          const float4 a = load4(sm.h2 + s * kHRow + j), w = load4(sm.w4 + j);
          g[j] = a.x > 0.f ? dz * w.x : 0.f;
          g[j + 1] = a.y > 0.f ? dz * w.y : 0.f;
          g[j + 2] = a.z > 0.f ? dz * w.z : 0.f;
          g[j + 3] = a.w > 0.f ? dz * w.w : 0.f;
          if (i0 == 0)
            *reinterpret_cast<float4*>(sm.g2 + s * kHRow + j) = make_float4(g[j], g[j + 1], g[j + 2], g[j + 3]);
        }
        for (int i = i0; i < i0 + kH / 2; i += 4) {
          float d[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < kH; j += 4) {
              const float4 w = load4(sm.w2 + (i + k) * kH + j);
              sum = fmaf(g[j], w.x, sum);
              sum = fmaf(g[j + 1], w.y, sum);
              sum = fmaf(g[j + 2], w.z, sum);
              sum = fmaf(g[j + 3], w.w, sum);
            }
            d[k] = sum;
          }
          const float4 a = load4(sm.h1 + s * kHRow + i);
          *reinterpret_cast<float4*>(sm.dh1 + s * kHRow + i) =
              make_float4(a.x > 0.f ? d[0] : 0.f, a.y > 0.f ? d[1] : 0.f, a.z > 0.f ? d[2] : 0.f, a.w > 0.f ? d[3] : 0.f);
        }
      }
      __syncthreads();
      if (first || second) {
#pragma unroll 4
        for (int s = 0; s < kTile; ++s) {
          const float4 a = load4(rowsOf + s * rowStride), b = load4(colsOf + s * kHRow);
          fma4(acc, a.x, b);
          fma4(acc + 4, a.y, b);
          fma4(acc + 8, a.z, b);
          fma4(acc + 12, a.w, b);
        }
      } else {
        for (int s = 0; s < kTile; ++s) {
          const float dz = sm.dz[s];
          fma4(acc, dz, load4(colsOf + s * kHRow));
          accDz += dz;
        }
      }
    }
    float* out = partial + size_t(blockIdx.x) * kParams;
    if (first || second) {
      const int rowsW = first ? kIn : kH;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int row = 4 * r + k;
        const int at = row < rowsW ? (first ? kW0 : kW2) + row * kH : (first ? kB0 : kB2);
        if (row <= rowsW)
          for (int j = 0; j < 4; ++j)
            out[at + 4 * c + j] = acc[4 * k + j];
      }
    } else {
      for (int j = 0; j < 4; ++j)
        out[kW4 + 4 * c + j] = acc[j];
      if (c == 0)
        out[kB4] = accDz;
    }
  }

  // grad[g] = sum of the blocks' partial sums, each warp of a block taking every
  // 32nd of them for 32 parameters (coalesced), then the warps in order.
  __global__ void __launch_bounds__(1024) kDnnGradReduce(const float* __restrict__ partial, int nPartials,
                                                         float* __restrict__ grad) {
    __shared__ float sSum[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = blockIdx.x * 32 + lane;
    float acc = 0.f;
    if (g < kParams)
      for (int p = warp; p < nPartials; p += 32)
        acc += partial[size_t(p) * kParams + g];
    sSum[warp][lane] = acc;
    __syncthreads();
    // warp w folds parameter w of the block: lane l holds warp l's sum
    float v = sSum[lane][warp];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_down_sync(0xffffffffu, v, o);
    const int gw = blockIdx.x * 32 + warp;
    if (lane == 0 && gw < kParams)
      grad[gw] = v;
  }

  thread_local std::string g_dnnError;

  int dnnFail(const char* what) {
    cudaError_t e = cudaGetLastError();
    g_dnnError = std::string(what) + ": " + cudaGetErrorString(e);
    return -1;
  }

  // Blocks of a kernel that strides over n samples, `tile` at a time: at most
  // four resident per SM of the current device (the backward pass keeps 51 KB of
  // shared memory a block, and a block's gradient sums are written once).
  int blocksFor(int n, int tile, int perSM) {
    int device = 0, sms = 148;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
      cudaGetLastError();
      sms = 148;
    }
    const int tiles = (n - 1) / tile + 1;
    return tiles < perSM * sms ? tiles : perSM * sms;
  }
  constexpr int kBwdPerSM = 4;

}  // namespace

// No C++ exception crosses the C ABI (see lst_event.cu): host-side failures
// become a -1 status with a message.
#define LST_ABI_TRY try {
#define LST_ABI_CATCH_INT        \
  }                              \
  catch (...) {                  \
    try {                        \
      g_dnnError = "host error"; \
    } catch (...) {              \
    }                            \
    return -1;                   \
  }

extern "C" {

size_t lst_t5dnn_scratch_floats(int n) {
  // (The backward pass uses kParams floats per block, at most one block per 64
  // samples, which is less than this for every n; the size is part of the
  // interface and stays.)
  constexpr size_t kChunk = 256;
  const size_t chunks = (size_t(n > 0 ? n : 0) + kChunk - 1) / kChunk;
  return 2 * size_t(kH) * size_t(n > 0 ? n : 0) + chunks * kParams;
}

int lst_t5dnn_forward(const float* weights, const float* x, int n, float* h1, float* h2, float* logit, void* stream) {
  LST_ABI_TRY
  if (n <= 0)
    return 0;
  if (!weights || !x || !h1 || !h2 || !logit)
    return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaGetLastError();
  if (n >= kFwdPairFrom)
    kDnnForward<2><<<blocksFor(n, 2 * kFwdThreads, 16), kFwdThreads, 0, s>>>(weights, x, n, h1, h2, logit);
  else
    kDnnForward<1><<<blocksFor(n, kFwdThreads, 16), kFwdThreads, 0, s>>>(weights, x, n, h1, h2, logit);
  if (cudaPeekAtLastError() != cudaSuccess)
    return dnnFail("kDnnForward");
  return 0;
  LST_ABI_CATCH_INT
}

int lst_t5dnn_backward(const float* weights, const float* x, const float* h1, const float* h2, const float* dlogit,
                       int n, float* grad, float* scratch, void* stream) {
  LST_ABI_TRY
  if (!weights || !x || !h1 || !h2 || !dlogit || !grad || !scratch)
    return -1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaGetLastError();
  if (n <= 0) {
    if (cudaMemsetAsync(grad, 0, sizeof(float) * kParams, s) != cudaSuccess)
      return dnnFail("cudaMemsetAsync");
    return 0;
  }
  // (per device, so set on every call: it only records the limit)
  if (cudaFuncSetAttribute(kDnnBackward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(sizeof(BwdShared))) != cudaSuccess)
    return dnnFail("kDnnBackward shared memory");
  const int blocks = blocksFor(n, kTile, kBwdPerSM);
  kDnnBackward<<<blocks, kBwdThreads, sizeof(BwdShared), s>>>(weights, x, h1, h2, dlogit, n, scratch);
  if (cudaPeekAtLastError() != cudaSuccess)
    return dnnFail("kDnnBackward");
  kDnnGradReduce<<<(kParams + 31) / 32, 1024, 0, s>>>(scratch, blocks, grad);
  if (cudaPeekAtLastError() != cudaSuccess)
    return dnnFail("kDnnGradReduce");
  return 0;
  LST_ABI_CATCH_INT
}

const char* lst_t5dnn_last_error(void) { return g_dnnError.c_str(); }

}  // extern "C"
