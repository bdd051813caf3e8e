// Learned hybrid sensor: training-data harvest from the plain FP64 method,
// BF16 tensor-core forward/backward kernels (FP32 accumulation), Adam.
//
// The reference's hybrid switch (fortran/rhs_hybrid_high_llf.m4:239-256)
// sends a level-0 cell to WENO when any of six density-ratio tests falls
// below 0.9999.  The learned sensor predicts from 40 stencil features
// (enl_mlp.cuh) whether WENO is needed, trained on the plain switch and on
// the local difference between the DRP and WENO right-hand sides.
#include <cstddef>
#include <cstring>
#include <cstdio>

#include "enl_mlp.cuh"
#include "enl_rhs_cell.cuh"

namespace enl {

// ---------------------------------------------------------------------------
// Training: one block of 4 warps handles chunks of 64 samples (16 per warp).
//
// The six matrix products of a chunk are small (64 x 48 x 64 and 64 x 64 x 64),
// so what bounds the kernel is everything around them: operand loads, the
// activations and the reductions over samples.
//   * Every fragment comes from shared memory by ldmatrix (four 8 x 8 tiles per
//     instruction, transposed where the product runs over samples) from
//     conflict-free padded rows; W2 is kept once, its transpose read from it.
//   * GELU and its derivative are evaluated once per activation, not once more
//     where the derivative is needed.
//   * Bias gradients are a product with a row of ones on the tensor cores,
//     done by the warp that has no rows of dW1, and dw3 is accumulated in
//     registers; one warp summing 64 samples column by column kept the other
//     three waiting.
//   * As many blocks as fit (no second wave that stages the parameters again),
//     features read 16 bytes at a time.
// 65,536 samples: 84 -> 53 us a call among others (with its two clears; a call
// alone 86 -> 54).
// ---------------------------------------------------------------------------
constexpr int kChunk = 64;

// (every matrix starts and every row lies on 16 bytes: ldmatrix and the wide
// copies need it)
struct alignas(16) TrainSmem {
  alignas(16) MlpSmem S;
  alignas(16) __nv_bfloat16 xs[kChunk][kLdF];
  alignas(16) __nv_bfloat16 h1[kChunk][kLdH];
  alignas(16) __nv_bfloat16 dz1[kChunk][kLdH];
  alignas(16) __nv_bfloat16 dz2[kChunk][kLdH];
};
static_assert(offsetof(MlpSmem, w1t) % 16 == 0 && offsetof(MlpSmem, w2t) % 16 == 0 && offsetof(TrainSmem, xs) % 16 == 0 &&
                  offsetof(TrainSmem, h1) % 16 == 0 && offsetof(TrainSmem, dz1) % 16 == 0 &&
                  offsetof(TrainSmem, dz2) % 16 == 0 && kLdF * 2 % 16 == 0 && kLdH * 2 % 16 == 0,
              "16-byte rows");

// GELU and its derivative at one argument, in one place so that the compiler
// shares Phi(x) between them (erf_as's exponential and the density's round their
// arguments differently and stay two).
__device__ __forceinline__ void gelu_both(float x, float& g, float& d) {
  g = gelu(x);
  d = gelu_grad(x);
}

// C (16 x 64, n-tiles of 8) += A (16 x 16 fragment) B, B's 16 x 64 slice at p
// stored [k][n] (rows of ld).
__device__ __forceinline__ void mma_row64(float c[8][4], const uint32_t a[4], const __nv_bfloat16* p, int ld,
                                          int lane) {
  const __nv_bfloat16* q = p + (lane & 15) * ld + (lane >> 4) * 8;
#pragma unroll
  for (int n = 0; n < 8; n += 2) {
    uint32_t b[4];
    ldsm4t(b, q + n * 8);
    mma_bf16(c[n], a[0], a[1], a[2], a[3], b[0], b[1]);
    mma_bf16(c[n + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
  }
}
// The same with B stored [n][k].
__device__ __forceinline__ void mma_col64(float c[8][4], const uint32_t a[4], const __nv_bfloat16* p, int ld,
                                          int lane) {
  const __nv_bfloat16* q = p + ((lane >> 4) * 8 + (lane & 7)) * ld + ((lane >> 3) & 1) * 8;
#pragma unroll
  for (int n = 0; n < 8; n += 2) {
    uint32_t b[4];
    ldsm4(b, q + n * 8 * ld);
    mma_bf16(c[n], a[0], a[1], a[2], a[3], b[0], b[1]);
    mma_bf16(c[n + 1], a[0], a[1], a[2], a[3], b[2], b[3]);
  }
}

__device__ __forceinline__ float2 bf16_pair(uint32_t v) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
}

__global__ void __launch_bounds__(128, 3) mlp_grad_kernel(const __nv_bfloat16* __restrict__ X,
                                                          const float* __restrict__ y, const float* __restrict__ wgt,
                                                          long N, const float* __restrict__ P, float* grad,
                                                          double* loss_sum) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  TrainSmem& T = *reinterpret_cast<TrainSmem*>(sm_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  mlp_stage_params(T.S, P, tid, 128);
  for (int e = tid; e < kChunk * (kFeatPad - kFeat); e += 128)
    T.xs[e / (kFeatPad - kFeat)][kFeat + e % (kFeatPad - kFeat)] = __float2bfloat16_rn(0.0f);
  const bool wide = (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  // the block's weight gradients: rows 16 warp .. of dW2; of dW1 (warps 0-2)
  // or, warp 3, db1 in row 0 and db2 in row 8 of products with ones
  float aw2[8][4], aw1[8][4];
  float aw3[8][2], ab3 = 0.f;
#pragma unroll
  for (int n = 0; n < 8; ++n) {
#pragma unroll
    for (int q = 0; q < 4; ++q) aw2[n][q] = aw1[n][q] = 0.f;
    aw3[n][0] = aw3[n][1] = 0.f;
  }
  // A fragments with ones in row 0 and in row 8
  const uint32_t one = g == 0 ? 0x3f803f80u : 0u;
  const uint32_t ones0[4] = {one, 0u, one, 0u}, ones8[4] = {0u, one, 0u, one};
  double lsum = 0.0;
  for (long c0 = (long)blockIdx.x * kChunk; c0 < N; c0 += (long)gridDim.x * kChunk) {
    if (wide && c0 + kChunk <= N) {
      const uint4* src = reinterpret_cast<const uint4*>(X + c0 * kFeat);
      for (int e = tid; e < kChunk * kFeat / 8; e += 128) {
        const int r = e / (kFeat / 8), q = e % (kFeat / 8);
        *reinterpret_cast<uint4*>(&T.xs[r][8 * q]) = src[e];
      }
    } else {
      for (int e = tid; e < kChunk * kFeat; e += 128) {
        const int r = e / kFeat, k = e % kFeat;
        T.xs[r][k] = c0 + r < N ? X[(c0 + r) * kFeat + k] : __float2bfloat16_rn(0.0f);
      }
    }
    __syncthreads();
    // forward, 16 rows per warp
    const int r0 = warp * 16 + g, r1 = r0 + 8, arow = warp * 16 + (lane & 15), acol = (lane >> 4) * 8;
    float z1[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) z1[n][q] = T.S.b1[n * 8 + 2 * t + (q & 1)];
#pragma unroll
    for (int kc = 0; kc < 3; ++kc) {
      uint32_t a[4];
      ldsm4(a, &T.xs[arow][kc * 16 + acol]);
      mma_col64(z1, a, &T.S.w1t[0][kc * 16], kLdF, lane);
    }
    // hidden layer 1: BF16 A fragments of layer 2, kept for dW2; z1 becomes
    // the derivative of the activation
    float z2[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) z2[n][q] = T.S.b2[n * 8 + 2 * t + (q & 1)];
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {
      uint32_t a[4];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int n = 2 * kc + half, col = n * 8 + 2 * t;
        float h[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) gelu_both(z1[n][q], h[q], z1[n][q]);
        a[2 * half] = pack_bf16(h[0], h[1]);
        a[2 * half + 1] = pack_bf16(h[2], h[3]);
        *reinterpret_cast<uint32_t*>(&T.h1[r0][col]) = a[2 * half];
        *reinterpret_cast<uint32_t*>(&T.h1[r1][col]) = a[2 * half + 1];
      }
      mma_col64(z2, a, &T.S.w2t[0][kc * 16], kLdH, lane);
    }
    // last layer: hidden activations rounded to BF16 like the tensor-core
    // layers' inputs; z2 becomes the derivative
    float s0 = 0.f, s1 = 0.f;
    uint32_t h2[8][2];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int col = n * 8 + 2 * t;
      float h[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) gelu_both(z2[n][q], h[q], z2[n][q]);
      h2[n][0] = pack_bf16(h[0], h[1]);
      h2[n][1] = pack_bf16(h[2], h[3]);
      const float2 u = bf16_pair(h2[n][0]), v = bf16_pair(h2[n][1]);
      s0 += u.x * T.S.w3[col] + u.y * T.S.w3[col + 1];
      s1 += v.x * T.S.w3[col] + v.y * T.S.w3[col + 1];
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    // BCE-with-logits gradient of rows r0, r1 (lanes t == 0)
    float dl0 = 0.f, dl1 = 0.f;
    if (t == 0) {
      const long i0 = c0 + r0, i1 = c0 + r1;
      const float l0 = s0 + T.S.b3, l1 = s1 + T.S.b3;
      if (i0 < N) {
        const float w = wgt[i0], yy = y[i0];
        dl0 = w * (1.0f / (1.0f + __expf(-l0)) - yy);
        lsum += (double)(w * (fmaxf(l0, 0.f) - yy * l0 + log1pf(__expf(-fabsf(l0)))));
      }
      if (i1 < N) {
        const float w = wgt[i1], yy = y[i1];
        dl1 = w * (1.0f / (1.0f + __expf(-l1)) - yy);
        lsum += (double)(w * (fmaxf(l1, 0.f) - yy * l1 + log1pf(__expf(-fabsf(l1)))));
      }
      ab3 += dl0 + dl1;
    }
    dl0 = __shfl_sync(0xffffffffu, dl0, lane & ~3);
    dl1 = __shfl_sync(0xffffffffu, dl1, lane & ~3);
    // dw3, and dZ2 = (dl w3) gelu'(z2) as A fragments and in shared memory;
    // dH1 = dZ2 W2^T on the tensor cores
    float dh1[8][4];
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) dh1[n][q] = 0.f;
#pragma unroll
    for (int kc = 0; kc < 4; ++kc) {
      uint32_t a[4];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int n = 2 * kc + half, col = n * 8 + 2 * t;
        const float2 u = bf16_pair(h2[n][0]), v = bf16_pair(h2[n][1]);
        aw3[n][0] += dl0 * u.x + dl1 * v.x;
        aw3[n][1] += dl0 * u.y + dl1 * v.y;
        const float w0 = T.S.w3[col], w1 = T.S.w3[col + 1];
        a[2 * half] = pack_bf16(dl0 * w0 * z2[n][0], dl0 * w1 * z2[n][1]);
        a[2 * half + 1] = pack_bf16(dl1 * w0 * z2[n][2], dl1 * w1 * z2[n][3]);
        *reinterpret_cast<uint32_t*>(&T.dz2[r0][col]) = a[2 * half];
        *reinterpret_cast<uint32_t*>(&T.dz2[r1][col]) = a[2 * half + 1];
      }
      // B(kk = hidden-2 index, col = hidden-1 index) = W2[col][kk] = w2t[kk][col]
      mma_row64(dh1, a, &T.S.w2t[kc * 16][0], kLdH, lane);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int col = n * 8 + 2 * t;
      *reinterpret_cast<uint32_t*>(&T.dz1[r0][col]) = pack_bf16(dh1[n][0] * z1[n][0], dh1[n][1] * z1[n][1]);
      *reinterpret_cast<uint32_t*>(&T.dz1[r1][col]) = pack_bf16(dh1[n][2] * z1[n][2], dh1[n][3] * z1[n][3]);
    }
    __syncthreads();
    // weight gradients, sums over the 64 samples on the tensor cores:
    // dW2[k][n] = sum_s H1[s][k] dZ2[s][n] (warp w: rows k of m-tile w)
    // dW1[k][n] = sum_s X[s][k] dZ1[s][n]  (warps 0-2: m-tiles of k < 48)
    // db2[n], db1[n] = sum_s dZ2[s][n], dZ1[s][n] (warp 3: ones in place of A)
    const int trow = ((lane >> 4) & 1) * 8 + (lane & 7), tcol = warp * 16 + ((lane >> 3) & 1) * 8;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t a[4];
      ldsm4t(a, &T.h1[ks * 16 + trow][tcol]);
      mma_row64(aw2, a, &T.dz2[ks * 16][0], kLdH, lane);
      if (warp < 3) {
        ldsm4t(a, &T.xs[ks * 16 + trow][tcol]);
        mma_row64(aw1, a, &T.dz1[ks * 16][0], kLdH, lane);
      } else {
        mma_row64(aw1, ones0, &T.dz1[ks * 16][0], kLdH, lane);
        mma_row64(aw1, ones8, &T.dz2[ks * 16][0], kLdH, lane);
      }
    }
    __syncthreads();
  }
  // flush the block's partial gradients, two neighbouring weights an atomic (a
  // warp's then fill their 32-byte sectors: a call alone 57.3 -> 55.8 us for 65,536
  // samples, 92.7 -> 90.6 for 200,000; one block of three teams an SM that sums its weight
  // gradients in shared memory first gained no more and cost 6 us on 3,000)
  static_assert(kOffW1 % 2 == 0 && kOffW2 % 2 == 0 && kOffB1 % 2 == 0 && kOffB2 % 2 == 0 && kHid % 2 == 0,
                "pairs start on 8 bytes where grad does");
  const bool pairs = (reinterpret_cast<uintptr_t>(grad) & 7) == 0;
  auto add2 = [&](int o, float a, float b) {
    if (pairs) {
      atomicAdd(reinterpret_cast<float2*>(&grad[o]), make_float2(a, b));
    } else {
      atomicAdd(&grad[o], a);
      atomicAdd(&grad[o + 1], b);
    }
  };
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int col = n * 8 + 2 * t;
    const int k0 = warp * 16 + g, k1 = k0 + 8;
    add2(kOffW2 + k0 * kHid + col, aw2[n][0], aw2[n][1]);
    add2(kOffW2 + k1 * kHid + col, aw2[n][2], aw2[n][3]);
    if (warp < 3) {
      if (k0 < kFeat) add2(kOffW1 + k0 * kHid + col, aw1[n][0], aw1[n][1]);
      if (k1 < kFeat) add2(kOffW1 + k1 * kHid + col, aw1[n][2], aw1[n][3]);
    } else if (g == 0) {  // rows 0 and 8
      add2(kOffB1 + col, aw1[n][0], aw1[n][1]);
      add2(kOffB2 + col, aw1[n][2], aw1[n][3]);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      float v = aw3[n][q];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (g == 0) atomicAdd(&grad[kOffW3 + col + q], v);
    }
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) ab3 += __shfl_xor_sync(0xffffffffu, ab3, o);
  if (lane == 0) atomicAdd(&grad[kOffB3], ab3);
  if (loss_sum) {
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if (lane == 0) atomicAdd(loss_sum, lsum);
  }
}

// Inference on a feature matrix (evaluation and tests): logits of N rows.
__global__ void __launch_bounds__(128) mlp_forward_kernel(const __nv_bfloat16* __restrict__ X, long N,
                                                          const float* __restrict__ P, float* __restrict__ logit) {
  __shared__ MlpSmem S;
  __shared__ __align__(16) __nv_bfloat16 xs[kChunk][kLdF];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  mlp_stage_params(S, P, tid, 128);
  __syncthreads();
  for (long c0 = (long)blockIdx.x * kChunk; c0 < N; c0 += (long)gridDim.x * kChunk) {
    for (int e = tid; e < kChunk * kFeatPad; e += 128) {
      int r = e / kFeatPad, k = e % kFeatPad;
      long s = c0 + r;
      xs[r][k] = (s < N && k < kFeat) ? X[s * kFeat + k] : __float2bfloat16_rn(0.0f);
    }
    __syncthreads();
    MlpFwd16 F;
    mlp_forward16(S, &xs[warp * 16][0], kLdF, lane, F);
    if ((lane & 3) == 0) {
      long s0 = c0 + warp * 16 + (lane >> 2);
      if (s0 < N) logit[s0] = F.logit[0];
      if (s0 + 8 < N) logit[s0 + 8] = F.logit[1];
    }
    __syncthreads();
  }
}

// Adam on the FP32 master parameters; the gradient is a sum over samples and
// is scaled by inv_n (1 / total sample weight).
__global__ void adam_kernel(float* P, const float* grad, float* m, float* v, int n, float lr, float b1, float b2,
                            float eps, float inv_n, int step) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float gr = grad[i] * inv_n;
  float mm = b1 * m[i] + (1.f - b1) * gr;
  float vv = b2 * v[i] + (1.f - b2) * gr * gr;
  m[i] = mm;
  v[i] = vv;
  float mh = mm / (1.f - powf(b1, (float)step));
  float vh = vv / (1.f - powf(b2, (float)step));
  P[i] -= lr * mh / (sqrtf(vh) + eps);
}

}  // namespace enl

using namespace enl;

// Largest |erf_as(x) - erff(x)| over n points evenly spread in [-6, 6]
// (bits of a non-negative float: ordered as unsigned integers).
__global__ void erf_check_kernel(int n, unsigned* max_bits) {
  float m = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float x = -6.0f + 12.0f * (float)i / (float)(n - 1);
    m = fmaxf(m, fabsf(erf_as(x) - erff(x)));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(max_bits, __float_as_uint(m));
}

extern "C" {

int enl_mlp_erf_error(double* max_err) {
  if (!max_err) return ENL_ERR_ARG;
  unsigned* d = nullptr;
  if (cudaMalloc(&d, sizeof(unsigned)) != cudaSuccess) return ENL_ERR_CUDA;
  cudaMemsetAsync(d, 0, sizeof(unsigned), stream());
  erf_check_kernel<<<256, 256, 0, stream()>>>(1 << 22, d);
  unsigned h = 0;
  cudaMemcpyAsync(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost, stream());
  cudaStreamSynchronize(stream());
  cudaFree(d);
  float f;
  memcpy(&f, &h, sizeof(f));
  *max_err = f;
  return check_launch("mlp erf check");
}

int enl_mlp_nparams(void) { return kNParams; }

int enl_mlp_grad(const void* X, const float* y, const float* wgt, long n, const float* params, float* grad,
                 double* loss_sum) {
  if (!X || !y || !wgt || !params || !grad || n < 0) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  if (n == 0) return ENL_OK;
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrainSmem));
    attr = true;
  }
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, 0);
  long chunks = (n + kChunk - 1) / kChunk;
  int blocks = (int)std::min<long>(chunks, (long)nsm * 3);  // resident at once
  mlp_grad_kernel<<<blocks, 128, sizeof(TrainSmem), stream()>>>((const __nv_bfloat16*)X, y, wgt, n, params, grad,
                                                               loss_sum);
  return check_launch("mlp_grad");
}

int enl_mlp_forward(const void* X, long n, const float* params, float* logits) {
  if (!X || !params || !logits || n < 0) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  if (n == 0) return ENL_OK;
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, 0);
  long chunks = (n + kChunk - 1) / kChunk;
  int blocks = (int)std::min<long>(chunks, (long)nsm * 8);
  mlp_forward_kernel<<<blocks, 128, 0, stream()>>>((const __nv_bfloat16*)X, n, params, logits);
  return check_launch("mlp_forward");
}

int enl_mlp_adam(float* params, const float* grad, float* m, float* v, float lr, float beta1, float beta2, float eps,
                 float inv_n, int step) {
  if (!params || !grad || !m || !v || step < 1) {
    set_error(ENL_ERR_ARG);
    return ENL_ERR_ARG;
  }
  adam_kernel<<<(kNParams + 255) / 256, 256, 0, stream()>>>(params, grad, m, v, kNParams, lr, beta1, beta2, eps, inv_n,
                                                          step);
  return check_launch("mlp_adam");
}

}  // extern "C"
