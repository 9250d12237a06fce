// mlp.cu — learned warm start of the obstacle-contact forces (no counterpart
// in the reference): a per-contact MLP 10 -> 64 -> 64 -> 3 with ReLU, BF16
// weights and activations on the tensor cores (mma.sync m16n8k16, FP32
// accumulation), FP32 master weights, trained on the GPU with Adam on contact
// samples the solver itself logs.
//
// Parameter vector (FP32, kMlpParams values, row-major weights):
//   W1[64][10] b1[64] W2[64][64] b2[64] W3[3][64] b3[3]
// Features of obstacle contact k at vertex i (dimensionless; s_v = |g| dt,
// s_r = m_i |g| dt; B = contact basis with columns n, t, b):
//   x0..2 = B^T (t_n,i - w_k) / s_v   predictor velocity relative to the obstacle
//   x3    = gap_k / 1 cm              signed distance to the obstacle surface
//   x4..6 = B^T R_i / s_r             R_i = world-frame impulse of the contacts of
//                                     vertex i at the end of the previous step
//                                     (0 if it had none)
//   x7    = mu_k
//   x8    = n . g / |g|
//   x9    = 1
// Output y: predicted converged local force r_k / s_r.  The warm start uses
// r = cone(y s_r) instead of the projection in the first PD iteration of the
// step (the fixed point of the iteration is unchanged; only its starting
// force is).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include "device.cuh"
#include "kernels.hpp"
#include "mlp.hpp"

namespace pdfb {

namespace {

constexpr int kIn = kMlpIn, kH = kMlpHidden, kOut = kMlpOut;
constexpr int OW1 = 0, OB1 = OW1 + kH * kIn, OW2 = OB1 + kH, OB2 = OW2 + kH * kH, OW3 = OB2 + kH, OB3 = OW3 + kOut * kH;
static_assert(OB3 + kOut == kMlpParams, "parameter layout");

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// D = A(16x16) B(16x8) + C, BF16 inputs, FP32 accumulate.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Fragment loaders from FP32 matrices in shared memory with arbitrary
// strides: element (r, c) of the logical matrix is at p[r * rs + c * cs].
// A fragment (16 x 16 at (r0, c0)):  a0 = (g, 2t..2t+1), a1 = (g+8, 2t..),
// a2 = (g, 2t+8..), a3 = (g+8, 2t+8..) with g = lane / 4, t = lane % 4.
__device__ __forceinline__ void load_a(uint32_t (&a)[4], const float* p, int rs, int cs, int r0, int c0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto e = [&](int r, int c) { return p[(r0 + r) * rs + (c0 + c) * cs]; };
  a[0] = pack_bf16(e(g, 2 * t), e(g, 2 * t + 1));
  a[1] = pack_bf16(e(g + 8, 2 * t), e(g + 8, 2 * t + 1));
  a[2] = pack_bf16(e(g, 2 * t + 8), e(g, 2 * t + 9));
  a[3] = pack_bf16(e(g + 8, 2 * t + 8), e(g + 8, 2 * t + 9));
}
// B fragment (16 x 8 at (k0, n0)): b0 = (k = 2t..2t+1, n = g), b1 = (k = 2t+8.., n = g).
__device__ __forceinline__ void load_b(uint32_t (&b)[2], const float* p, int ks, int ns, int k0, int n0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto e = [&](int k, int n) { return p[(k0 + k) * ks + (n0 + n) * ns]; };
  b[0] = pack_bf16(e(2 * t, g), e(2 * t + 1, g));
  b[1] = pack_bf16(e(2 * t + 8, g), e(2 * t + 9, g));
}
// C fragment (16 x 8 at (r0, n0)): c0 = (g, 2t), c1 = (g, 2t+1), c2 = (g+8, 2t), c3 = (g+8, 2t+1).
__device__ __forceinline__ void store_c(const float (&c)[4], float* p, int rs, int r0, int n0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  p[(r0 + g) * rs + n0 + 2 * t] = c[0];
  p[(r0 + g) * rs + n0 + 2 * t + 1] = c[1];
  p[(r0 + g + 8) * rs + n0 + 2 * t] = c[2];
  p[(r0 + g + 8) * rs + n0 + 2 * t + 1] = c[3];
}

// Shared-memory image of the parameters, zero padded for the tensor-core tiles:
//   w1[64][16] (k 10..15 zero), w2[64][64], w3[8][64] (rows 3..7 zero), b1, b2, b3[8].
struct SmemWeights {
  float w1[kH * 16];
  float w2[kH * kH];
  float w3[8 * kH];
  float b1[kH], b2[kH], b3[8];
};

__device__ void load_weights(SmemWeights& s, const float* __restrict__ prm) {
  for (int i = threadIdx.x; i < kH * 16; i += blockDim.x) {
    const int n = i / 16, k = i % 16;
    s.w1[i] = k < kIn ? prm[OW1 + n * kIn + k] : 0.f;
  }
  for (int i = threadIdx.x; i < kH * kH; i += blockDim.x) s.w2[i] = prm[OW2 + i];
  for (int i = threadIdx.x; i < 8 * kH; i += blockDim.x) s.w3[i] = i < kOut * kH ? prm[OW3 + i] : 0.f;
  for (int i = threadIdx.x; i < kH; i += blockDim.x) {
    s.b1[i] = prm[OB1 + i];
    s.b2[i] = prm[OB2 + i];
  }
  for (int i = threadIdx.x; i < 8; i += blockDim.x) s.b3[i] = i < kOut ? prm[OB3 + i] : 0.f;
}

// Per-warp activations of 16 samples.
struct WarpBuf {
  float x[16 * 16];   // inputs (cols 10..15 zero)
  float z1[16 * kH];  // pre-activations layer 1 (then gradients)
  float h1[16 * kH];  // relu(z1)
  float z2[16 * kH];
  float h2[16 * kH];
  float y[16 * 8];    // outputs (cols 3..7 zero), then output gradients
};

// Forward pass of 16 samples held by this warp.
__device__ void warp_forward(const SmemWeights& w, WarpBuf& b) {
  // layer 1: z1 = x w1^T + b1   (A = x [16 x 16], B(k, n) = w1[n][k])
  for (int nt = 0; nt < kH / 8; ++nt) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t a[4], bb[2];
    load_a(a, b.x, 16, 1, 0, 0);
    load_b(bb, w.w1, 1, 16, 0, nt * 8);
    mma16816(c, a, bb);
    store_c(c, b.z1, kH, 0, nt * 8);
  }
  __syncwarp();
  for (int i = threadIdx.x & 31; i < 16 * kH; i += 32) {
    const float z = b.z1[i] + w.b1[i % kH];
    b.z1[i] = z;
    b.h1[i] = fmaxf(z, 0.f);
  }
  __syncwarp();
  // layer 2: z2 = h1 w2^T + b2
  for (int nt = 0; nt < kH / 8; ++nt) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    for (int kt = 0; kt < kH / 16; ++kt) {
      uint32_t a[4], bb[2];
      load_a(a, b.h1, kH, 1, 0, kt * 16);
      load_b(bb, w.w2, 1, kH, kt * 16, nt * 8);
      mma16816(c, a, bb);
    }
    store_c(c, b.z2, kH, 0, nt * 8);
  }
  __syncwarp();
  for (int i = threadIdx.x & 31; i < 16 * kH; i += 32) {
    const float z = b.z2[i] + w.b2[i % kH];
    b.z2[i] = z;
    b.h2[i] = fmaxf(z, 0.f);
  }
  __syncwarp();
  // layer 3: y = h2 w3^T + b3   (N padded to 8)
  {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    for (int kt = 0; kt < kH / 16; ++kt) {
      uint32_t a[4], bb[2];
      load_a(a, b.h2, kH, 1, 0, kt * 16);
      load_b(bb, w.w3, 1, kH, kt * 16, 0);
      mma16816(c, a, bb);
    }
    store_c(c, b.y, 8, 0, 0);
  }
  __syncwarp();
  for (int i = threadIdx.x & 31; i < 16 * 8; i += 32) b.y[i] += w.b3[i % 8];
  __syncwarp();
}

// Loads up to 16 samples [s0, s0+16) of X (n x kIn) into the warp buffer.
__device__ void warp_load_x(WarpBuf& b, const float* __restrict__ X, int s0, int n) {
  for (int i = threadIdx.x & 31; i < 16 * 16; i += 32) {
    const int r = i / 16, c = i % 16;
    b.x[i] = (c < kIn && s0 + r < n) ? X[(int64_t)(s0 + r) * kIn + c] : 0.f;
  }
  __syncwarp();
}

// n samples, or min(*n_dev, n) when n_dev is given (count on the device).
__global__ void k_mlp_forward(const float* __restrict__ prm, const float* __restrict__ X, int n,
                              const int* __restrict__ n_dev, float* __restrict__ Y) {
  extern __shared__ unsigned char smem[];
  if (n_dev) n = min(n, *n_dev);
  SmemWeights& w = *reinterpret_cast<SmemWeights*>(smem);
  WarpBuf* bufs = reinterpret_cast<WarpBuf*>(smem + sizeof(SmemWeights));
  load_weights(w, prm);
  __syncthreads();
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  WarpBuf& b = bufs[warp];
  for (int s0 = (blockIdx.x * nw + warp) * 16; s0 < n; s0 += gridDim.x * nw * 16) {
    warp_load_x(b, X, s0, n);
    warp_forward(w, b);
    for (int i = threadIdx.x & 31; i < 16 * kOut; i += 32) {
      const int r = i / kOut, c = i % kOut;
      if (s0 + r < n) Y[(int64_t)(s0 + r) * kOut + c] = b.y[r * 8 + c];
    }
    __syncwarp();
  }
}

// ---- training
//
// Shared-memory matrices of the training kernel are BF16, rows padded by 8
// values: the eight rows of a fragment start in different banks.  ldmatrix
// reads a fragment, .trans the transposed one, so every matrix is stored once.
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm2t(uint32_t (&r)[2], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
// Fragments (fragment loaders above define the element places): A (16 x 16 at
// (r0, k0)) of a matrix stored [r][k], or [k][r] (at); B (16 x 8 at (k0, n0)) of
// a matrix stored [n][k], or [k][n] (bt).
__device__ __forceinline__ void frag_a(uint32_t (&a)[4], const __nv_bfloat16* p, int ld, int r0, int k0) {
  const int lane = threadIdx.x & 31;
  ldsm4(a, p + (r0 + (lane & 15)) * ld + k0 + (lane >> 4) * 8);
}
__device__ __forceinline__ void frag_at(uint32_t (&a)[4], const __nv_bfloat16* p, int ld, int r0, int k0) {
  const int lane = threadIdx.x & 31;
  ldsm4t(a, p + (k0 + (lane & 7) + (lane >> 4) * 8) * ld + r0 + ((lane >> 3) & 1) * 8);
}
__device__ __forceinline__ void frag_b(uint32_t (&b)[2], const __nv_bfloat16* p, int ld, int k0, int n0) {
  const int lane = threadIdx.x & 15;
  ldsm2(b, p + (n0 + (lane & 7)) * ld + k0 + (lane >> 3) * 8);
}
__device__ __forceinline__ void frag_bt(uint32_t (&b)[2], const __nv_bfloat16* p, int ld, int k0, int n0) {
  const int lane = threadIdx.x & 15;
  ldsm2t(b, p + (k0 + lane) * ld + n0);
}
// two values of a C fragment (row, cols n0 + 2t, n0 + 2t + 1)
__device__ __forceinline__ void put2(__nv_bfloat16* p, int ld, int row, int col, float lo, float hi) {
  *reinterpret_cast<uint32_t*>(p + row * ld + col) = pack_bf16(lo, hi);
}

constexpr int kTrainWarps = 8, kTrainRows = 64;  // warps a CTA, samples of a tile
constexpr int kLdW = kH + 8, kLdN = 16 + 8;      // row strides of 64- and 16-wide matrices
static_assert(OW2 % 4 == 0, "16-byte loads of W2");
static_assert(kH == 8 * kTrainWarps && kIn <= 16 && kOut <= 4, "the tiling of k_mlp_grad");
struct TrainSmem {
  __nv_bfloat16 w1[kH * kLdN], w2[kH * kLdW], w3[16 * kLdW];  // [out][in], zero padded
  __nv_bfloat16 x[kTrainRows * kLdN], dy[kTrainRows * kLdN];  // zero padded
  __nv_bfloat16 h1[kTrainRows * kLdW], h2[kTrainRows * kLdW], dz1[kTrainRows * kLdW], dz2[kTrainRows * kLdW];
  float b1[kH], b2[kH], b3[8];
  int last;
};

// Adam (Kingma & Ba 2015) on the FP32 master weights, by the last CTA of the
// gradient kernel; null prm: no update.  done: CTAs that have added their
// gradient (zero before and after a launch).
struct AdamStep {
  float *prm, *m1, *m2;
  unsigned int* done;
  float lr, b1, b2, eps, c1, c2;
};

// Gradient of the mean squared error over the samples idx[0..n) (or 0..n
// when idx is null), accumulated into grad (kMlpParams) and loss; with an Adam
// step, the weights' update and grad cleared for the next launch.
//
// A mini-batch of thousands of samples is a chain of seven small matrix products,
// bound by latency.  A CTA takes 64 samples at a time; warp w owns the 8 hidden
// units [8w, 8w + 8) as columns of every activation and of every weight
// gradient, so a product is 16 independent mma chains across the CTA, the
// weight gradients stay in registers over all the tiles of the CTA, and only
// they meet in atomics, once per CTA.  A batch of 4096 with its Adam step: 18 us;
// with a tile of 16 samples per warp, every weight gradient of every tile added
// by shared-memory atomics, and Adam in a launch of its own: 45 + 4 us (ncu).
__global__ void __launch_bounds__(32 * kTrainWarps)
    k_mlp_grad(const float* prm, const float* __restrict__ X, const float* __restrict__ T,
               const int* __restrict__ idx, int n, float* grad, double* loss, AdamStep adam) {
  extern __shared__ __align__(16) unsigned char smem[];
  TrainSmem& s = *reinterpret_cast<TrainSmem*>(smem);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  const int n0 = 8 * w;
  const float inv_n = 1.f / (float)n;
  griddep_launch_dependents();
  auto sample = [&](int r) -> int64_t { return idx ? idx[r] : r; };
  auto load_x = [&](int s0) {
    for (int i = tid; i < kTrainRows * 16; i += blockDim.x) {
      const int r = i / 16, c = i % 16;
      s.x[r * kLdN + c] = __float2bfloat16(c < kIn && s0 + r < n ? X[sample(s0 + r) * kIn + c] : 0.f);
    }
  };
  // samples and targets do not come from the launch before this one
  load_x(blockIdx.x * kTrainRows);
  for (int i = tid; i < kTrainRows * kLdN; i += blockDim.x) s.dy[i] = __float2bfloat16(0.f);
  griddep_wait();
  for (int i = tid; i < kH * 16; i += blockDim.x) {
    const int r = i / 16, c = i % 16;
    s.w1[r * kLdN + c] = __float2bfloat16(c < kIn ? __ldcg(prm + OW1 + r * kIn + c) : 0.f);
  }
  {
    float4 v[kH * kH / 4 / (32 * kTrainWarps)];
#pragma unroll
    for (int k = 0; k < kH * kH / 4 / (32 * kTrainWarps); ++k)
      v[k] = __ldcg(reinterpret_cast<const float4*>(prm + OW2) + tid + k * 32 * kTrainWarps);
#pragma unroll
    for (int k = 0; k < kH * kH / 4 / (32 * kTrainWarps); ++k) {
      const int i = 4 * (tid + k * 32 * kTrainWarps);
      put2(s.w2, kLdW, i / kH, i % kH, v[k].x, v[k].y);
      put2(s.w2, kLdW, i / kH, i % kH + 2, v[k].z, v[k].w);
    }
  }
  for (int i = tid; i < 16 * kH; i += blockDim.x)
    s.w3[(i / kH) * kLdW + i % kH] = __float2bfloat16(i < kOut * kH ? __ldcg(prm + OW3 + i) : 0.f);
  for (int i = tid; i < kH; i += blockDim.x) {
    s.b1[i] = __ldcg(prm + OB1 + i);
    s.b2[i] = __ldcg(prm + OB2 + i);
  }
  if (tid < 8) s.b3[tid] = tid < kOut ? __ldcg(prm + OB3 + tid) : 0.f;
  float dw1[4] = {}, dw2[4][4] = {}, dw3[4] = {}, db1[2] = {}, db2[2] = {}, db3[2] = {};
  double lsum = 0.;
  for (int s0 = blockIdx.x * kTrainRows; s0 < n; s0 += gridDim.x * kTrainRows) {
    if (s0 != (int)blockIdx.x * kTrainRows) load_x(s0);
    __syncthreads();
    uint32_t a[4], b[2];
    uint32_t on1 = 0, on2 = 0;  // bit 4 mt + c: the unit of C element c is active
    // h1 = relu(x w1^T + b1)
    frag_b(b, s.w1, kLdN, 0, n0);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      frag_a(a, s.x, kLdN, 16 * mt, 0);
      mma16816(c, a, b);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        c[k] += s.b1[n0 + 2 * t + (k & 1)];
        on1 |= (c[k] > 0.f ? 1u : 0u) << (4 * mt + k);
        c[k] = fmaxf(c[k], 0.f);
      }
      put2(s.h1, kLdW, 16 * mt + g, n0 + 2 * t, c[0], c[1]);
      put2(s.h1, kLdW, 16 * mt + g + 8, n0 + 2 * t, c[2], c[3]);
    }
    __syncthreads();
    // h2 = relu(h1 w2^T + b2)
    {
      float c[4][4] = {};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        frag_b(b, s.w2, kLdW, 16 * kt, n0);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          frag_a(a, s.h1, kLdW, 16 * mt, 16 * kt);
          mma16816(c[mt], a, b);
        }
      }
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          c[mt][k] += s.b2[n0 + 2 * t + (k & 1)];
          on2 |= (c[mt][k] > 0.f ? 1u : 0u) << (4 * mt + k);
          c[mt][k] = fmaxf(c[mt][k], 0.f);
        }
        put2(s.h2, kLdW, 16 * mt + g, n0 + 2 * t, c[mt][0], c[mt][1]);
        put2(s.h2, kLdW, 16 * mt + g + 8, n0 + 2 * t, c[mt][2], c[mt][3]);
      }
    }
    __syncthreads();
    // y = h2 w3^T + b3 and dL/dy = 2 (y - t) / n: one row tile each of warps 0 - 3
    if (w < 4) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        frag_a(a, s.h2, kLdW, 16 * w, 16 * kt);
        frag_b(b, s.w3, kLdW, 16 * kt, 0);
        mma16816(c, a, b);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int col = 2 * t + (k & 1), row = 16 * w + g + 8 * (k >> 1);
        float d = 0.f;
        if (col < kOut && s0 + row < n) {
          const float e = c[k] + s.b3[col] - T[sample(s0 + row) * kOut + col];
          lsum += (double)e * e;
          d = 2.f * e * inv_n;
        }
        db3[k & 1] += d;
        c[k] = d;
      }
      put2(s.dy, kLdN, 16 * w + g, 2 * t, c[0], c[1]);
      put2(s.dy, kLdN, 16 * w + g + 8, 2 * t, c[2], c[3]);
    }
    __syncthreads();
    // dz2 = (dy w3) where z2 > 0; dw3 += dy^T h2
    frag_bt(b, s.w3, kLdW, 0, n0);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      frag_a(a, s.dy, kLdN, 16 * mt, 0);
      mma16816(c, a, b);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!(on2 >> (4 * mt + k) & 1)) c[k] = 0.f;
        db2[k & 1] += c[k];
      }
      put2(s.dz2, kLdW, 16 * mt + g, n0 + 2 * t, c[0], c[1]);
      put2(s.dz2, kLdW, 16 * mt + g + 8, n0 + 2 * t, c[2], c[3]);
    }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      frag_at(a, s.dy, kLdN, 0, 16 * kt);
      frag_bt(b, s.h2, kLdW, 16 * kt, n0);
      mma16816(dw3, a, b);
    }
    __syncthreads();
    // dz1 = (dz2 w2) where z1 > 0; dw2 += dz2^T h1
    {
      float c[4][4] = {};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        frag_bt(b, s.w2, kLdW, 16 * kt, n0);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          frag_a(a, s.dz2, kLdW, 16 * mt, 16 * kt);
          mma16816(c[mt], a, b);
        }
      }
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (!(on1 >> (4 * mt + k) & 1)) c[mt][k] = 0.f;
          db1[k & 1] += c[mt][k];
        }
        put2(s.dz1, kLdW, 16 * mt + g, n0 + 2 * t, c[mt][0], c[mt][1]);
        put2(s.dz1, kLdW, 16 * mt + g + 8, n0 + 2 * t, c[mt][2], c[mt][3]);
      }
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        frag_bt(b, s.h1, kLdW, 16 * kt, n0);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
          frag_at(a, s.dz2, kLdW, 16 * mt, 16 * kt);
          mma16816(dw2[mt], a, b);
        }
      }
    }
    __syncthreads();
    // dw1 += dz1^T x: one 16 x 8 tile of it a warp
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      frag_at(a, s.dz1, kLdW, 16 * (w & 3), 16 * kt);
      frag_bt(b, s.x, kLdN, 16 * kt, 8 * (w >> 2));
      mma16816(dw1, a, b);
    }
    __syncthreads();  // the next tile overwrites x
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int row = g + 8 * (k >> 1), col = 2 * t + (k & 1);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) atomicAdd(grad + OW2 + (16 * mt + row) * kH + n0 + col, dw2[mt][k]);
    if (8 * (w >> 2) + col < kIn)
      atomicAdd(grad + OW1 + (16 * (w & 3) + row) * kIn + 8 * (w >> 2) + col, dw1[k]);
    if (row < kOut) atomicAdd(grad + OW3 + row * kH + n0 + col, dw3[k]);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      db1[k] += __shfl_xor_sync(0xffffffffu, db1[k], o);
      db2[k] += __shfl_xor_sync(0xffffffffu, db2[k], o);
      db3[k] += __shfl_xor_sync(0xffffffffu, db3[k], o);
    }
    if (g == 0) {
      atomicAdd(grad + OB1 + n0 + 2 * t + k, db1[k]);
      atomicAdd(grad + OB2 + n0 + 2 * t + k, db2[k]);
      if (w < 4 && 2 * t + k < kOut) atomicAdd(grad + OB3 + 2 * t + k, db3[k]);
    }
  }
  for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
  if (lane == 0 && w < 4) atomicAdd(loss, lsum * inv_n);
  if (!adam.prm) return;
  __threadfence();
  __syncthreads();
  if (tid == 0) s.last = atomicAdd(adam.done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s.last) return;
  __threadfence();
  auto update = [&](float d, float& m1, float& m2, float& p) {
    const float m = adam.b1 * m1 + (1.f - adam.b1) * d;
    const float v = adam.b2 * m2 + (1.f - adam.b2) * d * d;
    m1 = m;
    m2 = v;
    p -= adam.lr * (m / adam.c1) / (sqrtf(v / adam.c2) + adam.eps);
  };
  // four parameters a load, every load of the thread in flight
  constexpr int kQuads = kMlpParams / 4, kRounds = (kQuads + 32 * kTrainWarps - 1) / (32 * kTrainWarps);
  float4 d4[kRounds], m4[kRounds], v4[kRounds], p4[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int i = tid + k * 32 * kTrainWarps;
    if (i < kQuads) {
      d4[k] = __ldcg(reinterpret_cast<const float4*>(grad) + i);
      m4[k] = __ldcg(reinterpret_cast<const float4*>(adam.m1) + i);
      v4[k] = __ldcg(reinterpret_cast<const float4*>(adam.m2) + i);
      p4[k] = __ldcg(reinterpret_cast<const float4*>(adam.prm) + i);
    }
  }
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int i = tid + k * 32 * kTrainWarps;
    if (i < kQuads) {
      update(d4[k].x, m4[k].x, v4[k].x, p4[k].x);
      update(d4[k].y, m4[k].y, v4[k].y, p4[k].y);
      update(d4[k].z, m4[k].z, v4[k].z, p4[k].z);
      update(d4[k].w, m4[k].w, v4[k].w, p4[k].w);
      reinterpret_cast<float4*>(adam.m1)[i] = m4[k];
      reinterpret_cast<float4*>(adam.m2)[i] = v4[k];
      reinterpret_cast<float4*>(adam.prm)[i] = p4[k];
      reinterpret_cast<float4*>(grad)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  if (4 * kQuads + tid < kMlpParams) {
    const int i = 4 * kQuads + tid;
    update(__ldcg(grad + i), adam.m1[i], adam.m2[i], adam.prm[i]);
    grad[i] = 0.f;
  }
  if (tid == 0) *adam.done = 0u;
}

#define CKM(x)                                                                                      \
  do {                                                                                              \
    cudaError_t e_ = (x);                                                                           \
    if (e_ != cudaSuccess) throw std::runtime_error(std::string(#x) + ": " + cudaGetErrorString(e_)); \
  } while (0)

constexpr int kMlpThreads = 128;  // 4 warps
size_t fwd_smem() { return sizeof(SmemWeights) + 4 * sizeof(WarpBuf); }
size_t grad_smem() { return sizeof(TrainSmem); }

template <typename T>
struct DBuf {
  T* p = nullptr;
  explicit DBuf(size_t n) { CKM(cudaMalloc((void**)&p, std::max<size_t>(1, n) * sizeof(T))); }
  ~DBuf() {
    if (p) cudaFree(p);
  }
};

}  // namespace

// cudaFuncSetAttribute is per device: done once per device ordinal.
static void ensure_smem_attrs() {
  static std::atomic<bool> done[64];
  int dev = 0;
  CKM(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || done[dev].load()) return;
  CKM(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem()));
  CKM(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_smem()));
  done[dev].store(true);
}

void mlp_forward_device(const float* prm, const float* X, int n, float* Y, cudaStream_t st) {
  if (n <= 0) return;
  ensure_smem_attrs();
  const int grid = std::min(148 * 4, (n + 63) / 64);
  k_mlp_forward<<<grid, kMlpThreads, fwd_smem(), st>>>(prm, X, n, nullptr, Y);
}

void mlp_forward_counted(const float* prm, const float* X, const int* n_dev, int cap, float* Y, cudaStream_t st) {
  if (cap <= 0) return;
  ensure_smem_attrs();
  const int grid = std::min(148 * 4, (cap + 63) / 64);
  k_mlp_forward<<<grid, kMlpThreads, fwd_smem(), st>>>(prm, X, cap, n_dev, Y);
}

static void launch_grad(const float* prm, const float* X, const float* T, const int* idx, int n, float* grad,
                        double* loss, const AdamStep& adam, cudaStream_t st) {
  ensure_smem_attrs();
  const int grid = std::min(148 * 2, (n + kTrainRows - 1) / kTrainRows);
  launch_dependent(k_mlp_grad, grid, 32 * kTrainWarps, grad_smem(), st, prm, X, T, idx, n, grad, loss, adam);
}

void mlp_grad_device(const float* prm, const float* X, const float* T, const int* idx, int n, float* grad,
                     double* loss, cudaStream_t st) {
  if (n <= 0) return;
  launch_grad(prm, X, T, idx, n, grad, loss, AdamStep{}, st);
}

double mlp_train_device(float* prm, const float* X, const float* T, int n, int epochs, int batch, double lr,
                        uint64_t seed, double* val_loss, cudaStream_t st) {
  if (n < 2 || batch <= 0 || epochs <= 0 || !(lr > 0.)) throw std::invalid_argument("invalid training arguments");
  // seeded shuffle, 90 / 10 split
  std::mt19937_64 rng(seed);
  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  std::shuffle(order.begin(), order.end(), rng);
  const int nval = std::max(1, n / 10), ntr = n - nval;
  DBuf<float> dg(kMlpParams), m1(kMlpParams), m2(kMlpParams);
  DBuf<double> dl(1);
  DBuf<int> didx(n);
  DBuf<unsigned int> done(1);
  CKM(cudaMemsetAsync(dg.p, 0, kMlpParams * sizeof(float), st));
  CKM(cudaMemsetAsync(done.p, 0, sizeof(unsigned int), st));
  CKM(cudaMemsetAsync(m1.p, 0, kMlpParams * sizeof(float), st));
  CKM(cudaMemsetAsync(m2.p, 0, kMlpParams * sizeof(float), st));
  int64_t step = 0;
  double last = 0.;
  std::vector<int> tr(order.begin(), order.begin() + ntr);
  for (int ep = 0; ep < epochs; ++ep) {
    std::shuffle(tr.begin(), tr.end(), rng);
    CKM(cudaMemcpyAsync(didx.p, tr.data(), ntr * sizeof(int), cudaMemcpyHostToDevice, st));
    CKM(cudaMemsetAsync(dl.p, 0, sizeof(double), st));
    int nbatches = 0;
    for (int s0 = 0; s0 < ntr; s0 += batch) {
      const int nb = std::min(batch, ntr - s0);
      const double b1 = 0.9, b2 = 0.999;
      ++step;
      const AdamStep adam{prm,       m1.p,      m2.p, done.p, (float)lr, (float)b1, (float)b2, 1e-8f,
                          (float)(1. - std::pow(b1, (double)step)), (float)(1. - std::pow(b2, (double)step))};
      launch_grad(prm, X, T, didx.p + s0, nb, dg.p, dl.p, adam, st);
      ++nbatches;
    }
    double sum = 0.;
    CKM(cudaMemcpyAsync(&sum, dl.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    CKM(cudaStreamSynchronize(st));  // also keeps `tr` alive until its copy is done
    last = sum / std::max(nbatches, 1);
  }
  // loss on the held-out part
  std::vector<int> va(order.begin() + ntr, order.end());
  CKM(cudaMemcpyAsync(didx.p, va.data(), nval * sizeof(int), cudaMemcpyHostToDevice, st));
  CKM(cudaMemsetAsync(dg.p, 0, kMlpParams * sizeof(float), st));
  CKM(cudaMemsetAsync(dl.p, 0, sizeof(double), st));
  mlp_grad_device(prm, X, T, didx.p, nval, dg.p, dl.p, st);
  double vl = 0.;
  CKM(cudaMemcpyAsync(&vl, dl.p, sizeof(double), cudaMemcpyDeviceToHost, st));
  CKM(cudaStreamSynchronize(st));
  CKM(cudaGetLastError());
  if (val_loss) *val_loss = vl;
  return last;
}

// ---------------------------------------------------------------------------
// Standardised training: per-column mean / standard deviation of the samples
// (double accumulation), standardised copies, training, and the
// standardisation folded back into the first and last layers so that the
// network takes the raw features and returns raw forces.

__global__ void k_col_stats(const float* __restrict__ A, int64_t n, int ncol, double* __restrict__ acc) {
  // acc[2c] += sum of column c, acc[2c+1] += sum of squares (ncol <= 16)
  __shared__ double red[2 * 16];
  for (int i = threadIdx.x; i < 2 * 16; i += blockDim.x) red[i] = 0.;
  __syncthreads();
  double loc[2 * 16];
  for (int c = 0; c < 2 * ncol; ++c) loc[c] = 0.;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x)
    for (int c = 0; c < ncol; ++c) {
      const double v = A[r * ncol + c];
      loc[2 * c] += v;
      loc[2 * c + 1] += v * v;
    }
  for (int c = 0; c < 2 * ncol; ++c) atomicAdd(&red[c], loc[c]);
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * ncol; c += blockDim.x) atomicAdd(&acc[c], red[c]);
}

__global__ void k_standardize(const float* __restrict__ A, int64_t n, int ncol, const float* __restrict__ shift,
                              const float* __restrict__ scale, float* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * ncol;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % ncol);
    out[i] = (A[i] - shift[c]) / scale[c];
  }
}

double mlp_train_standardized(float* prm, const float* X, const float* T, int n, int epochs, int batch, double lr,
                              uint64_t seed, double* val_loss, cudaStream_t st) {
  if (n < 2) throw std::invalid_argument("fewer than 2 samples");
  DBuf<double> acc(2 * (kIn + kOut));
  CKM(cudaMemsetAsync(acc.p, 0, 2 * (kIn + kOut) * sizeof(double), st));
  k_col_stats<<<2 * 148, 256, 0, st>>>(X, n, kIn, acc.p);
  k_col_stats<<<2 * 148, 256, 0, st>>>(T, n, kOut, acc.p + 2 * kIn);
  std::vector<double> a(2 * (kIn + kOut));
  CKM(cudaMemcpyAsync(a.data(), acc.p, a.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  CKM(cudaStreamSynchronize(st));
  std::vector<float> shift(kIn + kOut), scale(kIn + kOut);
  for (int c = 0; c < kIn + kOut; ++c) {
    const double mean = a[2 * c] / n, var = std::max(0., a[2 * c + 1] / n - mean * mean);
    double sd = std::sqrt(var), sh = mean;
    if (sd < 1e-12) {  // constant column (the bias feature): left alone
      sd = 1.;
      if (c < kIn) sh = 0.;
    }
    shift[c] = (float)sh;
    scale[c] = (float)sd;
  }
  DBuf<float> dshift(kIn + kOut), dscale(kIn + kOut), Xs((size_t)n * kIn), Ts((size_t)n * kOut);
  CKM(cudaMemcpyAsync(dshift.p, shift.data(), shift.size() * sizeof(float), cudaMemcpyHostToDevice, st));
  CKM(cudaMemcpyAsync(dscale.p, scale.data(), scale.size() * sizeof(float), cudaMemcpyHostToDevice, st));
  k_standardize<<<4 * 148, 256, 0, st>>>(X, n, kIn, dshift.p, dscale.p, Xs.p);
  k_standardize<<<4 * 148, 256, 0, st>>>(T, n, kOut, dshift.p + kIn, dscale.p + kIn, Ts.p);
  std::vector<float> w(kMlpParams);
  mlp_init_params(w.data(), seed);
  CKM(cudaMemcpyAsync(prm, w.data(), kMlpParams * sizeof(float), cudaMemcpyHostToDevice, st));
  const double tl = mlp_train_device(prm, Xs.p, Ts.p, n, epochs, batch, lr, seed, val_loss, st);
  // fold: W1' = W1 / sigma, b1' = b1 - W1 (mu / sigma); W3' = tau W3, b3' = tau b3 + nu
  CKM(cudaMemcpyAsync(w.data(), prm, kMlpParams * sizeof(float), cudaMemcpyDeviceToHost, st));
  CKM(cudaStreamSynchronize(st));
  for (int h = 0; h < kH; ++h) {
    double b = w[OB1 + h];
    for (int i = 0; i < kIn; ++i) {
      const double wi = w[OW1 + h * kIn + i];
      b -= wi * (double)shift[i] / (double)scale[i];
      w[OW1 + h * kIn + i] = (float)(wi / (double)scale[i]);
    }
    w[OB1 + h] = (float)b;
  }
  for (int o = 0; o < kOut; ++o) {
    const double tau = scale[kIn + o], nu = shift[kIn + o];
    for (int h = 0; h < kH; ++h) w[OW3 + o * kH + h] = (float)(tau * w[OW3 + o * kH + h]);
    w[OB3 + o] = (float)(tau * w[OB3 + o] + nu);
  }
  CKM(cudaMemcpyAsync(prm, w.data(), kMlpParams * sizeof(float), cudaMemcpyHostToDevice, st));
  CKM(cudaStreamSynchronize(st));
  return tl;
}

// ---------------------------------------------------------------------------
// In the step loop.  This file is compiled without FMA contraction, so the
// feature arithmetic below rounds every product and sum separately, in the
// order written (the CPU oracle evaluates the same expressions).

__device__ __forceinline__ double gnorm_of(double gx, double gy, double gz) {
  const double gn = sqrt((gx * gx + gy * gy) + gz * gz);
  return gn > 1e-12 ? gn : 1e-12;
}

// Features of every obstacle contact (definitions at the top of this file).
__global__ void k_mlp_features(DContacts c, const double* __restrict__ tn, const double* __restrict__ mass,
                               const double* __restrict__ rprev, const int* __restrict__ rprev_tag, int tag_prev,
                               double gx, double gy, double gz, double dt, float* __restrict__ X) {
  const int C = *c.n_contacts;
  const double g = gnorm_of(gx, gy, gz);
  const double sv = g * dt;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < C; k += gridDim.x * blockDim.x) {
    const int v = c.c_vertex[k];
    const double* B = c.c_basis + 9 * (int64_t)k;
    const double3 w = ld3(c.c_speed, k);
    const double3 t = ld3(tn, v);
    const double dx = t.x - w.x, dy = t.y - w.y, dz = t.z - w.z;
    float* x = X + (int64_t)k * kIn;
    x[0] = (float)(((B[0] * dx + B[1] * dy) + B[2] * dz) / sv);
    x[1] = (float)(((B[3] * dx + B[4] * dy) + B[5] * dz) / sv);
    x[2] = (float)(((B[6] * dx + B[7] * dy) + B[8] * dz) / sv);
    x[3] = (float)(c.c_gap[k] / 1e-2);
    const double sr = mass[v] * sv;
    if (rprev_tag[v] == tag_prev) {
      const double3 R = ld3(rprev, v);
      x[4] = (float)(((B[0] * R.x + B[1] * R.y) + B[2] * R.z) / sr);
      x[5] = (float)(((B[3] * R.x + B[4] * R.y) + B[5] * R.z) / sr);
      x[6] = (float)(((B[6] * R.x + B[7] * R.y) + B[8] * R.z) / sr);
    } else {
      x[4] = x[5] = x[6] = 0.f;
    }
    x[7] = (float)c.c_mu[k];
    x[8] = (float)(((B[0] * gx + B[1] * gy) + B[2] * gz) / g);
    x[9] = 1.f;
  }
}

// End of step, pass 1: the r_prev memory of every contact vertex starts from zero.
__global__ void k_mlp_rprev_clear(DContacts c, double* __restrict__ rprev, int* __restrict__ rprev_tag, int tag) {
  const int C = *c.n_contacts;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < C; k += gridDim.x * blockDim.x) {
    const int v = c.c_vertex[k];
    st3(rprev, v, make_double3(0., 0., 0.));
    rprev_tag[v] = tag;
  }
}

// Pass 2: world-frame impulse B r of every contact that was active in the last
// iteration, summed per vertex; with a log, (features, r / s_r) samples in
// contact order after the samples already logged (target 0 for a contact
// that took off).
__global__ void k_mlp_record(DContacts c, const double* __restrict__ mass, double* __restrict__ rprev, double gx,
                             double gy, double gz, double dt, const float* __restrict__ X, float* __restrict__ SX,
                             float* __restrict__ ST, const int* __restrict__ n_samples, int cap) {
  const int C = *c.n_contacts;
  const double sv = gnorm_of(gx, gy, gz) * dt;
  const int base = SX ? *n_samples : 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < C; k += gridDim.x * blockDim.x) {
    const int v = c.c_vertex[k];
    const bool active = c.c_active[k] != 0;
    const double3 r = active ? ld3(c.c_force, k) : make_double3(0., 0., 0.);
    if (active) {
      const double* B = c.c_basis + 9 * (int64_t)k;
      atomicAdd(rprev + 3 * (int64_t)v, (B[0] * r.x + B[3] * r.y) + B[6] * r.z);
      atomicAdd(rprev + 3 * (int64_t)v + 1, (B[1] * r.x + B[4] * r.y) + B[7] * r.z);
      atomicAdd(rprev + 3 * (int64_t)v + 2, (B[2] * r.x + B[5] * r.y) + B[8] * r.z);
    }
    if (SX && (int64_t)base + k < cap) {
      const int64_t s = (int64_t)base + k;
      for (int d = 0; d < kIn; ++d) SX[s * kIn + d] = X[(int64_t)k * kIn + d];
      const double sr = mass[v] * sv;
      ST[s * kOut] = (float)(r.x / sr);
      ST[s * kOut + 1] = (float)(r.y / sr);
      ST[s * kOut + 2] = (float)(r.z / sr);
    }
  }
}

__global__ void k_mlp_count(DContacts c, int* n_samples, int cap) {
  const int64_t n = (int64_t)*n_samples + *c.n_contacts;
  *n_samples = (int)(n < cap ? n : cap);
}

void launch_mlp_features(cudaStream_t st, DContacts c, const double* tn, const double* mass, const double* rprev,
                         const int* rprev_tag, int tag_prev, const double g[3], double dt, float* X) {
  k_mlp_features<<<2 * 148, 256, 0, st>>>(c, tn, mass, rprev, rprev_tag, tag_prev, g[0], g[1], g[2], dt, X);
}

void launch_mlp_record(cudaStream_t st, DContacts c, const double* mass, double* rprev, int* rprev_tag, int tag,
                       const double g[3], double dt, const float* X, float* SX, float* ST, int* n_samples, int cap) {
  k_mlp_rprev_clear<<<2 * 148, 256, 0, st>>>(c, rprev, rprev_tag, tag);
  k_mlp_record<<<2 * 148, 256, 0, st>>>(c, mass, rprev, g[0], g[1], g[2], dt, X, SX, ST, n_samples, cap);
  if (SX) k_mlp_count<<<1, 1, 0, st>>>(c, n_samples, cap);
}

}  // namespace pdfb
