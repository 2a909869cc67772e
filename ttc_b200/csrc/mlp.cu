// Kernels of the learned schedule selector: a small fp32 MLP is trained and evaluated on the GPU with
// these. The matrices are tiny (batch x 128), so what bounds a step is launches and latency, not
// arithmetic (0.3 GFLOP): the whole forward pass of a block of rows is one kernel, and so is the
// backward pass, whose weight gradients (sums over all rows) are split over every CTA. All arithmetic
// stays fp32 FFMA; the tiled GEMM serves other hidden sizes.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "../../include/ttcb200_mlp.h"

extern "C" void ttcb_internal_set_error(const char* msg);

namespace {

constexpr int TM = 64, TN = 64, TK = 16;  // block tile
constexpr int RM = 4, RN = 4;             // per-thread tile; 16 x 16 threads

// C = op(A) op(B) (+ bias) (relu). Row-major storage.
__global__ void __launch_bounds__(256) gemm_kernel(int transA, int transB, int M, int N, int K,
                                                   const float* __restrict__ A, int lda,
                                                   const float* __restrict__ B, int ldb, float* __restrict__ C,
                                                   int ldc, const float* __restrict__ bias, int relu) {
  __shared__ float As[TK][TM + 1];
  __shared__ float Bs[TK][TN + 1];
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  float acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += TK) {
    for (int e = threadIdx.x; e < TM * TK; e += 256) {
      const int mm = e / TK, kk = e % TK;
      const int m = m0 + mm, k = k0 + kk;
      float v = 0.f;
      if (m < M && k < K) v = transA ? A[(size_t)k * lda + m] : A[(size_t)m * lda + k];
      As[kk][mm] = v;
    }
    for (int e = threadIdx.x; e < TN * TK; e += 256) {
      const int nn = e % TN, kk = e / TN;
      const int n = n0 + nn, k = k0 + kk;
      float v = 0.f;
      if (n < N && k < K) v = transB ? B[(size_t)n * ldb + k] : B[(size_t)k * ldb + n];
      Bs[kk][nn] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < TK; ++kk) {
      float a[RM], b[RN];
#pragma unroll
      for (int i = 0; i < RM; ++i) a[i] = As[kk][ty * RM + i];
#pragma unroll
      for (int j = 0; j < RN; ++j) b[j] = Bs[kk][tx * RN + j];
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = m0 + ty * RM + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < RN; ++j) {
      const int n = n0 + tx * RN + j;
      if (n >= N) continue;
      float v = acc[i][j] + (bias ? bias[n] : 0.f);
      if (relu) v = fmaxf(v, 0.f);
      C[(size_t)m * ldc + n] = v;
    }
  }
}

__global__ void relu_grad_kernel(const float* __restrict__ Y, const float* __restrict__ dY, float* __restrict__ dZ,
                                 int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dZ[i] = Y[i] > 0.f ? dY[i] : 0.f;
}

__global__ void colsum_kernel(const float* __restrict__ X, int M, int N, float* __restrict__ out) {
  const int n = blockIdx.x;
  float s = 0.f;
  for (int m = threadIdx.x; m < M; m += blockDim.x) s += X[(size_t)m * N + n];
  __shared__ float red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = red[0];
}

__global__ void mse_kernel(const float* __restrict__ pred, const float* __restrict__ target, int n,
                           float* __restrict__ dpred, float* __restrict__ loss) {
  __shared__ float red[256];
  float s = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float d = pred[i] - target[i];
    dpred[i] = 2.f * d / (float)n;
    s += d * d;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, red[0] / (float)n);
}

// The same in one CTA, which needs no zeroed loss: the batches of a training run (2048 rows) are far from
// filling more.
constexpr int kMseOneCta = 16384;
__global__ void __launch_bounds__(1024) mse_one_kernel(const float* __restrict__ pred, const float* __restrict__ target,
                                                       int n, float* __restrict__ dpred, float* __restrict__ loss) {
  __shared__ float red[32];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const float d = pred[i] - target[i];
    dpred[i] = 2.f * d / (float)n;
    s += d * d;
  }
  for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
    for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
    if (threadIdx.x == 0) loss[0] = s / (float)n;
  }
}

// ------------------------------------------------------------------------------------------------
// The network's passes (three layers, hidden size kH) over blocks of kR rows, one block per CTA: 2048
// rows give 128 CTAs. The layers of a row block follow each other in shared memory, so a pass is one
// launch, bound by the shared-memory reads of its operands (each thread holds one column of kR / 2
// rows, so a weight is read once per eight FFMAs and a row value is a broadcast) and by bringing the
// weights from L2. A training step of 2048 rows x 96 features took 1075 us as 22 launches; its weight
// gradients alone ran on four CTAs that each walked all 2048 rows. Now forward 10, loss 4, backward 22 and
// Adam 4 us on the device, in 5 launches.
constexpr int kH = 128, kR = 16, kT = 256;
constexpr int kMaxIn = 192;      // input features: W1, W2 and the rows fit shared memory
constexpr int kCluster = 4;      // CTAs whose weight gradients are summed through distributed shared memory (a cluster of
                                 // 8 leaves SMs of a GPC unused: 34 against 20 us for 2048 rows)
constexpr int kMaxClusters = 64; // per launch; longer batches loop
constexpr int kW2Pitch = kH + 4; // a row per lane without bank conflicts

__host__ __device__ constexpr int pad4(int n) { return (n + 3) & ~3; }
__host__ __device__ constexpr int grad_size(int nin) { return nin * kH + kH + kH * kH + kH + kH + 1; }
__host__ __device__ constexpr int forward_smem(int nin) { return 4 * (pad4(nin) * kH + kH * kH + kR * pad4(nin) + kR * kH); }
__host__ __device__ constexpr int backward_smem(int nin) {
  return 4 * (kH * kW2Pitch + kH * kH + kR * (pad4(nin) + 4 * kH) + kR + 3 * kH + 4);
}

// Asynchronous copies to shared memory: all of a CTA's operands are in flight at once, without registers.
__device__ __forceinline__ void copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_landed() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Rows [0, n) of kH floats to shared memory with the given pitch; rows [n, m) become zero.
__device__ __forceinline__ void load_wide(float* dst, int pitch, const float* __restrict__ src, int n, int m) {
  if (reinterpret_cast<uintptr_t>(src) % 16 == 0) {
    for (int e = threadIdx.x; e < n * (kH / 4); e += kT)
      copy16(dst + e / (kH / 4) * pitch + e % (kH / 4) * 4, src + (size_t)e * 4);
  } else {
    for (int e = threadIdx.x; e < n * kH; e += kT) copy4(dst + e / kH * pitch + e % kH, src + e);
  }
  for (int e = n * kH + threadIdx.x; e < m * kH; e += kT) dst[e / kH * pitch + e % kH] = 0.f;
}

// n rows of `width` floats (row-major, dense) to shared memory with the given pitch; zero to kR rows and
// `pitch` columns.
__device__ __forceinline__ void load_narrow(float* dst, int pitch, const float* __restrict__ src, int width, int n) {
  const int lane = threadIdx.x % 32;
  for (int r = threadIdx.x / 32; r < kR; r += kT / 32)
    for (int c = lane; c < pitch; c += 32) {
      if (r < n && c < width)
        copy4(dst + r * pitch + c, src + (size_t)r * width + c);
      else
        dst[r * pitch + c] = 0.f;
    }
}

// Column tid % kH of eight rows (those of the thread's half) of in (kR x K, K a multiple of 4) * W (K x kH).
__device__ __forceinline__ void dense_rows(const float* in, int pitch, int K, const float* W, float acc[kR / 2]) {
  const int j = threadIdx.x % kH, r0 = threadIdx.x / kH * (kR / 2);
#pragma unroll
  for (int r = 0; r < kR / 2; ++r) acc[r] = 0.f;
  for (int k = 0; k < K; k += 4) {
    float w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = W[(k + q) * kH + j];
#pragma unroll
    for (int r = 0; r < kR / 2; ++r) {
      const float4 x = *reinterpret_cast<const float4*>(in + (r0 + r) * pitch + k);
      acc[r] = fmaf(x.x, w[0], acc[r]);
      acc[r] = fmaf(x.y, w[1], acc[r]);
      acc[r] = fmaf(x.z, w[2], acc[r]);
      acc[r] = fmaf(x.w, w[3], acc[r]);
    }
  }
}

__global__ void __launch_bounds__(kT) mlp_forward_kernel(const float* __restrict__ X, int rows, int nin,
                                                         const float* __restrict__ W1, const float* __restrict__ b1,
                                                         const float* __restrict__ W2, const float* __restrict__ b2,
                                                         const float* __restrict__ W3, const float* __restrict__ b3,
                                                         float* __restrict__ H1, float* __restrict__ H2,
                                                         float* __restrict__ out) {
  extern __shared__ __align__(16) float sm[];
  const int np = pad4(nin);
  float* w1 = sm;
  float* w2 = w1 + np * kH;
  float* xs = w2 + kH * kH;
  float* hs = xs + kR * np;
  const int r0 = blockIdx.x * kR, tid = threadIdx.x;
  const int n = min(kR, rows - r0);
  load_narrow(xs, np, X + (size_t)r0 * nin, nin, n);
  load_wide(w1, kH, W1, nin, np);
  load_wide(w2, kH, W2, kH, kH);
  copies_landed();
  __syncthreads();
  const int j = tid % kH, rh = tid / kH * (kR / 2);
  float acc[kR / 2];
  dense_rows(xs, np, np, w1, acc);
  const float c1 = __ldg(b1 + j), c2 = __ldg(b2 + j), v3 = __ldg(W3 + j);
#pragma unroll
  for (int r = 0; r < kR / 2; ++r) {
    const float h = fmaxf(acc[r] + c1, 0.f);
    hs[(rh + r) * kH + j] = h;
    if (r0 + rh + r < rows) H1[(size_t)(r0 + rh + r) * kH + j] = h;
  }
  __syncthreads();
  dense_rows(hs, kH, kH, w2, acc);
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kR / 2; ++r) {
    const float h = fmaxf(acc[r] + c2, 0.f);
    hs[(rh + r) * kH + j] = h * v3;
    if (r0 + rh + r < rows) H2[(size_t)(r0 + rh + r) * kH + j] = h;
  }
  __syncthreads();
  const int lane = tid % 32;
  for (int r = tid / 32; r < kR; r += kT / 32) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < kH / 32; ++q) s += hs[r * kH + q * 32 + lane];
    for (int w = 16; w > 0; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
    if (lane == 0 && r0 + r < rows) out[r0 + r] = s + __ldg(b3);
  }
}

// buf (kH x kH) = A^T B for A (kR x kH columns from a0 of pitch pa, zero past `width`) and B (kR x kH).
__device__ __forceinline__ void outer_rows(const float* A, int pa, int a0, int width, const float* B, float* buf) {
  const int ty = threadIdx.x / 16 * 4, tx = threadIdx.x % 16 * 4;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
#pragma unroll 4
  for (int r = 0; r < kR; ++r) {
    float a[8], b[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = a0 + h * (kH / 2) + ty;
      const float4 x = c < width ? *reinterpret_cast<const float4*>(A + r * pa + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 y = *reinterpret_cast<const float4*>(B + r * kH + h * (kH / 2) + tx);
      a[4 * h] = x.x, a[4 * h + 1] = x.y, a[4 * h + 2] = x.z, a[4 * h + 3] = x.w;
      b[4 * h] = y.x, b[4 * h + 1] = y.y, b[4 * h + 2] = y.z, b[4 * h + 3] = y.w;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      *reinterpret_cast<float4*>(buf + ((i / 4) * (kH / 2) + ty + i % 4) * kH + h * (kH / 2) + tx) =
          make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]);
}

// Backward pass: every CTA forms the gradients of its rows; the kCluster CTAs of a cluster sum theirs
// through distributed shared memory, each a slice of the rows of the matrix, in a fixed order, and write
// one partial gradient per cluster (part[cluster][grad_size]), which grad_sum_kernel adds up.
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kT)
    mlp_backward_kernel(const float* __restrict__ X, int rows, int nin, const float* __restrict__ W2,
                        const float* __restrict__ W3, const float* __restrict__ H1, const float* __restrict__ H2,
                        const float* __restrict__ dout, float* __restrict__ part) {
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) float sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int np = pad4(nin), tid = threadIdx.x, rank = (int)cluster.block_rank();
  float* w2 = sm;
  float* buf = w2 + kH * kW2Pitch;
  float* xs = buf + kH * kH;
  float* h1 = xs + kR * np;
  float* h2 = h1 + kR * kH;
  float* z1 = h2 + kR * kH;
  float* z2 = z1 + kR * kH;
  float* vec = z2 + kR * kH;  // b1, b2, W3, b3 gradients of the CTA's rows
  float* dv = vec + 3 * kH + 4;
  float* mine = part + (size_t)(blockIdx.x / kCluster) * grad_size(nin);
  const int oW2 = nin * kH + kH, oW3 = oW2 + kH * kH + kH;
  load_wide(w2, kW2Pitch, W2, kH, kH);
  const int nblocks = (rows + kR - 1) / kR;
  // the same count for every CTA of a cluster: they meet at the cluster's barriers
  const int c0 = (int)(blockIdx.x / kCluster) * kCluster;
  for (int blk = c0; blk < nblocks; blk += (int)gridDim.x) {
    const bool first = blk == c0;
    const int r0 = (blk + rank) * kR, n = max(0, min(kR, rows - r0));
    load_wide(h2, kH, H2 + (size_t)r0 * kH, n, kR);
    load_wide(h1, kH, H1 + (size_t)r0 * kH, n, kR);
    load_narrow(xs, np, X + (size_t)r0 * nin, nin, n);
    copies_landed();
    if (tid < kR) dv[tid] = r0 + tid < rows ? __ldg(dout + r0 + tid) : 0.f;
    __syncthreads();
    for (int e = tid; e < kR * kH; e += kT) z2[e] = h2[e] > 0.f ? dv[e / kH] * __ldg(W3 + e % kH) : 0.f;
    __syncthreads();
    {
      // z1 = (z2 W2^T) where h1 > 0: column i of eight rows per thread
      const int i = tid % kH, rh = tid / kH * (kR / 2);
      float acc[kR / 2];
#pragma unroll
      for (int r = 0; r < kR / 2; ++r) acc[r] = 0.f;
      for (int k = 0; k < kH; k += 4) {
        const float4 w = *reinterpret_cast<const float4*>(w2 + i * kW2Pitch + k);
#pragma unroll
        for (int r = 0; r < kR / 2; ++r) {
          const float4 z = *reinterpret_cast<const float4*>(z2 + (rh + r) * kH + k);
          acc[r] = fmaf(z.x, w.x, acc[r]);
          acc[r] = fmaf(z.y, w.y, acc[r]);
          acc[r] = fmaf(z.z, w.z, acc[r]);
          acc[r] = fmaf(z.w, w.w, acc[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < kR / 2; ++r) z1[(rh + r) * kH + i] = h1[(rh + r) * kH + i] > 0.f ? acc[r] : 0.f;
    }
    __syncthreads();
    if (tid < kH) {
      float g1 = 0.f, g2 = 0.f, g3 = 0.f, s = 0.f;
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        g1 += z1[r * kH + tid];
        g2 += z2[r * kH + tid];
        g3 = fmaf(h2[r * kH + tid], dv[r], g3);
        s += dv[r];
      }
      vec[tid] = g1;
      vec[kH + tid] = g2;
      vec[2 * kH + tid] = g3;
      if (tid == 0) vec[3 * kH] = s;
    }
    // W2's gradient, then W1's in pieces of kH input features
    for (int a0 = -kH; a0 < nin; a0 += kH) {
      const bool second = a0 < 0;
      if (second)
        outer_rows(h1, kH, 0, kH, z2, buf);
      else
        outer_rows(xs, np, a0, np, z1, buf);
      cluster.sync();
      float* dst = mine + (second ? oW2 : a0 * kH);
      const int limit = second ? kH : min(kH, nin - a0);
      constexpr int kSlice = kH / kCluster;
#pragma unroll
      for (int e0 = 0; e0 < kSlice * kH; e0 += 4 * kT) {
        const int at = rank * kSlice * kH + e0 + 4 * tid;
        if (at / kH >= limit) continue;
        float4 v[kCluster];
#pragma unroll
        for (int c = 0; c < kCluster; ++c) v[c] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(buf, c) + at);
        float s[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
        for (int c = 1; c < kCluster; ++c) s[0] += v[c].x, s[1] += v[c].y, s[2] += v[c].z, s[3] += v[c].w;
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[at + q] = first ? s[q] : dst[at + q] + s[q];
      }
      if (second && rank == 0) {
        for (int e = tid; e < 3 * kH + 1; e += kT) {
          float s = 0.f;
#pragma unroll
          for (int c = 0; c < kCluster; ++c) s += cluster.map_shared_rank(vec, c)[e];
          const int to = e < kH ? nin * kH + e : e < 2 * kH ? oW2 + kH * kH + e - kH : oW3 + e - 2 * kH;
          mine[to] = first ? s : mine[to] + s;
        }
      }
      cluster.sync();
    }
  }
}

__global__ void grad_sum_kernel(const float* __restrict__ part, int n, int parts, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.f;
#pragma unroll 8
  for (int c = 0; c < parts; ++c) s += __ldg(part + (size_t)c * n + i);
  out[i] = s;
}

// The parameter tensors of one optimiser step, in one launch (blockIdx.y: the tensor).
constexpr int kMaxTensors = 8;
struct AdamTensors {
  float* p[kMaxTensors];
  const float* g[kMaxTensors];
  float* m[kMaxTensors];
  float* v[kMaxTensors];
  int n[kMaxTensors];
};

// wd: L2 weight decay, added to the gradient before the moments (wd * p).
__global__ void adam_kernel(AdamTensors t, float lr, float b1, float b2, float eps, float c1, float c2, float wd) {
  float* __restrict__ p = t.p[blockIdx.y];
  const float* __restrict__ g = t.g[blockIdx.y];
  float* __restrict__ m = t.m[blockIdx.y];
  float* __restrict__ v = t.v[blockIdx.y];
  const int n = t.n[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i] + wd * p[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

ttcb_status check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return TTCB_OK;
  std::string m = std::string(what) + ": " + cudaGetErrorString(e);
  ttcb_internal_set_error(m.c_str());
  return TTCB_ERR_CUDA;
}

int grid_for(int n) { return std::max(1, std::min((n + 255) / 256, 148 * 8)); }

}  // namespace

extern "C" {

ttcb_status ttcb_mlp_gemm(int transA, int transB, int M, int N, int K, const float* A, int lda, const float* B,
                          int ldb, float* C, int ldc, const float* bias, int relu, ttcb_stream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C) {
    ttcb_internal_set_error("ttcb_mlp_gemm: bad arguments");
    return TTCB_ERR_INVALID_ARG;
  }
  dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
  gemm_kernel<<<grid, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(transA, transB, M, N, K, A, lda, B, ldb, C,
                                                                       ldc, bias, relu);
  return check_launch("ttcb_mlp_gemm");
}

ttcb_status ttcb_mlp_relu_grad(const float* Y, const float* dY, float* dZ, int n, ttcb_stream_t stream) {
  if (n <= 0) return TTCB_OK;
  relu_grad_kernel<<<grid_for(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(Y, dY, dZ, n);
  return check_launch("ttcb_mlp_relu_grad");
}

ttcb_status ttcb_mlp_colsum(const float* X, int M, int N, float* out, ttcb_stream_t stream) {
  if (M <= 0 || N <= 0) return TTCB_OK;
  colsum_kernel<<<N, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(X, M, N, out);
  return check_launch("ttcb_mlp_colsum");
}

ttcb_status ttcb_mlp_mse(const float* pred, const float* target, int n, float* dpred, float* loss,
                         ttcb_stream_t stream) {
  if (n <= 0) return TTCB_OK;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (n <= kMseOneCta) {
    mse_one_kernel<<<1, 1024, 0, s>>>(pred, target, n, dpred, loss);
    return check_launch("ttcb_mlp_mse");
  }
  cudaMemsetAsync(loss, 0, sizeof(float), s);
  mse_kernel<<<grid_for(n), 256, 0, s>>>(pred, target, n, dpred, loss);
  return check_launch("ttcb_mlp_mse");
}

int ttcb_mlp_passes_max_features(void) { return kMaxIn; }

ttcb_status ttcb_mlp_forward(int rows, int nin, const float* X, const float* const* params, float* H1, float* H2,
                             float* out, ttcb_stream_t stream) {
  if (rows <= 0 || nin <= 0 || nin > kMaxIn || !X || !params || !H1 || !H2 || !out) {
    ttcb_internal_set_error("ttcb_mlp_forward: bad arguments");
    return TTCB_ERR_INVALID_ARG;
  }
  cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       forward_smem(kMaxIn));
  if (e == cudaSuccess) {
    mlp_forward_kernel<<<(rows + kR - 1) / kR, kT, forward_smem(nin), reinterpret_cast<cudaStream_t>(stream)>>>(
        X, rows, nin, params[0], params[1], params[2], params[3], params[4], params[5], H1, H2, out);
  }
  return check_launch("ttcb_mlp_forward");
}

static int backward_clusters(int rows) {
  return std::min((((rows + kR - 1) / kR) + kCluster - 1) / kCluster, kMaxClusters);
}

size_t ttcb_mlp_backward_workspace(int rows, int nin) {
  if (rows <= 0 || nin <= 0 || nin > kMaxIn) return 0;
  return sizeof(float) * (size_t)backward_clusters(rows) * grad_size(nin);
}

ttcb_status ttcb_mlp_backward(int rows, int nin, const float* X, const float* const* params, const float* H1,
                              const float* H2, const float* dout, float* grads, void* workspace,
                              ttcb_stream_t stream) {
  if (rows <= 0 || nin <= 0 || nin > kMaxIn || !X || !params || !H1 || !H2 || !dout || !grads || !workspace) {
    ttcb_internal_set_error("ttcb_mlp_backward: bad arguments");
    return TTCB_ERR_INVALID_ARG;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e = cudaFuncSetAttribute(mlp_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       backward_smem(kMaxIn));
  if (e == cudaSuccess) {
    const int clusters = backward_clusters(rows), n = grad_size(nin);
    float* part = static_cast<float*>(workspace);
    mlp_backward_kernel<<<clusters * kCluster, kT, backward_smem(nin), s>>>(X, rows, nin, params[2], params[4], H1, H2,
                                                                            dout, part);
    grad_sum_kernel<<<(n + 255) / 256, 256, 0, s>>>(part, n, clusters, grads);
  }
  return check_launch("ttcb_mlp_backward");
}

ttcb_status ttcb_mlp_adam_multi(int count, float* const* param, const float* const* grad, float* const* m,
                                float* const* v, const int* n, float lr, float beta1, float beta2, float eps,
                                float weight_decay, int t, ttcb_stream_t stream) {
  const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
  for (int k0 = 0; k0 < count; k0 += kMaxTensors) {
    AdamTensors a = {};
    int used = 0, most = 0;
    for (int k = k0; k < count && k < k0 + kMaxTensors; ++k) {
      if (n[k] <= 0) continue;
      a.p[used] = param[k];
      a.g[used] = grad[k];
      a.m[used] = m[k];
      a.v[used] = v[k];
      a.n[used++] = n[k];
      most = std::max(most, n[k]);
    }
    if (!used) continue;
    adam_kernel<<<dim3(grid_for(most), used), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(a, lr, beta1, beta2,
                                                                                               eps, c1, c2,
                                                                                               weight_decay);
  }
  return check_launch("ttcb_mlp_adam");
}

ttcb_status ttcb_mlp_adam_l2(float* param, const float* grad, float* m, float* v, int n, float lr, float beta1,
                             float beta2, float eps, float weight_decay, int t, ttcb_stream_t stream) {
  return ttcb_mlp_adam_multi(1, &param, &grad, &m, &v, &n, lr, beta1, beta2, eps, weight_decay, t, stream);
}

ttcb_status ttcb_mlp_adam(float* param, const float* grad, float* m, float* v, int n, float lr, float beta1,
                          float beta2, float eps, int t, ttcb_stream_t stream) {
  return ttcb_mlp_adam_l2(param, grad, m, v, n, lr, beta1, beta2, eps, 0.f, t, stream);
}

}  // extern "C"
