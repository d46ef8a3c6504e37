// FP32 kernels of the learned predictor seed: a multilayer perceptron
// (input -> 3 hidden layers with GELU -> output) trained on the GPU.
// Row-major matrices; a batch of B samples is a B x features matrix.
#pragma once

#include <cuda_runtime.h>

#include "adg_gelu.cuh"

namespace adg {
namespace mlp {

enum Epilogue : int {
  EPI_SLICE = 0,      // split K: slice z of C, and the column sums of B behind it
  EPI_BIAS = 1,       // C = acc + bias
  EPI_BIAS_GELU = 2,  // Z = acc + bias (stored to aux), C = gelu(Z)
  EPI_GELU_BWD = 3,   // C = acc * gelu'(aux)   (aux = pre-activation Z)
  EPI_MSE = 4,        // Y = acc + bias; C = (2 / (M N)) (Y - target), loss += sum (Y - target)^2
};

struct GemmArgs {
  int M, N, K;
  const float *A, *B;
  float* C;
  const float* bias;
  float* aux;
  const int* rows;      // optional: sample r of A is stored in row rows[r]
  const float* target;  // EPI_MSE
  const int* target_rows;  // the same for the targets
  double* loss;
  int kchunk;           // EPI_SLICE: K range of a slice, a multiple of 16
};

// Packed pairs of FP32 FMAs (one issue slot, each IEEE as fmaf).
__device__ __forceinline__ unsigned long long pair2(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

constexpr int kGemmTile = 64, kGemmThreads = 256;
constexpr int kGemmK = 16;  // K step

// The (R0 .. R0 + BT) x (k0 .. k0 + 16) tile of an operand into registers, four
// floats a load where `vec` allows it (row stride and base multiples of 16
// bytes), zeros outside.  KC: stored rows x K (rows: sample rows through idx),
// else K x rows (idx indexes K).
template <bool KC, int BT, int NT>
__device__ __forceinline__ void gemm_fetch(float4* r, const float* X, int R0, int R, int ld, int k0, int kend,
                                           const int* idx, bool vec) {
#pragma unroll
  for (int i = 0; i < BT * kGemmK / 4 / NT; ++i) {
    const int f = threadIdx.x + i * NT;
    const int row = R0 + (KC ? f / 4 : f % (BT / 4) * 4), k = k0 + (KC ? f % 4 * 4 : f / (BT / 4));
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (row < R && k < kend) {
      const int line = KC ? row : k;
      const float* p = X + (size_t)(idx ? idx[line] : line) * ld + (KC ? k : row);
      const int left = KC ? kend - k : R - row;
      if (vec && left >= 4) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(p));
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (c < left) v[c] = __ldg(p + c);
      }
    }
    r[i] = make_float4(v[0], v[1], v[2], v[3]);
  }
}
template <bool KC, int BT, int NT>
__device__ __forceinline__ void gemm_stage(const float4* r, float (*S)[BT + 4]) {
#pragma unroll
  for (int i = 0; i < BT * kGemmK / 4 / NT; ++i) {
    const int f = threadIdx.x + i * NT;
    if constexpr (KC) {
      const int m = f / 4, k = f % 4 * 4;
      S[k][m] = r[i].x, S[k + 1][m] = r[i].y, S[k + 2][m] = r[i].z, S[k + 3][m] = r[i].w;
    } else {
      *reinterpret_cast<float4*>(&S[f / (BT / 4)][f % (BT / 4) * 4]) = r[i];
    }
  }
}

// C[M x N] = op(A) op(B) with op(A) = A[M x K] (TA = 0) or A^T with A[K x M]
// (TA = 1), op(B) = B[K x N] (TB = 0) or B^T with B[N x K] (TB = 1), FP32
// throughout, each output one chain of FMAs in the order of K (of its slice).
//
// 64 x 64 tile per block of 256 threads, 4 x 4 outputs a thread.  Bound by the
// latency of shared memory (56 % of its cycles, packed FMAs 46 % of the FP32
// pipe's) and, at the ends, of memory: four floats a load and the tile after
// next on its way while one is multiplied, where single floats were loaded and
// then multiplied in turn.  Network 41-128-128-128-80, a layer forward /
// backward / weight gradient: 16384 samples 38 / 45 / 57 us -> 18 / 20 / 16,
// 1000 samples 19 / 20 / 62 -> 7 / 8 / 6; an epoch of 16384 780 -> 266 us.
// Larger tiles gained nothing: 64 x 128 (4 x 8 a thread) 17 / 20 / 15 us, but
// 12 / 13 / 8 at 1000 samples; 128 x 128 19 / 25 / 16; 64 x 64 with 8 x 4 a
// thread 17 / 20 / 15 and 9 / 10 / 7.
// Split K (the weight gradients, K the samples): a slice a block, so an output
// of 128 x 128 fills the chip; k_adam adds the slices.
template <int TA, int TB, int EPI>
__global__ void __launch_bounds__(kGemmThreads) k_sgemm(GemmArgs g) {
  constexpr int BM = kGemmTile, BN = kGemmTile, TM = 4, TN = 4, NT = kGemmThreads, BK = kGemmK;
  constexpr int LA = BM + 4, LB = BN + 4, TX = BN / TN;
  __shared__ __align__(16) float smem[BM * LB > 2 * BK * (LA + LB) ? BM * LB : 2 * BK * (LA + LB)];
  auto As = reinterpret_cast<float(*)[BK][LA]>(smem);
  auto Bs = reinterpret_cast<float(*)[BK][LB]>(smem + 2 * BK * LA);
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int kz0 = EPI == EPI_SLICE ? blockIdx.z * g.kchunk : 0;
  const int kz1 = EPI == EPI_SLICE ? min(g.K, kz0 + g.kchunk) : g.K;
  const int lda = TA ? g.M : g.K, ldb = TB ? g.K : g.N;
  const bool va = (lda & 3) == 0 && (reinterpret_cast<size_t>(g.A) & 15) == 0;
  const bool vb = (ldb & 3) == 0 && (reinterpret_cast<size_t>(g.B) & 15) == 0;
  const bool vc = (g.N & 3) == 0 && ((reinterpret_cast<size_t>(g.C) | reinterpret_cast<size_t>(g.aux) |
                                      reinterpret_cast<size_t>(g.target)) & 15) == 0;
  unsigned long long acc[TM][TN / 2] = {};
  float csum = 0.f;  // EPI_SLICE: column tid of B
  // tile t is in stage t % 2, t + 1 on its way in the other set of registers
  float4 ra[2][BM * BK / 4 / NT], rb[2][BN * BK / 4 / NT];
  auto fetch = [&](int r, int k0) {
    gemm_fetch<!TA, BM, NT>(ra[r], g.A, m0, g.M, lda, k0, kz1, g.rows, va);
    gemm_fetch<TB, BN, NT>(rb[r], g.B, n0, g.N, ldb, k0, kz1, nullptr, vb);
  };
  auto stage = [&](int r) {
    gemm_stage<!TA, BM, NT>(ra[r], As[r]);
    gemm_stage<TB, BN, NT>(rb[r], Bs[r]);
  };
  fetch(0, kz0);
  if (kz0 + BK < kz1) fetch(1, kz0 + BK);
  stage(0);
  __syncthreads();
  for (int kt = kz0; kt < kz1; kt += 2 * BK) {
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int k0 = kt + s * BK;
      if (k0 >= kz1) break;
      if (k0 + 2 * BK < kz1) fetch(s, k0 + 2 * BK);
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        unsigned long long a[TM], b[TN / 2];
        const float4 q = *reinterpret_cast<const float4*>(&As[s][k][ty * 4]);
        a[0] = pair2(q.x), a[1] = pair2(q.y), a[2] = pair2(q.z), a[3] = pair2(q.w);
        const ulonglong2 p = *reinterpret_cast<const ulonglong2*>(&Bs[s][k][tx * 4]);
        b[0] = p.x, b[1] = p.y;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(a[i], b[j], acc[i][j]);
      }
      if (EPI == EPI_SLICE && blockIdx.y == 0 && tid < BN) {
#pragma unroll
        for (int k = 0; k < BK; ++k) csum += Bs[s][k][tid];
      }
      if (k0 + BK < kz1) stage(s ^ 1);
      __syncthreads();
    }
  }
  float* C = g.C;
  if (EPI == EPI_SLICE) {
    C += (size_t)blockIdx.z * ((size_t)g.M * g.N + g.N);
    if (blockIdx.y == 0 && tid < BN && n0 + tid < g.N) C[(size_t)g.M * g.N + n0 + tid] = csum;
  }
  // The tile through shared memory: whole rows to memory, and a short loop for
  // what follows the sum (unrolled over a thread's outputs it did not fit the
  // instruction caches: 26 us a layer of 16384 samples).
  double loss = 0.0;
#pragma unroll
  for (int i = 0; i < TM; ++i)
    *reinterpret_cast<ulonglong2*>(&smem[(ty * 4 + i) * LB + tx * 4]) =
        make_ulonglong2(acc[i][0], acc[i][1]);
  __syncthreads();
#pragma unroll 4
  for (int f0 = 0; f0 < BM * BN / 4; f0 += NT) {
    const int f = f0 + tid, r = f / (BN / 4), c4 = f % (BN / 4) * 4, gm = m0 + r, gn = n0 + c4;
    if (gm >= g.M || gn >= g.N) continue;
    const size_t o = (size_t)gm * g.N + gn;
    const int left = min(4, g.N - gn);
    const float4 q = *reinterpret_cast<const float4*>(&smem[r * LB + c4]);
    float v[4] = {q.x, q.y, q.z, q.w}, z[4] = {0.f, 0.f, 0.f, 0.f};
    if (EPI == EPI_GELU_BWD || EPI == EPI_MSE) {
      const float* p = EPI == EPI_MSE ? g.target + (size_t)(g.target_rows ? g.target_rows[gm] : gm) * g.N + gn : g.aux + o;
      if (vc) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        z[0] = a.x, z[1] = a.y, z[2] = a.z, z[3] = a.w;
      } else {
        for (int c = 0; c < left; ++c) z[c] = p[c];
      }
    }
    float e = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (c >= left) break;
      if (EPI == EPI_GELU_BWD) v[c] *= gelu_grad(z[c]);
      if (EPI == EPI_BIAS || EPI == EPI_BIAS_GELU || EPI == EPI_MSE) v[c] += g.bias[gn + c];
      if (EPI == EPI_BIAS_GELU) {
        z[c] = v[c];
        v[c] = gelu(v[c]);
      } else if (EPI == EPI_MSE) {
        const float d = v[c] - z[c];
        v[c] = 2.0f * d / ((float)g.M * (float)g.N);
        e += d * d;
      }
    }
    if (EPI == EPI_MSE) loss += (double)e;
    const bool save = EPI == EPI_BIAS_GELU && g.aux;
    if (vc) {
      if (save) *reinterpret_cast<float4*>(g.aux + o) = make_float4(z[0], z[1], z[2], z[3]);
      *reinterpret_cast<float4*>(C + o) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
      for (int c = 0; c < left; ++c) {
        if (save) g.aux[o + c] = z[c];
        C[o + c] = v[c];
      }
    }
  }
  if constexpr (EPI == EPI_MSE) {  // one addition to the loss per block
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    __shared__ double wsum[NT / 32];
    if (tid % 32 == 0) wsum[tid / 32] = loss;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < NT / 32; ++w) loss += wsum[w];
      atomicAdd(g.loss, loss);
    }
  }
}

// Where the parameters of layer l (weights, then biases) lie and where their
// gradient's slices are.
struct SliceTab {
  long long off[5], base[4];
  int ns[4];
};

// Gradients of 32 parameters of a block of 32 x 8 threads: row y adds slices y,
// y + 8, .., row 0 the eight sums in pairs (a gradient is not a random walk:
// one chain over all slices loses more than the chains within them).
// Valid in row 0.
constexpr int kSliceRows = 8;
__device__ __forceinline__ float sum_slices(const SliceTab& t, const float* red, int n, int i) {
  __shared__ float part[kSliceRows][32];
  float v = 0.f;
  if (i < n) {
    int l = 0;
    while (l < 3 && i >= t.off[l + 1]) ++l;
    const long long len = t.off[l + 1] - t.off[l];
    const float* p = red + t.base[l] + (i - t.off[l]);
#pragma unroll 8
    for (int s = threadIdx.y; s < t.ns[l]; s += kSliceRows) v += p[s * len];
  }
  part[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  float r[kSliceRows];
#pragma unroll
  for (int k = 0; k < kSliceRows; ++k) r[k] = part[k][threadIdx.x];
  return ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
}

__global__ void __launch_bounds__(256) k_sum_slices(int n, SliceTab t, const float* __restrict__ red,
                                                    float* __restrict__ g) {
  const int i = blockIdx.x * 32 + threadIdx.x;
  const float v = sum_slices(t, red, n, i);
  if (threadIdx.y == 0 && i < n) g[i] = v;
}

// Adam (Kingma & Ba 2015) on a flat parameter vector, the gradient from its
// slices.
__global__ void __launch_bounds__(256) k_adam(int n, float* p, SliceTab t, const float* __restrict__ red, float* m,
                                              float* v, float lr, float b1, float b2, float eps, float bc1,
                                              float bc2) {
  const int i = blockIdx.x * 32 + threadIdx.x;
  const bool mine = threadIdx.y == 0 && i < n;
  const float m0 = mine ? m[i] : 0.f, v0 = mine ? v[i] : 0.f, p0 = mine ? p[i] : 0.f;  // before the slices arrive
  const float gi = sum_slices(t, red, n, i);
  if (!mine) return;
  const float mi = b1 * m0 + (1.f - b1) * gi;
  const float vi = b2 * v0 + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] = p0 - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// (X - mean) * istd per column, in place.
__global__ void k_standardise(long long M, int F, float* X, const float* mean, const float* istd) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M * F) return;
  const int f = (int)(i % F);
  X[i] = (X[i] - mean[f]) * istd[f];
}

// Column sums and sums of squares (double) over M rows, per block:
// part[(f gridDim.x + block) 2 + {0, 1}], added in order by the host.
__global__ void __launch_bounds__(256) k_col_moments(long long M, int F, const float* X, double* part) {
  const int f = blockIdx.y;
  double s = 0.0, s2 = 0.0;
  for (long long m = (long long)blockIdx.x * blockDim.x + threadIdx.x; m < M; m += (long long)gridDim.x * blockDim.x) {
    const double v = X[m * F + f];
    s += v;
    s2 += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  __shared__ double ws[8][2];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    ws[w][0] = s;
    ws[w][1] = s2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      a += ws[k][0];
      b += ws[k][1];
    }
    double* p = part + ((size_t)f * gridDim.x + blockIdx.x) * 2;
    p[0] = a;
    p[1] = b;
  }
}

}  // namespace mlp
}  // namespace adg
