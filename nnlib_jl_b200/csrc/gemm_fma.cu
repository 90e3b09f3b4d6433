// Strided-batched matrix product on the CUDA cores, any shape, stride and element type, exact fp32 accumulation
// in ascending k: what the tensor-core kernel (gemm_umma.cu) does not take, Float32 above all.
//
// One block of 256 threads computes a BT x BT tile of C, a thread (BT/16)^2 elements of it, with K in steps of 16
// through two shared-memory stages: while a stage is multiplied, the next one's elements are on their way into
// registers.  BT = 128 (64 multiply-adds per four 16-byte shared-memory loads) is bound by the FMA pipe; smaller
// products take the largest tile that still gives every SM a block.  64 x 1728 x 2821, batch 5, bf16 (an odd leading
// dimension): 2427 us with one thread per element of C, 371 us so.
#include <algorithm>

#include "common.cuh"
#include "launchers.h"

namespace nb200 {
namespace {

constexpr int kGK = 16;

template <typename T, int BT>
__global__ void __launch_bounds__(256) gemm_fma_kernel(const GemmArgs g) {
  constexpr int R = BT / 16;                 // a thread's rows and columns
  constexpr int G = R < 4 ? R : 4;           // ... in runs of G, 16*G apart
  constexpr int LD = BT + 4;
  constexpr int NL = BT * kGK / 256;         // elements of one operand a thread copies per stage
  __shared__ __align__(16) float As[2][kGK][LD], Bs[2][kGK][LD];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.x * BT, n0 = blockIdx.y * BT, b = blockIdx.z;
  const T* A = reinterpret_cast<const T*>(g.A) + (g.a_bcast ? 0 : (long long)b * g.strideA);
  const T* B = reinterpret_cast<const T*>(g.B) + (g.b_bcast ? 0 : (long long)b * g.strideB);
  // element e of the thread's share of a stage: consecutive threads follow the contiguous direction in memory
  auto a_pos = [&](int e, int& k, int& m) {
    const int c = e * 256 + threadIdx.x;
    if (g.transA) { k = c % kGK; m = c / kGK; } else { m = c % BT; k = c / BT; }
  };
  auto b_pos = [&](int e, int& k, int& n) {
    const int c = e * 256 + threadIdx.x;
    if (g.transB) { n = c % BT; k = c / BT; } else { k = c % kGK; n = c / kGK; }
  };
  T ra[NL], rb[NL];                          // (converted when they are stored: converting would wait for the load)
  const T zero = Elem<T>::from_f(0.f);
  auto fetch = [&](int k0) {
#pragma unroll
    for (int e = 0; e < NL; ++e) {
      int k, r;
      a_pos(e, k, r);
      ra[e] = (k0 + k < g.K && m0 + r < g.M)
                  ? (g.transA ? A[(long long)(m0 + r) * g.lda + k0 + k] : A[(long long)(k0 + k) * g.lda + m0 + r]) : zero;
      b_pos(e, k, r);
      rb[e] = (k0 + k < g.K && n0 + r < g.N)
                  ? (g.transB ? B[(long long)(k0 + k) * g.ldb + n0 + r] : B[(long long)(n0 + r) * g.ldb + k0 + k]) : zero;
    }
  };
  auto stage = [&](int s) {
#pragma unroll
    for (int e = 0; e < NL; ++e) {
      int k, r;
      a_pos(e, k, r);
      As[s][k][r] = Elem<T>::to_f(ra[e]);
      b_pos(e, k, r);
      Bs[s][k][r] = Elem<T>::to_f(rb[e]);
    }
  };
  float acc[R][R];                           // [n][m]
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[i][j] = 0.f;

  if (g.K > 0) {
    fetch(0);
    stage(0);
  }
  __syncthreads();
  for (int k0 = 0, s = 0; k0 < g.K; k0 += kGK, s ^= 1) {
    const bool more = k0 + kGK < g.K;
    if (more) fetch(k0 + kGK);
    const int kn = min(kGK, g.K - k0);       // the padding is not multiplied: 0 * Inf would be a NaN
    auto step = [&](int k) {
      float am[R], bn[R];
#pragma unroll
      for (int r = 0; r < R; r += G) {
        if constexpr (G == 4) {
          const float4 va = *reinterpret_cast<const float4*>(&As[s][k][tx * 4 + r * 16]);
          const float4 vb = *reinterpret_cast<const float4*>(&Bs[s][k][ty * 4 + r * 16]);
          am[r] = va.x; am[r + 1] = va.y; am[r + 2] = va.z; am[r + 3] = va.w;
          bn[r] = vb.x; bn[r + 1] = vb.y; bn[r + 2] = vb.z; bn[r + 3] = vb.w;
        } else {
          const float2 va = *reinterpret_cast<const float2*>(&As[s][k][tx * 2]);
          const float2 vb = *reinterpret_cast<const float2*>(&Bs[s][k][ty * 2]);
          am[0] = va.x; am[1] = va.y;
          bn[0] = vb.x; bn[1] = vb.y;
        }
      }
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = fmaf(am[j], bn[i], acc[i][j]);
    };
    if (kn == kGK) {
#pragma unroll
      for (int k = 0; k < kGK; ++k) step(k);
    } else {
      for (int k = 0; k < kn; ++k) step(k);
    }
    if (more) stage(s ^ 1);
    __syncthreads();
  }

  T* C = reinterpret_cast<T*>(g.C) + (long long)b * g.strideC;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int n = n0 + ty * G + (i / G) * 16 * G + i % G;
    if (n >= g.N) continue;
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int m = m0 + tx * G + (j / G) * 16 * G + j % G;
      if (m >= g.M) continue;
      T* c = C + (long long)n * g.ldc + m;
      float out = g.alpha * acc[i][j];
      if (g.beta != 0.f) out = fmaf(g.beta, Elem<T>::to_f(*c), out);
      *c = Elem<T>::from_f(out);
    }
  }
}

// One thread per element of C, 32 m by 8 n a block.
template <typename T>
__global__ void __launch_bounds__(256) gemm_element_kernel(const GemmArgs g) {
  const int m = blockIdx.x * 32 + (threadIdx.x & 31);
  const int n = blockIdx.y * 8 + (threadIdx.x >> 5);
  const int b = blockIdx.z;
  if (m >= g.M || n >= g.N) return;
  const T* A = reinterpret_cast<const T*>(g.A) + (g.a_bcast ? 0 : (long long)b * g.strideA);
  const T* B = reinterpret_cast<const T*>(g.B) + (g.b_bcast ? 0 : (long long)b * g.strideB);
  const long long a_m = g.transA ? g.lda : 1, a_k = g.transA ? 1 : g.lda;
  const long long b_k = g.transB ? g.ldb : 1, b_n = g.transB ? 1 : g.ldb;
  float acc = 0.f;
  for (int k = 0; k < g.K; ++k)
    acc = fmaf(Elem<T>::to_f(A[m * a_m + k * a_k]), Elem<T>::to_f(B[k * b_k + n * b_n]), acc);
  T* c = reinterpret_cast<T*>(g.C) + (long long)b * g.strideC + (long long)n * g.ldc + m;
  float out = g.alpha * acc;
  if (g.beta != 0.f) out = fmaf(g.beta, Elem<T>::to_f(*c), out);
  *c = Elem<T>::from_f(out);
}

template <typename T>
cudaError_t launch_gemm_fma(const GemmArgs& g, cudaStream_t st) {
  auto tiles = [&](long long t) { return ((g.M + t - 1) / t) * ((g.N + t - 1) / t) * g.batch; };
  auto grid = [&](long long t) { return dim3((unsigned)((g.M + t - 1) / t), (unsigned)((g.N + t - 1) / t), (unsigned)g.batch); };
  // The largest tile that is not mostly padding and still gives every SM a block.  Results of at most 8 columns take one
  // thread per element where the lanes of a warp read A along its columns and the sum is not long (4096 x 8 x 512, batch
  // 4: 28 us against 45 of 64-square tiles; 4096 x 1 x 4096: 193 against 130 of 32-square ones), tiny ones always (8 x 8 x
  // 8, batch 10000: 14 us against 205 of the 128-square tiles that their number alone had chosen).
  if (g.N <= 8 && (g.M <= 8 || (!g.transA && g.K <= 1024)))
    gemm_element_kernel<T><<<dim3((unsigned)((g.M + 31) / 32), (unsigned)((g.N + 7) / 8), (unsigned)g.batch), 256, 0, st>>>(g);
  else if (g.M > 64 && g.N > 64 && tiles(128) >= 148) gemm_fma_kernel<T, 128><<<grid(128), 256, 0, st>>>(g);
  else if (g.M > 32 && g.N > 32 && tiles(64) >= 148) gemm_fma_kernel<T, 64><<<grid(64), 256, 0, st>>>(g);
  else gemm_fma_kernel<T, 32><<<grid(32), 256, 0, st>>>(g);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

cudaError_t gemm_simt(const GemmArgs& g, int dtype, cudaStream_t st) {
  if (g.M < 1 || g.N < 1 || g.batch < 1) return cudaSuccess;
  // (the grid of gemm_element_kernel; the tiles' grids hold more)
  if ((g.N + 7LL) / 8 > 65535 || g.batch > 65535) return cudaErrorInvalidConfiguration;
  switch (dtype) {
    case NNLIB_B200_F16:  return launch_gemm_fma<__half>(g, st);
    case NNLIB_B200_BF16: return launch_gemm_fma<__nv_bfloat16>(g, st);
    default:              return launch_gemm_fma<float>(g, st);
  }
}

}  // namespace nb200
