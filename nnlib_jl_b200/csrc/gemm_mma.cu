// Strided-batched matrix product of 16-bit arrays whose leading dimensions, batch strides or addresses the copy
// engine cannot address (an odd number of rows, say): warp-level m16n8k16 products on tiles that the threads copy
// themselves, fp32 accumulation.
//
// Roles as in gemm_umma.cu: the product's rows are n, its columns m, so that a thread ends up with neighbouring m of
// a column of C.  One block of 256 threads computes 128 n x 128 m, K in steps of 32 through two shared-memory stages;
// while one is multiplied the next one's elements are on their way into registers.  An operand is kept the way it lies
// in memory, [row][k] or [k][row], and the fragments are read with or without transposition.  Eight elements at any
// 2-byte alignment are fetched as aligned words and shifted into place.  What bounds it is that copying: five 4-byte
// loads per eight elements.  3395 x 3969 x 128, batch 13, f16: 7.51 ms with one thread per element of C, 3.32 in
// CUDA-core tiles, 0.67 so (68 TFLOP/s).
#include <type_traits>

#include "common.cuh"
#include "extras.cuh"
#include "launchers.h"

namespace nb200 {
namespace {

constexpr int kMT = 128;          // tile edge, both ways
constexpr int kMK = 32;
constexpr int kPitchK = 40;       // elements between rows of an [row][k] tile: 16-byte reads of 8 rows hit 8 bank groups
constexpr int kPitchR = 136;      // ... of a [k][row] tile
constexpr int kTileElems = kMT * kPitchK;   // the larger of the two forms (kMK * kPitchR is less)
static_assert(kMK * kPitchR <= kTileElems, "tile size");

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p, bool trans) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  if (trans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Two groups of eight elements per thread of a 128 x 32 operand tile.  KC: k is the contiguous direction.
// `rows`, `K`: extent of the stored matrix; what lies beyond reads as 0.
template <typename T, bool KC>
__device__ __forceinline__ void fetch_tile(const T* base, long long ld, int r0, int rows, int k0, int K, uint32_t (&w)[2][4]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int g = threadIdx.x + 256 * u;
    const int r = KC ? r0 + (g >> 2) : r0 + (g & 15) * 8, k = KC ? k0 + (g & 3) * 8 : k0 + (g >> 4);
    const int n = KC ? (r < rows ? min(8, K - k) : 0) : (k < K ? min(8, rows - r) : 0);   // elements inside
    if (n > 0) {
      const unsigned char* p = reinterpret_cast<const unsigned char*>(base + (KC ? (long long)r * ld + k : (long long)k * ld + r));
      load_shifted<4>(p, p + 2 * n, w[u]);
      if (n < 8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) w[u][i] = 2 * i >= n ? 0u : (2 * i + 1 >= n ? w[u][i] & 0xffffu : w[u][i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) w[u][i] = 0u;
    }
  }
}
template <bool KC>
__device__ __forceinline__ void store_tile(unsigned short* t, const uint32_t (&w)[2][4]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int g = threadIdx.x + 256 * u;
    unsigned short* d = KC ? t + (g >> 2) * kPitchK + (g & 3) * 8 : t + (g >> 4) * kPitchR + (g & 15) * 8;
    *reinterpret_cast<uint4*>(d) = make_uint4(w[u][0], w[u][1], w[u][2], w[u][3]);
  }
}

// NKC: k contiguous in the n-side operand (B 'N'); MKC: in the m-side operand (A 'T')
template <typename T, bool NKC, bool MKC>
__global__ void __launch_bounds__(256) gemm_mma_kernel(const GemmArgs g) {
  constexpr bool BF16 = std::is_same<T, __nv_bfloat16>::value;
  __shared__ __align__(16) unsigned short sn[2][kTileElems], sm[2][kTileElems];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * kMT, n0 = blockIdx.y * kMT, b = blockIdx.z;
  const int wn = (warp >> 1) * 32, wm = (warp & 1) * 64;       // this warp's 32 n x 64 m
  const T* A = reinterpret_cast<const T*>(g.A) + (g.a_bcast ? 0 : (long long)b * g.strideA);
  const T* B = reinterpret_cast<const T*>(g.B) + (g.b_bcast ? 0 : (long long)b * g.strideB);
  uint32_t rn[2][4], rm[2][4];
  float acc[2][8][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;

  fetch_tile<T, NKC>(B, g.ldb, n0, g.N, 0, g.K, rn);
  fetch_tile<T, MKC>(A, g.lda, m0, g.M, 0, g.K, rm);
  store_tile<NKC>(sn[0], rn);
  store_tile<MKC>(sm[0], rm);
  __syncthreads();
  for (int k0 = 0, s = 0; k0 < g.K; k0 += kMK, s ^= 1) {
    const bool more = k0 + kMK < g.K;
    if (more) {
      fetch_tile<T, NKC>(B, g.ldb, n0, g.N, k0 + kMK, g.K, rn);
      fetch_tile<T, MKC>(A, g.lda, m0, g.M, k0 + kMK, g.K, rm);
    }
#pragma unroll
    for (int kk = 0; kk < kMK; kk += 16) {
      uint32_t fa[2][4], fb[4][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wn + 16 * i;
        ldsm4(fa[i], NKC ? &sn[s][(r + (lane & 15)) * kPitchK + kk + (lane >> 4) * 8]
                         : &sn[s][(kk + (lane & 7) + (lane >> 4) * 8) * kPitchR + r + ((lane >> 3) & 1) * 8], !NKC);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = wm + 16 * j;
        ldsm4(fb[j], MKC ? &sm[s][(r + (lane & 7) + (lane >> 4) * 8) * kPitchK + kk + ((lane >> 3) & 1) * 8]
                         : &sm[s][(kk + (lane & 15)) * kPitchR + r + (lane >> 4) * 8], !MKC);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) mma_16816<BF16>(acc[i][j], fa[i], fb[j >> 1][(j & 1) * 2], fb[j >> 1][(j & 1) * 2 + 1]);
    }
    if (more) {
      store_tile<NKC>(sn[s ^ 1], rn);
      store_tile<MKC>(sm[s ^ 1], rm);
    }
    __syncthreads();
  }

  T* C = reinterpret_cast<T*>(g.C) + (long long)b * g.strideC;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int n = n0 + wn + 16 * i + (lane >> 2) + (e >> 1) * 8, m = m0 + wm + 8 * j + (lane & 3) * 2 + (e & 1);
        if (n < g.N && m < g.M) {
          T* c = C + (long long)n * g.ldc + m;
          float out = g.alpha * acc[i][j][e];
          if (g.beta != 0.f) out = fmaf(g.beta, Elem<T>::to_f(*c), out);
          *c = Elem<T>::from_f(out);
        }
      }
}

template <typename T>
cudaError_t launch_gemm_mma(const GemmArgs& g, cudaStream_t st) {
  const dim3 grid((unsigned)((g.M + kMT - 1) / kMT), (unsigned)((g.N + kMT - 1) / kMT), (unsigned)g.batch);
  const bool nkc = !g.transB, mkc = g.transA != 0;
  if (nkc && mkc) gemm_mma_kernel<T, true, true><<<grid, 256, 0, st>>>(g);
  else if (nkc) gemm_mma_kernel<T, true, false><<<grid, 256, 0, st>>>(g);
  else if (mkc) gemm_mma_kernel<T, false, true><<<grid, 256, 0, st>>>(g);
  else gemm_mma_kernel<T, false, false><<<grid, 256, 0, st>>>(g);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

// 16-bit products worth a 128 x 128 tile; thinner ones are left to the CUDA-core tiles, and so are sums of more than 4096
// terms: the products' accumulation does not round each step to nearest, which adds up (error against Float64, f16,
// all terms positive: as with one fused multiply-add after the other up to K = 1000, + 0.7 % at 4095, + 11 % at 16385).
// The columns are limited as for every product off the tcgen05 path (gemm_fma.cu).
bool gemm_mma_supports(const GemmArgs& g, int dtype) {
  return (dtype == NNLIB_B200_F16 || dtype == NNLIB_B200_BF16) && g.M >= 32 && g.N >= 32 && g.K >= 16 && g.K <= 4096 &&
         (g.N + 7LL) / 8 <= 65535 && g.batch >= 1 && g.batch <= 65535 && (reinterpret_cast<uintptr_t>(g.A) & 1u) == 0 &&
         (reinterpret_cast<uintptr_t>(g.B) & 1u) == 0;
}
cudaError_t gemm_mma(const GemmArgs& g, int dtype, cudaStream_t st) {
  return dtype == NNLIB_B200_BF16 ? launch_gemm_mma<__nv_bfloat16>(g, st) : launch_gemm_mma<__half>(g, st);
}

}  // namespace nb200
