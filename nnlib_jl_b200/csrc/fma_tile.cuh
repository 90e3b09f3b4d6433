// Building blocks of the tiled CUDA-core kernels (attn_fma.cu, attn_bwd_fma.cu): exact fp32 arithmetic on
// tiles in shared memory, register-blocked so that the FMA pipe, not shared memory or L1, is what bounds them.
//
// A block of NTHR threads is a grid of NTHR/16 (ty) x 16 (tx).  A thread owns MI consecutive rows
// (ty*MI ..) of a tile product and every 16th column (tx, tx+16, tx+32, tx+48) of a 64-column score tile,
// or the feature columns colmap(tx, .) of an output tile.  Rows of a row-major tile are LD = DP + 4 floats
// apart: 16 lanes that read 16 bytes of 16 consecutive rows then touch 16 different 16-byte bank groups
// in two wavefronts, the least possible for 256 bytes.
#pragma once

#include "common.cuh"

namespace nb200 {
namespace fma_tile {

constexpr int kBN = 64;        // columns of a score tile
constexpr int kLDP = kBN + 4;  // row pitch of a score tile in shared memory

__device__ __forceinline__ float ninf() { return __int_as_float(0xff800000); }
__device__ __forceinline__ float pinf() { return __int_as_float(0x7f800000); }
__device__ __forceinline__ float qnan() { return __int_as_float(0x7fc00000); }

// pairs along the contraction: one packed FMA does two multiply-adds
__device__ __forceinline__ void ffma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

__device__ __forceinline__ void cp_async16(float* dst, const void* src, bool valid) {
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
  const int n = valid ? 16 : 0;   // 0: nothing is read, 16 zero bytes are written
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Copy `ROWS` rows of `d` elements (row 0 at src, rows `stride` elements apart) into a float tile of pitch LD,
// zeros in columns d .. DP-1 and in rows >= rows_ok.  Float32 rows that start on 16-byte boundaries (`vec`)
// are copied asynchronously (the caller commits and waits), everything else element by element with conversion.
template <typename T, int ROWS, int DP, int LD, int NTHR>
__device__ __forceinline__ void load_tile(float* dst, const T* src, long long stride, int rows_ok, int d, bool vec) {
  if (sizeof(T) == 4 && vec) {
    constexpr int kChunks = DP / 4;
    for (int c = threadIdx.x; c < ROWS * kChunks; c += NTHR) {
      const int r = c / kChunks, e = (c % kChunks) * 4;
      const bool ok = r < rows_ok && e < d;     // d is a multiple of 4 here
      cp_async16(dst + r * LD + e, ok ? (const void*)(src + (long long)r * stride + e) : (const void*)src, ok);
    }
  } else {
    for (int c = threadIdx.x; c < ROWS * DP; c += NTHR) {
      const int r = c / DP, e = c % DP;
      dst[r * LD + e] = (r < rows_ok && e < d) ? Elem<T>::to_f(src[(long long)r * stride + e]) : 0.f;
    }
  }
}

// Did this thread just copy a value that is not finite?  (Same assignment of elements to threads as load_tile,
// so it may be asked before the block synchronises.)
template <typename T, int ROWS, int DP, int LD, int NTHR>
__device__ __forceinline__ bool tile_not_finite(const float* t, bool vec) {
  bool bad = false;
  if (sizeof(T) == 4 && vec) {
    constexpr int kChunks = DP / 4;
    for (int c = threadIdx.x; c < ROWS * kChunks; c += NTHR) {
      const float4 v = *reinterpret_cast<const float4*>(t + (c / kChunks) * LD + (c % kChunks) * 4);
      bad |= !(fabsf(v.x) < pinf()) || !(fabsf(v.y) < pinf()) || !(fabsf(v.z) < pinf()) || !(fabsf(v.w) < pinf());
    }
  } else {
    for (int c = threadIdx.x; c < ROWS * DP; c += NTHR) bad |= !(fabsf(t[(c / DP) * LD + c % DP]) < pinf());
  }
  return bad;
}

// s[i][j] = A[ty*MI + i] . B[tx + 16 j] over the first 4*d4 features
template <int MI, int LD>
__device__ __forceinline__ void dot_tile(const float* A, const float* B, int d4, int ty, int tx, float (&s)[MI][4]) {
  unsigned long long acc[MI][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  const float* ap = A + ty * MI * LD;
  const float* bp = B + tx * LD;
#pragma unroll 2
  for (int c = 0; c < d4; ++c) {
    ulonglong2 b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(bp + 16 * j * LD + 4 * c);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(ap + i * LD + 4 * c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        ffma2(acc[i][j], a.x, b[j].x);
        ffma2(acc[i][j], a.y, b[j].y);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      s[i][j] = __uint_as_float((unsigned int)acc[i][j]) + __uint_as_float((unsigned int)(acc[i][j] >> 32));
}

// Feature columns of a thread: CN = DP/16 of them; full float4 groups of 64 columns, then a float2 group of 32.
template <int DP>
__device__ __forceinline__ int colmap(int tx, int c) {
  constexpr int kFull = (DP / 64) * 4;
  return c < kFull ? (c / 4) * 64 + tx * 4 + (c & 3) : (DP / 64) * 64 + tx * 2 + (c - kFull);
}

template <int DP>
__device__ __forceinline__ void load_cols(const float* row, int tx, float (&v)[DP / 16]) {
#pragma unroll
  for (int g = 0; g < DP / 64; ++g) {
    const float4 f = *reinterpret_cast<const float4*>(row + g * 64 + tx * 4);
    v[4 * g] = f.x; v[4 * g + 1] = f.y; v[4 * g + 2] = f.z; v[4 * g + 3] = f.w;
  }
  if (DP % 64 == 32) {
    const float2 f = *reinterpret_cast<const float2*>(row + (DP / 64) * 64 + tx * 2);
    v[(DP / 64) * 4] = f.x;
    v[(DP / 64) * 4 + 1] = f.y;
  }
}

// o[i][c] += sum_k P[ty*MI + i][k] V[k][colmap(tx, c)] for the first nk (rounded up to 4) columns k of the tile.
// SKIP: a zero weight takes nothing from its row of V, whatever is stored there (a masked key may hold
// anything, also NaN); the caller asks for it when the V tile holds a value that is not finite.
template <int MI, int DP, int LD, bool SKIP>
__device__ __forceinline__ void accumulate_impl(const float* P, int pitch, const float* V, int nk, int ty,
                                                int tx, float (&o)[MI][DP / 16]) {
  constexpr int CN = DP / 16;
  const float* pp = P + ty * MI * pitch;
#pragma unroll 1
  for (int k = 0; k < nk; k += 4) {
    float4 p[MI];
#pragma unroll
    for (int i = 0; i < MI; ++i) p[i] = *reinterpret_cast<const float4*>(pp + i * pitch + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float v[CN];
      load_cols<DP>(V + (k + kk) * LD, tx, v);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const float pk = kk == 0 ? p[i].x : (kk == 1 ? p[i].y : (kk == 2 ? p[i].z : p[i].w));
        if (!SKIP || pk != 0.f) {
#pragma unroll
          for (int c = 0; c < CN; ++c) o[i][c] = fmaf(pk, v[c], o[i][c]);
        }
      }
    }
  }
}

template <int MI, int DP, int LD>
__device__ __forceinline__ void accumulate(const float* P, int pitch, const float* V, int nk, int ty, int tx,
                                           bool skip_zero, float (&o)[MI][DP / 16]) {
  if (skip_zero) accumulate_impl<MI, DP, LD, true>(P, pitch, V, nk, ty, tx, o);
  else accumulate_impl<MI, DP, LD, false>(P, pitch, V, nk, ty, tx, o);
}

// o[i][c] += sum_k P[k][ty*MI + i] V[k][colmap(tx, c)] over the tile's 64 rows k: the same with the transpose of a tile
template <int MI, int DP, int LD, bool SKIP>
__device__ __forceinline__ void accumulate_t_impl(const float* P, int pitch, const float* V, int ty, int tx, float (&o)[MI][DP / 16]) {
  static_assert(MI == 4 || MI == 8, "rows of a thread");
  constexpr int CN = DP / 16;
  const float* pp = P + ty * MI;
#pragma unroll 4
  for (int k = 0; k < kBN; ++k) {
    float p[MI], v[CN];
#pragma unroll
    for (int i = 0; i < MI; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(pp + k * pitch + i);
      p[i] = f.x; p[i + 1] = f.y; p[i + 2] = f.z; p[i + 3] = f.w;
    }
    load_cols<DP>(V + k * LD, tx, v);
#pragma unroll
    for (int i = 0; i < MI; ++i)
      if (!SKIP || p[i] != 0.f) {
#pragma unroll
        for (int c = 0; c < CN; ++c) o[i][c] = fmaf(p[i], v[c], o[i][c]);
      }
  }
}
template <int MI, int DP, int LD>
__device__ __forceinline__ void accumulate_t(const float* P, int pitch, const float* V, int ty, int tx, bool skip_zero,
                                             float (&o)[MI][DP / 16]) {
  if (skip_zero) accumulate_t_impl<MI, DP, LD, true>(P, pitch, V, ty, tx, o);
  else accumulate_t_impl<MI, DP, LD, false>(P, pitch, V, ty, tx, o);
}

// Keep bits of dropout for a tile of `rows` score rows x 64 keys (keys k0 .., k0 a multiple of 8): byte g of
// row r covers keys k0 + 8g .. +7.  One Philox call serves eight scores.
// row_of(r): the global score-row number of tile row r.
template <int NTHR, typename RowOf>
__device__ __forceinline__ void fill_keep(unsigned char* keep, const AttnArgs& a, int rows, int k0, RowOf row_of) {
  for (int c = threadIdx.x; c < rows * 8; c += NTHR) {
    const int r = c >> 3, g = c & 7;
    unsigned int w[4];
    dropout_words(a, row_of(r), (unsigned int)(k0 >> 3) + g, w);
    unsigned int byte = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      byte |= ((w[e] & 0xffffu) >= a.drop_thresh ? 1u : 0u) << (2 * e);
      byte |= ((w[e] >> 16) >= a.drop_thresh ? 1u : 0u) << (2 * e + 1);
    }
    keep[r * 8 + g] = (unsigned char)byte;
  }
}

// scaled logit of (key j, query i) from its raw dot product: + bias (src/attention.jl:129-131), then the masks
// (:133-138).  (j, i) must lie inside the arrays.
__device__ __forceinline__ float finish_logit(const AttnArgs& a, float s, int j, int i, int h, int b) {
  s *= a.scale;
  if (a.bias)
    s += load_bias(a.bias, j * a.bias_s[0] + i * a.bias_s[1] + h * a.bias_s[2] + b * a.bias_s[3], a.bias_dtype);
  bool keep = true;
  if (a.causal) keep = (j <= i + a.coff);
  if (a.mask) keep = keep && (a.mask[j * a.mask_s[0] + i * a.mask_s[1] + h * a.mask_s[2] + b * a.mask_s[3]] != 0);
  return keep ? s : ninf();
}

// 16-byte copies of Float32 rows are possible
inline bool rows_vec(const void* base, long long stride_l, long long stride_b, int d, int dtype) {
  return dtype == NNLIB_B200_F32 && (reinterpret_cast<uintptr_t>(base) & 15u) == 0 && stride_l % 4 == 0 &&
         stride_b % 4 == 0 && d % 4 == 0;
}

}  // namespace fma_tile
}  // namespace nb200
