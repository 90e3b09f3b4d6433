// Exact fp32 backward on the CUDA cores, tiled (head sizes up to 128): what attn_bwd_simt.cu computes, for the
// same element types and options, register-blocked (fma_tile.cuh).
//
// The formulas are those of attn_bwd_simt.cu: alpha = exp(logit - lse) recomputed, alpha' = alpha * keep/(1-p),
// D_i = dx_i . x_i, ds_ij = alpha_ij (keep/(1-p) dx_i.v_j - D_i), dq = scale ds k, dk = scale ds^T q,
// dv = alpha'^T dx, dbias = ds.  Two launches: D, then one grid whose blocks own either 64 keys of a unit
// (dk, dv; walking over the query tiles) or 64 queries (dq, dbias; walking over the key tiles).  Both kinds keep
// the two arrays of their own rows in shared memory and stream the two of the other side, so one code serves
// both; they share a launch because neither alone fills the GPU at the sizes Float32 is used for.  No atomics
// except for dbias: the gradients of a call are the same bits every time.
// One training step (forward and backward) at d = 64, 8 heads, 512 x 512 causal, batch 8: 23.06 ms with the warp-per-row
// kernels, 0.46 ms with these (16 TFLOP/s counting seven products over the causal half).
#include <algorithm>

#include "common.cuh"
#include "fma_tile.cuh"
#include "launchers.h"

namespace nb200 {
namespace {

using namespace fma_tile;

constexpr int kBM = 64;                                    // rows a block owns
constexpr int kVecQ = 1, kVecK = 2, kVecV = 4, kVecD = 8;  // 16-byte copies of that array's rows are possible

template <typename T>
__global__ void __launch_bounds__(128) attn_bwd_delta_kernel(const AttnArgs a, const BwdArgs g) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= (long long)a.Lq * a.H * a.B) return;
  const int i = (int)(row % a.Lq), h = (int)((row / a.Lq) % a.H), b = (int)(row / ((long long)a.Lq * a.H));
  const T* xrow = reinterpret_cast<const T*>(a.x) + (long long)i * a.x_sl + (long long)b * a.x_sb + (long long)h * a.dv;
  const T* dxrow = reinterpret_cast<const T*>(g.dx) + (long long)i * g.dx_sl + (long long)b * g.dx_sb + (long long)h * a.dv;
  float dl = 0.f;
  for (int e = lane; e < a.dv; e += 32) dl = fmaf(Elem<T>::to_f(dxrow[e]), Elem<T>::to_f(xrow[e]), dl);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) dl += __shfl_xor_sync(0xffffffffu, dl, off);
  if (lane == 0) g.delta[row] = dl;
}

template <int DP>
__host__ __device__ constexpr int bwd_smem() { return 4 * (4 * kBM * (DP + 4) + 2 * kBM * kLDP) + kBM * 8; }

// KEYS: the block owns keys (dk, dv); else queries (dq, dbias)
template <typename T, int DP, int NTHR, bool KEYS>
__device__ __forceinline__ void bwd_block(const AttnArgs& a, const BwdArgs& g, const int tile, const int unit, const int vec,
                                          float* sm) {
  constexpr int MI = kBM * 16 / NTHR, LD = DP + 4, CN = DP / 16;
  float* a1 = sm;                    // own rows: K, V  or  Q, dX
  float* a2 = a1 + kBM * LD;
  float* b1 = a2 + kBM * LD;         // the walk:  Q, dX  or  K, V
  float* b2 = b1 + kBN * LD;
  float* ps = b2 + kBN * LD;         // alpha' (KEYS only)
  float* ds = ps + kBM * kLDP;
  unsigned char* keep = reinterpret_cast<unsigned char*>(ds + kBM * kLDP);   // [query of the tile][8]

  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int h = unit % a.H, b = unit / a.H;
  const bool drop = a.dropout_p > 0.f;
  const T* q = reinterpret_cast<const T*>(a.q) + (long long)b * a.q_sb + (long long)h * a.d;
  const T* k = reinterpret_cast<const T*>(a.k) + (long long)b * a.k_sb + (long long)h * a.d;
  const T* v = reinterpret_cast<const T*>(a.v) + (long long)b * a.v_sb + (long long)h * a.dv;
  const T* dx = reinterpret_cast<const T*>(g.dx) + (long long)b * g.dx_sb + (long long)h * a.dv;
  const float* lse = a.lse + (long long)a.Lq * h + a.lse_sb * b;
  const float* delta = g.delta + (long long)a.Lq * h + (long long)a.Lq * a.H * b;
  const int r0 = tile * kBM, n_rows = KEYS ? a.Lkv : a.Lq, n_cols = KEYS ? a.Lq : a.Lkv;
  if (KEYS) {
    load_tile<T, kBM, DP, LD, NTHR>(a1, k + (long long)r0 * a.k_sl, a.k_sl, a.Lkv - r0, a.d, (vec & kVecK) != 0);
    load_tile<T, kBM, DP, LD, NTHR>(a2, v + (long long)r0 * a.v_sl, a.v_sl, a.Lkv - r0, a.dv, (vec & kVecV) != 0);
  } else {
    load_tile<T, kBM, DP, LD, NTHR>(a1, q + (long long)r0 * a.q_sl, a.q_sl, a.Lq - r0, a.d, (vec & kVecQ) != 0);
    load_tile<T, kBM, DP, LD, NTHR>(a2, dx + (long long)r0 * g.dx_sl, g.dx_sl, a.Lq - r0, a.dv, (vec & kVecD) != 0);
  }

  float row_lse[MI], row_delta[MI];   // queries as rows: theirs
  float acc1[MI][CN], acc2[KEYS ? MI : 1][CN];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int gi = r0 + ty * MI + i;
    row_lse[i] = (!KEYS && gi < a.Lq) ? lse[gi] : ninf();
    row_delta[i] = (!KEYS && gi < a.Lq) ? delta[gi] : 0.f;
#pragma unroll
    for (int c = 0; c < CN; ++c) {
      acc1[i][c] = 0.f;
      if (KEYS) acc2[i][c] = 0.f;
    }
  }

  // the columns that the causal pattern (key j <= query i + coff) leaves: keys 0 .. or queries .. n_cols-1
  int c_begin = 0, c_end = n_cols;
  if (a.causal) {
    if (KEYS) {
      const long long first = (long long)r0 - a.coff;
      c_begin = first <= 0 ? 0 : (first < n_cols ? (int)first / kBN * kBN : n_cols);
    } else {
      const long long last = (long long)min(r0 + kBM, a.Lq) - 1 + a.coff;
      c_end = last < 0 ? 0 : (last + 1 < n_cols ? (int)last + 1 : n_cols);
    }
  }
  const int d4 = (a.d + 3) >> 2, dv4 = (a.dv + 3) >> 2;
  for (int c0 = c_begin; c0 < c_end; c0 += kBN) {
    const bool v1 = (vec & (KEYS ? kVecQ : kVecK)) != 0, v2 = (vec & (KEYS ? kVecD : kVecV)) != 0;
    if (KEYS) {
      load_tile<T, kBN, DP, LD, NTHR>(b1, q + (long long)c0 * a.q_sl, a.q_sl, a.Lq - c0, a.d, v1);
      cp_async_commit();
      load_tile<T, kBN, DP, LD, NTHR>(b2, dx + (long long)c0 * g.dx_sl, g.dx_sl, a.Lq - c0, a.dv, v2);
    } else {
      load_tile<T, kBN, DP, LD, NTHR>(b1, k + (long long)c0 * a.k_sl, a.k_sl, a.Lkv - c0, a.d, v1);
      cp_async_commit();
      load_tile<T, kBN, DP, LD, NTHR>(b2, v + (long long)c0 * a.v_sl, a.v_sl, a.Lkv - c0, a.dv, v2);
    }
    cp_async_commit();
    const int i0 = KEYS ? c0 : r0, j0 = KEYS ? r0 : c0;    // first query and key of the score tile
    if (drop) fill_keep<NTHR>(keep, a, kBN, j0, [&](int r) { return score_row(a, i0 + r, h, b); });
    float col_lse[4], col_delta[4];                        // queries as columns: theirs
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gc = c0 + tx + 16 * j;
      col_lse[j] = (KEYS && gc < a.Lq) ? lse[gc] : ninf();
      col_delta[j] = (KEYS && gc < a.Lq) ? delta[gc] : 0.f;
    }
    cp_async_wait<1>();
    __syncthreads();
    float p[MI][4];
    dot_tile<MI, LD>(a1, b1, d4, ty, tx, p);
    unsigned int kept = 0u;                                // bit 4 i + j: dropout keeps that score
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int gr = r0 + ty * MI + i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int gc = c0 + tx + 16 * j;
        const int qi = KEYS ? gc : gr, kj = KEYS ? gr : gc;
        const float L = KEYS ? col_lse[j] : row_lse[i];
        const int ql = qi - i0, kl = kj - j0;
        float pv = ninf();                                 // marks a score without any part in the result
        if (gr < n_rows && gc < n_cols && L != ninf()) {
          const float t = finish_logit(a, p[i][j], kj, qi, h, b);
          if (t != ninf()) pv = expf(t - L);
        }
        const bool kp = !drop || ((keep[ql * 8 + (kl >> 3)] >> (kl & 7)) & 1);
        kept |= kp ? 1u << (4 * i + j) : 0u;
        p[i][j] = pv;
        if (KEYS) ps[(ty * MI + i) * kLDP + tx + 16 * j] = (pv == ninf() || !kp) ? 0.f : pv * a.inv_keep;
      }
    }
    cp_async_wait<0>();
    const bool bad = tile_not_finite<T, kBN, DP, LD, NTHR>(b1, v1) || (KEYS && tile_not_finite<T, kBN, DP, LD, NTHR>(b2, v2));
    const bool skip = __syncthreads_or(bad) != 0;
    {
      float dp[MI][4];
      dot_tile<MI, LD>(a2, b2, dv4, ty, tx, dp);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int gr = r0 + ty * MI + i;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int gc = c0 + tx + 16 * j;
          float d = 0.f;
          if (p[i][j] != ninf()) {
            const float f = ((kept >> (4 * i + j)) & 1u) ? a.inv_keep : 0.f;
            d = p[i][j] * (dp[i][j] * f - (KEYS ? col_delta[j] : row_delta[i]));
            if (!KEYS && g.dbias)
              atomicAdd(g.dbias + gc * g.dbias_s[0] + gr * g.dbias_s[1] + h * g.dbias_s[2] + b * g.dbias_s[3], d);
          }
          ds[(ty * MI + i) * kLDP + tx + 16 * j] = d;
        }
      }
    }
    __syncthreads();
    const int nk = min(kBN, c_end - c0);
    if constexpr (KEYS) accumulate<MI, DP, LD>(ps, kLDP, b2, nk, ty, tx, skip, acc2);
    accumulate<MI, DP, LD>(ds, kLDP, b1, nk, ty, tx, skip, acc1);
    __syncthreads();
  }
  cp_async_wait<0>();

  T* o1 = reinterpret_cast<T*>(KEYS ? g.dk : g.dq) + (long long)n_rows * b * ((long long)a.H * a.d) + (long long)h * a.d;
  T* o2 = reinterpret_cast<T*>(g.dv) + (long long)n_rows * b * ((long long)a.H * a.dv) + (long long)h * a.dv;
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int gr = r0 + ty * MI + i;
    if (gr >= n_rows) continue;
#pragma unroll
    for (int c = 0; c < CN; ++c) {
      const int e = colmap<DP>(tx, c);
      if (e < a.d) o1[(long long)gr * a.H * a.d + e] = Elem<T>::from_f(acc1[i][c] * a.scale);
      if (KEYS && e < a.dv) o2[(long long)gr * a.H * a.dv + e] = Elem<T>::from_f(acc2[KEYS ? i : 0][c]);
    }
  }
}

template <typename T, int DP, int NTHR>
__global__ void __launch_bounds__(NTHR, DP <= 64 ? 2 : 1)
attn_bwd_fma_kernel(const AttnArgs a, const BwdArgs g, const int nkt, const int nqt, const int vec) {
  extern __shared__ __align__(16) float sm[];
  const int units = a.H * a.B;
  const int t = blockIdx.x / units, unit = blockIdx.x % units;
  // causal: the first keys are seen by the most queries, the last queries see the most keys
  if (t < nkt) bwd_block<T, DP, NTHR, true>(a, g, t, unit, vec, sm);
  else bwd_block<T, DP, NTHR, false>(a, g, nkt + nqt - 1 - t, unit, vec, sm);
}

template <typename T, int DP, int NTHR>
cudaError_t launch_bwd(const AttnArgs& a, const BwdArgs& g, int vec, cudaStream_t st) {
  const long long rows = (long long)a.Lq * a.H * a.B, db = (rows + 3) / 4;
  const int nkt = (a.Lkv + kBM - 1) / kBM, nqt = (a.Lq + kBM - 1) / kBM;
  const long long blocks = ((long long)nkt + nqt) * a.H * a.B;
  if (db > 0x7fffffffLL || blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  if (db > 0) {
    attn_bwd_delta_kernel<T><<<(unsigned)db, 128, 0, st>>>(a, g);
    count_launch();
  }
  if (blocks > 0) {
    auto kern = attn_bwd_fma_kernel<T, DP, NTHR>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem<DP>());
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)blocks, NTHR, bwd_smem<DP>(), st>>>(a, g, nkt, nqt, vec);
    count_launch();
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_bwd_dims(const AttnArgs& a, const BwdArgs& g, int dtype, cudaStream_t st) {
  const int dm = std::max(a.d, a.dv);
  const int vec = (rows_vec(a.q, a.q_sl, a.q_sb, a.d, dtype) ? kVecQ : 0) |
                  (rows_vec(a.k, a.k_sl, a.k_sb, a.d, dtype) ? kVecK : 0) |
                  (rows_vec(a.v, a.v_sl, a.v_sb, a.dv, dtype) ? kVecV : 0) |
                  (rows_vec(g.dx, g.dx_sl, g.dx_sb, a.dv, dtype) ? kVecD : 0);
  if constexpr (sizeof(T) == 4) {
    if (dm <= 32) return launch_bwd<T, 32, 128>(a, g, vec, st);
    if (dm > 64 && dm <= 96) return launch_bwd<T, 96, 256>(a, g, vec, st);
  }
  // 256 threads of 4 x 4 scores each, sixteen warps on an SM, against 128 of 8 x 4: 457 against 473 us for the step above
  if (dm <= 64) return launch_bwd<T, 64, 256>(a, g, vec, st);
  return launch_bwd<T, 128, 256>(a, g, vec, st);
}

}  // namespace

cudaError_t fma_bwd(const AttnArgs& a, const BwdArgs& g, int dtype, cudaStream_t st) {
  if (a.H == 0 || a.B == 0) return cudaSuccess;
  switch (dtype) {
    case NNLIB_B200_F16:  return launch_bwd_dims<__half>(a, g, dtype, st);
    case NNLIB_B200_BF16: return launch_bwd_dims<__nv_bfloat16>(a, g, dtype, st);
    default:              return launch_bwd_dims<float>(a, g, dtype, st);
  }
}

}  // namespace nb200
