// Second stage of the split-key forwards (attn_tile.cu, attn_decode.cu): layout of the workspace their first
// stage fills, and the kernel that merges the partial results.  Everything sits in an unnamed namespace, so each
// translation unit gets its own copy.
#pragma once

#include "common.cuh"

namespace nb200 {
namespace {

// Workspace of the split-key forward, in floats: (maximum, sum) per (unit, split, query), rounded up so that
// the O rows behind them start on a 16-byte boundary, then dv floats of unnormalised O per (unit, split, query).
__host__ __device__ inline long long split_ml_floats(const AttnArgs& a, int n_splits) {
  return (((long long)a.H * a.B * n_splits * a.Lq * 2) + 3) & ~3LL;
}
__host__ __device__ inline long long split_ws_floats(const AttnArgs& a, int n_splits) {
  return split_ml_floats(a, n_splits) + (long long)a.H * a.B * n_splits * a.Lq * a.dv;
}

// Second stage of the split-key forward: one block per (unit, query) merges the partial results of the
// splits, x = sum_s 2^(m_s - M) O_s / sum_s 2^(m_s - M) l_s, and writes the query's log-sum-exp.
template <typename T>
__global__ void __launch_bounds__(128) attn_split_reduce_kernel(const AttnArgs a, const int n_splits) {
  const long long row = blockIdx.x;              // unit * Lq + i
  const int i = (int)(row % a.Lq);
  const int unit = (int)(row / a.Lq);
  const int h = unit % a.H, b = unit / a.H;
  const float* ml = a.ws + ((long long)unit * n_splits * a.Lq + i) * 2;
  const float* o = a.ws + split_ml_floats(a, n_splits) + ((long long)unit * n_splits * a.Lq + i) * a.dv;
  const long long sstride = a.Lq;                // splits of one unit are Lq slots apart
  float M = __int_as_float(0xff800000);
  bool any_nan = false;
  for (int s = 0; s < n_splits; ++s) {
    const float m = ml[s * sstride * 2], l = ml[s * sstride * 2 + 1];
    if (l != l) any_nan = true;
    if (l > 0.f) M = fmaxf(M, m);
  }
  const bool inf_row = (M == __int_as_float(0x7f800000));
  float L = 0.f;
  for (int s = 0; s < n_splits; ++s) {
    const float m = ml[s * sstride * 2], l = ml[s * sstride * 2 + 1];
    if (!(l > 0.f)) continue;
    const float w = inf_row ? (m == M ? 1.f : 0.f) : exp2f(m - M);
    L += w * l;
  }
  const bool dead = !(L > 0.f) && !any_nan;
  const float nanv = __int_as_float(0x7fc00000);
  if (threadIdx.x == 0 && a.lse) {
    float lse = dead ? __int_as_float(0xff800000) : (M + log2f(L)) * 0.6931471805599453f;
    if (inf_row && !dead) lse = lse_inf_rows(L);
    if (any_nan) lse = nanv;
    a.lse[i + (long long)a.Lq * h + a.lse_sb * b] = lse;
  }
  T* xrow = reinterpret_cast<T*>(a.x) + (long long)i * a.x_sl + (long long)b * a.x_sb + (long long)h * a.dv;
  for (int e = threadIdx.x; e < a.dv; e += blockDim.x) {
    float acc = 0.f;
    for (int s = 0; s < n_splits; ++s) {
      const float m = ml[s * sstride * 2], l = ml[s * sstride * 2 + 1];
      if (!(l > 0.f)) continue;
      const float w = inf_row ? (m == M ? 1.f : 0.f) : exp2f(m - M);
      acc = fmaf(w, o[(long long)s * sstride * a.dv + e], acc);
    }
    float out = acc * (a.inv_keep / L);
    if (dead) out = a.nan_fm ? nanv : 0.f;
    if (any_nan) out = nanv;
    xrow[e] = Elem<T>::from_f(out);
  }
}

}  // namespace
}  // namespace nb200
