// Second stage of the split-key forwards (attn_tile.cu, attn_decode.cu): layout of the workspace their first
// stage fills, and the kernel that merges the partial results.  Everything sits in an unnamed namespace, so each
// translation unit gets its own copy.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace nb200 {
namespace {

// Workspace of the split-key forward, in floats: (maximum, sum) per (unit, split, query), rounded up so that
// the O rows behind them start on a 16-byte boundary, then dv floats of O per (unit, split, query).
__host__ __device__ inline long long split_ml_floats(const AttnArgs& a, int n_splits) {
  return (((long long)a.H * a.B * n_splits * a.Lq * 2) + 3) & ~3LL;
}
__host__ __device__ inline long long split_ws_floats(const AttnArgs& a, int n_splits) {
  return split_ml_floats(a, n_splits) + (long long)a.H * a.B * n_splits * a.Lq * a.dv;
}

// Second stage of the split-key forward: one block per (unit, query) merges the partial results of the
// splits, x = sum_s 2^(m_s - M) O_s / sum_s 2^(m_s - M) l_s, and writes the query's log-sum-exp.
// Latency is what bounds it (a few hundred bytes per share), so the lanes of a warp take a share each for its maximum,
// sum and weight, and hand these round while the O rows of up to 32 shares are under way; both sums run over the shares
// in order.  (One query of one unit against 1M keys, 1024 shares: the whole call 493 us with the shares walked one load after
// the other, 129 so; 8 units, 131072 keys: 154 and 106 us.)
// EXACT (attn_fma.cu): the maxima are natural logarithms, not base 2, whose conversion would be one rounding more, and
// O_s is already divided by l_s.  The weights of the sum are taken 2^e times smaller, 2^e > Lkv, so
// that nothing overflows that the result does not, and a share whose weight vanishes takes no part, whatever its O holds.
template <typename T, bool EXACT>
__global__ void __launch_bounds__(128) attn_split_reduce_kernel(const AttnArgs a, const int n_splits) {
  const long long row = blockIdx.x;              // unit * Lq + i
  const int i = (int)(row % a.Lq);
  const int unit = (int)(row / a.Lq);
  const int h = unit % a.H, b = unit / a.H, lane = threadIdx.x & 31;
  const float* ml = a.ws + ((long long)unit * n_splits * a.Lq + i) * 2;
  const float* o = a.ws + split_ml_floats(a, n_splits) + ((long long)unit * n_splits * a.Lq + i) * a.dv;
  const long long sstride = a.Lq;                // splits of one unit are Lq slots apart
  const float ninf = __int_as_float(0xff800000), pinf = __int_as_float(0x7f800000), nanv = __int_as_float(0x7fc00000);
  float M = ninf;
  bool any_nan = false;
  for (int s = lane; s < n_splits; s += 32) {
    const float m = ml[s * sstride * 2], l = ml[s * sstride * 2 + 1];
    if (l != l) any_nan = true;
    if (l > 0.f) M = fmaxf(M, m);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
  any_nan = __any_sync(0xffffffffu, any_nan);
  const bool inf_row = (M == pinf);
  const int e_keys = 32 - __clz(a.Lkv);
  const float p_scale = __int_as_float((127 - e_keys) << 23), o_scale = __int_as_float((127 + e_keys) << 23);
  T* xrow = reinterpret_cast<T*>(a.x) + (long long)i * a.x_sl + (long long)b * a.x_sb + (long long)h * a.dv;
  for (int e0 = threadIdx.x - lane; e0 < a.dv; e0 += 128) {
    const int e = min(e0 + lane, a.dv - 1);      // (lanes past the end keep their warp company)
    float L = 0.f, acc = 0.f;
    for (int s0 = 0; s0 < n_splits; s0 += 32) {
      const int cnt = min(32, n_splits - s0);
      const int s = s0 + min(lane, cnt - 1);
      const float m = ml[s * sstride * 2], l = ml[s * sstride * 2 + 1];
      const float w = inf_row ? (m == M ? 1.f : 0.f) : (EXACT ? expf(m - M) : exp2f(m - M));
      const float wo = EXACT ? w * (l * p_scale) : w;   // the weight of the share's O
      const unsigned int live = __ballot_sync(0xffffffffu, l > 0.f);
      auto merge = [&](auto group, int j0) {
        constexpr int G = decltype(group)::value;
        float ov[G];
#pragma unroll
        for (int j = 0; j < G; ++j) ov[j] = o[(long long)(s0 + min(j0 + j, cnt - 1)) * sstride * a.dv + e];
#pragma unroll
        for (int j = 0; j < G; ++j) {
          const float wj = __shfl_sync(0xffffffffu, w, j0 + j), lj = __shfl_sync(0xffffffffu, l, j0 + j);
          const float oj = EXACT ? __shfl_sync(0xffffffffu, wo, j0 + j) : wj;
          if (j0 + j < cnt && ((live >> (j0 + j)) & 1u)) {
            L = fmaf(wj, lj, L);
            if (!EXACT || oj != 0.f) acc = fmaf(oj, ov[j], acc);
          }
        }
      };
      if (cnt == 32) merge(std::integral_constant<int, 32>(), 0);
      else for (int j0 = 0; j0 < cnt; j0 += 8) merge(std::integral_constant<int, 8>(), j0);
    }
    const bool dead = !(L > 0.f) && !any_nan;
    float out = acc * (a.inv_keep / L);
    if (EXACT) out *= o_scale;
    if (dead) out = a.nan_fm ? nanv : 0.f;
    if (any_nan) out = nanv;
    if (e0 + lane < a.dv) xrow[e] = Elem<T>::from_f(out);
    if (threadIdx.x == 0 && e0 == 0 && a.lse) {
      float lse = dead ? ninf : (EXACT ? M + logf(L) : fmaf(M, 0.6931471805599453f, logf(L)));
      if (inf_row && !dead) lse = lse_inf_rows(L);
      if (any_nan) lse = nanv;
      a.lse[i + (long long)a.Lq * h + a.lse_sb * b] = lse;
    }
  }
}

}  // namespace
}  // namespace nb200
