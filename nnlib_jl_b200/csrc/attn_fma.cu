// Exact fp32 attention on the CUDA cores, tiled: Float32 arrays (without TF32) and whatever 16-bit arrays the
// tensor-core kernels do not take, head sizes up to 128.
//
// The arithmetic is the reference's (NNlib.jl src/softmax.jl:69-79, src/attention.jl:96-98,117-126) in fp32
// with FMA accumulation; only the order differs.  What bounds it is the FMA pipe (128 multiply-adds per SM and
// cycle), so everything is register-blocked: see fma_tile.cuh for the thread grid.
//
//   attn_fma_kernel      one block = BM queries of one unit, key tiles of 64:
//     FM_FWD     x and the log-sum-exp in one pass (running maximum; O rescaled when it rises)
//     FM_STATS   the log-sum-exp only
//     FM_SCORES  alpha from a given log-sum-exp; the key tiles of a block row may be dealt to several blocks
//     FM_APPLY   x = V alpha for scores the caller holds
//     FM_SPLIT   FM_FWD for few queries against many keys: the key tiles of a unit are dealt to gridDim.y blocks,
//                each leaving its maximum, sum and O in a workspace (split_reduce.cuh merges them)
// A warp per query that walked the keys one lane per key (attn_simt.cu, still there for larger heads) re-read every
// key row through L1 for each query, uncoalesced: 441 us for x and alpha at d = 64, 8 heads, 128 x 128, batch 4,
// where a call of the row kernel takes 26 us, nearly all of it host time.
//
//   attn_fma_row_kernel  x, alpha and the log-sum-exp in one pass for short key sequences: the logits of a
//                        block's queries stay in shared memory, so each is computed and exponentiated once
#include <algorithm>

#include "common.cuh"
#include "fma_tile.cuh"
#include "launchers.h"
#include "split_reduce.cuh"

namespace nb200 {
namespace {

using namespace fma_tile;

enum : int { FM_FWD = 0, FM_STATS = 1, FM_SCORES = 2, FM_APPLY = 3, FM_SPLIT = 4 };
constexpr int kRowBM = 32;                       // queries of a block of the row kernel
constexpr int kVecQ = 1, kVecK = 2, kVecV = 4;   // 16-byte copies of that array's rows are possible

// keys 0 .. n-1 are all that the queries up to i_max can attend to (without the mask array)
__device__ __forceinline__ int key_end(const AttnArgs& a, int i_max) {
  if (!a.causal) return a.Lkv;
  const long long e = (long long)i_max + a.coff + 1;
  return e < 0 ? 0 : (e < a.Lkv ? (int)e : a.Lkv);
}

// Does dropout keep any key of this score row?  (Only asked for rows without an ordinary result.)
__device__ __forceinline__ bool any_kept(const AttnArgs& a, unsigned long long srow) {
  if (!(a.dropout_p > 0.f)) return a.Lkv > 0;
  for (int j = 0; j < a.Lkv; ++j)
    if (dropout_keep1(a, srow, (unsigned int)j)) return true;
  return false;
}

__device__ __forceinline__ float max16(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float sum16(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// exp(t - m) for a maximum m over the row's ordinary and +Inf logits: +Inf logits count 1 against m = +Inf
// (equal shares, src/softmax.jl:73-75), a masked one 0, NaN stays NaN
__device__ __forceinline__ float exp_rel(float t, float m) { return t == ninf() ? 0.f : (t == m ? 1.f : expf(t - m)); }

// log-sum-exp as the other kernels read it, from the maximum and the sum relative to it
__device__ __forceinline__ float make_lse(float m, float l) {
  if (l != l) return qnan();
  if (!(l > 0.f)) return ninf();
  return m == pinf() ? lse_inf_rows(l) : m + logf(l);
}

template <int DP, int BM>
__host__ __device__ constexpr int kp_floats() { return kBN * (DP + 4) > BM * kLDP ? kBN * (DP + 4) : BM * kLDP; }
// AHEAD (x in one pass, heads up to 96; launch_fma_mi says when): the P tile has a place of its own, and the next K and V
// tiles are copied while the block works on this one (with larger heads it would cost the second block on an SM); tiles
// that need nothing but the scale are told apart.  512 x 512, d = 64, 64 units 267 -> 217 us, causal 134 -> 122, 2048 x 2048 causal, 16 units
// 504 -> 432.
template <int DP, int BM, int MODE, bool AHEAD>
__host__ __device__ constexpr int fma_smem() {
  return 4 * ((MODE != FM_APPLY ? BM * (DP + 4) : 0) +
              (AHEAD ? kBN * (DP + 4) + BM * kLDP : kp_floats<DP, BM>()) +
              (MODE != FM_STATS && MODE != FM_SCORES ? kBN * (DP + 4) : 0)) + BM * 8;
}

__host__ __device__ constexpr bool fm_with_v(int mode) { return mode == FM_FWD || mode == FM_APPLY || mode == FM_SPLIT; }

// (d = 64, 8 rows a thread: three blocks on an SM with a few spilled words are faster than two without)
template <typename T, int DP, int MI, int NTHR, int MODE, bool AHEAD>
__global__ void __launch_bounds__(NTHR, MODE == FM_FWD && MI == 8 && DP == 64 ? 3 : 1) attn_fma_kernel(const AttnArgs a, const int n_tiles, const int vec) {
  constexpr int BM = NTHR / 16 * MI, LD = DP + 4, CN = DP / 16;
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;
  float* kp = qs + (MODE != FM_APPLY ? BM * LD : 0);       // the K tile, then the P tile
  float* ps = AHEAD ? kp + kBN * LD : kp;
  float* vs = AHEAD ? ps + BM * kLDP : kp + kp_floats<DP, BM>();
  unsigned char* keep = reinterpret_cast<unsigned char*>(vs + (fm_with_v(MODE) ? kBN * LD : 0));

  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int units = a.H * a.B;
  const int unit = blockIdx.x % units;
  const int tile = n_tiles - 1 - blockIdx.x / units;       // causal: the longest walks are dealt out first
  const int h = unit % a.H, b = unit / a.H;
  const int q0 = tile * BM;
  const bool drop = a.dropout_p > 0.f && MODE != FM_STATS && MODE != FM_APPLY;

  const T* kbase = reinterpret_cast<const T*>(a.k) + (long long)b * a.k_sb + (long long)h * a.d;
  const T* vbase = reinterpret_cast<const T*>(a.v) + (long long)b * a.v_sb + (long long)h * a.dv;
  T* alpha = reinterpret_cast<T*>(a.alpha) + a.alpha_sb * b + (long long)a.Lq * h * a.Lkv;
  if (MODE != FM_APPLY) {
    const T* qbase = reinterpret_cast<const T*>(a.q) + (long long)b * a.q_sb + (long long)h * a.d + (long long)q0 * a.q_sl;
    load_tile<T, BM, DP, LD, NTHR>(qs, qbase, a.q_sl, a.Lq - q0, a.d, (vec & kVecQ) != 0);
    if (!AHEAD) cp_async_commit();
  }

  float m[MI], l[MI], o[MI][CN];
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    m[i] = ninf();
    l[i] = 0.f;
    if (MODE == FM_SCORES) m[i] = (q0 + ty * MI + i < a.Lq) ? a.lse[q0 + ty * MI + i + (long long)a.Lq * h + a.lse_sb * b] : 0.f;
#pragma unroll
    for (int c = 0; c < CN; ++c) o[i][c] = 0.f;
  }

  const int kend = key_end(a, min(q0 + BM, a.Lq) - 1);
  // every score is written in FM_SCORES and read in FM_APPLY, the others end at the last key in reach
  int kstart = blockIdx.y * kBN, kstep = kBN * gridDim.y;
  int kstop = (MODE == FM_SCORES || MODE == FM_APPLY) ? a.Lkv : kend;
  if (MODE == FM_SPLIT) {                                  // a contiguous share
    const int per = ((kstop + kBN - 1) / kBN + gridDim.y - 1) / gridDim.y * kBN;
    kstart = blockIdx.y * per;
    kstop = min(kstop, kstart + per);
    kstep = kBN;
  }
  const int d4 = (a.d + 3) >> 2;
  // O is summed with weights up to 1 a key and divided by their sum at the end: the weights of the sum are taken 2^e
  // times smaller, 2^e > Lkv, so that values near the end of the type's range do not overflow on the way to their mean
  const int e_keys = 32 - __clz(a.Lkv);
  const float p_scale = MODE == FM_APPLY ? 1.f : __int_as_float((127 - e_keys) << 23);
  const float o_scale = MODE == FM_APPLY ? 1.f : __int_as_float((127 + e_keys) << 23);
  auto fetch_k = [&](int k0) {
    if (k0 < kstop)
      load_tile<T, kBN, DP, LD, NTHR>(kp, kbase + (long long)k0 * a.k_sl, a.k_sl, a.Lkv - k0, a.d, (vec & kVecK) != 0);
    cp_async_commit();
  };
  auto fetch_v = [&](int k0) {
    if (k0 < kstop)
      load_tile<T, kBN, DP, LD, NTHR>(vs, vbase + (long long)k0 * a.v_sl, a.v_sl, a.Lkv - k0, a.dv, (vec & kVecV) != 0);
    cp_async_commit();
  };
  if (AHEAD) {
    fetch_k(kstart);
    fetch_v(kstart);
  }
  for (int k0 = kstart; k0 < kstop; k0 += kstep) {
    const bool live = MODE == FM_APPLY || k0 < kend;       // false: all above the causal diagonal
    // nothing but the scale is to be applied to the tile's logits
    const bool plain = !a.bias && !a.mask && q0 + BM <= a.Lq && k0 + kBN <= a.Lkv && (!a.causal || k0 + kBN - 1 <= q0 + a.coff);
    if (!AHEAD && MODE != FM_APPLY && live) {
      load_tile<T, kBN, DP, LD, NTHR>(kp, kbase + (long long)k0 * a.k_sl, a.k_sl, a.Lkv - k0, a.d, (vec & kVecK) != 0);
      cp_async_commit();
    }
    if (!AHEAD && fm_with_v(MODE)) {
      load_tile<T, kBN, DP, LD, NTHR>(vs, vbase + (long long)k0 * a.v_sl, a.v_sl, a.Lkv - k0, a.dv, (vec & kVecV) != 0);
      cp_async_commit();
    }
    if (drop)
      fill_keep<NTHR>(keep, a, BM, k0, [&](int r) { return score_row(a, q0 + r, h, b); });
    if (MODE == FM_APPLY) {
      for (int c = threadIdx.x; c < BM * kBN; c += NTHR) {
        const int r = c / kBN, k = c % kBN;
        kp[r * kLDP + k] = (q0 + r < a.Lq && k0 + k < a.Lkv) ? Elem<T>::to_f(alpha[(long long)(q0 + r) * a.Lkv + k0 + k]) : 0.f;
      }
    } else {
      float s[MI][4];
      if (live) {
        if (fm_with_v(MODE)) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
        dot_tile<MI, LD>(qs, kp, d4, ty, tx, s);
      }
      __syncthreads();                                     // the K tile is free, the keep bits are there
      if (AHEAD) fetch_k(k0 + kstep);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int r = ty * MI + i, gi = q0 + r;
        float t[4];
        if (AHEAD && plain) {
#pragma unroll
          for (int j = 0; j < 4; ++j) t[j] = s[i][j] * a.scale;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int kj = k0 + tx + 16 * j;
            t[j] = (live && gi < a.Lq && kj < a.Lkv) ? finish_logit(a, s[i][j], kj, gi, h, b) : ninf();
          }
        }
        if (MODE == FM_SCORES) {
          if (gi < a.Lq) {
            const float lse = m[i];
            const bool inf_row = lse_is_inf_rows(lse);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int k = tx + 16 * j, kj = k0 + k;
              float al;
              if (lse == ninf())   al = a.nan_fm ? qnan() : 0.f;
              else if (inf_row)    al = (t[j] == pinf()) ? 1.f / lse_inf_count(lse) : 0.f;
              else if (lse != lse) al = qnan();
              else                 al = (t[j] == ninf()) ? 0.f : expf(t[j] - lse);
              if (drop) al = ((keep[r * 8 + (k >> 3)] >> (k & 7)) & 1) ? al * a.inv_keep : 0.f;
              if (kj < a.Lkv) alpha[(long long)gi * a.Lkv + kj] = Elem<T>::from_f(al);
            }
          }
        } else {
          const float mn = fmaxf(m[i], max16(fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3]))));
          const float f = (m[i] == mn) ? 1.f : expf(m[i] - mn);
          m[i] = mn;
          float sum = 0.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int k = tx + 16 * j;
            float p = exp_rel(t[j], mn);
            sum += p;
            if (fm_with_v(MODE)) {
              if (drop && !((keep[r * 8 + (k >> 3)] >> (k & 7)) & 1)) p = 0.f;
              ps[r * kLDP + k] = p * p_scale;
            }
          }
          l[i] = fmaf(l[i], f, sum);
          if (fm_with_v(MODE) && f != 1.f) {
#pragma unroll
            for (int c = 0; c < CN; ++c) o[i][c] = (f == 0.f) ? 0.f : o[i][c] * f;
          }
        }
      }
    }
    if (fm_with_v(MODE)) {
      cp_async_wait<AHEAD ? 1 : 0>();
      const bool bad = tile_not_finite<T, kBN, DP, LD, NTHR>(vs, (vec & kVecV) != 0);
      const bool skip = __syncthreads_or(bad) != 0;
      accumulate<MI, DP, LD>(ps, kLDP, vs, min(kBN, kstop - k0), ty, tx, skip, o);
    }
    __syncthreads();
    if (AHEAD) fetch_v(k0 + kstep);
  }
  cp_async_wait<0>();
  if (MODE == FM_SCORES) return;

#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int gi = q0 + ty * MI + i;
    float scale = 1.f, fixed = 0.f;
    bool special = false;
    if (MODE != FM_APPLY) {
      const float ls = sum16(l[i]);                        // all 16 lanes of a row take part
      if (gi >= a.Lq) continue;                            // whole half-warps
      if (MODE == FM_SPLIT) {
        const long long slot = ((long long)unit * gridDim.y + blockIdx.y) * a.Lq + gi;
        if (tx == 0) {
          a.ws[slot * 2] = m[i];
          a.ws[slot * 2 + 1] = ls;
        }
        float* ow = a.ws + split_ml_floats(a, gridDim.y) + slot * a.dv;
        const float inv = ls > 0.f ? 1.f / ls : 0.f;
#pragma unroll
        for (int c = 0; c < CN; ++c)
          if (colmap<DP>(tx, c) < a.dv) ow[colmap<DP>(tx, c)] = o[i][c] * inv * o_scale;
        continue;
      }
      if (a.lse && tx == 0) a.lse[gi + (long long)a.Lq * h + a.lse_sb * b] = make_lse(m[i], ls);
      if (MODE == FM_STATS) continue;
      scale = a.inv_keep / ls;
      if (!(ls > 0.f)) {                                   // nothing attended, or a NaN logit
        special = true;
        if ((ls != ls || a.nan_fm) && any_kept(a, score_row(a, gi, h, b))) fixed = qnan();
      }
    }
    if (gi < a.Lq) {
      T* xr = reinterpret_cast<T*>(a.x) + (long long)gi * a.x_sl + (long long)b * a.x_sb + (long long)h * a.dv;
#pragma unroll
      for (int c = 0; c < CN; ++c) {
        const int e = colmap<DP>(tx, c);
        if (e < a.dv) xr[e] = Elem<T>::from_f(special ? fixed : o[i][c] * scale * o_scale);
      }
    }
  }
}

// ---- x, alpha and the log-sum-exp of a block's queries with all their logits in shared memory ----------------
// pitch of the logits: 64 per key tile + 4 (rows two lanes groups apart fall into different banks)
__host__ __device__ inline int row_pitch(int n_ktiles) { return n_ktiles * kBN + 4; }
template <int DP, int BM>
inline int row_smem(int n_ktiles) {
  return 4 * (BM * (DP + 4) + 2 * kBN * (DP + 4) + BM * row_pitch(n_ktiles)) + BM * 8 * n_ktiles;
}

template <typename T, int DP, int MI, int NTHR>
__global__ void __launch_bounds__(NTHR) attn_fma_row_kernel(const AttnArgs a, const int n_tiles, const int n_ktiles,
                                                            const int vec) {
  constexpr int BM = NTHR / 16 * MI, LD = DP + 4, CN = DP / 16;
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;
  float* ring = qs + BM * LD;                              // two tiles: K tiles, then V tiles
  float* ss = ring + 2 * kBN * LD;
  const int pitch = row_pitch(n_ktiles);
  unsigned char* keep = reinterpret_cast<unsigned char*>(ss + BM * pitch);   // [key tile][query][8]

  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int units = a.H * a.B;
  const int unit = blockIdx.x % units;
  const int tile = n_tiles - 1 - blockIdx.x / units;
  const int h = unit % a.H, b = unit / a.H;
  const int q0 = tile * BM;
  const bool drop = a.dropout_p > 0.f;
  const T* qbase = reinterpret_cast<const T*>(a.q) + (long long)b * a.q_sb + (long long)h * a.d + (long long)q0 * a.q_sl;
  const T* kbase = reinterpret_cast<const T*>(a.k) + (long long)b * a.k_sb + (long long)h * a.d;
  const T* vbase = reinterpret_cast<const T*>(a.v) + (long long)b * a.v_sb + (long long)h * a.dv;

  const int kend = key_end(a, min(q0 + BM, a.Lq) - 1);
  const int nt = (kend + kBN - 1) / kBN;                   // tiles with a key in reach; the others are all masked
  // step t of 2*nt: the K tile of step t < nt, the V tile t - nt after that
  auto fetch = [&](int t) {
    if (t < nt)
      load_tile<T, kBN, DP, LD, NTHR>(ring + (t & 1) * kBN * LD, kbase + (long long)t * kBN * a.k_sl, a.k_sl,
                                      a.Lkv - t * kBN, a.d, (vec & kVecK) != 0);
    else if (t < 2 * nt)
      load_tile<T, kBN, DP, LD, NTHR>(ring + (t & 1) * kBN * LD, vbase + (long long)(t - nt) * kBN * a.v_sl, a.v_sl,
                                      a.Lkv - (t - nt) * kBN, a.dv, (vec & kVecV) != 0);
    cp_async_commit();
  };
  load_tile<T, BM, DP, LD, NTHR>(qs, qbase, a.q_sl, a.Lq - q0, a.d, (vec & kVecQ) != 0);
  fetch(0);
  if (drop)
    for (int t = 0; t < n_ktiles; ++t)
      fill_keep<NTHR>(keep + t * BM * 8, a, BM, t * kBN, [&](int r) { return score_row(a, q0 + r, h, b); });

  const int d4 = (a.d + 3) >> 2;
  float m[MI];
#pragma unroll
  for (int i = 0; i < MI; ++i) m[i] = ninf();
  for (int t = 0; t < nt; ++t) {
    fetch(t + 1);
    cp_async_wait<1>();
    __syncthreads();
    // nothing but the scale is to be applied to the tile's logits (128 x 128, d = 64, 32 units 15.9 -> 15.2 us)
    const bool plain = !a.bias && !a.mask && q0 + BM <= a.Lq && (t + 1) * kBN <= a.Lkv && (!a.causal || (t + 1) * kBN - 1 <= q0 + a.coff);
    float s[MI][4];
    dot_tile<MI, LD>(qs, ring + (t & 1) * kBN * LD, d4, ty, tx, s);
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int r = ty * MI + i, gi = q0 + r;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kj = t * kBN + tx + 16 * j;
        const float v = plain ? s[i][j] * a.scale
                              : (gi < a.Lq && kj < a.Lkv) ? finish_logit(a, s[i][j], kj, gi, h, b) : ninf();
        ss[r * pitch + kj] = v;
        m[i] = fmaxf(m[i], v);
      }
    }
    __syncthreads();                                       // step t's tile is free for step t + 2
  }

  // a thread reads back the logits it wrote itself
  T* alpha = reinterpret_cast<T*>(a.alpha) + a.alpha_sb * b + (long long)a.Lq * h * a.Lkv;
  if (nt == 0) __syncthreads();                            // the keep bits
  bool nan_out[MI];                                        // a NaN among the scores of the row
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = ty * MI + i, gi = q0 + r;
    const float mr = max16(m[i]);
    bool any_nan = false;
    float l = 0.f;
    for (int k = tx; k < nt * kBN; k += 16) {
      const float p = exp_rel(ss[r * pitch + k], mr);
      ss[r * pitch + k] = p;
      l += p;
    }
    l = sum16(l);
    if (a.lse && tx == 0 && gi < a.Lq) a.lse[gi + (long long)a.Lq * h + a.lse_sb * b] = make_lse(mr, l);
    const bool special = !(l > 0.f);
    const float fixed = (l != l || a.nan_fm) ? qnan() : 0.f;   // every score of such a row
    const float norm = a.inv_keep / l;
    for (int k = tx; k < n_ktiles * kBN; k += 16) {
      float al = special ? fixed : (k < nt * kBN ? ss[r * pitch + k] * norm : 0.f);
      if (drop && !((keep[(k >> 6) * BM * 8 + r * 8 + ((k & 63) >> 3)] >> (k & 7)) & 1)) al = 0.f;
      if (k < a.Lkv) {
        if (gi < a.Lq) alpha[(long long)gi * a.Lkv + k] = Elem<T>::from_f(al);
      } else {
        al = 0.f;
      }
      ss[r * pitch + k] = al;
      any_nan |= al != al;
    }
    nan_out[i] = (__ballot_sync(0xffffffffu, any_nan) >> (threadIdx.x & 16) & 0xffffu) != 0u;
  }

  float o[MI][CN];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int c = 0; c < CN; ++c) o[i][c] = 0.f;
  for (int t = nt; t < 2 * nt; ++t) {
    fetch(t + 1);
    cp_async_wait<1>();
    const float* vt = ring + (t & 1) * kBN * LD;
    const bool bad = tile_not_finite<T, kBN, DP, LD, NTHR>(vt, (vec & kVecV) != 0);
    const bool skip = __syncthreads_or(bad) != 0;
    const int k0 = (t - nt) * kBN;
    accumulate<MI, DP, LD>(ss + k0, pitch, vt, min(kBN, kend - k0), ty, tx, skip, o);
    __syncthreads();
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < MI; ++i) {
    const int r = ty * MI + i, gi = q0 + r;
    if (gi >= a.Lq) continue;
    T* xr = reinterpret_cast<T*>(a.x) + (long long)gi * a.x_sl + (long long)b * a.x_sb + (long long)h * a.dv;
#pragma unroll
    for (int c = 0; c < CN; ++c) {
      const int e = colmap<DP>(tx, c);
      if (e < a.dv) xr[e] = Elem<T>::from_f(nan_out[i] ? qnan() : o[i][c]);
    }
  }
}

// ---- launches ---------------------------------------------------------------------------------------------
// Rows of a block: 64 (8 per thread) reads shared memory least per FMA and is the choice once the blocks fill
// the GPU twice over; 32 when they do not, 8 for a handful of queries (a decode step), where most of a larger
// block would be padding.
template <typename T, int DP, int MI, int MODE, bool AHEAD = false>
cudaError_t launch_fma_mi(const AttnArgs& a, int vec, cudaStream_t st, int n_splits = 1) {
  // Ahead where most tiles can be plain and enough blocks share an SM for their number (two or three instead of three or
  // four) not to matter, by the tiles of 64 x 64 scores: 4 an SM, of causal calls, whose walks differ, 12.  Gains there
  // are 2 to 16 % (742 x 742 of 32 units, d = 64: 5), below them and with a bias or a mask array the same kernels lose as
  // much: 586 x 144 of 32 units, padding 60.0 us, 63.9 ahead; 126 x 343 of 8 units, d = 32, 33.8 and 36.2; 345 x 345 of 64
  // units, causal 95 and 98.  Walks of one or two tiles have nothing to gain: 102 x 102 causal, 320 units 61.5, 64.0 ahead.
  if constexpr (MODE == FM_FWD && DP <= 96 && !AHEAD) {
    const long long tiles = ((a.Lq + 63ll) / 64) * ((a.Lkv + kBN - 1ll) / kBN) * a.H * a.B;
    if (!a.bias && !a.mask && a.Lq >= 128 && a.Lkv > 2 * kBN && tiles >= (a.causal ? 2 * 12 : 4) * 148)
      return launch_fma_mi<T, DP, MI, MODE, true>(a, vec, st, n_splits);
  }
  constexpr int NTHR = 128, BM = NTHR / 16 * MI;
  constexpr int smem = fma_smem<DP, BM, MODE, AHEAD>();
  auto kern = attn_fma_kernel<T, DP, MI, NTHR, MODE, AHEAD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const long long n_tiles = ((long long)a.Lq + BM - 1) / BM, blocks = n_tiles * a.H * a.B;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  int ky = 1;
  if (MODE == FM_SCORES) {   // scores of different key tiles are independent: enough blocks for four per SM
    const long long nkt = ((long long)a.Lkv + kBN - 1) / kBN;
    ky = (int)std::max<long long>(1, std::min<long long>({nkt, (4 * 148 + blocks - 1) / blocks, 65535}));
  }
  if (MODE == FM_SPLIT) ky = n_splits;
  kern<<<dim3((unsigned)blocks, (unsigned)ky), NTHR, smem, st>>>(a, (int)n_tiles, vec);
  count_launch();
  if (MODE == FM_SPLIT) {
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    attn_split_reduce_kernel<T, true><<<(unsigned)(a.H * a.B * a.Lq), 128, 0, st>>>(a, n_splits);
    count_launch();
  }
  return cudaGetLastError();
}

template <typename T, int DP, int MODE>
cudaError_t launch_fma(const AttnArgs& a, int vec, cudaStream_t st) {
  const long long units = (long long)a.H * a.B;
  if constexpr (sizeof(T) == 4) {
    if (a.Lq <= 8) return launch_fma_mi<T, DP, 1, MODE>(a, vec, st);
    if (a.Lq > 32 && units * ((a.Lq + 63) / 64) >= 2 * 148) return launch_fma_mi<T, DP, 8, MODE>(a, vec, st);
  }
  return launch_fma_mi<T, DP, 4, MODE>(a, vec, st);
}

template <typename T, int MODE>
cudaError_t launch_fma_dims(const AttnArgs& a, int dtype, cudaStream_t st) {
  const int dm = MODE == FM_APPLY ? a.dv : (MODE == FM_FWD ? std::max(a.d, a.dv) : a.d);
  const int vec = (rows_vec(a.q, a.q_sl, a.q_sb, a.d, dtype) ? kVecQ : 0) |
                  (rows_vec(a.k, a.k_sl, a.k_sb, a.d, dtype) ? kVecK : 0) |
                  (rows_vec(a.v, a.v_sl, a.v_sb, a.dv, dtype) ? kVecV : 0);
  if constexpr (sizeof(T) == 4) {
    if (dm <= 32) return launch_fma<T, 32, MODE>(a, vec, st);
    if (dm > 64 && dm <= 96) return launch_fma<T, 96, MODE>(a, vec, st);
  }
  if (dm <= 64) return launch_fma<T, 64, MODE>(a, vec, st);
  return launch_fma<T, 128, MODE>(a, vec, st);
}

template <int MODE>
cudaError_t launch_fma_any(const AttnArgs& a, int dtype, cudaStream_t st) {
  if (a.Lq == 0 || a.H == 0 || a.B == 0) return cudaSuccess;
  switch (dtype) {
    case NNLIB_B200_F16:  return launch_fma_dims<__half, MODE>(a, dtype, st);
    case NNLIB_B200_BF16: return launch_fma_dims<__nv_bfloat16, MODE>(a, dtype, st);
    default:              return launch_fma_dims<float, MODE>(a, dtype, st);
  }
}

template <typename T, int DP>
cudaError_t launch_row(const AttnArgs& a, int vec, cudaStream_t st) {
  constexpr int NTHR = 256, MI = 2, BM = NTHR / 16 * MI;
  static_assert(BM == kRowBM, "rows of a block");
  const int nkt = (a.Lkv + kBN - 1) / kBN;
  const int smem = row_smem<DP, BM>(nkt);
  auto kern = attn_fma_row_kernel<T, DP, MI, NTHR>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const long long n_tiles = ((long long)a.Lq + BM - 1) / BM, blocks = n_tiles * a.H * a.B;
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  kern<<<(unsigned)blocks, NTHR, smem, st>>>(a, (int)n_tiles, nkt, vec);
  count_launch();
  return cudaGetLastError();
}

}  // namespace

// Split-key forward, Float32, at most 32 queries: 256 keys (four tiles) per block once there are more than 1024
// (below that one launch is quicker than two).
// A function of the number of keys alone, so that a (head, batch) unit gives the same bits in whatever company it is
// computed.  (Without dropout: the merge does not know whether a row without attended keys kept one.)
int fma_split_count(const AttnArgs& a, int dtype) {
  if (dtype != NNLIB_B200_F32 || a.Lq < 1 || a.Lq > 32 || a.H < 1 || a.B < 1 || !fma_supports(a.d, a.dv) || a.dropout_p > 0.f)
    return 1;
  const long long last = a.causal ? std::min<long long>(a.Lkv, std::max<long long>(0, (long long)a.Lq + a.coff)) : a.Lkv;
  if (last <= 1024 || (long long)a.H * a.B * a.Lq > 0x7fffffffLL) return 1;
  return (int)std::min<long long>((last + 255) / 256, 65535);
}
size_t fma_split_workspace_bytes(const AttnArgs& a, int dtype) {
  const int n = fma_split_count(a, dtype);
  return n > 1 ? (size_t)split_ws_floats(a, n) * sizeof(float) : 0;
}
cudaError_t fma_split(const AttnArgs& a, int dtype, cudaStream_t st) {
  const int n = fma_split_count(a, dtype), dm = std::max(a.d, a.dv);
  const int vec = (rows_vec(a.q, a.q_sl, a.q_sb, a.d, dtype) ? kVecQ : 0) |
                  (rows_vec(a.k, a.k_sl, a.k_sb, a.d, dtype) ? kVecK : 0) |
                  (rows_vec(a.v, a.v_sl, a.v_sb, a.dv, dtype) ? kVecV : 0);
  if (dm <= 64) return a.Lq <= 8 ? launch_fma_mi<float, 64, 1, FM_SPLIT>(a, vec, st, n) : launch_fma_mi<float, 64, 4, FM_SPLIT>(a, vec, st, n);
  return a.Lq <= 8 ? launch_fma_mi<float, 128, 1, FM_SPLIT>(a, vec, st, n) : launch_fma_mi<float, 128, 4, FM_SPLIT>(a, vec, st, n);
}

bool fma_supports(int d, int dv) { return d >= 1 && d <= 128 && dv >= 1 && dv <= 128; }

cudaError_t fma_fwd(const AttnArgs& a, int dtype, cudaStream_t st) { return launch_fma_any<FM_FWD>(a, dtype, st); }
cudaError_t fma_stats(const AttnArgs& a, int dtype, cudaStream_t st) { return launch_fma_any<FM_STATS>(a, dtype, st); }
cudaError_t fma_scores(const AttnArgs& a, int dtype, cudaStream_t st) { return launch_fma_any<FM_SCORES>(a, dtype, st); }
cudaError_t fma_apply(const AttnArgs& a, int dtype, cudaStream_t st) { return launch_fma_any<FM_APPLY>(a, dtype, st); }

// Float32 only (what 16-bit arrays come here is odd enough to take the two launches); the block has to fit
// twice on an SM, or the logits kept in shared memory cost more in occupancy than they save.
bool fma_row_supports(const AttnArgs& a, int dtype) {
  if (dtype != NNLIB_B200_F32 || a.Lkv < 1 || !fma_supports(a.d, a.dv)) return false;
  const int nkt = (a.Lkv + kBN - 1) / kBN, dm = std::max(a.d, a.dv);
  if (nkt > 64) return false;
  const int smem = dm <= 32 ? row_smem<32, kRowBM>(nkt) : dm <= 64 ? row_smem<64, kRowBM>(nkt)
                 : dm <= 96 ? row_smem<96, kRowBM>(nkt) : row_smem<128, kRowBM>(nkt);
  return smem <= 113 * 1024;
}
cudaError_t fma_row(const AttnArgs& a, int dtype, cudaStream_t st) {
  const int dm = std::max(a.d, a.dv);
  const int vec = (rows_vec(a.q, a.q_sl, a.q_sb, a.d, dtype) ? kVecQ : 0) |
                  (rows_vec(a.k, a.k_sl, a.k_sb, a.d, dtype) ? kVecK : 0) |
                  (rows_vec(a.v, a.v_sl, a.v_sb, a.dv, dtype) ? kVecV : 0);
  if (dm <= 32) return launch_row<float, 32>(a, vec, st);
  if (dm <= 64) return launch_row<float, 64>(a, vec, st);
  if (dm <= 96) return launch_row<float, 96>(a, vec, st);
  return launch_row<float, 128>(a, vec, st);
}

}  // namespace nb200
