// Few queries (at most 16) against many keys: one generated token, or a handful, against a key / value history.
//
// Every byte of K and V is used once per query, so HBM is the bound (one query: 4 FLOPs per 2 bytes and key
// feature), and what counts is how many bytes are in flight.  The 128-row tcgen05 tiles of the other forward
// kernels would be padding but for a few rows, and their one CTA per SM leaves the memory system waiting while
// the last tile's scores go through the softmax; here nothing is staged: warps stream K and V straight from
// global memory into the fragments of the 16-row warp-level products, eight 16-byte loads of each array ahead,
// every warp on its own keys.
//
//   S  = Q K^T   m16n8k16: rows = queries, columns = keys.  The contraction may run over the features in any
//                order, so lane (g, c) = (lane / 4, lane % 4) takes the 8 consecutive features 32 G + 8 c .. of key g
//                (one 16-byte load) as its part of two k-steps, and Q's fragments are loaded in the same order.
//   O += P V     the columns may be any features, so column g of product j is feature 64 F + 8 g + j: lane (g, c)
//                loads 16 bytes (j = 0 .. 7) of each of its four keys 2c, 2c+1, 2c+8, 2c+9 and pairs up the
//                halves of two keys with byte permutes.
// A warp takes 16 keys at a time, the four warps of a CTA alternate; a CTA covers a contiguous share of a unit's
// keys, merges its warps' running maxima, sums and outputs through shared memory and leaves the partial result in
// the workspace, where attn_split_reduce_kernel merges the shares.
// The logits carry no side input here (causal flag only): calls with a bias, a mask array or dropout take
// the other kernels.
#include <algorithm>

#include "common.cuh"
#include "launchers.h"
#include "split_reduce.cuh"

namespace nb200 {
namespace {

constexpr int kDecWarps = 4;
constexpr int kDecKeys = 16;            // keys a warp takes per step
constexpr float kLog2eD = 1.4426950408889634f;

__device__ __forceinline__ float dec_ninf() { return __int_as_float(0xff800000); }

__device__ __forceinline__ float dec_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 16 bytes that nobody reads again: not kept in L1
__device__ __forceinline__ uint4 load_stream(const void* p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// D = A B + C, 16 x 8 x 16; ROWS8: rows 8 .. 15 of A are zero and theirs of the result are not wanted
template <bool BF16, bool ROWS8>
__device__ __forceinline__ void mma16(float (&c)[ROWS8 ? 2 : 4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                      uint32_t b0, uint32_t b1) {
  if constexpr (ROWS8) {
    float u, v;
    if constexpr (BF16)
      asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %10, %10};"
          : "+f"(c[0]), "+f"(c[1]), "=f"(u), "=f"(v) : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.f));
    else
      asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %10, %10};"
          : "+f"(c[0]), "+f"(c[1]), "=f"(u), "=f"(v) : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    if constexpr (BF16)
      asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
          : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
      asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
          : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
}

template <bool BF16>
__device__ __forceinline__ uint32_t dec_pack2(float lo, float hi) {
  if constexpr (BF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}

__device__ __forceinline__ uint32_t u4w(const uint4& q, int w) { return w == 0 ? q.x : (w == 1 ? q.y : (w == 2 ? q.z : q.w)); }

// One past the last key any query of the call attends to.
__host__ __device__ inline int dec_key_end(const AttnArgs& a) {
  if (!a.causal) return a.Lkv;
  const long long e = (long long)a.Lq + a.coff;
  return e <= 0 ? 0 : (e < a.Lkv ? (int)e : a.Lkv);
}

// CTAs that fit an SM together: what registers allow without spilling the fragments in flight
template <int D, bool ROWS8>
struct DecCfg { static constexpr int kCtas = (D == 64) ? 4 : 2; };

template <typename T, int D, bool ROWS8>
__global__ void __launch_bounds__(kDecWarps * 32, DecCfg<D, ROWS8>::kCtas)
attn_decode_kernel(const AttnArgs a, const int n_splits, const int steps_per_split, const int splits_per_cta) {
  constexpr bool BF16 = sizeof(T) == 2 && !std::is_same<T, __half>::value;
  constexpr int R = ROWS8 ? 1 : 2;                 // rows of a lane: g, g + 8
  constexpr int GQ = D / 32, GV = D / 64;
  constexpr int ROWS = 8 * R;
  __shared__ float sm_o[kDecWarps][ROWS][D];
  __shared__ float sm_m[kDecWarps][ROWS], sm_l[kDecWarps][ROWS];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  // the heads of one batch element side by side: what runs at one time then reads whole rows of k and v, not one
  // head's 256 bytes of each
  const int units = a.H * a.B, unit = blockIdx.x % units;
  int split = blockIdx.x / units * splits_per_cta;           // this CTA's shares: split .. split_end - 1
  const int split_end = min(n_splits, split + splits_per_cta);
  const int h = unit % a.H, b = unit / a.H;
  const int kend = dec_key_end(a);
  const int n_steps = (kend + kDecKeys - 1) / kDecKeys;
  const float c2 = a.scale * kLog2eD;

  const T* kbase = reinterpret_cast<const T*>(a.k) + (long long)b * a.k_sb + (long long)h * a.d;
  const T* vbase = reinterpret_cast<const T*>(a.v) + (long long)b * a.v_sb + (long long)h * a.dv;
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);

  uint4 qf[R][GQ];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = g + 8 * r;
    const T* qp = reinterpret_cast<const T*>(a.q) + (long long)i * a.q_sl + (long long)b * a.q_sb + (long long)h * a.d;
#pragma unroll
    for (int G = 0; G < GQ; ++G) {
      const int f = 32 * G + 8 * c;
      qf[r][G] = (i < a.Lq && f < a.d) ? *reinterpret_cast<const uint4*>(qp + f) : zero4;
    }
  }
  // keys of step s; past the end the last attended key of K is read again (its score is not used) and V is zero (the
  // weight there is zero, but 0 * Inf would be a NaN; zeroing V where it is used instead costs every step 2 %)
  uint4 kf[2][GQ], vf[4][GV];
  auto load_k = [&](int s) {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const T* kp = kbase + (long long)min(s * kDecKeys + nt * 8 + g, kend - 1) * a.k_sl;
#pragma unroll
      for (int G = 0; G < GQ; ++G) {
        const int f = 32 * G + 8 * c;
        kf[nt][G] = (f < a.d) ? load_stream(kp + f) : zero4;
      }
    }
  };
  auto load_v = [&](int s) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = s * kDecKeys + 2 * c + (u & 1) + (u >> 1) * 8;
      const T* vp = vbase + (long long)j * a.v_sl;
#pragma unroll
      for (int F = 0; F < GV; ++F) {
        const int f = 64 * F + 8 * g;
        vf[u][F] = (f < a.dv && j < kend) ? load_stream(vp + f) : zero4;
      }
    }
  };

  float m[R], l[R], o[GV][8][2 * R];
  auto first_step = [&](int sp) { return sp * steps_per_split + warp; };
  auto end_step = [&](int sp) { return min(n_steps, (sp + 1) * steps_per_split); };
  // the step after s of share sp: of the same share, or the warp's first of the next one (its loads are then under
  // way while this share is merged); -1: none
  auto next_step = [&](int s, int sp) {
    if (s + kDecWarps < end_step(sp)) return s + kDecWarps;
    return (sp + 1 < split_end && first_step(sp + 1) < end_step(sp + 1)) ? first_step(sp + 1) : -1;
  };
  if (split < split_end && first_step(split) < end_step(split)) {
    load_k(first_step(split));
    load_v(first_step(split));
  }
  for (; split < split_end; ++split) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      m[r] = dec_ninf();
      l[r] = 0.f;
    }
#pragma unroll
    for (int F = 0; F < GV; ++F)
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 2 * R; ++e) o[F][j][e] = 0.f;

    const int s_end = end_step(split);
    // (a warp without a step in this share has none in the next one either: only the last share is not full)
    for (int s = first_step(split); s < s_end; s += kDecWarps) {
      const int s_next = next_step(s, split);
      float sc[2][2 * R];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
        for (int e = 0; e < 2 * R; ++e) sc[nt][e] = 0.f;
#pragma unroll
        for (int G = 0; G < GQ; ++G) {
          mma16<BF16, ROWS8>(sc[nt], qf[0][G].x, qf[R - 1][G].x, qf[0][G].y, qf[R - 1][G].y, kf[nt][G].x, kf[nt][G].y);
          mma16<BF16, ROWS8>(sc[nt], qf[0][G].z, qf[R - 1][G].z, qf[0][G].w, qf[R - 1][G].w, kf[nt][G].z, kf[nt][G].w);
        }
      }
      if (s_next >= 0) load_k(s_next);

      const int j0 = s * kDecKeys + 2 * c;           // this lane's keys: j0, j0 + 1, j0 + 8, j0 + 9
      uint32_t pa[R][2];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = g + 8 * r;
        const int lim = (a.causal ? min(i + a.coff, a.Lkv - 1) : a.Lkv - 1);   // last key of this query
        float t[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          t[u] = sc[u >> 1][2 * r + (u & 1)] * c2;
          if (j0 + (u & 1) + (u >> 1) * 8 > lim) t[u] = dec_ninf();
        }
        float mx = fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mn = fmaxf(m[r], mx);
        if (__any_sync(0xffffffffu, mn > m[r])) {
          const float f = (m[r] == dec_ninf()) ? 0.f : dec_ex2(m[r] - mn);   // (a row without any key so far holds zeros)
          l[r] *= f;
#pragma unroll
          for (int F = 0; F < GV; ++F)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              o[F][j][2 * r] *= f;
              o[F][j][2 * r + 1] *= f;
            }
          m[r] = mn;
        }
        const float ref = (mn == dec_ninf()) ? 0.f : mn;
        float p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = dec_ex2(t[u] - ref);
        l[r] += (p[0] + p[1]) + (p[2] + p[3]);       // this lane's keys only; the four lanes are added at the end
        pa[r][0] = dec_pack2<BF16>(p[0], p[1]);
        pa[r][1] = dec_pack2<BF16>(p[2], p[3]);
      }
#pragma unroll
      for (int F = 0; F < GV; ++F)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;   // the high or the low halves of two words
          const uint32_t b0 = __byte_perm(u4w(vf[0][F], j >> 1), u4w(vf[1][F], j >> 1), sel);
          const uint32_t b1 = __byte_perm(u4w(vf[2][F], j >> 1), u4w(vf[3][F], j >> 1), sel);
          mma16<BF16, ROWS8>(o[F][j], pa[0][0], pa[R - 1][0], pa[0][1], pa[R - 1][1], b0, b1);
        }
      if (s_next >= 0) load_v(s_next);
    }

    // merge the four warps
    __syncthreads();                                         // the last share's statistics and outputs have been read
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int row = g + 8 * r;
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
      l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
      if (c == 0) {
        sm_m[warp][row] = m[r];
        sm_l[warp][row] = l[r];
      }
      // columns 2c and 2c+1 of product j: features 64 F + 16 c + j and + 8
#pragma unroll
      for (int F = 0; F < GV; ++F)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(&sm_o[warp][row][64 * F + 16 * c + 8 * e + j]) =
                make_float4(o[F][j][2 * r + e], o[F][j + 1][2 * r + e], o[F][j + 2][2 * r + e], o[F][j + 3][2 * r + e]);
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < a.Lq * D; idx += kDecWarps * 32) {
      const int i = idx / D, e = idx % D;
      float M = dec_ninf(), L = 0.f, acc = 0.f;
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) M = fmaxf(M, sm_m[w][i]);
#pragma unroll
      for (int w = 0; w < kDecWarps; ++w) {
        const float f = (sm_m[w][i] == dec_ninf()) ? 0.f : dec_ex2(sm_m[w][i] - M);
        // (a warp that met nothing but NaN logits still has the maximum -Inf: its sum says so)
        L += (sm_l[w][i] != sm_l[w][i]) ? sm_l[w][i] : f * sm_l[w][i];
        acc = fmaf(f, sm_o[w][i][e], acc);
      }
      const long long slot = ((long long)unit * n_splits + split) * a.Lq + i;
      if (e == 0) {
        a.ws[slot * 2] = M;
        a.ws[slot * 2 + 1] = L;
      }
      if (e < a.dv) a.ws[split_ml_floats(a, n_splits) + slot * a.dv + e] = acc;
    }
  }
}

template <typename T, int D, bool ROWS8>
cudaError_t launch_decode(const AttnArgs& a, int n_splits, cudaStream_t st) {
  const int n_steps = (dec_key_end(a) + kDecKeys - 1) / kDecKeys;
  const int per = std::max(1, (n_steps + n_splits - 1) / n_splits);   // (every share but the last one whole)
  // consecutive shares of a unit in one CTA, as long as every SM still gets four rounds of the CTAs that fit it: a
  // share's first loads are then in flight while the one before is merged
  const long long units = (long long)a.H * a.B, slots = 148LL * DecCfg<D, ROWS8>::kCtas;
  const int spc = (int)std::max<long long>(1, std::min<long long>(n_splits, units * n_splits / (4 * slots)));
  const long long blocks = units * ((n_splits + spc - 1) / spc);
  if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  attn_decode_kernel<T, D, ROWS8><<<(unsigned)blocks, kDecWarps * 32, 0, st>>>(a, n_splits, per, spc);
  count_launch();
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  attn_split_reduce_kernel<T, false><<<(unsigned)(a.H * a.B * a.Lq), 128, 0, st>>>(a, n_splits);
  count_launch();
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_decode_dims(const AttnArgs& a, int n_splits, cudaStream_t st) {
  if (a.d <= 64 && a.dv <= 64)
    return a.Lq <= 8 ? launch_decode<T, 64, true>(a, n_splits, st) : launch_decode<T, 64, false>(a, n_splits, st);
  return a.Lq <= 8 ? launch_decode<T, 128, true>(a, n_splits, st) : launch_decode<T, 128, false>(a, n_splits, st);
}

bool dec_stride_ok(long long s) { return s > 0 && s % 8 == 0; }

}  // namespace

bool decode_supports(const AttnArgs& a, int dtype) {
  if (dtype != NNLIB_B200_F16 && dtype != NNLIB_B200_BF16) return false;
  if (a.Lq < 1 || a.Lq > 16 || a.Lkv < 1 || a.H < 1 || a.B < 1) return false;
  if (a.bias || a.mask || a.dropout_p > 0.f || !(a.scale > 0.f)) return false;
  if (a.d < 8 || a.d > 128 || a.d % 8 != 0 || a.dv < 8 || a.dv > 128 || a.dv % 8 != 0) return false;
  const void* ptrs[] = {a.q, a.k, a.v, a.x};
  for (const void* p : ptrs)
    if ((reinterpret_cast<uintptr_t>(p) & 15u) != 0) return false;
  const long long strides[] = {a.q_sl, a.q_sb, a.k_sl, a.k_sb, a.v_sl, a.v_sb};
  for (long long s : strides)
    if (!dec_stride_ok(s)) return false;
  return dec_key_end(a) > 0 && (long long)a.H * a.B * a.Lq <= 0x7fffffffLL &&
         (long long)a.H * a.B * (a.Lkv / 256 + 1) <= 0x7fffffffLL;
}

// Shares the keys of one unit are cut into.  A function of the number of keys alone, so that a (head, batch) unit gives
// the same bits in whatever company it is computed (a shard of a larger call, a batch of another size): 512 keys each,
// 1024 from 8192 keys on, where many units pay for the set-up and merge of a share (one query, d = 128, 256 units, bf16,
// in a graph: 8191 keys 198 us, 8192 keys 187 us = 5.7 TB/s; the two-tile kernel 200 and 209).  Few units pay for the
// longer shares instead (8 units, with a slower merge than now: 8191 keys 17.8 us, 8192 keys 20.5, both 34.6 with their
// keys split by the number of units on the one-tile kernels).  Up to 1024 keys (2048 for more than 8 queries, whose
// fragments take twice the registers) the call is left to the other kernels, whose one launch takes less than two (384
// keys, 256 units, d = 64: 23.5 us against 28.9; 16 queries, 1408 keys, 192 units: 45.1 against 47.1).
int decode_split_count(const AttnArgs& a) {
  const int kend = dec_key_end(a), per = kend < 8192 ? 512 : 1024;
  return kend > (a.Lq <= 8 ? 1024 : 2048) ? (kend + per - 1) / per : 1;
}
// Is a call of `units` units better left to the two-tile forward, one CTA per unit?  With heads of more than 64 features
// that kernel streams K and V about as fast once every SM has a CTA, so what decides is how full its last wave is:
// units / (148 waves).  This kernel's side of the scale grows with the queries (their fragments, 8 and 16 of them a
// step longer, and their partial outputs) and falls with the keys.  Times of this kernel over the other's, d = 128, 4096
// keys, at 96 / 128 / 148 | 192 / 256 / 288 units (65, 86, 100 | 65, 86, 97 %): 1 query 0.82 1.04 1.09 | 0.78 0.94 1.04,
// 4 queries 0.85 1.08 1.13 | 0.82 0.98 1.09, 8 queries 0.90 1.15 1.20 | 0.88 1.04 1.16, 16 queries 1.06 1.35 1.41 |
// 1.05 1.23 1.36; at 16384 keys 0.76 0.92 1.03 | 0.74 0.92 0.99, ..., 0.91 1.08 1.19 | 0.88 1.09 1.15.  The percentages
// below are where the ratio passes 1, in one wave | in more (101: nowhere); heads padded to 128 are 6 % better off here.
bool decode_leaves(const AttnArgs& a, long long units) {
  if (a.d <= 64 && a.dv <= 64) return false;
  constexpr int kFull[2][4][2] = {{{80, 101}, {80, 97}, {75, 86}, {56, 64}},       // fewer than 8192 keys in reach
                                  {{93, 101}, {93, 101}, {85, 95}, {75, 80}}};
  const long long waves = (units + 147) / 148;
  const int q = a.Lq <= 2 ? 0 : (a.Lq <= 4 ? 1 : (a.Lq <= 8 ? 2 : 3));
  const int full = kFull[dec_key_end(a) < 8192 ? 0 : 1][q][waves > 1 ? 1 : 0] + (a.d < 128 ? 6 : 0);
  return units * 100 >= full * waves * 148;
}
size_t decode_workspace_bytes(const AttnArgs& a) {
  const int n = decode_split_count(a);
  return n > 1 ? (size_t)split_ws_floats(a, n) * sizeof(float) : 0;   // 0: not split
}
cudaError_t decode_fwd(const AttnArgs& a, int dtype, int n_splits, cudaStream_t st) {
  return dtype == NNLIB_B200_BF16 ? launch_decode_dims<__nv_bfloat16>(a, n_splits, st) : launch_decode_dims<__half>(a, n_splits, st);
}

}  // namespace nb200
