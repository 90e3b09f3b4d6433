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
//
// With a workspace there is another form, of one pass: every block owns 64 keys and computes a tile of scores once, with
// five products instead of the two kinds' seven, and leaves its share of the queries' dq in the workspace, 16 KB a tile at
// d = 64; a third launch adds the shares up, in the same order every time.  Where the keys alone make too few blocks, the
// walks over the queries are cut as well and dk and dv are put together in the same way.  What bounds a tile is shared
// memory: 4 x 4 scores a thread read 8 floats for 16 multiply-adds.
// Backward at d = 64, 8 heads, 512 x 512 causal, batch 8: 306 us in two halves, 234 in one pass (222 with atomic
// additions of dq, whose bits change from call to call); 16 heads, 2048 x 2048 causal 1025 and 736; 2 units of 1815 x 1815
// 385 and 187; 4 units of 128 keys and 2000 queries 424 and 41, of 4000 keys and 40 queries 653 and 43.  One training step
// (forward and backward) of the first: 23.06 ms with the warp-per-row kernels, 0.44 ms in two halves, 0.36 in one pass.
#include <algorithm>

#include "common.cuh"
#include "fma_tile.cuh"
#include "launchers.h"

namespace nb200 {
namespace {

using namespace fma_tile;

constexpr int kBM = 64;                                    // rows a block owns
constexpr int kVecQ = 1, kVecK = 2, kVecV = 4, kVecD = 8;  // 16-byte copies of that array's rows are possible

// D_i = dx_i . x_i, sixteen lanes a query; rows of 16-byte pieces (VEC) are read as such
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) attn_bwd_delta_kernel(const AttnArgs a, const BwdArgs g) {
  const int lane = threadIdx.x & 15;
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 4);
  const bool row_ok = row < (long long)a.Lq * a.H * a.B;
  float dl = 0.f;
  if (row_ok) {
    const int i = (int)(row % a.Lq), h = (int)((row / a.Lq) % a.H), b = (int)(row / ((long long)a.Lq * a.H));
    const T* xrow = reinterpret_cast<const T*>(a.x) + (long long)i * a.x_sl + (long long)b * a.x_sb + (long long)h * a.dv;
    const T* dxrow = reinterpret_cast<const T*>(g.dx) + (long long)i * g.dx_sl + (long long)b * g.dx_sb + (long long)h * a.dv;
    if constexpr (VEC) {
      for (int e = lane * 4; e < a.dv; e += 64) {
        const float4 x = *reinterpret_cast<const float4*>(xrow + e), y = *reinterpret_cast<const float4*>(dxrow + e);
        dl = fmaf(y.x, x.x, dl);
        dl = fmaf(y.y, x.y, dl);
        dl = fmaf(y.z, x.z, dl);
        dl = fmaf(y.w, x.w, dl);
      }
    } else {
      for (int e = lane; e < a.dv; e += 16) dl = fmaf(Elem<T>::to_f(dxrow[e]), Elem<T>::to_f(xrow[e]), dl);
    }
  }
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) dl += __shfl_xor_sync(0xffffffffu, dl, off);
  if (row_ok && lane == 0) g.delta[row] = dl;
}

template <int DP>
__host__ __device__ constexpr int bwd_smem() { return 4 * (4 * kBM * (DP + 4) + 2 * kBM * kLDP) + kBM * 8; }

// Workspace of the one-pass form, in floats: D of all queries, then per unit and tile of 64 queries one partial dq from
// every tile of keys, then, where the walks are cut into chunks, per unit and tile of keys one partial dk and dv from
// every chunk.  Rows are dd = d (dv) rounded up to 4.
struct Parts {
  int kt, qt, chunks, len, dd, dvd;   // tiles, chunks of a walk, query tiles of a chunk
  long long dq_off, dk_off, floats;
};
inline Parts make_parts(const AttnArgs& a) {
  Parts p;
  p.kt = (a.Lkv + kBM - 1) / kBM;
  p.qt = (a.Lq + kBN - 1) / kBN;
  p.len = fma_bwd_chunk(a);
  p.chunks = (p.qt + p.len - 1) / p.len;
  p.dd = (a.d + 3) & ~3;
  p.dvd = (a.dv + 3) & ~3;
  const long long units = (long long)a.H * a.B;
  p.dq_off = ((long long)a.Lq * units + 3) & ~3ll;
  p.dk_off = p.dq_off + units * p.qt * p.kt * (kBN * p.dd);
  p.floats = p.dk_off + (p.chunks > 1 ? units * p.kt * p.chunks * (kBM * (p.dd + p.dvd)) : 0);
  return p;
}
// first query that the keys of tile `t` are seen by, rounded down to a tile
__device__ __forceinline__ int first_query(const AttnArgs& a, int t) {
  const long long first = (long long)t * kBM - a.coff;
  return !a.causal || first <= 0 ? 0 : (first < a.Lq ? (int)first / kBN * kBN : a.Lq);
}

// a thread's columns of a row of a partial result
template <int DP>
__device__ __forceinline__ void put_part(float* row, const float (&v)[DP / 16], float mul, int tx, int dd) {
#pragma unroll
  for (int c = 0; c < DP / 16; c += 2) {
    const int e = colmap<DP>(tx, c);
    if ((c & 3) == 0 && c + 3 < DP / 16) {
      if (e < dd) *reinterpret_cast<float4*>(row + e) = make_float4(v[c] * mul, v[c + 1] * mul, v[c + 2] * mul, v[c + 3] * mul);
    } else if ((c & 3) == 0) {
      if (e < dd) *reinterpret_cast<float2*>(row + e) = make_float2(v[c] * mul, v[c + 1] * mul);   // (dd is even)
    }
  }
}

// KEYS: the block owns keys (dk, dv); else queries (dq, dbias).  ALL (with KEYS, Float32): it walks over chunk `chunk` of
// the query tiles and leaves its part of their dq, and of dk and dv if there are several chunks, in the workspace.
template <typename T, int DP, int NTHR, bool KEYS, bool ALL>
__device__ __forceinline__ void bwd_block(const AttnArgs& a, const BwdArgs& g, const int tile, const int unit, const int vec,
                                          float* sm, const Parts& ws, const int chunk) {
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
  const bool part = ALL && ws.chunks > 1;
  if (ALL) {
    c_begin = max(c_begin, chunk * ws.len * kBN);
    c_end = min(c_end, (int)min((long long)n_cols, (long long)(chunk + 1) * ws.len * kBN));
    if (part && c_begin >= c_end) {    // the merge knows
      cp_async_commit();
      cp_async_wait<0>();
      return;
    }
  }
  const int d4 = (a.d + 3) >> 2, dv4 = (a.dv + 3) >> 2;
  bool a1_bad = false;
  if (ALL) {                         // a key that takes no part may hold anything (accumulate_t)
    cp_async_commit();
    cp_async_wait<0>();
    a1_bad = __syncthreads_or(tile_not_finite<T, kBM, DP, LD, NTHR>(a1, (vec & kVecK) != 0)) != 0;
  }
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
    // nothing but the scale is to be applied to the tile's logits
    const bool plain = !a.bias && !a.mask && !drop && r0 + kBM <= n_rows && c0 + kBN <= n_cols &&
                       (!a.causal || j0 + kBN - 1 <= i0 + a.coff);
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
        if (plain) {
          const float t = p[i][j] * a.scale;
          if (L != ninf() && t != ninf()) pv = expf(t - L);
        } else if (gr < n_rows && gc < n_cols && L != ninf()) {
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
    if constexpr (ALL) {
      float o[MI][CN];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int c = 0; c < CN; ++c) o[i][c] = 0.f;
      accumulate_t<MI, DP, LD>(ds, kLDP, a1, ty, tx, a1_bad, o);
#pragma unroll
      for (int i = 0; i < MI; ++i)
        put_part<DP>(a.ws + ws.dq_off + (((long long)unit * ws.qt + c0 / kBN) * ws.kt + tile) * (kBN * ws.dd) +
                     (ty * MI + i) * ws.dd, o[i], a.scale, tx, ws.dd);
    }
    __syncthreads();
  }
  cp_async_wait<0>();

  T* o1 = reinterpret_cast<T*>(KEYS ? g.dk : g.dq) + (long long)n_rows * b * ((long long)a.H * a.d) + (long long)h * a.d;
  T* o2 = reinterpret_cast<T*>(g.dv) + (long long)n_rows * b * ((long long)a.H * a.dv) + (long long)h * a.dv;
  if constexpr (ALL) {
    if (part) {
      float* w = a.ws + ws.dk_off + (((long long)unit * ws.kt + tile) * ws.chunks + chunk) * (kBM * (ws.dd + ws.dvd)) + ty * MI * ws.dd;
      float* wv = w + kBM * ws.dd + ty * MI * (ws.dvd - ws.dd);
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        put_part<DP>(w + i * ws.dd, acc1[i], a.scale, tx, ws.dd);
        put_part<DP>(wv + i * ws.dvd, acc2[i], 1.f, tx, ws.dvd);
      }
      return;
    }
  }
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

template <typename T, int DP, int NTHR, bool ALL>
__global__ void __launch_bounds__(NTHR, DP <= 64 ? 2 : 1)
attn_bwd_fma_kernel(const AttnArgs a, const BwdArgs g, const int nkt, const int nqt, const int vec, const Parts ws) {
  extern __shared__ __align__(16) float sm[];
  const int units = a.H * a.B;
  const int t = blockIdx.x / units, unit = blockIdx.x % units;
  // causal: the first keys are seen by the most queries, the last queries see the most keys
  if (ALL) bwd_block<T, DP, NTHR, true, ALL>(a, g, t / ws.chunks, unit, vec, sm, ws, t % ws.chunks);
  else if (t < nkt) bwd_block<T, DP, NTHR, true, false>(a, g, t, unit, vec, sm, ws, 0);
  else bwd_block<T, DP, NTHR, false, false>(a, g, nkt + nqt - 1 - t, unit, vec, sm, ws, 0);
}

// The parts of the one-pass form added up, always in the same order.  A block sums 1024 elements (a thread four) of the
// 64 rows of one tile of queries (dq) or, behind those, of keys (dk and dv).
__global__ void __launch_bounds__(256) attn_bwd_fma_merge_kernel(const AttnArgs a, const BwdArgs g, const Parts ws) {
  const int units = a.H * a.B;
  const int e = (blockIdx.y * 256 + threadIdx.x) * 4;
  int t = blockIdx.x / units;
  const int unit = blockIdx.x % units, h = unit % a.H, b = unit / a.H;
  const bool keys = t >= ws.qt;
  if (keys) t -= ws.qt;
  const float* w;
  long long stride;
  int n, first = 0, row, col, width, d = a.d;
  float* out;
  long long rows;
  if (!keys) {
    width = ws.dd;
    row = e / width; col = e % width;
    out = reinterpret_cast<float*>(g.dq);
    rows = a.Lq;
    stride = kBN * ws.dd;
    w = a.ws + ws.dq_off + ((long long)unit * ws.qt + t) * ws.kt * stride + e;
    // tiles of keys that the queries see any of: the first so many
    n = ws.kt;
    if (a.causal)
      for (n = 0; n < ws.kt && first_query(a, n) <= t * kBN;) ++n;
  } else {
    const bool v = e >= kBM * ws.dd;
    const int f = v ? e - kBM * ws.dd : e;
    width = v ? ws.dvd : ws.dd;
    row = f / width; col = f % width;
    out = reinterpret_cast<float*>(v ? g.dv : g.dk);
    rows = a.Lkv;
    stride = kBM * (ws.dd + ws.dvd);
    w = a.ws + ws.dk_off + ((long long)unit * ws.kt + t) * ws.chunks * stride + e;
    const int q = first_query(a, t);
    first = q / (ws.len * kBN);
    n = q < a.Lq ? ws.chunks : 0;
    d = v ? a.dv : a.d;
  }
  if (row >= kBM || (long long)t * kBM + row >= rows) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int k = first; k < n; ++k) {
    const float4 f = *reinterpret_cast<const float4*>(w + k * stride);
    s.x += f.x; s.y += f.y; s.z += f.z; s.w += f.w;
  }
  float* o = out + ((long long)t * kBM + row + rows * b) * ((long long)a.H * d) + (long long)h * d + col;
  const float r[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (col + u < d) o[u] = r[u];
}

template <typename T, int DP, int NTHR, bool ALL>
cudaError_t launch_bwd_form(const AttnArgs& a, const BwdArgs& g, int vec, cudaStream_t st) {
  const long long rows = (long long)a.Lq * a.H * a.B, db = (rows + 7) / 8;
  const int nkt = (a.Lkv + kBM - 1) / kBM, nqt = (a.Lq + kBM - 1) / kBM;
  Parts ws = {};
  if (ALL) ws = make_parts(a);
  const long long blocks = (ALL ? (long long)nkt * ws.chunks : (long long)nkt + nqt) * a.H * a.B;
  if (db > 0x7fffffffLL || blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  if (db > 0) {
    bool dvec = false;
    if constexpr (sizeof(T) == 4) {
      dvec = (vec & kVecD) != 0 && rows_vec(a.x, a.x_sl, a.x_sb, a.dv, NNLIB_B200_F32);
      if (dvec) attn_bwd_delta_kernel<T, true><<<(unsigned)db, 128, 0, st>>>(a, g);
    }
    if (!dvec) attn_bwd_delta_kernel<T, false><<<(unsigned)db, 128, 0, st>>>(a, g);
    count_launch();
  }
  if (blocks > 0) {
    auto kern = attn_bwd_fma_kernel<T, DP, NTHR, ALL>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_smem<DP>());
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)blocks, NTHR, bwd_smem<DP>(), st>>>(a, g, nkt, nqt, vec, ws);
    count_launch();
    if (ALL) {
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      const int keys = ws.chunks > 1, floats = kBM * (keys ? ws.dd + ws.dvd : ws.dd);
      attn_bwd_fma_merge_kernel<<<dim3((unsigned)((ws.qt + (keys ? ws.kt : 0)) * a.H * a.B), (unsigned)((floats + 1023) / 1024)), 256, 0,
                                  st>>>(a, g, ws);
      count_launch();
    }
  }
  return cudaGetLastError();
}

template <typename T, int DP, int NTHR>
cudaError_t launch_bwd(const AttnArgs& a, const BwdArgs& g, int vec, cudaStream_t st) {
  if constexpr (sizeof(T) == 4) {
    if (a.ws) return launch_bwd_form<T, DP, NTHR, true>(a, g, vec, st);
  }
  return launch_bwd_form<T, DP, NTHR, false>(a, g, vec, st);
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

// One pass: how many query tiles a block walks over.  All of them where the blocks of keys alone fill the GPU; otherwise
// so few that there are one and a half times as many blocks as fit on it at once.
int fma_bwd_chunk(const AttnArgs& a) {
  const long long kt = (a.Lkv + kBM - 1) / kBM, qt = (a.Lq + kBN - 1) / kBN, blocks = kt * a.H * a.B;
  const long long at_once = 148 * (a.d <= 64 && a.dv <= 64 ? 2 : 1);
  if (blocks >= at_once) return (int)std::max(qt, 1ll);
  const long long chunks = std::max(1ll, std::min(qt, (3 * at_once / 2 + blocks - 1) / std::max(blocks, 1ll)));
  return (int)((qt + chunks - 1) / chunks);
}

size_t fma_bwd_workspace_bytes(const AttnArgs& a) { return (size_t)make_parts(a).floats * sizeof(float); }

cudaError_t fma_bwd(const AttnArgs& a, const BwdArgs& g, int dtype, cudaStream_t st) {
  if (a.H == 0 || a.B == 0) return cudaSuccess;
  switch (dtype) {
    case NNLIB_B200_F16:  return launch_bwd_dims<__half>(a, g, dtype, st);
    case NNLIB_B200_BF16: return launch_bwd_dims<__nv_bfloat16>(a, g, dtype, st);
    default:              return launch_bwd_dims<float>(a, g, dtype, st);
  }
}

}  // namespace nb200
