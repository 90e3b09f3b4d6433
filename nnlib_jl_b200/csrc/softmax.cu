// softmax / logsoftmax over one dimension of a column-major array and their
// pullbacks (NNlib.jl src/softmax.jl:69-79 `_softmax!`, :147-157
// `_logsoftmax!`, :98-101 `_∇softmax!`, :170-190 `∇logsoftmax`), the op in the
// middle of the attention path as a stand-alone entry point.
//
// The array is seen as (inner, n, outer) with the reduction over the middle
// extent: element (i, j, o) lives at i + inner*(j + n*o).  Bound by HBM: one
// read and one write per element (the second pass over a column re-reads it
// from L2).  Arithmetic in fp32 whatever the element type.
//
// Non-finite inputs follow the reference (src/softmax.jl:71-76): a column
// whose maximum is +Inf puts its weight on the +Inf entries in equal shares, a
// column whose maximum is -Inf or that contains a NaN becomes NaN.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <type_traits>
#include "common.cuh"
#include "launchers.h"

namespace nb200 {
namespace {

enum : int { SM_FWD = 0, LSM_FWD = 1, SM_BWD = 2, LSM_BWD = 3 };

__device__ __forceinline__ float f_inf() { return __int_as_float(0x7f800000); }
__device__ __forceinline__ float f_ninf() { return __int_as_float(0xff800000); }
__device__ __forceinline__ float f_nan() { return __int_as_float(0x7fc00000); }

// running statistics of a column (forward): maximum, sum of exp(x - max), number of +Inf entries, NaN seen
struct ColStat {
  float m, s;
  int n_inf;
  int nan;
};
__device__ __forceinline__ ColStat stat_init() { return ColStat{f_ninf(), 0.f, 0, 0}; }
__device__ __forceinline__ void stat_add(ColStat& c, float x) {
  if (x != x) { c.nan = 1; return; }
  if (x == f_inf()) { c.n_inf += 1; c.m = f_inf(); return; }
  if (x > c.m) {
    c.s = c.s * ((c.m == f_ninf()) ? 0.f : __expf(c.m - x)) + 1.f;
    c.m = x;
  } else if (x != f_ninf()) {
    c.s += __expf(x - c.m);
  }
}
__device__ __forceinline__ ColStat stat_merge(const ColStat& a, const ColStat& b) {
  ColStat c;
  c.nan = a.nan | b.nan;
  c.n_inf = a.n_inf + b.n_inf;
  c.m = fmaxf(a.m, b.m);
  if (c.m == f_ninf() || c.m == f_inf()) {
    c.s = 0.f;
  } else {
    c.s = ((a.m == f_ninf()) ? 0.f : a.s * __expf(a.m - c.m)) + ((b.m == f_ninf()) ? 0.f : b.s * __expf(b.m - c.m));
  }
  return c;
}
__device__ __forceinline__ ColStat stat_shfl_xor(const ColStat& a, int off) {
  ColStat b;
  b.m = __shfl_xor_sync(0xffffffffu, a.m, off);
  b.s = __shfl_xor_sync(0xffffffffu, a.s, off);
  b.n_inf = __shfl_xor_sync(0xffffffffu, a.n_inf, off);
  b.nan = __shfl_xor_sync(0xffffffffu, a.nan, off);
  return b;
}
// value of one output element given the finished statistics of its column
template <int MODE>
__device__ __forceinline__ float fwd_value(const ColStat& c, float x, float log_s) {
  if (c.nan || c.m == f_ninf()) return f_nan();
  if (c.m == f_inf()) {
    if (MODE == SM_FWD) return (x == f_inf()) ? 1.f / (float)c.n_inf : 0.f;
    return (x == f_inf()) ? -log_s : f_ninf();       // log_s = log(number of +Inf entries)
  }
  if (MODE == SM_FWD) return __expf(x - c.m) / c.s;
  return x - c.m - log_s;
}

// 16-byte packets: V = 16 / sizeof(T) consecutive elements of a column
template <typename T> struct Pack { static constexpr int V = 16 / sizeof(T); };
template <typename T>
__device__ __forceinline__ void unpack(const uint4& q, float (&f)[Pack<T>::V]) {
  const T* e = reinterpret_cast<const T*>(&q);
#pragma unroll
  for (int u = 0; u < Pack<T>::V; ++u) f[u] = Elem<T>::to_f(e[u]);
}
template <typename T>
__device__ __forceinline__ uint4 repack(const float (&f)[Pack<T>::V]) {
  uint4 q;
  T* e = reinterpret_cast<T*>(&q);
#pragma unroll
  for (int u = 0; u < Pack<T>::V; ++u) e[u] = Elem<T>::from_f(f[u]);
  return q;
}
// 16-bit types: two values per conversion instruction
template <>
__device__ __forceinline__ uint4 repack<__nv_bfloat16>(const float (&f)[8]) {
  uint4 q;
  __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int u = 0; u < 4; ++u) e[u] = __floats2bfloat162_rn(f[2 * u], f[2 * u + 1]);
  return q;
}
template <>
__device__ __forceinline__ uint4 repack<__half>(const float (&f)[8]) {
  uint4 q;
  __half2* e = reinterpret_cast<__half2*>(&q);
#pragma unroll
  for (int u = 0; u < 4; ++u) e[u] = __floats2half2_rn(f[2 * u], f[2 * u + 1]);
  return q;
}
// Every kernel exists twice.  NA (no alias: the host saw that the output overlaps neither input) takes
// `__restrict__` pointers and loads through the non-coherent path, which lets the compiler start the next
// column's loads before this column's stores.  The other variant serves the in-place forms (softmax!(x, x) of the
// reference, a pullback written over dy): plain coherent loads, no promise about aliasing — a column longer than a
// thread's register share is read a second time after other threads may have written theirs.
template <typename T, bool NA> struct Ptrs { using In = const T*; using Out = T*; };
template <typename T> struct Ptrs<T, true> { using In = const T* __restrict__; using Out = T* __restrict__; };
template <typename T, bool NA>
__device__ __forceinline__ uint4 load_raw(const T* p) {
  if constexpr (NA) return __ldg(reinterpret_cast<const uint4*>(p));
  else return *reinterpret_cast<const uint4*>(p);
}
template <typename T, bool NA>
__device__ __forceinline__ T load_elem(const T* p) {
  if constexpr (NA) return __ldg(p);
  else return *p;
}
template <typename T, bool NA>
__device__ __forceinline__ void load_pack(const T* p, float (&f)[Pack<T>::V]) { unpack<T>(load_raw<T, NA>(p), f); }
template <typename T>
__device__ __forceinline__ void store_pack(T* p, const float (&f)[Pack<T>::V]) {
  *reinterpret_cast<uint4*>(p) = repack<T>(f);
}

// branch-free update of the running statistics with one packet of V values: one rescaling exponential
// per packet instead of a data-dependent branch per value
template <int V>
__device__ __forceinline__ void stat_add_pack(ColStat& c, const float (&f)[V]) {
  float pm = f_ninf();
  float xv[V];
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const float x = f[u];
    c.nan |= (x != x) ? 1 : 0;
    const bool is_inf = (x == f_inf());
    c.n_inf += is_inf ? 1 : 0;
    xv[u] = (is_inf || x != x) ? f_ninf() : x;      // +Inf and NaN are accounted for by the flags
    pm = fmaxf(pm, xv[u]);
  }
  const float m_new = fmaxf(c.m, pm);
  const float m_safe = (m_new == f_ninf()) ? 0.f : m_new;
  float s = c.s * __expf(c.m - m_safe);              // c.m = -Inf: exp(-Inf) = 0
#pragma unroll
  for (int u = 0; u < V; ++u) s += __expf(xv[u] - m_safe);
  c.s = s;
  c.m = m_new;
}
// first sweep over a register-cached column: a NaN-propagating maximum is all the common case needs
// (one instruction per value); +Inf entries are counted only when the maximum turns out to be +Inf
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// (the maximum above ignores +Inf entries; a column that has some is marked here)
__device__ __forceinline__ void stat_finish(ColStat& c) {
  if (c.n_inf > 0) c.m = f_inf();
}
// output values of a packet given the finished statistics
template <int MODE, int V>
__device__ __forceinline__ void fwd_pack(const ColStat& c, float inv_s, float log_s, float (&f)[V]) {
  const bool special = c.nan || c.m == f_ninf() || c.m == f_inf();
#pragma unroll
  for (int u = 0; u < V; ++u) {
    if (special) f[u] = fwd_value<MODE>(c, f[u], log_s);
    else f[u] = (MODE == SM_FWD) ? __expf(f[u] - c.m) * inv_s : f[u] - c.m - log_s;
  }
}

// ---- reduction dimension contiguous (inner == 1): G threads per column ----------------------------
// VECT: columns are whole 16-byte packets (n a multiple of the packet, arrays 16-byte aligned).
// KP > 0 (with VECT): a thread's packets (at most KP, as raw 16-byte words) stay in registers between
// the two passes, so the column is read from memory once.
template <typename T, int MODE, int G, bool VECT, int KP, bool NA>
__global__ void __launch_bounds__((G > 256 ? G : 256)) softmax_cols_kernel(typename Ptrs<T, NA>::In x, typename Ptrs<T, NA>::In dy,
                                                                            typename Ptrs<T, NA>::Out out, long long n, long long cols) {
  constexpr int kBlock = G > 256 ? G : 256;
  constexpr int kPerBlock = kBlock / G;
  constexpr int kWarps = kBlock / 32;
  constexpr int V = Pack<T>::V;
  constexpr bool FWD = (MODE == SM_FWD || MODE == LSM_FWD);
  const long long np = n / V;   // packets per column (VECT)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = threadIdx.x / G, t = threadIdx.x % G;
  __shared__ ColStat sh_stat[32];
  __shared__ float sh_sum[32];
  for (long long col = (long long)blockIdx.x * kPerBlock + g; col < cols || G >= 256; col += (long long)gridDim.x * kPerBlock) {
    if (G >= 256 && col >= cols) break;
    const T* xc = x + col * n;
    const T* dc = FWD ? xc : dy + col * n;
    T* oc = out + col * n;
    constexpr bool CACHE = KP > 0;
    uint4 cx[CACHE ? KP : 1];                 // forward: x; pullbacks: y
    uint4 cd[(CACHE && !FWD) ? KP : 1];       // pullbacks: dy
    ColStat c = stat_init();
    float acc = 0.f;
    // ---- pass 1: column statistics (forward) or the column sum (pullbacks)
    if (VECT && CACHE) {
#pragma unroll
      for (int k = 0; k < (CACHE ? KP : 1); ++k) {
        const long long jp = t + (long long)k * G;
        if (jp < np) {
          cx[k] = load_raw<T, NA>(xc + jp * V);
          if (!FWD) cd[k] = load_raw<T, NA>(dc + jp * V);
        }
      }
#pragma unroll
      for (int k = 0; k < (CACHE ? KP : 1); ++k) {
        const long long jp = t + (long long)k * G;
        if (jp < np) {
          float f[V];
          unpack<T>(cx[k], f);
          if (FWD) {
#pragma unroll
            for (int u = 0; u < V; ++u) c.m = max_nan(c.m, f[u]);   // the exponentials follow once the maximum is known
          } else {
            float d[V];
            unpack<T>(cd[k], d);
#pragma unroll
            for (int u = 0; u < V; ++u) acc += (MODE == SM_BWD) ? d[u] * f[u] : d[u];
          }
        }
      }
    } else if (VECT) {
      for (long long jp = t; jp < np; jp += G) {
        float f[V], d[V];
        load_pack<T, NA>(xc + jp * V, f);
        if (FWD) {
          stat_add_pack<V>(c, f);
        } else {
          load_pack<T, NA>(dc + jp * V, d);
#pragma unroll
          for (int u = 0; u < V; ++u) acc += (MODE == SM_BWD) ? d[u] * f[u] : d[u];
        }
      }
    } else {
      for (long long j = t; j < n; j += G) {
        if (FWD) {
          stat_add(c, Elem<T>::to_f(xc[j]));
        } else {
          const float d = Elem<T>::to_f(dc[j]);
          acc += (MODE == SM_BWD) ? d * Elem<T>::to_f(xc[j]) : d;
        }
      }
    }
    // ---- reduce over the G threads of the column
    auto group_sum = [&](float v) -> float {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if (G >= 256) {
        if (lane == 0) sh_sum[warp] = v;
        __syncthreads();
        v = 0.f;
        for (int w = 0; w < kWarps; ++w) v += sh_sum[w];
        __syncthreads();
      }
      return v;
    };
    if (FWD && VECT && CACHE) {
      // register-cached column: only the (NaN-propagating) maximum exists so far
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) c.m = max_nan(c.m, __shfl_xor_sync(0xffffffffu, c.m, off));
      if (G >= 256) {
        if (lane == 0) sh_sum[warp] = c.m;
        __syncthreads();
        c.m = sh_sum[0];
        for (int w = 1; w < kWarps; ++w) c.m = max_nan(c.m, sh_sum[w]);
        __syncthreads();
      }
      if (c.m != c.m) {            // a NaN somewhere in the column
        c.nan = 1;
        c.m = 0.f;
      } else if (c.m == f_inf()) { // rare: count the +Inf entries (src/softmax.jl:71-76 shares the weight among them)
        float cnt = 0.f;
#pragma unroll
        for (int k = 0; k < (CACHE ? KP : 1); ++k) {
          const long long jp = t + (long long)k * G;
          if (jp < np) {
            float f[V];
            unpack<T>(cx[k], f);
#pragma unroll
            for (int u = 0; u < V; ++u) cnt += (f[u] == f_inf()) ? 1.f : 0.f;
          }
        }
        c.n_inf = (int)group_sum(cnt);
      }
    } else if (FWD) {
      stat_finish(c);
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) c = stat_merge(c, stat_shfl_xor(c, off));
      if (G >= 256) {
        if (lane == 0) sh_stat[warp] = c;
        __syncthreads();
        c = sh_stat[0];
        for (int w = 1; w < kWarps; ++w) c = stat_merge(c, sh_stat[w]);
        __syncthreads();
      }
    }
    if (FWD) {
      if (VECT && CACHE) {
        // second sweep over the registers: one exponential per element, summed in fp32; softmax keeps the
        // exponentials (in the element type) in place of x for the write sweep
        const bool special = c.nan || c.m == f_ninf() || c.m == f_inf();
        float part = 0.f;
        if (!special) {
#pragma unroll
          for (int k = 0; k < (CACHE ? KP : 1); ++k) {
            const long long jp = t + (long long)k * G;
            if (jp < np) {
              float f[V];
              unpack<T>(cx[k], f);
#pragma unroll
              for (int u = 0; u < V; ++u) {
                f[u] = __expf(f[u] - c.m);
                part += f[u];
              }
              if (MODE == SM_FWD) cx[k] = repack<T>(f);
            }
          }
        }
        c.s = group_sum(part);
      }
    } else {
      acc = group_sum(acc);
    }
    const float sum_or_cnt = (c.m == f_inf()) ? (float)c.n_inf : c.s;
    const float log_s = (MODE == LSM_FWD) ? __logf(sum_or_cnt) : 0.f;
    const float inv_s = (MODE == SM_FWD) ? 1.f / c.s : 0.f;
    // ---- pass 2: write
    if (VECT && CACHE) {
#pragma unroll
      for (int k = 0; k < (CACHE ? KP : 1); ++k) {
        const long long jp = t + (long long)k * G;
        if (jp < np) {
          float f[V];
          unpack<T>(cx[k], f);
          if (FWD) {
            const bool special = c.nan || c.m == f_ninf() || c.m == f_inf();
            if (MODE == SM_FWD && !special) {
#pragma unroll
              for (int u = 0; u < V; ++u) f[u] *= inv_s;      // f holds exp(x - max) from the second sweep
            } else {
              // (logsoftmax: with the common case told apart here, too, 1024 threads a block need 46 registers instead of 32
              // and leave room for one on an SM: 18160 Float16 x 581 12.5 us, and 16.2)
              fwd_pack<MODE, V>(c, inv_s, log_s, f);
            }
            store_pack<T>(oc + jp * V, f);
          } else {
            float d[V];
            unpack<T>(cd[k], d);
#pragma unroll
            for (int u = 0; u < V; ++u) d[u] = (MODE == SM_BWD) ? f[u] * (d[u] - acc) : d[u] - __expf(f[u]) * acc;
            store_pack<T>(oc + jp * V, d);
          }
        }
      }
    } else if (VECT) {
      for (long long jp = t; jp < np; jp += G) {
        float f[V], d[V];
        load_pack<T, NA>(xc + jp * V, f);
        if (FWD) {
          fwd_pack<MODE, V>(c, inv_s, log_s, f);
          store_pack<T>(oc + jp * V, f);
        } else {
          load_pack<T, NA>(dc + jp * V, d);
#pragma unroll
          for (int u = 0; u < V; ++u) d[u] = (MODE == SM_BWD) ? f[u] * (d[u] - acc) : d[u] - __expf(f[u]) * acc;
          store_pack<T>(oc + jp * V, d);
        }
      }
    } else {
      for (long long j = t; j < n; j += G) {
        if (FWD) {
          oc[j] = Elem<T>::from_f(fwd_value<MODE>(c, Elem<T>::to_f(xc[j]), log_s));
        } else {
          const float d = Elem<T>::to_f(dc[j]), y = Elem<T>::to_f(xc[j]);
          oc[j] = Elem<T>::from_f((MODE == SM_BWD) ? y * (d - acc) : d - __expf(y) * acc);
        }
      }
    }
  }
}

// ---- reduction dimension strided (inner > 1): TI columns by NT / TI rows of the reduction ----------------------
// A block owns TI consecutive columns; each of its NT / TI rows of threads takes every (NT / TI)-th element of them,
// eight loads in flight per thread, and the partial statistics are merged through shared memory; with one row (TI = NT)
// a column is a thread's own, without a barrier.  FLAT: the columns (i, o) are numbered through, so that narrow slices
// leave no lane idle; else a block keeps to one slice o, whose columns then start on a sector.  The second pass over a
// column re-reads it from L2; a thread writes only what it has read itself, so the in-place forms are safe.
template <typename T, int MODE, int TI, int NT, bool FLAT, bool NA>
__global__ void __launch_bounds__(NT) softmax_strided_kernel(typename Ptrs<T, NA>::In x, typename Ptrs<T, NA>::In dy,
                                                             typename Ptrs<T, NA>::Out out, long long inner, long long n,
                                                             long long outer) {
  constexpr int TJ = NT / TI;
  constexpr bool FWD = (MODE == SM_FWD || MODE == LSM_FWD);
  __shared__ ColStat sh_stat[FWD && TJ > 1 ? TJ : 1][TI];
  __shared__ float sh_sum[!FWD && TJ > 1 ? TJ : 1][TI];
  const int ti = threadIdx.x % TI, tj = threadIdx.x / TI;
  const long long itiles = (inner + TI - 1) / TI, tiles = FLAT ? (inner * outer + TI - 1) / TI : itiles * outer;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    long long i, o;
    if (FLAT) {
      const long long p = tile * TI + ti;
      o = (p | inner) >> 32 ? p / inner : (long long)((unsigned)p / (unsigned)inner);
      i = p - o * inner;
    } else {
      o = tile / itiles;
      i = (tile - o * itiles) * TI + ti;
    }
    const long long base = i + inner * n * o;
    const long long nj = (FLAT ? o < outer : i < inner) ? n : 0;        // columns beyond the edge have nothing to do
    // f(number of elements, the first one's j) over the thread's elements: eight at a time, what is left of a column
    // that is a thread's own in fours and twos
    auto over = [&](auto f) {
      long long j = tj;
      for (; j + 7 * TJ < nj; j += 8 * TJ) f(std::integral_constant<int, 8>(), j);
      if constexpr (TJ == 1) {
        if (j + 3 < nj) {
          f(std::integral_constant<int, 4>(), j);
          j += 4;
        }
        if (j + 1 < nj) {
          f(std::integral_constant<int, 2>(), j);
          j += 2;
        }
      }
      for (; j < nj; j += TJ) f(std::integral_constant<int, 1>(), j);
    };
    if constexpr (FWD) {
      ColStat c = stat_init();
      over([&](auto cnt, long long j) {
        constexpr int U = decltype(cnt)::value;
        float f[U];
#pragma unroll
        for (int u = 0; u < U; ++u) f[u] = Elem<T>::to_f(load_elem<T, NA>(x + base + (j + u * TJ) * inner));
        stat_add_pack<U>(c, f);
      });
      if (TJ > 1) {
        sh_stat[tj][ti] = c;
        __syncthreads();
#pragma unroll
        for (int s = TJ / 2; s > 0; s >>= 1) {
          if (tj < s) sh_stat[tj][ti] = stat_merge(sh_stat[tj][ti], sh_stat[tj + s][ti]);
          __syncthreads();
        }
        c = sh_stat[0][ti];
      }
      stat_finish(c);
      const float inv_s = 1.f / c.s;
      const float log_s = (MODE == LSM_FWD) ? __logf(c.m == f_inf() ? (float)c.n_inf : c.s) : 0.f;
      over([&](auto cnt, long long j) {
        constexpr int U = decltype(cnt)::value;
        float f[U];
#pragma unroll
        for (int u = 0; u < U; ++u) f[u] = Elem<T>::to_f(load_elem<T, NA>(x + base + (j + u * TJ) * inner));
        if constexpr (TJ == 1) {   // (short sums: the division's one rounding counts)
#pragma unroll
          for (int u = 0; u < U; ++u) f[u] = fwd_value<MODE>(c, f[u], log_s);
        } else {
          fwd_pack<MODE, U>(c, inv_s, log_s, f);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) out[base + (j + u * TJ) * inner] = Elem<T>::from_f(f[u]);
      });
    } else {
      // sum of dy * y (softmax) or of dy (logsoftmax), then y * (dy - sum) or dy - exp(y) * sum
      float acc = 0.f;
      over([&](auto cnt, long long j) {
        constexpr int U = decltype(cnt)::value;
        float d[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          d[u] = Elem<T>::to_f(load_elem<T, NA>(dy + base + (j + u * TJ) * inner));
          y[u] = (MODE == SM_BWD) ? Elem<T>::to_f(load_elem<T, NA>(x + base + (j + u * TJ) * inner)) : 1.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) acc = (MODE == SM_BWD) ? fmaf(d[u], y[u], acc) : acc + d[u];
      });
      if (TJ > 1) {
        sh_sum[tj][ti] = acc;
        __syncthreads();
#pragma unroll
        for (int s = TJ / 2; s > 0; s >>= 1) {
          if (tj < s) sh_sum[tj][ti] += sh_sum[tj + s][ti];
          __syncthreads();
        }
        acc = sh_sum[0][ti];
      }
      over([&](auto cnt, long long j) {
        constexpr int U = decltype(cnt)::value;
        float d[U], y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          d[u] = Elem<T>::to_f(load_elem<T, NA>(dy + base + (j + u * TJ) * inner));
          y[u] = Elem<T>::to_f(load_elem<T, NA>(x + base + (j + u * TJ) * inner));
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
          out[base + (j + u * TJ) * inner] =
              Elem<T>::from_f((MODE == SM_BWD) ? y[u] * (d[u] - acc) : d[u] - __expf(y[u]) * acc);
      });
    }
    if (TJ > 1) __syncthreads();                   // the shared statistics are used again
  }
}

// ---- forward over long contiguous columns: the next column on its way while one is worked on -------------------
// A column that takes a whole block's registers leaves room for one block on an SM, and a block that loads, reduces
// twice and stores keeps the memory system idle for most of that time: 32000 BFloat16 x 4096, logsoftmax, 121 us =
// 4.3 TB/s with a column after the other loaded into the registers of 1024 threads.  Here the next S columns of a block
// arrive in shared memory (cp.async; a thread reads back only the packets that it copied itself, so its own wait is all
// that is needed, and refills their place at once), and blocks of G threads, 1024 / G on an SM, are in different phases:
// 107 us = 4.9 TB/s there (one block of 1024 threads, two columns arriving: 127), softmax 163 -> 110; 50000 BFloat16 x
// 2000 195 -> 112, softmax 211 -> 126 (113 with the exponentials kept as 16-bit values, see ONCE), 10000 Float32 x 4096 116 -> 64.
// The statistics are softmax_cols_kernel's with their sums in another order, so a column's last bit may depend on whether
// there are enough of them for this kernel.  ONCE: the 16-bit x stays in the registers and its exponentials are taken
// again for the result, which is rounded once; without it they are kept there as 16-bit values, as in the other kernel
// for columns of the same length (up to 4096 packets).
constexpr int kRingSmem = 226 * 1024;
template <typename T, int MODE, int G, int KP, int S, bool ONCE>
__global__ void __launch_bounds__(G, 1024 / G) softmax_ring_kernel(const T* __restrict__ x, T* __restrict__ out, long long n,
                                                                   long long cols) {
  constexpr int V = Pack<T>::V;
  constexpr int kWarps = G / 32;
  extern __shared__ __align__(16) uint4 ring[];
  const int np = (int)(n / V);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t = threadIdx.x;
  __shared__ float sh[2][kWarps];
  auto fetch = [&](long long col, int st) {
    if (col < cols) {
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        const int jp = t + k * G;
        if (jp < np) {
          const unsigned int d = (unsigned int)__cvta_generic_to_shared(ring + st * np + jp);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(x + col * n + (long long)jp * V) : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // over the block; `buf` alternates, so that one barrier a reduction is enough
  auto block_reduce = [&](float v, int buf, auto op) -> float {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, off));
    if (lane == 0) sh[buf][warp] = v;
    __syncthreads();
    v = sh[buf][lane % kWarps];
#pragma unroll
    for (int off = kWarps / 2; off > 0; off >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
  };
  auto add = [](float a, float b) { return a + b; };
#pragma unroll
  for (int st = 0; st < S; ++st) fetch(blockIdx.x + (long long)st * gridDim.x, st);
  int st = 0;
  for (long long col = blockIdx.x; col < cols; col += gridDim.x, st = st + 1 == S ? 0 : st + 1) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 1) : "memory");
    uint4 cx[KP];
    ColStat c = stat_init();
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int jp = t + k * G;
      if (jp < np) {
        cx[k] = ring[st * np + jp];
        float f[V];
        unpack<T>(cx[k], f);
#pragma unroll
        for (int u = 0; u < V; ++u) c.m = max_nan(c.m, f[u]);
      }
    }
    fetch(col + (long long)S * gridDim.x, st);
    c.m = block_reduce(c.m, 0, [](float a, float b) { return max_nan(a, b); });
    if (c.m != c.m) {            // a NaN somewhere in the column
      c.nan = 1;
      c.m = 0.f;
    }
    // the sum of the exponentials; of a column whose maximum is +Inf the number of its +Inf entries, which share
    // the weight (src/softmax.jl:71-76)
    const bool special = c.nan || c.m == f_ninf() || c.m == f_inf();
    float part = 0.f;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int jp = t + k * G;
      if (jp < np) {
        float f[V];
        unpack<T>(cx[k], f);
        if (!special) {
#pragma unroll
          for (int u = 0; u < V; ++u) {
            f[u] = __expf(f[u] - c.m);
            part += f[u];
          }
          if (MODE == SM_FWD && !ONCE) cx[k] = repack<T>(f);
        } else {
#pragma unroll
          for (int u = 0; u < V; ++u) part += (f[u] == f_inf()) ? 1.f : 0.f;
        }
      }
    }
    c.s = block_reduce(part, 1, add);
    c.n_inf = special ? (int)c.s : 0;
    const float log_s = (MODE == LSM_FWD) ? __logf(c.s) : 0.f;
    const float inv_s = (MODE == SM_FWD) ? 1.f / c.s : 0.f;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int jp = t + k * G;
      if (jp < np) {
        float f[V];
        unpack<T>(cx[k], f);
        if (special) {
          fwd_pack<MODE, V>(c, inv_s, log_s, f);
        } else {
#pragma unroll
          for (int u = 0; u < V; ++u) f[u] = MODE == SM_FWD ? (ONCE ? __expf(f[u] - c.m) : f[u]) * inv_s : f[u] - c.m - log_s;
        }
        store_pack<T>(out + col * n + (long long)jp * V, f);
      }
    }
  }
}

template <typename T, int MODE, int G, int KP, int S, bool ONCE>
cudaError_t launch_ring(const T* x, T* out, long long n, long long cols, cudaStream_t st) {
  auto kern = softmax_ring_kernel<T, MODE, G, KP, S, ONCE>;
  constexpr int per_sm = 1024 / G;
  const int smem = (int)(n * sizeof(T)) * S;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kRingSmem / per_sm);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)(cols < 148 * per_sm ? cols : 148 * per_sm), G, smem, st>>>(x, out, n, cols);
  count_launch();
  return cudaGetLastError();
}

template <typename T, int MODE>
cudaError_t launch_softmax(const void* x, const void* dy, void* out, long long inner, long long n, long long outer,
                           cudaStream_t st) {
  const T* xp = static_cast<const T*>(x);
  const T* dp = static_cast<const T*>(dy);
  T* op = static_cast<T*>(out);
  // does the output overlap an input?  (the in-place forms of the reference: the same array, same extent)
  const uintptr_t bytes = (uintptr_t)(inner * n * outer) * sizeof(T);
  auto overlaps = [bytes](const void* a, const void* b) {
    const uintptr_t pa = reinterpret_cast<uintptr_t>(a), pb = reinterpret_cast<uintptr_t>(b);
    return a != nullptr && b != nullptr && pa < pb + bytes && pb < pa + bytes;
  };
  const bool no_alias = !overlaps(x, out) && !overlaps(dy, out);
  if (inner == 1) {
    auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const bool vect = (n % Pack<T>::V) == 0 && al16(x) && al16(out) && (dy == nullptr || al16(dy));
    const long long np = n / Pack<T>::V;
    const long long cap = 148ll * 16;
    // a warp per short column, a 256- or 1024-thread block per long one; the column stays in registers
    // between the passes whenever a thread's share is small enough (1024-thread blocks have 64 registers
    // per thread: 8 raw packets for Float32 forward, 4 otherwise, 4 + 4 in the pullbacks)
    constexpr bool FWD = (MODE == SM_FWD || MODE == LSM_FWD);
    constexpr int kBig = (FWD && sizeof(T) == 4) ? 8 : 4;
    // long columns, enough of them for every block to have a next one (20000 Float16 x 300: 15 us in the other kernel, 19
    // here; x 700: 24 and 22).  Columns that 256 threads hold (2048 packets) leave enough blocks on an SM as it is: 16384
    // BFloat16 x 4096 52 us, and 60 with the next column arriving.  In-place calls keep the other kernel, too.
    if constexpr (FWD) {
      if (vect && no_alias && outer >= 4 * 148) {
        if (np > 256ll * 8 && np <= 512ll * 8) return launch_ring<T, MODE, 512, 8, 1, false>(xp, op, n, outer, st);
        if (np > 512ll * 8 && np <= 1024ll * 7)
          return launch_ring<T, MODE, 1024, 7, 2, MODE == SM_FWD && sizeof(T) == 2>(xp, op, n, outer, st);
      }
    }
#define NB_SM_LAUNCH(GG, VV, KK)                                                                       \
  do {                                                                                                 \
    constexpr int kBlock = (GG) > 256 ? (GG) : 256;                                                    \
    const long long need = (outer + (kBlock / (GG)) - 1) / (kBlock / (GG));                            \
    const long long blocks = need < cap ? need : cap;                                                  \
    if (no_alias)                                                                                      \
      softmax_cols_kernel<T, MODE, GG, VV, KK, true><<<(unsigned)blocks, kBlock, 0, st>>>(xp, dp, op, n, outer);  \
    else                                                                                               \
      softmax_cols_kernel<T, MODE, GG, VV, KK, false><<<(unsigned)blocks, kBlock, 0, st>>>(xp, dp, op, n, outer); \
  } while (0)
    if (!vect) {
      if (n > 2048) NB_SM_LAUNCH(256, false, 0); else NB_SM_LAUNCH(32, false, 0);
    } else if (np <= 32ll * 2) {
      // short columns (attention-sized rows of scores): two packets per lane, few registers, so that enough
      // warps are resident to keep the memory system busy with so little in flight per warp
      NB_SM_LAUNCH(32, true, 2);
    } else if (np <= 32ll * 4) {
      NB_SM_LAUNCH(32, true, 4);
    } else if (np <= 32ll * 8) {
      NB_SM_LAUNCH(32, true, 8);
    } else if (sizeof(T) == 2 && FWD && np <= 32ll * 16) {
      // 16-bit columns of up to 4096 elements still fit a warp's registers (16 packets per lane): no block-wide
      // barrier between the passes, sixteen independent loads in flight per lane
      NB_SM_LAUNCH(32, true, 16);
    } else if (np <= 256ll * 8) {
      NB_SM_LAUNCH(256, true, 8);
    } else if (np <= 1024ll * kBig) {
      NB_SM_LAUNCH(1024, true, kBig);
    } else {
      NB_SM_LAUNCH(1024, true, 0);
    }
#undef NB_SM_LAUNCH
  } else {
    constexpr int kW = 32 / (int)sizeof(T);
    const long long cols = inner * outer;
    auto tiles_of = [&](long long ti, bool flat) { return flat ? (cols + ti - 1) / ti : (inner + ti - 1) / ti * outer; };
#define NB_SM_STRIDED(TI, NT, FLAT)                                                                                \
  do {                                                                                                             \
    const long long tiles = tiles_of(TI, FLAT), cap = 148ll * 32 * ((NT) < 256 ? 256 / (NT) : 1);                  \
    const unsigned blocks = (unsigned)(tiles < cap ? tiles : cap);                                                 \
    if (no_alias) softmax_strided_kernel<T, MODE, TI, NT, FLAT, true><<<blocks, NT, 0, st>>>(xp, dp, op, inner, n, outer);   \
    else softmax_strided_kernel<T, MODE, TI, NT, FLAT, false><<<blocks, NT, 0, st>>>(xp, dp, op, inner, n, outer); \
  } while (0)
    // The shorter the reduction and the more the columns, the fewer threads share one: a column is a thread's own up to 8
    // elements, or up to 24 / 48 once the columns alone fill the GPU (30000 / 100000), else four or eight share it, or
    // the 32 / 16 that are left beside the columns of one 32-byte sector (narrower blocks would fetch sectors twice).
    // Float32, forward, against one thread a column walking it one load at a time and against eight rows of 32 columns of
    // a slice for everything: (2, 4, 1M) 26 and 2633 -> 26 us, (8, 10, 2.5M) 598 and 8662 -> 494, (16, 64, 50000) 199 and
    // 285 -> 110, (46, 192, 260) 98 and 13 -> 8, (428, 8704, 1) 4163 and 25 -> 25; over 2816 shapes within 10 % of the
    // better of the two but for 25, and 20 % below it on average.
    if (n <= 8 || (n <= 24 && cols >= 30000) || (n <= 48 && cols >= 100000)) NB_SM_STRIDED(128, 128, true);
    else if (n < 24) NB_SM_STRIDED(32, 128, true);
    else if (n >= 1024 && cols < 148ll * kW) NB_SM_STRIDED(kW, 1024, false);
    else if (n >= 512 ? (inner < 32 || cols < 25000) : (cols < 5000 || (inner < 8 && n >= 48 && n * 400 >= cols)))
      NB_SM_STRIDED(kW, 256, true);
    else if (n >= 200 || (n >= 48 && cols < 25000)) NB_SM_STRIDED(32, 256, true);
    else NB_SM_STRIDED(32, 128, true);
#undef NB_SM_STRIDED
  }
  count_launch();
  return cudaGetLastError();
}

template <int MODE>
cudaError_t dispatch_softmax(int dtype, const void* x, const void* dy, void* out, long long inner, long long n,
                             long long outer, cudaStream_t st) {
  switch (dtype) {
    case NNLIB_B200_F16:  return launch_softmax<__half, MODE>(x, dy, out, inner, n, outer, st);
    case NNLIB_B200_BF16: return launch_softmax<__nv_bfloat16, MODE>(x, dy, out, inner, n, outer, st);
    default:              return launch_softmax<float, MODE>(x, dy, out, inner, n, outer, st);
  }
}

}  // namespace

cudaError_t softmax_forward(int dtype, bool log, const void* x, void* y, long long inner, long long n, long long outer,
                            cudaStream_t st) {
  return log ? dispatch_softmax<LSM_FWD>(dtype, x, nullptr, y, inner, n, outer, st)
             : dispatch_softmax<SM_FWD>(dtype, x, nullptr, y, inner, n, outer, st);
}

cudaError_t softmax_backward(int dtype, bool log, const void* dy, const void* y, void* dx, long long inner, long long n,
                             long long outer, cudaStream_t st) {
  return log ? dispatch_softmax<LSM_BWD>(dtype, y, dy, dx, inner, n, outer, st)
             : dispatch_softmax<SM_BWD>(dtype, y, dy, dx, inner, n, outer, st);
}

}  // namespace nb200
