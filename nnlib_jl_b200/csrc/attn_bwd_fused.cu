// One-pass backward of attention on the sm_100a tensor cores: five products per 128 x 128 block of scores.
//
// With P = exp(scale q.k - lse), D_i = dx_i . x_i and dS = P (dP - D) (attn_bwd_umma.cu has the gradients and their
// sources in the reference), a CTA owns 128 keys, walks over the tiles of 128 queries and issues per tile
//   S^T  = K Q^T          dP^T = V dX^T          dQ   = dS K          dK  += dS^T Q        (operands in shared memory)
//   dV  += P^T dX                                                                         (P^T in tensor memory)
// The tile's share of dQ is added to a Float32 array in the caller's workspace by the copy engine; a small kernel before
// clears it and computes D, a small one behind scales and rounds it.  The two half backwards of attn_bwd_umma.cu, which
// need no workspace and add in a fixed order, compute S, dP and the exponentials twice: seven products.
//   warps 0-3, 4-7   compute: keys 32 (warp % 4) .. + 31, queries 0-63 / 64-127 of the tile.  They read tensor memory
//                    in the fragment layout (tmem_ld_frag): 16 queries per thread, so that the per-query lse and D
//                    cost 16 8-byte shared-memory reads a step and thread instead of 32 16-byte ones (1 KB a warp
//                    instead of 4, on the pipe that feeds the products)
//   warps 8-11       dQ: tensor memory -> registers -> shared memory -> additions to global memory; dropout's keep bits
//   warp 12          TMA: the first loads of all, then the ring of Q with the queries' lse and D;   warp 15: ring of dX
//   warp 13          issues S and dV;   warp 14: issues dP, dQ and dK
// Tensor memory columns, D = 128: S [0,128) | dP [128,256) | dV | dK; D = 64: S | dP | dV [256,320) | dK | dQ [384,448).
// P^T (16 bits) is written over S, each warp over lanes and columns that it alone reads, once all its lanes have read
// them.  With D = 128 there is no room left and dQ is written over dP, which makes a chain of a step: dP, the compute
// warps' dS, dQ, its way into registers, the next dP.  So dQ is issued before dK, and a warp that takes dQ out holds a
// whole row of it in registers.
//
// What bounds it, at config "bf16 causal, L = 4096, d = 128, 32 heads, 8 sequences" (cycles of a step, from clock reads
// in a copy of the kernel): 3970 a step of 2560 cycles of tensor work.  The chain above takes about all of it: dP 770,
// its way into registers 170, dS 990, hand-over 430, dQ 800, registers 240, hand-over 440.  Beside it the additions
// take 2860: 64 KB at the 22 bytes a cycle and SM at which L2 takes them (6.0 TB/s for 148 CTAs that do nothing else).
// Added from registers instead (red.v4.f32) they go at the same rate but keep the load / store queue, and the compute
// warps' tensor memory stores behind them in it, waiting: 5600 a step.  Polynomials in place of a quarter to half of
// the exponentials shorten that phase (1345 -> 1080) and nothing else.  One backward (pre and post included) went
// 4140 -> 2940 us there, 3560 -> 2670 for one sequence of 16384 and 16 heads, 473 -> 325 for 16 heads of d = 64,
// L = 2048, 8 sequences, 1604 -> 773 for the same not causal with dropout.  Of a CTA's 46 us there 2.3 pass before its
// first scores and 3.9 behind its last dS.
#include <cuda.h>

#include "common.cuh"
#include "extras.cuh"
#include "launchers.h"
#include "umma.cuh"
#include "umma_shared.cuh"

namespace nb200 {

__device__ int g_bwd_fused_abort = 0;  // sticky: a bounded wait of the kernel ran out

namespace {

constexpr int kFuThreads = 512;
constexpr int kColBytes = 1024;        // per tile of queries: -lse (base 2) of 128 queries, then -D

template <int D, bool DROP>
struct FuCfg {
  // features of a piece of dQ on its way out (with dropout at D = 128 half as many, for the room of the keep bits)
  static constexpr int kPieceFeat = DROP && D == 128 ? 16 : 32, kPieceBytes = 32 * kPieceFeat * 4;
  static constexpr int kTile = (D / 64) * kChunkBytes;     // 128 rows x D halves
  static constexpr int kFixOff = 0;                        // K, V
  static constexpr int kQOff = 2 * kTile;
  static constexpr int kXStages = D == 128 ? 1 : 2;        // with D = 128 there is no room for more
  static constexpr int kXOff = kQOff + 2 * kTile;          // dX
  static constexpr int kDsOff = kXOff + kXStages * kTile;  // dS^T: 128 keys x 128 queries, halves
  static constexpr int kOutOff = kDsOff + 2 * kChunkBytes; // dQ on its way out: per warp two pieces of 32 queries
  static constexpr int kKeepOff = kOutOff + 8 * kPieceBytes;   // keep bits of two steps: [step & 1][32 keys][query]
  static constexpr int kColOff = kKeepOff + (DROP ? 4096 : 0);
  static constexpr int kBarOff = kColOff + 2 * kColBytes;
  static constexpr int kSmemBytes = kBarOff + 256;         // no slack: the kernel checks its 1 KB alignment
  static constexpr uint32_t kColS = 0, kColDP = 128, kColDV = 256, kColDK = 256 + D, kColDQ = D == 128 ? 128 : 384;
};
static_assert(FuCfg<128, false>::kSmemBytes <= 232448 && FuCfg<128, true>::kSmemBytes <= 232448, "shared memory budget");

struct FuBarriers {
  uint64_t k_full, v_full, q_full[2], q_empty[2], x_full[2], x_empty[2];
  uint64_t keep_full[2], keep_free[2], s_full, p_ready, dp_full, dp_read, ds_ready, dq_full, dq_read, acc_full;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(FuBarriers) <= 256, "barrier block");

// floats of workspace per tile of 128 queries of a unit: the column values of all tiles come first, then dQ
__host__ __device__ constexpr long long fused_tile_floats(int dpad) { return kColBytes / 4 + 128ll * dpad; }

// all ones where the sign of byte k of w is set, and the same of two words in the halves of a word
__device__ __forceinline__ unsigned int byte_sign(unsigned int w, int k) {
  unsigned int m;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(m) : "r"(w), "r"(0x8888u + 0x1111u * k));
  return m;
}
__device__ __forceinline__ unsigned int byte_sign_pair(unsigned int w0, unsigned int w1, int k) {
  unsigned int m;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(m) : "r"(w0), "r"(w1), "r"(0xcc88u + 0x1111u * k));
  return m;
}

// FEAT: 1 = Bool mask array, 2 = dropout, 4 = bias (as in attn_bwd_umma.cu)
template <int D, bool BF16, int FEAT>
__global__ void __launch_bounds__(kFuThreads, 1)
attn_bwd_fused_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                      const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_dx,
                      const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv, const AttnArgs a, const BwdArgs g, const int n_tiles, const int tail_units) {
  constexpr bool MASKED = (FEAT & 1) != 0, DROP = (FEAT & 2) != 0, BIAS = (FEAT & 4) != 0;
  using C = FuCfg<D, DROP>;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {
    // the swizzled tiles need 1 KB alignment and the budget leaves no room to round up: refuse cleanly
    if (threadIdx.x == 0) {
      atomicExch(&g_bwd_fused_abort, 1);
      if (a.status) atomicExch(a.status, NNLIB_B200_CUDA_ERROR);
    }
    return;
  }
  FuBarriers* bars = reinterpret_cast<FuBarriers*>(smem + C::kBarOff);
  volatile int* abort_flag = &bars->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // block -> (unit, key tile): unit by unit, the longest causal walks first; the last `tail_units` units are dealt
  // out together so that the launch does not end on the long walks of the last unit
  int unit, tix;
  {
    const int n_units = gridDim.x / n_tiles;
    const int head = (n_units - tail_units) * n_tiles;
    if ((int)blockIdx.x < head) {
      unit = blockIdx.x / n_tiles;
      tix = blockIdx.x % n_tiles;
    } else {
      const int j = blockIdx.x - head;
      unit = (n_units - tail_units) + j % tail_units;
      tix = j / tail_units;
    }
  }
  const int h = unit % a.H, b = unit / a.H;
  const int t0 = tix * 128;             // first key

  // query tiles: the causal walk goes from the key tile's own to the last; otherwise the CTAs of a unit start at
  // different ones, so that they do not all add to the same tile of dQ at once
  const int n_q = (a.Lq + 127) / 128;
  if (a.causal && tix >= n_q) {         // keys behind the last query: no query sees them, dk = dv = 0
    const int pieces = a.d / 8, rows = min(128, a.Lkv - t0);
    for (int i = threadIdx.x; i < rows * pieces; i += kFuThreads) {
      const long long o = ((long long)(t0 + i / pieces) + (long long)a.Lkv * b) * ((long long)a.H * a.d) + (long long)h * a.d +
                          (i % pieces) * 8;
      *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(g.dk) + 2 * o) = make_uint4(0u, 0u, 0u, 0u);
      *reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(g.dv) + 2 * o) = make_uint4(0u, 0u, 0u, 0u);
    }
    return;
  }
  const int r0 = tix % n_q;             // (causal: tix itself)
  const int n = a.causal ? n_q - r0 : n_q;
  auto tile_of = [&](int it) { const int t = r0 + it; return t < n_q ? t : t - n_q; };
  const long long tiles_all = (long long)n_q * a.H * a.B;
  const float* cols_u = a.ws + (long long)unit * n_q * (kColBytes / 4);
  float* dq_u = a.ws + tiles_all * (kColBytes / 4) + (long long)unit * n_q * (128 * D);

  auto load_tile = [&](int off, const CUtensorMap* m, uint64_t* bar, int first) {
    for (int c = 0; c < D / 64; ++c) tma_load_4d(smem + off + c * kChunkBytes, m, bar, c * 64, h, first, b);
  };
  auto load_q = [&](int it) {
    const int s = it & 1;
    mbar_arrive_expect_tx(&bars->q_full[s], C::kTile + kColBytes);
    load_tile(C::kQOff + s * C::kTile, &tm_q, &bars->q_full[s], tile_of(it) * 128);
    bulk_load(smem + C::kColOff + s * kColBytes, cols_u + (long long)tile_of(it) * (kColBytes / 4), &bars->q_full[s], kColBytes);
  };
  auto load_x = [&](int it) {
    const int s = it % C::kXStages;
    mbar_arrive_expect_tx(&bars->x_full[s], C::kTile);
    load_tile(C::kXOff + s * C::kTile, &tm_dx, &bars->x_full[s], tile_of(it) * 128);
  };
  if (threadIdx.x == 12 * 32) {
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_q);
    mbar_init(&bars->k_full, 1);
    mbar_init(&bars->v_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bars->q_full[s], 1);
      mbar_init(&bars->q_empty[s], 1);
      mbar_init(&bars->x_full[s], 1);
      mbar_init(&bars->x_empty[s], 2);   // dV and dP
      mbar_init(&bars->keep_full[s], 4);
      mbar_init(&bars->keep_free[s], 8);
    }
    mbar_init(&bars->s_full, 1);
    mbar_init(&bars->p_ready, 8);
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->dp_read, 8);
    mbar_init(&bars->ds_ready, 8);
    mbar_init(&bars->dq_full, 1);
    mbar_init(&bars->dq_read, 4);
    mbar_init(&bars->acc_full, 2);
    fence_mbar_init();
    // the first loads at once, while tensor memory is allocated and the block comes together (3 of a CTA's 48 us went
    // by before its first scores were there)
    mbar_arrive_expect_tx(&bars->k_full, C::kTile);
    load_tile(C::kFixOff, &tm_k, &bars->k_full, t0);
    load_q(0);
    mbar_arrive_expect_tx(&bars->v_full, C::kTile);
    load_tile(C::kFixOff + C::kTile, &tm_v, &bars->v_full, t0);
    load_x(0);
    bars->abort_flag = *reinterpret_cast<volatile int*>(&g_bwd_fused_abort);
  }
  if (warp == 13) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  const bool start_ok = (*abort_flag == 0);

  // registers: 256 x compute + 128 x dQ + 128 x 64 = the 512 x 128 that the block was launched with.  A warp that takes
  // dQ out holds all of a row (so that the tensor memory is free again at once) where the compute warps can spare them.
  constexpr int kRegOut = D == 64 ? 96 : (FEAT == 0 ? 144 : 128), kRegCompute = (512 * 128 - 128 * 64 - 128 * kRegOut) / 256;
  if (warp >= 12) {
    setmaxnreg_dec<64>();
    if (warp == 12) {
      // ------------------------------------------------ TMA: ring of Q with its column values
      if (lane == 0) {
        bool ok = true;
        int it = 1;
        for (; it < n && start_ok; ++it) {
          if (it >= 2) ok = mbar_wait(&bars->q_empty[it & 1], ((it >> 1) - 1) & 1, abort_flag);
          if (!ok) break;
          load_q(it);
        }
        if (*abort_flag) {
          mbar_wait_drain(&bars->k_full, 0, kDrainNs);
          mbar_wait_drain(&bars->v_full, 0, kDrainNs);
          for (int jj = max(0, it - 2); jj < it; ++jj) mbar_wait_drain(&bars->q_full[jj & 1], (jj >> 1) & 1, kDrainNs);
        }
      }
    } else if (warp == 15) {
      // ------------------------------------------------ TMA: ring of dX
      if (lane == 0) {
        bool ok = true;
        int it = 1;
        for (; it < n && start_ok; ++it) {
          if (it >= C::kXStages) ok = mbar_wait(&bars->x_empty[it % C::kXStages], (it / C::kXStages - 1) & 1, abort_flag);
          if (!ok) break;
          load_x(it);
        }
        if (*abort_flag)
          for (int jj = max(0, it - C::kXStages); jj < it; ++jj)
            mbar_wait_drain(&bars->x_full[jj % C::kXStages], (jj / C::kXStages) & 1, kDrainNs);
      }
    } else if (start_ok) {
      // ------------------------------------------------ MMA issuers
      if (lane == 0) {
        constexpr uint32_t idesc_nt = make_idesc_f16(BF16, 128, 128, false, false);  // both operands K-major
        constexpr uint32_t idesc_acc = make_idesc_f16(BF16, 128, D, false, true);    // B MN-major
        constexpr uint32_t idesc_dq = make_idesc_f16(BF16, 128, D, true, true);      // both MN-major
        constexpr uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
        constexpr uint32_t lbo_k = (16u >> 4) << 16;
        constexpr uint32_t lbo_mn = (static_cast<uint32_t>(kChunkBytes) >> 4) << 16;
        constexpr uint32_t tile16 = C::kTile >> 4;
        const uint32_t base16 = smem_u32(smem) >> 4;
        const uint32_t k16 = base16 + (C::kFixOff >> 4), v16 = k16 + tile16, q16 = base16 + (C::kQOff >> 4),
                       x16 = base16 + (C::kXOff >> 4), ds16 = base16 + (C::kDsOff >> 4);

        // product of two K-major tiles, D terms
        auto issue_nt = [&](uint32_t dcol, uint32_t a16, uint32_t b16) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = (kk >> 2) * (kChunkBytes >> 4) + (kk & 3) * 2;
            umma_ss_lohi(tmem + dcol, (a16 + off) | lbo_k, (b16 + off) | lbo_k, desc_hi, idesc_nt, kk > 0 ? 1u : 0u);
          }
        };
        // accumulator += (16-bit values in tensor memory, half 0 from acol, half 1 64 columns on) * MN-major tile
        auto issue_acc = [&](uint32_t dcol, uint32_t acol, uint32_t b16, bool first) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)
            umma_ts_lohi(tmem + dcol, tmem + acol + (kk >> 2) * 64 + (kk & 3) * 8, (b16 + kk * (2048 >> 4)) | lbo_mn, desc_hi,
                         idesc_acc, (first && kk == 0) ? 0u : 1u);
        };

        bool ok = mbar_wait(&bars->k_full, 0, abort_flag);
        if (warp == 13) {
          if (ok) ok = mbar_wait(&bars->q_full[0], 0, abort_flag);
          if (ok) {
            issue_nt(C::kColS, k16, q16);
            umma_commit(&bars->s_full);
          }
          for (int it = 0; it < n && ok; ++it) {
            const int s1 = (it + 1) & 1, sx = it % C::kXStages;
            ok = mbar_wait(&bars->x_full[sx], (it / C::kXStages) & 1, abort_flag);
            if (ok) ok = mbar_wait(&bars->p_ready, it & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            issue_acc(C::kColDV, C::kColS, x16 + sx * tile16, it == 0);
            umma_commit(&bars->x_empty[sx]);
            if (it + 1 < n) {
              ok = mbar_wait(&bars->q_full[s1], ((it + 1) >> 1) & 1, abort_flag);
              if (!ok) break;
              issue_nt(C::kColS, k16, q16 + s1 * tile16);    // over P^T: behind the product with it
              umma_commit(&bars->s_full);
            }
          }
          if (ok) umma_commit(&bars->acc_full);
        } else {
          if (ok) ok = mbar_wait(&bars->v_full, 0, abort_flag);
          if (ok) ok = mbar_wait(&bars->x_full[0], 0, abort_flag);
          if (ok) {
            issue_nt(C::kColDP, v16, x16);
            umma_commit(&bars->dp_full);
            umma_commit(&bars->x_empty[0]);
          }
          for (int it = 0; it < n && ok; ++it) {
            const int s = it & 1;
            auto next_dp = [&](uint64_t* free_bar) {
              const int sx = (it + 1) % C::kXStages;
              ok = mbar_wait(&bars->x_full[sx], ((it + 1) / C::kXStages) & 1, abort_flag);
              if (ok) ok = mbar_wait(free_bar, it & 1, abort_flag);
              if (!ok) return;
              tc_fence_after();
              issue_nt(C::kColDP, v16, x16 + sx * tile16);
              umma_commit(&bars->dp_full);
              umma_commit(&bars->x_empty[sx]);
            };
            if (D == 64 && it + 1 < n) next_dp(&bars->dp_read);    // dP is in registers
            if (ok) ok = mbar_wait(&bars->q_full[s], (it >> 1) & 1, abort_flag);
            if (D == 64 && ok && it > 0) ok = mbar_wait(&bars->dq_read, (it - 1) & 1, abort_flag);
            if (ok) ok = mbar_wait(&bars->ds_ready, it & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_ss_lohi(tmem + C::kColDQ, (ds16 + kk * (2048 >> 4)) | lbo_mn, (k16 + kk * (2048 >> 4)) | lbo_mn, desc_hi,
                           idesc_dq, kk > 0 ? 1u : 0u);
            umma_commit(&bars->dq_full);
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_ss_lohi(tmem + C::kColDK, (ds16 + (kk >> 2) * (kChunkBytes >> 4) + (kk & 3) * 2) | lbo_k,
                           (q16 + s * tile16 + kk * (2048 >> 4)) | lbo_mn, desc_hi, idesc_acc, (it == 0 && kk == 0) ? 0u : 1u);
            umma_commit(&bars->q_empty[s]);                         // also tells that dS has been read
            if (D == 128 && it + 1 < n) next_dp(&bars->dq_read);    // dQ, over which dP is written, is in registers
          }
          if (ok) umma_commit(&bars->acc_full);
        }
      }
    }
  } else if (warp >= 8) {
    if (kRegOut > 128) setmaxnreg_inc<kRegOut>(); else setmaxnreg_dec<kRegOut>();
    if (start_ok) {
      // ------------------------------------------------ dQ: one query per thread
      const int wq = warp & 3;
      const uint32_t tDQ = tmem + (static_cast<uint32_t>(wq * 32) << 16) + C::kColDQ;
      bool ok = true;
      // A warp's 32 queries x 32 features at a time, staged as [feature / 4][query][4] (the workspace's order, a warp's
      // queries together) and added by the copy engine.  Additions from registers keep the load / store queue busy
      // at the rate L2 takes them (22 bytes a cycle and SM), and everything else behind them in it waits.
      uint8_t* out_s = smem + C::kOutOff + wq * 2 * C::kPieceBytes;
      // Which scores of the warp's 32 keys survived the forward's dropout, a word per query: drawn here, two steps ahead,
      // because these warps have the time: d = 64, 2048 x 2048, 128 units 882 us with the compute warps drawing and trading
      // by votes, 773 so; d = 80, 1000 x 777, padding 139 and 128.  Lane L draws the call of (query L % 8 of eight, keys
      // 8 (L / 8) ..), and the bytes of a query's four calls are put together by exchanges.  Four calls in lockstep hide
      // each other's latency; beside a bias, with its stores, two in turn are quicker (256 x 2048, 256 units 906 and 978).
      auto draw_keep = [&](int it) {
        const unsigned int j8 = (unsigned int)(t0 + wq * 32) / 8u + (unsigned int)(lane >> 3);
        unsigned int* words = reinterpret_cast<unsigned int*>(smem + C::kKeepOff) + ((it & 1) * 4 + wq) * 128;
        const unsigned long long row0 = score_row(a, tile_of(it) * 128 + (lane & 7), h, b);
#pragma unroll 1
        for (int q32 = 0; q32 < 4; ++q32) {
          unsigned int word = 0u, w[4][4];
          if (!BIAS) dropout_words4(a, row0 + (unsigned int)(q32 * 32), 8u, j8, 0u, w);
#pragma unroll(BIAS ? 2 : 4)
          for (int q8 = 0; q8 < 4; ++q8) {
            unsigned int (&wq8)[4] = w[BIAS ? 0 : q8];
            if (BIAS) dropout_words(a, row0 + (unsigned int)(q32 * 32 + q8 * 8), j8, wq8);
            // bits 15 / 31 of a word's test belong to keys 2 e / 2 e + 1
            unsigned int k = keep_lanes(a, wq8[0]) >> 15;
            k |= keep_lanes(a, wq8[1]) >> 13;
            k |= keep_lanes(a, wq8[2]) >> 11;
            k |= keep_lanes(a, wq8[3]) >> 9;
            unsigned int v = ((k & 0x55u) | ((k >> 15) & 0xaau)) << (8 * (lane >> 3));
            v |= __shfl_xor_sync(0xffffffffu, v, 8);
            v |= __shfl_xor_sync(0xffffffffu, v, 16);
            if ((lane >> 3) == q8) word = v;
          }
          words[q32 * 32 + lane] = word;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->keep_full[it & 1]);
      };
      if (DROP) {
        draw_keep(0);
        if (n > 1) draw_keep(1);
      }
      for (int it = 0; it < n; ++it) {
        ok = mbar_wait(&bars->dq_full, it & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        float* p = dq_u + (long long)tile_of(it) * (128 * D) + wq * (32 * D);
        constexpr int kHeld = kRegOut == 128 ? 3 : D / 32;   // of the D / 32 pieces of 32 features
        uint32_t v[kHeld][32];
#pragma unroll
        for (int c = 0; c < kHeld; ++c) tmem_ld32(tDQ + 32 * c, v[c]);
        tmem_wait_ld();
        auto release = [&] {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->dq_read);
        };
        if (kHeld == D / 32) release();
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t (&vc)[32] = v[c % kHeld];
          constexpr int PF = C::kPieceFeat;
#pragma unroll
          for (int f = 0; f < 32; f += PF) {
            uint8_t* piece = out_s + ((c * 32 + f) / PF & 1) * C::kPieceBytes;
            if (lane == 0) tma_store_wait_read<1>();          // the piece before the last has been read
            __syncwarp();
#pragma unroll
            for (int e = 0; e < PF; e += 4)
              *reinterpret_cast<uint4*>(piece + (e >> 2) * 512 + lane * 16) =
                  make_uint4(vc[f + e], vc[f + e + 1], vc[f + e + 2], vc[f + e + 3]);
            if (kHeld < D / 32 && c == 0 && f + PF == 32) {
              __syncwarp();
              tmem_ld32(tDQ + 32 * kHeld, v[0]);
              tmem_wait_ld();
              release();
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              bulk_add_f32(p + c * 1024 + f * 32, piece, C::kPieceBytes);
              tma_store_commit();
            }
          }
        }
        if (DROP && it + 2 < n) {
          ok = mbar_wait(&bars->keep_free[it & 1], (it >> 1) & 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          draw_keep(it + 2);
        }
      }
      if (lane == 0) tma_store_wait_read<0>();
    }
  } else {
    setmaxnreg_inc<kRegCompute>();
    if (start_ok) {
      // ------------------------------------------------ compute
      // element (hh, 4 j + 2 s + e) of a thread: key t0 + 32 wq + 16 hh + 8 s + lane / 4,
      // query 64 half + 8 j + 2 (lane % 4) + e of the tile
      const int half = warp >> 2, wq = warp & 3;
      const uint32_t lane_base = tmem + (static_cast<uint32_t>(wq * 32) << 16);
      const uint32_t tS = lane_base + C::kColS + half * 64, tDP = lane_base + C::kColDP + half * 64;
      const unsigned long long c2 = pair_of(a.scale * kLog2e);
      const int rb = t0 + wq * 32 + (lane >> 2);        // first of the thread's four keys (8 apart)
      const int cb = half * 64 + 2 * (lane & 3);        // first of its columns in a tile
      const float* col_s = reinterpret_cast<const float*>(smem + C::kColOff) + cb;
      // stmatrix rows: lane 8 m + i gives row i of matrix m = (s = m & 1, j + (m >> 1))
      const int st_row = wq * 32 + (lane & 7) + 8 * ((lane >> 3) & 1);
      const uint32_t st_base = smem_u32(smem) + C::kDsOff + half * kChunkBytes + st_row * 128;
      const int st_j = lane >> 4, st_x = st_row & 7;
      const bool edge_rows = t0 + 128 > a.Lkv;
      bool ok = true;

      // key-padding masks (no dependence on the query): one byte per key for the whole kernel
      const unsigned char* mask_u = nullptr;
      bool mask_per_step = false, mask_rows = false, mask_vec = false;
      unsigned int dead_rows = 0;                       // bit 2 hh + s: nothing attends to that key
      if (MASKED) {
        mask_u = a.mask + (long long)h * a.mask_s[2] + (long long)b * a.mask_s[3];
        mask_per_step = a.mask_s[1] != 0;
        mask_rows = a.mask_s[0] == 1 && t0 + wq * 32 + 32 <= a.Lkv;
        mask_vec = ((reinterpret_cast<uintptr_t>(mask_u) | (uintptr_t)a.mask_s[1]) & 15u) == 0;   // (t0 + 32 wq: a multiple of 32)
        if (!mask_per_step) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (rb + 8 * k < a.Lkv && __ldg(mask_u + (long long)(rb + 8 * k) * a.mask_s[0]) == 0) dead_rows |= 1u << k;
        }
      }
      const unsigned char* bias_u = nullptr;
      const int bias_esz = (BIAS && a.bias_dtype == NNLIB_B200_F32) ? 4 : 2;
      if (BIAS)
        bias_u = reinterpret_cast<const unsigned char*>(a.bias) +
                 ((long long)h * a.bias_s[2] + (long long)b * a.bias_s[3]) * bias_esz;
      float* dbias_u = nullptr;
      bool dbias_exclusive = false;
      if (BIAS && g.dbias) {
        dbias_u = g.dbias + (long long)h * g.dbias_s[2] + (long long)b * g.dbias_s[3];
        dbias_exclusive = (g.dbias_s[0] != 0 || a.Lkv == 1) && (g.dbias_s[1] != 0 || a.Lq == 1) &&
                          (g.dbias_s[2] != 0 || a.H == 1) && (g.dbias_s[3] != 0 || a.B == 1);
      }

      for (int it = 0; it < n; ++it) {
        const int st = it & 1;
        const int c0 = tile_of(it) * 128;               // first query of the tile
        const float* cols = col_s + st * (kColBytes / 4);

        // mask bytes of the warp's 32 keys x 64 queries, a word of 32 bits per query: the threads need those of their 16
        // queries, shifted so that key 8 k + lane / 4 is the sign of byte k.  Where a query's keys lie side by side a lane reads
        // the 32 bytes of two queries and the words change hands; otherwise a query's keys are read by the 32 lanes
        // and voted into a word.
        unsigned int mv[16];
        if (MASKED && mask_per_step) {
          if (mask_rows) {
            unsigned int wd[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              unsigned int w[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
              const int col = c0 + half * 64 + 32 * k + lane;
              if (col < a.Lq) {
                const unsigned char* mp = mask_u + (t0 + wq * 32) + (long long)col * a.mask_s[1];
                if (mask_vec) {
                  const uint4 x = __ldg(reinterpret_cast<const uint4*>(mp)), y = __ldg(reinterpret_cast<const uint4*>(mp) + 1);
                  w[0] = x.x; w[1] = x.y; w[2] = x.z; w[3] = x.w;
                  w[4] = y.x; w[5] = y.y; w[6] = y.z; w[7] = y.w;
                } else {
                  load_shifted<8>(mp, mp + 32, w);
                }
              }
              wd[k] = 0u;
#pragma unroll
              for (int u = 0; u < 8; ++u) {
                // bit 7 of a byte: the byte is not zero; the four of them gathered in the top four bits of a product
                const unsigned int nz = ((((w[u] & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w[u]) & 0x80808080u) >> 7;
                wd[k] |= ((nz * 0x10204080u) >> 28) << (4 * u);
              }
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 16; ++k)
              mv[k] = __shfl_sync(0xffffffffu, wd[k >> 3], (8 * (k >> 1) + 2 * (lane & 3) + (k & 1)) & 31);
          } else {
            const int row = t0 + wq * 32 + lane;
            const unsigned char* mp = mask_u + (long long)row * a.mask_s[0] + (long long)(c0 + half * 64) * a.mask_s[1];
            const int n_cols = row < a.Lkv ? a.Lq - c0 - half * 64 : 0;
#pragma unroll
            for (int c = 0; c < 64; ++c) {
              const bool keep = c < n_cols && __ldg(mp + (long long)c * a.mask_s[1]) != 0;
              const unsigned int v = __ballot_sync(0xffffffffu, keep);
              if ((lane & 3) == ((c & 7) >> 1)) mv[2 * (c >> 3) + (c & 1)] = v;
            }
          }
#pragma unroll
          for (int k = 0; k < 16; ++k) mv[k] <<= 7 - (lane >> 2);
        }
        // survivors of the forward's dropout, in the same form
        unsigned int kw[16];
        if (DROP) {
          ok = mbar_wait(&bars->keep_full[st], (it >> 1) & 1, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const unsigned int* words = reinterpret_cast<const unsigned int*>(smem + C::kKeepOff) + (st * 4 + wq) * 128 + cb;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint2 w = *reinterpret_cast<const uint2*>(words + 8 * j);
            kw[2 * j] = w.x << (7 - (lane >> 2));
            kw[2 * j + 1] = w.y << (7 - (lane >> 2));
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->keep_free[st]);
        }
        // 16-bit bias: element pairs (one key, two queries) packed to a word
        unsigned int bw[2][16];
        if (BIAS && bias_esz == 2) {
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const long long row = min(rb + 16 * hh + 8 * (k & 1), a.Lkv - 1);
              const int col = c0 + cb + 8 * (k >> 1);
              const unsigned char* bp = bias_u + 2 * row * a.bias_s[0];
              const unsigned int lo = __ldg(reinterpret_cast<const unsigned short*>(bp + 2ll * min(col, a.Lq - 1) * a.bias_s[1]));
              const unsigned int hi = __ldg(reinterpret_cast<const unsigned short*>(bp + 2ll * min(col + 1, a.Lq - 1) * a.bias_s[1]));
              bw[hh][k] = lo | (hi << 16);
            }
        }

        ok = mbar_wait(&bars->q_full[st], (it >> 1) & 1, abort_flag);   // the column values
        if (ok) ok = mbar_wait(&bars->s_full, st, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        uint32_t su[2][32];
        tmem_ld_frag(tS, su[0]);
        tmem_ld_frag(tS + (16u << 16), su[1]);
        tmem_wait_ld();
        // P = exp2(S scale log2(e) - lse)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 nl = *reinterpret_cast<const float2*>(cols + 8 * j);
          const unsigned long long nlp = pair_pack(nl.x, nl.y);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              uint32_t& u0 = su[hh][4 * j + 2 * s];
              uint32_t& u1 = su[hh][4 * j + 2 * s + 1];
              unsigned long long t = nlp;
              if (BIAS) {
                float b0, b1;
                if (bias_esz == 2) {
                  const unsigned int w = bw[hh][2 * j + s];
                  if (a.bias_dtype == NNLIB_B200_BF16) {
                    b0 = __uint_as_float(w << 16);
                    b1 = __uint_as_float(w & 0xffff0000u);
                  } else {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
                    b0 = f.x; b1 = f.y;
                  }
                } else {
                  const long long row = min(rb + 16 * hh + 8 * s, a.Lkv - 1);
                  const int col = c0 + cb + 8 * j;
                  const float* bp = reinterpret_cast<const float*>(bias_u) + row * a.bias_s[0];
                  b0 = __ldg(bp + (long long)min(col, a.Lq - 1) * a.bias_s[1]);
                  b1 = __ldg(bp + (long long)min(col + 1, a.Lq - 1) * a.bias_s[1]);
                }
                t = pair_fma(pair_pack(b0, b1), pair_of(kLog2e), t);
              }
              t = pair_fma(pair_pack(__uint_as_float(u0), __uint_as_float(u1)), c2, t);
              float p0, p1;
              pair_unpack(t, p0, p1);
              u0 = __float_as_uint(ex2_approx(p0));
              u1 = __float_as_uint(ex2_approx(p1));
            }
        }
        // queries before a key (causal, on the diagonal tile) and padded or masked-out keys contribute nothing
        const bool diag = a.causal && c0 == t0;
        // padded queries have lse = +inf, and the last query's bias, read in their place, may be that, too, or NaN.  (In a
        // block of its own this took 8 % with dropout: 256 x 2048, 256 units 750 us.)
        const bool edge_cols = BIAS && c0 + 128 > a.Lq;
        if (edge_rows || diag || edge_cols || (MASKED && dead_rows != 0u)) {
          const int last = edge_cols ? a.Lq - c0 - cb : 0x40000000;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int row = rb + 8 * k;
            int first = diag ? row - c0 - cb : -0x40000000;            // columns (from cb on) before it are zero
            if (row >= a.Lkv || (MASKED && ((dead_rows >> k) & 1u))) first = 0x40000000;
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e)
                if (8 * j + e < first || (BIAS && 8 * j + e >= last)) su[k >> 1][4 * j + 2 * (k & 1) + e] = 0u;
          }
        }
        if (MASKED && mask_per_step) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e)
                su[k >> 1][4 * j + 2 * (k & 1) + e] &= byte_sign(mv[2 * j + e], k);
        }
        // P^T rounded to the element type over S: what dV takes, with dropout alpha' = P keep / (1 - p)
        uint32_t pk[16];
        __syncwarp();
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              float p0 = __uint_as_float(su[hh][4 * j + 2 * s]), p1 = __uint_as_float(su[hh][4 * j + 2 * s + 1]);
              if (DROP) pair_unpack(pair_mul(pair_pack(p0, p1), pair_of(a.inv_keep)), p0, p1);
              pk[2 * j + s] = pack2<BF16>(p0, p1);
              if (DROP) pk[2 * j + s] &= byte_sign_pair(kw[2 * j], kw[2 * j + 1], 2 * hh + s);
            }
          tmem_st_frag16(tS + (static_cast<uint32_t>(16 * hh) << 16), pk);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_ready);

        // dS = P (dP - D), with dropout P (dP keep / (1 - p) - D), rounded to the element type, in shared memory, once the
        // previous step's products have read it.  (1 / (1 - p) belongs in front of the roundings: left to the results, dS of
        // a p near 1 falls among Float16's subnormal numbers.)
        ok = mbar_wait(&bars->dp_full, st, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        uint32_t dp[2][32];
        tmem_ld_frag(tDP, dp[0]);
        tmem_ld_frag(tDP + (16u << 16), dp[1]);
        if (it > 0) ok = mbar_wait(&bars->q_empty[st ^ 1], ((it - 1) >> 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tmem_wait_ld();
        if (D == 64) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->dp_read);
        }
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            uint32_t pk4[4];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              const float2 nd = *reinterpret_cast<const float2*>(cols + 128 + 8 * (j + jj));
              const unsigned long long ndp = pair_pack(nd.x, nd.y);
#pragma unroll
              for (int s = 0; s < 2; ++s) {
                const int e0 = 4 * (j + jj) + 2 * s;
                if (DROP) {
                  dp[hh][e0] &= byte_sign(kw[2 * (j + jj)], 2 * hh + s);
                  dp[hh][e0 + 1] &= byte_sign(kw[2 * (j + jj) + 1], 2 * hh + s);
                }
                const float g0 = __uint_as_float(dp[hh][e0]), g1 = __uint_as_float(dp[hh][e0 + 1]);
                float d0, d1;
                const unsigned long long gp = pair_pack(g0, g1);
                pair_unpack(pair_mul(DROP ? pair_fma(gp, pair_of(a.inv_keep), ndp) : pair_add(gp, ndp),
                                     pair_pack(__uint_as_float(su[hh][e0]), __uint_as_float(su[hh][e0 + 1]))), d0, d1);
                pk4[2 * jj + s] = pack2<BF16>(d0, d1);
                if (BIAS) {
                  su[hh][e0] = __float_as_uint(d0);
                  su[hh][e0 + 1] = __float_as_uint(d1);
                }
              }
            }
            stmatrix_x4(st_base + hh * 2048 + (((j + st_j) ^ st_x) << 4), pk4[0], pk4[1], pk4[2], pk4[3]);
          }
        }
        tc_fence_before();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->ds_ready);

        if (BIAS && dbias_u) {
          // gradient of the bias = dS in fp32: plain stores when every score has its own element, atomic additions
          // when a stride of 0 folds several scores onto one
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int row = rb + 8 * k;
            if (row >= a.Lkv) continue;
            float* o = dbias_u + (long long)row * g.dbias_s[0];
#pragma unroll
            for (int j = 0; j < 8; ++j)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int col = c0 + cb + 8 * j + e;
                if (col >= a.Lq) continue;
                const float v = __uint_as_float(su[k >> 1][4 * j + 2 * (k & 1) + e]);
                float* oc = o + (long long)col * g.dbias_s[1];
                if (dbias_exclusive) *oc = v; else atomicAdd(oc, v);
              }
          }
          __syncwarp();
        }
      }

      // ------------------------------------------------ dV (warps 0-3) and dK (warps 4-7): one key per thread
      if (ok) {
        ok = mbar_wait(&bars->acc_full, 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok) {
        tc_fence_after();
        // through K's place (dV through V's: every product has read them) in the layout of the copy engine, which leaves
        // out keys past the end and padding; stored from here, 16 bytes a row and thread, they took 3 us
        const int r = wq * 32 + lane;
        uint8_t* stage = smem + C::kFixOff + (half == 0 ? C::kTile : 0);
        const float mul = half == 0 ? 1.f : a.scale;
        const uint32_t col = lane_base + (half == 0 ? C::kColDV : C::kColDK);
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t o[32];
          tmem_ld32(col + c * 32, o);
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 v;
            v.x = pack2<BF16>(__uint_as_float(o[e]) * mul, __uint_as_float(o[e + 1]) * mul);
            v.y = pack2<BF16>(__uint_as_float(o[e + 2]) * mul, __uint_as_float(o[e + 3]) * mul);
            v.z = pack2<BF16>(__uint_as_float(o[e + 4]) * mul, __uint_as_float(o[e + 5]) * mul);
            v.w = pack2<BF16>(__uint_as_float(o[e + 6]) * mul, __uint_as_float(o[e + 7]) * mul);
            const int piece = (c & 1) * 4 + e / 8;
            *reinterpret_cast<uint4*>(stage + (c >> 1) * kChunkBytes + r * 128 + ((piece ^ (r & 7)) << 4)) = v;
          }
        }
        fence_proxy_async_smem();
        asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory");
        if (wq == 0 && lane == 0) {
          for (int c = 0; c < D / 64; ++c)
            if (c * 64 < a.d) tma_store_4d(half == 0 ? &tm_dv : &tm_dk, stage + c * kChunkBytes, c * 64, h, t0, b);
          tma_store_commit();
          tma_store_wait_read<0>();
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) {
    atomicExch(&g_bwd_fused_abort, 1);
    if (a.status) atomicExch(a.status, NNLIB_B200_TIMEOUT);
  }
}

// Before: D_i = dx_i . x_i and lse of a tile's queries, negated and (lse) in base 2, and zeros for its dQ.  One block
// per tile of 128 queries of a unit; LANES threads share a query.  Bound by memory: reads dx and x, writes the zeros.
template <int DPAD, bool BF16>
__global__ void __launch_bounds__(256) attn_bwd_fused_pre_kernel(const AttnArgs a, const BwdArgs g, const int n_q) {
  constexpr int LANES = DPAD / 8;                 // 16-byte pieces of a row
  constexpr int ROWS = 256 / LANES;               // queries at a time
  const long long tile = blockIdx.x;
  const int t = (int)(tile % n_q), unit = (int)(tile / n_q), h = unit % a.H, b = unit / a.H;
  const long long tiles_all = gridDim.x;
  float4* z = reinterpret_cast<float4*>(a.ws + tiles_all * (kColBytes / 4) + tile * (128 * DPAD));
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 128 * DPAD / 4 / 256; ++i) z[i * 256 + threadIdx.x] = zero;
  float* cols = a.ws + tile * (kColBytes / 4);
  const int piece = threadIdx.x % LANES;
#pragma unroll 4
  for (int r = threadIdx.x / LANES; r < 128; r += ROWS) {
    const int q = t * 128 + r;
    float acc = 0.f;
    if (q < a.Lq && piece * 8 < a.d) {
      const uint4 x = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(a.x) +
                            2ll * ((long long)q * a.x_sl + (long long)b * a.x_sb + (long long)h * a.d + piece * 8)));
      const uint4 y = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(g.dx) +
                            2ll * ((long long)q * g.dx_sl + (long long)b * g.dx_sb + (long long)h * a.d + piece * 8)));
      const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float2 fx, fy;
        if (BF16) {
          fx = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xs[e]));
          fy = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ys[e]));
        } else {
          fx = __half22float2(*reinterpret_cast<const __half2*>(&xs[e]));
          fy = __half22float2(*reinterpret_cast<const __half2*>(&ys[e]));
        }
        acc = fmaf(fx.x, fy.x, acc);
        acc = fmaf(fx.y, fy.y, acc);
      }
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (piece == 0) {
      float nl = neg_inf(), nd = 0.f;                 // padded query, or one that attends to nothing: P = 0
      if (q < a.Lq) {
        const float l = __ldg(a.lse + (long long)a.Lq * h + a.lse_sb * b + q);
        if (l != neg_inf()) {
          nl = -(l * kLog2e);
          nd = -acc;
        }
      }
      cols[r] = nl;
      cols[128 + r] = nd;
    }
  }
}

// Behind: dq = scale dQ in the element type.  One block per tile; a thread takes 16 features of a query (32 bytes).
template <int DPAD, bool BF16>
__global__ void __launch_bounds__(256) attn_bwd_fused_post_kernel(const AttnArgs a, const BwdArgs g, const int n_q) {
  const long long tile = blockIdx.x;
  const int t = (int)(tile % n_q), unit = (int)(tile / n_q), h = unit % a.H, b = unit / a.H;
  const long long tiles_all = gridDim.x;
  const int r = threadIdx.x & 127, q = t * 128 + r;
  if (q >= a.Lq) return;
  const float mul = a.scale;
  const float4* w = reinterpret_cast<const float4*>(a.ws + tiles_all * (kColBytes / 4) + tile * (128 * DPAD)) + (r >> 5) * (8 * DPAD) + (r & 31);
  uint8_t* out = reinterpret_cast<uint8_t*>(g.dq) +
                 2ll * (((long long)q + (long long)a.Lq * b) * ((long long)a.H * a.d) + (long long)h * a.d);
#pragma unroll
  for (int i = 0; i < DPAD / 32; ++i) {
    const int f = ((threadIdx.x >> 7) + 2 * i) * 16;
    if (f >= a.d) break;
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = __ldcg(w + (f / 4 + u) * 32);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (f + 8 * u >= a.d) break;
      uint4 o;
      o.x = pack2<BF16>(v[2 * u].x * mul, v[2 * u].y * mul);
      o.y = pack2<BF16>(v[2 * u].z * mul, v[2 * u].w * mul);
      o.z = pack2<BF16>(v[2 * u + 1].x * mul, v[2 * u + 1].y * mul);
      o.w = pack2<BF16>(v[2 * u + 1].z * mul, v[2 * u + 1].w * mul);
      *reinterpret_cast<uint4*>(out + (f + 8 * u) * 2) = o;
    }
  }
}

template <int D, bool BF16, int FEAT>
cudaError_t launch_fused(const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mq, const CUtensorMap& mdx,
                         const CUtensorMap& mdk, const CUtensorMap& mdv, const AttnArgs& a, const BwdArgs& g, cudaStream_t st) {
  auto kern = attn_bwd_fused_kernel<D, BF16, FEAT>;
  constexpr int smem = FuCfg<D, (FEAT & 2) != 0>::kSmemBytes;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int n_tiles = (a.Lkv + 127) / 128, n_q = (a.Lq + 127) / 128;
  const long long n_units = (long long)a.H * a.B;
  const long long blocks = n_tiles * n_units, q_blocks = n_q * n_units;
  if (blocks > 0x7fffffffLL || q_blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  // causal walks differ in length: the units of the last two waves are dealt out longest walks first, as long as
  // their arrays stay well inside L2 together (attn_bwd_umma.cu)
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      sms < 1)
    sms = 148;
  long long tail_units = a.causal ? 2 * ((sms + n_tiles - 1) / n_tiles) : 0;
  if (tail_units > n_units) tail_units = n_units;
  const long long unit_bytes = 2ll * ((long long)a.Lq + a.Lkv) * a.d * 2 + 4ll * a.Lq * D;
  if (tail_units * unit_bytes > (48ll << 20)) tail_units = (48ll << 20) / unit_bytes;
  if (tail_units < 2) tail_units = 0;
  attn_bwd_fused_pre_kernel<D, BF16><<<(unsigned)q_blocks, 256, 0, st>>>(a, g, n_q);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)blocks, kFuThreads, smem, st>>>(mk, mv, mq, mdx, mdk, mdv, a, g, n_tiles, (int)tail_units);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  attn_bwd_fused_post_kernel<D, BF16><<<(unsigned)q_blocks, 256, 0, st>>>(a, g, n_q);
  count_launch(3);
  return cudaGetLastError();
}

}  // namespace

size_t umma_bwd_fused_workspace_bytes(const AttnArgs& a) {
  const long long tiles = ((long long)a.Lq + 127) / 128 * a.H * a.B;
  return (size_t)(tiles * fused_tile_floats(a.d > 64 ? 128 : 64)) * sizeof(float);
}

cudaError_t umma_bwd_fused(const AttnArgs& a, const BwdArgs& g, int dtype, cudaStream_t st) {
  CUtensorMap mq, mk, mv, mdx, mdk, mdv;
  if (!make_head_map(&mq, a.q, dtype, a.d, a.H, a.Lq, a.B, a.q_sl, a.q_sb)) return cudaErrorInvalidValue;
  if (!make_head_map(&mk, a.k, dtype, a.d, a.H, a.Lkv, a.B, a.k_sl, a.k_sb)) return cudaErrorInvalidValue;
  if (!make_head_map(&mv, a.v, dtype, a.d, a.H, a.Lkv, a.B, a.v_sl, a.v_sb)) return cudaErrorInvalidValue;
  if (!make_head_map(&mdx, g.dx, dtype, a.d, a.H, a.Lq, a.B, g.dx_sl, g.dx_sb)) return cudaErrorInvalidValue;
  const long long E = (long long)a.H * a.d;
  if (!make_head_map(&mdk, g.dk, dtype, a.d, a.H, a.Lkv, a.B, E, E * a.Lkv)) return cudaErrorInvalidValue;
  if (!make_head_map(&mdv, g.dv, dtype, a.d, a.H, a.Lkv, a.B, E, E * a.Lkv)) return cudaErrorInvalidValue;
  const bool bf16 = dtype == NNLIB_B200_BF16;
  const int feat = (a.mask ? 1 : 0) | (a.dropout_p > 0.f ? 2 : 0) | (a.bias ? 4 : 0);
#define NB_FU(DD, BF)                                                  \
  switch (feat) {                                                      \
    case 0: return launch_fused<DD, BF, 0>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    case 1: return launch_fused<DD, BF, 1>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    case 2: return launch_fused<DD, BF, 2>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    case 3: return launch_fused<DD, BF, 3>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    case 4: return launch_fused<DD, BF, 4>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    case 5: return launch_fused<DD, BF, 5>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    case 6: return launch_fused<DD, BF, 6>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
    default: return launch_fused<DD, BF, 7>(mk, mv, mq, mdx, mdk, mdv, a, g, st); \
  }
  if (a.d > 64) {
    if (bf16) { NB_FU(128, true) } else { NB_FU(128, false) }
  } else {
    if (bf16) { NB_FU(64, true) } else { NB_FU(64, false) }
  }
#undef NB_FU
}

// Reads and clears the kernel's sticky "a bounded wait ran out" flag of the current device.  Synchronises the stream.
cudaError_t umma_bwd_fused_take_abort(int* out, cudaStream_t st) {
  int v = 0;
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyFromSymbol(&v, g_bwd_fused_abort, sizeof(int));
  if (e != cudaSuccess) return e;
  if (v) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(g_bwd_fused_abort, &zero, sizeof(int));
  }
  *out = v;
  return e;
}

}  // namespace nb200
