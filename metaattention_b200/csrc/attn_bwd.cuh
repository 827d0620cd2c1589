// Backward of attention for sm_100a, generic over a functor that gives P and dS per score element (head dims
// 128 / 128 or 64 / 64, 16-bit inputs, fp32 accumulation):
//
//   dV = P^T dO,   dP = dO V^T,   dS = dP o dP/dS,   dK = dS^T Q,   dQ = dS K
//
// One kernel template in two roles.  A CTA keeps one 128-row tile pair resident (X: K_j, V_j or Q_i, dO_i) and streams
// the other (Y1: Q_i or K_j through a three-stage TMA ring, Y2: dO_i or V_j through a two-stage one).  Per streamed tile:
//   S  = X1 Y1^T, dP = X2 Y2^T           tcgen05 SS, fp32 in tensor memory (attn_bwd_cta has the columns)
//   row threads (thread = TMEM lane x column half): P and dS as 16-bit pairs
//   acc1 += P  Y2   (dV; KV role only)    tcgen05 TS, A from tensor memory, B = the streamed tile MN-major
//   acc2 += dS Y1   (dK or dQ)
// With the KV role the lanes are KV rows and the columns query rows (S^T, dP^T), so that P^T and dS^T are the A
// operands as they stand.  The functor F supplies
//   F::kUsesStats            per-query-row statistics (softmax: lse and delta) travel with the query tiles
//   F::kFiniteTail           without statistics: P and g are finite at a score of 0, so zero rows need no mask
//   F::kNegInfMask           P and dS vanish at a score of -inf: masked pairs are given that score
//   F::Ctx F::make(params)   per-thread constants
//   F::score(s, lse2, ctx, b, h, q_idx, kv_idx, p_out, g_out)   P, and the factor g that turns dP into dS
//   F::grad(g, dp, ctx)                                          dS without its constant factor; with statistics instead
//   F::score_row, F::grad_row                                    score() for a row of an unmasked tile, and dS of a row
//   F::out_scale(ctx)                                            the constant factor, applied to the finished dK, dQ rows
// softmax_bwd.cu instantiates it for the built-in softmax; lowered score_mod functors (elementwise programs: no row
// scales) get a library of their own, compiled from the forward-mode derivative of the traced expression.
//
// What bounds it: the row threads, whose phases for a tile follow one another (take S, exponentials, hand over P, take dP, dS,
// hand over), and in long calls the power that the seven products draw.  So a tile's S and dP leave their buffers for
// registers at once and the next ones are computed under the row threads' work, P and dS have columns of their own (over
// S and dP each product waited for the one that read them: 3330 and 2550 cycles a tile for the KV and the query
// role), S and dP are issued by one warp and the accumulators by another, and four threads share a row, four row warps
// to a scheduler.  Now 3000 and 2400 cycles with D = 128 (1 x 32 x 4096 non-causal forward and backward; products alone 2048 and
// 1536), 2400 and 1960 with D = 64; training step of 4 x 32 x 4096 x 128 causal 2775 -> 2610 us (at its power cap), of
// 4 x 8 / 2 x 2118 x 128 237 -> 215.  In the KV role the statistics of a tile's columns come through shared memory, 256
// sixteen-byte broadcasts a tile of ~3 cycles each beside the operands of the products (2048 cycles of its bandwidth).
//   KV role, D = 128  S and dP take one buffer in turn: S(i+1) is issued once dP(i) is in registers, dV(i) and dK(i) behind it.
//   Otherwise         a buffer each: S(i+1) and dP(i+1) are issued once S(i) and dP(i) are in registers.
//   Q role            dS sits in two buffers (the role has no second accumulator).
#pragma once

#include <cstring>
#include <type_traits>

#include "../../include/attn_b200.h"
#include "common_host.cuh"
#include "parallel_launch.cuh"  // tensor_map_encoder(), encode_rows_map(), CoordOrder, tma_load_rows()
#include "sm100.cuh"

namespace b200 {

constexpr int kBwdT = 128;                // rows of a tile, both ways
constexpr int kBwdRowGroups = 4;                                // threads that share a row of a tile
constexpr int kBwdRowWarps = kBwdRowGroups * kBwdT / 32;        // row warps: one TMEM lane and a part of the columns per thread
constexpr int kBwdThreads = kBwdRowWarps * 32 + 96;             // plus the loading warp and two that issue MMAs
constexpr int kBwdStages1 = 3;            // ring of Y1 (read by the first and by the last MMA of its tile)
constexpr int kBwdStages2 = 2;            // ring of Y2

struct BwdParams {
  const void* custom[ATTN_B200_MAX_CUSTOM];   // device pointers of the functor's custom inputs (lowered functors)
  void* dq;
  void* dk;
  void* dv;
  const float* lse2;    // [batch, heads, seq_q_pad] lse * log2(e); +inf past seq_q (those rows get P = 0)
  const float* delta;   // [batch, heads, seq_q_pad]
  int batch, heads, heads_kv, kv_group, seq_q, seq_kv, seq_q_pad;
  int mask_left, mask_right;   // keep q_idx - mask_left <= kv_idx <= q_idx + mask_right; ATTN_B200_MASK_OPEN = no bound
  // kBits kernels (any mask that does not depend on batch or head, as keep bits): bits_q[q][kv tile][4 words] = the
  // 128 keep bits of query row q in that KV tile, bits_kv[kv][query tile][4 words] the same matrix transposed; both
  // padded with zeros to whole tiles.  Every pair of tiles is visited.
  const uint32_t* bits_q;
  const uint32_t* bits_kv;
  // optional with the bits: which tiles keep anything at all, so that the others are not visited.  tiles_q[query tile]
  // [tile_words_k] = bitmap over the KV tiles, tiles_kv[KV tile][tile_words_q] = bitmap over the query tiles
  const uint32_t* tiles_q;
  const uint32_t* tiles_kv;
  int tile_words_k, tile_words_q;
  float scale;
  long long dq_s[3], dk_s[3], dv_s[3];   // element strides (batch, seq, head)
  CoordOrder oq, ok, ov, odo;
  int heads_at_once;   // of so many (query head, batch) pairs at a time the longest CTAs first; 0: of each
  int* status;
};

enum BwdWaitSite { kBwdXFull = 61, kBwdYFull, kBwdYEmpty, kBwdSFull, kBwdPReady, kBwdAccDone, kBwdSFree, kBwdDpFull, kBwdDsReady, kBwdSmemAlign, kBwdDpFree, kBwdPFree, kBwdDsFree, kBwdSIssued };
enum BwdBarrier {
  kBarXFull = 0,
  kBarY1Full,                               // kBwdStages1 of them
  kBarY1Empty = kBarY1Full + kBwdStages1,
  kBarY2Full = kBarY1Empty + kBwdStages1,   // kBwdStages2 of them
  kBarY2Empty = kBarY2Full + kBwdStages2,
  kBarSFull = kBarY2Empty + kBwdStages2,    // scores / dP of a tile in tensor memory, and in the row threads' registers
  kBarSFree,
  kBarDpFull,
  kBarDpFree,
  kBarPReady,                               // P of a tile in tensor memory, and read by its product (KV role)
  kBarPFree,
  kBarDsReady,                              // the same of dS, one per buffer of the query role
  kBarDsFree = kBarDsReady + 2,
  kBarSIssued = kBarDsFree + 2,             // the next tile's S is in the pipe (KV role with a shared buffer)
  kBarAccDone,
  kNumBwdBarriers
};

template <int D>
struct BwdSmem {
  static constexpr int kTileBytes = kBwdT * D * 2;            // D/64 chunks of 128 rows x 128 B (64 columns)
  static constexpr int kChunkBytes = kBwdT * 128;
  static constexpr int kOffX1 = 0;
  static constexpr int kOffX2 = kOffX1 + kTileBytes;
  static constexpr int kOffY1 = kOffX2 + kTileBytes;                   // [kBwdStages1] tiles
  static constexpr int kOffY2 = kOffY1 + kBwdStages1 * kTileBytes;     // [kBwdStages2] tiles
  static constexpr int kOffLse = kOffY2 + kBwdStages2 * kTileBytes;    // [kBwdStages1][128] fp32, with Y1 (KV role)
  static constexpr int kStatBytes = kBwdT * 4;
  static constexpr int kOffDelta = kOffLse + kBwdStages1 * kStatBytes; // [kBwdStages2][128] fp32, with Y2 (KV role)
  static constexpr int kOffBar = kOffDelta + kBwdStages2 * kStatBytes;
  static constexpr int kOffMisc = kOffBar + 8 * kNumBwdBarriers;
  static constexpr int kBytes = kOffMisc + 16;                // the dynamic shared memory is declared 1024-byte aligned
  static_assert(kBytes <= 232448, "shared memory layout exceeds an SM");
};

// plain (untiled) bulk copy global -> shared, counted on an mbarrier; both addresses 16-byte aligned, bytes % 16 == 0
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)),
               "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// The set bits of one row of a tile bitmap, in order, over and over (the KV role walks its row once per query head of
// its group).  The caller knows how many there are and never asks an empty row.
struct KeptTiles {
  const uint32_t* words;
  int nwords, w;
  uint32_t bits;
  __device__ KeptTiles(const uint32_t* p, int n) : words(p), nwords(n), w(-1), bits(0) {}
  __device__ int next() {
    while (bits == 0) {
      if (++w >= nwords) w = 0;
      bits = words[w];
    }
    const int j = w * 32 + __ffs(bits) - 1;
    bits &= bits - 1;
    return j;
  }
  __device__ int count() const {
    int c = 0;
    for (int i = 0; i < nwords; ++i) c += __popc(words[i]);
    return c;
  }
};

// kRoleQ = false: CTA = (KV tile, KV head, batch), streams the query tiles (of every query head of its group) and
// writes dK, dV.  kRoleQ = true: CTA = (query tile, query head, batch), streams the KV tiles and writes dQ.
// Tensor memory.  KV role: accumulators dV, dK (D columns each), P and dS (64 each, 16-bit pairs), then S and dP: with D = 128
// one buffer that they take in turn, with D = 64 one each.  Query role: accumulator dQ, two dS buffers, S, dP.
template <class F, bool kRoleQ, bool kBf16, int D, bool kBits>
__device__ __forceinline__ void attn_bwd_cta(const CUtensorMap& tmQ, const CUtensorMap& tmK, const CUtensorMap& tmV, const CUtensorMap& tmDO,
                                             const BwdParams& p, const int tile, const int hx, const int b) {
  using L = BwdSmem<D>;
  constexpr int T = kBwdT, KC = D / 64;   // chunks of a tile
  constexpr int C = T / kBwdRowGroups, AC = D / kBwdRowGroups, kRowWarps = kBwdRowWarps;   // columns per thread: of a tile, of an accumulator
  constexpr int N1 = kBwdStages1, N2 = kBwdStages2;
  static_assert(D == 64 || D == 128, "head dims 64 and 128");
  constexpr bool kShared = !kRoleQ && D == 128;   // S and dP share a buffer
  constexpr uint32_t kTmemCols = 512, kColA = 0, kColB = D, kColP = 2 * D, kColDS = kRoleQ ? 128 : 2 * D + 64, kColDP = 384,
                     kColS = kShared ? 384 : 256;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sX1 = smem + L::kOffX1;
  uint8_t* sX2 = smem + L::kOffX2;
  uint8_t* sY1 = smem + L::kOffY1;
  uint8_t* sY2 = smem + L::kOffY2;
  float* sLse = reinterpret_cast<float*>(smem + L::kOffLse);
  float* sDelta = reinterpret_cast<float*>(smem + L::kOffDelta);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* x_full = bars + kBarXFull;
  uint64_t* y1_full = bars + kBarY1Full;
  uint64_t* y1_empty = bars + kBarY1Empty;
  uint64_t* y2_full = bars + kBarY2Full;
  uint64_t* y2_empty = bars + kBarY2Empty;
  uint64_t* s_full = bars + kBarSFull;
  uint64_t* s_free = bars + kBarSFree;
  uint64_t* dp_full = bars + kBarDpFull;
  uint64_t* dp_free = bars + kBarDpFree;
  uint64_t* p_ready = bars + kBarPReady;
  uint64_t* p_free = bars + kBarPFree;
  uint64_t* ds_ready = bars + kBarDsReady;
  uint64_t* ds_free = bars + kBarDsFree;
  uint64_t* s_issued = bars + kBarSIssued;
  uint64_t* acc_done = bars + kBarAccDone;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 8);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const AbortState ab{abort_flag, p.status};
  if constexpr (kBits) pdl_wait();   // the tile bitmaps are read right away
  const int nq = (p.seq_q + T - 1) / T, nk = (p.seq_kv + T - 1) / T;
  // The streamed tiles are those the band q_idx - left <= kv_idx <= q_idx + right lets the resident tile meet: KV tiles
  // [j0, j0 + n_iter) for a query tile; for a KV tile the query tiles [i0, i0 + per_head) of every query head of its
  // group, head after head.  (No mask: both sides open; causal: left open, right 0.)
  const long long r0 = static_cast<long long>(tile) * T, r1 = r0 + T - 1;   // rows of the resident tile
  const int i0 = static_cast<int>(max(r0 - p.mask_right, 0LL) / T);
  const int i1 = static_cast<int>(min(static_cast<long long>(nq) - 1, (r1 + p.mask_left) / T));
  const int j0 = static_cast<int>(max(r0 - p.mask_left, 0LL) / T);
  const int j1 = static_cast<int>(min(static_cast<long long>(nk) - 1, (r1 + p.mask_right) / T));
  // with keep bits and a tile bitmap: the tiles whose bit is set in this tile's row of the bitmap
  const bool walk_tiles = kBits && p.tiles_q != nullptr;
  const uint32_t* tiles_row = !walk_tiles ? nullptr
                              : kRoleQ  ? p.tiles_q + static_cast<long long>(tile) * p.tile_words_k
                                        : p.tiles_kv + static_cast<long long>(tile) * p.tile_words_q;
  const int tiles_words = kRoleQ ? p.tile_words_k : p.tile_words_q;
  const int n_kept = walk_tiles ? KeptTiles(tiles_row, tiles_words).count() : 0;
  const int per_head = kRoleQ ? 0 : (walk_tiles ? n_kept : max(i1 - i0 + 1, 0));
  const int n_iter = kRoleQ ? (walk_tiles ? n_kept : max(j1 - j0 + 1, 0)) : p.kv_group * per_head;

  if (tid == 0) {
    *abort_flag = 0;
    // the operand tiles use the 128-byte swizzle, whose pattern repeats every 1024 bytes of the shared window
    if ((smem_u32(smem) & 1023u) != 0) {
      *abort_flag = 1;
      atomicCAS(p.status, 0, kStatusTimeoutBase + kBwdSmemAlign);
    }
    pdl_wait();
    if (*reinterpret_cast<volatile int*>(p.status) != 0) *abort_flag = 1;
  }
  // Loads.  The loading warp sets the barriers up and sends the resident pair and the first streamed pair off at once, under
  // the tensor-memory allocation and the CTA-wide sync.  (If the status word turns out set nobody takes them, and the
  // teardown below gives them time to land.)
  auto load_y1 = [&](int it, int ys, int hq) {   // streamed tile: row offset and head in the tensors it comes from
    const int st = it % N1;
    mbar_arrive_expect_tx(y1_full + st, L::kTileBytes + ((!kRoleQ && F::kUsesStats) ? L::kStatBytes : 0));
    for (int c = 0; c < KC; ++c)
      tma_load_rows(sY1 + st * L::kTileBytes + c * L::kChunkBytes, kRoleQ ? &tmK : &tmQ, y1_full + st, c * 64, ys * T, hq, b, kRoleQ ? p.ok : p.oq);
    if constexpr (!kRoleQ && F::kUsesStats)
      bulk_load(sLse + st * T, p.lse2 + (static_cast<long long>(b) * p.heads + hq) * p.seq_q_pad + ys * T, L::kStatBytes, y1_full + st);
  };
  auto load_y2 = [&](int it, int ys, int hq) {
    const int st = it % N2;
    mbar_arrive_expect_tx(y2_full + st, L::kTileBytes + ((!kRoleQ && F::kUsesStats) ? L::kStatBytes : 0));
    for (int c = 0; c < KC; ++c)
      tma_load_rows(sY2 + st * L::kTileBytes + c * L::kChunkBytes, kRoleQ ? &tmV : &tmDO, y2_full + st, c * 64, ys * T, hq, b, kRoleQ ? p.ov : p.odo);
    if constexpr (!kRoleQ && F::kUsesStats)
      bulk_load(sDelta + st * T, p.delta + (static_cast<long long>(b) * p.heads + hq) * p.seq_q_pad + ys * T, L::kStatBytes, y2_full + st);
  };
  KeptTiles load_walk(tiles_row, tiles_words);
  if (warp == kRowWarps) {
    static_assert(kNumBwdBarriers <= 32, "a barrier for each lane");
    const bool rows = lane == kBarSFree || lane == kBarDpFree || lane == kBarPReady || lane == kBarDsReady || lane == kBarDsReady + 1;
    if (lane < kNumBwdBarriers) mbar_init(bars + lane, rows ? kRowWarps : 1);
    fence_barrier_init();
    __syncwarp();
    if (lane == 0 && n_iter > 0) {
      pdl_wait();
      mbar_arrive_expect_tx(x_full, 2 * L::kTileBytes);
      for (int c = 0; c < KC; ++c) {
        tma_load_rows(sX1 + c * L::kChunkBytes, kRoleQ ? &tmQ : &tmK, x_full, c * 64, tile * T, hx, b, kRoleQ ? p.oq : p.ok);
        tma_load_rows(sX2 + c * L::kChunkBytes, kRoleQ ? &tmDO : &tmV, x_full, c * 64, tile * T, hx, b, kRoleQ ? p.odo : p.ov);
      }
      const int ys = walk_tiles ? load_walk.next() : (kRoleQ ? j0 : i0), hq = kRoleQ ? hx / p.kv_group : hx * p.kv_group;
      load_y1(0, ys, hq);
      load_y2(0, ys, hq);
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
    pdl_launch_dependents();   // behind the allocation: see sm100.cuh
  }
  pdl_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const bool start_ok = warp_all(!*abort_flag);

  if (warp == kRowWarps) {
    // ======================= loading warp =======================
    if (lane == 0 && start_ok && n_iter > 0) {
      for (int it = 1; it < n_iter; ++it) {
        const int ys = walk_tiles ? load_walk.next() : (kRoleQ ? j0 + it : i0 + it % max(per_head, 1));   // the streamed tile
        const int hq = kRoleQ ? hx / p.kv_group : hx * p.kv_group + it / max(per_head, 1);
        if (!mbar_wait(y1_empty + it % N1, ((it / N1) & 1) ^ 1, ab, kBwdYEmpty)) break;
        load_y1(it, ys, hq);
        if (!mbar_wait(y2_empty + it % N2, ((it / N2) & 1) ^ 1, ab, kBwdYEmpty)) break;
        load_y2(it, ys, hq);
      }
    }
  } else if (warp > kRowWarps) {
    // ======================= issuing warps: one for S and dP, one for the accumulators =======================
    // Each runs its loop converged and one elected lane issues a batch of MMAs with its commits: the descriptors then live
    // in uniform registers, and a batch leaves at the pipe's rate whatever the row warps do (issued from inside an
    // `if (lane == 0)` region an MMA with N = 128 took ~90 cycles under load, against the 64 the pipe needs for it).  Two
    // warps, because a batch occupies its warp until the pipe has nearly done with it: what one warp does between its
    // batches is covered by the other's.
    if (__all_sync(0xffffffffu, start_ok) && n_iter > 0) {
      constexpr uint64_t kChunk = L::kChunkBytes >> 4;
      auto wait = [&](uint64_t* bar, uint32_t parity, int site) -> bool {
        return __all_sync(0xffffffffu, mbar_wait_poll(bar, parity, ab, site));
      };
      if (warp == kRowWarps + 1) {
        constexpr uint32_t idesc_kk = make_idesc_f16(T, T, kBf16, false, false);      // both operands K-major
        const uint64_t x1_desc = make_smem_desc(smem_u32(sX1), 16, 1024), x2_desc = make_smem_desc(smem_u32(sX2), 16, 1024);
        // out = X Y^T, then up to two commits
        auto issue_xy = [&](uint32_t out_col, uint64_t x_desc, const uint8_t* y_tile, uint64_t* c1, uint64_t* c2) {
          tc_fence_after_sync();
          const uint64_t y_desc = make_smem_desc(smem_u32(y_tile), 16, 1024);
          if (elect_one()) {
#pragma unroll
            for (int ch = 0; ch < KC; ++ch)
              umma_ss_x4<2, 2>(tmem_base + out_col, x_desc + ch * kChunk, y_desc + ch * kChunk, idesc_kk, ch > 0 ? 1u : 0u);
            umma_commit(c1);
            if (c2 != nullptr) umma_commit(c2);
          }
        };
        bool ok = wait(x_full, 0, kBwdXFull);
        for (int it = 0; ok && it < n_iter; ++it) {
          const int s1 = it % N1, s2 = it % N2;
          if (!wait(y1_full + s1, (it / N1) & 1, kBwdYFull)) break;
          // the buffer's last contents are in the row threads' registers.  The row threads learn from s_full and dp_full
          // what else they need for a tile (every barrier that they look at costs them 50-200 cycles behind their
          // exponentials): query role: dS's buffer has been read; KV role: the statistics have arrived.  They came by bulk
          // copies on the tiles' barriers, which this warp waits for and the row threads do not: that the row threads see them
          // rests on this wait, the commit behind it and their own wait for that commit.
          if (it > 0 && !(kShared ? wait(dp_free, (it - 1) & 1, kBwdDpFree) : wait(s_free, (it - 1) & 1, kBwdSFree))) break;
          issue_xy(kColS, x1_desc, sY1 + s1 * L::kTileBytes, s_full, nullptr);
          if (kShared && it > 0 && lane == 0) mbar_arrive(s_issued);
          if (!wait(y2_full + s2, (it / N2) & 1, kBwdYFull)) break;
          if constexpr (kShared) ok = wait(s_free, it & 1, kBwdSFree);
          else ok = it == 0 || wait(dp_free, (it - 1) & 1, kBwdDpFree);
          if (kRoleQ && ok && it >= 2) ok = wait(ds_free + (it & 1), ((it >> 1) - 1) & 1, kBwdDsFree);
          if (!ok) break;
          issue_xy(kColDP, x2_desc, sY2 + s2 * L::kTileBytes, dp_full, kRoleQ ? y2_empty + s2 : nullptr);   // V is read by dP only
        }
      } else {
        constexpr uint32_t idesc_mn = make_idesc_f16(T, D, kBf16, false, true);       // B = streamed tile, MN-major
        // acc += A (16-bit, tensor memory columns a_col...) x streamed tile (MN-major), then up to three commits; c0 is
        // for what was issued before this batch
        auto issue_acc = [&](uint32_t acc_col, uint32_t a_col, const uint8_t* y_tile, bool accumulate, uint64_t* c0, uint64_t* c1, uint64_t* c2,
                             uint64_t* c3) {
          tc_fence_after_sync();
          const uint64_t y_mn = make_smem_desc(smem_u32(y_tile), L::kChunkBytes, 1024);
          if (elect_one()) {
            if (c0 != nullptr) umma_commit(c0);
#pragma unroll
            for (int g = 0; g < T / 64; ++g)
              umma_ts_x4<8, 128>(tmem_base + acc_col, tmem_base + a_col + g * 32, y_mn + g * 512, idesc_mn, (accumulate || g > 0) ? 1u : 0u);
            umma_commit(c1);
            if (c2 != nullptr) umma_commit(c2);
            if (c3 != nullptr) umma_commit(c3);
          }
        };
        for (int it = 0; it < n_iter; ++it) {
          const int s1 = it % N1, s2 = it % N2;
          uint64_t* last = it + 1 == n_iter ? acc_done : nullptr;
          if (!wait(y1_full + s1, (it / N1) & 1, kBwdYFull)) break;
          if constexpr (kRoleQ) {
            if (!wait(ds_ready + (it & 1), (it >> 1) & 1, kBwdDsReady)) break;
            issue_acc(kColA, kColDS + (it & 1) * 64, sY1 + s1 * L::kTileBytes, it > 0, nullptr, ds_free + (it & 1), y1_empty + s1, last);   // dQ += dS K
          } else {
            if (!wait(y2_full + s2, (it / N2) & 1, kBwdYFull)) break;
            if (!wait(p_ready, it & 1, kBwdPReady)) break;
            // Where S waits for the buffer that dP was taken from, the row threads wait for S while dV would do a tile later
            // as well: it queues up behind S (in front of it: 3300 cycles a tile)
            if (kShared && it + 1 < n_iter && !wait(s_issued, it & 1, kBwdSIssued)) break;
            issue_acc(kColA, kColP, sY2 + s2 * L::kTileBytes, it > 0, nullptr, p_free, nullptr, nullptr);    // dV += P^T dO
            if (!wait(ds_ready, it & 1, kBwdDsReady)) break;
            // dO(it) has been read by dP(it) and, behind this commit, by dV(it); its stage also holds delta(it), which
            // the row threads have now used
            issue_acc(kColB, kColDS, sY1 + s1 * L::kTileBytes, it > 0, y2_empty + s2, ds_free, y1_empty + s1, last);   // dK += dS^T Q
          }
        }
      }
    }
  } else {
    // ======================= row threads: one TMEM lane each, C columns =======================
    const int wq = warp & 3, wg = warp >> 2;
    const int row = wq * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tS = tmem_base + lane_base + kColS, tDP = tmem_base + lane_base + kColDP;
    const uint32_t tP = tmem_base + lane_base + kColP, tDS = tmem_base + lane_base + kColDS;
    const typename F::Ctx fctx = F::make(p);
    float lse2_r = 0.0f, delta_r = 0.0f;
    if constexpr (kRoleQ && F::kUsesStats) {
      const long long idx = (static_cast<long long>(b) * p.heads + hx) * p.seq_q_pad + tile * T + row;
      lse2_r = p.lse2[idx];
      delta_r = p.delta[idx];
    }
    // P and g of one element.  KV role: lanes are KV rows, columns query rows; query role the other way round.  The
    // band and the sequence's end keep, for this thread's row, the columns [col_lo, col_hi] of the tile (set per streamed
    // tile; everything when neither crosses the pair); a functor whose P vanishes at a score of -inf (softmax) gets the mask
    // through the score
    int col_lo = 0, col_hi = T;   // counted from this thread's first column
    uint32_t keep_bits = 0;       // kBits: this thread's part of its row of the streamed tile
    auto score_of = [&](auto edge_tile, float s, float l2, int ys, int hq, int k, float& pr, float& g) {
      const int col = wg * C + k;
      const int q_idx = kRoleQ ? tile * T + row : ys * T + col;
      const int kv_idx = kRoleQ ? ys * T + col : tile * T + row;
      bool masked;
      if constexpr (kBits) {
        masked = ((keep_bits >> k) & 1u) == 0u;
      } else {
        masked = decltype(edge_tile)::value && (k < col_lo || k > col_hi);
      }
      F::score((F::kNegInfMask && masked) ? -INFINITY : s, l2, fctx, b, hq, q_idx, kv_idx, pr, g);
      if (!F::kNegInfMask && masked) pr = g = 0.0f;
    };
    // KV role: the statistics belong to the columns and sit in shared memory; every lane reads the same four at a time
    auto stat_of = [&](const float* base, int k) -> float {
      const float4 v4 = *reinterpret_cast<const float4*>(base + (k & ~3));
      return (k & 3) == 0 ? v4.x : (k & 3) == 1 ? v4.y : (k & 3) == 2 ? v4.z : v4.w;
    };
    KeptTiles kept(tiles_row, tiles_words);
    int next_i = 0, next_hq = kRoleQ ? hx : hx * p.kv_group;   // without a division per tile: rows are the serial chain
    for (int it = 0; start_ok && it < n_iter; ++it) {
      // the streamed tile index, its query head, and whether an edge of the band crosses this pair of tiles
      const int ys = walk_tiles ? kept.next() : (kRoleQ ? j0 : i0) + next_i;
      const int hq = next_hq;
      if (++next_i == per_head && !kRoleQ) {
        next_i = 0;
        ++next_hq;
      }
      // Pairs of tiles that an edge of the band crosses take a second copy of the row loops, with the mask: the row
      // phases sit on the kernel's serial chain, and two compares per element on every tile cost 15 %
      const int kv_minus_q = (kRoleQ ? ys - tile : tile - ys) * T;   // of the tiles' first rows
      // So does a tile that the sequence ends in, where its columns past the end would not come out as zeros: their score is 0
      // (zero rows), and dS there is exp(-lse) times a finite value, which a row of strongly negative logits makes infinite --
      // infinity times the zero rows of K is NaN for the whole row of dQ.  (Query rows past the end have lse = +inf; without
      // statistics theirs are such columns too, where P or its derivative may be anything at a score of 0.)
      const int col_last = (kRoleQ ? p.seq_kv : p.seq_q) - 1 - ys * T;
      const bool tail = (F::kUsesStats ? kRoleQ : !F::kFiniteTail) && col_last < T - 1;
      const bool edge = kBits || tail || kv_minus_q + T - 1 > p.mask_right || kv_minus_q - (T - 1) < -p.mask_left;
      if constexpr (kBits) {
        const uint32_t* bits = kRoleQ ? p.bits_q : p.bits_kv;
        const long long pitch = 4LL * (kRoleQ ? nk : nq);   // words per row: four per streamed tile
        keep_bits = bits[(static_cast<long long>(tile) * T + row) * pitch + 4LL * ys + wg];
      } else if (edge) {
        // kv - q of (row, col) is base + col (query role) or base - col (KV role); kept where -left <= kv - q <= right
        const long long base = kRoleQ ? kv_minus_q - row : kv_minus_q + row;
        const long long lo = kRoleQ ? -static_cast<long long>(p.mask_left) - base : base - p.mask_right;
        const long long hi = kRoleQ ? static_cast<long long>(p.mask_right) - base : base + p.mask_left;
        col_lo = static_cast<int>(max(lo, 0LL)) - wg * C;
        col_hi = static_cast<int>(min(hi, static_cast<long long>(tail ? col_last : T))) - wg * C;
      }
      // this thread's columns of S or dP to registers, their buffer free behind them
      auto take = [&](uint32_t taddr, uint64_t* free_bar, float (&x)[C]) {
        tc_fence_after_sync();
        tmem_ld32f(taddr + wg * C, x);
        tmem_wait_ld();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(free_bar);
      };
      auto hand_over = [&](uint32_t taddr, const float (&x)[C], uint64_t* ready_bar) {   // as 16-bit pairs
        uint32_t pk[C / 2];
#pragma unroll
        for (int k = 0; k < C / 2; ++k) pk[k] = pack2<kBf16>(x[2 * k], x[2 * k + 1]);
        tmem_st16(taddr + wg * (C / 2), pk);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(ready_bar);
      };
      static_assert(C == 32, "one tensor-memory load and one store of a row's part, one word of its keep bits");
      mbar_wait_rows(s_full, it & 1, ab, kBwdSFull);
      // the statistics of the query rows: this thread's own (query role) or those of its columns, which came with the tiles
      const float* st_lse = sLse + (it % N1) * T + wg * C;
      const float* st_delta = sDelta + (it % N2) * T + wg * C;
      float s[C], g[C];
      take(tS, s_free, s);
      auto probabilities = [&](auto edge_tile) {
#pragma unroll
        for (int k = 0; k < C; ++k) {
          float pr;
          score_of(edge_tile, s[k], kRoleQ ? lse2_r : F::kUsesStats ? stat_of(st_lse, k) : 0.0f, ys, hq, k, pr, g[k]);
          s[k] = pr;
        }
      };
      if (edge) {
        probabilities(std::true_type{});
      } else {
        if constexpr (F::kUsesStats) F::template score_row<C, !kRoleQ>(s, g, kRoleQ ? &lse2_r : st_lse, fctx);
        else probabilities(std::false_type{});
      }
      if constexpr (!kRoleQ) {
        if (it > 0) {   // dV of the last tile has read its P
          mbar_wait_rows(p_free, (it - 1) & 1, ab, kBwdPFree);
          tc_fence_after_sync();
        }
        hand_over(tP, s, p_ready);
      }
      // ---- dP -> dS ----
      mbar_wait_rows(dp_full, it & 1, ab, kBwdDpFull);
      take(tDP, dp_free, s);
      if constexpr (F::kUsesStats) {
        F::template grad_row<C, !kRoleQ>(g, s, kRoleQ ? &delta_r : st_delta);
      } else {
#pragma unroll
        for (int k = 0; k < C; ++k) s[k] = F::grad(g[k], s[k], fctx);
      }
      if (!kRoleQ && it > 0) {   // dK of the last tile has read its dS
        mbar_wait_rows(ds_free, (it - 1) & 1, ab, kBwdDsFree);
        tc_fence_after_sync();
      }
      const int ds_buf = kRoleQ ? it & 1 : 0;
      hand_over(tDS + ds_buf * 64, s, ds_ready + ds_buf);
    }
    // ---- epilogue: the accumulators as 16-bit rows (dK and dQ times the functor's constant factor) ----
    if (n_iter > 0) {
      mbar_wait_rows(acc_done, 0, ab, kBwdAccDone);
      tc_fence_after_sync();
    }
    if (warp_all(!*abort_flag)) {
      const int r = tile * T + row;
      const int n_out = kRoleQ ? 1 : 2;
      for (int a = 0; a < n_out; ++a) {
        // a = 0: dQ (query role) or dV; a = 1: dK
        uint16_t* base;
        if constexpr (kRoleQ) {
          base = static_cast<uint16_t*>(p.dq) + b * p.dq_s[0] + static_cast<long long>(r) * p.dq_s[1] + hx * p.dq_s[2];
        } else {
          const long long* sd = a == 0 ? p.dv_s : p.dk_s;
          base = static_cast<uint16_t*>(a == 0 ? p.dv : p.dk) + b * sd[0] + static_cast<long long>(r) * sd[1] + hx * sd[2];
        }
        const float f = (kRoleQ || a == 1) ? F::out_scale(fctx) : 1.0f;
        const bool in_range = r < (kRoleQ ? p.seq_q : p.seq_kv);
#pragma unroll
        for (int u = 0; u < AC / 16; ++u) {
          const int c0 = wg * AC + u * 16;
          float v[16];
          if (n_iter > 0) {
            tmem_ld16f(tmem_base + lane_base + (a == 0 ? kColA : kColB) + c0, v);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] = 0.0f;
          }
          if (in_range) {
            uint4* dst = reinterpret_cast<uint4*>(base + c0);
#pragma unroll
            for (int q4 = 0; q4 < 2; ++q4) {
              uint4 pk;
              pk.x = pack2<kBf16>(v[8 * q4 + 0] * f, v[8 * q4 + 1] * f);
              pk.y = pack2<kBf16>(v[8 * q4 + 2] * f, v[8 * q4 + 3] * f);
              pk.z = pack2<kBf16>(v[8 * q4 + 4] * f, v[8 * q4 + 5] * f);
              pk.w = pack2<kBf16>(v[8 * q4 + 6] * f, v[8 * q4 + 7] * f);
              dst[q4] = pk;
            }
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Both roles in one launch, the CTAs of the KV role (the longer ones) first: those of the query role fill the SMs that the
// last of them leave idle, which two launches one after the other could not.  Training step of 2 x 16 / 4 x 1111 x 64 with
// a window (72 CTAs of 28 us and 288 of 6): 94 -> 84 us; 4 x 32 x 4096 x 128 causal: unchanged (2.82 ms).
template <class F, bool kBf16, int D, bool kBits>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ BwdParams p) {
  const int nq = (p.seq_q + kBwdT - 1) / kBwdT, nk = (p.seq_kv + kBwdT - 1) / kBwdT;
  const int n_kv_ctas = nk * p.heads_kv * p.batch;
  const int i = static_cast<int>(blockIdx.x);
  // the longest first: a causal KV tile meets the more query tiles the earlier it lies, a query tile the fewer KV tiles
  if (i < n_kv_ctas) {
    int tile, pair;
    heavy_order(i, nk, p.heads_kv * p.batch, max(p.heads_at_once / p.kv_group, 1), tile, pair);
    attn_bwd_cta<F, false, kBf16, D, kBits>(tmQ, tmK, tmV, tmDO, p, tile, pair % p.heads_kv, pair / p.heads_kv);
  } else {
    int tile, pair;
    heavy_order(i - n_kv_ctas, nq, p.heads * p.batch, max(p.heads_at_once, 1), tile, pair);
    attn_bwd_cta<F, true, kBf16, D, kBits>(tmQ, tmK, tmV, tmDO, p, nq - 1 - tile, pair % p.heads, pair / p.heads);
  }
}

// What a backward launch needs beside the functor: filled from the C-ABI argument structs.
struct BwdCall {
  const void *q, *k, *v, *d_o;
  void *dq, *dk, *dv;
  int batch, heads, heads_kv, seq_q, seq_kv, dim, dtype, mask_left, mask_right;
  float scale;
  const int64_t *q_stride, *k_stride, *v_stride, *do_stride, *dq_stride, *dk_stride, *dv_stride;
  const float* lse2;
  const float* delta;
  const void* const* custom;
  const uint32_t *bits_q, *bits_kv;   // both or neither: keep bits of a general mask (the band then has to be open)
  const uint32_t *tiles_q, *tiles_kv; // with the bits, optional (both or neither): bitmaps of the tiles that keep anything
};

// One CTA per KV tile and KV head (dK, dV) and one per query tile and head (dQ) for functor F.
template <class F, bool kBf16, int D>
int launch_attn_bwd(const BwdCall& a, cudaStream_t stream, int* status) {
  using L = BwdSmem<D>;
  const int T = kBwdT;
  const int nq = (a.seq_q + T - 1) / T, nk = (a.seq_kv + T - 1) / T;
  CUtensorMap tmQ, tmK, tmV, tmDO;
  BwdParams p;
  std::memset(&p, 0, sizeof(p));
  int rc = encode_rows_map(&tmQ, &p.oq, a.q, a.dtype, D, a.batch, a.seq_q, a.heads, a.q_stride, T);
  if (rc != ATTN_B200_OK) return rc;
  rc = encode_rows_map(&tmK, &p.ok, a.k, a.dtype, D, a.batch, a.seq_kv, a.heads_kv, a.k_stride, T);
  if (rc != ATTN_B200_OK) return rc;
  rc = encode_rows_map(&tmV, &p.ov, a.v, a.dtype, D, a.batch, a.seq_kv, a.heads_kv, a.v_stride, T);
  if (rc != ATTN_B200_OK) return rc;
  rc = encode_rows_map(&tmDO, &p.odo, a.d_o, a.dtype, D, a.batch, a.seq_q, a.heads, a.do_stride, T);
  if (rc != ATTN_B200_OK) return rc;
  p.dq = a.dq;
  p.dk = a.dk;
  p.dv = a.dv;
  p.lse2 = a.lse2;
  p.delta = a.delta;
  p.batch = a.batch;
  p.heads = a.heads;
  p.heads_kv = a.heads_kv;
  p.kv_group = a.heads / a.heads_kv;
  p.seq_q = a.seq_q;
  p.seq_kv = a.seq_kv;
  p.seq_q_pad = nq * T;
  p.mask_left = a.mask_left;
  p.mask_right = a.mask_right;
  p.bits_q = a.bits_q;
  p.bits_kv = a.bits_kv;
  p.tiles_q = a.bits_q != nullptr ? a.tiles_q : nullptr;
  p.tiles_kv = a.bits_q != nullptr ? a.tiles_kv : nullptr;
  p.tile_words_k = (nk + 31) / 32;
  p.tile_words_q = (nq + 31) / 32;
  p.scale = a.scale;
  for (int i = 0; i < 3; ++i) {
    p.dq_s[i] = a.dq_stride[i];
    p.dk_s[i] = a.dk_stride[i];
    p.dv_s[i] = a.dv_stride[i];
  }
  for (int i = 0; i < ATTN_B200_MAX_CUSTOM; ++i) p.custom[i] = a.custom != nullptr ? a.custom[i] : nullptr;
  p.status = status;
  const bool with_bits = a.bits_q != nullptr;
  if (a.mask_left >= ATTN_B200_MASK_OPEN && a.mask_right == 0)
    p.heads_at_once = heavy_heads_at_once(static_cast<long long>(a.seq_q) * D * 4, static_cast<long long>(a.batch) * a.heads);
  auto kernel = with_bits ? attn_bwd_kernel<F, kBf16, D, true> : attn_bwd_kernel<F, kBf16, D, false>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes) != cudaSuccess) {
    cudaGetLastError();
    return ATTN_B200_E_LAUNCH;
  }
  const long long ctas = (static_cast<long long>(nk) * a.heads_kv + static_cast<long long>(nq) * a.heads) * a.batch;
  if (ctas > 0x7fffffffLL) return ATTN_B200_E_UNSUPPORTED;
  if (!launch_pdl(kernel, dim3(static_cast<unsigned>(ctas)), dim3(kBwdThreads), L::kBytes, stream, tmQ, tmK, tmV, tmDO, p)) return ATTN_B200_E_LAUNCH;
  return ATTN_B200_OK;
}

// mask_kind, the band and the keep bits of an argument struct as the mask of a call; false = not a mask the backward covers
inline bool bwd_mask_of(int mask_kind, int left, int right, const void* bits_q, const void* bits_kv, const void* tiles_q,
                        const void* tiles_kv, BwdCall& call) {
  call.bits_q = call.bits_kv = call.tiles_q = call.tiles_kv = nullptr;
  if (mask_kind == ATTN_B200_MASK_BITS) {
    if (bits_q == nullptr || bits_kv == nullptr) return false;
    if ((tiles_q == nullptr) != (tiles_kv == nullptr)) return false;
    call.tiles_q = static_cast<const uint32_t*>(tiles_q);
    call.tiles_kv = static_cast<const uint32_t*>(tiles_kv);
    if (((reinterpret_cast<uintptr_t>(bits_q) | reinterpret_cast<uintptr_t>(bits_kv)) & 15) != 0) return false;
    call.bits_q = static_cast<const uint32_t*>(bits_q);
    call.bits_kv = static_cast<const uint32_t*>(bits_kv);
    call.mask_left = call.mask_right = ATTN_B200_MASK_OPEN;
  } else if (mask_kind == ATTN_B200_MASK_NONE) {
    call.mask_left = call.mask_right = ATTN_B200_MASK_OPEN;
  } else if (mask_kind == ATTN_B200_MASK_CAUSAL) {
    call.mask_left = ATTN_B200_MASK_OPEN;
    call.mask_right = 0;
  } else if (mask_kind == ATTN_B200_MASK_BAND) {
    if (left < 0 || right < 0 || left > ATTN_B200_MASK_OPEN || right > ATTN_B200_MASK_OPEN) return false;
    call.mask_left = left;
    call.mask_right = right;
  } else {
    return false;
  }
  return true;
}

// Checks shared by every backward entry point (pointers, dims, strides, alignment of the outputs).
inline int validate_bwd_call(const BwdCall& a) {
  if (a.q == nullptr || a.k == nullptr || a.v == nullptr || a.d_o == nullptr || a.dq == nullptr || a.dk == nullptr || a.dv == nullptr)
    return ATTN_B200_E_INVALID_ARG;
  if (a.batch <= 0 || a.heads <= 0 || a.seq_q <= 0 || a.seq_kv <= 0) return ATTN_B200_E_INVALID_ARG;
  if (a.dtype != ATTN_B200_DTYPE_FP16 && a.dtype != ATTN_B200_DTYPE_BF16) return ATTN_B200_E_INVALID_ARG;
  if (a.heads_kv <= 0 || a.heads % a.heads_kv != 0) return ATTN_B200_E_INVALID_ARG;
  if (a.dim != 64 && a.dim != 128) return ATTN_B200_E_UNSUPPORTED;
  if (a.batch > 65535 || a.heads > 65535) return ATTN_B200_E_UNSUPPORTED;
  const void* outs[3] = {a.dq, a.dk, a.dv};
  const int64_t* strides[3] = {a.dq_stride, a.dk_stride, a.dv_stride};
  for (int i = 0; i < 3; ++i) {
    if ((reinterpret_cast<uintptr_t>(outs[i]) & 15) != 0) return ATTN_B200_E_UNSUPPORTED;
    for (int d = 0; d < 3; ++d)
      if (strides[i][d] % 8 != 0) return ATTN_B200_E_UNSUPPORTED;
  }
  return ATTN_B200_OK;
}

}  // namespace b200
