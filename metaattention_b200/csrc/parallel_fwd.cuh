// Kernel family (1): parallel-pattern attention forward for sm_100a.
//
//   O = epilogue( sum over KV tiles of  o_scale-rescaled  P.V ),
//   P = online_fwd( score_mod( mask + Q.K^T ) )
//
// with score_mod / online_fwd / epilogue supplied by a device functor F (the
// lowered form of the user's score_mod and OnlineFunc).  Replaces the
// generated TileLang kernel of the reference
// (attention_engine/core/template/tl_template/attn/attn_tl.py:93-190) and its
// CuTe warp-specialised forward (core/template/cute_template/flash_fwd_kernel.h:28-199).
//
// One CTA owns two 128-row query tiles (NT; one for the widest heads) of one (batch, head) and walks the KV
// sequence in 128-row tiles.  Warps, with RT threads to a query row (two where the functor allows it):
//   4 RT per query tile   functor stage: scores from tensor memory to registers, P back to tensor memory
//   1                     loads of Q and K (TMA rings), 1 loads of V
//   1                     issues S = Q_t.K^T (tcgen05.mma), 1 issues O_t += P_t.V with P_t read from tensor memory
// What bounds it is the functor stage: 128 x 128 exponentials are 1024 cycles of the special-function unit, and both
// tiles' together equal the 2048 cycles of their MMAs.  So the functor warps never wait for each other's tile or for the
// pipe: P has columns of its own, and a score tile leaves its buffer for registers as soon as it is there, so the
// next one (the other tile's, where there is one buffer) is computed under the exponentials; the four service warps wait
// for nothing but their own operands (one warp that issued both products in turn: 4950 cycles for a step of both tiles
// against 3300, its barriers and bookkeeping of 400-600 cycles a product standing in front of an idle pipe).  With P
// written over its own scores (so that a tile's chain functor -> P.V -> Q.K^T was serial), 192 / 128 causal
// 2 x 16 x 3000 took 154 us, now 124; sigmoid 2 x 32 x 4096 523, now 488; causal 8 x 32 x 4096 1216, now 1157 (at its power cap).
// Two threads to a row (16 functor warps, four to a scheduler) against one: causal 6 x 8 x 965 33 us against 34-37, long
// calls 2 % slower for softmax and sigmoid alike.
// Tensor memory: O0 O1 (DV columns each), P0 P1 (64 each), then one or two score buffers (128 each).
// Masks are bands kv_idx in [q_idx - left, q_idx + right] (none / causal / explicit bounds): a query tile
// walks only the KV tiles its band touches, the CTA loads the union of its two tiles' ranges, and tiles
// that cross an edge of the band are masked element by element.  K/V heads may be shared by groups of
// query heads (kv_group).  The same kernel serves q_len != kv_len (decode patterns).
// Start and end of a CTA: the producer lane initialises the barriers and issues the query tiles and the first K/V
// tiles before the tensor-memory allocation and the CTA-wide sync; the output rows of a tile are staged in its
// query buffer and stored as whole rows.
#pragma once

#include <type_traits>

#include "sm100.cuh"

namespace b200 {

constexpr int kMaxCustom = 4;
constexpr int kNoBound = 0x3fffffff;   // an open side of the mask band
constexpr int kMaxRowScales = 4;

struct FunctorArgs {
  float f[8];
  const void* custom[kMaxCustom];
  long long cstride[kMaxCustom][4];  // element strides of (batch, heads, seq_len, seq_len_kv)
};

// Threads that share a row: two where the functor allows it (it keeps nothing per row, or its row values are a maximum
// that the threads exchange and a sum that is added up at the end; its epilogue works on each accumulator column by itself), so
// that four functor warps run on each scheduler.
template <class F, class = void>
struct functor_split_sum : std::false_type {};
template <class F>
struct functor_split_sum<F, std::void_t<decltype(F::kSplitSum)>> : std::true_type {};
template <class F>
constexpr int kRowThreads = functor_split_sum<F>::value || (F::kRowScales == 0 && F::kUnitOScale && !F::kRowEpilogue) ? 2 : 1;

// What a functor knows about the row it is working on.
struct RowCtx {
  int b, h, q_idx;   // batch, head, query position of this thread's row
  int kv0;           // first KV position of the current tile
  int seq_q, seq_kv;
  const FunctorArgs* fa;
};

// Position (1..3) of the head / sequence / batch coordinate inside a 4-D
// tensor map whose dimension 0 is the feature dimension; the host sorts the
// three outer dimensions by stride.
struct CoordOrder {
  int pos_s, pos_h, pos_b;
};

struct ParallelParams {
  void* o;
  float* final_out[kMaxRowScales];
  int batch, heads, seq_q, seq_kv;
  int kv_group;                // query heads per KV head (1 = one KV head per query head)
  int kv_splits;               // > 1: blockIdx.z = batch * kv_splits + split, each split covers tiles_per_split KV tiles
  int tiles_per_split;
  float* part_o;               // [batch, kv_splits, heads, seq_q, dim_v] fp32 results of the splits (kv_splits > 1)
  float* part_final;           // [kFinal][batch, kv_splits, heads, seq_q] their final row scales
  long long part_final_stride; // elements between two final row scales in part_final
  // Block sparsity (kSparse kernels): per (sparse batch, sparse head, 128-row query tile) a bitmap of the 128-row KV
  // tiles to visit and one of the tiles among them that need the element mask.
  const uint32_t* tile_keep;   // [sparse_batch][sparse_heads][q_tiles][tile_words]
  const uint32_t* tile_partial;
  const int* tile_mask_base;   // [sparse_batch][sparse_heads][q_tiles] first element-mask slot of the query tile, or null
  const uint32_t* elem_mask;   // slots of [elem_mask_rows][4] words (bit = keep), or with elem_mask_rows == 0 one
                               // [4]-word column mask per (sparse batch, sparse head, KV tile)
  int sparse_batch, sparse_heads, tile_words, elem_mask_rows;
  long long o_sb, o_ss, o_sh;  // element strides of o
  int heads_at_once;           // causal: of so many (head, batch) pairs at a time the heaviest query tiles first; 0: of each
  int mask_kind;               // 0 none, 1 causal (keep q_idx >= kv_idx), 2 band
  int win_left, win_right;     // band: keep kv_idx in [q_idx - win_left, q_idx + win_right]; kNoBound = open side
  CoordOrder oq, ok, ov;
  int* status;
  FunctorArgs fa;
};

__device__ __forceinline__ void tma_load_rows(void* dst, const CUtensorMap* tm, uint64_t* bar, int c0, int s, int h,
                                              int b, const CoordOrder& o) {
  const int c1 = (o.pos_s == 1) ? s : (o.pos_h == 1) ? h : b;
  const int c2 = (o.pos_s == 2) ? s : (o.pos_h == 2) ? h : b;
  const int c3 = (o.pos_s == 3) ? s : (o.pos_h == 3) ? h : b;
  tma_load_4d(dst, tm, bar, c0, c1, c2, c3);
}

// The i-th CTA of `pairs` (head, batch) pairs with `tiles` tiles each, taken `at_once` pairs at a time, tile by tile.
__device__ __forceinline__ void heavy_order(int i, int tiles, int pairs, int at_once, int& tile, int& pair) {
  const int group = i / (tiles * at_once), first = group * at_once, n = min(at_once, pairs - first);
  const int r = i - first * tiles;
  tile = r / n;
  pair = first + r - tile * n;
}

// wait-site ids reported through the device status word
enum ParallelWaitSite {
  kSiteQFull = 1, kSiteKFull, kSiteVFull, kSiteKEmpty, kSiteVEmpty, kSiteSFull, kSitePReady, kSiteODone, kSiteOFinal, kSiteSFree, kSiteSmemAlign
};

// Walks the set bits of one bitmap, or of the union of two, in increasing order (KV tile indices of a sparse walk).
struct TileWalk {
  const uint32_t* a;
  const uint32_t* b;
  int words, w;
  uint32_t bits;
  __device__ TileWalk(const uint32_t* a_, const uint32_t* b_, int words_) : a(a_), b(b_), words(words_), w(-1), bits(0) {}
  __device__ int next() {
    while (bits == 0) {
      if (++w >= words) return -1;
      bits = a[w] | (b != nullptr ? b[w] : 0u);
    }
    const int j = w * 32 + __ffs(bits) - 1;
    bits &= bits - 1;
    return j;
  }
};

// four functor warps per query tile and thread of a row, two loading and two issuing warps
template <int NT, int RT>
constexpr int kParallelThreads = (4 * NT * RT + 4) * 32;

constexpr int kMaxTileWords = 128;   // sparse walks: at most 4096 KV tiles (512 k tokens)

// NT = query tiles per CTA: 2 (K/V shared by both tiles, in two stages; with dim_qk = 192 the tiles leave room for one
// stage of V: it is free from the second tile's P.V on and needed again behind the other tile's Q.K^T and functor stage,
// later than its load takes) or 1 (single-staged K/V; the layout that fits dim_qk = 256: one 64 KB query tile, 64 KB
// of K, 32 KB of V)
template <int D, int DV, int NT = 2>
struct ParallelSmem {
  static constexpr int kBM = 128, kBN = 128, kStages = NT == 2 ? 2 : 1, kVStages = NT == 2 && D <= 128 ? 2 : 1;
  static constexpr int kQBytes = kBM * D * 2;
  static constexpr int kKBytes = kBN * D * 2;
  static constexpr int kVBytes = kBN * DV * 2;
  static constexpr int kOffQ = 0;
  static constexpr int kOffK = kOffQ + NT * kQBytes;
  static constexpr int kOffV = kOffK + kStages * kKBytes;
  static constexpr int kOffBar = kOffV + kVStages * kVBytes;
  static constexpr int kNumBars = 2 + 2 * kStages + 2 * kVStages + 8;
  static constexpr int kOffMisc = kOffBar + 8 * kNumBars;
  static constexpr int kOffExchange = kOffMisc + 16;   // row maxima of the two threads of a row: [steps][NT][2][128]
  // one step's only where the tiles leave no room for two: a second barrier then keeps the next step's write off
  static constexpr int kExchangeSteps = NT == 2 && D > 128 ? 1 : 2;
  static constexpr int kOffSparse = kOffExchange + kExchangeSteps * NT * 2 * kBM * 4;     // sparse kernels: keep / partial bitmaps of the two query tiles
  static constexpr int kBytes = kOffSparse;            // the dynamic shared memory is declared 1024-byte aligned
  static constexpr int kBytesSparse = kBytes + 4 * kMaxTileWords * 4;
};

template <class F, int D, int DV, bool kBf16, int NT = 2, bool kSparse = false>
__global__ void __launch_bounds__(kParallelThreads<NT, kRowThreads<F>>, 1)
parallel_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const ParallelParams p) {
  using L = ParallelSmem<D, DV, NT>;
  constexpr int BM = L::kBM, BN = L::kBN, ST = L::kStages, STV = L::kVStages;
  static_assert(D % 64 == 0 && DV % 64 == 0 && DV <= 128 && (D <= 192 || (D <= 256 && NT == 1)), "unsupported head dims");
  static_assert((kSparse ? L::kBytesSparse : L::kBytes) <= 232448, "shared memory layout exceeds an SM");
  // score buffers: one that both query tiles take in turn where the accumulators leave room for no more (dim_v 128),
  // else one per query tile; a CTA with a single query tile takes two in turn
  constexpr int NSB = NT == 2 && DV > 64 ? 1 : 2;
  constexpr uint32_t kTmemCols = 512;
  constexpr uint32_t kColO = 0, kColP = NT * DV, kColS = 512 - NSB * BN;
  static_assert(kColP + NT * (BN / 2) <= kColS, "tensor memory layout");
  constexpr int RT = kRowThreads<F>, TC = BN / RT;   // threads per query row, score columns per thread
  constexpr int kKWarp = 4 * NT * RT, kVWarp = kKWarp + 1, kQkWarp = kKWarp + 2, kPvWarp = kKWarp + 3;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem + L::kOffQ;
  uint8_t* sK = smem + L::kOffK;
  uint8_t* sV = smem + L::kOffV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint64_t* q_full = bars;          // [2] one per query tile
  uint64_t* k_full = bars + 2;
  uint64_t* k_empty = k_full + ST;
  uint64_t* v_full = k_empty + ST;
  uint64_t* v_empty = v_full + STV;
  uint64_t* s_full = v_empty + STV;   // [2] one per query tile; with one query tile one per score buffer
  uint64_t* s_free = s_full + 2;      // [2] one per score buffer: its scores are in registers
  uint64_t* p_ready = s_free + 2;     // [2] one per query tile
  uint64_t* o_done = p_ready + 2;     // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const AbortState ab{abort_flag, p.status};
  if constexpr (kSparse) pdl_wait();   // the bitmaps are read right away

  // Every mask is a band kv_idx in [q_idx - left, q_idx + right]: none = open on both sides, causal = open
  // to the left with right = 0, sliding windows bound the left side as well.
  const bool causal = p.mask_kind == 1;
  const int left = p.mask_kind == 2 ? p.win_left : kNoBound;
  const int right = p.mask_kind == 0 ? kNoBound : (p.mask_kind == 1 ? 0 : p.win_right);
  const bool banded = p.mask_kind != 0;
  // heaviest query tiles (largest KV range under a causal mask) are launched first
  int m_of = blockIdx.x, h = blockIdx.y, z = blockIdx.z;
  if (p.heads_at_once > 0) {
    int pair;
    heavy_order(blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z), gridDim.x, gridDim.y * gridDim.z, p.heads_at_once, m_of, pair);
    z = pair / static_cast<int>(gridDim.y);
    h = pair - z * static_cast<int>(gridDim.y);
  }
  const int m_pair = causal ? gridDim.x - 1 - m_of : m_of;
  const int b = p.kv_splits > 1 ? z / p.kv_splits : z;
  const int split = p.kv_splits > 1 ? z % p.kv_splits : 0;
  const int m0 = m_pair * NT * BM;
  const int n_kv_tiles = (p.seq_kv + BN - 1) / BN;
  // KV tiles [j_lo, j_hi) of each query tile; the CTA walks the union [j_min, j_max)
  int j_lo[2], j_hi[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int row0 = m0 + t * BM;
    j_lo[t] = j_hi[t] = 0;
    if (t < NT && row0 < p.seq_q) {
      j_lo[t] = (left >= kNoBound || row0 <= left) ? 0 : (row0 - left) / BN;
      j_hi[t] = right >= kNoBound ? n_kv_tiles : min(n_kv_tiles, (row0 + BM - 1 + right) / BN + 1);
      if (p.kv_splits > 1) {   // this CTA's share of the KV tiles
        j_lo[t] = max(j_lo[t], split * p.tiles_per_split);
        j_hi[t] = min(j_hi[t], (split + 1) * p.tiles_per_split);
      }
      if (j_hi[t] < j_lo[t]) j_hi[t] = j_lo[t];
    }
  }
  bool act0 = j_hi[0] > j_lo[0], act1 = j_hi[1] > j_lo[1];
  const int j_min = act0 ? (act1 ? min(j_lo[0], j_lo[1]) : j_lo[0]) : j_lo[1];
  const int j_max = max(act0 ? j_hi[0] : 0, act1 ? j_hi[1] : 0);
  int n_max = (act0 || act1) ? j_max - j_min : 0;
  // Sparse walk: the bitmaps of this CTA's two query tiles are copied to shared memory (a query tile past the end of
  // the sequence gets an empty one); n_tiles[t] = KV tiles of tile t, n_max = tiles of the union.
  uint32_t* sp_keep = reinterpret_cast<uint32_t*>(smem + L::kOffSparse);      // [2][kMaxTileWords]
  uint32_t* sp_part = sp_keep + 2 * kMaxTileWords;                           // [2][kMaxTileWords]
  int n_tiles[2] = {0, 0};
  int sp_row[2] = {0, 0};       // index of (sparse batch, sparse head, query tile) for each of the two tiles
  if constexpr (kSparse) {
    const int sb = p.sparse_batch > 1 ? b : 0;
    const int sh = p.sparse_heads <= 1 ? 0 : (p.sparse_heads == p.heads ? h : h / (p.heads / p.sparse_heads));
    const int q_tiles = (p.seq_q + BM - 1) / BM;
    for (int t = 0; t < 2; ++t) {
      const int qt = m_pair * NT + t;
      const bool exists = t < NT && qt < q_tiles;
      sp_row[t] = (sb * p.sparse_heads + sh) * q_tiles + (exists ? qt : 0);
      for (int w = threadIdx.x; w < p.tile_words; w += blockDim.x) {
        sp_keep[t * kMaxTileWords + w] = exists ? p.tile_keep[static_cast<long long>(sp_row[t]) * p.tile_words + w] : 0u;
        sp_part[t * kMaxTileWords + w] = exists ? p.tile_partial[static_cast<long long>(sp_row[t]) * p.tile_words + w] : 0u;
      }
    }
    __syncthreads();
    n_max = 0;
    for (int w = 0; w < p.tile_words; ++w) {
      n_tiles[0] += __popc(sp_keep[w]);
      n_tiles[1] += __popc(sp_keep[kMaxTileWords + w]);
      n_max += __popc(sp_keep[w] | sp_keep[kMaxTileWords + w]);
    }
    act0 = n_tiles[0] > 0;
    act1 = n_tiles[1] > 0;
  }
  auto active = [&](int t, int j) {
    if constexpr (kSparse) return j >= 0 && ((sp_keep[t * kMaxTileWords + (j >> 5)] >> (j & 31)) & 1u) != 0;
    else return t == 0 ? (j >= j_lo[0] && j < j_hi[0]) : (j >= j_lo[1] && j < j_hi[1]);
  };

  // ---------------- setup ----------------
  // The producer lane initialises the barriers and sends off the query tiles and the first K and V tiles at once:
  // their ~2800 cycles of latency start before the tensor-memory allocation and the CTA-wide sync, not after.
  auto load_k_tile = [&](int i, int j) {   // KV tile j into the stage of step i
    const int st = i % ST;
    mbar_arrive_expect_tx(&k_full[st], L::kKBytes);
    for (int c = 0; c < D / 64; ++c)
      tma_load_rows(sK + st * L::kKBytes + c * (BN * 128), &tmK, &k_full[st], c * 64, j * BN, h / p.kv_group, b, p.ok);
  };
  auto load_v_tile = [&](int i, int j) {
    const int st = i % STV;
    mbar_arrive_expect_tx(&v_full[st], L::kVBytes);
    for (int c = 0; c < DV / 64; ++c)
      tma_load_rows(sV + st * L::kVBytes + c * (BN * 128), &tmV, &v_full[st], c * 64, j * BN, h / p.kv_group, b, p.ov);
  };
  auto load_q = [&](int t) {
    mbar_arrive_expect_tx(&q_full[t], L::kQBytes);
    for (int c = 0; c < D / 64; ++c)
      tma_load_rows(sQ + t * L::kQBytes + c * (BM * 128), &tmQ, &q_full[t], c * 64, m0 + t * BM, h, b, p.oq);
  };
  if (warp == kVWarp && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == kKWarp) {   // one barrier a lane
    constexpr int kSFreeBar = 2 + 2 * ST + 2 * STV + 2;   // s_free and p_ready: an arrival from each functor warp of a tile
    if (lane < L::kNumBars) mbar_init(bars + lane, lane >= kSFreeBar && lane < kSFreeBar + 4 ? 4 * RT : 1);
    static_assert(L::kNumBars <= 32, "a barrier for each lane");
    fence_barrier_init();
    __syncwarp();
  }
  if (warp == kKWarp && lane == 0) {
    pdl_wait();
    if (n_max > 0 && !kSparse) {
      // in the order of first use: query tile 0 and K so that its scores can start, then query tile 1, then V
      if (act0) load_q(0);
      load_k_tile(0, j_min);
      if (act1) load_q(1);
      load_v_tile(0, j_min);
    }
  }
  // The device status word (set by a CTA whose wait ran out) is read by another thread meanwhile: a global-memory
  // round trip that the first loads do not wait for.  If it is set, nobody consumes those loads and the teardown
  // below gives them time to land.
  if (threadIdx.x == 0) {
    pdl_wait();
    *abort_flag = (*reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    // the operand tiles use the 128-byte swizzle, whose pattern repeats every 1024 bytes of the shared window
    if ((smem_u32(smem) & 1023u) != 0) {
      *abort_flag = 1;
      atomicCAS(p.status, 0, kStatusTimeoutBase + kSiteSmemAlign);
    }
  }
  if (warp == kQkWarp) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
    pdl_launch_dependents();   // behind the allocation: see sm100.cuh
  }
  pdl_wait();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // the steps of the walk: `body(i, j)` for the i-th KV tile j of the union, until it returns false
  auto for_steps = [&](auto&& body) {
    if constexpr (kSparse) {
      TileWalk walk(sp_keep, sp_keep + kMaxTileWords, p.tile_words);
      for (int i = 0; i < n_max; ++i)
        if (!body(i, walk.next())) break;
    } else {
      for (int i = 0; i < n_max; ++i)
        if (!body(i, j_min + i)) break;
    }
  };
  if (warp == kKWarp) {
    // =============== loads of Q and K ===============
    if (lane == 0 && n_max > 0 && !*abort_flag) {
      for_steps([&](int i, int j) {
        if (i == 0) {
          if constexpr (kSparse) {
            if (act0) load_q(0);
            load_k_tile(0, j);
            if (act1) load_q(1);
          }
          return true;   // otherwise on their way since before the CTA-wide sync
        }
        if (i >= ST && !mbar_wait(&k_empty[i % ST], ((i / ST) & 1) ^ 1, ab, kSiteKEmpty)) return false;
        load_k_tile(i, j);
        return true;
      });
    }
  } else if (warp == kVWarp) {
    // =============== loads of V ===============
    if (lane == 0 && n_max > 0 && !*abort_flag) {
      for_steps([&](int i, int j) {
        if (i == 0 && !kSparse) return true;
        if (i >= STV && !mbar_wait(&v_empty[i % STV], ((i / STV) & 1) ^ 1, ab, kSiteVEmpty)) return false;
        load_v_tile(i, j);
        return true;
      });
    }
  } else if (warp == kQkWarp || warp == kPvWarp) {
    // =============== MMA issuers: one warp for Q.K^T, one for P.V ===============
    // Each warp runs its loop converged; one elected lane issues each batch of MMAs with its commits.  The
    // descriptors then live in uniform registers and a batch leaves at the tensor pipe's rate whatever the functor
    // warps do: issued from inside an `if (lane == 0)` region an MMA with N = 128 took ~90 cycles beside busy warps,
    // against the 64 the pipe needs for it.  A batch occupies its warp until the pipe has nearly done with it, so what
    // a warp does between two batches (barriers, tile bookkeeping: 400-600 cycles beside the functor warps) is time
    // without MMAs unless the other warp's are queued: one warp for both products took 4950 cycles a pair-step.
    if (n_max > 0 && __all_sync(0xffffffffu, !*abort_flag)) {
      auto wait = [&](uint64_t* bar, uint32_t parity, int site) -> bool {
        return __all_sync(0xffffffffu, mbar_wait(bar, parity, ab, site));
      };
      // Descriptors are built once; per MMA only the start-address field moves (units of 16 bytes), and four
      // K steps go out per asm block.
      if (warp == kQkWarp) {
        constexpr uint32_t idesc_qk = make_idesc_f16(BM, BN, kBf16, false, false);
        const uint64_t q_desc0 = make_smem_desc(smem_u32(sQ), 16, 1024);
        const uint64_t k_desc0 = make_smem_desc(smem_u32(sK), 16, 1024);
        int n = 0, own[2] = {0, 0};   // score tiles issued: all, and per query tile
        for_steps([&](int i, int j) {
          const int st = i % ST;
          if (!wait(&k_full[st], (i / ST) & 1, kSiteKFull)) return false;
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            if (!active(t, j)) continue;
            if (own[t] == 0 && !wait(&q_full[t], 0, kSiteQFull)) return false;
            // the scores that were in this buffer before have left it for registers
            const int buf = NSB == 1 ? 0 : (NT == 1 ? n & 1 : t);
            const int use = NSB == 1 ? n : (NT == 1 ? n >> 1 : own[t]);
            if (use > 0 && !wait(&s_free[buf], (use - 1) & 1, kSiteSFree)) return false;
            tc_fence_after_sync();
            const uint64_t a = q_desc0 + static_cast<uint64_t>(t * (L::kQBytes >> 4));
            const uint64_t bq = k_desc0 + static_cast<uint64_t>(st * (L::kKBytes >> 4));
            const bool last = t == NT - 1 || !active(1, j);
            if (elect_one()) {
#pragma unroll
              for (int ch = 0; ch < D / 64; ++ch)
                umma_ss_x4<2, 2>(tmem_base + kColS + buf * BN, a + ch * ((BM * 128) >> 4), bq + ch * ((BN * 128) >> 4), idesc_qk,
                                 ch > 0 ? 1u : 0u);
              umma_commit(&s_full[NT == 1 ? n & 1 : t]);
              if (last) umma_commit(&k_empty[st]);   // the step's last scores: its K tile may be overwritten behind them
            }
            ++n;
            ++own[t];
          }
          return true;
        });
      } else {
        constexpr uint32_t idesc_pv = make_idesc_f16(BM, DV, kBf16, false, true);
        const uint64_t v_desc0 = make_smem_desc(smem_u32(sV), BN * 128, 1024);
        int own[2] = {0, 0};
        for_steps([&](int i, int j) {
          const int st = i % STV;
          if (!wait(&v_full[st], (i / STV) & 1, kSiteVFull)) return false;
          const uint64_t bv = v_desc0 + static_cast<uint64_t>(st * (L::kVBytes >> 4));
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            if (!active(t, j)) continue;
            if (!wait(&p_ready[t], own[t] & 1, kSitePReady)) return false;
            tc_fence_after_sync();
            const bool last = t == NT - 1 || !active(1, j);
            if (elect_one()) {
#pragma unroll
              for (int g = 0; g < BN / 64; ++g)   // 16 KV rows (2048 B) per K step, P advances 8 TMEM columns
                umma_ts_x4<8, 128>(tmem_base + kColO + t * DV, tmem_base + kColP + t * (BN / 2) + g * 32, bv + g * 512, idesc_pv,
                                   (own[t] > 0 || g > 0) ? 1u : 0u);
              umma_commit(&o_done[t]);
              if (last) umma_commit(&v_empty[st]);
            }
            ++own[t];
          }
          return true;
        });
      }
    }
  } else {
    // =============== functor stage: RT threads per query row, TC of its columns each ===============
    const int t = warp / (4 * RT);
    const int half = RT == 1 ? 0 : (warp >> 2) & 1;
    const int row = (warp & 3) * 32 + lane;
    const int q_idx = m0 + t * BM + row;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem_base + lane_base + kColS + (NSB == 2 && NT == 2 ? t * BN : 0) + half * TC;
    const uint32_t tP = tmem_base + lane_base + kColP + t * (BN / 2) + half * (TC / 2);
    constexpr int OC = DV / RT;   // output columns per thread
    const uint32_t tO = tmem_base + lane_base + kColO + t * DV + half * OC;
    const int pair_bar = 1 + t * 4 + (warp & 3);   // named barrier of the two warps that share rows
    float* xch = reinterpret_cast<float*>(smem + L::kOffExchange) + t * 2 * BM + row;
    const int n = kSparse ? n_tiles[t] : j_hi[t] - j_lo[t];
    const int row0 = m0 + t * BM;
    TileWalk walk(sp_keep + t * kMaxTileWords, nullptr, kSparse ? p.tile_words : 0);
    int mask_slot = (kSparse && p.tile_mask_base != nullptr) ? p.tile_mask_base[sp_row[t]] : 0;
    float rs[F::kRowScales > 0 ? F::kRowScales : 1];
    RowCtx ctx{b, h, q_idx, 0, p.seq_q, p.seq_kv, &p.fa};
    F::init(rs, ctx);
    // Where two warps share rows they leave this loop together: each passes what it knows through the exchange of the
    // row maxima, and one that has given up a wait goes on to the next exchange, so that its partner never waits there alone.
    // Other warps leave where a wait has failed.  Their lanes poll one barrier and read one abort flag together, without
    // anything in front of it that parts them, and so agree; every other form that was tried (a vote behind the wait, one in
    // the place of either warp barrier, no leaving at all) took 4 to 8 % of sigmoid 7 x 8 x 3544 x 64 (247 us).
    constexpr bool kPairs = functor_split_sum<F>::value;
    bool ok = !*abort_flag;
    for (int j = 0; j < n && (kPairs || ok); ++j) {   // j counts this query tile's own KV tiles
      const int buf = NSB == 1 ? 0 : (NT == 1 ? j & 1 : t);
      ok = ok && (NT == 1 ? mbar_wait(&s_full[buf], (j >> 1) & 1, ab, kSiteSFull) : mbar_wait(&s_full[t], j & 1, ab, kSiteSFull));
      if (!kPairs && !ok) break;
      tc_fence_after_sync();
      float s[TC];
#pragma unroll
      for (int c = 0; c < TC / 32; ++c) tmem_ld32f(tS + (NT == 1 ? buf * BN : 0) + c * 32, &s[c * 32]);
      tmem_wait_ld();
      // the scores are in registers: their buffer may take the next ones
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_free[buf]);
      // before P is written: the P.V that reads this tile's previous P (and whose sum a rescale would touch) is done
      auto p_free = [&]() {
        if (j > 0) {
          ok = ok && mbar_wait(&o_done[t], (j - 1) & 1, ab, kSiteODone);
          tc_fence_after_sync();
        }
      };
      const int jt = kSparse ? walk.next() : j_lo[t] + j;   // KV tile of this step
      const int kv0 = jt * BN;
      ctx.kv0 = kv0 + half * TC;
      if constexpr (kSparse) {
        // element mask of a partial tile: 128 keep bits for this thread's row (or one column mask for all rows)
        if (F::kNegInfMask && ((sp_part[t * kMaxTileWords + (jt >> 5)] >> (jt & 31)) & 1u) != 0) {
          const uint32_t* mrow;
          if (p.elem_mask_rows > 0) {
            mrow = p.elem_mask + (static_cast<long long>(mask_slot) * p.elem_mask_rows + row) * 4;
            ++mask_slot;
          } else {
            const int n_kv = (p.seq_kv + BN - 1) / BN;
            mrow = p.elem_mask + ((static_cast<long long>(sp_row[t]) / ((p.seq_q + BM - 1) / BM)) * n_kv + jt) * 4;
          }
          uint32_t words[TC / 32];
#pragma unroll
          for (int i = 0; i < TC / 32; i += 2) {
            const uint2 mw = *reinterpret_cast<const uint2*>(mrow + half * (TC / 32) + i);
            words[i] = mw.x;
            words[i + 1] = mw.y;
          }
#pragma unroll
          for (int i = 0; i < TC; ++i) s[i] = ((words[i >> 5] >> (i & 31)) & 1u) ? s[i] : -INFINITY;
        }
      }
      // a tile needs element masking when it crosses an edge of the mask band or the end of the KV sequence
      const bool crosses = (banded && ((right < kNoBound && kv0 + BN - 1 > row0 + right) ||
                                       (left < kNoBound && kv0 < row0 + BM - 1 - left))) || (kv0 + BN > p.seq_kv);
      if (F::kNegInfMask && crosses) {
        // 32 columns at a time, those that a warp's 32 rows keep as a whole left alone, and a compare per element for an open
        // side left out: two compares on every element took 1000 of 2960 cycles on a lone causal tile
        const int q_w = row0 + (warp & 3) * 32;   // the warp's first row
        const int kv_end = p.seq_kv - 1;
        const int k0 = kv0 + half * TC;
        const int first_max = left < kNoBound ? q_w + 31 - left : -kNoBound;
        const int last_min = right < kNoBound ? min(q_w + right, kv_end) : kv_end;
        const int hi = (right < kNoBound ? min(q_idx + right, kv_end) : kv_end) - k0;
#pragma unroll
        for (int c = 0; c < TC; c += 32) {
          if (k0 + c + 31 > last_min) {
#pragma unroll
            for (int i = c; i < c + 32; ++i) s[i] = i <= hi ? s[i] : -INFINITY;
          }
        }
        if (k0 < first_max) {
          const int lo = q_idx - left - k0;
#pragma unroll
          for (int i = 0; i < TC; ++i) s[i] = i >= lo ? s[i] : -INFINITY;
        }
      }
      // P: 16-bit, two per column, in columns of its own
      auto store_half = [&](int c) {
        uint32_t pk[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) pk[i] = pack2<kBf16>(s[c * 64 + 2 * i], s[c * 64 + 2 * i + 1]);
        tmem_st32(tP + c * 32, pk);
      };
      float o_scale;
      bool both_ok = true;
      if constexpr (kPairs) {
        // the functor hands over a piece of the row (32 columns) as soon as its probabilities are final: the piece is on
        // its way to tensor memory while the exponentials of the next one run
        auto row_max = [&](float mx) {   // two buffers in turn: the partner may still read the last step's
          float* x = xch + (L::kExchangeSteps == 2 ? (j & 1) * (NT * 2 * BM) : 0);
          x[half * BM] = mx;
          ok = named_sync_and(pair_bar, 64, ok);
          both_ok = ok;
          mx = fmaxf(mx, x[(half ^ 1) * BM]);
          if constexpr (L::kExchangeSteps == 1) named_sync(pair_bar, 64);
          return mx;
        };
        o_scale = F::template tile_pieces<TC, TC / 32>(s, rs, ctx, row_max, [&](int c) {
          if (c == 0) p_free();
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = pack2<kBf16>(s[c * 32 + 2 * i], s[c * 32 + 2 * i + 1]);
          tmem_st16(tP + c * 16, pk);
        });
      } else if constexpr (F::kUnitOScale) {
        // no rescale: the row can be handed to the functor as narrower tiles, each stored as soon as it is done
        o_scale = 1.0f;
#pragma unroll
        for (int c = 0; c < TC / 32; ++c) {
          ctx.kv0 = kv0 + half * TC + c * 32;
          F::template tile<32>(reinterpret_cast<float(&)[32]>(s[c * 32]), rs, ctx);
          // keys past the end of the sequence weigh nothing: a weight that is not finite, times their zero rows of V, would be
          // NaN.  (On functors that need none of it these lines cost 9 % of sigmoid 7 x 8 x 3544 x 64.)
          if constexpr (!F::kFiniteTail) {
            if (kv0 + BN > p.seq_kv) {
#pragma unroll
              for (int i = 0; i < 32; ++i) s[c * 32 + i] = ctx.kv0 + i < p.seq_kv ? s[c * 32 + i] : 0.0f;
            }
          }
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = pack2<kBf16>(s[c * 32 + 2 * i], s[c * 32 + 2 * i + 1]);
          if (c == 0) p_free();
          tmem_st16(tP + c * 16, pk);
        }
      } else {
        o_scale = F::template tile<TC>(s, rs, ctx);
        p_free();
#pragma unroll
        for (int c = 0; c < TC / 64; ++c) store_half(c);
      }
      if (kPairs && !both_ok) break;
      if (!F::kUnitOScale && j > 0) {
        const bool need = (o_scale != 1.0f);
        if (__any_sync(0xffffffffu, need)) {
#pragma unroll
          for (int c = 0; c < OC / 32; ++c) {
            float o[32];
            tmem_ld32f(tO + c * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= o_scale;
            tmem_st32f(tO + c * 32, o);
          }
        }
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[t]);
    }
    // a query tile of a sparse walk that visits no KV tile at all still owes its output rows: the epilogue of an
    // empty accumulator (what the reference's kernel leaves there as well)
    const bool empty_tile = kSparse && n == 0 && row0 < p.seq_q;
    if (n > 0 || empty_tile) {
      if (n > 0) ok = ok && mbar_wait(&o_done[t], (n - 1) & 1, ab, kSiteOFinal);
      if constexpr (kPairs) {   // the row's sum from its two threads' parts
        float* x = xch + (L::kExchangeSteps == 2 ? (n & 1) * (NT * 2 * BM) : 0);   // not the buffer of the last exchange
        x[half * BM] = rs[F::kSplitSum];
        ok = named_sync_and(pair_bar, 64, ok);
        rs[F::kSplitSum] += x[(half ^ 1) * BM];
      }
      if (ok) {
        tc_fence_after_sync();
        const bool in_range = q_idx < p.seq_q;
        float o[OC];
        if (n > 0) {
#pragma unroll
          for (int c = 0; c < OC / 32; ++c) tmem_ld32f(tO + c * 32, &o[c * 32]);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < OC; ++i) o[i] = 0.0f;
        }
        F::template epilogue<OC>(o, rs, ctx);
        if (p.kv_splits > 1) {
          // split-KV: the normalised rows and their log-sum-exp go to the scratch the combine kernel reads
          if (in_range) {
            const long long prow = ((static_cast<long long>(b) * p.kv_splits + split) * p.heads + h) * p.seq_q + q_idx;
            float4* dst = reinterpret_cast<float4*>(p.part_o + prow * DV + half * OC);
#pragma unroll
            for (int v = 0; v < OC / 4; ++v) dst[v] = make_float4(o[4 * v], o[4 * v + 1], o[4 * v + 2], o[4 * v + 3]);
#pragma unroll
            for (int i = 0; i < (half == 0 ? F::kFinal : 0); ++i) p.part_final[i * p.part_final_stride + prow] = F::final_rowscale(i, rs, ctx);
          }
        } else {
          // Output rows leave through the tile's own Q buffer (free: its last Q.K^T ran before the P.V that o_done
          // reports).  Each warp owns the 32 rows it computed, so a warp-level sync is enough: every lane writes its
          // row in 16-byte pieces (piece index xor row: conflict-free), then the warp stores whole rows, DV*2
          // contiguous bytes per row and 512 bytes per instruction.  A thread storing its own row put 32 pieces
          // into 32 different rows with every instruction, and the tile's last output took ~3100 cycles.
          static_assert(DV <= D, "the output tile is staged in the query tile's buffer");
          constexpr int PR = OC / 8;     // 16-byte pieces of a row's columns
          constexpr int RPI = 32 / PR;   // rows per warp instruction
          const uint32_t stage = smem_u32(sQ + t * L::kQBytes) + ((warp & 3) * RT + half) * (32 * OC * 2);
          const uint32_t mine = stage + lane * (OC * 2);
#pragma unroll
          for (int v = 0; v < PR; ++v) {
            uint4 pk;
            pk.x = pack2<kBf16>(o[8 * v + 0], o[8 * v + 1]);
            pk.y = pack2<kBf16>(o[8 * v + 2], o[8 * v + 3]);
            pk.z = pack2<kBf16>(o[8 * v + 4], o[8 * v + 5]);
            pk.w = pack2<kBf16>(o[8 * v + 6], o[8 * v + 7]);
            st_shared_v4(mine + ((v ^ (lane & (PR - 1))) << 4), pk);
          }
          __syncwarp();
          const int c = lane & (PR - 1), rsub = lane / PR;
          const int row_first = row0 + (warp & 3) * 32;
          uint8_t* obase = reinterpret_cast<uint8_t*>(p.o) +
                           2 * (static_cast<long long>(b) * p.o_sb + static_cast<long long>(h) * p.o_sh + half * OC) + c * 16;
          uint4 val[PR];   // all loads first, then all stores: one after the other each pair costs a shared-memory round trip
#pragma unroll
          for (int i = 0; i < PR; ++i) {
            const int r = i * RPI + rsub;
            val[i] = ld_shared_v4(stage + r * (OC * 2) + ((c ^ (r & (PR - 1))) << 4));
          }
#pragma unroll
          for (int i = 0; i < PR; ++i) {
            const int r = i * RPI + rsub;
            if (row_first + r < p.seq_q)
              *reinterpret_cast<uint4*>(obase + 2 * static_cast<long long>(row_first + r) * p.o_ss) = val[i];
          }
        }
        if (in_range && half == 0 && p.kv_splits <= 1) {
#pragma unroll
          for (int i = 0; i < F::kFinal; ++i) {
            if (p.final_out[i] != nullptr) {
              p.final_out[i][(static_cast<long long>(b) * p.heads + h) * p.seq_q + q_idx] = F::final_rowscale(i, rs, ctx);
            }
          }
        }
      }
    }
  }

  // a split whose share of the KV tiles is empty for a query tile contributes nothing
  if (p.kv_splits > 1 && warp < 4 * NT * RT) {
    const int t = warp / (4 * RT);
    const int q_idx = m0 + t * BM + (warp & 3) * 32 + lane;
    if (j_hi[t] <= j_lo[t] && q_idx < p.seq_q)
      p.part_final[((static_cast<long long>(b) * p.kv_splits + split) * p.heads + h) * p.seq_q + q_idx] = -INFINITY;
  }

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // a wait was abandoned: give copies and MMAs still in flight time to land before the CTA's
    // shared and tensor memory are released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kQkWarp) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}


// Split-KV combine: o[b,q,h,:] = sum_i w_i part_o[b,i,h,q,:] with w_i = F::combine(i, splits, final row scales of
// all splits) -- the lowered OnlineFunc.combine of the reference (core/lower/lower_decode.py:287-302, combine kernel
// of attn_decode_tl.py:158-206).  For the built-in softmax that is exp(lse_i - lse), lse = log sum_i exp(lse_i), and
// the combined lse is written out as the call's final row scale.  One warp per (batch, head, query row).
template <class F, int DV, bool kBf16>
__global__ void __launch_bounds__(256) parallel_combine_kernel(const float* part_o, const float* part_final,
                                                             long long part_final_stride, void* o,
                                                             float* final_out, int batch, int heads, int seq_q,
                                                             int splits, long long o_sb, long long o_ss, long long o_sh) {
  pdl_launch_dependents();
  pdl_wait();
  const long long row = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= static_cast<long long>(batch) * heads * seq_q) return;
  const int q = static_cast<int>(row % seq_q);
  const int h = static_cast<int>((row / seq_q) % heads);
  const int b = static_cast<int>(row / (static_cast<long long>(seq_q) * heads));
  const long long split_stride = static_cast<long long>(heads) * seq_q;
  const long long prow0 = (static_cast<long long>(b) * splits * heads + h) * seq_q + q;   // split 0
  const float* fin = part_final + prow0;
  constexpr int E = DV / 32;   // columns per lane
  float acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  for (int i = 0; i < splits; ++i) {
    const float w = F::combine(i, splits, fin, split_stride, part_final_stride);
    if (w == 0.0f) continue;   // an empty split (its partial rows were never written)
    const float* src = part_o + (prow0 + i * split_stride) * DV + lane * E;
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] += w * src[e];
  }
  uint8_t* orow = reinterpret_cast<uint8_t*>(o) + 2 * (b * o_sb + q * o_ss + h * o_sh + lane * E);
#pragma unroll
  for (int e = 0; e < E; e += 2) *reinterpret_cast<uint32_t*>(orow + 2 * e) = pack2<kBf16>(acc[e], acc[e + 1]);
  if constexpr (F::kCombinedFinal) {
    if (lane == 0 && final_out != nullptr)
      final_out[(static_cast<long long>(b) * heads + h) * seq_q + q] = F::combined_final(splits, fin, split_stride, part_final_stride);
  }
}

}  // namespace b200
