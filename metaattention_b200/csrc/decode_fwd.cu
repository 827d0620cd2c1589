// Decode attention for sm_100a: a few query rows per sequence against a long KV cache, softmax(scale * Q.K^T).V, with
// grouped KV heads, per-sequence lengths and block-sparse caches.  Bound by the bytes of the kept cache.
//
// Stands in for the reference's split-KV decode kernels (core/lower/lower_decode.py:375-449, the GQA decode of
// core/template/tl_template/attn/attn_gqa_tl.py and blockattn_decode_varlen_tl.py) where the program is the built-in softmax;
// other programs decode on the forward kernel (parallel_fwd.cuh).
//
// What the forward kernel spends on such a call: one 128-row query tile per QUERY head with one row used, so a group of
// heads reads its K/V head once per query head; one CTA per (head, sequence) or a whole number of splits of it; a sparse
// call visits 128-row tiles for kept blocks of 32 and needs a launch of its own for the tile bitmaps.  Here
//   * the rows of a query tile are the (query position, head of the group) pairs of one KV head: K/V are read once;
//   * the KV tiles of all (sequence, KV head) pairs form one list that is cut into one equal share per SM; a share walks
//     its pieces ("units") with every ring and barrier phase carried across units, so that loads never stop between them;
//   * kept blocks are GATHERED: a 128-row tile is filled with the next 128 / block kept blocks by one TMA box each, and
//     the counts that cut the list are taken from the block mask and the lengths by every CTA itself;
//   * two softmax groups take alternate tiles with score tiles and accumulators of their own, merged at the end of a
//     unit through tensor memory (both accumulators of a row are in the lane of its thread).  With one group the warp that
//     holds the only used rows is the bound: ~1600 cycles a tile, against 1480 for the bytes of a 64-wide tile;
//   * K and V each have a ring of 96 KB: ~190 KB in flight per SM, three times what latency times bandwidth asks for.
// Measured (calls back to back, bf16, D = 128): 1 sequence x 32 heads x 32768 tokens 93-103 us from box to box = 5.2-5.8 TB/s of
// K and V, x 4312 tokens 23.7-28 (25.2 before the first loads went ahead of the CTA's set-up and the merge kernel fetched its code early); 8
// sequences x 32 heads on 8 KV heads, up to 8192 tokens, 30 % of the 32-token blocks kept 38 -> 30: of its 26 us in the
// kernel 8 went to counting the mask at four flags a load, 2 to a list of kept blocks made the same way, 2 to boxes issued
// by one lane.  8 such sequences of 16384 tokens, dense: 5.8 TB/s.
// A unit that is a whole (sequence, KV head) pair writes its output; the others leave fp32 partial rows that a second
// small kernel adds up, launched early (programmatic dependent launch) so that only its own microseconds show.
#include <cstring>

#include "../../include/attn_b200.h"
#include "common_host.cuh"
#include "functors.cuh"
#include "parallel_launch.cuh"

namespace b200 {

constexpr int kDecTile = 128;         // KV rows of a tile
constexpr int kDecThreads = 320;      // softmax group 0 (warps 0-3), group 1 (4-7), loading warp 8, issuing warp 9
constexpr int kDecMaxPairs = 1024;    // (sequence, KV head) pairs of a call with lengths or a block mask
constexpr int kDecMaxBlocks = 4096;   // blocks of a block mask's row

struct DecodeParams {
  void* o;
  float* lse;                    // [batch, heads, seq_q] or null
  long long o_sb, o_ss, o_sh;
  int batch, heads, heads_kv, group, seq_q, seq_kv;
  int rows, rows_pad;            // group * seq_q rows of a query tile; padded to a multiple of 8
  int q_bufs, q_bytes;           // query tile buffers in shared memory and the bytes of one
  int head_major;                // row = g * seq_q + q (1) or q * group + g (0): the order the tensor map delivers
  const uint8_t* block_mask;     // [batch, heads_kv, n_blocks] or null
  const int* seq_lens;           // [batch] or null
  int n_blocks, block;           // blocks of a mask row, rows of a block (divides 128)
  float* part_o;                 // [2 * CTAs][rows][D]
  float* part_lse;               // [2 * CTAs][rows]
  int* cum;                      // [batch * heads_kv + 1] tiles in front of each pair, for the merge (lengths or mask)
  CoordOrder oq, ok, ov;
  int* status;
  FunctorArgs fa;
};

enum DecodeWaitSite { kDecQFull = 81, kDecQEmpty, kDecKFull, kDecKEmpty, kDecVFull, kDecVEmpty, kDecSFull, kDecPReady, kDecODone, kDecStats, kDecOFree };

// kCounted: calls with lengths or a block mask, whose shares are cut from counts made on the device
template <int D, bool kCounted>
struct DecodeSmem {
  static constexpr int kTileBytes = kDecTile * D * 2;
  static constexpr int kStages = 98304 / kTileBytes;          // 3 of 32 KB or 6 of 16 KB, for K and for V
  // query tiles; an MMA reads 128 rows from a tile's start whatever its rows, so what follows must be shared memory too
  static constexpr int kQRegion = kCounted ? D * 128 : D * 256;
  static constexpr int kOffK = kQRegion;
  static constexpr int kOffV = kOffK + kStages * kTileBytes;
  static constexpr int kOffBar = kOffV + kStages * kTileBytes;
  static constexpr int kQFull = 0, kQEmpty = 2, kSFull = 4, kPReady = 6, kODone = 8, kStats = 10, kOFree = 11, kKFull = 12;
  static constexpr int kKEmpty = kKFull + kStages, kVFull = kKEmpty + kStages, kVEmpty = kVFull + kStages, kNumBars = kVEmpty + kStages;
  static constexpr int kOffMisc = kOffBar + 8 * kNumBars;
  static constexpr int kOffMl = kOffMisc + 16;                  // float2 [128]: group 1's (reference maximum, sum) of a row
  static constexpr int kOffCum = kOffMl + 128 * 8;              // kCounted: int [pairs + 1] tiles in front, int [pairs] valid rows
  static constexpr int kOffList = kOffCum + (kCounted ? (2 * kDecMaxPairs + 4) * 4 : 0);   // uint16: kept blocks of the unit
  static constexpr int kBytes = kOffList + (kCounted ? 2 * kDecMaxBlocks : 0) + 1024;
  static_assert(kBytes <= 232448, "shared memory layout exceeds an SM");
};

// tile range of CTA c of n <= T: [c T / n, (c + 1) T / n); the CTA that holds tile t is ((t + 1) n - 1) / T
__host__ __device__ __forceinline__ int dec_share(long long total, int c, int n) { return static_cast<int>(total * c / n); }
__device__ __forceinline__ int dec_owner(int t, int n, int total) {
  return static_cast<int>((static_cast<long long>(t + 1) * n - 1) / total);
}

// The units of one CTA, in order: pair, first tile of the pair, tiles, KV rows of the pair that take part.
struct DecodeWalk {
  const int* cum;   // null: every pair has `per` tiles and `rows` valid rows
  const int* valid;
  int per, all_rows, t, t_end;
  int pair, t0, n, total, rows;
  __device__ DecodeWalk(const int* cum_, const int* valid_, int pairs, int per_, int all_rows_, int t_, int t_end_)
      : cum(cum_), valid(valid_), per(per_), all_rows(all_rows_), t(t_), t_end(t_end_) {
    if (cum == nullptr) {
      pair = t / per - 1;
    } else {
      int lo = 0, hi = pairs;   // last pair with cum[pair] <= t
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cum[mid] <= t) lo = mid; else hi = mid;
      }
      pair = lo - 1;
    }
    n = 0;
  }
  __device__ bool next() {
    if (t >= t_end) return false;
    int first;
    do {
      ++pair;
      first = cum == nullptr ? pair * per : cum[pair];
      total = cum == nullptr ? per : cum[pair + 1] - first;
    } while (first + total <= t);   // pairs without tiles
    rows = cum == nullptr ? all_rows : valid[pair];
    t0 = t - first;
    n = min(total - t0, t_end - t);
    t += n;
    return true;
  }
};

// Flags [i, i + 16) of a mask row as bits, those from `n` on as zeros; `wide`: the row may be read sixteen flags at a time.
__device__ __forceinline__ uint32_t dec_flags16(const uint8_t* row, int i, int n, bool wide) {
  uint32_t m = 0;
  if (wide) {
    if (i < n) {   // rows are whole pieces of sixteen
      const uint4 v = *reinterpret_cast<const uint4*>(row + i);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) m |= ((__vsetne4(w[k], 0u) * 0x10204080u) >> 28) << (4 * k);   // four bytes of 0 / 1 to four bits
    }
  } else {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (i + k < n && row[i + k] != 0) m |= 1u << k;
  }
  const int in = min(max(n - i, 0), 16);
  return m & ((1u << in) - 1u);
}

template <int D, bool kBf16, bool kCounted>
__global__ void __launch_bounds__(kDecThreads, 1)
decode_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const DecodeParams p) {
  using L = DecodeSmem<D, kCounted>;
  using F = SoftmaxFunctor;
  constexpr int N = kDecTile, ST = L::kStages, KC = D / 64, kChunk = N * 128;
  constexpr uint32_t kTmemCols = 512, kColS = 0, kColO = 256;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = smem + L::kOffK;
  uint8_t* sV = smem + L::kOffV;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kOffBar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kOffMisc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kOffMisc + 8);
  float2* s_ml = reinterpret_cast<float2*>(smem + L::kOffMl);
  int* s_cum = reinterpret_cast<int*>(smem + L::kOffCum);
  int* s_valid = s_cum + kDecMaxPairs + 1;
  uint16_t* s_list = reinterpret_cast<uint16_t*>(smem + L::kOffList);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const AbortState ab{abort_flag, p.status};
  const int pairs = p.batch * p.heads_kv;
  const int active_warps = (p.rows + 31) / 32;   // of each softmax group
  const bool sparse = kCounted && p.block_mask != nullptr;

  // The merge kernel may be made ready, ahead of this kernel's own allocation (behind it a dense call of 1 x 32 x 13172 x 64 took
  // 34.2 us, so 32.8): the rule of sm100.cuh is kept by shared memory, of which no kernel with tensor memory takes less than 64 KB.
  static_assert(L::kBytes + 65536 > 233472, "a CTA with tensor memory could share the SM");
  pdl_launch_dependents();

  const int per_pair = (p.seq_kv + N - 1) / N;
  const int cta = static_cast<int>(blockIdx.x);
  // The loading lane sets the barriers up; without counts to wait for it sends the first loads off at once, under the
  // tensor-memory allocation and the CTA-wide sync.  (If the status word turns out set nobody takes them, and the teardown
  // below gives them time to land.)
  auto load_q = [&](int buf, int pair) {
    const int b = pair / p.heads_kv, hk = pair - b * p.heads_kv;
    mbar_arrive_expect_tx(bars + L::kQFull + buf, KC * p.rows * 128);
    for (int c = 0; c < KC; ++c)
      tma_load_rows(sQ + buf * p.q_bytes + c * (p.rows_pad * 128), &tmQ, bars + L::kQFull + buf, c * 64, 0, hk * p.group, b, p.oq);
  };
  int early = 0;   // tiles of the first unit on their way
  if (warp == 8) {   // two barriers a lane
    for (int i = lane; i < L::kNumBars; i += 32) {
      const bool rows = i == L::kPReady || i == L::kPReady + 1 || i == L::kStats || i == L::kOFree;
      mbar_init(bars + i, rows ? active_warps * 32 : 1);
    }
    fence_barrier_init();
    __syncwarp();
  }
  if (warp == 8 && lane == 0) {
    if constexpr (!kCounted) {
      pdl_wait();
      const int total = pairs * per_pair, shares = min(static_cast<int>(gridDim.x), total);
      if (cta < shares) {
        DecodeWalk u(nullptr, nullptr, pairs, per_pair, p.seq_kv, dec_share(total, cta, shares), dec_share(total, cta + 1, shares));
        u.next();
        load_q(0, u.pair);
        const int b = u.pair / p.heads_kv, hk = u.pair - b * p.heads_kv;
        early = min(u.n, ST);
#pragma unroll 1
        for (int i = 0; i < early; ++i) {
          mbar_arrive_expect_tx(bars + L::kKFull + i, L::kTileBytes);
          mbar_arrive_expect_tx(bars + L::kVFull + i, L::kTileBytes);
          for (int c = 0; c < KC; ++c)
            tma_load_rows(sK + i * L::kTileBytes + c * kChunk, &tmK, bars + L::kKFull + i, c * 64, (u.t0 + i) * N, hk, b, p.ok);
          for (int c = 0; c < KC; ++c)
            tma_load_rows(sV + i * L::kTileBytes + c * kChunk, &tmV, bars + L::kVFull + i, c * 64, (u.t0 + i) * N, hk, b, p.ov);
        }
      }
    } else {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
    }
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  pdl_wait();
  if (tid == 0) *abort_flag = (*reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
  // ---- how many KV rows of every pair take part, and the tiles in front of it ----
  const bool wide = sparse && (p.n_blocks & 15) == 0 && (reinterpret_cast<uintptr_t>(p.block_mask) & 15) == 0;
  if constexpr (kCounted) {
    auto len_of = [&](int b) { return p.seq_lens != nullptr ? min(max(p.seq_lens[b], 0), p.seq_kv) : p.seq_kv; };
    if (sparse) {
      for (int i = tid; i < pairs; i += kDecThreads) s_valid[i] = 0;
      __syncthreads();
      // Sixteen flags per item; the items of a thread are independent loads, all of them in flight at once where there
      // are no more than four (64 rows of 256 flags: 5.4 k cycles, 12.4 k at four flags an item)
      const int ipr = (p.n_blocks + 15) / 16;
#pragma unroll 4
      for (int i = tid; i < pairs * ipr; i += kDecThreads) {
        const int pair = i / ipr, at = 16 * (i - pair * ipr);
        const uint32_t m = dec_flags16(p.block_mask + static_cast<long long>(pair) * p.n_blocks, at, p.n_blocks, wide);
        const int len = len_of(pair / p.heads_kv);
        const int nb = min(p.n_blocks, (len + p.block - 1) / p.block);   // blocks that begin inside the sequence
        const int in = min(max(nb - at, 0), 16), last = nb - 1 - at;     // the sequence's last block may be cut by its end
        int r = __popc(m & ((1u << in) - 1u)) * p.block;
        if (last >= 0 && last < 16 && ((m >> last) & 1u)) r -= max(nb * p.block - len, 0);
        if (r > 0) atomicAdd(&s_valid[pair], r);
      }
      __syncthreads();
    } else {
      for (int i = tid; i < pairs; i += kDecThreads) s_valid[i] = len_of(i / p.heads_kv);
      __syncthreads();
    }
    if (warp == 0) {
      int run = 0;
      for (int i0 = 0; i0 < pairs; i0 += 32) {
        const int tiles = i0 + lane < pairs ? (s_valid[i0 + lane] + N - 1) / N : 0;
        int x = tiles;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, x, d);
          if (lane >= d) x += y;
        }
        if (i0 + lane < pairs) s_cum[i0 + lane] = run + x - tiles;
        run += __shfl_sync(0xffffffffu, x, 31);
      }
      if (lane == 0) s_cum[pairs] = run;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int total = kCounted ? s_cum[pairs] : pairs * per_pair;
  const int shares = min(static_cast<int>(gridDim.x), total);   // none is empty
  const int T0 = cta < shares ? dec_share(total, cta, shares) : 0, T1 = cta < shares ? dec_share(total, cta + 1, shares) : 0;
  if (kCounted && blockIdx.x == 0)
    for (int i = tid; i <= pairs; i += kDecThreads) p.cum[i] = s_cum[i];
  const bool run_cta = warp_all(T1 > T0 && !*abort_flag);
  auto make_walk = [&]() { return DecodeWalk(kCounted ? s_cum : nullptr, s_valid, pairs, per_pair, p.seq_kv, T0, T1); };

  if (warp == 8) {
    // ======================= loading warp =======================
    if (run_cta) {
      DecodeWalk u = make_walk();
      const int n_early = __shfl_sync(0xffffffffu, early, 0);
      bool ok = true;
      int J = 0;
      for (int ui = 0; ok && u.next(); ++ui) {
        const int b = u.pair / p.heads_kv, hk = u.pair - b * p.heads_kv;
        const int bpt = sparse ? N / p.block : 1;
        int kept_here = 0;
        if (sparse) {
          // ranks [t0 * bpt, (t0 + n) * bpt) of the row's kept blocks, sixteen flags per lane and step
          const uint8_t* row = p.block_mask + static_cast<long long>(u.pair) * p.n_blocks;
          const int len = p.seq_lens != nullptr ? min(max(p.seq_lens[b], 0), p.seq_kv) : p.seq_kv;
          const int nb = min(p.n_blocks, (len + p.block - 1) / p.block);
          const int r0 = u.t0 * bpt, r1 = r0 + u.n * bpt;
          __syncwarp();   // the previous unit's list has been read
          int rank = 0;
          for (int base = 0; base < p.n_blocks && rank < r1; base += 512) {
            const int i0 = base + 16 * lane;
            uint32_t flags = dec_flags16(row, i0, p.n_blocks, wide);   // does not wait for the length
            flags &= (1u << min(max(nb - i0, 0), 16)) - 1u;
            const int mine = __popc(flags);
            int x = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
              const int y = __shfl_up_sync(0xffffffffu, x, d);
              if (lane >= d) x += y;
            }
            int r = rank + x - mine;
            for (; flags != 0; flags &= flags - 1, ++r)
              if (r >= r0 && r < r1) s_list[r - r0] = static_cast<uint16_t>(i0 + __ffs(flags) - 1);
            rank += __shfl_sync(0xffffffffu, x, 31);
          }
          kept_here = min(rank, r1) - r0;
          __syncwarp();
        }
        // A tile's boxes are spread over the lanes: K's and V's bpt blocks of KC column chunks (at most 32 boxes; one lane
        // issuing all of them, sixteen a tile with blocks of 32, took 3100 cycles a tile against 2400 for its bytes)
        const int qb = ui % p.q_bufs;
        if (ui >= p.q_bufs) ok = warp_all(mbar_wait(bars + L::kQEmpty + qb, (ui / p.q_bufs - 1) & 1, ab, kDecQEmpty));
        if (lane == 0 && ok && (kCounted || ui > 0)) load_q(qb, u.pair);
        const int blk = lane / KC, chunk = lane - blk * KC;
        for (int i = 0; i < u.n && ok; ++i) {
          const int jj = J + i, st = jj % ST;
          if (!kCounted && jj < n_early) continue;
          const uint32_t par = ((jj / ST) & 1) ^ 1;
          // slots past the last kept block repeat it: masked, but what lies there is multiplied by zero
          const int r = sparse ? s_list[min(i * bpt + blk, kept_here - 1)] * p.block : (u.t0 + i) * N;
          const int off = st * L::kTileBytes + chunk * kChunk + (sparse ? blk * p.block * 128 : 0);
          for (int kv = 0; kv < 2 && ok; ++kv) {
            uint64_t* full = bars + (kv == 0 ? L::kKFull : L::kVFull) + st;
            ok = warp_all(mbar_wait(bars + (kv == 0 ? L::kKEmpty : L::kVEmpty) + st, par, ab, kv == 0 ? kDecKEmpty : kDecVEmpty));
            if (!ok) break;
            if (lane == 0) mbar_arrive_expect_tx(full, L::kTileBytes);
            __syncwarp();
            if (blk < bpt) {
              if (kv == 0) tma_load_rows(sK + off, &tmK, full, chunk * 64, r, hk, b, p.ok);
              else tma_load_rows(sV + off, &tmV, full, chunk * 64, r, hk, b, p.ov);
            }
          }
        }
        J += u.n;
      }
    }
  } else if (warp == 9) {
    // ======================= issuing warp (converged, one elected lane per batch) =======================
    if (run_cta) {
      constexpr uint32_t idesc_qk = make_idesc_f16(128, N, kBf16, false, false);
      constexpr uint32_t idesc_pv = make_idesc_f16(128, D, kBf16, false, true);
      auto wait = [&](uint64_t* bar, uint32_t parity, int site) -> bool { return warp_all(mbar_wait_poll(bar, parity, ab, site)); };
      const uint64_t k_desc0 = make_smem_desc(smem_u32(sK), 16, 1024);
      const uint64_t v_desc0 = make_smem_desc(smem_u32(sV), kChunk, 1024);
      DecodeWalk uq = make_walk();
      int uq_i = -1, uq_left = 0, Jq = 0;   // unit and tile of the next scores
      auto issue_qk = [&]() -> bool {
        if (uq_left == 0) {
          uq.next();
          uq_left = uq.n;
          ++uq_i;
          if (!wait(bars + L::kQFull + uq_i % p.q_bufs, (uq_i / p.q_bufs) & 1, kDecQFull)) return false;
        }
        const int st = Jq % ST, t = Jq & 1, qb = uq_i % p.q_bufs;
        if (!wait(bars + L::kKFull + st, (Jq / ST) & 1, kDecKFull)) return false;
        tc_fence_after_sync();
        --uq_left;
        const uint64_t a = make_smem_desc(smem_u32(sQ + qb * p.q_bytes), 16, 1024);
        const uint64_t bk = k_desc0 + static_cast<uint64_t>(st * (L::kTileBytes >> 4));
        const uint64_t a_chunk = static_cast<uint64_t>(p.rows_pad * 128) >> 4;
        if (elect_one()) {
#pragma unroll
          for (int ch = 0; ch < KC; ++ch)
            umma_ss_x4<2, 2>(tmem_base + kColS + t * N, a + ch * a_chunk, bk + ch * (kChunk >> 4), idesc_qk, ch > 0 ? 1u : 0u);
          umma_commit(bars + L::kSFull + t);
          umma_commit(bars + L::kKEmpty + st);
          if (uq_left == 0) umma_commit(bars + L::kQEmpty + qb);
        }
        ++Jq;
        return true;
      };
      const int n_all = T1 - T0;
      bool ok = issue_qk();
      if (ok && n_all > 1) ok = issue_qk();
      DecodeWalk u = make_walk();
      int J = 0;
      for (int ui = 0; ok && u.next(); ++ui) {
        for (int i = 0; i < u.n && ok; ++i, ++J) {
          const int t = J & 1, st = J % ST;
          if (i == 0 && ui > 0) ok = wait(bars + L::kOFree, (ui - 1) & 1, kDecOFree);   // the accumulators have been read
          ok = ok && wait(bars + L::kVFull + st, (J / ST) & 1, kDecVFull) && wait(bars + L::kPReady + t, (J >> 1) & 1, kDecPReady);
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t bv = v_desc0 + static_cast<uint64_t>(st * (L::kTileBytes >> 4));
          if (elect_one()) {
#pragma unroll
            for (int g = 0; g < N / 64; ++g)
              umma_ts_x4<8, 128>(tmem_base + kColO + t * D, tmem_base + kColS + t * N + g * 32, bv + g * 512, idesc_pv,
                                 (i >= 2 || g > 0) ? 1u : 0u);
            umma_commit(bars + L::kODone + t);
            umma_commit(bars + L::kVEmpty + st);
          }
          if (Jq < n_all) ok = issue_qk();   // over the scores of tile J, behind its P.V in the pipe
        }
      }
    }
  } else if ((warp & 3) < active_warps && run_cta) {
    // ======================= softmax groups: one query row per thread, alternate tiles =======================
    const int t = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t tS = tmem_base + lane_base + kColS + t * N;
    const uint32_t tO = tmem_base + lane_base + kColO + t * D;
    const RowCtx ctx{0, 0, 0, 0, p.seq_q, p.seq_kv, &p.fa};   // softmax asks for the scale only
    DecodeWalk u = make_walk();
    int J0 = 0;   // tiles of the units before this one
    for (int ui = 0; u.next(); ++ui, J0 += u.n) {
      float rs[2];
      F::init(rs, ctx);
      for (int J = J0 + ((J0 ^ t) & 1); J < J0 + u.n; J += 2) {
        mbar_wait_rows(bars + L::kSFull + t, (J >> 1) & 1, ab, kDecSFull);
        tc_fence_after_sync();
        float s[N];
#pragma unroll
        for (int c = 0; c < N / 32; ++c) tmem_ld32f(tS + c * 32, &s[c * 32]);
        tmem_wait_ld();
        const int left = u.rows - (u.t0 + J - J0) * N;   // rows of the pair from this tile on
        if (left < N) {
#pragma unroll
          for (int i = 0; i < N; ++i) s[i] = i < left ? s[i] : -INFINITY;
        }
        const float o_scale = F::template tile_pieces<N, 4, false>(s, rs, ctx, [](float mx) { return mx; }, [&](int c) {
          constexpr int W = N / 4 / 2;
          uint32_t pk[W];
#pragma unroll
          for (int i = 0; i < W; ++i) pk[i] = pack2<kBf16>(s[c * 2 * W + 2 * i], s[c * 2 * W + 2 * i + 1]);
          static_assert(W == 16, "a quarter of the row per store");
          tmem_st16(tS + c * W, pk);
        });
        if (J - J0 >= 2 && __any_sync(0xffffffffu, o_scale != 1.0f)) {
          mbar_wait_rows(bars + L::kODone + t, ((J >> 1) - 1) & 1, ab, kDecODone);
          tc_fence_after_sync();
#pragma unroll
          for (int c = 0; c < D / 32; ++c) {
            float o[32];
            tmem_ld32f(tO + c * 32, o);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= o_scale;
            tmem_st32f(tO + c * 32, o);
          }
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bars + L::kPReady + t);
      }
      if (t == 1) {
        if (ui > 0) mbar_wait_rows(bars + L::kOFree, (ui - 1) & 1, ab, kDecOFree);   // group 0 has read the last unit's
        s_ml[row] = make_float2(rs[0], rs[1]);
        mbar_arrive(bars + L::kStats);
        continue;
      }
      // ---- end of a unit (group 0): both accumulators of the row, weighted ----
      const int Jl = J0 + u.n - 1, l0 = (Jl & 1) == 0 ? Jl : Jl - 1, l1 = (Jl & 1) == 1 ? Jl : Jl - 1;
      const bool has0 = l0 >= J0, has1 = l1 >= J0;
      mbar_wait_rows(bars + L::kStats, ui & 1, ab, kDecStats);
      if (has0) mbar_wait_rows(bars + L::kODone, (l0 >> 1) & 1, ab, kDecODone);
      if (has1) mbar_wait_rows(bars + L::kODone + 1, (l1 >> 1) & 1, ab, kDecODone);
      if (!warp_all(!*abort_flag)) break;
      tc_fence_after_sync();
      const float2 ml1 = s_ml[row];
      const float c2 = p.fa.f[0] * 1.4426950408889634f;
      const float m = fmaxf(rs[0], ml1.x);
      const float w0 = fast_exp2((rs[0] - m) * c2), w1 = fast_exp2((ml1.x - m) * c2);
      const float sum = rs[1] * w0 + ml1.y * w1;
      const float inv = 1.0f / sum, f0 = has0 ? w0 * inv : 0.0f, f1 = has1 ? w1 * inv : 0.0f;
      const float lse = logf(sum) + m * p.fa.f[0];
      const int g = p.head_major ? row / p.seq_q : row % p.group;
      const int qi = p.head_major ? row % p.seq_q : row / p.group;
      const int b = u.pair / p.heads_kv, h = (u.pair - b * p.heads_kv) * p.group + g;
      const bool whole = u.n == u.total;
      // a partial result: the pair's first share leaves it in the second slot of its CTA, the later ones in the first
      const long long slot = (2LL * blockIdx.x + (u.t0 == 0 ? 1 : 0)) * p.rows + row;
      uint16_t* orow = static_cast<uint16_t*>(p.o) + b * p.o_sb + qi * p.o_ss + h * p.o_sh;
      // not unrolled: it runs once or twice a call, and fetching 13 KB of code for it took 2700 cycles
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        float a0[32], a1[32];
        tmem_ld32f(tO + c * 32, a0);
        tmem_ld32f(tO + D + c * 32, a1);
        tmem_wait_ld();
        if (has0 && has1) {   // an accumulator that the unit has not used holds anything
#pragma unroll
          for (int i = 0; i < 32; ++i) a0[i] = fmaf(a0[i], f0, a1[i] * f1);
        } else {
          const float f = has0 ? f0 : f1;
#pragma unroll
          for (int i = 0; i < 32; ++i) a0[i] = (has0 ? a0[i] : a1[i]) * f;
        }
        if (row < p.rows) {
          if (whole) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 pk;
              pk.x = pack2<kBf16>(a0[8 * v + 0], a0[8 * v + 1]);
              pk.y = pack2<kBf16>(a0[8 * v + 2], a0[8 * v + 3]);
              pk.z = pack2<kBf16>(a0[8 * v + 4], a0[8 * v + 5]);
              pk.w = pack2<kBf16>(a0[8 * v + 6], a0[8 * v + 7]);
              reinterpret_cast<uint4*>(orow + c * 32)[v] = pk;
            }
          } else {
            float4* dst = reinterpret_cast<float4*>(p.part_o + slot * D + c * 32);
#pragma unroll
            for (int v = 0; v < 8; ++v) dst[v] = make_float4(a0[4 * v], a0[4 * v + 1], a0[4 * v + 2], a0[4 * v + 3]);
          }
        }
      }
      if (row < p.rows) {
        if (!whole) p.part_lse[slot] = lse;
        else if (p.lse != nullptr) p.lse[(static_cast<long long>(b) * p.heads + h) * p.seq_q + qi] = lse;
      }
      tc_fence_before_sync();
      mbar_arrive(bars + L::kOFree);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 9) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Adds up the partial rows of the pairs that were cut: o = sum_i exp(lse_i - lse) part_i.  One warp per (pair, row).  Pairs
// that one CTA held whole were written by it; a pair without a kept row gets what an empty softmax is (nan, -inf).
template <int D, bool kBf16>
__global__ void __launch_bounds__(128) decode_merge_kernel(const DecodeParams p, int ctas, int counted) {
  pdl_launch_dependents();
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  const int pairs = p.batch * p.heads_kv;
  if (w >= pairs * p.rows) return;   // (the block's first warp never does)
  const int pair = w / p.rows, row = w - pair * p.rows;
  const int per = (p.seq_kv + kDecTile - 1) / kDecTile;
  const int g = p.head_major ? row / p.seq_q : row % p.group, qi = p.head_major ? row % p.seq_q : row / p.group;
  const int b = pair / p.heads_kv, h = (pair - b * p.heads_kv) * p.group + g;
  constexpr int E = D / 32;
  uint16_t* orow = static_cast<uint16_t*>(p.o) + b * p.o_sb + qi * p.o_ss + h * p.o_sh + lane * E;
  // The blocks of this kernel stand ready while the decode kernel still runs.  A first pass over the same code, on scratch
  // that is not written yet and without a store, fetches the instructions and page translations meanwhile: the pass that
  // counts took 4 to 5 us without it, behind the decode kernel's end.  All reads pass L1 by, so nothing stale is kept there.
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const bool real = pass == 1;
    if (real) pdl_wait();   // the decode kernel's results are complete and visible
    int total = pairs * per, first = pair * per, end = first + per;
    if (counted) {
      total = __ldcg(p.cum + pairs);
      first = __ldcg(p.cum + pair);
      end = __ldcg(p.cum + pair + 1);
    }
    const int shares = min(ctas, total);
    int c_lo = 0, c_hi = -1;
    if (end > first && shares > 0) {
      c_lo = dec_owner(first, shares, total);
      c_hi = dec_owner(end - 1, shares, total);
    }
    if (!real) {   // what the counts say is not to be relied on yet: two slots that exist
      c_lo = 0;
      c_hi = min(1, ctas - 1);
    } else if (c_lo == c_hi) {
      return;
    }
    auto slot_of = [&](int c) { return (2LL * c + (c == c_lo ? 1 : 0)) * p.rows + row; };
    // Four shares at a time, their statistics and rows loaded together (one after the other they are two round trips to
    // memory), added up against a running maximum.
    float mx = -INFINITY, den = 0.0f;
    float acc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = 0.0f;
#pragma unroll 1
    for (int c0 = c_lo; c0 <= c_hi; c0 += 4) {
      float l[4], x[4][E];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = c0 + k <= c_hi;
        const long long slot = slot_of(in ? c0 + k : c_hi);
        const float* src = p.part_o + slot * D + lane * E;
        l[k] = __ldcg(p.part_lse + slot);
#pragma unroll
        for (int e = 0; e < E; e += 2) {
          const float2 v = __ldcg(reinterpret_cast<const float2*>(src + e));
          x[k][e] = v.x;
          x[k][e + 1] = v.y;
        }
        if (!in) l[k] = -INFINITY;
      }
      // Shares whose scores are all -inf count nothing, in front of others as well as behind them (their rows are 0 / 0); NaN
      // passes through: the maxima ignore it, its weight does not.
      const float m = fmaxf(mx, fmaxf(fmaxf(l[0], l[1]), fmaxf(l[2], l[3])));
      const float old = mx == -INFINITY ? 0.0f : __expf(mx - m);
      den *= old;
#pragma unroll
      for (int e = 0; e < E; ++e) acc[e] *= old;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool in = l[k] != -INFINITY;
        const float wgt = in ? __expf(l[k] - m) : 0.0f;
        den += wgt;
#pragma unroll
        for (int e = 0; e < E; ++e) acc[e] = in ? fmaf(wgt, x[k][e], acc[e]) : acc[e];
      }
      mx = m;
    }
    const float inv = 1.0f / den;   // no partial result at all: 0 * inf
    const float lse = end > first ? mx + logf(den) : -INFINITY;
#pragma unroll
    for (int e = 0; e < E; e += 2) {
      const uint32_t two = pack2<kBf16>(acc[e] * inv, acc[e + 1] * inv);
      if (real) *reinterpret_cast<uint32_t*>(orow + e) = two;
    }
    if (real && lane == 0 && p.lse != nullptr) p.lse[(static_cast<long long>(b) * p.heads + h) * p.seq_q + qi] = lse;
  }
}

struct DecodePlan {
  int group, rows, ctas;
  bool counted, sparse;
  long long off_lse, off_cum, bytes;
};

// What a call needs, or an error: the shapes this kernel covers are the ones whose query rows fit one tile.
inline int plan_decode(const AttnB200DecodeArgs* a, int sms, DecodePlan* d) {
  if (a->batch <= 0 || a->heads <= 0 || a->heads_kv <= 0 || a->seq_q <= 0 || a->seq_kv <= 0 || a->heads % a->heads_kv != 0) return ATTN_B200_E_INVALID_ARG;
  if (a->dim != 64 && a->dim != 128) return ATTN_B200_E_UNSUPPORTED;
  d->group = a->heads / a->heads_kv;
  const long long rows = static_cast<long long>(d->group) * a->seq_q;
  d->sparse = a->block_mask != nullptr;
  d->counted = d->sparse || a->seq_lens != nullptr;
  if (rows > (d->counted ? 64 : 128)) return ATTN_B200_E_UNSUPPORTED;
  d->rows = static_cast<int>(rows);
  const long long pairs = static_cast<long long>(a->batch) * a->heads_kv;
  if (d->sparse) {
    if (a->n_blocks <= 0 || a->block_size <= 0) return ATTN_B200_E_INVALID_ARG;
    if (a->block_size < 8 || kDecTile % a->block_size != 0 || a->n_blocks > kDecMaxBlocks) return ATTN_B200_E_UNSUPPORTED;
  }
  if (d->counted && pairs > kDecMaxPairs) return ATTN_B200_E_UNSUPPORTED;
  const long long most = pairs * ((static_cast<long long>(a->seq_kv) + kDecTile - 1) / kDecTile);
  if (most > 0x3fffffff || pairs * rows > 0x3ffffff) return ATTN_B200_E_UNSUPPORTED;
  d->ctas = static_cast<int>(std::min<long long>(sms, most));
  d->off_lse = 2LL * d->ctas * rows * a->dim * 4;
  d->off_cum = d->off_lse + 2LL * d->ctas * rows * 4;
  d->bytes = (d->off_cum + (d->counted ? (pairs + 1) * 4 : 0) + 255) / 256 * 256;
  return ATTN_B200_OK;
}

template <int D, bool kBf16, bool kCounted>
int launch_decode(const AttnB200DecodeArgs* a, const DecodePlan& d, cudaStream_t stream, int* status) {
  using L = DecodeSmem<D, kCounted>;
  CUtensorMap tmQ, tmK, tmV;
  DecodeParams p;
  std::memset(&p, 0, sizeof(p));
  int rc = encode_rows_map(&tmQ, &p.oq, a->q, a->dtype, D, a->batch, a->seq_q, a->heads, a->q_stride, a->seq_q, d.group);
  if (rc != ATTN_B200_OK) return rc;
  const int box = d.sparse ? a->block_size : kDecTile;
  rc = encode_rows_map(&tmK, &p.ok, a->k, a->dtype, D, a->batch, a->seq_kv, a->heads_kv, a->k_stride, box);
  if (rc != ATTN_B200_OK) return rc;
  rc = encode_rows_map(&tmV, &p.ov, a->v, a->dtype, D, a->batch, a->seq_kv, a->heads_kv, a->v_stride, box);
  if (rc != ATTN_B200_OK) return rc;
  p.o = a->o;
  p.lse = a->lse;
  p.o_sb = a->o_stride[0];
  p.o_ss = a->o_stride[1];
  p.o_sh = a->o_stride[2];
  p.batch = a->batch;
  p.heads = a->heads;
  p.heads_kv = a->heads_kv;
  p.group = d.group;
  p.seq_q = a->seq_q;
  p.seq_kv = a->seq_kv;
  p.rows = d.rows;
  p.rows_pad = (d.rows + 7) / 8 * 8;
  p.q_bytes = (D / 64) * p.rows_pad * 128;
  p.q_bufs = 2 * p.q_bytes <= L::kQRegion ? 2 : 1;
  p.head_major = p.oq.pos_s < p.oq.pos_h ? 1 : 0;
  p.block_mask = a->block_mask;
  p.seq_lens = a->seq_lens;
  p.n_blocks = a->n_blocks;
  p.block = a->block_size;
  p.part_o = static_cast<float*>(a->workspace);
  p.part_lse = reinterpret_cast<float*>(static_cast<uint8_t*>(a->workspace) + d.off_lse);
  p.cum = reinterpret_cast<int*>(static_cast<uint8_t*>(a->workspace) + d.off_cum);
  p.status = status;
  p.fa.f[0] = a->scale;
  auto kernel = decode_fwd_kernel<D, kBf16, kCounted>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes) != cudaSuccess) {
    cudaGetLastError();
    return ATTN_B200_E_LAUNCH;
  }
  if (!launch_pdl(kernel, dim3(d.ctas), dim3(kDecThreads), L::kBytes, stream, tmQ, tmK, tmV, p)) return ATTN_B200_E_LAUNCH;
  const long long pairs = static_cast<long long>(a->batch) * a->heads_kv;
  // every share of a dense call is whole pairs: nothing to merge
  if (!d.counted && pairs % d.ctas == 0) return ATTN_B200_OK;
  const dim3 merge_grid(static_cast<unsigned>((pairs * d.rows + 3) / 4));
  return launch_pdl(decode_merge_kernel<D, kBf16>, merge_grid, dim3(128), 0, stream, p, d.ctas, d.counted ? 1 : 0) ? ATTN_B200_OK : ATTN_B200_E_LAUNCH;
}

}  // namespace b200

extern "C" {

int64_t attn_b200_decode_workspace_bytes(const AttnB200DecodeArgs* a) {
  if (a == nullptr) return -1;
  b200::DecodePlan d;
  const int sms = b200::device_sms();
  if (sms <= 0) return -1;
  return b200::plan_decode(a, sms, &d) == ATTN_B200_OK ? d.bytes : -1;
}

int attn_b200_decode_fwd(const AttnB200DecodeArgs* a, void* cuda_stream) {
  if (a == nullptr || a->q == nullptr || a->k == nullptr || a->v == nullptr || a->o == nullptr) return ATTN_B200_E_INVALID_ARG;
  if (a->dtype != ATTN_B200_DTYPE_FP16 && a->dtype != ATTN_B200_DTYPE_BF16) return ATTN_B200_E_INVALID_ARG;
  const int sms = b200::device_sms();
  if (sms <= 0) return ATTN_B200_E_LAUNCH;
  b200::DecodePlan d;
  const int rc = b200::plan_decode(a, sms, &d);
  if (rc != ATTN_B200_OK) return rc;
  if ((reinterpret_cast<uintptr_t>(a->o) & 15) != 0) return ATTN_B200_E_UNSUPPORTED;
  for (int i = 0; i < 3; ++i)
    if (a->o_stride[i] % 8 != 0) return ATTN_B200_E_UNSUPPORTED;
  if (a->workspace == nullptr || a->workspace_bytes < d.bytes || (reinterpret_cast<uintptr_t>(a->workspace) & 15) != 0) return ATTN_B200_E_WORKSPACE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return ATTN_B200_E_LAUNCH;
  int* status = b200::device_status_word(dev);
  if (status == nullptr) return ATTN_B200_E_LAUNCH;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  const bool bf16 = a->dtype == ATTN_B200_DTYPE_BF16;
#define ATTN_B200_DECODE(DIM)                                                                                                  \
  return d.counted ? (bf16 ? b200::launch_decode<DIM, true, true>(a, d, stream, status) : b200::launch_decode<DIM, false, true>(a, d, stream, status)) \
                  : (bf16 ? b200::launch_decode<DIM, true, false>(a, d, stream, status) : b200::launch_decode<DIM, false, false>(a, d, stream, status))
  if (a->dim == 64) { ATTN_B200_DECODE(64); }
  ATTN_B200_DECODE(128);
#undef ATTN_B200_DECODE
}

}  // extern "C"
