// Hand-tuned functors of the parallel pattern.  A functor is the device-side
// form of (score_mod, OnlineFunc.online_fwd, OnlineFunc.online_fwd_epilogue):
//
//   kRowScales   number of running per-row values (OnlineFunc.online_rowscales)
//   kFinal       number of per-row outputs        (OnlineFunc.final_rowscales)
//   kUnitOScale  o_scale is identically 1: the accumulator is never rescaled
//   kNegInfMask  masked positions are pre-filled with -inf before score_mod
//                (mask_value "-inf" of the reference, attn_tl.py:140-153)
//   init(rs, ctx)                  initial row-scale values
//   tile<N>(s, rs, ctx) -> o_scale in-place score tile -> probabilities for one row
//   kSplitSum, tile_pieces  instead of tile(): rows that several threads share, see SoftmaxFunctor
//   kRowEpilogue epilogue() reduces over the columns it is given: it gets a whole row of dim_v
//   kFiniteTail  with kUnitOScale: tile() makes finite values of what stands for keys past the end of the sequence
//   epilogue<N>(o, rs, ctx)        in-place transform of N accumulator columns
//   final_rowscale(i, rs, ctx)     i-th per-row output
//   combine(i, n, fin, ...)        split-KV: weight of split i among n (OnlineFunc.combine), from all splits' final
//                                  row scales; kCombinedFinal / combined_final(): the call's final row scale 0 after
//                                  the combine, where the functor can give one
//
// Functors for arbitrary user DAGs are generated by core/lower/functor.py and
// obey the same interface.
#pragma once

#include "parallel_fwd.cuh"

namespace b200 {

// Online softmax, the pattern of examples/mha.py:26-83 of the reference
// (score_mod = score*scale; m_new = max(m, rowmax); p = exp(s - m_new);
//  r = r*exp(m - m_new) + rowsum(p); o_scale = exp(m - m_new);
//  epilogue o/r, lse = log(r) + m).
// Evaluated in the exp2 domain with the scale folded into one FMA per
// element.  The running maximum used as exponent reference only moves when
// the true maximum has grown by more than 2^8: p stays below 256 and the
// accumulator rescale (a TMEM round trip) becomes rare.  The result is
// unchanged because numerator and denominator share the reference.
//   fa.f[0] = scale
struct SoftmaxFunctor {
  static constexpr int kRowScales = 2;  // rs[0] = reference max of raw scores, rs[1] = running sum
  static constexpr int kFinal = 1;      // lse
  static constexpr bool kUnitOScale = false;
  static constexpr bool kNegInfMask = true;
  static constexpr bool kRowEpilogue = false;

  __device__ static void init(float* rs, const RowCtx&) {
    rs[0] = -1.0e30f;  // stands for -inf; finite so that differences stay finite
    rs[1] = 0.0f;
  }

  // One tile of a row, or of the part of it that this thread holds (N columns): `row_max` turns the maximum of this
  // thread's columns into the row's; rs[kSplitSum], its sum, stays the part of this thread until the row is finished.
  // Each piece (N / kPieces columns) is handed to `store_piece(index)` as soon as its probabilities are final, so that it
  // is on its way to tensor memory while the next piece's exponentials run.  Multiply-adds and sums go two elements to
  // an instruction and the maximum three: with two or four warps to a scheduler this stage is bound by the
  // special-function unit (16 exponentials a cycle) and, in long calls, by the power it draws; prefill of
  // 8 x 32 x 4096 x 128 causal 1203 -> 1165 us against one element to an instruction, with the same bits.  kPacked false: one
  // element to an instruction.  A thread with a whole row of 128 columns (the decode kernel, bound by memory) has no room
  // for the aligned register pairs: 20 to 96 bytes of spills in its instances, none without.
  static constexpr int kSplitSum = 1;
  template <int N, int kPieces, bool kPacked = true, class RowMax, class StorePiece>
  __device__ static float tile_pieces(float (&s)[N], float* rs, const RowCtx& c, RowMax&& row_max, StorePiece&& store_piece) {
    static_assert(N % (4 * kPieces) == 0 && N % 8 == 0, "pieces of whole groups");
    const float c2 = c.fa->f[0] * 1.4426950408889634f;
    float mx0 = s[0], mx1 = s[1], mx2 = s[2], mx3 = s[3];
#pragma unroll
    for (int i = 4; i + 8 <= N; i += 8) {
      mx0 = max3(mx0, s[i], s[i + 4]);
      mx1 = max3(mx1, s[i + 1], s[i + 5]);
      mx2 = max3(mx2, s[i + 2], s[i + 6]);
      mx3 = max3(mx3, s[i + 3], s[i + 7]);
    }
    mx0 = max3(mx0, s[N - 4], s[N - 3]);
    mx1 = max3(mx1, s[N - 2], s[N - 1]);
    const float mx = row_max(fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)));
    float m_ref = rs[0];
    float o_scale = 1.0f;
    if ((mx - m_ref) * c2 > 8.0f) {
      o_scale = fast_exp2((m_ref - mx) * c2);
      m_ref = mx;
      rs[0] = mx;
      rs[1] *= o_scale;
    }
    const float neg = -m_ref * c2;
    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
    for (int hf = 0; hf < kPieces; ++hf) {
#pragma unroll
      for (int i = hf * (N / kPieces); i < (hf + 1) * (N / kPieces); i += 4) {
        if constexpr (kPacked) {
          fma_x2(s[i], s[i + 1], c2, c2, neg, neg);
          fma_x2(s[i + 2], s[i + 3], c2, c2, neg, neg);
        } else {
#pragma unroll
          for (int k = i; k < i + 4; ++k) s[k] = fmaf(s[k], c2, neg);
        }
        s[i] = fast_exp2(s[i]);
        s[i + 1] = fast_exp2(s[i + 1]);
        s[i + 2] = fast_exp2(s[i + 2]);
        s[i + 3] = fast_exp2(s[i + 3]);
        if constexpr (kPacked) {
          add_x2(a0, a1, s[i], s[i + 1]);
          add_x2(a2, a3, s[i + 2], s[i + 3]);
        } else {
          a0 += s[i];
          a1 += s[i + 1];
          a2 += s[i + 2];
          a3 += s[i + 3];
        }
      }
      store_piece(hf);
    }
    rs[1] += (a0 + a1) + (a2 + a3);
    return o_scale;
  }

  template <int N>
  __device__ static void epilogue(float (&o)[N], const float* rs, const RowCtx&) {
    const float inv = 1.0f / rs[1];
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] *= inv;
  }

  __device__ static float final_rowscale(int, const float* rs, const RowCtx& c) {
    return logf(rs[1]) + rs[0] * c.fa->f[0];
  }

  // Split-KV: weight of split i among n, from the splits' final row scales fin[final * final_stride + split *
  // split_stride] (here one: the log-sum-exp).  w_i = exp(lse_i - lse), lse = log sum_k exp(lse_k): the combine of
  // examples/mha_decode.py:69-77 with natural exponentials.  An empty split has lse = -inf and weight 0.
  static constexpr bool kCombinedFinal = true;
  __device__ static float combined_final(int n, const float* fin, long long split_stride, long long) {
    float mx = -INFINITY;
    for (int k = 0; k < n; ++k) mx = fmaxf(mx, fin[k * split_stride]);
    float den = 0.f;
    for (int k = 0; k < n; ++k) den += __expf(fin[k * split_stride] - mx);
    return mx + __logf(den);
  }
  __device__ static float combine(int i, int n, const float* fin, long long split_stride, long long final_stride) {
    const float li = fin[i * split_stride];
    if (li == -INFINITY) return 0.0f;
    return __expf(li - combined_final(n, fin, split_stride, final_stride));
  }
};

}  // namespace b200
