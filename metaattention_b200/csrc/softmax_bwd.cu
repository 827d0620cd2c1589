// Backward of softmax attention for sm_100a (head dims 128 / 128 or 64 / 64, 16-bit inputs, fp32 accumulation).
//
//   P  = exp(scale * Q K^T - lse)            (recomputed from the forward's log-sum-exp, masked like the forward)
//   dV = P^T dO
//   dP = dO V^T,   delta_i = sum_d dO_id O_id,   dS = P o (dP - delta) * scale
//   dK = dS^T Q,   dQ = dS K
//
// the algorithm of the reference's generated backward (attention_engine/core/template/tl_template/attn/attn_tl.py:
// preprocess :212-244 = delta, main kernel :309-503 = dK/dV per KV tile with atomic adds into an fp32 dQ, postprocess
// :246-275 = dQ to 16 bits; autograd wrapper :669-694), for the built-in softmax.  Differences: three launches
// without atomics or an fp32 dQ buffer -- (1) delta and log2-domain lse into a padded scratch, (2) one CTA per KV tile
// accumulating dK and dV over the query tiles, (3) one CTA per query tile accumulating dQ over the KV tiles (S and dP
// are computed a second time there: 7 tile products instead of 5 for no read-modify-write traffic on dQ; (2) and (3) are
// one launch).  Their kernel template is attn_bwd.cuh, shared with the lowered functors.
#include "attn_bwd.cuh"

namespace b200 {

// The built-in softmax: P = exp2(s * scale * log2e - lse2), dS = P (dP - delta) * scale; the scale is left to the
// finished dK and dQ rows.
struct SoftmaxBwdFunctor {
  static constexpr bool kUsesStats = true, kFiniteTail = false;
  static constexpr bool kNegInfMask = true;
  struct Ctx {
    float c2, scale;
  };
  __device__ static Ctx make(const BwdParams& p) { return Ctx{p.scale * 1.4426950408889634f, p.scale}; }
  __device__ static void score(float s, float lse2, const Ctx& c, int, int, int, int, float& p_out, float& g_out) {
    p_out = g_out = fast_exp2(fmaf(s, c.c2, -lse2));
  }
  // For the N columns of a row, two to an instruction; kColumns: one statistic per column, else one for the row.
  template <int N, bool kColumns>
  __device__ static void score_row(float (&s)[N], float (&g)[N], const float* lse2, const Ctx& c) {
#pragma unroll
    for (int k = 0; k < N; k += 4) {
      const float4 l = kColumns ? *reinterpret_cast<const float4*>(lse2 + k) : make_float4(*lse2, *lse2, *lse2, *lse2);
      fma_x2(s[k], s[k + 1], c.c2, c.c2, -l.x, -l.y);
      fma_x2(s[k + 2], s[k + 3], c.c2, c.c2, -l.z, -l.w);
#pragma unroll
      for (int i = k; i < k + 4; ++i) s[i] = g[i] = fast_exp2(s[i]);
    }
  }
  template <int N, bool kColumns>
  __device__ static void grad_row(const float (&g)[N], float (&dp)[N], const float* delta) {
#pragma unroll
    for (int k = 0; k < N; k += 4) {
      const float4 d = kColumns ? *reinterpret_cast<const float4*>(delta + k) : make_float4(*delta, *delta, *delta, *delta);
      add_x2(dp[k], dp[k + 1], -d.x, -d.y);
      add_x2(dp[k + 2], dp[k + 3], -d.z, -d.w);
      mul_x2(dp[k], dp[k + 1], g[k], g[k + 1]);
      mul_x2(dp[k + 2], dp[k + 3], g[k + 2], g[k + 3]);
    }
  }
  __device__ static float out_scale(const Ctx& c) { return c.scale; }
};

// delta[b,h,s] = sum_d dO[b,s,h,d] * O[b,s,h,d] and lse2 = lse * log2(e), both padded to whole tiles (delta 0,
// lse2 +inf past the end).  attn_tl.py:212-244 of the reference computes the same delta.  Bound by reading o and dO once:
// a block takes 32 tokens x 8 heads, heads fastest, so that its reads run through memory in 2 KB pieces (D = 128); D / 8
// lanes share a row, 16 bytes each, four rows of a lane group in flight; results leave through shared memory as whole
// lines per head.  One warp per row with 4-byte loads and tokens fastest took 160 us on 4 x 32 x 4096 x 128, this one
// 56 us (268 MB: 42 us at the copy rate).
constexpr int kPrepTokens = 32, kPrepHeads = 8;

template <bool kBf16, int D, bool kAligned>
__global__ void __launch_bounds__(256) bwd_prepare_kernel(const void* o, const void* d_o,
                                                        const float* lse, float* delta,
                                                        float* lse2, int heads, int seq_q, int seq_q_pad, long long o_sb,
                                                        long long o_ss, long long o_sh, long long do_sb, long long do_ss, long long do_sh) {
  constexpr int G = D / 8;             // lanes of a row
  constexpr int kGroups = 256 / G;     // rows a block reads at a time
  constexpr int kRows = kPrepTokens * kPrepHeads;
  __shared__ float acc_s[kPrepHeads][kPrepTokens + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int s0 = blockIdx.x * kPrepTokens, h0 = blockIdx.y * kPrepHeads, b = blockIdx.z;
  const int grp = threadIdx.x / G, l = threadIdx.x % G;
  auto load = [&](const void* base, long long off) -> uint4 {
    const uint16_t* src = static_cast<const uint16_t*>(base) + off + l * 8;
    if constexpr (kAligned) return *reinterpret_cast<const uint4*>(src);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
    return make_uint4(w[0], w[1], w[2], w[3]);
  };
  auto dot2 = [](uint32_t a, uint32_t c, float acc) {
    float a0, a1, c0, c1;
    if constexpr (kBf16) {
      const float2 x = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&a)), y = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&c));
      a0 = x.x; a1 = x.y; c0 = y.x; c1 = y.y;
    } else {
      const float2 x = __half22float2(*reinterpret_cast<__half2*>(&a)), y = __half22float2(*reinterpret_cast<__half2*>(&c));
      a0 = x.x; a1 = x.y; c0 = y.x; c1 = y.y;
    }
    return fmaf(a0, c0, fmaf(a1, c1, acc));
  };
#pragma unroll
  for (int r0 = 0; r0 < kRows; r0 += 4 * kGroups) {
    uint4 x[4], y[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + u * kGroups + grp, s = s0 + r / kPrepHeads, h = h0 + r % kPrepHeads;
      const bool in = s < seq_q && h < heads;
      x[u] = in ? load(o, b * o_sb + s * o_ss + h * o_sh) : make_uint4(0u, 0u, 0u, 0u);
      y[u] = in ? load(d_o, b * do_sb + s * do_ss + h * do_sh) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + u * kGroups + grp;
      float acc = dot2(x[u].x, y[u].x, dot2(x[u].y, y[u].y, dot2(x[u].z, y[u].z, dot2(x[u].w, y[u].w, 0.0f))));
#pragma unroll
      for (int d = G / 2; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
      if (l == 0) acc_s[r % kPrepHeads][r / kPrepHeads] = acc;
    }
  }
  __syncthreads();
  static_assert(kRows == 256 && kPrepTokens == 32, "one warp per head writes a line of tokens");
  const int h = h0 + (threadIdx.x >> 5), s = s0 + (threadIdx.x & 31);
  if (h < heads && s < seq_q_pad) {
    const long long bh = static_cast<long long>(b) * heads + h;
    delta[bh * seq_q_pad + s] = acc_s[threadIdx.x >> 5][threadIdx.x & 31];
    // rows past the end, and rows whose mask kept nothing (lse = -inf), get P = 0 everywhere
    const float v = s < seq_q ? lse[bh * seq_q + s] : INFINITY;
    lse2[bh * seq_q_pad + s] = v == -INFINITY ? INFINITY : v * 1.4426950408889634f;
  }
}

template <bool kBf16, int D>
int launch_softmax_bwd(const AttnB200SoftmaxBwdArgs* a, const BwdCall& call_in, cudaStream_t stream, int* status) {
  const int T = kBwdT;
  const int seq_q_pad = (a->seq_q + T - 1) / T * T;
  const long long rows = static_cast<long long>(a->batch) * a->heads * seq_q_pad;
  float* delta = static_cast<float*>(a->workspace);
  float* lse2 = delta + rows;
  {
    bool aligned = ((reinterpret_cast<uintptr_t>(a->o) | reinterpret_cast<uintptr_t>(a->d_o)) & 15) == 0;
    for (int d = 0; d < 3; ++d) aligned = aligned && a->o_stride[d] % 8 == 0 && a->do_stride[d] % 8 == 0;
    const dim3 grid((seq_q_pad + kPrepTokens - 1) / kPrepTokens, (a->heads + kPrepHeads - 1) / kPrepHeads, a->batch);
    auto kernel = aligned ? bwd_prepare_kernel<kBf16, D, true> : bwd_prepare_kernel<kBf16, D, false>;
    if (!launch_pdl(kernel, grid, dim3(256), 0, stream, a->o, a->d_o, a->lse, delta, lse2, a->heads, a->seq_q, seq_q_pad, a->o_stride[0], a->o_stride[1],
                    a->o_stride[2], a->do_stride[0], a->do_stride[1], a->do_stride[2]))
      return ATTN_B200_E_LAUNCH;
  }
  BwdCall call = call_in;
  call.lse2 = lse2;
  call.delta = delta;
  return launch_attn_bwd<SoftmaxBwdFunctor, kBf16, D>(call, stream, status);
}

}  // namespace b200

extern "C" {

int64_t attn_b200_softmax_bwd_workspace_bytes(const AttnB200SoftmaxBwdArgs* a) {
  if (a == nullptr || a->batch <= 0 || a->heads <= 0 || a->seq_q <= 0) return -1;
  const int64_t seq_q_pad = (static_cast<int64_t>(a->seq_q) + b200::kBwdT - 1) / b200::kBwdT * b200::kBwdT;
  return 2 * static_cast<int64_t>(a->batch) * a->heads * seq_q_pad * 4;
}

int attn_b200_softmax_bwd(const AttnB200SoftmaxBwdArgs* a, void* cuda_stream) {
  if (a == nullptr || a->o == nullptr || a->lse == nullptr) return ATTN_B200_E_INVALID_ARG;
  if (a->dim_qk != a->dim_v) return ATTN_B200_E_UNSUPPORTED;
  b200::BwdCall call{};
  if (!b200::bwd_mask_of(a->mask_kind, a->mask_left, a->mask_right, a->mask_bits_q, a->mask_bits_kv, a->mask_tiles_q, a->mask_tiles_kv, call)) return ATTN_B200_E_UNSUPPORTED;
  call.q = a->q; call.k = a->k; call.v = a->v; call.d_o = a->d_o;
  call.dq = a->dq; call.dk = a->dk; call.dv = a->dv;
  call.batch = a->batch; call.heads = a->heads; call.heads_kv = a->heads_kv > 0 ? a->heads_kv : a->heads;
  call.seq_q = a->seq_q; call.seq_kv = a->seq_kv; call.dim = a->dim_qk; call.dtype = a->dtype;
  call.scale = a->scale;
  call.q_stride = a->q_stride; call.k_stride = a->k_stride; call.v_stride = a->v_stride; call.do_stride = a->do_stride;
  call.dq_stride = a->dq_stride; call.dk_stride = a->dk_stride; call.dv_stride = a->dv_stride;
  const int rc = b200::validate_bwd_call(call);
  if (rc != ATTN_B200_OK) return rc;
  for (int d = 0; d < 3; ++d)
    if (a->o_stride[d] % 2 != 0 || a->do_stride[d] % 2 != 0) return ATTN_B200_E_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(a->o) & 3) != 0 || (reinterpret_cast<uintptr_t>(a->d_o) & 3) != 0) return ATTN_B200_E_UNSUPPORTED;
  const int64_t need = attn_b200_softmax_bwd_workspace_bytes(a);
  if (a->workspace == nullptr || a->workspace_bytes < need || (reinterpret_cast<uintptr_t>(a->workspace) & 15) != 0)
    return ATTN_B200_E_WORKSPACE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return ATTN_B200_E_LAUNCH;
  int* status = b200::device_status_word(dev);
  if (status == nullptr) return ATTN_B200_E_LAUNCH;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  const bool bf16 = a->dtype == ATTN_B200_DTYPE_BF16;
  if (a->dim_qk == 64)
    return bf16 ? b200::launch_softmax_bwd<true, 64>(a, call, stream, status) : b200::launch_softmax_bwd<false, 64>(a, call, stream, status);
  return bf16 ? b200::launch_softmax_bwd<true, 128>(a, call, stream, status) : b200::launch_softmax_bwd<false, 128>(a, call, stream, status);
}

}  // extern "C"
