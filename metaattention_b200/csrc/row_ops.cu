// Row passes around the linear-attention backward (sm_100a), which adds up fp32 partial results of the forward kernel.
// torch does each step as a pass of its own (slice + contiguous, add, cast, multiply, sum); here each is one pass.
//   rows_copy16:    dst[o][s'][0:width] = src[o][s][col0:col0+width],  s' = reverse ? seq-1-s : s   (16-bit elements)
//   rows_sum_cast:  dst16[o][s'][:]     = a[o][s][:] (+ b[o][s][:])                                 (fp32 -> fp16 / bf16)
//   decay_grad:     dq, dk as rows_sum_cast, and the gradient of the log-decays from the same reads
#include <cstdint>

#include "../../include/attn_b200.h"
#include "common_host.cuh"
#include "sm100.cuh"

namespace b200 {

__global__ void __launch_bounds__(256) rows_copy16_kernel(const uint16_t* src, uint16_t* dst, long long rows,
                                                         int seq, int src_cols, int col0, int width, int reverse) {
  pdl_launch_dependents();
  pdl_wait();
  const int vpr = width / 8;   // 16-byte vectors per row
  const long long total = rows * vpr;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / vpr;
    const int v = static_cast<int>(i - r * vpr);
    const long long o = r / seq;
    const int s = static_cast<int>(r - o * seq);
    const long long rd = o * seq + (reverse ? seq - 1 - s : s);
    const uint4 x = *reinterpret_cast<const uint4*>(src + r * src_cols + col0 + v * 8);
    *reinterpret_cast<uint4*>(dst + rd * width + v * 8) = x;
  }
}

template <bool kBf16>
__global__ void __launch_bounds__(256) rows_sum_cast_kernel(const float* a, const float* b,
                                                           uint16_t* dst, long long rows, int seq, int cols, int reverse) {
  pdl_launch_dependents();
  pdl_wait();
  const int vpr = cols / 8;
  const long long total = rows * vpr;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / vpr;
    const int v = static_cast<int>(i - r * vpr);
    const long long o = r / seq;
    const int s = static_cast<int>(r - o * seq);
    const long long rd = o * seq + (reverse ? seq - 1 - s : s);
    const float4* pa = reinterpret_cast<const float4*>(a + r * cols + v * 8);
    float4 x0 = pa[0], x1 = pa[1];
    if (b != nullptr) {
      const float4* pb = reinterpret_cast<const float4*>(b + r * cols + v * 8);
      const float4 y0 = pb[0], y1 = pb[1];
      x0.x += y0.x; x0.y += y0.y; x0.z += y0.z; x0.w += y0.w;
      x1.x += y1.x; x1.y += y1.y; x1.z += y1.z; x1.w += y1.w;
    }
    uint4 pk;
    pk.x = pack2<kBf16>(x0.x, x0.y);
    pk.y = pack2<kBf16>(x0.z, x0.w);
    pk.z = pack2<kBf16>(x1.x, x1.y);
    pk.w = pack2<kBf16>(x1.z, x1.w);
    *reinterpret_cast<uint4*>(dst + rd * cols + v * 8) = pk;
  }
}

// Gradient of the log-decays (see the header).  A warp per row reads the fp32 results and the operands once, rounds the
// gradients and leaves the row's term; torch took six passes over [rows, cols] fp32 for the same (93 us of 2 x 8 x 2000 x
// 128, now 16 with the scan below).  Bound by HBM.
template <bool kBf16>
__global__ void __launch_bounds__(256) decay_grad_rows_kernel(const uint16_t* q, const uint16_t* k,
                                                             const float* dq_a, const float* dq_b,
                                                             const float* dk_a, const float* dk_b,
                                                             uint16_t* dq, uint16_t* dk,
                                                             float* row_term, long long rows, int cols) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  for (long long r = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
    float term = 0.0f;
    for (int c = lane * 4; c < cols; c += 128) {
      const long long at = r * cols + c;
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        float4 x = *reinterpret_cast<const float4*>((side == 0 ? dq_a : dk_a) + at);
        const float* second = side == 0 ? dq_b : dk_b;
        if (second != nullptr) {
          const float4 y = *reinterpret_cast<const float4*>(second + at);
          x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
        }
        const uint2 w = *reinterpret_cast<const uint2*>((side == 0 ? q : k) + at);
        float2 w0, w1;
        if constexpr (kBf16) {
          w0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.x));
          w1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w.y));
        } else {
          w0 = __half22float2(*reinterpret_cast<const __half2*>(&w.x));
          w1 = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
        }
        const float dot = fmaf(w0.x, x.x, fmaf(w0.y, x.y, fmaf(w1.x, x.z, w1.y * x.w)));
        term += side == 0 ? dot : -dot;
        *reinterpret_cast<uint2*>((side == 0 ? dq : dk) + at) = make_uint2(pack2<kBf16>(x.x, x.y), pack2<kBf16>(x.z, x.w));
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) term += __shfl_xor_sync(0xffffffffu, term, d);
    if (lane == 0) row_term[r] = term;
  }
}

// dg[t] = sum of row_term from t to the end: a CTA per sequence, from the last 1024 tokens to the first, the sum so far
// carried along.
__global__ void __launch_bounds__(1024) decay_grad_scan_kernel(const float* row_term, float* dg, int seq) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* in = row_term + static_cast<long long>(blockIdx.x) * seq;
  float* out = dg + static_cast<long long>(blockIdx.x) * seq;
  float carry = 0.0f;
  for (int end = seq; end > 0; end -= 1024) {
    const int t = end - 1 - static_cast<int>(threadIdx.x);
    float x = t >= 0 ? in[t] : 0.0f;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) warp_sum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      float y = warp_sum[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const float z = __shfl_up_sync(0xffffffffu, y, d);
        if (lane >= d) y += z;
      }
      warp_sum[lane] = y;
    }
    __syncthreads();
    x += carry + (warp > 0 ? warp_sum[warp - 1] : 0.0f);
    if (t >= 0) out[t] = x;
    carry += warp_sum[31];
    __syncthreads();
  }
}

inline unsigned row_ops_grid(long long total_vectors) {
  const long long blocks = (total_vectors + 255) / 256;
  const long long cap = 148LL * 16;   // a multiple of the SM count; the loops stride over the rest
  return static_cast<unsigned>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

}  // namespace b200

extern "C" {

int attn_b200_rows_copy16(const void* src, void* dst, int64_t outer, int32_t seq, int32_t src_cols, int32_t col0, int32_t width,
                          int32_t reverse, void* cuda_stream) {
  if (src == nullptr || dst == nullptr || outer <= 0 || seq <= 0 || width <= 0) return ATTN_B200_E_INVALID_ARG;
  if (col0 < 0 || col0 + width > src_cols) return ATTN_B200_E_INVALID_ARG;
  if (width % 8 != 0 || col0 % 8 != 0 || src_cols % 8 != 0) return ATTN_B200_E_UNSUPPORTED;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) != 0) return ATTN_B200_E_UNSUPPORTED;
  const long long rows = static_cast<long long>(outer) * seq;
  return b200::launch_pdl(b200::rows_copy16_kernel, dim3(b200::row_ops_grid(rows * (width / 8))), dim3(256), 0,
                          static_cast<cudaStream_t>(cuda_stream), static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst), rows, seq, src_cols,
                          col0, width, reverse)
             ? ATTN_B200_OK
             : ATTN_B200_E_LAUNCH;
}

int attn_b200_linear_decay_grad(const void* q, const void* k, const float* dq_a, const float* dq_b, const float* dk_a,
                                const float* dk_b, void* dq, void* dk, float* row_term, float* dg, int32_t dtype, int64_t outer,
                                int32_t seq, int32_t cols, void* cuda_stream) {
  if (q == nullptr || k == nullptr || dq_a == nullptr || dk_a == nullptr || dq == nullptr || dk == nullptr || row_term == nullptr ||
      dg == nullptr || outer <= 0 || seq <= 0 || cols <= 0)
    return ATTN_B200_E_INVALID_ARG;
  if (dtype != ATTN_B200_DTYPE_FP16 && dtype != ATTN_B200_DTYPE_BF16) return ATTN_B200_E_INVALID_ARG;
  if (cols % 4 != 0 || outer > 0x7fffffff) return ATTN_B200_E_UNSUPPORTED;
  uintptr_t bits = 0;
  for (const void* ptr : {q, k, static_cast<const void*>(dq_a), static_cast<const void*>(dq_b), static_cast<const void*>(dk_a),
                          static_cast<const void*>(dk_b), static_cast<const void*>(dq), static_cast<const void*>(dk)})
    bits |= reinterpret_cast<uintptr_t>(ptr);
  if ((bits & 15) != 0) return ATTN_B200_E_UNSUPPORTED;
  const long long rows = static_cast<long long>(outer) * seq;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  const unsigned grid = b200::row_ops_grid(rows * 32);
  auto kernel = dtype == ATTN_B200_DTYPE_BF16 ? b200::decay_grad_rows_kernel<true> : b200::decay_grad_rows_kernel<false>;
  if (!b200::launch_pdl(kernel, dim3(grid), dim3(256), 0, stream, static_cast<const uint16_t*>(q), static_cast<const uint16_t*>(k), dq_a, dq_b, dk_a,
                        dk_b, static_cast<uint16_t*>(dq), static_cast<uint16_t*>(dk), row_term, rows, cols))
    return ATTN_B200_E_LAUNCH;
  return b200::launch_pdl(b200::decay_grad_scan_kernel, dim3(static_cast<unsigned>(outer)), dim3(1024), 0, stream, row_term, dg, seq) ? ATTN_B200_OK
                                                                                                                                   : ATTN_B200_E_LAUNCH;
}

int attn_b200_rows_sum_cast(const float* a, const float* b, void* dst, int32_t dtype, int64_t outer, int32_t seq, int32_t cols,
                            int32_t reverse, void* cuda_stream) {
  if (a == nullptr || dst == nullptr || outer <= 0 || seq <= 0 || cols <= 0) return ATTN_B200_E_INVALID_ARG;
  if (dtype != ATTN_B200_DTYPE_FP16 && dtype != ATTN_B200_DTYPE_BF16) return ATTN_B200_E_INVALID_ARG;
  if (cols % 8 != 0) return ATTN_B200_E_UNSUPPORTED;
  if (((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(dst)) & 15) != 0)
    return ATTN_B200_E_UNSUPPORTED;
  const long long rows = static_cast<long long>(outer) * seq;
  const unsigned grid = b200::row_ops_grid(rows * (cols / 8));
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  auto kernel = dtype == ATTN_B200_DTYPE_BF16 ? b200::rows_sum_cast_kernel<true> : b200::rows_sum_cast_kernel<false>;
  return b200::launch_pdl(kernel, dim3(grid), dim3(256), 0, stream, a, b, static_cast<uint16_t*>(dst), rows, seq, cols, reverse) ? ATTN_B200_OK
                                                                                                                                : ATTN_B200_E_LAUNCH;
}

}  // extern "C"
