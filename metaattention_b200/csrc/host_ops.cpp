// Host side of a call in native code: from tensors to the argument structs of include/attn_b200.h, outputs and scratch from
// torch's allocator, the launch on the current stream, and the autograd functions.
//
// A short call's kernel runs for 5 to 30 microseconds; filling a ctypes struct field by field in Python took 35 to 50, and a
// forward and backward through Python autograd functions 220.  Everything here works on what the engine decided once at
// construction (`Plan`) and on the shapes and strides of this call.  Nothing is kept between calls but the plan's copies of
// its mask on each device.
//
// A call whose operands are not what a kernel takes is declined (`None` / false): the Python side then raises the error
// that names what is wrong.  Entry points of libattn_b200.so and of functor libraries come in as addresses, from the
// libraries that Python has loaded.
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <ATen/cuda/CUDAContext.h>
#include <torch/csrc/Exceptions.h>
#include <torch/extension.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <memory>
#include <tuple>

#include "../../include/attn_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = c10::optional<Tensor>;

struct Api {
  int (*parallel_fwd)(const AttnB200ParallelArgs*, void*) = nullptr;
  int64_t (*decode_bytes)(const AttnB200DecodeArgs*) = nullptr;
  int (*decode_fwd)(const AttnB200DecodeArgs*, void*) = nullptr;
  int64_t (*decode_tiles_bytes)(int32_t, int32_t, int32_t) = nullptr;
  int (*decode_tiles)(const uint8_t*, const int32_t*, int32_t, int32_t, int32_t, int32_t, int32_t, void*, int64_t, void*) = nullptr;
  int64_t (*softmax_bwd_bytes)(const AttnB200SoftmaxBwdArgs*) = nullptr;
  int (*softmax_bwd)(const AttnB200SoftmaxBwdArgs*, void*) = nullptr;
  int (*status_word)(int32_t, int32_t**) = nullptr;
  int64_t (*linear_bytes)(const AttnB200LinearArgs*) = nullptr;
  int (*linear_fwd)(const AttnB200LinearArgs*, void*) = nullptr;
  decltype(&attn_b200_linear_decay_grad) linear_decay_grad = nullptr;
  decltype(&attn_b200_rows_sum_cast) rows_sum_cast = nullptr;
  int (*mla_plan)(const AttnB200MlaShape*, int32_t, int32_t*) = nullptr;
  int64_t (*mla_bytes)(const AttnB200MlaShape*, int32_t) = nullptr;
  int32_t (*mla_num_parts)(int32_t, int32_t) = nullptr;
  int (*mla_decode)(const AttnB200MlaArgs*, void*) = nullptr;
} api;

template <class F>
void take(F& slot, const py::dict& d, const char* name) {
  slot = reinterpret_cast<F>(py::cast<uintptr_t>(d[name]));
}

PyObject* raise_status = nullptr;   // core.native.lib.check: raises NativeError for a status code; held to the end of the process

void bind(const py::dict& d, py::object check) {
  take(api.parallel_fwd, d, "attn_b200_parallel_fwd");
  take(api.decode_bytes, d, "attn_b200_decode_workspace_bytes");
  take(api.decode_fwd, d, "attn_b200_decode_fwd");
  take(api.decode_tiles_bytes, d, "attn_b200_decode_tiles_bytes");
  take(api.decode_tiles, d, "attn_b200_decode_tiles");
  take(api.softmax_bwd_bytes, d, "attn_b200_softmax_bwd_workspace_bytes");
  take(api.softmax_bwd, d, "attn_b200_softmax_bwd");
  take(api.status_word, d, "attn_b200_device_status_word");
  take(api.linear_bytes, d, "attn_b200_linear_workspace_bytes");
  take(api.linear_fwd, d, "attn_b200_linear_fwd");
  take(api.linear_decay_grad, d, "attn_b200_linear_decay_grad");
  take(api.rows_sum_cast, d, "attn_b200_rows_sum_cast");
  take(api.mla_plan, d, "attn_b200_mla_plan");
  take(api.mla_bytes, d, "attn_b200_mla_workspace_bytes");
  take(api.mla_num_parts, d, "attn_b200_mla_num_parts");
  take(api.mla_decode, d, "attn_b200_mla_decode");
  raise_status = check.release().ptr();
}

// Raises the Python NativeError of a status code; callable without the GIL (autograd threads).
void check(int rc, const char* what) {
  if (rc == ATTN_B200_OK) return;
  py::gil_scoped_acquire gil;
  try {
    py::reinterpret_borrow<py::object>(raise_status)(rc, what);
  } catch (py::error_already_set& e) {
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}

int dtype_code(const Tensor& t) {
  return t.scalar_type() == at::kHalf ? ATTN_B200_DTYPE_FP16 : t.scalar_type() == at::kBFloat16 ? ATTN_B200_DTYPE_BF16 : -1;
}
void strides_bsh(int64_t (&dst)[3], const Tensor& t) {
  for (int i = 0; i < 3; ++i) dst[i] = t.stride(i);
}
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
Tensor f32(at::IntArrayRef size, const Tensor& like) { return at::empty(size, like.options().dtype(at::kFloat)); }
Tensor bytes(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }

// One custom input of a program: per dimension the axis it stands for (0..3 = batch, heads, seq_len, seq_len_kv; -1 = none,
// then `literal` is its declared extent or -1), and the type the functor reads.
struct Custom {
  std::vector<int> axes;
  std::vector<int64_t> literal;
  at::ScalarType dtype;
};

// Block-sparse walk of a mask on one device (core/lower/sparse.py).
struct Sparse {
  Tensor keep, partial, mask_base, elem_mask, bits_q, bits_kv, tiles_q, tiles_kv;
  int batch = 1, heads = 1, rows = 128;

  // Around a launch on the current stream: the tensors go when the engine does, perhaps with that launch still to run.
  static void used(const Tensor& q, std::initializer_list<const Tensor*> by_it) {
    const auto now = c10::cuda::getCurrentCUDAStream(q.device().index());
    for (const Tensor* t : by_it)
      if (t->defined()) c10::cuda::CUDACachingAllocator::recordStream(t->storage().data_ptr(), now);
  }
  void used_by_forward(const Tensor& q) const { used(q, {&keep, &partial, &mask_base, &elem_mask}); }
  void used_by_backward(const Tensor& q) const { used(q, {&bits_q, &bits_kv, &tiles_q, &tiles_kv}); }
};

// What an engine of the parallel pattern decided at construction.
struct Plan {
  bool builtin = false;        // the built-in softmax; else `fn` is attn_b200_parallel_fwd_jit of its functor library
  uintptr_t fn = 0;
  std::vector<float> fparams;
  int n_final = 0;
  int mask_kind = 0, left = 0, right = 0;
  bool may_decode = false;     // attn_b200_decode_fwd computes this program
  bool may_split = false;      // results over parts of the KV sequence merge into the whole one
  int decode_block = 0;        // > 0: block_mask / cache_seqlens arrive with the call
  bool has_mask_walk = false;  // a general mask_mod, evaluated for mask_q x mask_kv positions of mask_bh (batch, head) pairs
  int64_t mask_q = 0, mask_kv = 0, mask_bh = 1;
  std::vector<Custom> custom;
  int backward = 0;            // 0 none, 1 softmax, 2 elementwise
  py::object load_mask;        // device -> dict of tensors
  py::object load_backward;    // () -> address of attn_b200_elementwise_bwd_jit
  std::atomic<uintptr_t> bwd_fn{0};   // loaded by the first backward; autograd runs one thread per device
  std::map<int, std::shared_ptr<const Sparse>> masks;

  std::shared_ptr<const Sparse> mask_on(const Tensor& like) {   // with the GIL
    const int dev = like.device().index();
    auto it = masks.find(dev);
    if (it != masks.end()) return it->second;
    py::dict d = load_mask(like.device());
    Sparse s;
    auto get = [&](const char* k, Tensor& t) {
      if (d.contains(k) && !d[k].is_none()) t = py::cast<Tensor>(d[k]);
    };
    get("keep", s.keep); get("partial", s.partial); get("mask_base", s.mask_base); get("elem_mask", s.elem_mask);
    get("bits_q", s.bits_q); get("bits_kv", s.bits_kv); get("tiles_q", s.tiles_q); get("tiles_kv", s.tiles_kv);
    s.batch = py::cast<int>(d["batch"]);
    s.heads = py::cast<int>(d["heads"]);
    s.rows = py::cast<int>(d["mask_rows"]);
    return masks.emplace(dev, std::make_shared<const Sparse>(std::move(s))).first->second;
  }
};

// The call-time masks of a decode as the types the library reads; false = not a shape it takes.
bool decode_operands(OptTensor& block_mask, OptTensor& lens, int64_t B, int64_t Hkv, const Tensor& q) {
  if (block_mask.has_value()) {
    Tensor& m = *block_mask;
    if (m.dim() != 3 || m.size(0) != B || m.size(1) != Hkv) return false;
    if (m.device() != q.device()) m = m.to(q.device());
    m = m.contiguous();
    m = m.scalar_type() == at::kBool ? m.view(at::kByte) : m.to(at::kByte);
  }
  if (lens.has_value()) {
    if (lens->numel() != B) return false;
    lens = lens->to(q.device(), at::kInt).contiguous();
  }
  return true;
}

struct Forward {
  bool done = false;
  std::shared_ptr<const Sparse> mask;   // the general mask it ran under, kept for the backward
  Tensor o;
  std::vector<Tensor> finals;   // empty when split results were merged without them
};

int splits_on(int64_t B, int64_t H, int64_t Sq, int64_t Skv, int64_t sms) {
  // 1 unless the (query tile pair, head, batch) grid fills less than half of the SMs; then as many as fit, each keeping at
  // least four 128-row KV tiles (a split re-reads Q and adds a combine pass)
  const int64_t ctas = B * H * ((Sq + 255) / 256);
  const int64_t tiles = (Skv + 127) / 128;
  if (ctas <= 0 || 2 * ctas > sms || tiles < 8) return 1;   // nothing to compute: nothing to split
  return static_cast<int>(std::max<int64_t>(1, std::min({sms / ctas, tiles / 4, int64_t{65535} / std::max<int64_t>(B, 1)})));
}
int kv_splits_for(int64_t B, int64_t H, int64_t Sq, int64_t Skv, int device) {
  return splits_on(B, H, Sq, Skv, at::cuda::getDeviceProperties(device)->multiProcessorCount);
}

// What is wrong with the extents of a call's 4-dimensional operands, or null.  The kernels walk k and v with the batch and
// head dim of q and the length of k: an operand that has less would be read past its end.  One that has more is read in
// part (caches laid out for more sequences).
const char* fault(const Plan& plan, const Tensor& q, const Tensor& k, const Tensor& v) {
  if (q.numel() == 0 || k.numel() == 0 || v.numel() == 0) return "q, k and v must not be empty";
  if (k.size(0) < q.size(0) || v.size(0) < q.size(0)) return "k and v hold fewer sequences than q";
  if (k.size(3) < q.size(3)) return "k has a smaller head dim than q";
  if (v.size(1) < k.size(1)) return "v is shorter than k";
  if (plan.has_mask_walk) {
    // The bitmaps have a row of `words` words per query tile, the rows of the (batch, head) pairs one after the other: a
    // call may be shorter than what the mask was evaluated for where that leaves the rows in their places.
    const int64_t Sq = q.size(1), Skv = k.size(1);
    auto tiles = [](int64_t n) { return (n + 127) / 128; };
    auto words = [&](int64_t n) { return (tiles(n) + 31) / 32; };
    if (Sq > plan.mask_q || Skv > plan.mask_kv) return "longer than the lengths that mask_mod was evaluated for";
    if ((plan.mask_bh > 1 && tiles(Sq) != tiles(plan.mask_q)) || (words(Skv) != words(plan.mask_kv) && (plan.mask_bh > 1 || tiles(Sq) > 1)))
      return "too much shorter than the lengths that mask_mod was evaluated for";
  }
  return nullptr;
}

// The forward of one call; `done` false = declined.  `mask`: the plan's on q's device, if it has one.
Forward forward(const Plan& plan, const std::shared_ptr<const Sparse>& mask, const Tensor& q, const Tensor& k, const Tensor& v,
                const std::vector<Tensor>& custom, int forced_splits, OptTensor block_mask, OptTensor lens) {
  Forward r;
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4 || fault(plan, q, k, v) != nullptr) return r;
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device()) return r;
  const int dt = dtype_code(q);
  if (dt < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return r;
  if (q.stride(3) != 1 || k.stride(3) != 1 || v.stride(3) != 1) return r;
  const int64_t B = q.size(0), Sq = q.size(1), H = q.size(2), D = q.size(3), Skv = k.size(1), Hkv = k.size(2), Dv = v.size(3);
  if (Hkv <= 0 || v.size(2) != Hkv || H % Hkv != 0 || custom.size() != plan.custom.size()) return r;
  c10::cuda::CUDAGuard guard(q.device());
  void* stream = stream_of(q);
  if (plan.decode_block == 0) {   // nothing is made of them: they are not in a form a kernel takes
    block_mask.reset();
    lens.reset();
  }

  if (plan.may_decode && forced_splits < 0 && Sq * H <= 128 * Hkv && Skv > 128 && D == Dv) {
    // the query rows of the heads that share a KV head fit one tile: the decode kernel, if it covers the call
    OptTensor bm = block_mask, ln = lens;
    if (plan.decode_block > 0 && !decode_operands(bm, ln, B, Hkv, q)) return r;
    AttnB200DecodeArgs a;
    std::memset(&a, 0, sizeof(a));
    a.batch = B; a.heads = H; a.heads_kv = Hkv; a.seq_q = Sq; a.seq_kv = Skv; a.dim = D; a.dtype = dt; a.scale = plan.fparams[0];
    if (bm.has_value()) {
      a.block_mask = bm->data_ptr<uint8_t>();
      a.n_blocks = bm->size(2);
      a.block_size = plan.decode_block;
    }
    if (ln.has_value()) a.seq_lens = ln->data_ptr<int32_t>();
    const int64_t need = api.decode_bytes(&a);
    if (need >= 0) {
      Tensor ws = bytes(need, q), lse = f32({B, H, Sq}, q);
      r.o = at::empty({B, Sq, H, Dv}, q.options());
      a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = r.o.data_ptr();
      a.lse = lse.data_ptr<float>();
      a.workspace = ws.data_ptr();
      a.workspace_bytes = need;
      strides_bsh(a.q_stride, q); strides_bsh(a.k_stride, k); strides_bsh(a.v_stride, v); strides_bsh(a.o_stride, r.o);
      check(api.decode_fwd(&a, stream), "attn_b200_decode_fwd");
      r.finals.push_back(lse);
      r.done = true;
      return r;
    }
  }

  AttnB200ParallelArgs a;
  std::memset(&a, 0, sizeof(a));
  // custom inputs: addressed by strides alone, so a named axis must have extent 1 (broadcast) or exactly the call's
  const int64_t extent[4] = {B, H, Sq, Skv};
  std::vector<Tensor> held;
  for (size_t c = 0; c < custom.size(); ++c) {
    const Custom& spec = plan.custom[c];
    Tensor t = custom[c];
    if (!t.defined() || t.dim() != static_cast<int64_t>(spec.axes.size()) || (t.is_cuda() && t.device() != q.device())) return r;
    for (size_t d = 0; d < spec.axes.size(); ++d) {
      const int64_t n = t.size(d);
      if (spec.axes[d] < 0 ? (n != 1 || (spec.literal[d] >= 0 && spec.literal[d] != n)) : (n != 1 && n != extent[spec.axes[d]])) return r;
    }
    t = t.to(q.device(), spec.dtype);
    for (size_t d = 0; d < spec.axes.size(); ++d)
      if (spec.axes[d] >= 0 && t.size(d) > 1) a.custom_stride[c][spec.axes[d]] = t.stride(d);
    a.custom[c] = t.data_ptr();
    held.push_back(std::move(t));
  }

  Tensor tiles;   // call-time block_mask / cache_seqlens as tile bitmaps and column masks
  if (plan.decode_block > 0) {
    if (!decode_operands(block_mask, lens, B, Hkv, q)) return r;
    const int64_t nt = (Skv + 127) / 128, words = (nt + 31) / 32, bh = B * Hkv;
    const int64_t need = api.decode_tiles_bytes(B, Hkv, Skv);
    tiles = bytes(need, q);
    check(api.decode_tiles(block_mask.has_value() ? block_mask->data_ptr<uint8_t>() : nullptr, lens.has_value() ? lens->data_ptr<int32_t>() : nullptr, B,
                           Hkv, block_mask.has_value() ? block_mask->size(2) : 0, plan.decode_block, Skv, tiles.data_ptr(), need, stream),
          "attn_b200_decode_tiles");
    uint32_t* col = static_cast<uint32_t*>(tiles.data_ptr());
    a.elem_mask = col;
    a.tile_keep = col + bh * nt * 4;
    a.tile_partial = col + bh * nt * 4 + bh * words;
    a.sparse_batch = B;
    a.sparse_heads = Hkv;
  } else if (plan.has_mask_walk) {
    r.mask = mask;
    const Sparse& s = *mask;
    s.used_by_forward(q);
    a.tile_keep = static_cast<const uint32_t*>(s.keep.data_ptr());
    a.tile_partial = static_cast<const uint32_t*>(s.partial.data_ptr());
    a.tile_mask_base = s.mask_base.defined() ? s.mask_base.data_ptr<int32_t>() : nullptr;
    a.elem_mask = s.elem_mask.defined() ? static_cast<const uint32_t*>(s.elem_mask.data_ptr()) : nullptr;
    a.sparse_batch = s.batch;
    a.sparse_heads = s.heads;
    a.elem_mask_rows = s.rows;
  }

  r.o = at::empty({B, Sq, H, Dv}, q.options());
  for (int i = 0; i < plan.n_final; ++i) {
    r.finals.push_back(f32({B, H, Sq}, q));
    a.final_rowscales[i] = r.finals.back().data_ptr<float>();
  }
  // split-KV when the launch would leave most SMs idle; the split results are added up with the weights of the functor's
  // combine (lowered functors: the user's, which needs every split to be non-empty, i.e. no mask).  A program without one
  // whose results do not add up is split on demand only
  int splits = 1;
  Tensor ws;
  if (a.tile_keep == nullptr && Dv <= 128 && D <= 128 && (plan.builtin || plan.mask_kind == ATTN_B200_MASK_NONE)) {
    splits = forced_splits >= 0 ? forced_splits : plan.may_split ? kv_splits_for(B, H, Sq, Skv, q.device().index()) : 1;
    if (splits > 1 && !plan.builtin) {
      const int64_t nt = (Skv + 127) / 128, per = (nt + std::min<int64_t>(splits, nt) - 1) / std::min<int64_t>(splits, nt);
      splits = (nt + per - 1) / per;   // no split without KV tiles
    }
    if (splits > 1) {
      ws = bytes(B * splits * H * Sq * (Dv + ATTN_B200_MAX_ROWSCALES) * 4, q);
      a.workspace = ws.data_ptr();
      a.workspace_bytes = ws.numel();
    }
  }
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = r.o.data_ptr();
  a.batch = B; a.heads = H; a.seq_q = Sq; a.seq_kv = Skv; a.dim_qk = D; a.dim_v = Dv; a.heads_kv = Hkv;
  strides_bsh(a.q_stride, q); strides_bsh(a.k_stride, k); strides_bsh(a.v_stride, v); strides_bsh(a.o_stride, r.o);
  a.dtype = dt;
  a.mask_kind = plan.mask_kind;
  a.mask_left = plan.left;
  a.mask_right = plan.right;
  a.functor = ATTN_B200_FUNCTOR_SOFTMAX;
  a.num_splits = splits;
  for (size_t i = 0; i < plan.fparams.size() && i < 8; ++i) a.fparams[i] = plan.fparams[i];
  if (plan.builtin) {
    check(api.parallel_fwd(&a, stream), "attn_b200_parallel_fwd");
  } else {
    int32_t* status = nullptr;
    check(api.status_word(q.device().index(), &status), "attn_b200_device_status_word");
    auto fn = reinterpret_cast<int (*)(const AttnB200ParallelArgs*, void*, int32_t*)>(plan.fn);
    check(fn(&a, stream, status), "attn_b200_parallel_fwd_jit");
    if (splits > 1) r.finals.clear();   // the combine gives output weights only
  }
  r.done = true;
  return r;
}

// ---------------------------------------------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------------------------------------------

Tensor grad_like(const Tensor& t) {   // the strides of t where its last dimension is contiguous and it has no holes
  Tensor g = at::empty_like(t);
  return g.stride(3) == 1 ? g : at::empty(t.sizes(), t.options());
}

struct Mask {
  int kind, left, right;
  Tensor bits_q, bits_kv, tiles_q, tiles_kv;
};

template <class Args>
void fill_bwd(Args& a, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& d_o, const Tensor& dq, const Tensor& dk, const Tensor& dv,
              const Mask& m) {
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.d_o = d_o.data_ptr();
  a.dq = dq.data_ptr(); a.dk = dk.data_ptr(); a.dv = dv.data_ptr();
  a.batch = q.size(0); a.heads = q.size(2); a.heads_kv = k.size(2); a.seq_q = q.size(1); a.seq_kv = k.size(1);
  a.dim_qk = q.size(3); a.dim_v = v.size(3);
  a.dtype = dtype_code(q);
  a.mask_kind = m.kind;
  a.mask_left = m.left;
  a.mask_right = m.right;
  if (m.bits_q.defined()) {
    const int64_t nq = (q.size(1) + 127) / 128, nk = (k.size(1) + 127) / 128;
    const std::vector<int64_t> want_q{nq * 128, nk, 4}, want_kv{nk * 128, nq, 4};
    if (m.bits_q.sizes() != want_q || m.bits_kv.sizes() != want_kv)
      check(ATTN_B200_E_INVALID_ARG, "backward at other lengths than mask_mod was evaluated for");
    a.mask_kind = ATTN_B200_MASK_BITS;
    a.mask_bits_q = m.bits_q.data_ptr();
    a.mask_bits_kv = m.bits_kv.data_ptr();
    if (m.tiles_q.defined()) {
      if (m.tiles_q.numel() != nq * ((nk + 31) / 32) || m.tiles_kv.numel() != nk * ((nq + 31) / 32))
        check(ATTN_B200_E_INVALID_ARG, "backward with bitmaps of other lengths than the call's");
      a.mask_tiles_q = m.tiles_q.data_ptr();
      a.mask_tiles_kv = m.tiles_kv.data_ptr();
    }
  }
  strides_bsh(a.q_stride, q); strides_bsh(a.k_stride, k); strides_bsh(a.v_stride, v); strides_bsh(a.do_stride, d_o);
  strides_bsh(a.dq_stride, dq); strides_bsh(a.dk_stride, dk); strides_bsh(a.dv_stride, dv);
}

std::vector<Tensor> softmax_bwd_one(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& d_o,
                                    float scale, const Mask& m) {
  Tensor dq = grad_like(q), dk = grad_like(k), dv = grad_like(v);
  AttnB200SoftmaxBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  fill_bwd(a, q, k, v, d_o, dq, dk, dv, m);
  a.o = o.data_ptr();
  a.lse = lse.data_ptr<float>();
  a.scale = scale;
  strides_bsh(a.o_stride, o);
  const int64_t need = api.softmax_bwd_bytes(&a);
  Tensor ws = bytes(std::max<int64_t>(need, 16), q);
  a.workspace = ws.data_ptr();
  a.workspace_bytes = need;
  check(api.softmax_bwd(&a, stream_of(q)), "attn_b200_softmax_bwd");
  return {dq, dk, dv};
}

std::vector<Tensor> elementwise_bwd_one(uintptr_t fn, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& d_o,
                                        const std::vector<Tensor>& custom, const Mask& m) {
  Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(k.sizes(), k.options()), dv = at::empty(v.sizes(), v.options());
  AttnB200ElementwiseBwdArgs a;
  std::memset(&a, 0, sizeof(a));
  fill_bwd(a, q, k, v, d_o, dq, dk, dv, m);
  std::vector<Tensor> held;
  for (size_t i = 0; i < custom.size() && i < ATTN_B200_MAX_CUSTOM; ++i) {
    held.push_back(custom[i].to(q.device(), at::kFloat).contiguous());
    a.custom[i] = held.back().data_ptr();
  }
  int32_t* status = nullptr;
  check(api.status_word(q.device().index(), &status), "attn_b200_device_status_word");
  check(reinterpret_cast<int (*)(const AttnB200ElementwiseBwdArgs*, void*, int32_t*)>(fn)(&a, stream_of(q), status), "attn_b200_elementwise_bwd_jit");
  return {dq, dk, dv};
}

// dim_v a multiple of dim_qk: the backward is linear in dP = dO V^T and in delta, sums over the columns of v, and dV's
// columns are independent: one run per dim_qk-wide column slice, dQ and dK added up in fp32
template <class Run>
std::vector<Tensor> over_dim_v(const Tensor& q, const Tensor& v, const Run& run) {
  const int64_t D = q.size(3), Dv = v.size(3);
  if (Dv == D) return run(0, D);
  Tensor dq, dk;
  std::vector<Tensor> dvs;
  for (int64_t c = 0; c < Dv; c += D) {
    auto part = run(c, D);
    dq = dq.defined() ? dq + part[0].to(at::kFloat) : part[0].to(at::kFloat);
    dk = dk.defined() ? dk + part[1].to(at::kFloat) : part[1].to(at::kFloat);
    dvs.push_back(part[2]);
  }
  return {dq.to(q.scalar_type()), dk.to(q.scalar_type()), at::cat(dvs, -1)};
}

Tensor cols(const Tensor& t, int64_t c, int64_t w) { return t.size(3) == w ? t : t.narrow(3, c, w); }

std::vector<Tensor> softmax_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& d_o, float scale,
                                const Mask& m) {
  return over_dim_v(q, v, [&](int64_t c, int64_t w) {
    return softmax_bwd_one(q, k, cols(v, c, w), cols(o, c, w), lse, cols(d_o, c, w), scale, m);
  });
}

// Of a k or v larger than the call, gradients of what the forward left unread would not be written.
void whole(const Tensor& q, const Tensor& k, const Tensor& v) {
  if (k.size(0) != q.size(0) || v.size(0) != q.size(0) || k.size(3) != q.size(3) || v.size(1) != k.size(1) || v.size(2) != k.size(2))
    check(ATTN_B200_E_INVALID_ARG, "backward with k or v of another batch, length or head dim than the call");
}

Tensor last_contiguous(Tensor t, const Tensor& like) {
  if (t.scalar_type() != like.scalar_type()) t = t.to(like.scalar_type());
  return t.stride(3) == 1 ? t : t.contiguous();
}

// What a backward needs beside the saved tensors.  The mask's tensors belong to the plan: they are no variables of the
// graph (saved ones would go through the user's saved-tensor hooks, and may not have been made in inference mode).
struct PlanRef : torch::CustomClassHolder {
  std::shared_ptr<Plan> plan;
  std::shared_ptr<const Sparse> mask;
};

// The forward with its backward (attn_b200_softmax_bwd, attn_b200_elementwise_bwd_jit): the counterpart of the reference's
// `_attention` autograd function (core/template/tl_template/attn/attn_tl.py:654-694).  Outputs: o, then the final row
// scales, which carry no gradient.
struct Attention : torch::autograd::Function<Attention> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const std::shared_ptr<Plan>& plan, const Forward& done,
                                                const Tensor& q, const Tensor& k, const Tensor& v, const std::vector<Tensor>& custom) {
    auto ref = c10::make_intrusive<PlanRef>();
    ref->plan = plan;
    ref->mask = done.mask;
    ctx->saved_data["plan"] = c10::IValue::make_capsule(ref);
    torch::autograd::variable_list saved{q, k, v};
    if (plan->backward == 1) {
      saved.push_back(done.o);
      saved.push_back(done.finals[0]);
    } else {
      for (const Tensor& t : custom) saved.push_back(t);
    }
    ctx->save_for_backward(saved);
    torch::autograd::variable_list out{done.o};
    for (const Tensor& t : done.finals) out.push_back(t);
    ctx->mark_non_differentiable(done.finals);
    ctx->set_materialize_grads(false);   // nobody reads the zeros that would be made for them
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto ref = c10::static_intrusive_pointer_cast<PlanRef>(ctx->saved_data["plan"].toCapsule());
    const std::shared_ptr<Plan>& plan = ref->plan;
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
    whole(q, k, v);
    c10::cuda::CUDAGuard guard(q.device());
    Tensor g = grads[0].defined() ? grads[0] : at::zeros({q.size(0), q.size(1), q.size(2), v.size(3)}, q.options());
    const Tensor d_o = last_contiguous(g, q);
    Mask m{plan->mask_kind, plan->left, plan->right, {}, {}, {}, {}};
    if (ref->mask != nullptr) {
      ref->mask->used_by_backward(q);
      m.bits_q = ref->mask->bits_q; m.bits_kv = ref->mask->bits_kv; m.tiles_q = ref->mask->tiles_q; m.tiles_kv = ref->mask->tiles_kv;
    }
    std::vector<Tensor> d;
    if (plan->backward == 1) {
      d = softmax_bwd(q, k, v, saved[3], saved[4], d_o, plan->fparams[0], m);
    } else {
      if (plan->bwd_fn == 0) {   // compiled when a gradient is first asked for
        py::gil_scoped_acquire gil;
        try {
          plan->bwd_fn = py::cast<uintptr_t>(plan->load_backward());
        } catch (py::error_already_set& e) {
          e.restore();
          python_error err;
          err.persist();
          throw err;
        }
      }
      const std::vector<Tensor> custom(saved.begin() + 3, saved.end());
      d = over_dim_v(q, v, [&](int64_t c, int64_t w) {
        return elementwise_bwd_one(plan->bwd_fn, q, k, cols(v, c, w), cols(d_o, c, w), custom, m);
      });
    }
    return {Tensor(), Tensor(), d[0], d[1], d[2], Tensor()};   // one entry per argument of forward
  }
};

// One call of an engine: None (declined) or [o, final row scales...].  `grad`: the call is recorded for the backward.
py::object run(const std::shared_ptr<Plan>& plan, const Tensor& q, const Tensor& k, const Tensor& v, const std::vector<Tensor>& custom,
               int forced_splits, const OptTensor& block_mask, const OptTensor& lens, bool grad) {
  std::shared_ptr<const Sparse> mask;
  if (plan->has_mask_walk && q.is_cuda()) {
    c10::cuda::CUDAGuard guard(q.device());
    at::AutoDispatchBelowADInplaceOrView below;
    mask = plan->mask_on(q);   // calls Python the first time
  }
  std::vector<Tensor> results;
  {
    py::gil_scoped_release others_run;   // a launch waits while the stream's queue is full
    Forward f;
    {
      at::AutoDispatchBelowADInplaceOrView below;   // outputs are made, nothing is recorded
      f = forward(*plan, mask, q, k, v, custom, forced_splits, block_mask, lens);
    }
    if (f.done && grad) {
      results = Attention::apply(plan, f, q, k, v, custom);
    } else if (f.done) {
      results.push_back(std::move(f.o));
      for (Tensor& t : f.finals) results.push_back(std::move(t));
    }
  }
  if (results.empty()) return py::none();
  py::list out;
  for (Tensor& t : results) out.append(std::move(t));
  return out;
}

// The softmax backward by itself (core.native.lib.softmax_bwd, which has looked at types, devices and strides).  `bits`:
// empty, or bits_q, bits_kv and optionally tiles_q, tiles_kv of a general mask.
std::vector<Tensor> softmax_bwd_call(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& d_o,
                                     float scale, int kind, int left, int right, const std::vector<Tensor>& bits) {
  whole(q, k, v);
  if (o.size(0) != q.size(0) || o.size(1) != q.size(1) || o.size(2) != q.size(2) || o.size(3) != v.size(3) || d_o.sizes() != o.sizes() ||
      lse.numel() != q.size(0) * q.size(1) * q.size(2))
    check(ATTN_B200_E_INVALID_ARG, "backward with o, lse or a gradient of another shape than the output");
  c10::cuda::CUDAGuard guard(q.device());
  Mask m{kind, left, right, {}, {}, {}, {}};
  if (bits.size() >= 2) {
    m.bits_q = bits[0];
    m.bits_kv = bits[1];
  }
  if (bits.size() == 4) {
    m.tiles_q = bits[2];
    m.tiles_kv = bits[3];
  }
  py::gil_scoped_release others_run;
  at::AutoDispatchBelowADInplaceOrView below;
  return softmax_bwd(q, k, v, o, lse, d_o, scale, m);
}

std::shared_ptr<Plan> make_plan(const py::dict& d) {
  // the last reference may be dropped by an autograd thread: Python objects go under the GIL
  std::shared_ptr<Plan> p(new Plan, [](Plan* x) {
    py::gil_scoped_acquire gil;
    delete x;
  });
  p->builtin = py::cast<bool>(d["builtin"]);
  p->fn = py::cast<uintptr_t>(d["fn"]);
  p->fparams = py::cast<std::vector<float>>(d["fparams"]);
  p->n_final = py::cast<int>(d["n_final"]);
  p->mask_kind = py::cast<int>(d["mask_kind"]);
  p->left = py::cast<int>(d["left"]);
  p->right = py::cast<int>(d["right"]);
  p->may_decode = py::cast<bool>(d["may_decode"]);
  p->may_split = py::cast<bool>(d["may_split"]);
  p->decode_block = py::cast<int>(d["decode_block"]);
  p->has_mask_walk = py::cast<bool>(d["has_mask_walk"]);
  std::tie(p->mask_q, p->mask_kv, p->mask_bh) = py::cast<std::tuple<int64_t, int64_t, int64_t>>(d["mask_extents"]);
  p->backward = py::cast<int>(d["backward"]);
  p->load_mask = d["load_mask"];
  p->load_backward = d["load_backward"];
  for (const auto& item : py::cast<py::list>(d["custom"])) {
    const py::tuple t = py::cast<py::tuple>(item);
    p->custom.push_back({py::cast<std::vector<int>>(t[0]), py::cast<std::vector<int64_t>>(t[1]), py::cast<bool>(t[2]) ? at::kFloat
                                                                                                 : py::cast<bool>(t[3]) ? at::kBFloat16
                                                                                                                        : at::kHalf});
  }
  return p;
}

// ---------------------------------------------------------------------------------------------------------------
// chunked linear attention
// ---------------------------------------------------------------------------------------------------------------

// The row pitch of t [B, H, T, w] if it is a column range of a contiguous [B, H, T, ld] tensor that the kernel can read in
// place (16-byte aligned start, ld a multiple of 8), else 0.
int64_t column_range_ld(const Tensor& t) {
  const int64_t ld = t.stride(2), T = t.size(2);
  return t.stride(3) == 1 && ld > t.size(3) && ld % 8 == 0 && t.stride(1) == T * ld && t.stride(0) == t.size(1) * T * ld &&
                 (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0
             ? ld
             : 0;
}

// Why attn_engine/linear_attn_engine.py refuses a call (it words the errors).
enum LinearRefusal { kLinearOk = 0, kLinearShapes, kLinearFit, kLinearDevice, kLinearType, kLinearHeads, kLinearNormalize };

LinearRefusal linear_refusal(const Tensor& q, const Tensor& k, const Tensor& v, bool normalize) {
  if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) return kLinearShapes;
  // the kernel walks k and v with the extents of q: what has others would be read askew or past its end
  if (k.size(3) != q.size(3) || k.size(2) != q.size(2) || v.size(2) != q.size(2) || k.size(0) < q.size(0) || v.size(0) < q.size(0)) return kLinearFit;
  if (!q.is_cuda() || !k.is_cuda() || !v.is_cuda()) return kLinearDevice;
  if (dtype_code(q) < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return kLinearType;
  if (q.size(1) <= 0 || k.size(1) <= 0 || v.size(1) % q.size(1) != 0 || v.size(1) % k.size(1) != 0) return kLinearHeads;
  if (normalize && v.size(3) % 128 != 0) return kLinearNormalize;
  return kLinearOk;
}

struct LinearCall {
  double q_scale, eps;
  bool normalize, f32_out, precise, reverse;
  int segments;
};

Tensor linear_forward(Tensor q, Tensor k, Tensor v, Tensor log_decay, OptTensor v_scale, const LinearCall& c) {
  const int64_t B = q.size(0), T = q.size(2), Dk = q.size(3), H = v.size(1), Dv = v.size(3);
  if (Dv % 8 != 0 || (c.f32_out && Dv % 128 != 0)) {
    // rows of v that are not whole 16-byte pieces, or fp32 rows that are not whole slices: padded with zero columns,
    // which stay zero in the output and are cut off again (otherwise the kernel reads the columns that a slice of 128
    // is short of as zeros)
    Tensor o = linear_forward(q, k, at::constant_pad_nd(v, {0, 128 - Dv % 128}), log_decay, v_scale, c);
    return o.narrow(3, 0, Dv).contiguous();
  }
  // q and k may be column ranges of wider contiguous tensors (the backward's contractions over ranges of dim_v)
  const int64_t q_ld = column_range_ld(q), k_ld = column_range_ld(k);
  if (q_ld == 0) q = q.contiguous();
  if (k_ld == 0) k = k.contiguous();
  v = v.contiguous();
  log_decay = log_decay.to(q.device(), at::kFloat).expand({B, H, T}).contiguous();
  if (v_scale.has_value()) v_scale = v_scale->to(q.device(), at::kFloat).expand({B, H, T}).contiguous();
  c10::cuda::CUDAGuard guard(q.device());
  Tensor o = at::empty({B, H, T, Dv}, c.f32_out ? q.options().dtype(at::kFloat) : q.options());
  AttnB200LinearArgs a;
  std::memset(&a, 0, sizeof(a));
  a.dtype_out = c.f32_out ? ATTN_B200_DTYPE_FP32 : ATTN_B200_DTYPE_SAME;
  a.q = q.data_ptr(); a.k = k.data_ptr(); a.v = v.data_ptr(); a.o = o.data_ptr();
  a.log_decay = log_decay.data_ptr<float>();
  a.v_scale = v_scale.has_value() ? v_scale->data_ptr<float>() : nullptr;
  a.batch = B; a.heads = H; a.seq = T; a.dim_qk = Dk; a.dim_v = Dv;
  a.heads_q = q.size(1); a.heads_k = k.size(1);
  a.q_ld = q_ld; a.k_ld = k_ld;
  a.dtype = dtype_code(q);
  a.normalize = c.normalize; a.precise = c.precise; a.segments = c.segments; a.reverse = c.reverse; a.any_dim_v = 1;
  a.q_scale = c.q_scale; a.norm_eps = c.eps;
  const int64_t need = api.linear_bytes(&a);
  Tensor ws;
  if (need > 0) {
    ws = bytes(need, q);
    a.workspace = ws.data_ptr();
    a.workspace_bytes = need;
  }
  check(api.linear_fwd(&a, stream_of(q)), "attn_b200_linear_fwd");
  return o;
}

// The output, or the number of a refusal.
py::object linear_forward_call(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& log_decay, double q_scale, bool normalize, double eps,
                               bool f32_out, const OptTensor& v_scale, bool precise, int segments, bool reverse) {
  const LinearRefusal why = linear_refusal(q, k, v, normalize);
  if (why != kLinearOk) return py::int_(static_cast<int>(why));
  Tensor o;
  {
    py::gil_scoped_release others_run;
    at::AutoDispatchBelowADInplaceOrView below;
    o = linear_forward(q, k, v, log_decay, v_scale, {q_scale, eps, normalize, f32_out, precise, reverse, segments});
  }
  return py::cast(o);
}

// dq, dk rounded to the dtype of q [B, H, T, cols] and the gradient of the log-decays [B, H, T], from one or two fp32
// partial results each (attn_b200_linear_decay_grad).
std::vector<Tensor> linear_decay_grad(const Tensor& q_in, const Tensor& k_in, const std::vector<Tensor>& dq_in, const std::vector<Tensor>& dk_in) {
  py::gil_scoped_release others_run;
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor q = q_in.contiguous(), k = k_in.contiguous();
  std::vector<Tensor> parts;   // alive until the launch
  auto part = [&](const std::vector<Tensor>& from, size_t i) -> const float* {
    if (i >= from.size()) return nullptr;
    parts.push_back(from[i].contiguous());
    return parts.back().data_ptr<float>();
  };
  const float *dq_a = part(dq_in, 0), *dq_b = part(dq_in, 1), *dk_a = part(dk_in, 0), *dk_b = part(dk_in, 1);
  c10::cuda::CUDAGuard guard(q.device());
  Tensor dq = at::empty_like(q), dk = at::empty_like(k), dg = f32({q.size(0), q.size(1), q.size(2)}, q), term = at::empty_like(dg);
  check(api.linear_decay_grad(q.data_ptr(), k.data_ptr(), dq_a, dq_b, dk_a, dk_b, dq.data_ptr(), dk.data_ptr(), term.data_ptr<float>(),
                              dg.data_ptr<float>(), dtype_code(q), q.size(0) * q.size(1), static_cast<int32_t>(q.size(2)),
                              static_cast<int32_t>(q.size(3)), stream_of(q)),
        "attn_b200_linear_decay_grad");
  return {dq, dk, dg};
}

// a (+ b), fp32 [..., seq, cols], rounded to fp16 or bf16, the rows of every sequence reversed if asked.
Tensor rows_sum_cast(const Tensor& a_in, const OptTensor& b_in, bool bf16, bool reverse) {
  py::gil_scoped_release others_run;
  at::AutoDispatchBelowADInplaceOrView below;
  const Tensor a = a_in.contiguous();
  Tensor b;
  if (b_in.has_value()) b = b_in->contiguous();
  const int64_t cols = a.size(-1), seq = a.size(-2);
  c10::cuda::CUDAGuard guard(a.device());
  Tensor dst = at::empty(a.sizes(), a.options().dtype(bf16 ? at::kBFloat16 : at::kHalf));
  check(api.rows_sum_cast(a.data_ptr<float>(), b.defined() ? b.data_ptr<float>() : nullptr, dst.data_ptr(),
                          bf16 ? ATTN_B200_DTYPE_BF16 : ATTN_B200_DTYPE_FP16, seq * cols > 0 ? a.numel() / (seq * cols) : 0,
                          static_cast<int32_t>(seq), static_cast<int32_t>(cols), reverse ? 1 : 0, stream_of(a)),
        "attn_b200_rows_sum_cast");
  return dst;
}

// ---------------------------------------------------------------------------------------------------------------
// MLA decode
// ---------------------------------------------------------------------------------------------------------------

// [B, R, C] view of a [B, R, C], [B, 1, R, C] or [B, R, 1, C] tensor with contiguous columns.
bool rows_of(const Tensor& t, Tensor& out) {
  out = t;
  if (t.dim() == 4) {
    if (t.size(1) == 1) out = t.select(1, 0);
    else if (t.size(2) == 1) out = t.select(2, 0);
    else return false;
  }
  return out.dim() == 3 && out.stride(2) == 1;
}

// Why attn_engine/mla.py refuses a call (it words the errors).
enum MlaRefusal { kMlaRows = 1, kMlaDevice, kMlaTable, kMlaMaxLen, kMlaLens, kMlaRope, kMlaType, kMlaDims, kMlaSchedule, kMlaOtherSchedule };

struct MlaResult {
  int refusal = 0, num_splits = 0, parts = 0;
  Tensor o, lse;
};

MlaResult mla_decode(const Tensor& q_in, const Tensor& kv_in, int64_t dim_v, double scale, const OptTensor& q_rope, const OptTensor& kv_rope,
                     c10::optional<int64_t> num_splits, const OptTensor& workspace, const OptTensor& lens_in, const OptTensor& table_in,
                     c10::optional<int64_t> max_seqlen, const OptTensor& sched, const OptTensor& sched_cum) {
  MlaResult r;
  auto refuse = [&](int why) {
    r.refusal = why;
    return r;
  };
  Tensor q, kv, qr, kr, table, lens;
  if (!rows_of(q_in, q) || !rows_of(kv_in, kv)) return refuse(kMlaRows);
  if (!q.is_cuda() || !kv.is_cuda()) return refuse(kMlaDevice);
  const int64_t B = q.size(0), H = q.size(1);
  int64_t S = kv.size(1);
  if (table_in.has_value()) {
    table = *table_in;
    if (table.scalar_type() != at::kInt || !table.is_cuda() || table.dim() != 2 || table.size(0) != B) return refuse(kMlaTable);
    if (table.stride(1) != 1) table = table.contiguous();
    const int64_t most = table.size(1) * kv.size(1);
    S = max_seqlen.value_or(most);
    if (S > most) return refuse(kMlaMaxLen);
  }
  if (lens_in.has_value()) {
    if (lens_in->scalar_type() != at::kInt || !lens_in->is_cuda() || lens_in->numel() != B) return refuse(kMlaLens);
    lens = lens_in->contiguous();
  }
  if (q_rope.has_value() != kv_rope.has_value()) return refuse(kMlaRope);
  int64_t rope = 0;
  if (q_rope.has_value()) {
    if (!rows_of(*q_rope, qr) || !rows_of(*kv_rope, kr)) return refuse(kMlaRows);
    rope = qr.size(2);
  }
  if (dtype_code(q) < 0 || kv.scalar_type() != q.scalar_type()) return refuse(kMlaType);
  c10::cuda::CUDAGuard guard(q.device());
  const int sms = at::cuda::getDeviceProperties(q.device().index())->multiProcessorCount;
  AttnB200MlaArgs a;
  std::memset(&a, 0, sizeof(a));
  a.shape.batch = B; a.shape.heads_q = H; a.shape.seq_kv = S; a.shape.dim_qk = q.size(2) + rope; a.shape.dim_v = dim_v;
  int32_t splits = 0;
  if (num_splits.has_value()) splits = static_cast<int32_t>(*num_splits);
  else if (!lens.defined() && !sched.has_value()) check(api.mla_plan(&a.shape, sms, &splits), "attn_b200_mla_plan");
  r.num_splits = splits;
  r.parts = api.mla_num_parts(H, sms);
  const int64_t need = api.mla_bytes(&a.shape, splits);
  if (need < 0) return refuse(kMlaDims);
  Tensor ws;
  if (need > 0) {
    ws = workspace.has_value() && static_cast<int64_t>(workspace->nbytes()) >= need ? *workspace : bytes(need, q);
    a.workspace = ws.data_ptr();
  }
  a.workspace_bytes = need;
  r.o = at::empty({B, H, dim_v}, q.options());
  r.lse = f32({B, H}, q);
  a.q = q.data_ptr(); a.kv = kv.data_ptr(); a.o = r.o.data_ptr();
  a.lse = r.lse.data_ptr<float>();
  for (int i = 0; i < 2; ++i) {
    a.q_stride[i] = q.stride(i);
    a.kv_stride[i] = kv.stride(i);
    if (rope > 0 || qr.defined()) {
      a.q_rope_stride[i] = qr.stride(i);
      a.kv_rope_stride[i] = kr.stride(i);
    }
  }
  if (qr.defined()) {
    a.q_rope = qr.data_ptr();
    a.kv_rope = kr.data_ptr();
  }
  a.num_splits = splits;
  a.dtype = dtype_code(q);
  a.scale = scale;
  if (lens.defined()) a.seq_lens = lens.data_ptr<int32_t>();
  if (splits == 0 && sched.has_value()) {
    if (!sched_cum.has_value() || sched->scalar_type() != at::kInt || sched_cum->scalar_type() != at::kInt) return refuse(kMlaSchedule);
    if (sched->size(0) != r.parts || sched_cum->numel() != B + 1) return refuse(kMlaOtherSchedule);
    a.sched_meta = sched->data_ptr<int32_t>();
    a.sched_num_splits = sched_cum->data_ptr<int32_t>();
    a.sched_parts = r.parts;
  }
  if (table.defined()) {
    a.block_table = table.data_ptr<int32_t>();
    a.block_table_stride = table.stride(0);
    a.page_size = kv.size(1);
    a.num_pages = kv.size(0);
  }
  check(api.mla_decode(&a, stream_of(q)), "attn_b200_mla_decode");
  return r;
}

// (o, lse, splits, parts), or the number of a refusal.
py::object mla_decode_call(const Tensor& q, const Tensor& kv, int64_t dim_v, double scale, const OptTensor& q_rope, const OptTensor& kv_rope,
                           c10::optional<int64_t> num_splits, const OptTensor& workspace, const OptTensor& lens, const OptTensor& table,
                           c10::optional<int64_t> max_seqlen, const OptTensor& sched, const OptTensor& sched_cum) {
  MlaResult r;
  {
    py::gil_scoped_release others_run;
    at::AutoDispatchBelowADInplaceOrView below;
    r = mla_decode(q, kv, dim_v, scale, q_rope, kv_rope, num_splits, workspace, lens, table, max_seqlen, sched, sched_cum);
  }
  if (r.refusal != 0) return py::int_(r.refusal);
  return py::make_tuple(r.o, r.lse, r.num_splits, r.parts);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Plan, std::shared_ptr<Plan>>(m, "Plan");
  m.def("bind", &bind);
  m.def("make_plan", &make_plan);
  m.def("run", &run);
  m.def("softmax_bwd", &softmax_bwd_call);
  m.def("kv_splits", &kv_splits_for);
  m.def("splits_on", &splits_on);
  m.def("fault", &fault);
  m.def("linear_forward", &linear_forward_call);
  m.def("linear_decay_grad", &linear_decay_grad);
  m.def("rows_sum_cast", &rows_sum_cast);
  m.def("mla_decode", &mla_decode_call);
}
