"""``LinearAttentionEngine``: chunked linear attention / retention on the native
sm_100a kernel (reference: attention_engine/attn_engine/linear_attn_engine.py:11-65,
lowering core/lower/lower_linear.py:290-409, wrapper linear_tl.py:1240-1268).

``mod(q, k, v, decay, *custom)`` with q ``[B,HQ,T,Dk]``, k ``[B,HK,T,Dk]``,
v ``[B,H,T,Dv]``, decay ``[B,H,T]`` fp32 returns o ``[B,H,T,Dv]``.

The user's ``decay_mod`` / ``k_mod`` / ``v_mod`` are traced once and applied as
whole-tensor torch operations on the device before the kernel, which is what
the reference does with generated PyTorch statements (lower_linear.py:138-206);
``decay_mod`` must produce the natural log of the per-token decay (RetNet:
``decay.log()``).  A ``q_mod`` of the form ``q * const`` is folded into the
kernel (the reference fuses q_mod into its output kernel, linear_tl.py:368-370);
any other ``q_mod`` is applied like the others.  Tuning arguments are accepted
and ignored.
"""

from __future__ import annotations

import torch

from core.native import lib as native
from core.transform.core import CustomIO, SymbolicArray, SymbolScalar
from core.transform.graph import Var


def _align(a, b):
    """Broadcast rule of the reference's whole-tensor statements (codegen/tl_gen.py:253-262):
    operands are aligned on their LEADING axes; the shorter one gets trailing singleton axes."""
    if isinstance(a, torch.Tensor) and isinstance(b, torch.Tensor) and a.dim() != b.dim():
        if a.dim() < b.dim():
            a = a.reshape(a.shape + (1,) * (b.dim() - a.dim()))
        else:
            b = b.reshape(b.shape + (1,) * (a.dim() - b.dim()))
    return a, b


def eval_tensor_expr(sym: SymbolScalar, env: dict, memo: dict | None = None):
    """Evaluate a traced whole-tensor expression with torch (on whatever device the leaves live)."""
    memo = {} if memo is None else memo
    key = id(sym)
    if key in memo:
        return memo[key]
    if key in env:
        return env[key]
    t = sym.code.type
    if t == "Const":
        val = float(sym.code.value)
    elif t == "Var":
        raise ValueError(f"free variable {sym.code.name!r} in a linear-attention mod")
    else:
        a = [eval_tensor_expr(p, env, memo) for p in sym.prev]
        if len(a) == 2:
            a = list(_align(a[0], a[1]))
        as_t = lambda x: x if isinstance(x, torch.Tensor) else torch.tensor(x)  # noqa: E731
        if t == "Add":
            val = a[0] + a[1]
        elif t == "Sub":
            val = a[0] - a[1]
        elif t == "Mul":
            val = a[0] * a[1]
        elif t == "Div":
            val = a[0] / a[1]
        elif t == "Neg":
            val = -a[0]
        elif t == "Abs":
            val = torch.abs(as_t(a[0]))
        elif t == "Exp":
            val = torch.exp(as_t(a[0]))
        elif t == "Exp2":
            val = torch.exp2(as_t(a[0]))
        elif t == "Log":
            val = torch.log(as_t(a[0]))
        elif t == "Log2":
            val = torch.log2(as_t(a[0]))
        elif t == "Tanh":
            val = torch.tanh(as_t(a[0]))
        elif t == "Max":
            val = torch.maximum(*[x if isinstance(x, torch.Tensor) else torch.tensor(x, device=as_t(a[0]).device if isinstance(a[0], torch.Tensor) else a[1].device, dtype=torch.float32) for x in a])
        else:
            raise NotImplementedError(f"op {t} in a linear-attention mod")
    memo[key] = val
    return val


def _depends_on(sym: SymbolScalar, leaf: SymbolScalar) -> bool:
    return sym is leaf or any(_depends_on(p, leaf) for p in sym.prev)


def _constant_multiple(out: SymbolScalar, leaf: SymbolScalar):
    """If ``out`` is ``leaf * c`` (or ``c * leaf``, ``leaf / c``) for a Python constant c, return c."""
    if out is leaf:
        return 1.0
    if out.code.type in ("Mul", "Div") and len(out.prev) == 2:
        a, b = out.prev
        if a is leaf and b.code.type == "Const":
            c = float(b.code.value)
            return c if out.code.type == "Mul" else 1.0 / c
        if out.code.type == "Mul" and b is leaf and a.code.type == "Const":
            return float(a.code.value)
    return None


def linear_attention_forward(q, k, v, log_decay, q_scale: float = 1.0, normalize: bool = False, eps: float = 1e-5,
                             out_dtype=None, v_scale=None, precise: bool = False, segments: int = 0, reverse: bool = False):
    """q,k: [B,H,T,Dk]; v: [B,H,T,Dv] (fp16/bf16 CUDA); log_decay: [B,H,T] fp32, natural log of the
    per-token decay.  Returns o [B,H,T,Dv] in the input dtype, or in fp32 with ``out_dtype=torch.float32``
    (the kernel's accumulators without the output rounding).  ``normalize`` applies a per-(batch, head,
    token) normalisation over Dv (zero mean, unit variance, no affine) to the output.  ``v_scale`` [B,H,T] (fp32) is a
    per-token factor on the rows of v, applied inside the kernel.  ``precise``: the decayed scores of a block keep a
    16-bit remainder beside their 16-bit value (a second P V pass).  ``segments``: CTAs that share
    a chain's sequence, 0 = planned from the shape (the result has the same bits).  ``reverse``: the sums run over the
    tokens from a row's own to the end of the sequence (see ``_reversed_forward``)."""
    if out_dtype not in (None, q.dtype, torch.float32):
        raise native.NativeError("out_dtype must be the input dtype or torch.float32")
    o = native.host().linear_forward(q, k, v, log_decay, q_scale, normalize, eps, out_dtype == torch.float32, v_scale, precise, segments,
                                     reverse)
    if not isinstance(o, torch.Tensor):
        _refuse(o, q, k, v)
    return o


def _refuse(why: int, q, k, v):
    """The error of a call that the native host side refuses (LinearRefusal in csrc/host_ops.cpp)."""
    (_, _, _, _), (_, _, _, _), (_, _, _, _) = q.shape, k.shape, v.shape
    raise native.NativeError({
        2: f"q, k, v do not fit together: {tuple(q.shape)}, {tuple(k.shape)}, {tuple(v.shape)}",
        3: "linear attention needs CUDA tensors",
        4: "q, k, v must share dtype float16 or bfloat16",
        5: "the heads of v must be a multiple of the heads of q and of k",
        6: "normalize needs dim_v to be a multiple of 128"}[why])


def _reversed_forward(q, k, v, log_decay, q_scale, out_dtype=None, precise=False):
    """o_j = q_scale * sum_{i>=j} exp(G_i - G_j) (q_j . k_i) v_i, G the inclusive cumulative sum of log_decay: the kernel
    walks the sequence from its end.  The same on time-reversed operands, where position u carries the log-decay of token
    T - u (0 for u = 0), is how the composition is followed without a GPU, the oracle in the kernel's place."""
    if q.is_cuda:
        return linear_attention_forward(q, k, v, log_decay, q_scale, out_dtype=out_dtype, precise=precise, reverse=True)
    ld_rev = torch.cat([torch.zeros_like(log_decay[..., :1]), log_decay.flip(-1)[..., :-1]], dim=-1)
    return linear_attention_forward(q.flip(2), k.flip(2), v.flip(2), ld_rev, q_scale, out_dtype=out_dtype, precise=precise).flip(2)


def _sum_cast(parts, dtype):
    """Sum of the partial results, rounded to ``dtype``: one pass for two parts, none for one that has the dtype already."""
    parts = _at_most_two(parts)
    if len(parts) == 1 and parts[0].dtype == dtype:
        return parts[0]
    if parts[0].shape[-1] % 8 == 0:
        return native.rows_sum_cast(parts[0], parts[1] if len(parts) > 1 else None, dtype)
    return (parts[0] + parts[1] if len(parts) > 1 else parts[0]).to(dtype)


def _at_most_two(parts):
    while len(parts) > 2:
        parts = [parts[0] + parts[1]] + parts[2:]
    return parts


def _retention_parts(qc, kc, vc, log_decay, q_scale, precise=False, reverse=False, fp32=True):
    """o_i = q_scale * sum_{j<=i} exp(G_i - G_j) (qc_i . kc_j) vc_j (``reverse``: the sum over j >= i) on the forward
    kernel, for any width of the contraction, as a list of fp32 partial results to be added: the sum is linear in the
    scores, so a contraction wider than the kernel's 256 columns is the sum over column ranges it does cover (widths
    256 / 128 / 64, the last one zero-padded), which the kernel reads in place.  A single result that is only to be
    rounded (``fp32`` = False) leaves the kernel in the operands' dtype."""
    run = _reversed_forward if reverse else linear_attention_forward
    D = qc.shape[-1]
    out_dtype = torch.float32 if fp32 or D > 256 or D not in (64, 128, 256) else None
    parts, start = [], 0
    while start < D:
        width = next((w for w in (256, 128, 64) if D - start >= w), 64)
        have = min(width, D - start)
        qs, ks = qc[..., start:start + have], kc[..., start:start + have]
        if have < width:
            qs, ks = torch.nn.functional.pad(qs, (0, width - have)), torch.nn.functional.pad(ks, (0, width - have))
        parts.append(run(qs, ks, vc, log_decay, q_scale, out_dtype=out_dtype, precise=precise))
        start += width
    return parts


def linear_attention_backward(q, k, v, log_decay, d_o, q_scale: float = 1.0, need_dg: bool = False):
    """(dq, dk, dv[, dg]) of ``linear_attention_forward`` (no normalisation), the job of the reference's three backward
    kernels (core/template/tl_template/linear/linear_tl.py:461-975), as runs of the forward kernel.  With
    D_ij = exp(G_i - G_j) for j <= i:

        dq_i = q_scale * sum_{j<=i} D_ij (do_i . v_j) k_j      = retention(q = do, k = v, v = k)
        dv_j = q_scale * sum_{i>=j} D_ij (q_i . k_j) do_i      = reversed retention(q = k, k = q, v = do)
        dk_j = q_scale * sum_{i>=j} D_ij (do_i . v_j) q_i      = reversed retention(q = v, k = do, v = q)

    The two contractions over dim_v go through ``_retention_parts`` (dim_v may exceed the kernel's 256 columns of dim_qk).

    ``need_dg``: also the gradient with respect to the per-token log-decay, fp32 [B, H, T].  A score A_ij depends on the
    log-decays of tokens j+1..i, so dg_t = sum_{i>=t, j<t} dA_ij A_ij; with dG_i = q_i . dq_i - k_i . dk_i (row sums
    minus column sums of dA o A) that is the reversed cumulative sum of dG — what the reference's dqkg kernel and its
    ``compute_final_dg`` produce per chunk (linear_tl.py:63-76, 638-814).  dg is a difference of sums over dq and dk:
    those runs then keep the 16-bit remainder of their decayed scores, and leave fp32 results for the row sums."""
    d_o = d_o.to(q.dtype)
    B, H, T, _ = q.shape
    q, k, v, d_o = q.contiguous(), k.contiguous(), v.contiguous(), d_o.contiguous()
    ld = log_decay.to(dtype=torch.float32, device=q.device).expand(B, H, T).contiguous()
    dq_parts = _retention_parts(d_o, v, k, ld, q_scale, precise=need_dg, fp32=need_dg)
    dv = _reversed_forward(k, q, d_o, ld, q_scale)
    dk_parts = _retention_parts(v, d_o, q, ld, q_scale, precise=need_dg, reverse=True, fp32=need_dg)
    if not need_dg:
        return _sum_cast(dq_parts, q.dtype), _sum_cast(dk_parts, k.dtype), dv
    dq_parts, dk_parts = _at_most_two(dq_parts), _at_most_two(dk_parts)
    if q.is_cuda and q.shape[-1] % 8 == 0:
        dq, dk, dg = native.linear_decay_grad(q, k, dq_parts, dk_parts)
        return dq, dk, dv, dg
    d_cum = (q.float() * sum(dq_parts)).sum(-1) - (k.float() * sum(dk_parts)).sum(-1)
    return _sum_cast(dq_parts, q.dtype), _sum_cast(dk_parts, k.dtype), dv, d_cum.flip(-1).cumsum(-1).flip(-1)


class _ForwardOnly(torch.autograd.Function):
    @staticmethod
    def forward(ctx, runner, *tensors):
        return runner(*[t.detach() for t in tensors])

    @staticmethod
    def backward(ctx, *grads):
        raise NotImplementedError("the B200-native backend differentiates linear attention only without output "
                                  "normalisation")


class _LinearAttention(torch.autograd.Function):
    """Chunked linear attention of operands that have been through their mods, with its backward
    (``linear_attention_backward``): the counterpart of the kernels inside the reference's ``LinearAttention`` autograd
    function (core/template/tl_template/linear/linear_tl.py:1237-1333).  The reference differentiates the mods with
    generated statements (``*_mod_bwd_expr``, :1322-1329); here they are torch operations in front of this function and
    torch's autograd carries dq, dk, dv and the log-decay's gradient through them, custom inputs included."""

    @staticmethod
    def forward(ctx, q, k, v, log_decay, q_scale):
        o = linear_attention_forward(q.detach(), k.detach(), v.detach(), log_decay.detach(), q_scale=q_scale)
        ctx.save_for_backward(q, k, v, log_decay)
        ctx.q_scale = q_scale
        return o

    @staticmethod
    def backward(ctx, d_o):
        q, k, v, log_decay = ctx.saved_tensors
        B, H, T, _ = v.shape
        hq, hk = q.shape[1], k.shape[1]
        qe = q.repeat_interleave(H // hq, dim=1) if hq != H else q
        ke = k.repeat_interleave(H // hk, dim=1) if hk != H else k
        need_dg = ctx.needs_input_grad[3]
        res = linear_attention_backward(qe, ke, v, log_decay, d_o, ctx.q_scale, need_dg=need_dg)
        dq, dk, dv = res[:3]
        if hq != H:   # heads that shared one q head: their gradients add up
            dq = dq.view(B, hq, H // hq, T, -1).float().sum(2).to(dq.dtype)
        if hk != H:
            dk = dk.view(B, hk, H // hk, T, -1).float().sum(2).to(dk.dtype)
        dg = res[3].sum_to_size(log_decay.shape).to(log_decay.dtype) if need_dg else None
        return dq, dk, dv, dg, None


class LinearAttentionEngine:
    def __init__(self, qkv_meta, q_mod=None, k_mod=None, v_mod=None, decay_mod=None, custom_io=None,
                 tune=False, tune_filename="tune_result", tune_bwd=False):
        self.qkv_meta = qkv_meta
        self.custom_io = custom_io if custom_io is not None else CustomIO()
        self.custom_names = list(self.custom_io.input_tensors.keys())
        self.normalize_output = False
        B, HQ, T, Dk = qkv_meta[0].shape
        self.HK = qkv_meta[1].shape[1]
        self.H = qkv_meta[2].shape[1]
        self.Dv = qkv_meta[2].shape[3]
        if Dk not in (64, 128, 256):
            raise NotImplementedError(f"linear attention kernel covers dim_qk in (64,128,256) (got {Dk})")
        if self.H % HQ != 0 or self.H % self.HK != 0:
            raise NotImplementedError(f"v heads ({self.H}) must be a multiple of q heads ({HQ}) and k heads ({self.HK})")
        # trace the mods once
        self._leaves = {
            "q": SymbolicArray("q", Var("q"), shape_idx=["B", "H", "T", "D"]),
            "k": SymbolicArray("k", Var("k"), shape_idx=["B", "H", "T", "D"]),
            "v": SymbolicArray("v", Var("v"), shape_idx=["B", "H", "T", "D"]),
            "decay": SymbolicArray("decay", Var("decay"), shape_idx=["B", "H", "T"]),
        }
        self._mods = {}
        for name, fn in (("q", q_mod), ("k", k_mod), ("v", v_mod), ("decay", decay_mod)):
            self._mods[name] = fn(self._leaves[name], self.custom_io) if fn is not None else None
        self.q_scale = 1.0
        if self._mods["q"] is not None:
            c = _constant_multiple(self._mods["q"], self._leaves["q"])
            if c is not None:
                self.q_scale = c
                self._mods["q"] = None
        # v_mod = v * t with t free of v (Mamba2: v * dt[batch, heads, seq_len]): the factor goes into the kernel, which
        # rescales the rows of v anyway, instead of a whole-tensor multiply before it (the fused v_mod of the
        # reference, core/lower/lower_linear.py:211-287)
        self._v_scale_expr = None
        vm = self._mods["v"]
        if vm is not None and vm.code.type == "Mul" and len(vm.prev) == 2:
            a, b = vm.prev
            other = b if a is self._leaves["v"] else a if b is self._leaves["v"] else None
            if other is not None and not _depends_on(other, self._leaves["v"]):
                self._v_scale_expr = other
                self._mods["v"] = None
        self.attention = self._run

    def _apply(self, name, tensor, custom_env):
        out = self._mods[name]
        if out is None:
            return tensor
        env = dict(custom_env)
        env[id(self._leaves[name])] = tensor.float()
        res = eval_tensor_expr(out, env)
        return res if name == "decay" else res.to(tensor.dtype)

    def has_backward(self) -> bool:
        """Gradients flow to q, k, v, the decay and the custom inputs, through every mod, unless the output is
        normalised."""
        return not self.normalize_output

    def _run(self, q, k, v, decay, *custom):
        tensors = [t for t in (q, k, v, decay) + tuple(custom) if isinstance(t, torch.Tensor)]
        if torch.is_grad_enabled() and any(t.requires_grad for t in tensors):
            if self.has_backward():
                return self._run_differentiable(q, k, v, decay, *custom)
            return _ForwardOnly.apply(self._run_impl, q, k, v, decay, *custom)
        return self._run_impl(q, k, v, decay, *custom)

    def _run_differentiable(self, q, k, v, decay, *custom):
        """The mods as torch operations that autograd records (a factor on v that the forward-only path hands to the
        kernel is an explicit multiply here), then the kernel with its backward."""
        if len(custom) != len(self.custom_names):
            raise TypeError(f"expected custom tensors {self.custom_names}")
        cenv = {id(self.custom_io.input_tensors[n]): t.float() for n, t in zip(self.custom_names, custom)}
        q = self._apply("q", q, cenv)
        k = self._apply("k", k, cenv)
        v = self._apply("v", v, cenv)
        if self._v_scale_expr is not None:
            t = eval_tensor_expr(self._v_scale_expr, cenv)
            t = t if isinstance(t, torch.Tensor) else torch.tensor(float(t), device=v.device)
            f, g = _align(v.float(), t)
            v = (f * g).to(v.dtype)
        log_decay = self._apply("decay", decay.float(), cenv)
        return _LinearAttention.apply(q, k, v, log_decay, self.q_scale)

    def _run_impl(self, q, k, v, decay, *custom):
        if len(custom) != len(self.custom_names):
            raise TypeError(f"expected custom tensors {self.custom_names}")
        cenv = {id(self.custom_io.input_tensors[n]): t.float() for n, t in zip(self.custom_names, custom)}
        q = self._apply("q", q, cenv)
        k = self._apply("k", k, cenv)
        v = self._apply("v", v, cenv)
        v_scale = None
        if self._v_scale_expr is not None:
            t = eval_tensor_expr(self._v_scale_expr, cenv)
            t = t if isinstance(t, torch.Tensor) else torch.tensor(float(t), device=v.device)
            if t.dim() <= 3 and (t.dim() < 3 or t.shape[-1] in (1, v.shape[2])):
                v_scale = t.reshape(t.shape + (1,) * (3 - t.dim())) if t.dim() < 3 else t   # leading axes: batch, heads, token
            else:   # a factor with a feature axis: no per-token scalar, multiply before the kernel
                f, g = _align(v.float(), t)
                v = (f * g).to(v.dtype)
        log_decay = self._apply("decay", decay.float(), cenv)
        B, _, T, _ = q.shape
        H = v.shape[1]
        # fewer q / k heads than v heads: each group serves H / HQ consecutive heads (the grouping of the
        # Mamba2 reference, testing/test.py:222,271); the kernel reads the shared head, nothing is replicated
        return linear_attention_forward(q, k, v, log_decay, q_scale=self.q_scale, normalize=self.normalize_output, v_scale=v_scale)

    def __call__(self, *args, **kargs):
        return self.attention(*args, **kargs)
