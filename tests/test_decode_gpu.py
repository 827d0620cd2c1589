"""Decode calls of the built-in softmax (attn_b200_decode_fwd) against softmax attention in fp32: query rows packed by KV head,
shares of the tile list that cut sequences, lengths, gathered blocks, and the calls it leaves to the forward kernel."""

import pytest
import torch

from attn_engine import AttentionEngine
from core import CustomIO, meta_tensor
from core.native import lib
from examples_b200 import programs

pytestmark = pytest.mark.gpu


def reference(q, k, v, scale, keep=None):
    """q [B,Sq,H,D], k/v [B,S,Hkv,D] on the GPU, keep [B,Hkv,S] or None -> (o, lse) in fp32"""
    g = q.shape[2] // k.shape[2]
    kf, vf = (t.float().repeat_interleave(g, 2) for t in (k, v))
    s = torch.einsum("bshd,bthd->bhst", q.float(), kf) * scale
    if keep is not None:
        s = s.masked_fill(~keep.repeat_interleave(g, 1)[:, :, None], -float("inf"))
    return torch.einsum("bhst,bthd->bshd", s.softmax(-1), vf), s.logsumexp(-1)


def check(got, want, dtype):
    """o: the roundings of P (one unit of its 16-bit type, relative) and of o itself; |o| stays below ~4 here.  lse: fp32
    sums of ex2.approx results, whose errors are below 2^-20."""
    o, lse = got
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    ref = want[0].abs().max().item()
    assert (o.float() - want[0]).abs().max().item() <= 2 * eps * max(1.0, ref)
    assert (lse - want[1]).abs().max().item() <= 2e-5 * max(1.0, want[1].abs().max().item())


def run(eng, *args, **kwargs):
    o = eng(*args, **kwargs)
    return o, eng.last_final_rowscales["lse"]


def rand(gen, *shape, dtype):
    return torch.randn(*shape, generator=gen, device="cuda").to(dtype)


@pytest.mark.parametrize("B,H,Hkv,Sq,S,D,dtype", [
    (1, 1, 1, 1, 129, 128, torch.bfloat16),       # two tiles, the second with one row
    (1, 4, 1, 1, 128 * 149, 128, torch.bfloat16),   # one tile more than an SM each
    (2, 32, 8, 1, 1000, 128, torch.float16),      # shares that begin and end inside a pair
    (3, 8, 8, 1, 257, 64, torch.bfloat16),        # fewer tiles than SMs
    (37, 8, 4, 1, 300, 64, torch.float16),        # a whole pair per share: 148 pairs, nothing to merge
    (40, 16, 8, 1, 130, 128, torch.bfloat16),     # shares of several pairs of two tiles
    (2, 33, 1, 1, 700, 128, torch.bfloat16),      # two warps of a softmax group, the second with one row
    (2, 16, 2, 8, 513, 64, torch.float16),        # 64 rows
    (3, 32, 1, 4, 900, 128, torch.bfloat16),      # 128 rows: one query buffer
    (5, 8, 2, 25, 2000, 64, torch.bfloat16),      # 100 rows
])
def test_dense(B, H, Hkv, Sq, S, D, dtype):
    gen = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v = rand(gen, B, Sq, H, D, dtype=dtype), rand(gen, B, S, Hkv, D, dtype=dtype), rand(gen, B, S, Hkv, D, dtype=dtype)
    k[..., S // 2:, :, :] *= 3.0   # the running maximum moves: accumulators are rescaled
    eng = programs.gqa_engine(B, H, Hkv, Sq, S, D, D, dtype=dtype)
    got = run(eng, q, k, v)
    want = reference(q, k, v, D ** -0.5)
    check(got, want, dtype)
    # another order of the query rows: heads outside the sequence axis
    qh = q.transpose(1, 2).contiguous().transpose(1, 2)
    check(run(eng, qh, k.transpose(1, 2).contiguous().transpose(1, 2), v), want, dtype)
    eng.kv_splits = 1   # the forward kernel
    check(run(eng, q, k, v), want, dtype)
    assert lib.last_device_status() == 0


def decode_engine(B, H, Hkv, Sq, S, D, block):
    scale = D ** -0.5

    def score_mod(score, custom, b, h, q_idx, kv_idx):
        return score * scale
    meta = (meta_tensor(B, H, Sq, D, dtype=torch.bfloat16),) + (meta_tensor(B, Hkv, S, D, dtype=torch.bfloat16),) * 2
    return AttentionEngine(meta, CustomIO({}), score_mod=score_mod, mask_mod=None, online_func=programs.NaturalSoftmax(),
                           extern_block_mask=True, use_varlen=True, infer_mask_block_N=block)


@pytest.mark.parametrize("B,H,Hkv,Sq,S,D,block,masked,varlen", [
    (3, 8, 2, 1, 1024, 128, 32, True, True),
    (2, 8, 8, 1, 1000, 128, 8, True, True),        # 125 blocks: rows of the mask are read byte by byte
    (5, 16, 4, 4, 777, 64, 16, True, False),       # the last block lies partly behind the sequence
    (4, 32, 4, 1, 4096, 128, 64, True, True),
    (70, 8, 4, 1, 640, 64, 128, True, True),       # more pairs than SMs
    (6, 8, 2, 2, 2000, 128, 32, False, True),      # lengths only
    (2, 4, 2, 1, 5120, 64, 8, True, True),         # 640 blocks: a row's list takes two steps of 512 flags
    (2, 4, 2, 1, 4808, 128, 8, True, True),        # 601 blocks, byte by byte
    (2, 4, 2, 1, 960, 64, 48, True, True),         # a block that does not divide a tile: left to the forward kernel
    (2, 8, 1, 9, 640, 128, 32, True, True),        # 72 rows with a block mask: left to the forward kernel
])
def test_blocks_and_lengths(B, H, Hkv, Sq, S, D, block, masked, varlen):
    dtype = torch.bfloat16
    gen = torch.Generator(device="cuda").manual_seed(S + block)
    q, k, v = rand(gen, B, Sq, H, D, dtype=dtype), rand(gen, B, S, Hkv, D, dtype=dtype), rand(gen, B, S, Hkv, D, dtype=dtype)
    nb = -(-S // block)
    mask = torch.rand(B, Hkv, nb, generator=gen, device="cuda") < 0.4 if masked else None
    lens = torch.randint(1, S + 1, (B,), generator=gen, device="cuda", dtype=torch.int32) if varlen else None
    if varlen:
        lens[0], lens[1] = S, 1
    if masked:
        mask[:, :, 0] = True
        mask[1, 0] = False        # a pair without a kept block
    keep = torch.ones(B, Hkv, S, dtype=torch.bool, device="cuda")
    if masked:
        keep &= mask.repeat_interleave(block, -1)[..., :S]
    if varlen:
        keep &= (torch.arange(S, device="cuda") < lens[:, None])[:, None]
    eng = decode_engine(B, H, Hkv, Sq, S, D, block)
    o, lse = run(eng, q, k, v, block_mask=mask, cache_seqlens=lens)
    want_o, want_lse = reference(q, k, v, D ** -0.5, keep)
    some = keep.any(-1).repeat_interleave(H // Hkv, 1)     # [B, H]
    assert torch.isnan(o.transpose(1, 2)[~some]).all() and (lse[~some] == -float("inf")).all()
    check((o.transpose(1, 2)[some], lse[some]), (want_o.transpose(1, 2)[some], want_lse[some]), dtype)
    if masked:   # a mask that does not begin on a 16-byte boundary is read byte by byte
        mask = torch.cat([mask.new_zeros(1), mask.flatten()])[1:].view(mask.shape)
    again = run(eng, q, k, v, block_mask=mask, cache_seqlens=lens)
    assert torch.equal(o.nan_to_num(7.0), again[0].nan_to_num(7.0)) and torch.equal(lse, again[1])
    assert lib.last_device_status() == 0


def test_shares_whose_scores_are_all_minus_infinity():
    """One sequence cut into twenty shares, the keys of the first six tiles and of one in the middle -inf against every query
    row: those shares count nothing wherever they stand, and NaN in one of them reaches the result."""
    B, H, Hkv, S, D = 1, 4, 1, 20 * 128, 128
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (rand(gen, B, n, h, D, dtype=torch.bfloat16) for n, h in ((1, H), (S, Hkv), (S, Hkv)))
    q[..., 0] = 1.0
    keep = torch.ones(B, Hkv, S, dtype=torch.bool, device="cuda")
    keep[..., :6 * 128] = keep[..., 11 * 128:12 * 128] = False
    k[0, ~keep[0, 0], 0, 0] = -float("inf")
    eng = programs.gqa_engine(B, H, Hkv, 1, S, D, D)
    kz = k.clone()
    kz[0, ~keep[0, 0]] = 0
    check(run(eng, q, k, v), reference(q, kz, v, D ** -0.5, keep), torch.bfloat16)
    k[0, :8 * 128, 0, 1] = float("nan")
    o, lse = run(eng, q, k, v)
    assert torch.isnan(o).all() and torch.isnan(lse).all()
    assert lib.last_device_status() == 0
