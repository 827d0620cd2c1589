"""The native host side of a call (csrc/host_ops.cpp) without a GPU: the calls it refuses before anything is launched, and
the life of the plans that engines give it."""

import copy
import gc
import os
import pickle
import shutil
import weakref

import pytest
import torch

from core.native import lib
from examples_b200 import programs


@pytest.fixture(scope="module")
def host(native_lib):
    lib.build_host_ops()
    return lib.host()


def operands(*shapes):
    return [torch.zeros(*s, dtype=torch.bfloat16) for s in shapes]


@pytest.mark.parametrize("B,H,Sq", [(0, 8, 1), (1, 8, 0), (1, 0, 1), (0, 0, 0)])
def test_empty_calls_are_refused(host, B, H, Sq):
    """against a cache long enough to be split: the split plan divides by the number of CTAs"""
    assert host.splits_on(B, H, Sq, 4096, 148) == 1
    eng = programs.gqa_engine(1, 8, 8, 1, 4096, 128, 128)
    with pytest.raises(ValueError, match="empty"):
        eng(*operands((B, Sq, H, 128), (B, 4096, max(H, 1), 128), (B, 4096, max(H, 1), 128)))


def test_split_plan(host):
    assert host.splits_on(1, 32, 1, 32768, 148) == 4      # 32 CTAs of 148 SMs
    assert host.splits_on(1, 1, 1, 2048, 148) == 4        # four tiles to a split
    assert host.splits_on(8, 32, 1, 32768, 148) == 1


@pytest.mark.parametrize("q,k,v,what", [
    ((2, 1, 8, 128), (1, 2048, 2, 128), (2, 2048, 2, 128), "fewer sequences"),
    ((2, 1, 8, 128), (2, 2048, 2, 128), (1, 2048, 2, 128), "fewer sequences"),
    ((2, 1, 8, 128), (2, 2048, 2, 64), (2, 2048, 2, 128), "smaller head dim"),
    ((2, 1, 8, 128), (2, 2048, 2, 128), (2, 2047, 2, 128), "shorter"),
    ((2, 300, 8, 128), (2, 300, 8, 128), (2, 172, 8, 128), "shorter"),
])
def test_operands_that_would_be_read_past_their_end_are_refused(host, q, k, v, what):
    with pytest.raises(ValueError, match=what):
        programs.gqa_engine(2, 8, 2, q[1], k[1], 128, 128)(*operands(q, k, v))


def test_larger_caches_are_read_in_part(host):
    """a batch of three out of caches laid out for eight, and rows of v past the last of k"""
    eng = programs.gqa_engine(3, 8, 8, 1, 512, 128, 128)
    assert host.fault(eng._make_plan(), *operands((3, 1, 8, 128), (8, 512, 8, 128), (8, 600, 8, 128))) is None


def document(b, h, q_idx, kv_idx):
    return (q_idx // 200 == kv_idx // 200) & (q_idx >= kv_idx)


def document_of_head(b, h, q_idx, kv_idx):
    return (q_idx // (200 + h) == kv_idx // (200 + h)) & (q_idx >= kv_idx)


@pytest.mark.parametrize("mask,built,call,refused", [
    (document, 500, 500, None),
    (document, 500, 505, "longer"),              # the same tiles, but rows the mask was not evaluated for
    (document, 500, 700, "longer"),              # bitmaps and element masks would be read past their end
    (document, 500, 400, None),                  # the same tiles
    (document, 500, 130, None),                  # fewer tiles of the same rows
    (document, 4200, 4200, None),
    (document, 4200, 4000, "too much shorter"),  # rows of one word instead of two
    (document, 4200, 100, None),                 # one row
    (document_of_head, 500, 390, None),
    (document_of_head, 500, 380, "too much shorter"),   # rows of the second head further in front
    (document_of_head, 4200, 100, "too much shorter"),
])
def test_lengths_that_a_mask_was_not_evaluated_for(host, mask, built, call, refused):
    eng = programs.masked_softmax_engine(1, 2, built, 64, 64, mask)
    q, k, v = operands(*[(1, call, 2, 64)] * 3)
    got = host.fault(eng._make_plan(), q, k, v)
    assert got is None if refused is None else refused in got
    with pytest.raises(lib.NativeError if refused is None else ValueError, match=refused or "CUDA"):
        eng(q, k, v)


def test_reading_of_a_mask_at_the_lengths_of_a_call(host):
    """The lengths that are accepted are those at which the bitmaps, read as the kernel does with the rows and words of the
    call, are the ones that the mask gives when it is evaluated for the call."""
    from core.lower import sparse
    for mask in (document, document_of_head):
        for built in (300, 4200):
            eng = programs.masked_softmax_engine(1, 2, built, 64, 64, mask)
            plan, was = eng._make_plan(), eng._sparse_host
            for sq in {100, 128, 129, 256, 300, 4100} & set(range(built + 1)):
                for skv in {100, 128, 300, 4096, 4097} & set(range(built + 1)):
                    q, k = torch.zeros(1, sq, 2, 64), torch.zeros(1, skv, 2, 64)
                    now = sparse.build_block_sparse(mask, 1, 2, sq, skv)
                    rows, words = now["keep"].shape[1] * now["keep"].shape[2], now["keep"].shape[3]
                    flat = was["keep"].flatten()
                    same = rows * words <= flat.numel() and now["heads"] == was["heads"]
                    if same:   # tiles past the call's last are loaded as zeros and masked
                        live = torch.tensor([(1 << min(32, max(0, -(-skv // 128) - 32 * w))) - 1 for w in range(words)])
                        read = flat[:rows * words].view(rows, words).long() & live
                        want = now["keep"].view(rows, words).long() & live
                        base = was["mask_base"].flatten()[:rows]
                        same = torch.equal(read, want) and torch.equal(base, was["mask_base"].reshape(
                            was["mask_base"].shape[1], -1)[:, :now["keep"].shape[2]].reshape(-1)[:rows])
                    assert (host.fault(plan, q, k, k) is None) == same, (mask.__name__, built, sq, skv)


@pytest.mark.parametrize("make", [
    lambda: programs.gqa_engine(1, 8, 2, 256, 256, 128, 128, is_causal=True),
    lambda: programs.masked_softmax_engine(1, 2, 500, 64, 64, document),
])
def test_an_engine_goes_when_its_last_user_does(host, make):
    """with its plan, and so with the device copies of its mask"""
    eng = make()
    plan = eng._make_plan()
    left = weakref.ref(eng)
    del eng
    gc.collect()
    assert left() is None and plan is not None


@pytest.mark.parametrize("duplicate", [copy.copy, copy.deepcopy, lambda eng: pickle.loads(pickle.dumps(eng))])
def test_engines_that_have_been_called_are_copied_and_pickled(host, duplicate):
    eng = programs.masked_softmax_engine(1, 2, 500, 64, 64, document)
    plan = eng._make_plan()
    twin = duplicate(eng)
    assert twin._plan is None and eng._plan is plan
    assert host.fault(twin._make_plan(), *operands(*[(1, 700, 2, 64)] * 3)) is not None


def test_backward_refuses_what_it_would_leave_unwritten(host):
    """a status of the library, raised from native code, arrives as the library's error"""
    q, k, v, o = operands((2, 256, 8, 64), (3, 256, 8, 64), (3, 256, 8, 64), (2, 256, 8, 64))
    lse = torch.zeros(2, 8, 256)
    with pytest.raises(lib.NativeError, match="invalid argument"):
        host.softmax_bwd(q, k, v, o, lse, o, 0.125, lib.MASK_CAUSAL, 0, 0, ())
    with pytest.raises(lib.NativeError, match="invalid argument"):
        host.softmax_bwd(q, k[:2], v[:2], o, lse[:1], o, 0.125, lib.MASK_CAUSAL, 0, 0, ())


def test_a_host_side_of_other_sources_is_not_loaded(host, monkeypatch, tmp_path):
    """the header gives the layout of the structs that it fills"""
    assert host.__file__ == lib.host_path() == lib.build_host_ops()
    shutil.copy(os.path.join(lib.INCLUDE_DIR, "attn_b200.h"), tmp_path)
    with monkeypatch.context() as m:
        m.setattr(lib, "INCLUDE_DIR", str(tmp_path))
        assert lib.host_path() == host.__file__
        with open(tmp_path / "attn_b200.h", "a") as f:
            f.write("/* a field more */")
        assert lib.host_path() != host.__file__
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "0.0")
        assert lib.host_path() != host.__file__


def test_refusals_of_linear_and_mla_calls_keep_their_errors():
    """Shapes, types and devices that the native host side refuses, before anything is launched."""
    from attn_engine.linear_attn_engine import linear_attention_forward
    from attn_engine.mla import mla_decode_forward
    from core.native.lib import NativeError
    q, k, v, g = torch.zeros(2, 2, 64, 64), torch.zeros(2, 2, 64, 64), torch.zeros(2, 4, 64, 128), torch.zeros(2, 4, 64)
    with pytest.raises(NativeError, match="needs CUDA tensors"):
        linear_attention_forward(q, k, v, g)
    with pytest.raises(NativeError, match="do not fit together"):
        linear_attention_forward(q, k[:1], v, g)
    with pytest.raises(ValueError):
        linear_attention_forward(q[0], k, v, g)
    with pytest.raises(NativeError, match="out_dtype"):
        linear_attention_forward(q, k, v, g, out_dtype=torch.float64)
    with pytest.raises(NativeError, match="needs CUDA tensors"):
        mla_decode_forward(torch.zeros(2, 128, 576), torch.zeros(2, 64, 576), 512, 1.0)
    with pytest.raises(ValueError, match="q: expected a singleton axis"):
        mla_decode_forward(torch.zeros(2, 2, 128, 576), torch.zeros(2, 64, 576), 512, 1.0)
    with pytest.raises(ValueError, match="kv: expected .batch, rows, cols. with contiguous columns"):
        mla_decode_forward(torch.zeros(2, 128, 576), torch.zeros(2, 576, 64).transpose(1, 2), 512, 1.0)


def test_mla_lengths_may_be_any_number():
    """max_seqlen and scale as what a program computes them as; the call is refused for its CPU tensors, not for their type"""
    from attn_engine.mla import mla_decode_forward
    from core.native.lib import NativeError
    table = torch.zeros(2, 1, dtype=torch.int32)
    for length in (64, 64.0, torch.tensor(64), torch.tensor(64.0)):
        with pytest.raises(NativeError, match="needs CUDA tensors"):
            mla_decode_forward(torch.zeros(2, 128, 576), torch.zeros(2, 64, 576), 512, torch.tensor(0.5), block_table=table, max_seqlen=length)
