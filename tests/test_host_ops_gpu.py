"""The native host side of a call (csrc/host_ops.cpp) on the GPU: what surrounds the launches."""

import ctypes
import gc
import threading
import time

import pytest
import torch

from core.native import lib
from examples_b200 import programs

pytestmark = pytest.mark.gpu


def document(b, h, q_idx, kv_idx):
    return (q_idx // 200 == kv_idx // 200) & (q_idx >= kv_idx)


def rand(*shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(len(shape) + shape[1]), device="cuda").to(torch.bfloat16)


def test_training_after_a_first_call_in_inference_mode():
    """the mask's device copies are made by the first call: here as inference tensors, which autograd does not save"""
    grads = []
    for first in (False, True):
        eng = programs.masked_softmax_engine(1, 2, 512, 64, 64, document)
        q, k, v = (rand(1, 512, 2, 64).mul_(s) for s in (1.0, 0.5, 2.0))
        if first:
            with torch.inference_mode():
                eng(q, k, v)
        for t in (q, k, v):
            t.requires_grad_()
        grads.append(torch.autograd.grad(eng(q, k, v), (q, k, v), rand(1, 512, 2, 64)))
    assert all(torch.equal(a, b) for a, b in zip(*grads))
    assert lib.last_device_status() == 0


def test_saved_tensor_hooks_see_the_call_s_tensors_only():
    eng = programs.masked_softmax_engine(1, 2, 512, 64, 64, document)
    q, k, v = (rand(1, 512, 2, 64).requires_grad_() for _ in range(3))
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.dtype) or t, lambda t: t):
        o = eng(q, k, v)
    assert sorted(map(str, seen)) == ["torch.bfloat16"] * 4 + ["torch.float32"]     # q, k, v, o and lse
    o.sum().backward()
    assert q.grad is not None and lib.last_device_status() == 0


def test_masks_of_engines_that_are_gone_give_their_memory_back():
    """each engine's mask takes 4 MB of bits twice; used on another stream as well as on the one it was made on"""
    q, k, v = (rand(1, 6000, 2, 64) for _ in range(3))
    other = torch.cuda.Stream()
    want, held = None, []
    for _ in range(3):
        eng = programs.masked_softmax_engine(1, 2, 6000, 64, 64, document)
        o = eng(q, k, v)
        other.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(other):
            o2 = eng(q, k, v)
        del eng
        gc.collect()
        torch.cuda.synchronize()
        assert torch.equal(o, o2) and (want is None or torch.equal(o, want))
        want = o
        del o, o2
        torch.cuda.empty_cache()
        held.append(torch.cuda.memory_allocated())
    assert held[2] - held[0] < 1 << 20
    assert lib.last_device_status() == 0


def test_decode_arguments_of_an_engine_without_them_are_left_alone():
    eng = programs.gqa_engine(2, 8, 2, 1, 1024, 128, 128)
    q, k, v = rand(2, 1, 8, 128), rand(2, 1024, 2, 128), rand(2, 1024, 2, 128)
    want = eng(q, k, v)
    mask = torch.zeros(2, 2, 8, dtype=torch.bool, device="cuda")
    assert torch.equal(eng.attention(q, k, v, block_mask=mask, cache_seqlens=torch.tensor([3, 5])), want)
    assert lib.last_device_status() == 0


def test_other_threads_run_while_a_call_waits_for_the_stream():
    """Behind 0.7 s of work on the stream, calls fill its queue (about a thousand launches) and the next one waits."""
    eng = programs.gqa_engine(1, 2, 2, 128, 128, 64, 64, is_causal=True)
    q, k, v = (rand(1, 128, 2, 64) for _ in range(3))
    eng(q, k, v)
    torch.cuda.synchronize()
    longest, stop = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            longest[0], last = max(longest[0], now - last), now

    ticker = threading.Thread(target=tick)
    ticker.start()
    time.sleep(0.05)
    torch.cuda._sleep(int(0.7 * 1.9e9))
    start = time.perf_counter()
    for _ in range(3000):
        eng(q, k, v)
    waited = time.perf_counter() - start
    stop.set()
    ticker.join()
    torch.cuda.synchronize()
    if waited < 0.4:
        pytest.skip("this driver's queue holds all of the calls")
    assert longest[0] < 0.5 * waited, (longest[0], waited)


def test_refusals_of_the_library_arrive_as_its_error():
    """from a forward, outside the interpreter lock, and from a backward on autograd's thread; nothing is launched"""
    eng = programs.gqa_engine(1, 2, 2, 256, 256, 64, 64, is_causal=True)
    q, k, v = (rand(1, 256, 2, 64) for _ in range(3))
    with pytest.raises(lib.NativeError, match="unsupported"):
        eng(rand(1, 256, 2, 65)[..., :64], k, v)       # heads 65 elements apart: no 16-byte pieces
    k, v = (rand(2, 256, 2, 64).requires_grad_() for _ in range(2))     # a cache of two sequences, a call of one
    o = eng(q, k, v)
    assert torch.equal(o, eng(q, k[:1].detach(), v[:1].detach()))
    with pytest.raises(lib.NativeError, match="invalid argument"):
        o.sum().backward()
    # keep bits of another extent than the call's, in each of their dimensions
    q, k, v, o = (t.detach() for t in (q, k[:1], v[:1], o))
    for shape in ((384, 2, 4), (256, 3, 4), (256, 2, 2)):
        bits = [torch.zeros(*shape, dtype=torch.int32, device="cuda")] * 2
        with pytest.raises(lib.NativeError, match="invalid argument"):
            lib.softmax_bwd(q, k, v, o, torch.zeros(1, 2, 256, device="cuda"), o, 0.125, lib.MASK_NONE, mask_bits=bits)
    assert lib.last_device_status() == 0


def _chains():
    """Calls whose output is the next call's input as it stands, one per kernel family: name -> (start tensor, step).  No torch
    kernel runs between two calls: it would end before the next of the library's kernels is made ready."""
    from attn_engine.mla import mla_decode_forward
    gen = torch.Generator(device="cuda").manual_seed(3)

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)
    k, v, ones = rnd(1, 700, 4, 64), rnd(1, 700, 4, 64), torch.ones(1, 700, 4, 64, device="cuda", dtype=torch.bfloat16)
    prefill = programs.softmax_engine(1, 4, 700, 64, 64, is_causal=True)
    decode = programs.gqa_engine(2, 8, 2, 1, 900, 128, 128)
    dk, dv = rnd(2, 900, 2, 128), rnd(2, 900, 2, 128)
    lin = programs.gla_engine(1, 4, 600, 128, 128)
    lk, lv, lg, ld = rnd(1, 4, 600, 128), rnd(1, 4, 600, 128), torch.full((1, 4, 600), -0.3, device="cuda"), rnd(1, 4, 600, 128) * 0.1
    lk.requires_grad_()
    lg_leaf = lg.clone().requires_grad_()
    kv, q_rope = rnd(2, 500, 576), rnd(2, 128, 64)

    def mla(q):   # the output's 512 columns are the next call's
        return mla_decode_forward(q, kv[..., :512], 512, 576 ** -0.5, q_rope=q_rope, kv_rope=kv[..., 512:], num_splits=0)[0]

    def train(x):
        x = x.detach().requires_grad_()
        return torch.autograd.grad(prefill(x, k, v), x, ones)[0]

    def train_linear(x):   # dk depends on q (dq would not), and is the next call's q
        return torch.autograd.grad(lin(x, lk, lv, lg_leaf), (lk, lg_leaf), ld)[0]
    return {"prefill": (rnd(1, 700, 4, 64), lambda x: prefill(x, k, v)), "train": (rnd(1, 700, 4, 64), train),
            "decode": (rnd(2, 1, 8, 128), lambda x: decode(x, dk, dv)),
            "linear": (rnd(1, 4, 600, 128), lambda x: lin(x, lk.detach(), lv, lg)),
            "linear_train": (rnd(1, 4, 600, 128), train_linear), "mla": (rnd(2, 128, 512), mla)}


@pytest.mark.parametrize("name", ["prefill", "train", "decode", "linear", "linear_train", "mla"])
def test_calls_that_feed_one_another(name):
    """A kernel is made ready while the one in front of it still runs: what it reads and overwrites must wait all the same,
    the allocator handing scratch and outputs from one call to the next.  The same bits as with a wait behind every call."""
    x0, step = _chains()[name]
    want = x0
    for _ in range(12):
        want = step(want)
        torch.cuda.synchronize()
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            for _ in range(5):
                x = x0
                for _ in range(12):
                    x = step(x)
                assert torch.equal(x, want)
    if "train" not in name:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            x = x0
            for _ in range(12):
                x = step(x)
        for _ in range(3):
            graph.replay()
            assert torch.equal(x, want)
    assert lib.last_device_status() == 0


def _more_families():
    gen = torch.Generator(device="cuda").manual_seed(4)

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device="cuda").to(torch.bfloat16)
    k, v, bias = rnd(1, 300, 2, 64), rnd(1, 300, 2, 64), torch.tensor([-3.0], device="cuda")
    masked, sigmoid = programs.masked_softmax_engine(1, 2, 300, 64, 64, document), programs.sigmoid_engine(1, 2, 300, 64, 64)
    other = programs.softmax_engine_noprobe(1, 2, 300, 64, 64, is_causal=True)

    def train(engine, *custom):
        def step(x):
            x = x.detach().requires_grad_()
            return torch.autograd.grad(engine(x, k, v, *custom), x, v)[0]
        return rnd(1, 300, 2, 64), step
    return {"sparse": train(masked), "elementwise": train(sigmoid, bias), "rows": (rnd(1, 300, 2, 64), lambda x: other(x, k, v))}


class _Word:
    """The device status word as an array that torch can write."""

    def __init__(self):
        ptr = ctypes.c_void_p()
        lib.check(lib.load_library().attn_b200_device_status_word(0, ctypes.byref(ptr)), "attn_b200_device_status_word")
        self.__cuda_array_interface__ = {"shape": (1,), "typestr": "<i4", "data": (ptr.value, False), "version": 3}


@pytest.mark.parametrize("name", ["prefill", "train", "decode", "linear", "linear_train", "mla", "sparse", "elementwise", "rows"])
def test_calls_behind_a_recorded_failure_leave(name):
    """The status word says that a wait ran out: every kernel of a call leaves, its warps together, with copies under way or
    not; once the word has been read the same call is right again."""
    x0, step = {**_chains(), **_more_families()}[name]
    want = step(x0)
    assert lib.last_device_status() == 0
    torch.as_tensor(_Word(), device="cuda").fill_(177)
    step(x0)
    assert lib.last_device_status() == 177
    assert torch.equal(step(x0), want)
    assert lib.last_device_status() == 0
