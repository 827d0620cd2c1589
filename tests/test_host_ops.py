"""The native host side of a call (csrc/host_ops.cpp) without a GPU: the calls it refuses before anything is launched, and
the life of the plans that engines give it."""

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
    assert host.fault(*operands((3, 1, 8, 128), (8, 512, 8, 128), (8, 600, 8, 128))) is None
