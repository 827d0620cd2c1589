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
