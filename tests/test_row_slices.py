"""The row-slice kernel (few chains) against the one-kernel forward of the same call, bit for bit, where its shapes change: two or
four CTAs per chain, one or two chunks per stage, odd and even numbers of chunks around its ring, slabs, ragged batches."""
import pytest
import torch

import flashkda_b200
from flashkda_b200 import _lib
from flashkda_b200.synth import Workload, make_inputs
from test_one_kernel_forward import _call

pytestmark = pytest.mark.gpu


def _compare(w, every=None, seed=5):
    inp = make_inputs(w, seed=seed)
    a = _call(inp, every=every)
    launches = flashkda_b200.last_launch_count()
    b = _call(inp, flags=_lib.FLAG_NO_WIDE, every=every)
    assert launches > flashkda_b200.last_launch_count()   # the second call was the one-kernel form
    for x, y in zip(a, b):
        assert x is None or torch.equal(x, y)


@pytest.mark.parametrize("chains", ["4 CTAs", "2 CTAs", "most of 2 CTAs"])
@pytest.mark.parametrize("T", [17, 33, 48, 127, 128, 129, 144, 145, 300])
def test_lengths_around_the_ring(chains, T):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = {"4 CTAs": sms // 4, "2 CTAs": sms // 4 + 1, "most of 2 CTAs": sms // 2}[chains]
    _compare(Workload("r", n, T, 1, state_in="fp32", state_out="fp32", lower_bound=-2.0))


@pytest.mark.parametrize("chains", [1, 6, 24, 25, 58])
@pytest.mark.parametrize("T", [1024, 1025, 4999])
def test_slabs(chains, T):
    _compare(Workload("s", 1, T, chains, state_in="bf16", state_out="bf16", lower_bound=-1.0), every=None if T == 1024 else 3)


@pytest.mark.parametrize("H", [1, 5, 8, 20])
def test_ragged(H):
    lens = [300, 1, 17, 0, 64, 33, 16, 129, 500]   # 9 to 180 chains: four, two and two CTAs per chain, two CTAs per SM
    _compare(Workload("v", 1, sum(lens), H, state_in="fp32", state_out="fp32", lower_bound=-2.0, seq_lens=lens), every=1)
