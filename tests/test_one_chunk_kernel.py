"""The one-chunk kernel (sequences of 1 .. 16 tokens, persistent CTAs that stream states through shared memory) against the general
kernels, bit for bit: chain counts around its grid, its two groups and its ring, many rounds per CTA with and without states to
load, both state types, missing states, a final state written over the initial one, and decode steps on both sides of the
dispatch line."""
import pytest
import torch

import flashkda_b200
from flashkda_b200 import _lib
from flashkda_b200.synth import Workload, make_inputs, to_device

pytestmark = pytest.mark.gpu
GENERAL = _lib.FLAG_NO_DECODE | _lib.FLAG_NO_SHORT


def _call(d, flags=0, h0="initial_state"):
    out = torch.zeros_like(d["out"])
    h_in = None if d["initial_state"] is None else d["initial_state"].clone()
    hT = h_in if h0 == "in place" else (None if d["final_state"] is None else torch.zeros_like(d["final_state"]))
    flashkda_b200.fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], out, d["A_log"], d["dt_bias"], d["lower_bound"],
                      h_in, hT, d["cu_seqlens"], flags=flags)
    return out, hT


@pytest.mark.parametrize("B,T,H", [(1, 2, 1), (147, 9, 1), (149, 8, 1), (74, 7, 4), (297, 16, 3), (250, 1, 9)])
@pytest.mark.parametrize("state_in,state_out", [("bf16", "bf16"), ("fp32", "fp32"), (None, "bf16"), ("fp32", None), (None, None)])
def test_fixed_batches_equal_the_general_kernels(B, T, H, state_in, state_out):
    d = to_device(make_inputs(Workload("oc", B, T, H, state_in=state_in, state_out=state_out, lower_bound=-2.0), seed=B + T), "cuda")
    got = _call(d)
    assert flashkda_b200.last_launch_count() == 1
    ref = _call(d, GENERAL)
    assert flashkda_b200.last_launch_count() >= 1
    exact = T > 1 or "fp32" not in (state_in, state_out)   # (a decode step with fp32 states: the decode kernel)
    for x, y in zip(got, ref):
        if x is not None:
            assert torch.equal(x, y) if exact else torch.allclose(x.float(), y.float(), atol=2e-2)


@pytest.mark.parametrize("state", ["bf16", "fp32"])
def test_final_state_over_the_initial_state(state):
    d = to_device(make_inputs(Workload("ip", 160, 5, 4, state_in=state, state_out=state, lower_bound=-2.0), seed=3), "cuda")
    ref, got = _call(d), _call(d, h0="in place")
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


@pytest.mark.parametrize("chains", [2048, 2049])
def test_decode_steps_on_both_sides_of_the_dispatch_line(chains):
    d = to_device(make_inputs(Workload("dl", chains, 1, 1, state_in="bf16", state_out="bf16", lower_bound=-2.0), seed=5), "cuda")
    got = _call(d)
    assert flashkda_b200.last_launch_count() == 1
    ref = _call(d, GENERAL)
    if chains > 2048:   # (the decode kernel sums its dot products in another order)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
    assert torch.allclose(got[0].float(), ref[0].float(), atol=2e-2) and torch.allclose(got[1].float(), ref[1].float(), atol=2e-2)


@pytest.mark.parametrize("state", ["bf16", "fp32"])
def test_ragged_with_empty_sequences_over_several_rounds(state):
    g = torch.Generator().manual_seed(2)
    lens = torch.randint(0, 17, (333,), generator=g).tolist()
    lens[0] = lens[-1] = 0
    d = to_device(make_inputs(Workload("re", 1, sum(lens), 4, state_in=state, state_out=state, lower_bound=-2.0, seq_lens=lens), seed=6), "cuda")
    got, ref = _call(d), _call(d, GENERAL)
    assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


@pytest.mark.parametrize("T", [2, 16])
@pytest.mark.parametrize("state_in,state_out", [(None, "bf16"), (None, "fp32"), ("bf16", "bf16"), ("fp32", "fp32")])
@pytest.mark.parametrize("ragged", [False, True])
def test_many_rounds_per_cta(T, state_in, state_out, ragged):
    """Dozens of chains per CTA, repeated: nothing but the kernel's own barriers keeps the warps of a group in step, and without
    states to load there is no arrival of a load to hold one back."""
    n, H = 1100, 4
    lens = [T] * n if ragged else None
    w = Workload("mr", 1 if ragged else n, n * T if ragged else T, H, state_in=state_in, state_out=state_out, lower_bound=-2.0, seq_lens=lens)
    d = to_device(make_inputs(w, seed=T), "cuda")
    ref = _call(d, GENERAL)
    for _ in range(10):
        got = _call(d)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])


@pytest.mark.parametrize("state", ["bf16", "fp32"])
def test_empty_sequences_pass_their_state_through(state):
    """Bit for bit, whatever the state holds (signed zeros, infinities, NaN) and whatever the tokens of other sequences hold: the
    batch's first token is made of NaN."""
    lens = [5, 0, 16, 0, 1, 0] * 24
    d = to_device(make_inputs(Workload("ep", 1, sum(lens), 3, state_in=state, state_out=state, lower_bound=-2.0, seq_lens=lens), seed=8), "cuda")
    for name in "qkvg":
        d[name][0, 0] = float("nan")
    h0 = d["initial_state"]
    h0[1, :, 3] = -0.0
    h0[3, :, 5, 7], h0[3, :, 6] = float("inf"), float("nan")
    got, ref = _call(d), _call(d, GENERAL)
    assert flashkda_b200.last_launch_count() == 3
    bits = lambda x: x.contiguous().view(torch.int16 if x.dtype == torch.bfloat16 else torch.int32)
    empty, rest = [i for i, n in enumerate(lens) if n == 0], [i for i, n in enumerate(lens) if n > 0 and i > 0]
    want = h0[empty].to(torch.bfloat16).to(h0.dtype)
    assert torch.equal(bits(got[1][empty]), bits(ref[1][empty]))
    assert torch.allclose(got[1][empty], want, rtol=0, atol=0, equal_nan=True)
    assert torch.equal(got[1][rest], ref[1][rest]) and torch.equal(got[0][0, 5:], ref[0][0, 5:])
