"""The one-kernel forward (batches with enough chains to fill the GPU) against the two-kernel form of the same call, bit for
bit, and against the CPU oracle: sizes at the edges of its dispatch, of its chunks and of the ranges its CTAs walk (ranges that
start and end inside a chain, chains longer than a range, sequences without tokens)."""
import pytest
import torch

import flashkda_b200
from flashkda_b200 import _lib
from flashkda_b200.synth import Workload, make_inputs, to_device
from test_gpu_parity import check_against, run_oracle

pytestmark = pytest.mark.gpu

BOTH = _lib.PHASE_PREPARE | _lib.PHASE_RECURRENCE   # both stages by name: the two-kernel form

CASES = {
    "one_chain_per_cta": Workload("a", 75, 17, 1, state_in="fp32", state_out="fp32"),
    "ranges_cut_chains": Workload("b", 3, 500, 53, state_in="bf16", state_out="bf16", lower_bound=-2.0),
    "one_more_than_sms": Workload("c", 149, 33, 1, state_out="fp32"),
    "fewer_chunks_than_ctas": Workload("d", 1, 300, 60, lower_bound=-1.0, seq_lens=[300] + [0] * 4),
    "ragged": Workload("e", 1, 3000 + 34 + 61 * 40, 5, state_in="fp32", state_out="fp32", lower_bound=-2.0,
                       seq_lens=[0, 1, 16, 3000, 17, 0] + [40] * 61 + [0]),
    "ragged_stateless_out": Workload("f", 1, 70 * 35, 5, state_out="bf16", seq_lens=[0, 70] * 35),
}


def _call(inp, flags=0, phase_mask=0, every=None):
    d = to_device(inp, "cuda")
    B, T, H = d["beta"].shape
    lens = [T] * B if d["cu_seqlens"] is None else d["cu_seqlens"].diff().tolist()
    ws = torch.full((flashkda_b200.get_workspace_size(B * T, H, len(lens)),), 0xAB, dtype=torch.uint8, device="cuda")
    extra = {}
    if every is not None:
        slots = flashkda_b200.chunk_states_slots(1, 0, every, seq_lens=lens)
        extra = dict(chunk_states=torch.zeros(slots, H, 128, 128, dtype=torch.bfloat16, device="cuda"), chunk_states_every=every)
    flashkda_b200.fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], d["out"], d["A_log"], d["dt_bias"], d["lower_bound"],
                      d["initial_state"], d["final_state"], d["cu_seqlens"], workspace=ws, flags=flags, phase_mask=phase_mask, **extra)
    assert flashkda_b200.device_status(ws) == 0
    return d["out"].cpu(), None if d["final_state"] is None else d["final_state"].cpu(), extra.get("chunk_states")


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("every", [None, 2])
def test_one_kernel_forward_equals_the_two_kernel_form(name, every):
    w = CASES[name]
    inp = make_inputs(w, seed=7)
    ragged = w.seq_lens is not None
    out, hT, cs = _call(inp, flags=_lib.FLAG_NO_WIDE, every=every)
    assert flashkda_b200.last_launch_count() == (2 if ragged else 1)
    out2, hT2, cs2 = _call(inp, phase_mask=BOTH, every=every)
    assert flashkda_b200.last_launch_count() == (3 if ragged else 2)
    assert torch.equal(out, out2)
    assert hT is None or torch.equal(hT, hT2)
    assert cs is None or torch.equal(cs, cs2)
    if every is None:
        check_against(out, hT, *run_oracle(inp))


def test_dispatch_line():
    """Fixed batches take the one kernel from one row slice more than SMs, ragged batches from two chains per SM."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for B, expect in ((sms // 2, 2), (sms // 2 + 1, 1)):
        _call(make_inputs(Workload("l", B, 40, 1), seed=1))
        assert flashkda_b200.last_launch_count() == expect
    for n, expect in ((2 * sms - 1, 3), (2 * sms, 2)):
        _call(make_inputs(Workload("l", 1, 18 * n, 1, seq_lens=[18] * n), seed=1))
        assert flashkda_b200.last_launch_count() == expect


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
@pytest.mark.parametrize("length", [64, 65])
def test_dispatch_line_of_short_sequences(dtype, length):
    """fp32 states in and out: the one kernel from more than four chunks per sequence, with the same results."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for w, one in ((Workload("s", sms, length, 1, state_in=dtype, state_out=dtype), 1),
                   (Workload("s", 1, length * 2 * sms, 1, state_in=dtype, state_out=dtype, seq_lens=[length] * (2 * sms)), 2)):
        inp = make_inputs(w, seed=3)
        out, hT, _ = _call(inp)
        assert flashkda_b200.last_launch_count() == one + (1 if dtype == "fp32" and length == 64 else 0)
        out2, hT2, _ = _call(inp, flags=_lib.FLAG_NO_WIDE)
        assert torch.equal(out, out2) and torch.equal(hT, hT2)


def test_dispatch_line_of_long_ragged_sequences():
    """Ragged batches of more than ten chunks per sequence take the one kernel from 1.6 chains per SM."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = (8 * sms + 4) // 5
    for count, length, expect in ((n, 161, 2), (n, 160, 3), (n - 1, 161, 3)):
        _call(make_inputs(Workload("l", 1, length * count, 1, seq_lens=[length] * count), seed=1))
        assert flashkda_b200.last_launch_count() == expect


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("kind", ["one_kernel", "one_kernel_ragged", "one_token", "short", "one_chunk", "short_ragged", "two_kernels", "empty"])
def test_recurrence_alone_behind_any_call(kind):
    """PHASE_RECURRENCE on a workspace whose last call left no records (a one-kernel form), left records, or left those of other
    inputs before a call that left none: the result of the whole forward with this call's values, each time."""
    n = _sms()
    shape = {"one_kernel": (n, 70, 1, None), "one_kernel_ragged": (1, 70 * 2 * n, 1, [70] * (2 * n)), "one_token": (70, 1, 2, None),
             "short": (70, 5, 2, None), "one_chunk": (70, 16, 2, None), "short_ragged": (1, 7 * 64, 2, [3, 0, 16, 9] * 16),
             "two_kernels": (1, 100, 3, None), "empty": (3, 0, 2, None)}[kind]
    w = Workload("ra", *shape[:3], state_in="fp32", state_out="fp32", lower_bound=-2.0, seq_lens=shape[3])
    a, b = (to_device(make_inputs(w, seed=s), "cuda") for s in (1, 2))
    ws = torch.full((flashkda_b200.get_workspace_size(w.tokens, w.H, w.n_seqs),), 0xAB, dtype=torch.uint8, device="cuda")

    def call(d, phase_mask, v=None):
        flashkda_b200.fwd(d["q"], d["k"], d["v"] if v is None else v, d["g"], d["beta"], d["scale"], d["out"].zero_(), d["A_log"],
                          d["dt_bias"], d["lower_bound"], d["initial_state"], d["final_state"].zero_(), d["cu_seqlens"],
                          workspace=ws, phase_mask=phase_mask)
        assert flashkda_b200.device_status(ws) == 0
        return d["out"].clone(), d["final_state"].clone()

    v2 = torch.flip(b["v"], [1])
    general = _lib.FLAG_NO_DECODE | _lib.FLAG_NO_SHORT
    flashkda_b200.fwd(b["q"], b["k"], v2, b["g"], b["beta"], b["scale"], b["out"].zero_(), b["A_log"], b["dt_bias"], b["lower_bound"],
                      b["initial_state"], b["final_state"].zero_(), b["cu_seqlens"], flags=general)
    want = b["out"].clone(), b["final_state"].clone()
    for before in (0, BOTH, _lib.PHASE_PREPARE, None):   # None: nothing, the records of the call before are still there
        if before is not None:
            call(a, _lib.PHASE_PREPARE)
            call(b, before)
            if before == 0 and kind in ("one_kernel", "one_kernel_ragged", "one_token", "short", "one_chunk"):
                assert flashkda_b200.last_launch_count() == (2 if shape[3] else 1)   # no records left
        for _ in range(2):
            got = call(b, _lib.PHASE_RECURRENCE, v2)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), before
