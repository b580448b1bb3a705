"""The give-up path of the device-side waits, and persistent launches that share the GPU.

Every wait inside the kernels (mbarrier, flag of another range) is bounded: when its limit runs out the kernel
records FKDA_ERR_DEVICE_STATUS in the workspace header, tells the other warps of its CTA, waits for its own copies in
flight and returns, so the context stays usable.  The first test makes that happen without any fault: a test-only flag
stops the one-kernel forward from publishing the states it hands on, so that the ranges behind starve and run out
a limit shortened to a few milliseconds.  Nothing here traps, faults or waits without bound.
"""
import time

import pytest
import torch

import flashkda_b200
from flashkda_b200 import _lib
from flashkda_b200.synth import Workload, make_inputs, to_device

pytestmark = pytest.mark.gpu


def _call(d, ws, flags=0, phase_mask=0):
    flashkda_b200.fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], d["out"], A_log=d["A_log"],
                      dt_bias=d["dt_bias"], lower_bound=d["lower_bound"], initial_state=d["initial_state"],
                      final_state=d["final_state"], cu_seqlens=d["cu_seqlens"], algo="tc", workspace=ws, flags=flags, phase_mask=phase_mask)


def _many_chains(seed, n_seq=100, H=5):
    # 500 chains of 10 to 40 chunks: the one-kernel forward, with chains cut by the ranges
    gen = torch.Generator().manual_seed(seed)
    lens = torch.randint(160, 640, (n_seq,), generator=gen).tolist()
    w = Workload("bw", 1, sum(lens), H, state_in="fp32", state_out="fp32", seq_lens=lens, lower_bound=-2.0)
    d = to_device(make_inputs(w, seed=seed), "cuda")
    ws = torch.empty(flashkda_b200.get_workspace_size(w.tokens, w.H, n_seq), dtype=torch.uint8, device="cuda")
    return d, ws


def test_starved_ranges_give_up_cleanly_and_the_next_call_succeeds():
    d, ws = _many_chains(1)
    _call(d, ws)                                   # a normal call: the expected result
    assert flashkda_b200.device_status(ws) == 0
    good_out, good_state = d["out"].clone(), d["final_state"].clone()

    flags = _lib.FLAG_TEST_DROP_PUSH | _lib.flags_wait_ms(5)
    t0 = time.perf_counter()
    _call(d, ws, flags)
    status = flashkda_b200.device_status(ws)       # synchronises
    dt = time.perf_counter() - t0
    assert status == 9, "starved ranges must be reported as FKDA_ERR_DEVICE_STATUS"
    assert dt < 2.0, f"the kernel took {dt:.2f} s to give up with a 5 ms limit"

    # the context is intact: the same call without the hook is correct again
    d["out"].zero_()
    d["final_state"].zero_()
    _call(d, ws)
    assert flashkda_b200.device_status(ws) == 0
    assert torch.equal(d["out"], good_out) and torch.equal(d["final_state"], good_state)


def test_two_persistent_launches_on_two_streams():
    """Two calls that each fill the GPU, on two streams at once: the CTAs of the second launch find the SMs taken.  Ranges are
    numbered by the CTAs as they start, so neither launch waits for CTAs that have not started; both must finish with
    the results of lone calls and a clean status."""
    probs = [_many_chains(seed) for seed in (2, 3)]
    expect = []
    for d, ws in probs:
        _call(d, ws)
        assert flashkda_b200.device_status(ws) == 0
        expect.append((d["out"].clone(), d["final_state"].clone()))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    limit = _lib.flags_wait_ms(1000)
    for _ in range(5):
        for (d, ws), s in zip(probs, streams):
            d["out"].zero_()
            d["final_state"].zero_()
            s.wait_stream(torch.cuda.current_stream())
        for (d, ws), s in zip(probs, streams):
            with torch.cuda.stream(s):
                _call(d, ws, limit)
        for s in streams:
            s.synchronize()
        for (d, ws), (out, state) in zip(probs, expect):
            assert flashkda_b200.device_status(ws) == 0
            assert torch.equal(d["out"], out) and torch.equal(d["final_state"], state)


def test_a_chain_longer_than_the_limit_of_a_wait():
    """One long sequence among many short ones: its chain is walked range after range, so the last CTA's turn comes when all of it
    but the end is done (4 ms here, under a limit of 1 ms).  That is no reason to give up."""
    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    lens = [64000 - n] + [1] * (n - 1)
    w = Workload("lc", 1, sum(lens), 1, state_in="bf16", state_out="bf16", seq_lens=lens, lower_bound=-2.0)
    d = to_device(make_inputs(w, seed=4), "cuda")
    ws = torch.empty(flashkda_b200.get_workspace_size(w.tokens, w.H, n), dtype=torch.uint8, device="cuda")
    _call(d, ws, _lib.flags_wait_ms(1))
    assert flashkda_b200.last_launch_count() == 2      # the one-kernel form
    assert flashkda_b200.device_status(ws) == 0
    out, state = d["out"].clone(), d["final_state"].clone()
    d["out"].zero_()
    d["final_state"].zero_()
    _call(d, ws, phase_mask=_lib.PHASE_PREPARE | _lib.PHASE_RECURRENCE)
    assert flashkda_b200.device_status(ws) == 0
    assert torch.equal(d["out"], out) and torch.equal(d["final_state"], state)
