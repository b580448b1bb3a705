"""Calls one behind the other on a stream, with the caller's kernels or nothing between them, each working on what the one before
wrote, without a synchronisation in between (their kernels are launched as dependents of whatever is in front of them): the
results of the same calls with one after each."""
import pytest
import torch

import flashkda_b200
from flashkda_b200.synth import Workload, make_inputs, to_device

pytestmark = pytest.mark.gpu

SHAPES = {   # B, T, H, sequence lengths
    "decode": (7, 1, 8, None), "decode_many": (600, 1, 4, None), "decode_packed": (1, 70, 4, [1] * 70), "short": (9, 5, 8, None),
    "short_packed": (1, 9 * 20, 8, [5, 0, 16, 15] * 5), "prompt": (1, 100, 8, None), "slabs": (1, 1100, 4, None),
    "ragged": (1, 400, 4, [300, 1, 99]), "one_kernel": (80, 40, 1, None), "one_kernel_ragged": (1, 20 * 300, 1, [20] * 300),
}


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_steps_in_a_row(name, dtype):
    B, T, H, lens = SHAPES[name]
    w = Workload("b", B, T, H, state_in=dtype, state_out=dtype, lower_bound=-0.2, seq_lens=lens)
    d = to_device(make_inputs(w, seed=3), "cuda")
    ws = torch.empty((flashkda_b200.get_workspace_size(w.tokens, H, w.n_seqs),), dtype=torch.uint8, device="cuda")

    def run(sync):
        q, v, state = d["q"].clone(), d["v"].clone(), d["initial_state"].clone()
        outs = []
        for _ in range(6):
            out, new = torch.empty_like(v), torch.empty_like(state)
            flashkda_b200.fwd(q, d["k"], v, d["g"], d["beta"], d["scale"], out, d["A_log"], d["dt_bias"], d["lower_bound"], state,
                              new, d["cu_seqlens"], workspace=ws)
            if sync:
                torch.cuda.synchronize()
            outs.append(out)
            state = new
            v = (v + out).mul_(0.5)        # the caller's own kernels, before and behind
            q.add_(out)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        assert flashkda_b200.device_status(ws) == 0
        return outs, state

    (a, sa), (b, sb) = run(True), run(False)
    assert all(torch.equal(x, y) for x, y in zip(a, b)) and torch.equal(sa, sb)


def _nothing_between(d, ws, shapes, calls, sync):
    """`calls` calls in a row with nothing between them: out of one call is v of the next, final states are the next initial states.
    shapes: (B, T, cu_seqlens) in turn, of one number of tokens each."""
    H = d["v"].shape[2]
    tokens = [d["v"].clone(), torch.zeros_like(d["v"])]
    states = [d["initial_state"].clone(), torch.zeros_like(d["initial_state"])]
    if not sync:
        torch.cuda._sleep(20_000_000)   # 10 ms: the calls below are all in the queue when the first one starts
    for i in range(calls):
        B, T, cu = shapes[i % len(shapes)]
        n = B if cu is None else cu.numel() - 1
        v, out = (t.view(B, T, H, 128) for t in (tokens[i % 2], tokens[1 - i % 2]))
        q, k, g = (d[x].view(B, T, H, 128) for x in "qkg")
        flashkda_b200.fwd(q, k, v, g, d["beta"].view(B, T, H), 4.0, out, d["A_log"], d["dt_bias"], d["lower_bound"],
                          states[i % 2][:n], states[1 - i % 2][:n], cu, workspace=ws)
        if sync:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    if ws is not None:
        assert flashkda_b200.device_status(ws) == 0
    return tokens + states


def _check_nothing_between(d, ws, shapes, calls):
    want = _nothing_between(d, ws, shapes, calls, True)
    assert all(bool(x.float().abs().sum() > 0) and bool(x.isfinite().all()) for x in want)
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(want, _nothing_between(d, ws, shapes, calls, False)))


@pytest.mark.parametrize("own_scratch", [False, True])
@pytest.mark.parametrize("name", sorted(SHAPES) + ["chains_between"])
def test_calls_with_nothing_between(name, own_scratch):
    B, T, H, lens = (1, 1100, 80, None) if name == "chains_between" else SHAPES[name]
    dtype = "bf16" if own_scratch else "fp32"
    w = Workload("b", B, T, H, state_in=dtype, state_out=dtype, lower_bound=-0.2, seq_lens=lens)
    d = to_device(make_inputs(w, seed=3), "cuda")
    ws = None if own_scratch else torch.empty((flashkda_b200.get_workspace_size(w.tokens, H, w.n_seqs),), dtype=torch.uint8, device="cuda")
    _check_nothing_between(d, ws, [(B, T, d["cu_seqlens"])], 12)


@pytest.mark.parametrize("own_scratch", [False, True])
def test_calls_of_other_kinds_with_nothing_between(own_scratch):
    """1 280 tokens of 4 heads as steps of decoding, drafts, prompts, ragged batches and a long prompt in turn, one workspace."""
    def cu(lens):
        return torch.tensor([0] + lens, dtype=torch.int64).cumsum(0).cuda()
    n = 1280
    shapes = [(n, 1, None), (1, n, None), (1, n, cu([1] * n)), (160, 8, None), (1, n, cu([700, 0, 1, 79, 500])), (1, n, cu([5, 0, 16, 11] * 40)),
              (40, 32, None), (n, 1, None), (n, 1, None), (1, n, cu([16] * 70 + [160])), (8, 160, None), (1, n, cu([20] * 64))]
    w = Workload("b", n, 1, 4, state_in="fp32", state_out="fp32", lower_bound=-0.2)
    d = to_device(make_inputs(w, seed=3), "cuda")
    ws = None if own_scratch else torch.empty((max(flashkda_b200.get_workspace_size(n, 4, m) for m in (1, n)),), dtype=torch.uint8, device="cuda")
    _check_nothing_between(d, ws, shapes, 2 * len(shapes))
