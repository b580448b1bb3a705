"""Calls one behind the other on a stream, each working on what the one before wrote, without a synchronisation in between (their
kernels are launched as dependents of whatever is in front of them): the results of the same calls with one after each."""
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
