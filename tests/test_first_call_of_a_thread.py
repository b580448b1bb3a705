"""A call that is the first CUDA work of its host thread, in every form of the forward."""
import threading

import pytest
import torch

import flashkda_b200
from flashkda_b200.synth import Workload, make_inputs, to_device

pytestmark = pytest.mark.gpu

SHAPES = {   # B, T, H, sequence lengths
    "decode": (7, 1, 8, None), "decode_packed": (1, 70, 4, [1] * 70), "short": (9, 5, 8, None), "prompt": (1, 100, 8, None),
    "slabs": (1, 1100, 4, None), "chains_between": (1, 1100, 80, None), "one_kernel": (80, 40, 1, None), "ragged": (1, 400, 4, [300, 1, 99]),
}


@pytest.mark.parametrize("own_scratch", [False, True])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_first_call_of_a_thread(name, own_scratch):
    B, T, H, lens = SHAPES[name]
    w = Workload("t", B, T, H, state_in="fp32", state_out="fp32", lower_bound=-1.0, seq_lens=lens)
    d = to_device(make_inputs(w, seed=3), "cuda")
    ws = None if own_scratch else torch.empty((flashkda_b200.get_workspace_size(w.tokens, H, w.n_seqs),), dtype=torch.uint8, device="cuda")
    errors = []

    def call():
        try:
            flashkda_b200.fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], d["out"], d["A_log"], d["dt_bias"], d["lower_bound"],
                              d["initial_state"], d["final_state"], d["cu_seqlens"], workspace=ws)
        except Exception as e:
            errors.append(e)

    call()
    torch.cuda.synchronize()
    want = d["out"].clone(), d["final_state"].clone()
    d["out"].zero_()
    d["final_state"].zero_()
    torch.cuda.synchronize()
    t = threading.Thread(target=call)
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert not errors
    assert torch.equal(d["out"], want[0]) and torch.equal(d["final_state"], want[1])
