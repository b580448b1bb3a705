"""Fixed batches with fewer chains than SMs but more than half as many: the one-kernel form walks the first chunks while the idle SMs
prepare the records of the others for a row-slice kernel.  Against the one-kernel form alone, bit for bit: sizes at the edges of the
dispatch and of the chunks, states of both types, exported states, and a workspace that holds no records."""
import pytest
import torch

import flashkda_b200
from flashkda_b200 import _lib
from flashkda_b200.synth import Workload, make_inputs, to_device
from test_one_kernel_forward import _call

pytestmark = pytest.mark.gpu


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("chains,T,state,every", [
    ("least", 1024, "fp32", None), ("least", 1025, "bf16", 3), ("least", 4099, None, None), ("most", 192 * 16, "fp32", None),
    ("most", 192 * 16 - 1, "bf16", None), ("most", 256 * 16 + 7, "fp32", 5), ("least", 94 * 16, "bf16", 3), ("least", 94 * 16 + 1, "bf16", 3),
    ("most", 287 * 16, "fp32", 5), ("most", 288 * 16 - 9, "fp32", 5)])
def test_equals_the_one_kernel_form(chains, T, state, every):
    n = {"least": _sms() // 2 + 1, "most": _sms() - 24}[chains]
    inp = make_inputs(Workload("m", 1, T, n, state_in=state, state_out=state, lower_bound=-1.0), seed=11)
    a = _call(inp, every=every)
    expect = 5 if T <= 255 * 16 else 7
    if every is not None and (T + 15) // 16 * (_sms() - n) < 6912:
        expect = 1   # below the line of calls that export states
    assert flashkda_b200.last_launch_count() == expect
    b = _call(inp, flags=_lib.FLAG_NO_WIDE, every=every)
    assert flashkda_b200.last_launch_count() == 1
    for x, y in zip(a, b):
        assert x is None or torch.equal(x, y)


def test_several_sequences_and_its_lines():
    sms = _sms()
    for B, T, H, expect in ((3, 2000, 30, 5), (1, 1008, sms // 2 + 1, 1), (1, 8192, sms - 23, 1), (1, 191 * 16, sms - 24, 1)):
        inp = make_inputs(Workload("l", B, T, H, state_out="fp32", lower_bound=-1.0), seed=2)
        a = _call(inp)
        assert flashkda_b200.last_launch_count() == expect
        b = _call(inp, flags=_lib.FLAG_NO_SLABS)
        assert flashkda_b200.last_launch_count() == 1
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_a_workspace_without_room_for_records_and_none():
    inp = to_device(make_inputs(Workload("w", 1, 2048, 80, state_out="fp32", lower_bound=-1.0), seed=4), "cuda")
    sms, outs = _sms(), []
    least = 256 + 256 + (sms * 4 + 255) // 256 * 256 + sms * 32768   # header, tables, flags, hand-over states
    for ws, expect in ((None, 5), (torch.empty(least, dtype=torch.uint8, device="cuda"), 1)):
        inp["out"].zero_()
        flashkda_b200.fwd(inp["q"], inp["k"], inp["v"], inp["g"], inp["beta"], inp["scale"], inp["out"], inp["A_log"], inp["dt_bias"],
                          inp["lower_bound"], None, inp["final_state"], None, workspace=ws)
        assert flashkda_b200.last_launch_count() == expect
        outs.append((inp["out"].clone(), inp["final_state"].clone()))
    assert all(torch.equal(x, y) for x, y in zip(*outs))
