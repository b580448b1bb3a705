"""Scratch that a call makes use of but can do without (records of the later chunks, 75 to 124 chains of a fixed batch): taken only
where the allocator has room for it, so that nobody else's cached memory is given back for it, and not into a graph."""
import pytest
import torch

import flashkda_b200
from flashkda_b200.synth import Workload, make_inputs, to_device

pytestmark = pytest.mark.gpu

T, H = 2048, 80
WANTED = 80 * 128 * 14656   # the records, the better part of it


def _problem(seed=4):
    return to_device(make_inputs(Workload("w", 1, T, H, state_out="fp32", lower_bound=-1.0), seed=seed), "cuda")


def _call(d):
    flashkda_b200.fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], d["out"], d["A_log"], d["dt_bias"], d["lower_bound"],
                      None, d["final_state"], None)
    return flashkda_b200.last_launch_count()


@pytest.fixture
def limited():
    """Limits this process to what it holds now and `room` bytes more, none of it cached."""
    def limit(room):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(0).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / total)
    yield limit
    torch.cuda.set_per_process_memory_fraction(1.0)


def _counts():
    s = torch.cuda.memory_stats()
    return s["num_alloc_retries"], s["num_ooms"]


@pytest.mark.parametrize("room,launches", [(0.5, (1,)), (1.6, (1, 5)), (2.4, (5,))])
def test_room_for_records(limited, room, launches):
    """Whatever form a call takes, nothing is given back to the device for it.  In between it depends on what is cached, which
    includes the unused ends of segments that other tests' tensors hold."""
    d = _problem()
    limited(int(room * WANTED))
    before = _counts()
    cached = torch.empty(WANTED // 4, dtype=torch.uint8, device="cuda")
    del cached                                   # a block that stays in the cache
    reserved = torch.cuda.memory_reserved()
    outs = []
    for _ in range(3):
        assert _call(d) in launches
        outs.append((d["out"].cpu(), d["final_state"].cpu()))
    assert torch.cuda.memory_reserved() >= reserved and _counts() == before
    torch.cuda.set_per_process_memory_fraction(1.0)
    assert _call(d) == 5
    assert all(torch.equal(d["out"].cpu(), o) and torch.equal(d["final_state"].cpu(), s) for o, s in outs)


def test_a_graph_does_not_keep_the_records():
    d = _problem()
    assert _call(d) == 5
    out, state = d["out"].clone(), d["final_state"].clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    reserved = torch.cuda.memory_reserved()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert _call(d) == 1
    assert torch.cuda.memory_reserved() - reserved < WANTED // 4
    d["out"].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(d["out"], out) and torch.equal(d["final_state"], state)
