"""Calls that use the library's side stream for 75 to 124 chains of a fixed batch, beside other threads' and streams' calls: no call
is refused for another's capture or waits for what another's stream waits for, and the bits are those of a lone call."""
import threading

import pytest
import torch

import flashkda_b200
from flashkda_b200.synth import Workload, make_inputs, to_device

pytestmark = pytest.mark.gpu

HEADS = {"mid": 80, "few": 8}


class Problem:
    def __init__(self, kind, seed):
        w = Workload("s", 1, 2048, HEADS[kind], state_out="fp32", lower_bound=-1.0)
        self.d = to_device(make_inputs(w, seed=seed), "cuda")
        self.ws = torch.empty(flashkda_b200.get_workspace_size(w.T, w.H, 1), dtype=torch.uint8, device="cuda")
        self.launches = self.call()
        self.want = self.results()

    def call(self):
        d = self.d
        flashkda_b200.fwd(d["q"], d["k"], d["v"], d["g"], d["beta"], d["scale"], d["out"], d["A_log"], d["dt_bias"], d["lower_bound"],
                          None, d["final_state"], None, workspace=self.ws)
        return flashkda_b200.last_launch_count()

    def results(self):
        torch.cuda.synchronize()
        got = self.d["out"].clone(), self.d["final_state"].clone()
        self.d["out"].zero_()
        self.d["final_state"].zero_()
        torch.cuda.synchronize()
        return got

    def check(self):
        assert all(torch.equal(x, y) for x, y in zip(self.results(), self.want))
        assert flashkda_b200.device_status(self.ws) == 0


def _in_threads(*fns):
    """Their results, each from a thread of its own; an exception is raised here."""
    box = [None] * len(fns)

    def run(i):
        try:
            box[i] = fns[i]()
        except Exception as e:
            box[i] = e
    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(fns))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x in box:
        if isinstance(x, Exception):
            raise x
    return box


@pytest.mark.parametrize("captured,eager", [("mid", "mid"), ("mid", "few"), ("few", "mid")])
def test_beside_another_threads_capture(captured, eager):
    a, b = Problem(captured, 1), Problem(eager, 2)
    stream, other, graph = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()

    def on_other():
        with torch.cuda.stream(other):
            return b.call()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            assert a.call() == a.launches
            n = _in_threads(on_other)[0]
            assert a.call() == a.launches   # a second call in the same capture
        finally:
            graph.capture_end()
    assert n == (1 if (captured, eager) == ("mid", "mid") else b.launches)
    b.check()
    for _ in range(2):
        graph.replay()
        a.check()
    with torch.cuda.stream(other):
        assert b.call() == b.launches   # the side stream is free again
    b.check()


@pytest.mark.parametrize("blocked,free", [("mid", "mid"), ("few", "mid"), ("mid", "few")])
def test_beside_a_stream_that_waits(blocked, free):
    a, b = Problem(blocked, 1), Problem(free, 2)
    s1, s2, e1, e2 = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Event(), torch.cuda.Event()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(600_000_000)   # 0.3 s
        assert a.call() == a.launches
        e1.record()
    with torch.cuda.stream(s2):
        assert b.call() == (1 if (blocked, free) == ("mid", "mid") else b.launches)
        e2.record()
    e2.synchronize()
    assert not e1.query()
    e1.synchronize()
    a.check()
    b.check()


def test_two_threads():
    problems = [Problem("mid", 5), Problem("mid", 6)]

    def worker(p, wait):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(20):
                p.call()
                if wait:   # the side stream falls free for the other one now and then
                    stream.synchronize()
        stream.synchronize()
    _in_threads(lambda: worker(problems[0], True), lambda: worker(problems[1], False))
    for p in problems:
        p.check()
