"""Seeded random problems (ragged and fixed batches, short and long sequences, all state options): whatever path
the dispatch picks (decode kernel, one-chunk kernel, one-kernel forward, row slices with or without the slab pipeline) must
give what the plain two-kernel form gives on the same inputs, bit for bit (the decode kernel: to its summation-order
tolerance), and must agree with the CUDA-core implementation within the parity tolerances."""
import random

import pytest
import torch

import flashkda_b200
import oracle
from flashkda_b200 import _lib
from flashkda_b200.synth import Workload, make_inputs
from test_gpu_parity import run_gpu

pytestmark = pytest.mark.gpu

# both stages by name and no one-chunk kernel: prepare and row slices in one launch each
PLAIN = dict(flags=_lib.FLAG_NO_DECODE | _lib.FLAG_NO_SHORT | _lib.FLAG_NO_SLABS, phase_mask=_lib.PHASE_PREPARE | _lib.PHASE_RECURRENCE)


def _random_workload(rng):
    H = rng.choice([1, 2, 3, 4, 8, 16])
    st_in = rng.choice([None, "bf16", "fp32"])
    st_out = st_in if st_in is not None and rng.random() < 0.8 else rng.choice([None, st_in or "fp32"])
    if st_in is not None and st_out is not None:
        st_out = st_in
    lb = rng.choice([-5.0, -2.0, -0.5])
    kind = rng.choice(["fixed_short", "fixed_one", "fixed_long", "ragged_short", "ragged_ones", "ragged_mixed", "ragged_long"])
    if kind == "fixed_short":
        return Workload("r", rng.randint(1, 70), rng.randint(2, 16), H, state_in=st_in, state_out=st_out, lower_bound=lb)
    if kind == "fixed_one":
        return Workload("r", rng.randint(1, 90), 1, H, state_in=st_in, state_out=st_out, lower_bound=lb)
    if kind == "fixed_long":
        return Workload("r", rng.randint(1, 6), rng.choice([17, 64, 100, 257, 1024, 1500]), H, state_in=st_in, state_out=st_out,
                        lower_bound=lb)
    n = rng.randint(2, 80)
    if kind == "ragged_short":
        lens = [rng.randint(0, 16) for _ in range(n)]
    elif kind == "ragged_ones":
        lens = [1] * n
    elif kind == "ragged_mixed":
        lens = [rng.choice([0, 1, 2, 5, 16, 17, 40, 130]) for _ in range(n)]
    else:
        lens = [rng.randint(1, 600) for _ in range(rng.randint(2, 12))]
    if sum(lens) == 0:
        lens[0] = 3
    return Workload("r", 1, sum(lens), H, state_in=st_in, state_out=st_out, lower_bound=lb, seq_lens=lens)


@pytest.mark.parametrize("seed", range(48))
def test_dispatch_paths_agree(seed):
    rng = random.Random(1000 + seed)
    w = _random_workload(rng)
    inp = make_inputs(w, seed=seed)
    out_d, hT_d = run_gpu(inp, "tc")
    launches = flashkda_b200.last_launch_count()
    out_p, hT_p = run_gpu(inp, "tc", **PLAIN)
    assert flashkda_b200.last_launch_count() == (2 if w.seq_lens is None else 3)
    one_token_each = (w.seq_lens is None and w.T == 1) or (w.seq_lens is not None and all(L == 1 for L in w.seq_lens))
    if one_token_each and launches in (1, 5):      # the decode kernel served the call
        assert oracle.err_ratio(out_p, out_d) <= 2e-3
        if hT_d is not None:
            assert oracle.err_ratio(hT_p.float(), hT_d.float()) <= 1e-3
    else:
        assert torch.equal(out_d, out_p), (w, launches)
        if hT_d is not None:
            assert torch.equal(hT_d, hT_p), (w, launches)
    out_c, hT_c = run_gpu(inp, "twopass")
    assert oracle.err_ratio(out_c, out_d) <= 4e-3
    if hT_d is not None:
        assert oracle.err_ratio(hT_c.float(), hT_d.float()) <= 4e-3
