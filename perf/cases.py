"""The calls that users of this package make, as measurable cases.

Everything goes through ``flash_kda.fwd`` with the reference signature, as FLA's ``chunk_kda`` and serving code call it:
outputs allocated by the caller, scratch left to the operator.  One case is one shape of such a call: a step of decoding, a
verification step over a few drafted tokens, a prompt, a packed batch of prompts, a throughput batch, a long document.
"""
import math

import torch

import flash_kda
from flashkda_b200 import chunk_states_slots
from flashkda_b200.synth import (BYTES_PER_TOKEN_HEAD, D, FLOPS_PER_TOKEN_HEAD, Workload, make_inputs, varlen_lengths)

STATE_BYTES = {"none": 0, "bf16": 2, "fp32": 4}
EXPORT_EVERY = 4   # 64-token groups: the states that FLA returns for return_intermediate_states


def _case(name, B, T, H, state_in, state_out, lower_bound=-5.0, lens="", export=False):
    """B sequences of T tokens, or (``lens``) one packed batch of sequences of those lengths; the dtypes of the initial and
    final state; the gate's lower bound; whether the states before every 64 tokens are exported as well."""
    return {"name": name, "B": B, "T": T, "H": H, "state_in": state_in, "state_out": state_out,
            "lower_bound": lower_bound, "lens": lens, "export": export}


def _packed(name, lens, H, state_in, state_out, lower_bound=-5.0, export=False):
    return _case(name, 1, sum(lens), H, state_in, state_out, lower_bound, "+".join(str(n) for n in lens), export)


def _lengths(case):
    return [int(n) for n in case["lens"].split("+")] if case["lens"] else None


def listed():
    return [
        # one user's next token: the smallest call there is, all of it latency
        _case("decode_single", 1, 1, 32, "fp32", "fp32"),
        # next token of a full serving batch, states kept in bf16: the states have to be read and written once
        _case("decode_batch", 512, 1, 64, "bf16", "bf16"),
        # the same step from an engine with continuous batching, which hands every batch over as packed sequences
        _packed("decode_packed", [1] * 128, 32, "fp32", "fp32"),
        # verification of speculative decoding: a few drafted tokens behind every sequence of the batch
        _case("verify_drafts", 192, 5, 64, "bf16", "bf16"),
        # one user's prompt of ordinary length: time to first token
        _case("prompt_single", 1, 777, 32, "none", "fp32"),
        # a packed handful of short prompts whose 64-token states are kept for a prefix cache
        _packed("prompts_prefix_cache", [300, 1, 211, 512], 32, "fp32", "fp32", export=True),
        # one dense prefill without states
        _case("prefill_8k", 1, 8192, 32, "none", "none"),
        # the reference's benchmark: one sequence of 8192 tokens, wide model, state in and out
        _case("prefill_8k_wide", 1, 8192, 96, "fp32", "fp32"),
        # the reference's benchmark: the same tokens as six uneven sequences
        _packed("packed_6_wide", [1300, 547, 2048, 963, 271, 3063], 96, "fp32", "fp32"),
        # a packed batch of 64 sequences of 1 to 4096 tokens with bf16 states
        _packed("packed_64", varlen_lengths(), 32, "bf16", "bf16"),
        # offline throughput: a full batch of long sequences (the largest case)
        _case("throughput_32k", 8, 32768, 64, "fp32", "fp32", lower_bound=-3.0),
        # a long document in one call
        _case("document_128k", 1, 131072, 32, "none", "fp32"),
    ]


MAX_TOKEN_HEADS = 8 * 32768 * 64 // 4   # a drawn case stays below the largest listed one
MAX_STATES = 512 * 64                   # (sequence, head) pairs of one call


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more call of the same kinds: sizes over their whole range, odd ones included."""
    kind = rng.choice(["decode", "decode_packed", "verify", "prompt", "batch", "packed", "packed", "long"])
    H = rng.choice([4, 8, 16, 24, 32, 48, 64, 96])
    dtype = rng.choice(["bf16", "fp32"])
    lower_bound = rng.choice([-5.0, -3.0])
    most = max(1, MAX_STATES // H)
    if kind == "decode":
        c = _case("", _log_int(rng, 1, min(512, most)), 1, H, dtype, dtype, lower_bound)
    elif kind == "decode_packed":
        c = _packed("", [1] * _log_int(rng, 2, min(512, most)), H, dtype, dtype, lower_bound)
    elif kind == "verify":
        c = _case("", _log_int(rng, 1, min(512, most)), rng.randint(2, 16), H, dtype, dtype, lower_bound)
    elif kind == "prompt":      # a single prompt, with or without a state to continue from
        c = _case("", 1, _log_int(rng, 17, 16384), H, rng.choice(["none", dtype]), dtype, lower_bound, "", rng.random() < 0.2)
    elif kind == "batch":       # equal sequences side by side
        T = _log_int(rng, 17, 32768)
        B = _log_int(rng, 2, max(2, min(64, MAX_TOKEN_HEADS // (T * H))))
        s = rng.choice(["none", dtype])
        c = _case("", B, T, H, s, s, lower_bound)
    elif kind == "packed":      # unequal sequences, packed
        n = _log_int(rng, 2, 128)
        top = _log_int(rng, 32, max(32, min(8192, 2 * MAX_TOKEN_HEADS // (n * H))))
        lens = [rng.randint(1, top) for _ in range(n)]
        c = _packed("", lens, H, dtype, dtype, lower_bound, rng.random() < 0.2)
    else:                       # one long sequence
        T = _log_int(rng, 16384, max(16385, min(131072, MAX_TOKEN_HEADS // H)))
        c = _case("", 1, T, H, "none", rng.choice(["none", dtype]), lower_bound)
    del c["name"]
    return c


def prepare(case, seed):
    opt = lambda s: None if s == "none" else s
    w = Workload("case", case["B"], case["T"], case["H"], lower_bound=case["lower_bound"], state_in=opt(case["state_in"]),
                 state_out=opt(case["state_out"]), seq_lens=_lengths(case))
    state = make_inputs(w, device="cuda", seed=seed)
    state["extra"] = {}
    if case["export"]:
        slots = chunk_states_slots(case["B"], case["T"], EXPORT_EVERY, seq_lens=_lengths(case))
        states = torch.zeros(slots, case["H"], D, D, dtype=torch.bfloat16, device="cuda")
        state["extra"] = {"chunk_states": states, "chunk_states_every": EXPORT_EVERY}
    return state


def run(state):
    s = state
    flash_kda.fwd(s["q"], s["k"], s["v"], s["g"], s["beta"], s["scale"], s["out"], s["A_log"], s["dt_bias"],
                  s["lower_bound"], s["initial_state"], s["final_state"], s["cu_seqlens"], **s["extra"])
    return {"out": s["out"], "final_state": s["final_state"], "chunk_states": s["extra"].get("chunk_states")}


def work(case):
    """Every input read once and every output written once; the operations of the chunked form."""
    lens = _lengths(case)
    n_seqs = case["B"] if lens is None else len(lens)
    token_heads = case["B"] * case["T"] * case["H"]
    n = token_heads * BYTES_PER_TOKEN_HEAD + case["H"] * (D + 1) * 4
    n += n_seqs * case["H"] * D * D * (STATE_BYTES[case["state_in"]] + STATE_BYTES[case["state_out"]])
    if case["export"]:
        n += chunk_states_slots(case["B"], case["T"], EXPORT_EVERY, seq_lens=lens) * case["H"] * D * D * 2
    return {"bytes": n, "flops": token_heads * FLOPS_PER_TOKEN_HEAD}


def tolerance(case):
    """bf16 operands and a state rounded to bf16 after every chunk; fp32 states hold such values widened."""
    return {"rel": 1e-2}
