"""flashkda_b200: Kimi Delta Attention forward for NVIDIA B200 (sm_100a).

Host-side mirror of the reference operator API (``flash_kda/__init__.py:5-41`` and the
checks of ``csrc/flash_kda.cpp:44-174`` in the reference project): the same ``fwd``
signature, argument meaning and error conditions, on top of a C-ABI CUDA library
(``include/flashkda_b200.h``).  There is no CPU path: calling ``fwd`` without the built
library or without CUDA tensors raises.
"""
import os

import torch

from . import _lib

__all__ = ["fwd", "get_workspace_size", "last_launch_count", "default_algo", "device_status", "chunk_states_slots"]

D = 128
_ENV_ALGO = "FLASHKDA_B200_ALGO"


def default_algo() -> str:
    return os.environ.get(_ENV_ALGO, "auto")


def get_workspace_size(T_total: int, H: int, N: int = 1, algo: str = None) -> int:
    """Scratch bytes one ``fwd`` call allocates (reference: ``get_workspace_size``,
    csrc/flash_kda.cpp:5-26)."""
    a = _lib.ALGOS[algo or default_algo()]
    return int(_lib.lib().fkda_workspace_bytes(int(T_total), int(H), int(N), a))


def _load_host_fwd(*args):
    """First call: binds the native host side (argument checks, scratch allocation, launch)."""
    global _host_fwd
    _lib.lib()   # the CUDA library, with its own error when it has not been built
    try:
        from . import _host
    except ImportError as e:
        raise RuntimeError("flashkda_b200/_host.so is missing or does not load: build it with "
                           f"`python -m flashkda_b200.build` ({e})") from e
    _host_fwd = _host.fwd
    return _host_fwd(*args)


_host_fwd = _load_host_fwd


def fwd(q, k, v, g, beta, scale, out, A_log, dt_bias, lower_bound, initial_state=None, final_state=None,
        cu_seqlens=None, *, algo: str = None, workspace: torch.Tensor = None, phase_mask: int = 0, flags: int = 0,
        chunk_states: torch.Tensor = None, chunk_states_every: int = 4):
    """FlashKDA forward; writes ``out`` (and ``final_state``) in place and returns ``None``.

    q, k, v, g, out: bf16 ``[B, T, H, 128]``; beta: bf16 ``[B, T, H]`` logits; A_log: fp32
    ``[H]``; dt_bias: fp32 ``[H, 128]``; states: bf16 or fp32 ``[N, H, 128, 128]`` (``[V, K]``
    layout); cu_seqlens: int64 ``[N + 1]`` (then ``B`` must be 1).  Work is enqueued on the
    current CUDA stream of ``q.device`` without synchronising.

    ``algo`` and ``workspace`` are additions to the reference signature: the implementation
    selector (default from ``$FLASHKDA_B200_ALGO`` or "auto") and an optional caller-owned
    uint8 scratch tensor of at least ``get_workspace_size(...)`` bytes.  ``phase_mask`` runs the
    two stages of the forward apart (see ``fkda_fwd_params.phase_mask``) and ``flags`` selects kernel variants for tests
    (``fkda_fwd_params.flags``); leave both 0.

    ``chunk_states`` (optional, bf16 ``[slots, H, 128, 128]``) receives the state of every sequence before each
    group of ``chunk_states_every`` 16-token chunks (``chunk_states_slots`` gives the slot count); with the default
    of 4 these are the states FLA's ``chunk_kda`` returns as ``h`` for ``return_intermediate_states=True``.

    The call returns without synchronising, so it cannot tell whether a kernel gave up on one of its
    bounded internal waits (possible only when other long-running kernels hold the GPU's SMs for
    seconds); ``device_status(workspace)`` reports that after the stream has been synchronised.
    """
    _host_fwd(q, k, v, g, beta, scale, out, A_log, dt_bias, lower_bound, initial_state, final_state, cu_seqlens, algo,
              workspace, phase_mask, flags, chunk_states, chunk_states_every)


def chunk_states_slots(B: int, T: int, every: int = 4, seq_lens=None) -> int:
    """Slots a ``chunk_states`` tensor needs: per sequence ``ceil(len / (16 * every))``; pass the lengths of a
    ragged batch as ``seq_lens``."""
    group = 16 * int(every)
    if seq_lens is not None:
        return int(sum((int(x) + group - 1) // group for x in seq_lens))
    return int(B) * ((int(T) + group - 1) // group)


def device_status(workspace: torch.Tensor) -> int:
    """Synchronises the current stream and returns the device status word of the last call that used
    ``workspace`` (0 = ok; see ``fkda_device_status``)."""
    with torch.cuda.device(workspace.device):
        stream = torch.cuda.current_stream(workspace.device).cuda_stream
        return int(_lib.lib().fkda_device_status(workspace.data_ptr(), stream))


def last_launch_count() -> int:
    """Kernels launched by the last successful ``fwd`` on this thread."""
    return int(_lib.lib().fkda_last_launch_count())
