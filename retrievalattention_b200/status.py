"""The process's status word, on the host.

Prefill, dense decode and wave decode kernels record in it that a device-side wait gave up, and the dense append that a row did
not fit (0: none of it): one word in page-locked host memory for all devices and streams, replays of CUDA graphs among them.  The
kernels only write it, so a failure stays inside its call; it stays set until it is reported, by ``check`` or by the first call
that finds it set.
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib

_word = None
_devices: set = set()


def word(device) -> C.c_int32:
    """The word, for calls that run on ``device``."""
    global _word
    if _word is None:
        address = _lib.lib.ri_status_word()          # the same for every thread that gets here
        if not address:
            raise RuntimeError(f"ri_status_word: {_lib.lib.ri_last_error().decode()}")
        _word = C.c_int32.from_address(address)
    _devices.add(device)
    return _word


def _kernel(code: int) -> str:
    # what the kernels' waits are numbered by; a second bound of a wait, by count, adds 100
    return {2: "ri_prefill_attn", 3: "ri_prefill_attn", 4: "ri_dense_decode", 5: "ri_wave_decode_layer"}.get(code % 100 // 10, "a kernel")


def check() -> None:
    """Raise if any prefill or decode call since the last check, replays of captured ones among them, gave up on a device-side
    wait, or a dense cache was full when a row was appended (synchronises)."""
    for device in list(_devices):
        torch.cuda.synchronize(device)
    code = 0 if _word is None else _word.value
    if code:
        _word.value = 0
        if code == _lib.RI_STATUS_CACHE_FULL:
            raise RuntimeError("a token's rows did not fit the dense cache (more decode steps than max_length has room for)")
        raise RuntimeError(f"{_kernel(code)} gave up on a device-side wait (code {code})")


def report(status: C.c_int32) -> None:
    """``check`` where the word is set; for calls, after their launches.  Under a capture nothing has run that could have
    set it."""
    if status.value and not torch.cuda.is_current_stream_capturing():
        check()
