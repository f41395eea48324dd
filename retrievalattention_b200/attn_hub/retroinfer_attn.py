"""The two entry points of the reference's ``attn_hub/retroinfer_attn.py``."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _lib

# Where the prefill and dense decode kernels record that a device-side wait gave up, and the dense append that a row did not
# fit (0: none of it): one word in page-locked host memory for all devices and streams, replays of CUDA graphs among them.  The kernels only write it, so a failure stays
# inside its call; it stays set until it is reported, by ``check_prefill_errors`` or by the first call that finds it set.
_word = None
_devices: set = set()


def _status_word(device) -> C.c_int32:
    global _word
    if _word is None:
        address = _lib.lib.ri_status_word()          # the same for every thread that gets here
        if not address:
            raise RuntimeError(f"ri_status_word: {_lib.lib.ri_last_error().decode()}")
        _word = C.c_int32.from_address(address)
    _devices.add(device)
    return _word


def retroinfer_prefill_attn(query_states, key_states, value_states, causal):
    """Dense prefill attention (attn_hub/retroinfer_attn.py:4-13: ``flash_attn_with_kvcache(q, k_cache, v_cache,
    causal)`` over the whole prompt), on this library's tcgen05 kernel ``ri_prefill_attn``.
    query_states [batch, seq_len, heads, 128]; key/value_states [batch, seq_len, kv_heads, 128].  Asynchronous on the
    current stream; ``check_prefill_errors()`` (which synchronises) raises if a device-side wait ever ran out."""
    b, s, hq, d = query_states.shape
    hk = key_states.shape[2]
    if d != 128 or key_states.shape != (b, s, hk, d) or value_states.shape != key_states.shape or hq % hk:
        raise ValueError("retroinfer_prefill_attn: expected q [B,S,Hq,128] and k, v [B,S,Hk,128] with Hq a multiple of Hk")
    if not query_states.is_cuda or any(x.device != query_states.device or x.dtype != query_states.dtype
                                       for x in (key_states, value_states)):
        raise ValueError("retroinfer_prefill_attn: expected q, k and v of one type on one GPU")
    q, k, v = query_states.contiguous(), key_states.contiguous(), value_states.contiguous()
    out = torch.empty_like(q)
    status = _status_word(q.device)
    _lib.check(_lib.lib.ri_prefill_attn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None,
                                        C.addressof(status), b, s, hq, hk, int(bool(causal)), _lib.dtype_code(q.dtype),
                                        _lib.current_stream()), "ri_prefill_attn")
    if status.value and not torch.cuda.is_current_stream_capturing():
        check_prefill_errors()
    return out


def check_prefill_errors() -> None:
    """Raise if any prefill or dense decode call since the last check, replays of captured ones among them, gave up on a
    device-side wait, or a dense cache was full when a row was appended (synchronises)."""
    for device in list(_devices):
        torch.cuda.synchronize(device)
    code = 0 if _word is None else _word.value
    if code:
        _word.value = 0
        if code == _lib.RI_STATUS_CACHE_FULL:
            raise RuntimeError("a token's rows did not fit the dense cache (more decode steps than max_length has room for)")
        raise RuntimeError(f"ri_prefill_attn or ri_dense_decode gave up on a device-side wait (code {code})")


def retroinfer_decode_attn(query_states, key_states, value_states, layer_idx, retroinfer_cache, query_states_next=None):
    """attn_hub/retroinfer_attn.py:17-24 — decode attention is the cache's ``compute``."""
    return retroinfer_cache.compute(
        query_states.contiguous(), layer_idx,
        query_states_next.contiguous() if query_states_next is not None else None)
