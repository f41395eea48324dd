"""The two entry points of the reference's ``attn_hub/retroinfer_attn.py``."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _lib, status as _status

_status_word = _status.word


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
    _status.report(status)
    return out


def check_prefill_errors() -> None:
    """Raise if any prefill or decode call (dense or wave index) since the last check, replays of captured ones among them, gave
    up on a device-side wait, or a dense cache was full when a row was appended (synchronises)."""
    _status.check()


def retroinfer_decode_attn(query_states, key_states, value_states, layer_idx, retroinfer_cache, query_states_next=None):
    """attn_hub/retroinfer_attn.py:17-24 — decode attention is the cache's ``compute``."""
    return retroinfer_cache.compute(
        query_states.contiguous(), layer_idx,
        query_states_next.contiguous() if query_states_next is not None else None)
