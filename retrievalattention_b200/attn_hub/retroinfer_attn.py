"""The two entry points of the reference's ``attn_hub/retroinfer_attn.py``."""
from __future__ import annotations

import torch

from .. import _lib

# Status words of the prefill and dense decode kernels, one per device: 0, or where a device-side wait gave up.  A word stays set until
# ``check_prefill_errors`` reports it; every CHECK_EVERY calls a copy of it is sent to the host and looked at when it has
# arrived, so that a failure surfaces without a call ever waiting for the GPU.
CHECK_EVERY = 64
_words: dict = {}
_captured: list = []      # words of calls captured in a graph before the device had one


class _StatusWord:
    def __init__(self, device):
        self.word = torch.zeros((1,), dtype=torch.int32, device=device)
        torch.cuda.current_stream(device).synchronize()      # cleared before a kernel of any other stream looks at it
        self.address = self.word.data_ptr()
        self.calls = 0
        self.host = None                                     # (pinned copy, event) on its way

    def tick(self):
        self.calls += 1
        pending = self.host                                  # read once: another thread's call may clear it
        if pending is not None:
            copy, arrived = pending
            if arrived.query():
                self.host = None
                if int(copy):
                    check_prefill_errors()
        elif self.calls >= CHECK_EVERY:
            self.calls = 0
            copy = torch.empty((1,), dtype=torch.int32, pin_memory=True)
            copy.copy_(self.word, non_blocking=True)
            arrived = torch.cuda.Event()
            arrived.record()
            self.host = (copy, arrived)


def _status_word(device, capturing: bool) -> _StatusWord:
    word = _words.get(device)
    if word is None:
        if capturing:      # nothing may be waited for here: this word is cleared by the graph itself
            word = _StatusWord.__new__(_StatusWord)
            word.word = torch.zeros((1,), dtype=torch.int32, device=device)
            word.address, word.calls, word.host = word.word.data_ptr(), 0, None
            _captured.append(word.word)
            return word
        word = _words.setdefault(device, _StatusWord(device))
    return word


def retroinfer_prefill_attn(query_states, key_states, value_states, causal):
    """Dense prefill attention (attn_hub/retroinfer_attn.py:4-13: ``flash_attn_with_kvcache(q, k_cache, v_cache,
    causal)`` over the whole prompt), on this library's tcgen05 kernel ``ri_prefill_attn``.
    query_states [batch, seq_len, heads, 128]; key/value_states [batch, seq_len, kv_heads, 128].  Asynchronous on the
    current stream; ``check_prefill_errors()`` (which synchronises) raises if a device-side wait ever ran out."""
    b, s, hq, d = query_states.shape
    hk = key_states.shape[2]
    if d != 128 or key_states.shape != (b, s, hk, d) or value_states.shape != key_states.shape or hq % hk:
        raise ValueError("retroinfer_prefill_attn: expected q [B,S,Hq,128] and k, v [B,S,Hk,128] with Hq a multiple of Hk")
    q, k, v = query_states.contiguous(), key_states.contiguous(), value_states.contiguous()
    out = torch.empty_like(q)
    capturing = torch.cuda.is_current_stream_capturing()
    status = _status_word(q.device, capturing)
    _lib.check(_lib.lib.ri_prefill_attn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None,
                                        status.address, b, s, hq, hk, int(bool(causal)), _lib.dtype_code(q.dtype),
                                        _lib.current_stream()), "ri_prefill_attn")
    if not capturing:
        status.tick()
    return out


def check_prefill_errors() -> None:
    """Raise if any prefill call since the last check gave up on a device-side wait (synchronises)."""
    bad = {int(w.item()) for w in _captured} - {0}
    _captured.clear()
    for status in list(_words.values()):
        torch.cuda.synchronize(status.word.device)
        code = int(status.word.item())
        if code:
            bad.add(code)
            status.word.zero_()
            torch.cuda.synchronize(status.word.device)
        status.calls, status.host = 0, None
    if bad:
        raise RuntimeError(f"ri_prefill_attn or ri_dense_decode gave up on a device-side wait (codes {sorted(bad)})")


def retroinfer_decode_attn(query_states, key_states, value_states, layer_idx, retroinfer_cache, query_states_next=None):
    """attn_hub/retroinfer_attn.py:17-24 — decode attention is the cache's ``compute``."""
    return retroinfer_cache.compute(
        query_states.contiguous(), layer_idx,
        query_states_next.contiguous() if query_states_next is not None else None)
