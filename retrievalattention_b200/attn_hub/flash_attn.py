"""Full attention over the dense cache, with the reference's interface (attn_hub/flash_attn.py:4-30): the comparator
of the wave-index path.  Decoding runs ``ri_dense_decode`` over the head-major cache of ``cache_hub.flash_attn_cache``;
``check_prefill_errors()`` reports its device-side waits too."""
from __future__ import annotations

import ctypes as C

import torch

from .. import _lib
from ..kernels import weighted_flash_decoding
from ..status import report
from .retroinfer_attn import _status_word, check_prefill_errors, retroinfer_prefill_attn  # noqa: F401


def prefill_full_flash_attn(query_states, key_states, value_states, causal):
    """attn_hub/flash_attn.py:4-13 — dense (causal) attention over the prompt."""
    return retroinfer_prefill_attn(query_states, key_states, value_states, causal)


def _dense_form(q, k, v, valid_length) -> bool:
    """Whether the call has the form the dense cache's own kernel takes (everything as ``flash_attn_cache`` keeps it);
    any other goes through the general operator.  Written out: it runs once per layer and token."""
    if q.dim() != 4 or k.dim() != 4 or not q.is_cuda:
        return False
    dev, dtype = q.device, q.dtype
    if dev.index != torch.cuda.current_device() or (dtype != torch.bfloat16 and dtype != torch.float16):
        return False
    b, one, hq, d = q.shape
    kb, hk, length, kd = kv = k.shape
    g = b * hk
    return (one == 1 and d == 128 and kb == b and kd == 128 and v.shape == kv and hk > 0 and hq % hk == 0
            and 1 <= hq // hk <= 8 and 1 <= g <= 65535 and g * length < (1 << 31) - 16 and length > 0
            and valid_length.shape == (b,) and valid_length.dtype == torch.int32 and valid_length.device == dev
            and valid_length.is_contiguous() and q.is_contiguous() and k.is_contiguous() and v.is_contiguous()
            and k.device == dev and v.device == dev and k.dtype == dtype and v.dtype == dtype
            and (q.data_ptr() | k.data_ptr() | v.data_ptr()) % 16 == 0)


def decode_full_flash_attn(query_states, key_states, value_states, layer_idx, full_attn_cache):
    """attn_hub/flash_attn.py:17-30.  query_states [batch, 1, heads, 128]; key/value_states: the cache tensors
    ``[batch, kv_heads, max_length, 128]`` that ``flash_attn_cache.decode_update_kv_cache`` returned."""
    c = full_attn_cache
    extra = 1 if layer_idx < c.layer_num - 1 else 0                                      # :19
    b, _, hq, d = query_states.shape
    hk, length = key_states.shape[1], key_states.shape[2]
    g, gs = b * hk, hq // hk
    if _dense_form(query_states, key_states, value_states, c.valid_length):
        out = torch.empty_like(query_states)
        status = _status_word(out.device)
        scratch = torch.empty((_lib.lib.ri_dense_decode_scratch_bytes(b, hk, gs),), dtype=torch.uint8, device=out.device)
        _lib.check(_lib.lib.ri_dense_decode(
            query_states.data_ptr(), key_states.data_ptr(), value_states.data_ptr(), c.valid_length.data_ptr(), extra,
            out.data_ptr(), scratch.data_ptr(), C.addressof(status), b, hk, gs, length, _lib.dtype_code(out.dtype), _lib.current_stream()),
            "ri_dense_decode")
        report(status)
        return out
    valid = c.valid_length + extra
    seqlens = valid.to(query_states.device).to(torch.int32).repeat_interleave(hk)
    out = weighted_flash_decoding(query_states.reshape(g, 1, gs, d), key_states.view(g, length, 1, d),
                                  value_states.view(g, length, 1, d), cache_seqlens=seqlens)
    return out.view(b, 1, hq, d)
