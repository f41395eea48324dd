"""Dense KV cache with the reference's ``flash_attn_cache`` interface (cache_hub/flash_attn_cache.py:5-151): the
full-attention comparator of the wave index.

Same constructor, ``prefill_update_kv_cache`` / ``sync`` / ``decode_update_kv_cache`` / ``move_gpu`` and attributes
(``key_cache``, ``value_cache``, ``valid_length``, ``context``).  The cache is always resident on the layer's GPU (the
reference falls back to pinned host memory during prefill when HBM is short, :54-76), and it is kept head-major,
``[batch, kv_heads, max_length, head_dim]``, which is the layout this library's decode kernel streams; the tensors
``decode_update_kv_cache`` returns are meant for ``attn_hub.decode_full_flash_attn`` of this package only.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from .. import _lib
from ..attn_hub.retroinfer_attn import _status_word
from .cache import KV_Cache


class flash_attn_cache(KV_Cache):
    def __init__(self, valid_start, layer_num: int, batch_size: int, max_length: int, num_key_value_heads: int,
                 num_heads: int, head_dim: int, dtype: torch.dtype, layer_mapping: dict, num_gpus: int,
                 model_size: int) -> None:
        super().__init__(layer_num, batch_size, max_length, num_key_value_heads, num_heads, head_dim, dtype,
                         layer_mapping, num_gpus, model_size)
        if head_dim != 128:
            raise ValueError("the decode kernel is built for head_dim 128")
        self.valid_start = valid_start
        self._longest = None                # rows of the longest request, counted on the host from the first prefill call on
        self.valid_length = None            # [batch] int32 on the first layer's device, set by the first prefill call
        self.allocated = True
        mk = lambda ldx: torch.zeros((batch_size, self.kv_head, max_length, head_dim), dtype=dtype,   # noqa: E731
                                     device=layer_mapping[str(ldx)])
        self.key_cache = [mk(ldx) for ldx in range(layer_num)]
        self.value_cache = [mk(ldx) for ldx in range(layer_num)]
        self._rows = torch.arange(batch_size, device=layer_mapping[str(0)])

    def move_gpu(self):
        """The reference moves a host-resident cache to the GPUs here (:85-89); this one is already there."""
        return None

    def prefill_update_kv_cache(self, query_states, key_states, value_states, layer_idx, start_bdx):
        """One request, one layer (:92-127).  key/value_states: [1, seq_len, kv_heads, head_dim]."""
        bsz, seq_len, _, _ = key_states.shape
        assert bsz == 1, "Multi-batch prefilling only support prefill single batch one by one."
        assert seq_len <= self.max_length, f"Prefilling sequence length {seq_len} exceeds max length {self.max_length}."
        if self.valid_length is None:
            vs = np.asarray(self.valid_start)
            self._longest = int(seq_len - vs.min())
            self.valid_length = torch.from_numpy(seq_len - vs).to(torch.int32).to(self.layer_mapping[str(0)])
        vs = int(self.valid_start[start_bdx])
        n = seq_len - vs
        self.key_cache[layer_idx][start_bdx, :, :n].copy_(key_states[0, vs:].transpose(0, 1))
        self.value_cache[layer_idx][start_bdx, :, :n].copy_(value_states[0, vs:].transpose(0, 1))
        if layer_idx == self.layer_num - 1 and start_bdx + bsz == self.batch_size:
            self.context += seq_len
        return key_states[:, vs:], value_states[:, vs:]

    def sync(self, layer_idx, start_bdx):
        """The reference waits for its side-stream copy (:129-130); the copy above is in stream order."""
        return None

    def _one_launch(self, keys, key_states, value_states, values=None) -> bool:
        """Whether the rows can be appended by one kernel for both tensors: what a decode step hands over, 16-bit rows of
        the cache's own type, dense and aligned, on the current device, into tensors as they were made (a caller may have
        put others in their place), and rows that fit (a full cache is refused by the indexing below).  The lengths are counted on the host here; where they move on without it, as in
        replays of a CUDA graph, the kernel itself leaves out a row that does not fit, and ``check_prefill_errors`` or the
        next ``decode_full_flash_attn`` says so.  Six launches of indexing kernels otherwise."""
        if not keys.is_cuda or self._longest is None or self._longest >= self.max_length:
            return False
        if values is None:
            values = keys
        dev, dtype, n, b, hk, d = keys.device, keys.dtype, self.valid_length, self.batch_size, self.kv_head, self.head_dim
        if not (dev.index == torch.cuda.current_device() and n.device == dev and n.dtype == torch.int32
                and n.is_contiguous() and n.shape == (b,) and key_states.element_size() == 2):
            return False
        cache, rows = (b, hk, self.max_length, d), (b, 1, hk, d)
        if not (keys.shape == cache and values.shape == cache and key_states.shape == rows and value_states.shape == rows):
            return False
        for x in (keys, values, key_states, value_states):
            if x.dtype != dtype or x.device != dev or x.requires_grad or not x.is_contiguous() or x.data_ptr() % 16:
                return False
        return True

    def decode_update_kv_cache(self, key_states, value_states, layer_idx):
        """Append one token per request (:133-151).  key/value_states: [batch, 1, kv_heads, head_dim]."""
        keys, values = self.key_cache[layer_idx], self.value_cache[layer_idx]
        if self._one_launch(keys, key_states, value_states, values):
            _lib.check(_lib.lib.ri_dense_append(key_states.data_ptr(), value_states.data_ptr(), keys.data_ptr(),
                                                values.data_ptr(), self.valid_length.data_ptr(),
                                                C.addressof(_status_word(keys.device)), self.batch_size, self.kv_head,
                                                self.max_length, _lib.current_stream()), "ri_dense_append")
            torch.autograd.graph.increment_version((keys, values))      # as the indexing form does by itself
        else:
            pos = self.valid_length.to(keys.device).long()
            keys[self._rows.to(pos.device), :, pos] = key_states[:, 0]
            values[self._rows.to(pos.device), :, pos] = value_states[:, 0]
        if layer_idx == self.layer_num - 1:
            self.context += 1
            self.valid_length += 1
            if self._longest is not None:
                self._longest += 1
        return self.key_cache[layer_idx], self.value_cache[layer_idx]
