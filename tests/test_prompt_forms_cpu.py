"""Which prompts the index build reads in place, and what it refuses before anything reaches a kernel."""
from types import SimpleNamespace

import pytest
import torch


def index_tensors(z, c, n, steady, d=128, dt=torch.bfloat16):
    mk = lambda *s, t=dt: torch.zeros(s, dtype=t)        # noqa: E731
    return dict(centroids=mk(z, c, d), value_sum=mk(z, c, d), cluster_size=mk(z, c), cluster_count=mk(z, c, t=torch.int32),
                cluster_offset=mk(z, c + 1, t=torch.int32), empty=mk(z, c, t=torch.bool), keys=mk(z, n, d), values=mk(z, n, d),
                steady_keys=mk(z, steady, d), steady_values=mk(z, steady, d))


@pytest.mark.parametrize("head_dim", [64, 128, 256])
def test_prompt_build_refuses_host_tensors_and_other_head_dims(head_dim):
    from retrievalattention_b200.cache_hub.kmeans import build_prompt_index

    k = torch.zeros((200, 2, head_dim), dtype=torch.bfloat16)
    with pytest.raises(AssertionError, match="GPU only"):
        build_prompt_index(k, k, 1, 4, 64, index_tensors(2, 32, 132, 68))


class Rows:
    """What the rule looks at, without memory behind it."""

    def __init__(self, shape, dtype=torch.bfloat16, device="cuda:0", requires_grad=False):
        self.shape, self.dtype, self.device, self.requires_grad = torch.Size(shape), dtype, torch.device(device), requires_grad


@pytest.mark.parametrize("wanted,change", [
    (True, {}),
    (True, dict(requires_grad=True, grad=False)),
    (False, dict(requires_grad=True)),
    (False, dict(device="cuda:1")),                       # clustered where it lies, then copied
    (False, dict(device="cpu")),
    (False, dict(dtype=torch.float16)),                   # clustered in its own type
    (False, dict(dtype=torch.float32)),
    (False, dict(shape=(1, 200, 2, 64))),
    (False, dict(shape=(1, 200, 2, 256))),
    (False, dict(shape=(1, 200, 1, 128))),                # one head for all of the cache's
    (False, dict(current=1)),
    (False, dict(clustered=0)),
    (False, dict(table=48)),
])
def test_rule_for_reading_the_prompt_in_place(monkeypatch, wanted, change):
    from retrievalattention_b200.cache_hub.retroinfer_cache import retroinfer_cache

    monkeypatch.setattr(torch.cuda, "current_device", lambda: change.get("current", 0))
    cache = SimpleNamespace(kv_head=2, head_dim=128, dtype=torch.bfloat16, n_centroids=32)
    plain = Rows((1, 200, 2, 128))
    other = Rows(change.get("shape", (1, 200, 2, 128)), **{k: v for k, v in change.items() if k in ("dtype", "device", "requires_grad")})
    centroids = Rows((2, change.get("table", 32), 128))
    with torch.set_grad_enabled(change.get("grad", True)):
        for keys, values in ((other, plain), (plain, other)):      # either tensor decides
            assert retroinfer_cache._prompt_form(cache, keys, values, centroids, change.get("clustered", 132)) is wanted


def test_prefill_attention_refuses_host_tensors():
    from retrievalattention_b200.attn_hub import retroinfer_prefill_attn

    x = torch.zeros((1, 8, 2, 128), dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="one GPU"):
        retroinfer_prefill_attn(x, x, x, True)
