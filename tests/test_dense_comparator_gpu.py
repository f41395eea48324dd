"""The dense comparator (``cache_hub.flash_attn_cache`` + ``attn_hub.decode_full_flash_attn``, the reference's full-attention
baseline, cache_hub/flash_attn_cache.py and attn_hub/flash_attn.py) against fp32 attention over every token, and the
wave-index path beside it on the same prompt — what the comparator is for."""
import pytest
import torch

from retrievalattention_b200.config import generate_config
from retrievalattention_b200.synthetic import make_kv, make_queries

pytestmark = pytest.mark.gpu


def test_dense_decode_matches_fp32_attention_beside_the_wave_index():
    from retrievalattention_b200.attn_hub import decode_full_flash_attn, retroinfer_decode_attn
    from retrievalattention_b200.cache_hub import flash_attn_cache, retroinfer_cache

    batch, layers, kv_heads, q_heads, seq_len, max_new = 2, 2, 2, 8, 2048 + 68, 6
    valid_start = [0, 37]
    mapping = {str(l): "cuda:0" for l in range(layers)}
    dense = flash_attn_cache(valid_start, layers, batch, seq_len + max_new, kv_heads, q_heads, 128, torch.bfloat16,
                             mapping, num_gpus=1, model_size=8)
    cfg = generate_config(seq_len, 0.05, 0.2, n_segments=2)
    wave = retroinfer_cache(valid_start, layers, batch, seq_len + max_new, kv_heads, q_heads, 128, torch.bfloat16,
                            mapping, max_new, num_gpus=1, model_size=8, **cfg.as_kwargs())
    prompts = {}
    for b in range(batch):
        for l in range(layers):
            k, v = make_kv(kv_heads, seq_len, 128, seed=100 * l + b, device="cuda")
            prompts[(l, b)] = (k, v)
            rk, _ = dense.prefill_update_kv_cache(None, k, v, l, b)
            assert rk.shape[1] == seq_len - valid_start[b]
            dense.sync(l, b)
            wave.prefill_update_kv_cache(None, k, v, l, b)
    wave.prepare_cache()
    assert dense.context == seq_len and dense.valid_length.tolist() == [seq_len, seq_len - 37]

    new_rows = {l: [] for l in range(layers)}
    for step in range(3):
        for l in range(layers):
            k_new = make_queries(batch, kv_heads, 128, seed=7000 + 10 * step + l, device="cuda")
            v_new = make_queries(batch, kv_heads, 128, seed=8000 + 10 * step + l, device="cuda")
            q = make_queries(batch, q_heads, 128, seed=9000 + 10 * step + l, device="cuda")
            new_rows[l].append((k_new, v_new))
            kc, vc = dense.decode_update_kv_cache(k_new, v_new, l)
            out = decode_full_flash_attn(q, kc, vc, l, dense)
            wave.decode_update_kv_cache(k_new, v_new, l)
            approx = retroinfer_decode_attn(q, k_new, v_new, l, wave)
            for b in range(batch):
                k, v = prompts[(l, b)]
                ks = torch.cat([k[0, valid_start[b]:]] + [r[0][b] for r in new_rows[l]]).float()      # [tokens, Hk, d]
                vs = torch.cat([v[0, valid_start[b]:]] + [r[1][b] for r in new_rows[l]]).float()
                qb = q[b, 0].float().view(kv_heads, q_heads // kv_heads, 128)
                s = torch.einsum("hgd,thd->hgt", qb, ks) / 128 ** 0.5
                ref = torch.einsum("hgt,thd->hgd", torch.softmax(s, -1), vs).reshape(q_heads, 128)
                err = (out[b, 0].float() - ref).abs()
                assert err.max() <= 2e-2 and err.mean() <= 2e-3, (step, l, b, float(err.max()))
                # the wave index approximates the same quantity (how closely depends on the prompt: these keys are
                # random, the worst case for clustering), so only its sanity is checked here
                assert torch.isfinite(approx[b, 0].float()).all()
    assert dense.context == seq_len + 3 and dense.valid_length.tolist() == [seq_len + 3, seq_len - 37 + 3]


@pytest.mark.parametrize("lengths,kv_heads,group,extra,dtype", [
    ((1,), 1, 1, 0, torch.bfloat16),                        # one row: one step, one warp
    ((0, 15, 16, 17), 2, 3, 0, torch.float16),              # a request without rows, edges of a 16-row step
    ((0, 0, 1), 1, 8, 0, torch.bfloat16),                   # requests without rows in front
    ((2047, 0, 130), 3, 5, 1, torch.float16),               # partial last steps, a CTA's range over several groups
    ((4095,), 1, 7, 1, torch.bfloat16),                     # one group over the whole chip
    ((37,) * 90, 8, 2, 1, torch.bfloat16),                  # more groups than warps
])
def test_dense_decode_kernel_equals_fp32_attention(lengths, kv_heads, group, extra, dtype):
    """Tolerances as above: probabilities and outputs are rounded to 16 bits (2^-8 relative for bf16)."""
    from types import SimpleNamespace

    from retrievalattention_b200.attn_hub import decode_full_flash_attn, flash_attn

    batch, room = len(lengths), max(lengths) + 3
    gen = torch.Generator(device="cuda").manual_seed(5)
    q = torch.randn((batch, 1, kv_heads * group, 128), generator=gen, device="cuda").to(dtype)
    k, v = (torch.randn((batch, kv_heads, room, 128), generator=gen, device="cuda").to(dtype) for _ in range(2))
    cache = SimpleNamespace(valid_length=torch.tensor(lengths, dtype=torch.int32, device="cuda"), layer_num=2)
    assert flash_attn._dense_form(q, k, v, cache.valid_length)
    out = decode_full_flash_attn(q, k, v, 1 - extra, cache)
    for b, n in enumerate(lengths):
        n += extra
        if n == 0:
            assert not out[b].any()
            continue
        s = torch.einsum("hgd,htd->hgt", q[b, 0].float().view(kv_heads, group, 128), k[b, :, :n].float()) / 128 ** 0.5
        ref = torch.einsum("hgt,htd->hgd", torch.softmax(s, -1), v[b, :, :n].float()).reshape(-1, 128)
        err = (out[b, 0].float() - ref).abs()
        assert err.max() <= 2e-2 and err.mean() <= 2e-3, (b, float(err.max()), float(err.mean()))
    # a view that is not dense takes the general operator: the same attention up to the order of the sums
    wide = torch.randn((batch, 1, kv_heads * group, 256), generator=gen, device="cuda").to(dtype)
    wide[..., :128] = q
    assert flash_attn._dense_form(wide[..., :128], k, v, cache.valid_length) == (kv_heads * group == 1)
    other = decode_full_flash_attn(wide[..., :128], k, v, 1 - extra, cache)
    assert (other.float() - out.float()).abs().max() <= 2e-2


@pytest.mark.parametrize("form", ["dense", "strided", "one_request", "full"])
def test_dense_append_forms(form):
    """Rows go where the indexing form puts them, whatever their strides; a full cache is refused."""
    from retrievalattention_b200.cache_hub import flash_attn_cache

    batch, hk, n = 3, 2, 40
    cache = flash_attn_cache([0, 7, 3], 2, batch, n + (0 if form == "full" else 2), hk, 8, 128, torch.bfloat16,
                             {"0": "cuda:0", "1": "cuda:0"}, 1, 8)
    gen = torch.Generator(device="cuda").manual_seed(6)
    for layer in range(2):
        for b in range(batch):
            k, v = (torch.randn((1, n, hk, 128), generator=gen, device="cuda").bfloat16() for _ in range(2))
            cache.prefill_update_kv_cache(None, k, v, layer, b)
    new = torch.randn((batch, 1, hk, 256), generator=gen, device="cuda").bfloat16()
    k, v = new[..., :128], new[..., 128:]
    if form == "dense":
        k, v = k.contiguous(), v.contiguous()
    if form == "one_request":
        k, v = k[:1], v[:1]
    wanted = form == "dense"
    assert cache._one_launch(cache.key_cache[0], k, v) == wanted
    if form == "full":                 # refused by the rule already: the indexing form is not run into its device check
        assert not cache._one_launch(cache.key_cache[0], k.contiguous(), v.contiguous())
        return
    before = [t.clone() for t in (cache.key_cache[0], cache.value_cache[0])]
    got = cache.decode_update_kv_cache(k, v, 0)
    for old, now, rows in zip(before, got, (k, v)):
        for b, start in enumerate((0, 7, 3)):
            old[b, :, n - start] = rows[b if rows.shape[0] > 1 else 0, 0]
        assert torch.equal(old, now)


def test_rows_behind_the_end_of_the_cache_are_reported():
    """Where the lengths move on without the host, in replays of a captured step, a row that no longer fits is left out and
    said to be."""
    from retrievalattention_b200.attn_hub import decode_full_flash_attn, retroinfer_attn as ra
    from retrievalattention_b200.cache_hub import flash_attn_cache

    n, hk = 40, 2
    cache = flash_attn_cache([0, 1], 1, 2, n + 2, hk, 8, 128, torch.bfloat16, {"0": "cuda:0"}, 1, 8)
    gen = torch.Generator(device="cuda").manual_seed(6)
    mk = lambda b, s, h: torch.randn((b, s, h, 128), generator=gen, device="cuda").bfloat16()      # noqa: E731
    for b in range(2):
        cache.prefill_update_kv_cache(None, mk(1, n, hk), mk(1, n, hk), 0, b)
    k, v, q = mk(2, 1, hk), mk(2, 1, hk), mk(2, 1, 8)
    assert cache._one_launch(cache.key_cache[0], k, v)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = decode_full_flash_attn(q, *cache.decode_update_kv_cache(k, v, 0), 0, cache)
    for step in range(2):
        graph.replay()
        ra.check_prefill_errors()
        assert cache.valid_length.tolist() == [n + step + 1, n + step] and torch.isfinite(out.float()).all()
    assert torch.equal(cache.key_cache[0][0, :, n + 1], k[0, 0]) and torch.equal(cache.value_cache[0][1, :, n], v[1, 0])
    before = [t.clone() for t in (cache.key_cache[0], cache.value_cache[0])]
    graph.replay()                                  # the first request is full, the second has room for one more row
    with pytest.raises(RuntimeError, match="did not fit"):
        ra.check_prefill_errors()
    ra.check_prefill_errors()
    for old, now, rows in zip(before, (cache.key_cache[0], cache.value_cache[0]), (k, v)):
        old[1, :, n + 1] = rows[1, 0]
        assert torch.equal(old, now)


@pytest.mark.parametrize("form", ["longer", "strided", "other_type"])
def test_dense_append_into_tensors_put_in_place_of_the_cache(form):
    from retrievalattention_b200.cache_hub import flash_attn_cache

    n, hk = 40, 2
    cache = flash_attn_cache([0, 7], 2, 2, n + 2, hk, 8, 128, torch.bfloat16, {"0": "cuda:0", "1": "cuda:0"}, 1, 8)
    gen = torch.Generator(device="cuda").manual_seed(6)
    mk = lambda s: torch.randn((2, s, hk, 128), generator=gen, device="cuda").bfloat16()      # noqa: E731
    for b in range(2):
        cache.prefill_update_kv_cache(None, mk(n)[:1], mk(n)[:1], 0, b)
    for tensors in (cache.key_cache, cache.value_cache):
        old = tensors[0]
        if form == "longer":
            tensors[0] = torch.cat((old, torch.zeros_like(old)), dim=2)
        elif form == "strided":
            tensors[0] = torch.cat((old, old), dim=3)[..., :128]
    if form == "other_type":
        cache.value_cache[0] = cache.value_cache[0].half()
    k, v = mk(1), mk(1)
    v = v.to(cache.value_cache[0].dtype)
    assert not cache._one_launch(cache.key_cache[0], k, v, cache.value_cache[0])
    before = [cache.key_cache[0].clone(), cache.value_cache[0].clone()]
    got = cache.decode_update_kv_cache(k, v, 0)
    for old, now, rows in zip(before, got, (k, v)):
        for b, start in enumerate((0, 7)):
            old[b, :, n - start] = rows[b, 0]
        assert torch.equal(old, now)


def test_rows_written_by_kernels_count_as_changes_in_place():
    """A backward pass that saved a cache tensor must not run on rows written since (autograd compares versions)."""
    from retrievalattention_b200.cache_hub import flash_attn_cache, retroinfer_cache

    n, hk = 1024 + 68, 2
    dense = flash_attn_cache([0], 2, 1, n + 2, hk, 8, 128, torch.bfloat16, {"0": "cuda:0", "1": "cuda:0"}, 1, 8)
    cfg = generate_config(n, 0.05, 0.2, n_segments=1)
    wave = retroinfer_cache([0], 1, 1, n + 6, hk, 8, 128, torch.bfloat16, {"0": "cuda:0"}, 6, num_gpus=1, model_size=8,
                            **cfg.as_kwargs())
    k, v = make_kv(hk, n, 128, seed=3, device="cuda")
    dense.prefill_update_kv_cache(None, k, v, 0, 0)
    wave_tensors = [getattr(wave, name)[0] for name in ("centroids", "value_sum", "cluster_size", "cluster_count", "cluster_offset",
                                                        "centroids_mask", "list_keys", "list_values", "steady_zone_keys",
                                                        "steady_zone_values")]
    before = [t._version for t in wave_tensors]
    wave.prefill_update_kv_cache(None, k, v, 0, 0)
    assert all(t._version > old for t, old in zip(wave_tensors, before))
    weight = torch.ones(128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    loss = (dense.key_cache[0] * weight).sum()
    row = k[:, :1].contiguous()
    assert dense._one_launch(dense.key_cache[0], row, row, dense.value_cache[0])
    dense.decode_update_kv_cache(row, row, 0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        loss.backward()
    with torch.inference_mode():                    # tensors made there keep no version
        other = flash_attn_cache([0], 2, 1, n + 2, hk, 8, 128, torch.bfloat16, {"0": "cuda:0", "1": "cuda:0"}, 1, 8)
        other.prefill_update_kv_cache(None, k, v, 0, 0)
        other.decode_update_kv_cache(row, row, 0)
        assert torch.equal(other.key_cache[0][0, :, n], row[0, 0])
