"""Dense prefill attention (``ri_prefill_attn`` behind ``retroinfer_prefill_attn``, the replacement of the reference's
flash-attn call, attn_hub/retroinfer_attn.py:4-13) against fp32 PyTorch attention.

Tolerance (bf16 probabilities and outputs, fp32 accumulation): max-abs <= 2e-2, mean-abs <= 2e-3."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(q, k, v, causal):
    b, s, hq, d = q.shape
    hk = k.shape[2]
    qf = q.float().permute(0, 2, 1, 3)                                   # [B, Hq, S, d]
    kf = k.float().permute(0, 2, 1, 3).repeat_interleave(hq // hk, dim=1)
    vf = v.float().permute(0, 2, 1, 3).repeat_interleave(hq // hk, dim=1)
    out = torch.nn.functional.scaled_dot_product_attention(qf, kf, vf, is_causal=bool(causal))
    return out.permute(0, 2, 1, 3)


@pytest.mark.parametrize("batch,seq,hq,hk,causal,dtype", [
    (1, 1024, 4, 1, True, torch.bfloat16),
    (2, 1000, 8, 2, True, torch.bfloat16),       # ragged: last tile partly empty, rows of the next request behind it
    (1, 128, 2, 2, True, torch.bfloat16),        # a single tile
    (1, 77, 4, 4, True, torch.float16),          # shorter than one tile
    (2, 640, 4, 2, False, torch.bfloat16),       # not causal
    (1, 4096, 8, 2, True, torch.bfloat16),
    (1, 16384, 2, 1, True, torch.bfloat16),
])
def test_prefill_attention_matches_fp32(batch, seq, hq, hk, causal, dtype):
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    g = torch.Generator(device="cuda").manual_seed(seq + hq)
    mk = lambda h, scale: (torch.randn((batch, seq, h, 128), generator=g, device="cuda") * scale).to(dtype)   # noqa: E731
    q, k, v = mk(hq, 1.5), mk(hk, 1.5), mk(hk, 1.0)
    out = ra.retroinfer_prefill_attn(q, k, v, causal)
    ra.check_prefill_errors()
    ref = reference(q, k, v, causal)
    err = (out.float() - ref).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))


def test_large_scores_move_the_reference_maximum():
    """Scores that keep growing along the sequence force the lazy reference maximum to move (the accumulator is
    rescaled in tensor memory) many times."""
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    torch.manual_seed(3)
    seq = 1536
    q = torch.randn((1, seq, 2, 128), device="cuda")
    k = torch.randn((1, seq, 1, 128), device="cuda")
    ramp = torch.linspace(0.2, 6.0, seq, device="cuda")[None, :, None, None]
    k = (k * 0.3 + q[:, :, :1] * 0.05 * ramp)             # later keys score higher against every query
    q, k = q.to(torch.bfloat16), k.to(torch.bfloat16)
    v = torch.randn((1, seq, 1, 128), device="cuda").to(torch.bfloat16)
    out = ra.retroinfer_prefill_attn(q, k, v, True)
    ra.check_prefill_errors()
    err = (out.float() - reference(q, k, v, True)).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))


def test_bad_arguments_are_rejected():
    from retrievalattention_b200 import _lib

    assert _lib.lib.ri_prefill_attn(None, None, None, None, None, None, 1, 128, 4, 1, 1, 0, None) == -1
    assert _lib.lib.ri_prefill_attn_scratch_bytes(1, 0, 1) == -1
    assert _lib.lib.ri_prefill_attn_scratch_bytes(2, 1000, 2) == 2 * 2 * 128 * 1024 * 2


# two query tiles per CTA or one with its key/value tiles split over two groups (fewer pairs of query tiles than SMs), an
# odd number of tiles, more items than SMs (persistent CTAs), rows of the next request behind a request's last tile.
# Same tolerance as above; NaN in a neighbouring request must not leak in.
@pytest.mark.parametrize("batch,seq,hq,hk,causal", [
    (1, 129, 2, 1, True), (1, 257, 1, 1, False), (3, 385, 5, 1, True), (2, 1200, 40, 8, True), (2, 1300, 28, 4, False),
    (1, 2500, 24, 8, True),
])
def test_query_tile_pairs_and_split_walks(batch, seq, hq, hk, causal):
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    g = torch.Generator(device="cuda").manual_seed(seq)
    mk = lambda h: torch.randn((batch, seq, h, 128), generator=g, device="cuda").to(torch.bfloat16)   # noqa: E731
    q, k, v = mk(hq), mk(hk), mk(hk)
    if batch > 1:
        k[1:], v[1:] = float("nan"), float("nan")
    out = ra.retroinfer_prefill_attn(q, k, v, causal)[:1]
    ra.check_prefill_errors()
    err = (out.float() - reference(q[:1], k[:1], v[:1], causal)).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))


def two_walks(scores, v, tiles, dtype):
    """Attention of rows of scores (log2 domain, fp32, masked) as two walks over the even and the odd tiles of 128 keys give
    it, each with its own reference maximum that follows in steps of more than 2^8, probabilities rounded to `dtype`."""
    parts = []
    for first in (0, 1):
        m = torch.full(scores.shape[:1], -torch.inf, device=scores.device)
        total, acc = torch.zeros_like(m), torch.zeros((scores.shape[0], 128), device=scores.device)
        for t in range(first, tiles, 2):
            s = scores[:, t * 128:(t + 1) * 128]
            top = s.max(1).values
            new = torch.where(top > m + 8, top, m)
            ref = new.nan_to_num(neginf=0.0)
            factor, p = torch.exp2(m - ref), torch.exp2(s - ref[:, None])
            total = total * factor + p.sum(1)
            acc = acc * factor[:, None] + p.to(dtype).float() @ v[t * 128:(t + 1) * 128].float()
            m = new
        parts.append((m, total, acc))
    top = torch.maximum(parts[0][0], parts[1][0])
    weight = [torch.exp2(m - top) for m, _, _ in parts]
    return sum(w[:, None] * a for w, (_, _, a) in zip(weight, parts)) / sum(w * t for w, (_, t, _) in zip(weight, parts))[:, None]


@pytest.mark.parametrize("seq,hq,hk,dtype", [(2500, 32, 8, torch.bfloat16), (5001, 28, 4, torch.float16), (8192, 8, 8, torch.bfloat16)])
def test_pairs_are_as_accurate_as_two_walks(seq, hq, hk, dtype):
    """Where two query tiles share the keys there is one walk per row.  Its distance from 64-bit attention must not exceed
    that of the same rows in two walks (computed here); the keys are clustered, so some scores stand out."""
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra
    from retrievalattention_b200.synthetic import make_kv

    assert takes_pairs(1, seq, hq)
    q = torch.randn((1, seq, hq, 128), generator=torch.Generator(device="cuda").manual_seed(17), device="cuda").to(dtype)
    k, v = make_kv(hk, seq, 128, seed=93, device="cuda", dtype=dtype)
    out = ra.retroinfer_prefill_attn(q, k, v, True)
    ra.check_prefill_errors()
    rows = torch.randperm(seq, generator=torch.Generator().manual_seed(1))[:1024].cuda()
    mine = theirs = 0.0
    torch.backends.cuda.matmul.allow_tf32 = False
    for h in range(0, hq, hq // 8):
        keys, vals = k[0, :, h // (hq // hk)], v[0, :, h // (hq // hk)]
        s = q[0, rows, h].double() @ keys.double().T * (1.4426950408889634 / 128 ** 0.5)
        s = s.masked_fill(torch.arange(seq, device="cuda")[None] > rows[:, None], -torch.inf)
        exact = torch.softmax(s * 0.6931471805599453, -1) @ vals.double()
        mine += float((out[0, rows, h].double() - exact).pow(2).sum())
        theirs += float((two_walks(s.float(), vals, -(-seq // 128), dtype).to(dtype).double() - exact).pow(2).sum())
    assert mine <= theirs, ((mine / theirs) ** 0.5)


@pytest.mark.parametrize("seq,hq", [(300, 2), (1300, 32)])       # one query tile per CTA, and pairs
def test_a_recorded_failure_is_reported_once_and_stops_no_later_call(seq, hq):
    import ctypes as C

    from retrievalattention_b200 import _lib
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    g = torch.Generator(device="cuda").manual_seed(seq)
    q, k, v = (torch.randn((1, seq, h, 128), generator=g, device="cuda").to(torch.bfloat16) for h in (hq, 2, 2))
    good = ra.retroinfer_prefill_attn(q, k, v, True)
    ra.check_prefill_errors()
    status = ra._status_word(q.device)
    out = torch.zeros_like(q)
    status.value = 31                                     # as a kernel of an earlier call would have left it
    _lib.check(_lib.lib.ri_prefill_attn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None, C.addressof(status), 1, seq,
                                        hq, 2, 1, _lib.dtype_code(q.dtype), _lib.current_stream()))
    torch.cuda.synchronize()
    assert status.value == 31 and torch.equal(good, out)
    with pytest.raises(RuntimeError, match="31"):         # the first call that finds it says so
        ra.retroinfer_prefill_attn(q, k, v, True)
    assert torch.equal(good, ra.retroinfer_prefill_attn(q, k, v, True))
    ra.check_prefill_errors()


def test_status_of_captured_calls():
    """The word is clear before a captured call's first replay, and failures of any replay are reported, also behind an
    earlier check."""
    from types import SimpleNamespace

    from retrievalattention_b200.attn_hub import decode_full_flash_attn, retroinfer_attn as ra

    g = torch.Generator(device="cuda").manual_seed(9)
    q, k, v = (torch.randn((1, 300, h, 128), generator=g, device="cuda").to(torch.bfloat16) for h in (4, 2, 2))
    kc, vc = (x.transpose(1, 2).contiguous() for x in (k, v))
    cache = SimpleNamespace(valid_length=torch.tensor([290], dtype=torch.int32, device="cuda"), layer_num=1)
    calls = (lambda: ra.retroinfer_prefill_attn(q, k, v, True), lambda: decode_full_flash_attn(q[:, :1], kc, vc, 0, cache))
    want = [f() for f in calls]
    ra.check_prefill_errors()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [f() for f in calls]
    ra.check_prefill_errors()
    for _ in range(2):
        for x in got:
            x.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
        ra.check_prefill_errors()
        ra._status_word(q.device).value = 24
        with pytest.raises(RuntimeError, match="24"):
            ra.check_prefill_errors()


def test_first_call_of_a_process_may_be_captured():
    """Its status word is made under the capture."""
    import subprocess
    import sys

    code = """
import torch
from retrievalattention_b200.attn_hub import retroinfer_attn as ra
q, k = (torch.randn((1, 300, h, 128), device="cuda").bfloat16() for h in (4, 2))
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = ra.retroinfer_prefill_attn(q, k, k, True)
ra.check_prefill_errors()
graph.replay()
ra.check_prefill_errors()
assert torch.equal(out, ra.retroinfer_prefill_attn(q, k, k, True))
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)


def takes_pairs(batch, seq, hq):
    """Whether a call has a pair of query tiles for every SM, so that CTAs take pairs (else single tiles, split walks)."""
    tiles = -(-seq // 128)
    return (tiles + 1) // 2 * hq * batch >= torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("batch,seq,hq,hk,causal,dtype,grows", [
    (1, 1300, 32, 8, True, torch.float16, False),
    (3, 900, 28, 4, True, torch.bfloat16, False),       # NaN in the middle request, both neighbours compared
    (3, 901, 28, 4, False, torch.float16, False),
    (1, 1536, 32, 1, True, torch.bfloat16, True),       # scores grow along the sequence: accumulators are rescaled
    (1, 1600, 28, 1, True, torch.float16, True),
    (1, 8192, 8, 8, True, torch.bfloat16, False),       # a walk of 64 key tiles
])
def test_pairs_of_query_tiles(batch, seq, hq, hk, causal, dtype, grows):
    """Same tolerance as above."""
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    assert takes_pairs(batch, seq, hq)
    g = torch.Generator(device="cuda").manual_seed(seq)
    q, k, v = (torch.randn((batch, seq, h, 128), generator=g, device="cuda") for h in (hq, hk, hk))
    if grows:
        ramp = torch.linspace(0.2, 6.0, seq, device="cuda")[None, :, None, None]
        k = k * 0.3 + q[:, :, :hk] * 0.05 * ramp
    q, k, v = q.to(dtype), k.to(dtype), v.to(dtype)
    if batch > 2:
        k[1], v[1] = float("nan"), float("nan")
    out = ra.retroinfer_prefill_attn(q, k, v, causal)
    ra.check_prefill_errors()
    for b in range(0, batch, 2):
        err = (out[b:b + 1].float() - reference(q[b:b + 1], k[b:b + 1], v[b:b + 1], causal)).abs()
        assert err.max() <= 2e-2 and err.mean() <= 2e-3, (b, float(err.max()), float(err.mean()))
