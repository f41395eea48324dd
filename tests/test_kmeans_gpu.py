"""Parity of the CUDA clustering (tcgen05 assignment GEMM + bucket + update + layout, through the
C ABI) against (a) the fixtures recorded from the reference's own kmeans.py and (b) the CPU oracle.

Bar (cluster assignments bit-exact except ties):

* one or two Lloyd iterations — both sides start from the same centroids — EVERY assignment that differs
  must be a tie: the two clusters' inner products with the token, evaluated on the oracle's centroids of
  the last assignment pass, differ by no more than the noise a tie can hide (fp32 accumulation order
  with identical centroids: 1e-5 of |x||c|; one 16-bit rounding step of a centroid after an update:
  2 ulp of |x||c|);
* more iterations: a flipped tie moves a centroid by a rounding step and the runs drift apart from
  there, which no tie rule at the end can excuse; the stated bound is <= 1 % of the assignments and
  >= 97 % of the cluster sizes equal, with centroids and value sums within one ulp of the 16-bit
  dtype wherever the sizes agree."""
import os
import sys

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))

import make_golden as mg  # noqa: E402
from oracle import kmeans as okm  # noqa: E402
from retrievalattention_b200.synthetic import make_kv  # noqa: E402

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(HERE, "golden")
DRIFT_ASSIGN, DRIFT_SIZES = 0.01, 0.97


def last_pass_centroids(centred, cents, iters, segs):
    """The oracle's centroids that the LAST assignment pass of ``segment_k_means`` compares against
    (cache_hub/kmeans.py:232-248): the evenly spaced initial rows, moved by iters - 1 segmented passes."""
    groups, n, d = centred.shape
    cen = torch.index_select(centred, 1, okm.initial_centroid_indices(n, cents))
    n_seg, c_seg = n // segs, cents // segs
    data = centred[:, :n_seg * segs].reshape(-1, n_seg, d)
    cen = cen.reshape(-1, c_seg, d)
    for _ in range(iters - 1):
        cen, _, _ = okm.train_step(data, cen, normalize=True)
    return cen.reshape(groups, cents, d)


def tie_margin(data, centroids, a, b):
    """|x.c_a - x.c_b| relative to |x| times the mean norm of the two centroids."""
    ip = torch.bmm(data.float(), centroids.float().transpose(1, 2))
    sa = torch.gather(ip, 2, a.long()[..., None])[..., 0]
    sb = torch.gather(ip, 2, b.long()[..., None])[..., 0]
    cn = centroids.float().norm(dim=-1)
    scale = data.float().norm(dim=-1) * 0.5 * (torch.gather(cn, 1, a.long()) + torch.gather(cn, 1, b.long()))
    return (sa - sb).abs() / scale.clamp_min(1e-20)


def check_assignments(got, want, centred, cents, iters, segs):
    """The parity bar of the module docstring.  Returns the mask of differing assignments."""
    diff = got != want
    if iters <= 2:
        if diff.any():
            ulp = 2.0 ** -10 if centred.dtype == torch.float16 else 2.0 ** -7
            tol = 1e-5 if iters == 1 else 2 * ulp
            margin = tie_margin(centred, last_pass_centroids(centred, cents, iters, segs), got, want)[diff]
            assert (margin <= tol).all(), f"{int((margin > tol).sum())} of {int(diff.sum())} differing assignments are no ties (worst {float(margin.max()):.3g})"
    else:
        assert diff.float().mean() <= DRIFT_ASSIGN, f"{int(diff.sum())} of {diff.numel()} assignments differ"
    return diff


@pytest.mark.parametrize("name", sorted(mg.KMEANS_CASES))
def test_segment_k_means_against_reference_fixture(name):
    from retrievalattention_b200.cache_hub import kmeans as gk

    heads, tokens, cents, segs, iters, seed, planted = mg.KMEANS_CASES[name]
    gold = torch.load(os.path.join(GOLDEN, name + ".pt"))
    k, v, centred = mg.kmeans_inputs(heads, tokens, seed, planted)
    assert mg.sha(centred) == gold["input_sha"]["centred"]
    cen, vsum, clusters, sizes = gk.segment_k_means(centred.cuda(), v.cuda(), cents, num_iters=iters, num_segments=segs)
    torch.cuda.synchronize()
    cen, vsum, clusters, sizes = cen.cpu(), vsum.cpu(), clusters.cpu(), sizes.cpu()
    assign = torch.full((heads, tokens), -1, dtype=torch.int32)
    for h in range(heads):
        for c in range(cents):
            m = int(sizes[h, c])
            members = clusters[h, c, :m]
            assert (members[1:] > members[:-1]).all(), "members must be in ascending token order"
            assign[h, members.long()] = c
    assert (assign >= 0).all() and int(sizes.sum()) == heads * tokens
    want = gold["assignments"].to(torch.int32)
    check_assignments(assign, want, centred, cents, iters, segs)
    same = (sizes == gold["sizes"])
    assert same.float().mean() >= DRIFT_SIZES
    torch.testing.assert_close(cen.float()[same], gold["centroids"].float()[same], rtol=2 ** -9, atol=2e-3)
    torch.testing.assert_close(vsum.float()[same], gold["value_sum"].float()[same], rtol=2 ** -9, atol=2e-2)


BF16_CASES = {
    # heads, tokens, centroids, segments, iters, seed
    "one_tile": (2, 100, 32, 1, 3, 1),
    "ragged_tiles": (3, 1000, 96, 3, 4, 2),
    "many_tiles": (2, 5000, 512, 4, 5, 3),
    "wide": (1, 3000, 1024, 2, 3, 4),
    "one_iteration": (2, 4000, 256, 4, 1, 5),
    "two_iterations": (2, 4000, 256, 4, 2, 6),
    "two_iterations_wide": (1, 6000, 1024, 2, 2, 7),
    # centroid tiles of the resident-centroid kernel: three tiles (two rounds, the second with one tile), a partial
    # second tile, a partial third tile, token counts that are no multiple of 128
    "three_tiles": (2, 3000, 384, 1, 2, 8),
    "partial_second_tile": (2, 2600, 224, 1, 2, 9),
    "partial_third_tile": (1, 2053, 352, 1, 1, 10),
    # configuration 0 of the benchmark: 8 kv heads x (8192 - 68) clustered keys, 512 centroids, 10 iterations
    "cfg0_geometry": (8, 8192 - 68, 512, 1, 10, 0),
}


@pytest.mark.parametrize("name", sorted(BF16_CASES))
def test_build_index_against_oracle_bf16(name):
    from retrievalattention_b200.cache_hub import kmeans as gk

    heads, tokens, cents, segs, iters, seed = BF16_CASES[name]
    k, v = make_kv(heads, tokens, 128, seed=seed)
    k = k[0].transpose(0, 1).contiguous()
    v = v[0].transpose(0, 1).contiguous()
    r = gk.build_index(k.cuda(), v.cuda(), cents, segs, iters, want_lists=True)
    torch.cuda.synchronize()
    r = {n: t.cpu() for n, t in r.items() if not n.startswith("_")}
    assert int(r["error"]) == 0

    # mean key: fp32 sum in another order, so allow one bf16 step; then centre exactly as the kernel did
    ref_mean = torch.mean(k, dim=1, keepdim=True)
    torch.testing.assert_close(r["mean_key"].float(), ref_mean.float(), rtol=2 ** -7, atol=1e-3)
    centred = k - r["mean_key"]
    cen, vsum, clusters, sizes, assign = okm.segment_k_means(centred, v, cents, iters, segs, return_assignments=True)

    diff = check_assignments(r["assign"], assign, centred, cents, iters, segs)

    # structure: counts/offsets/order describe r["assign"] exactly, members ascending
    for h in range(heads):
        cnt = torch.bincount(r["assign"][h].long(), minlength=cents)
        assert torch.equal(cnt.to(torch.int32), r["cluster_count"][h])
        off = r["cluster_offset"][h].long()
        assert off[0] == 0 and off[-1] == tokens and torch.equal(off[1:] - off[:-1], cnt)
        order = r["order"][h].long()
        assert torch.equal(torch.sort(order).values, torch.arange(tokens))
        assert torch.equal(r["assign"][h].long()[order], torch.repeat_interleave(torch.arange(cents), cnt))
        same_cluster = r["assign"][h].long()[order][1:] == r["assign"][h].long()[order][:-1]
        assert (order[1:][same_cluster] > order[:-1][same_cluster]).all()
        # layout: rows copied bit-for-bit in member order
        assert torch.equal(r["keys"][h].view(torch.int16), k[h][order].view(torch.int16))
        assert torch.equal(r["values"][h].view(torch.int16), v[h][order].view(torch.int16))
    assert torch.equal(r["cluster_size"].view(torch.int16), r["cluster_count"].to(torch.bfloat16).view(torch.int16))

    same = sizes == r["cluster_count"]
    assert same.float().mean() >= DRIFT_SIZES
    want_cent = cen + r["mean_key"]
    torch.testing.assert_close(r["centroids"].float()[same], want_cent.float()[same], rtol=2 ** -6, atol=2e-2)
    torch.testing.assert_close(r["value_sum"].float()[same], vsum.float()[same], rtol=2 ** -6, atol=6e-2)
    if not diff.any():
        # identical member sets and a serial sum in the same order: value sums agree to the bit
        assert torch.equal(r["value_sum"].view(torch.int16), vsum.view(torch.int16))


def test_empty_clusters_keep_centroid_and_zero_value_sum():
    from retrievalattention_b200.cache_hub import kmeans as gk

    heads, tokens, cents = 2, 700, 64
    k, v = make_kv(heads, tokens, 128, seed=9)
    k = k[0].transpose(0, 1)[:, torch.arange(tokens) % 37].contiguous()
    v = v[0].transpose(0, 1).contiguous()
    r = gk.build_index(k.cuda(), v.cuda(), cents, 1, 5, want_lists=True)
    torch.cuda.synchronize()
    cnt = r["cluster_count"].cpu()
    assert int((cnt == 0).sum()) > 0
    assert (r["value_sum"].cpu()[cnt == 0] == 0).all()
    assert torch.isfinite(r["centroids"].float()).all()


def test_rejects_bad_shapes():
    import ctypes as C
    from retrievalattention_b200 import _lib

    p = _lib.KMeans()
    p.groups, p.n_tokens, p.n_centroids, p.n_segments, p.n_iters = 1, 100, 48, 1, 3
    assert _lib.lib.ri_kmeans_scratch_bytes(C.byref(p)) == -1
    assert b"multiple of 32" in _lib.lib.ri_last_error()


# sizes where the sort, the update and the assignment change form: one problem per 8, 4, 2, 1 CTAs of the sort, more tokens
# than its 16-bit counts take and more clusters than its tables hold (the one-CTA form), one partial centroid tile, 512 centroids (resident) and 544 (streamed),
# a prompt whose clustered rows are no multiple of anything.  Everything below is exact: the list is a stable sort of the
# assignment, and the prompt form is the array form on the same rows.
@pytest.mark.parametrize("heads,n,c,seg,dtype", [
    (1, 333, 32, 1, torch.bfloat16), (3, 5003, 512, 1, torch.bfloat16), (2, 9001, 544, 1, torch.float16),
    (8, 16411, 1024, 16, torch.bfloat16), (8, 20000, 1024, 8, torch.bfloat16), (5, 20011, 1280, 40, torch.float16),
    (1, 500009, 96, 1, torch.bfloat16), (1, 41051, 20512, 1, torch.bfloat16),
])
def test_lists_and_prompt_form(heads, n, c, seg, dtype):
    from retrievalattention_b200.cache_hub.kmeans import build_index, build_prompt_index

    sink, recent, z = 4, 64, heads
    g = torch.Generator(device="cuda").manual_seed(n)
    k, v = (torch.randn((sink + n + recent, z, 128), generator=g, device="cuda").to(dtype) for _ in range(2))
    mid_k, mid_v = (t[sink:sink + n].transpose(0, 1).contiguous() for t in (k, v))
    r = build_index(mid_k, mid_v, c, seg, 3, want_lists=True)
    assert int(r["error"]) == 0
    count = torch.stack([torch.bincount(a, minlength=c) for a in r["assign"].long()])
    assert torch.equal(r["cluster_count"].long(), count)
    assert torch.equal(r["cluster_offset"][:, 1:].long(), count.cumsum(1)) and int(r["cluster_offset"][:, 0].abs().max()) == 0
    assert torch.equal(r["order"].long(), torch.sort(r["assign"].long(), dim=1, stable=True)[1])
    pick = r["order"].long()[:, :, None].expand(-1, -1, 128)
    assert torch.equal(r["keys"], torch.gather(mid_k, 1, pick)) and torch.equal(r["values"], torch.gather(mid_v, 1, pick))
    owner = torch.gather(r["assign"].long(), 1, r["order"].long())[:, :, None].expand(-1, -1, 128)
    total = torch.zeros((z, c, 128), dtype=torch.float64, device="cuda").scatter_add_(1, owner, r["values"].double())
    bound = torch.zeros_like(total).scatter_add_(1, owner, r["values"].double().abs())
    # one rounding to 16 bits of a serial fp32 sum: half an ulp of the result plus n_c * 2^-24 of the summed magnitudes
    ulp = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert bool(((r["value_sum"].double() - total).abs() <= ulp * total.abs() + count.max() * 2.0 ** -24 * bound + 1e-12).all())
    mk = lambda *s, dt=dtype: torch.full(s, 7, dtype=dt, device="cuda")        # noqa: E731
    rows, steady = n + 9, sink + recent + 5
    out = dict(centroids=mk(z, c, 128), value_sum=mk(z, c, 128), cluster_size=mk(z, c), cluster_count=mk(z, c, dt=torch.int32),
               cluster_offset=mk(z, c + 1, dt=torch.int32), empty=torch.zeros((z, c), dtype=torch.bool, device="cuda"),
               keys=mk(z, rows, 128), values=mk(z, rows, 128), steady_keys=mk(z, steady, 128), steady_values=mk(z, steady, 128))
    assert int(build_prompt_index(k, v, seg, sink, recent, out, 3)) == 0
    for name in ("centroids", "value_sum", "cluster_size", "cluster_count", "cluster_offset"):
        assert torch.equal(out[name], r[name]), name
    assert torch.equal(out["empty"], r["cluster_count"] == 0)
    for name, raw in (("keys", k), ("values", v)):
        assert torch.equal(out[name][:, :n], r[name]) and bool((out[name][:, n:] == 7).all())
        ends = torch.cat((raw[:sink], raw[sink + n:]), 0).transpose(0, 1)
        assert torch.equal(out["steady_" + name][:, :sink + recent], ends) and bool((out["steady_" + name][:, sink + recent:] == 7).all())


def test_infinite_scores_keep_every_token():
    """fp16 keys whose centred form overflows give scores of +inf and -inf beside one another: every token still lands in
    exactly one cluster."""
    from retrievalattention_b200.cache_hub.kmeans import build_index

    n = 1024
    keys = torch.randn((1, n, 128), generator=torch.Generator().manual_seed(3)).half()
    keys[0, ::2, 0], keys[0, 1::2, 0] = -60000.0, -20000.0
    keys[0, 7::256, 0] = 65504.0
    values = torch.zeros_like(keys)
    values[0, :, 0], values[0, :, 1] = torch.arange(n) % 32, torch.arange(n) // 32
    for n_cen in (64, 1024):         # centroids resident in shared memory, and streamed
        r = build_index(keys.cuda(), values.cuda(), n_cen, 1)
        torch.cuda.synchronize()
        assert int(r["error"].item()) == 0 and int(r["cluster_count"].sum()) == n
        got = r["values"][0].float().cpu()
        assert (got[:, 0] + 32 * got[:, 1]).sort().values.tolist() == list(range(n))


# members of the long cluster: around the size from which a whole CTA sums it, a batch of rows more, and several rounds of batches
# with a remainder
@pytest.mark.parametrize("per_seg,segs,cents,dtype", [(511, 1, 32, torch.bfloat16), (512, 2, 64, torch.float16), (545, 1, 32, torch.bfloat16),
                                                       (701, 3, 96, torch.bfloat16), (2117, 2, 128, torch.float16), (6000, 1, 512, torch.bfloat16)])
def test_cluster_that_holds_a_whole_segment(per_seg, segs, cents, dtype):
    """The first initial centroid of every segment is a long key that wins all its tokens: after one update of that cluster (the
    others keep their rows) the assignments are the oracle's except for ties."""
    from retrievalattention_b200.cache_hub import kmeans as gk

    heads, n = 2, per_seg * segs
    gen = torch.Generator().manual_seed(per_seg)
    u = torch.randn((heads, 1, 128), generator=gen)
    k = (u + torch.randn((heads, n, 128), generator=gen)).to(dtype)
    start = okm.initial_centroid_indices(n, cents)
    k[:, start[::cents // segs]] = (u * 20).to(dtype)
    v = torch.randn((heads, n, 128), generator=gen).to(dtype)
    data = k.reshape(-1, per_seg, 128)
    cen = torch.index_select(k, 1, start).reshape(-1, cents // segs, 128)
    assert (okm.assign(data, cen) == 0).all()                    # the case is what it says
    want = okm.segment_k_means(k, v, cents, 2, segs, return_assignments=True)[4]
    got = gk._run(k.cuda(), v.cuda(), cents, 2, segs, False, False)
    assert int(got["error"]) == 0
    check_assignments(got["assign"].cpu(), want.to(torch.int32), k, cents, 2, segs)
