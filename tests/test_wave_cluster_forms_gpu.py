"""The forms of the single decode kernel over its cluster sizes, against the oracle: id outputs (which rank the candidates), a page
budget that cuts them, the global and the mixed lists, and new rows that the kernel appends."""
import pytest
import torch

from helpers import RECENT, SINK
from oracle import attention as oat
from oracle import score_select as oss
from test_wave_cluster_sizes_gpu import make_layer

pytestmark = pytest.mark.gpu

# groups, group size, centroids, retrieved, estimated, type; the CTAs per group are those of a GPU with 148 SMs
SIZES = {
    "16_ctas": (1, 8, 2568, 40, 500, torch.bfloat16),
    "16_ctas_4_keys": (7, 3, 12296, 200, 2900, torch.float16),
    "16_ctas_full_slices": (1, 8, 16384, 294, 3801, torch.bfloat16),
    "10_ctas_8_keys": (9, 8, 16384, 1024, 2000, torch.bfloat16),
    "7_ctas": (4, 2, 760, 13, 0, torch.bfloat16),
    "2_ctas": (60, 2, 200, 3, 40, torch.bfloat16),
    "1_cta": (100, 4, 136, 2, 30, torch.float16),
    "5_ctas_16_keys": (23, 1, 12296, 220, 2800, torch.bfloat16),
    "4_ctas_16_keys": (34, 2, 16384, 294, 3801, torch.float16),
}
LEN = SINK + RECENT + 1


def attend(q, t, ret, kept, est):
    """Attention over the given clusters: [groups, gs, 128]."""
    g, gs = ret.shape[0], q.numel() // ret.shape[0] // 128
    qg, out = q.reshape(g, 1, gs, 128), []
    for i in range(g):
        rows = [torch.arange(int(t["cluster_offset"][i, c]), int(t["cluster_offset"][i, c + 1])) for c in ret[i, :kept[i]].tolist()]
        rows = torch.cat(rows + [torch.empty(0, dtype=torch.int64)])
        k, v = (torch.cat((t["steady_" + x][i, :LEN], t[x][i, rows])).reshape(1, -1, 1, 128) for x in ("keys", "values"))
        before = {}
        if est.shape[1]:
            c = est[i]
            o, lse = oat.weighted_flash_decoding(qg[i:i + 1], t["centroids"][i, c].reshape(1, -1, 1, 128),
                                                 t["value_sum"][i, c].reshape(1, -1, 1, 128), t["cluster_size"][i, c],
                                                 return_softmax_lse=True, out_dtype=torch.float32)
            before = dict(previous_out=o, previous_lse=lse)
        out.append(oat.weighted_flash_decoding(qg[i:i + 1], k, v, out_dtype=torch.float32, **before))
    return torch.cat(out).reshape(g, gs, 128)


@pytest.mark.parametrize("size", SIZES)
def test_forms(size):
    from retrievalattention_b200 import _lib, wave

    groups, gs, c, nprobe, n_est, dtype = SIZES[size]
    made, t, q, page, pages = make_layer(groups, gs, c, nprobe, n_est, dtype, seed=c + groups)
    # the new token's rows: the layer's tensors hold others in their place before each call
    gen = torch.Generator().manual_seed(c)
    new = {x: torch.randn((groups, 128), generator=gen).to(dtype) for x in ("steady_keys", "steady_values")}
    stale = {x: t[x][:, LEN - 1].cuda() for x in new}
    for x in new:
        t[x][:, LEN - 1] = new[x]

    def run(budget, ids, cap=-1):
        shape = wave.WaveShape(groups, gs, c, nprobe, n_est, page, budget, made.shape.tokens_per_group, made.shape.steady_stride, dtype)
        layer = wave.WaveIndexLayer(shape, want_ids=ids, **{**made.t, "scratch": wave.new_scratch(shape, "cuda")})
        for x in new:
            layer.t[x][:, LEN - 1] = stale[x]
        layer.append_with_next_compute(new["steady_keys"].cuda(), new["steady_values"].cuda())
        _lib.lib.ri_wave_test_local_cap(cap)
        try:
            out = layer.compute(q.cuda()).cpu()
        finally:
            _lib.lib.ri_wave_test_local_cap(-1)
        for x in new:
            assert torch.equal(layer.t[x].cpu().view(torch.int16), t[x].view(torch.int16))
        return layer, out.float().reshape(groups, gs, 128)

    dist = oss.cluster_distance(q.reshape(groups, gs, 128), t["centroids"], t["cluster_count"] == 0)
    # members are 0 .. 6, a cluster has one page or none: the smaller budget cuts the list in half
    for budget in (pages, max(nprobe // 2, 1)):
        layer, out = run(budget, ids=True)
        ret, est = layer.retrieved_ids.cpu(), layer.estimated_ids.cpu()[:, :n_est]
        assert oss.selection_matches(dist, ret, nprobe)
        if n_est:
            assert oss.selection_matches(dist, torch.cat((ret, est), 1), nprobe + n_est)
        kept = layer.retrieved_kept.tolist()
        assert kept == [oat.surviving_clusters(ret[g], t["cluster_count"][g], page, budget) for g in range(groups)]
        assert budget == pages or nprobe < 3 or min(kept) < nprobe
        ref = attend(q, t, ret, kept, est)
        for form, got in {"ids": out, **{f"cap {cap}": run(budget, False, cap)[1] for cap in (-1, 0, 16)}}.items():
            err = (got - ref).abs()
            assert err.max() <= 2e-2 and err.mean() <= 2e-3, (budget, form, float(err.max()), float(err.mean()))
