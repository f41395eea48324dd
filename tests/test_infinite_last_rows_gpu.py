"""Infinite values in the last row of a list, which stands in for the rows that fill up a step of 16: those have no part in the
result, whatever the last row holds."""
import pytest
import torch

from oracle import attention as oat
from retrievalattention_b200 import kernels
from test_wave_cluster_sizes_gpu import make_layer

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("groups,gs,length,dtype", [(2, 4, 1, torch.bfloat16), (1, 8, 15, torch.float16), (3, 7, 16, torch.bfloat16),
                                                    (2, 1, 17, torch.float16), (1, 4, 333, torch.bfloat16), (2, 8, 1039, torch.float16)])
def test_operator(groups, gs, length, dtype):
    gen = torch.Generator().manual_seed(length)
    q, k, v = (torch.randn(s, generator=gen).to(dtype) for s in ((groups, 1, gs, 128), (groups, length, 1, 128), (groups, length, 1, 128)))
    ref = oat.weighted_flash_decoding(q, k, v, out_dtype=torch.float32)
    for x, channel in ((INF, 6), (-INF, 77)):
        v[:, -1, :, channel] = x
        ref[..., channel] = x
    out = kernels.weighted_flash_decoding(q.cuda(), k.cuda(), v.cuda()).cpu().float()
    assert torch.equal(out.isinf(), ref.isinf()) and torch.equal(out[out.isinf()], ref[ref.isinf()])
    err = (out - ref)[~ref.isinf()].abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))


# one to sixteen CTAs a group; estimation and exact steps that are not full
@pytest.mark.parametrize("form", ["compute", "compute_staged"])
@pytest.mark.parametrize("groups,gs,c,nprobe,n_est,dtype", [
    (1, 8, 2568, 40, 500, torch.bfloat16), (2, 8, 12288, 147, 17, torch.bfloat16), (8, 5, 1608, 28, 300, torch.float16),
    (60, 2, 200, 3, 41, torch.bfloat16), (100, 4, 136, 2, 30, torch.float16)])
def test_decode(groups, gs, c, nprobe, n_est, dtype, form):
    layer, _, q, _, _ = make_layer(groups, gs, c, nprobe, n_est, dtype, seed=c)
    q = q.cuda()
    plain = getattr(layer, form)(q).clone()
    layer.t["values"][..., 9] = INF                        # every retrieved row's, every estimated cluster's
    layer.t["value_sum"][..., 100] = -INF
    out = getattr(layer, form)(q)
    assert bool((out[..., 9] == INF).all()) and bool((out[..., 100] == -INF).all())
    rest = [x for x in range(128) if x not in (9, 100)]
    assert torch.equal(out[..., rest].view(torch.int16), plain[..., rest].view(torch.int16))
