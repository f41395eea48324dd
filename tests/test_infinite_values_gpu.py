"""Value rows with infinities: a channel that holds one comes out infinite with that sign (its probability is positive, whatever
part of it 16 bits leave over), every other channel as without them."""
import pytest
import torch

from helpers import RECENT, SINK, Case, build_cpu_index, queries, to_gpu_layer
from oracle import attention as oat
from retrievalattention_b200 import kernels

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.mark.parametrize("groups,gs,length,dtype", [(2, 4, 333, torch.bfloat16), (3, 8, 1040, torch.float16), (1, 1, 64, torch.bfloat16)])
def test_operator(groups, gs, length, dtype):
    gen = torch.Generator().manual_seed(length)
    q, k, v = (torch.randn(s, generator=gen).to(dtype) for s in ((groups, 1, gs, 128), (groups, length, 1, 128), (groups, length, 1, 128)))
    ref = oat.weighted_flash_decoding(q, k, v, out_dtype=torch.float32)
    rows = {0: (INF, 3), 9: (-INF, 70), 40: (INF, 127)}          # none is the last row, which stands in for rows past the end
    for row, (x, channel) in rows.items():
        v[:, row, :, channel] = x
        ref[..., channel] = x
    out = kernels.weighted_flash_decoding(q.cuda(), k.cuda(), v.cuda()).cpu().float()
    assert torch.equal(out.isinf(), ref.isinf()) and torch.equal(out[out.isinf()], ref[ref.isinf()])
    err = (out - ref)[~ref.isinf()].abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_single_kernel(dtype):
    case = Case(1, 2, 4, 1024 + 68, 64, 1, 4, 15, seed=61, dtype=dtype)
    cpu = build_cpu_index(case)
    layer = to_gpu_layer(case, cpu, SINK + RECENT)
    q = queries(case).cuda()
    plain = layer.compute(q).clone()
    layer.t["steady_values"][:, 2, 5] = INF
    layer.t["steady_values"][:, 17, 99] = -INF
    out = layer.compute(q)
    assert bool((out[..., 5] == INF).all()) and bool((out[..., 99] == -INF).all())
    rest = [c for c in range(128) if c not in (5, 99)]
    assert torch.equal(out[..., rest], plain[..., rest])
