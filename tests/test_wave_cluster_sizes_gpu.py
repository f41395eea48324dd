"""The single decode kernel over the cluster sizes and slice lengths that its dispatch picks, against the oracle: one to sixteen
CTAs per group, slices of which some CTAs hold little or nothing, 16 keys a thread, more groups than fit the GPU at once."""
import pytest
import torch

from helpers import RECENT, SINK
from oracle import attention as oat

pytestmark = pytest.mark.gpu

# groups, group size, centroids, retrieved, estimated, type.  The CTAs per group are those of a GPU with 148 SMs.
CASES = [
    (1, 8, 2568, 40, 500, torch.bfloat16),       # 16 CTAs, the last one nearly empty
    (7, 3, 12296, 200, 2900, torch.float16),     # 16 CTAs, 4 keys a thread
    (1, 1, 16384, 294, 3801, torch.bfloat16),    # 16 CTAs, slices of exactly 1024
    (8, 5, 1608, 28, 300, torch.bfloat16),       # 10 CTAs
    (4, 2, 760, 13, 0, torch.bfloat16),          # 7 CTAs
    (2, 4, 8, 1, 7, torch.bfloat16),             # 4 CTAs, one of which has the centroids; every cluster taken
    (40, 3, 648, 11, 150, torch.float16),        # 3 CTAs
    (60, 2, 200, 3, 40, torch.bfloat16),         # 2 CTAs
    (100, 4, 136, 2, 30, torch.bfloat16),        # 1 CTA
    (160, 8, 72, 2, 10, torch.bfloat16),         # 1 CTA, more groups than SMs
    (23, 1, 12296, 220, 2800, torch.bfloat16),   # 5 CTAs, 16 keys a thread, the last thread of a slice with 8 of them
    (34, 2, 16384, 294, 3801, torch.float16),    # 4 CTAs, full slices of 4096, groups that take turns
    (9, 8, 16384, 1024, 2000, torch.bfloat16),   # 10 CTAs, the longest candidate list
]


def make_layer(groups, gs, c, nprobe, n_est, dtype, seed):
    """An index of random clusters (0 .. 6 members, some empty), without the clustering: (wave layer, oracle's tensors, q)."""
    from retrievalattention_b200 import wave

    gen = torch.Generator().manual_seed(seed)
    count = torch.randint(0, 7, (groups, c), generator=gen, dtype=torch.int32)
    count[:, :nprobe + n_est] = count[:, :nprobe + n_est].clamp_min(1)
    n, stride = int(count.sum(1).max()), SINK + RECENT + 8
    offset = torch.zeros((groups, c + 1), dtype=torch.int32)
    offset[:, 1:] = count.cumsum(1)
    rand = lambda *shape: torch.randn(shape, generator=gen).to(dtype)        # noqa: E731
    t = dict(centroids=rand(groups, c, 128), value_sum=rand(groups, c, 128) * 2, cluster_size=count.to(dtype),
             cluster_count=count, cluster_offset=offset, keys=rand(groups, n, 128), values=rand(groups, n, 128),
             steady_keys=rand(groups, stride, 128), steady_values=rand(groups, stride, 128))
    page, pages = 8, max(nprobe * 4, 16)
    shape = wave.WaveShape(groups, gs, c, nprobe, n_est, page, pages, n, stride, dtype)
    on_gpu = {k: v.cuda().contiguous() for k, v in t.items()}
    static_len = torch.tensor([SINK + RECENT + 1], dtype=torch.int32, device="cuda")
    layer = wave.WaveIndexLayer(shape, static_len=static_len, scratch=wave.new_scratch(shape, "cuda"), **on_gpu)
    return layer, t, rand(1, 1, groups * gs, 128), page, pages


@pytest.mark.parametrize("groups,gs,c,nprobe,n_est,dtype", CASES)
def test_single_kernel_over_cluster_sizes(groups, gs, c, nprobe, n_est, dtype):
    layer, t, q, page, pages = make_layer(groups, gs, c, nprobe, n_est, dtype, seed=c + groups)
    # an output that starts two bytes behind an 8-byte boundary
    out = torch.empty(q.numel() + 1, dtype=dtype, device="cuda")[1:].view_as(q)
    layer.compute(q.cuda(), out)
    torch.cuda.synchronize()
    ref = oat.compute(q, t["centroids"], t["value_sum"], t["cluster_size"], t["cluster_count"] == 0, t["cluster_count"],
                      t["cluster_offset"], t["keys"], t["values"], t["steady_keys"], t["steady_values"], SINK + RECENT + 1,
                      nprobe, nprobe + n_est, page, pages)
    err = (out.cpu().float().reshape(ref.shape) - ref.float()).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))
