"""The entry points beyond the single kernel's range: they run the three stage kernels.  16448 centroids are what a layer of 256K
tokens has after its first re-index of generated tokens."""

import pytest
import torch

from helpers import RECENT, SINK, Case, build_cpu_index, gpu_built_layer, queries, to_gpu_layer
from oracle import attention as oat
from test_peer_gather_gpu import make_gather

pytestmark = pytest.mark.gpu

CENTROIDS, NPROBE, ESTIMATED = 16448, 296, 3815


def bits(x):
    return x.contiguous().view(torch.int16)


@pytest.fixture(scope="module")
def built():
    return gpu_built_layer(1, 2, 4, CENTROIDS * 16, CENTROIDS, 2, NPROBE, ESTIMATED, seed=12, want_ids=False, n_layers=2)


def oracle(layer, t, q, static_len):
    s = layer.shape
    c = {k: v.cpu() for k, v in t.items()}
    return oat.compute(q.cpu(), c["centroids"], c["value_sum"], c["cluster_size"], c["cluster_count"] == 0, c["cluster_count"],
                       c["cluster_offset"], c["keys"], c["values"], c["steady_keys"], c["steady_values"], static_len, s.nprobe,
                       s.nprobe + s.n_estimate, s.page_size, s.buffer_pages)


def check(out, ref):
    err = (out.cpu().float().reshape(ref.shape) - ref.float()).abs()
    assert err.max() <= 2e-2 and err.mean() <= 2e-3, (float(err.max()), float(err.mean()))


def test_gather_stores_every_slice(built):
    (a, b), t, q = built
    shape = (2, 2, 4, 128)
    outs = [torch.zeros(shape, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    flags = [torch.zeros((2,), dtype=torch.int32, device="cuda") for _ in range(2)]
    epoch, error = (torch.full((1,), x, dtype=torch.int32, device="cuda") for x in (1, 0))
    keep = []
    got = [x.compute(q, gather=make_gather(r, 2, outs, flags, epoch, error, 3000, keep)).clone() for r, x in enumerate((a, b))]
    check(got[0], oracle(a, t, q, SINK + RECENT))
    assert torch.equal(bits(a.compute_staged(q)), bits(got[0]))          # the stages are what ran
    for buf in outs:
        for r in range(2):
            assert torch.equal(bits(buf[r]), bits(got[r].reshape(shape[1:])))


def test_static_scratch_on_a_used_array():
    small = Case(1, 2, 4, 1024 + 68, 64, 1, 4, 15, seed=23)
    small_layer = to_gpu_layer(small, build_cpu_index(small), SINK + RECENT)
    (layer,), _, q = gpu_built_layer(1, 1, 4, CENTROIDS * 16, CENTROIDS, 2, NPROBE, ESTIMATED, seed=24)
    assert layer.shape.scratch_bytes() <= 16 << 20
    for call in range(2):
        small_layer.compute_static(queries(small, seed=40 + call).cuda())      # leaves its results in the shared array
        want = layer.compute(q).clone()
        assert torch.equal(bits(layer.compute_static(q)), bits(want))
        assert torch.equal(bits(layer.compute_staged(q)), bits(want))


@pytest.mark.parametrize("call", ["compute", "compute_static"])
def test_new_rows_are_appended_and_attended(call):
    (layer,), t, q = gpu_built_layer(1, 1, 4, CENTROIDS * 16, CENTROIDS, 2, NPROBE, ESTIMATED, seed=25, want_ids=False)
    gen = torch.Generator().manual_seed(25)
    k, v = (torch.randn((1, 128), generator=gen).to(torch.bfloat16).cuda() for _ in range(2))
    layer.t["static_len"].add_(1)
    layer.append_with_next_compute(k, v)
    out = getattr(layer, call)(q)
    row = SINK + RECENT
    assert torch.equal(bits(t["steady_keys"][:, row]), bits(k)) and torch.equal(bits(t["steady_values"][:, row]), bits(v))
    assert not t["steady_keys"][:, row + 1:].any() and not t["steady_values"][:, row + 1:].any()
    check(out, oracle(layer, t, q, row + 1))
