"""Where the decode kernel's outputs go: gather slots on any 2-byte boundary, every rank's with its own."""
import pytest
import torch

from helpers import RECENT, SINK, Case, build_cpu_index, queries, to_gpu_layer
from retrievalattention_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [Case(1, 2, 4, 1024 + 68, 64, 1, 4, 15, seed=71), Case(1, 3, 7, 1024 + 68, 64, 1, 4, 15, seed=72, dtype=torch.float16),
                                  Case(1, 1, 1, 1024 + 68, 64, 1, 4, 15, seed=73)], ids=["gs4", "gs7", "gs1"])
def test_slots_on_any_boundary(case):
    layer = to_gpu_layer(case, build_cpu_index(case), SINK + RECENT, want_ids=False)
    q = queries(case).cuda()
    want = layer.compute(q).flatten().view(torch.int16)
    n, words = want.numel(), [0, 1, 2, 3, 4, 6, 8]                   # 2-byte words in front of each rank's slot
    bufs = [torch.full((n + 16,), -7, dtype=torch.int16, device="cuda") for _ in words]
    slots = torch.tensor([b.data_ptr() + 2 * w for b, w in zip(bufs, words)], dtype=torch.int64).cuda()
    other = torch.zeros((len(words),), dtype=torch.int32, device="cuda")
    g = _lib.WaveGather()
    g.n_ranks, g.rank = len(words), 0
    g.d_out_slots = g.d_flag_slots = slots.data_ptr()
    g.d_flags = g.d_epoch = g.d_error = other.data_ptr()
    out = layer.compute(q, gather=g).flatten().view(torch.int16)
    assert torch.equal(out, want)
    for b, w in zip(bufs, words):
        assert torch.equal(b[w:w + n], want) and (b[:w] == -7).all() and (b[w + n:] == -7).all()
