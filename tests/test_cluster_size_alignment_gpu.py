"""Cluster sizes on an 8-byte boundary that is no 16-byte one, whatever kernel form the geometry gets."""
import pytest
import torch

from retrievalattention_b200 import wave
from test_wave_cluster_sizes_gpu import make_layer

pytestmark = pytest.mark.gpu


# 4, 8 and 16 keys a thread, and the stage kernels
@pytest.mark.parametrize("groups,c", [(8, 1608), (100, 136), (9, 16384), (60, 4104), (23, 12296), (150, 2056), (2, 16448)])
def test_sizes_on_an_eight_byte_boundary(groups, c):
    layer, _, q, _, _ = make_layer(groups, 3, c, 20, c // 5, torch.bfloat16, seed=c)
    q = q.cuda()
    want = layer.compute(q).clone()
    store = torch.empty((groups * c + 8,), dtype=torch.bfloat16, device="cuda")
    sizes = store[4:4 + groups * c].view(groups, c).copy_(layer.t["cluster_size"])
    assert store.data_ptr() % 16 == 0 and sizes.data_ptr() % 16 == 8
    moved = wave.WaveIndexLayer(layer.shape, **{**layer.t, "cluster_size": sizes})
    assert torch.equal(moved.compute(q).view(torch.int16), want.view(torch.int16))
