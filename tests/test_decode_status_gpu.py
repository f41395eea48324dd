"""A wave decode call whose device-side wait ran out is reported: by the next call, and by ``check_prefill_errors``."""
import subprocess
import sys

import pytest
import torch

from helpers import RECENT, SINK, Case, build_cpu_index, queries, to_gpu_layer

pytestmark = pytest.mark.gpu

CASE = Case(1, 2, 4, 1024 + 68, 64, 1, 4, 15, seed=51)


@pytest.fixture(scope="module")
def layer():
    return to_gpu_layer(CASE, build_cpu_index(CASE), SINK + RECENT)


@pytest.mark.parametrize("call", ["compute", "compute_static"])
def test_next_decode_call_reports_a_wait_that_ran_out(layer, call):
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    q = queries(CASE).cuda()
    want = getattr(layer, call)(q).clone()
    ra._status_word(q.device).value = 51
    with pytest.raises(RuntimeError, match="ri_wave_decode_layer.*51"):
        getattr(layer, call)(q)
    assert torch.equal(getattr(layer, call)(q), want)                 # reported once
    ra.check_prefill_errors()


def test_word_is_looked_at_after_a_capture_not_in_it(layer):
    from retrievalattention_b200.attn_hub import retroinfer_attn as ra

    q = queries(CASE).cuda()
    layer.compute(q)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    ra._status_word(q.device).value = 55
    with torch.cuda.graph(graph):
        layer.compute(q)
    graph.replay()
    with pytest.raises(RuntimeError, match="55"):
        ra.check_prefill_errors()
    ra.check_prefill_errors()


def test_process_that_only_decodes_is_told():
    code = """
import ctypes, sys
sys.path.insert(0, "tests")
from helpers import RECENT, SINK, Case, build_cpu_index, queries, to_gpu_layer
from retrievalattention_b200 import _lib
from retrievalattention_b200.attn_hub import retroinfer_attn as ra
case = Case(1, 2, 4, 1024 + 68, 64, 1, 4, 15, seed=51)
to_gpu_layer(case, build_cpu_index(case), SINK + RECENT).compute(queries(case).cuda())
ra.check_prefill_errors()
ctypes.c_int32.from_address(_lib.lib.ri_status_word()).value = 52
try:
    ra.check_prefill_errors()
except RuntimeError as e:
    assert "52" in str(e)
else:
    raise SystemExit("nothing reported")
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300)
