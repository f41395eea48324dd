"""The gather's report of a decode kernel that gave up and left its slice out.  The kernel's mark in the error word is set from the
host here; no wait of any kernel runs out."""
import ctypes as C

import pytest
import torch

from retrievalattention_b200 import _lib
from test_peer_gather_gpu import make_gather

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ranks,rank", [(2, 0), (2, 1), (33, 32), (64, 5)])
def test_a_missing_slice_raises_no_flags(ranks, rank):
    word = lambda n, x: torch.full((n,), x, dtype=torch.int32, device="cuda")        # noqa: E731
    outs = [torch.zeros((ranks, 1, 1, 128), dtype=torch.bfloat16, device="cuda") for _ in range(ranks)]
    flags = [word(ranks, 3) for _ in range(ranks)]
    flags[rank][torch.arange(ranks, device="cuda") != rank] = 4          # the others are done with this step
    epoch, error, keep = word(1, 4), word(1, 2), []
    gather = make_gather(rank, ranks, outs, flags, epoch, error, 3000, keep)

    def wait():
        _lib.check(_lib.lib.ri_wave_gather_wait(C.byref(gather), _lib.current_stream()))
        torch.cuda.synchronize()
        return [int(f[rank]) for f in flags]

    assert wait() == [3] * ranks and int(error) == 1                    # reported here; the other ranks will wait in vain
    assert wait() == [4] * ranks and int(error) == 1                    # once: a later call raises its flags, the report stays
