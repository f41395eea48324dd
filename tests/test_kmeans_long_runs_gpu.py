"""The first update of the index build where a warp has a run of several clusters and some of them hold 512 members or more: at the
first, a middle and the last place of a run, two of a run, two neighbours, and in several runs of a CTA."""
import pytest
import torch

from oracle import kmeans as okm
from test_kmeans_gpu import check_assignments

pytestmark = pytest.mark.gpu

CENTS = 2048
# clusters of a run on a GPU with 148 SMs -> problems of CENTS clusters that make it so (a run is a power of two, of 14208 or more)
PROBLEMS = {1: 2, 2: 14, 4: 28, 8: 56}
# which clusters are long: (a CTA has four runs, of 1 .. 8 clusters)
LONG = [[0, 3, 11, 24, 25, 31, 1000, 2047], [1, 2, 4, 7, 8, 15, 16, 2040], [0, 1, 2, 3, 4, 5, 6, 7]]
TOKENS = 8448


def make(problems, dtype):
    """Keys [problems, TOKENS, 128].  Of the initial centroids the LONG ones are long keys, the rest short: the former win all
    tokens and share them about evenly, and which token is whose depends on all of their members after the update."""
    gen = torch.Generator().manual_seed(problems)
    start = okm.initial_centroid_indices(TOKENS, CENTS)
    k = torch.randn((problems, TOKENS, 128), generator=gen)
    k[:, start] *= 0.01
    for p in range(problems):
        u = torch.randn((8, 128), generator=gen)
        k[p, start[LONG[p % 3]]] = u / u.norm(dim=1, keepdim=True) * 200
    return k.to(dtype)


@pytest.mark.parametrize("run,dtype", [(1, torch.float16), (2, torch.float16), (4, torch.float16), (4, torch.bfloat16), (8, torch.float16)])
def test_long_clusters_of_a_run(run, dtype):
    from retrievalattention_b200.cache_hub import kmeans as gk

    problems = PROBLEMS[run]
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the runs are those of a GPU with 148 SMs")
    k = make(problems, dtype)
    v = torch.randn(k.shape, generator=torch.Generator().manual_seed(1)).to(dtype)
    got = gk._run(k.cuda(), v.cuda(), CENTS, 2, 1, False, False)
    assert int(got["error"]) == 0
    start = okm.initial_centroid_indices(TOKENS, CENTS)
    for p in range(0, problems, 7):
        part = k[p:p + 7]
        first = okm.assign(part, part[:, start])
        for i, a in enumerate(first):                                # the case is what it says
            assert (a.bincount(minlength=CENTS)[LONG[(p + i) % 3]] >= 512).all()
        want = okm.segment_k_means(part, v[p:p + 7], CENTS, 2, 1, return_assignments=True)[4]
        check_assignments(got["assign"][p:p + 7].cpu(), want.to(torch.int32), part, CENTS, 2, 1)
