"""Small batches give a query a CTA (a team), large ones a warp: the same queries through both, at sizes around
the edges of each form, against one another and the oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from glide_b200 import api
from glide_b200.params import Metric, SearchParameter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [4, 127, 128, 132, 301, 960])    # a chunk per lane up to 128 in multiples of four, wide rows otherwise
@pytest.mark.parametrize("degree", [1, 32, 33, 64, 65])            # lanes, strip, and the widest a team takes and one more
@pytest.mark.parametrize("beam", [32, 64, 160, 288])
def test_a_team_and_a_warp_give_the_oracles_results(gpu_ctx, dim, degree, beam):
    rng = np.random.default_rng(dim + degree)
    n, nq = 900, 24
    base, q = rng.random((n, dim), np.float32), rng.random((nq, dim), np.float32)
    graph = rng.integers(0, n, (n, degree)).astype(np.uint32)
    graph[rng.random((n, degree)) < 0.1] = 0xFFFFFFFF
    cent, start = base[:2].copy(), np.array([3, 77], np.uint32)
    o = oracle.SearchParams.derive(beam, degree, top_k=min(beam, 50))
    metric = Metric.Cosine if degree == 64 else Metric.Euclidean
    want_ids, want_d = oracle.search(base, graph, cent, start, q, o, int(metric))
    t = lambda a: torch.from_numpy(a).to(gpu_ctx.torch_device)  # noqa: E731
    sp = SearchParameter(top_k=o.top_k, beam=o.beam, max_iterations=o.max_iterations, min_iterations=o.min_iterations,
                         hash_bit=o.hash_bit, hash_reset_interval=o.hash_reset_interval)
    args = (gpu_ctx, t(base), api.from_u32(gpu_ctx, graph), t(cent), api.from_u32(gpu_ctx, start))
    for copies in (1, 25, 50, 240):      # 24 queries and 5,760: more than the device holds as teams
        ids, d, _ = api.search(*args, t(np.tile(q, (copies, 1))), sp, metric)
        assert np.array_equal(api.to_u32(ids), np.tile(want_ids, (copies, 1)))
        assert np.array_equal(d.cpu().numpy(), np.tile(want_d, (copies, 1)))
