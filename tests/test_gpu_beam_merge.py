"""The beam's merge by insertion, by ranked survivors and by networks: searches on data whose distances
tie rarely, often and nearly always, on random graphs, against the oracle's networks, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from glide_b200 import api
from glide_b200.params import Metric, SearchParameter

pytestmark = pytest.mark.gpu


def _set(kind, n, dim, nq, degree, seed=5):
    rng = np.random.default_rng(seed)
    if kind == "floats":
        base, q = rng.random((n, dim)), rng.random((nq, dim))
    else:
        hi = {"some_ties": 200, "ties": 12, "all_tie": 2}[kind]
        base, q = rng.integers(0, hi, (n, dim)), rng.integers(0, hi, (nq, dim))
    base, q = base.astype(np.float32), q.astype(np.float32)
    graph = rng.integers(0, n, (n, degree)).astype(np.uint32)
    graph[rng.random((n, degree)) < 0.1] = 0xFFFFFFFF   # holes, as after pruning
    return base, q, graph


@pytest.mark.parametrize("kind", ["floats", "some_ties", "ties", "all_tie"])
@pytest.mark.parametrize("degree", [8, 32, 33, 130])      # lane-resident up to 32, one or two 32-slot groups, two-warp sort
@pytest.mark.parametrize("beam", [32, 64, 96, 128, 256, 512])
def test_search_on_tied_distances_matches_oracle(gpu_ctx, kind, degree, beam):
    n, dim, nq = 1500, 24, 40
    base, q, graph = _set(kind, n, dim, nq, degree)
    cent, start = base[:2].copy(), np.array([3, 77], np.uint32)
    o = oracle.SearchParams.derive(beam, degree, top_k=min(beam, 100))
    want_ids, want_d = oracle.search(base, graph, cent, start, q, o)
    t = lambda a: torch.from_numpy(a).to(gpu_ctx.torch_device)  # noqa: E731
    sp = SearchParameter(top_k=o.top_k, beam=o.beam, max_iterations=o.max_iterations, min_iterations=o.min_iterations,
                         hash_bit=o.hash_bit, hash_reset_interval=o.hash_reset_interval)
    ids, d, _ = api.search(gpu_ctx, t(base), api.from_u32(gpu_ctx, graph), t(cent), api.from_u32(gpu_ctx, start), t(q), sp,
                           Metric.Euclidean)
    assert np.array_equal(api.to_u32(ids), want_ids)
    assert np.array_equal(d.cpu().numpy(), want_d)
