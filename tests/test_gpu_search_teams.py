"""Small batches give a query a CTA (a team), large ones a warp: the same queries through both, at sizes around
the edges of each form, against one another and the oracle, bit for bit."""
import numpy as np
import pytest
import torch

import oracle
from glide_b200 import api, large
from glide_b200.params import IndexParameter, Metric, SearchParameter

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


@pytest.mark.parametrize("dim", [64, 128, 301])
@pytest.mark.parametrize("degree", [32, 48])
def test_small_batches_run_as_teams_and_count_what_they_read(gpu_ctx, dim, degree):
    """One query has a team, thousands have not; the rows scored and the expansions are the same, and what a team reads
    beside them is counted apart: whole adjacency rows where rows fit the lanes, nothing otherwise."""
    rng = np.random.default_rng(dim + degree)
    n, nq = 900, 24
    base, q = rng.random((n, dim), np.float32), rng.random((nq, dim), np.float32)
    graph = rng.integers(0, n, (n, degree)).astype(np.uint32)
    sp = SearchParameter(top_k=10, beam=64).derive(degree)
    t = lambda a: torch.from_numpy(a).to(gpu_ctx.torch_device)  # noqa: E731
    args = (gpu_ctx, t(base), api.from_u32(gpu_ctx, graph), t(base[:2].copy()), api.from_u32(gpu_ctx, np.array([3, 77], np.uint32)))
    counts = {}
    gpu_ctx.enable_counters(True)
    for copies in (1, 400):
        api.search(*args, t(np.tile(q, (copies, 1))), sp)
        counts[copies] = gpu_ctx.read_counters()[:3]
        assert (gpu_ctx.last_team_warps > 1) == (copies == 1)
    gpu_ctx.enable_counters(False)
    rows, expansions, beside = counts[1]
    assert counts[400] == (400 * rows, 400 * expansions, 0)
    assert beside == ((expansions + nq) * degree - rows if dim <= 128 and dim % 4 == 0 else 0)


@pytest.mark.parametrize("dim,degree", [(64, 48), (132, 32), (132, 48)])
def test_teams_over_several_partitions_give_the_streamed_results(gpu_ctx, dim, degree):
    """Large path: queries routed to resident partitions take teams, the streamed walk (checked against the oracle elsewhere)
    a warp per query."""
    rng = np.random.default_rng(dim + degree)
    base, queries = rng.random((4000, dim), np.float32), rng.random((30, dim), np.float32)
    pre = large.preprocess_for_large(gpu_ctx, base, 5, 0.2, batch_num=2, seed=2)
    index = large.GLIDE_large(gpu_ctx, degree, Metric.Euclidean, pre["h_reorder_data"], pre["h_map"], pre["h_centroids"],
                              pre["h_segment_start"], pre["h_segment_length"])
    pk, pr = SearchParameter(beam=64).derive(32), SearchParameter(beam=64).derive(32)
    index.build(IndexParameter(degree, 32, 1.05), pk, pr, seed=5)
    d_q = torch.from_numpy(queries).to(gpu_ctx.torch_device)
    sps = [SearchParameter(top_k=10, beam=beam).derive(degree) for beam in (32, 64, 128, 160)]
    streamed = [index.search(sp, 3, 1.2, d_q) for sp in sps]
    assert index.make_resident(10 ** 9) == 5
    for sp, (want_ids, want_d, _) in zip(sps, streamed):
        ids, d, _ = index.search(sp, 3, 1.2, d_q)
        assert gpu_ctx.last_team_warps > 1
        assert np.array_equal(ids, want_ids) and np.array_equal(d, want_d)
    index.close()
