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


def _sp(o):
    return SearchParameter(top_k=o.top_k, beam=o.beam, max_iterations=o.max_iterations, min_iterations=o.min_iterations,
                           hash_bit=o.hash_bit, hash_reset_interval=o.hash_reset_interval)


def _far_rows(n, dim, seed, how):
    """Rows of which one in twenty lies where the square of a distance is beyond fp32 (or holds an infinity)."""
    rng = np.random.default_rng(seed)
    base = rng.random((n, dim)).astype(np.float32)
    far = rng.choice(n, n // 20, replace=False)
    near = base.copy()
    if how == "infinity":
        base[far, 1] = np.inf
    else:
        base[far] *= np.float32(1e25)
    return base, near, far


@pytest.mark.parametrize("how", ["infinity", "square"])
@pytest.mark.parametrize("degree", [8, 32, 64, 130])
@pytest.mark.parametrize("beam", [32, 64, 128, 256, 512])
def test_search_with_infinite_distances_matches_oracle(gpu_ctx, how, degree, beam):
    """Infinite distances sort behind the empty slots; a seed step that meets them leaves a beam that is not ascending. Every
    third query is far from all rows, so that all of its distances are infinite."""
    n, dim, nq = 1500, 24, 60
    base, _, far = _far_rows(n, dim, 5, how)
    rng = np.random.default_rng(6)
    graph = rng.integers(0, n, (n, degree)).astype(np.uint32)
    graph[rng.random((n, degree)) < 0.1] = 0xFFFFFFFF
    graph[3, 1], graph[77, 1:3] = far[0], far[1:3]
    q = rng.random((nq, dim)).astype(np.float32)
    q[::3] = np.float32(3e24) * rng.choice([-1, 1], (nq // 3, 1)).astype(np.float32)
    cent = np.stack([base[np.setdiff1d(np.arange(n), far)[0]], np.full(dim, 3e24, np.float32), np.full(dim, -3e24, np.float32)])
    start = np.array([3, 77, 3], np.uint32)
    o = oracle.SearchParams.derive(beam, degree, top_k=min(beam, 100))
    want_ids, want_d = oracle.search(base, graph, cent, start, q, o)
    t = lambda a: torch.from_numpy(a).to(gpu_ctx.torch_device)  # noqa: E731
    for copies in (1, 100):      # a CTA per query, a warp per query
        ids, d, _ = api.search(gpu_ctx, t(base), api.from_u32(gpu_ctx, graph), t(cent), api.from_u32(gpu_ctx, start),
                               t(np.tile(q, (copies, 1))), _sp(o), Metric.Euclidean)
        assert np.array_equal(api.to_u32(ids), np.tile(want_ids, (copies, 1)))
        assert np.array_equal(d.cpu().numpy(), np.tile(want_d, (copies, 1)))


@pytest.mark.parametrize("degree,out", [(16, 24), (32, 32), (48, 64)])
@pytest.mark.parametrize("beams", [(32, 64), (64, 128), (288, 288)])
def test_build_with_infinite_distances_matches_oracle(gpu_ctx, degree, out, beams):
    n = 1200
    base, near, far = _far_rows(n, 24, 5, "square")
    ids = oracle.bruteforce_knn(near, near, degree + 1, want_dists=False)
    knn = np.array([[i for i in row if i != j][:degree] for j, row in enumerate(ids)], np.uint32)
    knn[9, [2, 5]] = far[:2]
    ob, orf = (oracle.SearchParams.derive(b, degree) for b in beams)
    one = np.array([0], np.uint32)
    want = oracle.build_rows(base, knn, one, np.array([n], np.uint32), np.array([9], np.uint32), np.arange(n, dtype=np.uint32),
                             n, out, ob, 1.05)
    rows = torch.from_numpy(base).to(gpu_ctx.torch_device)
    got = api.build_partition(gpu_ctx, rows, api.from_u32(gpu_ctx, knn), 9, out, _sp(ob), 1.05)
    assert np.array_equal(api.to_u32(got), want)
    oracle.reverse_graph(want)
    want[9, :2] = far[:2]
    refined = oracle.refine(base, want, None, 9, orf, 1.05)
    got = api.from_u32(gpu_ctx, want)
    api.refine_partition(gpu_ctx, rows, got, 9, _sp(orf), 1.05)
    assert np.array_equal(api.to_u32(got), refined)
