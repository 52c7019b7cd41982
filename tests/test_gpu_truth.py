"""bruteforce_knn through the tensor cores' candidates against bruteforce_tile_kernel, which takes what is too small for
them: one call over all queries, then slices of few queries, whose products of values are below the line between the two.
Bit for bit, ties by id included."""
import numpy as np
import pytest
import torch

from glide_b200 import api
from glide_b200.params import Metric, NNDescentParameter

pytestmark = pytest.mark.gpu


def _rows(kind, rng, n, dim):
    if kind == "ties":
        return rng.integers(0, 3, (n, dim)).astype(np.float32)
    x = rng.random((n, dim), dtype=np.float32)
    if kind == "unit":
        x -= np.float32(0.5)
        x /= np.linalg.norm(x, axis=1, keepdims=True)
    if kind == "offset":          # norms far above the distances: the candidates overflow and the other kernel answers
        x += np.float32(500)
    if kind == "nan":
        x[n // 2, 0] = np.nan
    return x


@pytest.mark.parametrize("kind", ["uniform", "ties", "unit", "offset", "nan"])
@pytest.mark.parametrize("n,dim,q,k", [
    (4097, 128, 129, 10),      # a tile and one more on both sides, four operand blocks
    (3000, 33, 128, 128),      # padded rows, the longest lists
    (127, 100, 200, 127),      # fewer rows than a tile, nearly all of them wanted
    (2000, 256, 40, 1),        # the most blocks that stay in shared memory
    (1500, 260, 70, 50),       # blocks of queries stream with the rows'
    (700, 961, 33, 10),        # wide and padded
    (20000, 16, 64, 10),       # one block, half of it filled; a sample of every other stride
])
def test_candidates_from_the_tensor_cores_give_the_tile_kernels_results(gpu_ctx, kind, n, dim, q, k):
    rng = np.random.default_rng(n + dim)
    base = torch.from_numpy(_rows(kind, rng, n, dim)).to(gpu_ctx.torch_device)
    queries = torch.from_numpy(_rows("uniform" if kind == "nan" else kind, rng, q, dim)).to(gpu_ctx.torch_device)
    assert n * q * dim >= 1 << 20
    metric = Metric.Cosine if kind == "unit" else Metric.Euclidean
    ids, dists = api.bruteforce_knn(gpu_ctx, base, queries, k, metric)
    few = max(1, ((1 << 20) - 1) // (n * dim))
    assert n * dim < 1 << 20
    for lo in range(0, q, few):
        want_ids, want = api.bruteforce_knn(gpu_ctx, base, queries[lo:lo + few].contiguous(), k, metric)
        assert torch.equal(ids[lo:lo + few], want_ids)
        assert torch.equal(dists[lo:lo + few].view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("kind", ["uniform", "ties", "offset", "nan"])
@pytest.mark.parametrize("dim", [16, 33, 100, 256, 260, 961])
@pytest.mark.parametrize("degree", [8, 32, 64])
def test_partition_graphs_from_the_tensor_cores_are_the_tile_kernels(gpu_ctx, kind, dim, degree):
    lens = np.array([1, 2, 40, 128, 129, 1000, 4200], np.uint32)   # padding, one tile, a tile and a row, several
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint32)
    rng = np.random.default_rng(dim + degree)
    rows = torch.from_numpy(_rows(kind, rng, int(lens.sum()), dim)).to(gpu_ctx.torch_device)
    got, _, _ = api.build_nnd(gpu_ctx, NNDescentParameter(degree), rows, start, lens, exact_max_rows=16384)
    got = got.cpu().numpy()
    for lo, n in zip(start, lens):
        lo, n = int(lo), int(n)
        part = rows[lo:lo + n].contiguous()
        if kind == "nan" and bool(torch.isnan(part).any()):
            continue      # a row that is no number is nobody's neighbour; which pads fill its own row is checked by its sums' order only
        k = min(degree, n - 1)
        if k == 0:
            continue
        few = max(1, ((1 << 20) - 1) // (n * dim))     # below the line: bruteforce_tile_kernel
        for q in range(0, n, max(few, n // 4)):
            hi = min(n, q + few)
            ids, _ = api.bruteforce_knn(gpu_ctx, part, part[q:hi].contiguous(), min(k + 1, n))
            ids = ids.cpu().numpy()
            for r in range(q, hi):
                want = [i for i in ids[r - q] if i != r][:k]
                assert list(got[lo + r][:k]) == want


@pytest.fixture
def short_passes(gpu_ctx):
    """Passes of a few hundred rows, so that small inputs take several of each kind."""
    def set_passes(**sizes):
        gpu_ctx.limit_exact_knn(**sizes)
        return gpu_ctx
    yield set_passes
    gpu_ctx.limit_exact_knn()


def _tile_kernel(ctx, base, queries, k, metric=Metric.Euclidean):
    """bruteforce_tile_kernel on every query: slices below the line between it and the tensor cores."""
    n, dim = base.shape
    few = max(1, ((1 << 20) - 1) // (n * dim))
    before = ctx.exact_knn_counts
    got = [api.bruteforce_knn(ctx, base, queries[lo:lo + few].contiguous(), k, metric) for lo in range(0, queries.shape[0], few)]
    assert ctx.exact_knn_counts == before      # none of them went through the tensor cores
    return torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])


@pytest.mark.parametrize("kind", ["uniform", "ties", "unit"])
@pytest.mark.parametrize("dim", [64, 33])
@pytest.mark.parametrize("k", [1, 10, 100])
def test_several_passes_give_the_tile_kernels_results(short_passes, kind, dim, k):
    """Three passes over the base rows (the last one ragged; equal rows on both sides of a boundary) times three over
    the queries."""
    rng = np.random.default_rng(dim + k)
    base = _rows(kind, rng, 1409, dim)
    base[512] = base[511]
    base[1024:1030] = base[100]
    queries = _rows(kind, rng, 300, dim)
    queries[7], queries[299] = base[511], base[1024]
    ctx = short_passes(base_rows=512, queries=128)
    base, queries = (torch.from_numpy(x).to(ctx.torch_device) for x in (base, queries))
    before = ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(ctx, base, queries, k)
    after = ctx.exact_knn_counts
    assert after[0] - before[0] == 300 and after[1] == before[1]     # all from the tensor cores' candidates
    want_ids, want = _tile_kernel(ctx, base, queries, k)
    assert torch.equal(ids, want_ids)
    assert torch.equal(dists.view(torch.int32), want.view(torch.int32))


def test_passes_cut_by_the_padded_copy_give_the_tile_kernels_results(short_passes):
    rng = np.random.default_rng(3)
    ctx = short_passes(padded_values=36 * 500)
    base = torch.from_numpy(_rows("uniform", rng, 1700, 35)).to(ctx.torch_device)
    queries = torch.from_numpy(_rows("uniform", rng, 150, 35)).to(ctx.torch_device)
    before = ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(ctx, base, queries, 20)
    after = ctx.exact_knn_counts
    assert after[0] - before[0] == 150 and after[1] == before[1]
    want_ids, want = _tile_kernel(ctx, base, queries, 20)
    assert torch.equal(ids, want_ids) and torch.equal(dists, want)


@pytest.mark.parametrize("kind", ["uniform", "ties"])
@pytest.mark.parametrize("dim,degree", [(36, 32), (33, 16)])
def test_several_launches_over_partitions_give_the_tile_kernels_graph(short_passes, kind, dim, degree):
    lens = np.array([2000, 129, 1400, 1, 600], np.uint32)
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint32)
    ctx = short_passes(tiles=4)
    rows = torch.from_numpy(_rows(kind, np.random.default_rng(dim), int(lens.sum()), dim)).to(ctx.torch_device)
    before = ctx.exact_knn_counts
    got, _, _ = api.build_nnd(ctx, NNDescentParameter(degree), rows, start, lens, exact_max_rows=16384)
    after = ctx.exact_knn_counts
    assert after[2] - before[2] == int(lens.sum()) and after[3] == before[3]
    got = got.cpu().numpy()
    for lo, n in zip(start, lens):
        k = min(degree, int(n) - 1)
        if k == 0:
            continue
        part = rows[int(lo):int(lo) + int(n)].contiguous()
        ids, _ = _tile_kernel(ctx, part, part, k + 1)
        for r, row in enumerate(ids.cpu().numpy()):
            assert list(got[int(lo) + r][:k]) == [i for i in row if i != r][:k]


def _sorted_by_cluster(rng, n, dim, size, spread=0.1):
    """`size` adjacent rows around each of n / size centres."""
    centres = rng.normal(0, 10, ((n + size - 1) // size, dim))
    return (np.repeat(centres, size, axis=0)[:n] + rng.normal(0, spread, (n, dim))).astype(np.float32)


@pytest.mark.parametrize("size,k", [(1000, 100), (300, 32), (64, 10)])
def test_files_sorted_by_cluster_keep_their_candidates_few(gpu_ctx, size, k):
    """A query's neighbours lie side by side in the file: sample and groups that follow the file's order would let many
    clusters through."""
    rng = np.random.default_rng(size)
    base = _sorted_by_cluster(rng, 60_000, 16, size)
    queries = base[rng.choice(60_000, 40, replace=False)] + rng.normal(0, 0.05, (40, 16)).astype(np.float32)
    base, queries = (torch.from_numpy(x).to(gpu_ctx.torch_device) for x in (base, queries.astype(np.float32)))
    before = gpu_ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(gpu_ctx, base, queries, k)
    after = gpu_ctx.exact_knn_counts
    assert after[0] - before[0] == 40 and after[1] == before[1]
    want_ids, want = _tile_kernel(gpu_ctx, base, queries, k)
    assert torch.equal(ids, want_ids) and torch.equal(dists, want)


@pytest.mark.parametrize("degree", [4, 32])
def test_tiny_partitions_and_partitions_sorted_by_cluster_stay_with_the_candidates(gpu_ctx, degree):
    lens = np.array([2, 3, 5, 8, 9000, 33], np.uint32)
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint32)
    rng = np.random.default_rng(degree)
    rows = torch.from_numpy(_sorted_by_cluster(rng, int(lens.sum()), 36, 400)).to(gpu_ctx.torch_device)
    before = gpu_ctx.exact_knn_counts
    got, _, _ = api.build_nnd(gpu_ctx, NNDescentParameter(degree), rows, start, lens, exact_max_rows=16384)
    after = gpu_ctx.exact_knn_counts
    assert after[2] - before[2] == int(lens.sum()) and after[3] == before[3]
    got = got.cpu().numpy()
    for lo, n in zip(start, lens):
        k = min(degree, int(n) - 1)
        part = rows[int(lo):int(lo) + int(n)].contiguous()
        check = np.arange(int(n)) if n < 100 else rng.choice(int(n), 60, replace=False)
        ids, _ = _tile_kernel(gpu_ctx, part, part[torch.from_numpy(check).to(part.device)].contiguous(), k + 1)
        for r, row in zip(check, ids.cpu().numpy()):
            assert list(got[int(lo) + r][:k]) == [i for i in row if i != r][:k]


def test_only_the_queries_that_overflow_or_hold_no_numbers_are_redone(gpu_ctx):
    """5,000 equal rows are too many candidates for the queries beside them; rows that hold an infinity, no number or squares
    beyond fp32 cost the other queries nothing."""
    rng = np.random.default_rng(8)
    n, dim, q, k = 20_000, 20, 120, 10
    base, queries = rng.random((n, dim), np.float32), rng.random((q, dim), np.float32)
    base[7000:12000] = base[7000] + np.float32(3)
    base[3, 2], base[4000, 0], base[19_999, 5], base[150] = np.nan, np.inf, -np.inf, np.float32(2e19)
    queries[[5, 64, 119]] = base[7000]
    queries[10, 3], queries[11, 0] = np.nan, np.inf
    base, queries = (torch.from_numpy(x).to(gpu_ctx.torch_device) for x in (base, queries))
    before = gpu_ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(gpu_ctx, base, queries, k)
    after = gpu_ctx.exact_knn_counts
    assert (after[0] - before[0], after[1] - before[1]) == (q, 5)
    want_ids, want = _tile_kernel(gpu_ctx, base, queries, k)
    assert torch.equal(ids, want_ids)
    assert torch.equal(dists.view(torch.int32), want.view(torch.int32))


def test_a_query_handed_back_in_one_pass_stays_so_in_the_next(short_passes):
    rng = np.random.default_rng(9)
    base, queries = rng.random((15_000, 24), np.float32), rng.random((200, 24), np.float32)
    base[:5000], base[9000:9003] = base[0] + np.float32(3), base[0]
    queries[[0, 130]] = base[0]
    ctx = short_passes(base_rows=6000, queries=128)
    base, queries = (torch.from_numpy(x).to(ctx.torch_device) for x in (base, queries))
    before = ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(ctx, base, queries, 10)
    after = ctx.exact_knn_counts
    assert (after[0] - before[0], after[1] - before[1]) == (200, 2)
    want_ids, want = _tile_kernel(ctx, base, queries, 10)
    assert torch.equal(ids, want_ids) and torch.equal(dists, want)


def test_bad_rows_of_one_partition_leave_the_others_on_the_tensor_cores(gpu_ctx):
    dim, degree = 36, 32
    lens = np.array([900, 900, 900, 4000], np.uint32)     # alone, 900 rows take segment_knn_kernel
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint32)
    rows = np.random.default_rng(4).random((int(lens.sum()), dim), np.float32)
    rows[900 + 130, 3] = np.nan
    rows[1800 + 64, 0], rows[1800 + 100, 1] = np.inf, -np.inf      # both in one half tile
    rows[2700 + 1000:2700 + 3500] = rows[0] + np.float32(2)        # halves 15 to 54 of the last partition
    rows = torch.from_numpy(rows).to(gpu_ctx.torch_device)
    before, stages = gpu_ctx.exact_knn_counts, gpu_ctx.tc_knn_fallbacks
    got, _, _ = api.build_nnd(gpu_ctx, NNDescentParameter(degree), rows, start, lens, exact_max_rows=16384)
    after = gpu_ctx.exact_knn_counts
    assert (after[2] - before[2], after[3] - before[3]) == (int(lens.sum()), 64 + 64 + 40 * 64)
    assert gpu_ctx.tc_knn_fallbacks == stages + 1
    got = got.cpu().numpy()
    for lo in (0, 900, 1800):
        alone, _, _ = api.build_nnd(gpu_ctx, NNDescentParameter(degree), rows[lo:lo + 900].contiguous(), np.array([0], np.uint32),
                                    np.array([900], np.uint32), exact_max_rows=16384)
        real = torch.isfinite(rows[lo:lo + 900]).all(dim=1).cpu().numpy()   # (the others' rows are padding, by the row's own number)
        assert real.sum() >= 898 and np.array_equal(got[lo:lo + 900][real], alone.cpu().numpy()[real])
    part = rows[2700:].contiguous()
    check = np.concatenate([np.arange(900, 1100), np.arange(3400, 3600)])
    ids, _ = _tile_kernel(gpu_ctx, part, part[torch.from_numpy(check).to(part.device)].contiguous(), degree + 1)
    for r, row in zip(check, ids.cpu().numpy()):
        assert list(got[2700 + r]) == [i for i in row if i != r][:degree]


def test_rows_that_overflow_one_tensor_core_path_are_not_given_to_the_other(gpu_ctx):
    rows = np.random.default_rng(4).random((5000, 64), np.float32)
    rows[1000:4500] = rows[0]
    rows = torch.from_numpy(rows).to(gpu_ctx.torch_device)
    before, stages = gpu_ctx.exact_knn_counts, gpu_ctx.tc_knn_fallbacks
    got, _, _ = api.build_nnd(gpu_ctx, NNDescentParameter(32), rows, np.array([0], np.uint32), np.array([5000], np.uint32))
    assert gpu_ctx.tc_knn_fallbacks == stages + 1 and gpu_ctx.exact_knn_counts == before
    ids, _ = _tile_kernel(gpu_ctx, rows, rows[900:1100].contiguous(), 33)
    for r, row in zip(range(900, 1100), ids.cpu().numpy()):
        assert list(got[r].cpu().numpy()) == [i for i in row if i != r][:32]


@pytest.mark.parametrize("lens", [[1500, 1600, 1, 1700, 0, 1800, 900], [1500, 4200, 1600, 1700]])
def test_padded_partitions_are_copied_a_run_at_a_time(lens):
    """Rows of 35 values need a padded copy: the context's scratch holds that of a run of partitions, not of all rows, and the
    graph is the one that a single run gives. A partition beyond the exact limit lies between them once."""
    lens = np.array(lens, np.uint32)
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint32)
    n, small = int(lens.sum()), lens <= 2000
    ctx = api.Context(0)
    rows = torch.from_numpy(np.random.default_rng(4).random((n, 35), np.float32)).to(ctx.torch_device)
    graphs, held = [], []
    for values in (36 * 2000, 0):
        ctx.limit_exact_knn(padded_values=values)
        got, _, _ = api.build_nnd(ctx, NNDescentParameter(16), rows, start, lens, exact_max_rows=2000, seed=3)
        graphs.append(got.cpu().numpy())
        held.append(int(ctx.lib.glide_ctx_workspace_bytes(ctx.handle)))
    counts = ctx.exact_knn_counts
    ctx.close()
    assert counts[2] == 2 * int(lens[small].sum()) and counts[3] == 0
    for lo, l in zip(start[small], lens[small]):
        assert np.array_equal(graphs[0][lo:lo + l], graphs[1][lo:lo + l])
    if small.all():       # (otherwise descent's scratch is the larger)
        assert held[1] - held[0] >= 4 * 36 * (n - 2000)


@pytest.mark.parametrize("dim", [64, 300])      # query blocks that stay in shared memory, blocks that ride along
def test_waits_that_run_out_leave_everything_to_the_tile_kernels(short_passes, dim):
    """As if a wait had run out: a CTA gives up, drains what it has in flight and returns; the results are the tile kernel's, and
    the context goes on."""
    rng = np.random.default_rng(dim)
    ctx = short_passes(give_up=True)
    base, queries = (torch.from_numpy(rng.random((m, dim), np.float32)).to(ctx.torch_device) for m in (3000, 150))
    before = ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(ctx, base, queries, 10)
    after = ctx.exact_knn_counts
    assert (after[0] - before[0], after[1] - before[1]) == (150, 150)
    ctx.limit_exact_knn()
    want_ids, want = api.bruteforce_knn(ctx, base, queries, 10)
    assert ctx.exact_knn_counts[1] == after[1]
    assert torch.equal(ids, want_ids) and torch.equal(dists, want)


@pytest.mark.parametrize("dim", [40, 35])
@pytest.mark.parametrize("offset", [1000, -30_000])
def test_rows_far_from_the_origin_are_taken_about_their_middle(gpu_ctx, dim, offset):
    """Norms far above the distances make every row a candidate; about a point amid the rows the bound is small again."""
    rng = np.random.default_rng(dim)
    base, queries = (torch.from_numpy(rng.random((m, dim), np.float32) + np.float32(offset)).to(gpu_ctx.torch_device) for m in (20_000, 100))
    base[77, 3] = float("nan")
    before = gpu_ctx.exact_knn_counts
    ids, dists = api.bruteforce_knn(gpu_ctx, base, queries, 10)
    after = gpu_ctx.exact_knn_counts
    assert (after[0] - before[0], after[1] - before[1]) == (100, 0)
    want_ids, want = _tile_kernel(gpu_ctx, base, queries, 10)
    assert torch.equal(ids, want_ids) and torch.equal(dists, want)


def test_partitions_far_from_the_origin_are_taken_about_their_middles(gpu_ctx):
    lens = np.array([5000, 300, 6000], np.uint32)
    start = np.concatenate([[0], np.cumsum(lens)[:-1]]).astype(np.uint32)
    rng = np.random.default_rng(2)
    rows = rng.random((int(lens.sum()), 36), np.float32)
    for lo, n, offset in zip(start, lens, (1000, -400, 3000)):
        rows[lo:lo + n] += np.float32(offset)
    rows = torch.from_numpy(rows).to(gpu_ctx.torch_device)
    before, stages = gpu_ctx.exact_knn_counts, gpu_ctx.tc_knn_fallbacks
    got, _, _ = api.build_nnd(gpu_ctx, NNDescentParameter(32), rows, start, lens, exact_max_rows=16384)
    after = gpu_ctx.exact_knn_counts
    assert (after[2] - before[2], after[3] - before[3]) == (int(lens.sum()), 0) and gpu_ctx.tc_knn_fallbacks == stages
    got = got.cpu().numpy()
    for lo, n in zip(start, lens):
        part = rows[int(lo):int(lo) + int(n)].contiguous()
        check = rng.choice(int(n), 60, replace=False)
        ids, _ = _tile_kernel(gpu_ctx, part, part[torch.from_numpy(check).to(part.device)].contiguous(), 33)
        for r, row in zip(check, ids.cpu().numpy()):
            assert list(got[int(lo) + r]) == [i for i in row if i != r][:32]
