"""The work that users of this package have it do, as cases that can be timed and compared.

Six kinds of calls, through the public entry points of `glide_b200`:

  search        `GLIDE.search`: queries in device memory against a finished index, results on the host
  pipe          `SearchPipe`: batches of queries in pinned host memory, several in flight
  build         `pipeline.build_small`: partition, kNN graph, subgraphs, boundary merge, reverse edges, refinement
  large_build   `GLIDE_large.build`: rows in pinned host memory streamed through the GPU, the graph back in host memory
  large_search  `GLIDE_large.search`: queries routed to several partitions that lie in device memory
  truth         `bruteforce_knn`: exact neighbours, what recall is measured against

Sizes, distributions and parameters are those of the repository's own configurations (`datasets.CONFIGS`),
its tests and its benchmark, or lie between them. Data are drawn on the GPU from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from glide_b200 import api, datasets, large, pipeline
from glide_b200.params import IndexParameter, Metric, NNDescentParameter, SearchParameter

_CONTEXT = None


def _ctx() -> api.Context:
    """One context per process, as a program that uses the package keeps one."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = api.Context(0)
    return _CONTEXT


def _case(name, kind, data, n, dim, components, metric, degree, partitions, queries=0, beam=0, top_k=0, batches=0,
          route_min=0, sample_factor=0.1, uint8=False):
    case = dict(kind=kind, data=data, n=n, dim=dim, components=components, metric=metric, degree=degree,
                partitions=partitions, sample_factor=sample_factor, queries=queries, beam=beam, top_k=top_k,
                batches=batches, route_min=route_min, uint8=uint8)
    return case if name is None else dict(case, name=name)


def listed():
    return [
        # one query against the small index of the correctness configuration (cfg0): an interactive lookup
        _case("lookup_one", "search", "uniform", 10_000, 32, 0, "Euclidean", 32, 1, queries=1, beam=32, top_k=10),
        # the headline workload (cfg1): 10,000 queries on a million integer-valued descriptors at recall@10 >= 0.95
        _case("search_cfg1", "search", "int_mixture", 1_000_000, 128, 1024, "Euclidean", 32, 1024, queries=10_000, beam=28, top_k=10),
        # unit vectors under cosine, a wide beam and a long result list: candidate generation for a re-ranker
        _case("search_cosine_k100", "search", "unit_lowrank_mixture", 300_007, 100, 16, "Cosine", 32, 16, queries=2_000, beam=128,
              top_k=100),
        # wide rows (cfg2's dimension and degree, fewer rows so that the index is made in a second)
        _case("search_wide_rows", "search", "scaled_mixture", 100_000, 960, 256, "Euclidean", 64, 25, queries=1_000, beam=49, top_k=10),
        # a service: eight batches of host queries through the pipe, three in flight
        _case("pipe_batches", "pipe", "int_lowrank_mixture", 500_000, 128, 32, "Euclidean", 32, 32, queries=1_250, beam=60, top_k=10,
              batches=8),
        # the correctness configuration built from its rows: launches and host work count
        _case("build_cfg0", "build", "uniform", 10_000, 32, 0, "Euclidean", 32, 1),
        # the headline build
        _case("build_cfg1", "build", "int_mixture", 1_000_000, 128, 1024, "Euclidean", 32, 1024),
        # the reference's default ten partitions on unit vectors whose dimension is no multiple of 32
        _case("build_cosine", "build", "unit_lowrank_mixture", 200_003, 100, 10, "Cosine", 32, 10),
        # wide rows, degree 64
        _case("build_wide_rows", "build", "scaled_mixture", 60_000, 960, 256, "Euclidean", 64, 15),
        # byte rows in host memory, partitions streamed through the GPU (the reference's large path holds bytes)
        _case("large_build_u8", "large_build", "int_lowrank_mixture", 400_000, 128, 8, "Euclidean", 32, 8, uint8=True),
        # queries routed to at least two of the partitions, all of them in device memory (cfg3's rows and metric)
        _case("large_search", "large_search", "unit_lowrank_mixture", 400_000, 96, 16, "Cosine", 32, 16, queries=10_000, beam=64, top_k=10,
              route_min=2),
        # ground truth for a recall figure
        _case("truth", "truth", "int_mixture", 1_000_000, 128, 1024, "Euclidean", 0, 1, queries=1_000, top_k=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "pipe", "build", "build", "build", "large_build", "large_search", "truth"])
    uint8 = kind == "large_build" and rng.random() < 0.5
    data = rng.choice(["uniform", "int_mixture", "int_lowrank_mixture", "unit_mixture", "unit_lowrank_mixture", "scaled_mixture"])
    if uint8:
        data = rng.choice(["int_mixture", "int_lowrank_mixture"])
    # dimensions: the usual ones, multiples of four and any
    dim = rng.choice([rng.choice([32, 64, 96, 128, 256, 768, 960]), 4 * _log_int(rng, 5, 64), _log_int(rng, 20, 300)])
    if uint8:
        dim = 4 * ((dim + 3) // 4)   # byte rows come in multiples of four
    # values per row bound the rows: no more than the listed cases hold, and the builds stay within a second
    most = {"search": 96e6, "pipe": 48e6, "build": 24e6, "large_build": 32e6, "large_search": 32e6, "truth": 96e6}[kind]
    n = _log_int(rng, 4_000, max(8_000, min(1_000_000, most / dim)))
    per_partition = _log_int(rng, 900, 12_000 if dim > 128 or dim % 32 else 40_000)
    partitions = max(1, min(1024, n // per_partition))
    components = max(1, min(1024, int(partitions * rng.choice([1, 1, 4]))))
    degree = rng.choice([16, 32, 32, 32, 64])
    metric = "Cosine" if data.startswith("unit") else "Euclidean"
    beam = rng.choice([10, 20, 28, 32, 50, 60, 64, 100, 128, 200])
    top_k = min(beam, rng.choice([1, 10, 10, 10, 50, 100]))
    case = _case(None, kind, data, n, dim, components, metric, degree, partitions, uint8=uint8)
    if kind in ("search", "large_search"):
        case.update(queries=_log_int(rng, 1, 10_000 if dim <= 128 else 2_000), beam=beam, top_k=top_k)
        if kind == "large_search":
            case.update(route_min=rng.randint(1, 4))
    elif kind == "pipe":
        case.update(queries=_log_int(rng, 1, 2_000), beam=beam, top_k=top_k, batches=rng.randint(2, 8))
    elif kind == "truth":
        case.update(queries=_log_int(rng, 10, 1_000), top_k=top_k, partitions=1)
    return case


def _spec(case, seed):
    return datasets.DatasetSpec("rows", case["n"], case["dim"], max(1, case["queries"] * max(1, case["batches"])), case["data"],
                                case["components"], case["metric"], max(1, case["degree"]), int(seed) % 1_000_003)


def _draw_rows(spec, count, stream, device):
    """Rows of the mixtures of `datasets` (uniform ones are drawn here: the device generator has none)."""
    if spec.kind == "uniform":
        g = torch.Generator(device=device)
        g.manual_seed(spec.seed * 8 + stream)
        return torch.rand((count, spec.dim), generator=g, device=device)
    return datasets.device_rows(spec, 0, count, device, stream=stream)


def _build_config(case, seed):
    return pipeline.BuildConfig(metric=Metric.parse(case["metric"]), centroid_num=case["partitions"], sample_factor=case["sample_factor"],
                                knn_degree=max(32, case["degree"]), graph_degree=case["degree"], seed=int(seed) % 1_000_003)


def prepare(case, seed):
    ctx = _ctx()
    spec = _spec(case, seed)
    kind = case["kind"]
    rows = _draw_rows(spec, case["n"], 1, ctx.torch_device)
    state = dict(case=case, kind=kind, ctx=ctx, metric=Metric.parse(case["metric"]), seed=int(seed) % 1_000_003)
    if case["queries"]:
        state["queries"] = _draw_rows(spec, spec.n_queries, 2, ctx.torch_device)
    if case["beam"]:
        state["params"] = pipeline.derive_search_params(case["beam"], case["degree"], case["top_k"])
    if kind == "truth":
        state["rows"] = rows
    elif kind == "build":
        state["rows"], state["config"] = rows, _build_config(case, seed)
    elif kind in ("search", "pipe"):
        state["index"] = pipeline.build_small(ctx, rows, _build_config(case, seed)).index
        if kind == "pipe":
            q, k, batches = case["queries"], case["top_k"], case["batches"]
            host = state.pop("queries").cpu().numpy()
            state["batches"] = [dict(q=large.pinned_copy(host[b * q:(b + 1) * q]), ids=large.pinned_copy(np.zeros((q, k), np.int32)),
                                     dists=large.pinned_copy(np.zeros((q, k), np.float32))) for b in range(batches)]
            state["pipe"] = state["index"].search_pipe(q, k, 3)
    else:
        # the large path starts from rows grouped by partition in host memory (preprocess_for_large)
        cfg = state["config"] = _build_config(case, seed)
        d_centroids, _ = api.get_centroids(ctx, rows, case["partitions"], case["sample_factor"], cfg.seed, 0, cfg.metric)
        d_segment, seg_start, seg_len = api.define_partition(ctx, rows, d_centroids, -1.0, cfg.metric)
        order = torch.argsort(d_segment[:, 0], stable=True)
        grouped = rows[order]
        h_rows = large.pinned_copy((grouped.to(torch.uint8) if case["uint8"] else grouped).cpu().numpy())
        index = large.GLIDE_large(ctx, case["degree"], cfg.metric, h_rows, order.cpu().numpy().astype(np.uint32),
                                  d_centroids.cpu().numpy(), seg_start[:case["partitions"]], seg_len[:case["partitions"]])
        state["index"] = index
        if kind == "large_search":
            _large_build(state)
            index.make_resident(1 << 40)
    return state


def _large_build(state):
    cfg = state["config"]
    p_knn, p_refine = pipeline.derive_build_search_params(cfg)
    state["index"].build(IndexParameter(cfg.graph_degree, cfg.knn_degree, cfg.relaxant_factor, cfg.metric), p_knn, p_refine,
                         seed=cfg.seed, nnd=NNDescentParameter(cfg.knn_degree))


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "search":
        ids, dists, _ = state["index"].search(state["params"], state["queries"])
        return dict(ids=ids.view(np.int32), dists=dists)
    if kind == "pipe":
        pipe, params = state["pipe"], state["params"]
        for b in state["batches"]:
            pipe.submit(params, b["q"], b["ids"], b["dists"])
        pipe.drain()
        return [dict(ids=b["ids"], dists=b["dists"]) for b in state["batches"]]
    if kind == "build":
        res = pipeline.build_small(ctx, state["rows"], state["config"])
        return dict(graph=res.index.graph_view(), start_points=res.index.start_point_view(), centroids=res.index.centroid_view(),
                    segment_length=res.h_segment_length.view(np.int32))
    if kind == "large_build":
        _large_build(state)
        return dict(graph=state["index"].graph_view().view(np.int32), start_points=state["index"].start_point_view().view(np.int32))
    if kind == "large_search":
        ids, dists, _ = state["index"].search(state["params"], state["case"]["route_min"], 1.2, state["queries"])
        return dict(ids=ids.view(np.int32), dists=dists)
    ids, dists = api.bruteforce_knn(ctx, state["rows"], state["queries"], state["case"]["top_k"], state["metric"])
    return dict(ids=ids, dists=dists)


def _search_work(case, searches, beam, data_rows):
    """A greedy search expands about `beam` nodes and scores most of each one's neighbours; rows and
    adjacency lists that several searches visit are counted once."""
    expansions = SearchParameter(beam=beam).derive(case["degree"]).max_iterations
    scored = searches * expansions * case["degree"]
    return dict(bytes=4.0 * (min(scored, data_rows) * case["dim"] + min(searches * expansions, data_rows) * case["degree"]),
                flops=3.0 * scored * case["dim"])


def work(case):
    n, dim, kind = case["n"], case["dim"], case["kind"]
    q = case["queries"] * max(1, case["batches"])
    result = 8.0 * q * case["top_k"]
    if kind == "truth":
        return dict(bytes=4.0 * (n + q) * dim + result, flops=2.0 * n * q * dim)
    if kind in ("search", "pipe", "large_search"):
        searches = q * max(1, case["route_min"])
        w = _search_work(case, searches, case["beam"], n)
        return dict(bytes=w["bytes"] + 4.0 * (q + case["partitions"]) * dim + result,
                    flops=w["flops"] + 2.0 * q * case["partitions"] * dim)
    # builds: rows in, graph out; every pair of a partition, one search per row, assignment
    w = _search_work(case, n, 64, n)
    row_bytes = 1.0 if case["uint8"] else 4.0
    return dict(bytes=row_bytes * n * dim + 4.0 * n * (case["degree"] + max(32, case["degree"])),
                flops=w["flops"] + 2.0 * n * (n / case["partitions"]) * dim + 2.0 * n * case["partitions"] * dim)


def tolerance(case):
    # Integer-valued rows: every sum of squares is below 2^24, so distances, and with them ids, are the same in
    # any order of summation. Other rows: the path was compared with itself on rows whose dimensions had been
    # permuted (all sums in another order), and four times the differences seen are allowed: results differed by
    # 5.4e-8 (norm) and 2.4e-7 (one value) with 1e-5 of the ids swapped among near ties; up to 6.8e-3 of a built
    # graph's entries changed where near ties decide an edge. Centroids are fp32 sums over thousands of rows.
    if case["data"].startswith("int_"):
        return "exact"
    if case["kind"] in ("build", "large_build"):
        return dict(rel=1e-5, differ=0.01)
    return dict(rel=2.5e-7, max=1e-6, differ=5e-5)
