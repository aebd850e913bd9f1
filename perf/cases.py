"""Workloads of this framework: searches of an index from one query to a large batch, and the two
ways the neighbor table of an index is made (by a scan of all rows, and by the index's own search).

A program loads its index once and searches it with ever new queries, so the handle of an index
(built here with the library's own builder from fixed rows) is shared by the states of a case and
by the cases that name the same index; what the seed makes is the queries. The cases that make a
table take new rows from every seed. Rows and queries have the distributions of
``octex_b200.synth``, drawn on the GPU.
"""
import collections
import tempfile

import torch

import octex_b200

# ---- the indexes ---------------------------------------------------------------------------------
# Fields of a case that describe its index; the first three name the rows, the rest are parameters
# of the builder.
INDEX_FIELDS = ("data", "rows", "dim", "copies", "blocks", "list_len", "min_cell", "log_buckets",
                "sketch_width", "table_len")

# a million local descriptors of 128 small integers: the default workload of bench.py
DESCRIPTORS = dict(data="descriptor", rows=1_000_000, dim=128, copies=64, blocks=4, list_len=32,
                   min_cell=16, log_buckets=18, sketch_width=64, table_len=64)
# a million unit-norm embeddings of 96 dimensions: needs many start points for a recall of 0.99
EMBEDDINGS = dict(data="embedding", rows=1_000_000, dim=96, copies=64, blocks=4, list_len=32,
                  min_cell=16, log_buckets=18, sketch_width=64, table_len=64)
# global descriptors of 960 dimensions, where the exact rerank and the query's own projections weigh
GLOBALS = dict(data="global", rows=100_003, dim=960, copies=48, blocks=4, list_len=64, min_cell=16,
               log_buckets=16, sketch_width=128, table_len=64)
# the small index of the tests: two blocks per copy, short lists
SMALL = dict(data="mixture", rows=20_000, dim=48, copies=8, blocks=2, list_len=16, min_cell=1,
             log_buckets=12, sketch_width=32, table_len=16)

SEARCH_FIELDS = ("read", "starts", "waves", "rerank", "wave_rerank", "batch", "sketch_rank",
                 "final_rerank")
# the default parameters of Index.search
DEFAULTS = dict(read=32, starts=128, waves=2, rerank=128, wave_rerank=128, batch=10_000,
                sketch_rank=False, final_rerank=32)
# the parameters with which the descriptors reach a recall of 0.99
TUNED = dict(DEFAULTS, read=16, starts=32, waves=1, rerank=128, wave_rerank=384)


def _search(name, index, queries, k, host, params):
    return dict(name=name, do="search", queries=queries, k=k, host=host, **index, **params)


def listed():
    return [
        # one request at a time: an interactive lookup, all latency
        _search("one query", DESCRIPTORS, 1, 10, False, TUNED),
        # a handful of requests gathered by a server, queries and answers in numpy arrays
        _search("17 queries on the host", DESCRIPTORS, 17, 10, True, TUNED),
        # an ordinary batch with nothing tuned: the call with its default parameters
        _search("1000 queries, defaults", DESCRIPTORS, 1_000, 10, False, DEFAULTS),
        # throughput: the 10 000-query batch the framework is quoted on, resident on the GPU ...
        _search("10000 queries", DESCRIPTORS, 10_000, 10, False, TUNED),
        # ... and from and to ordinary host memory
        _search("10000 queries on the host", DESCRIPTORS, 10_000, 10, True, TUNED),
        # a set that is no multiple of the batch size: one whole batch and a ragged rest
        _search("12345 queries, ragged", DESCRIPTORS, 12_345, 10, False, TUNED),
        # embedding search at a recall of 0.99: the heaviest parameters in earnest use, the largest search
        _search("10000 embeddings, heavy", EMBEDDINGS, 10_000, 10, False,
                dict(DEFAULTS, read=32, starts=256, waves=3, rerank=512, wave_rerank=512)),
        # ranking by the int8 sketch with an exact rerank at the end: how indexes are searched whose
        # vectors are far away
        _search("2500 embeddings by sketch", EMBEDDINGS, 2_500, 10, False,
                dict(DEFAULTS, read=16, starts=512, waves=3, sketch_rank=True, final_rerank=32)),
        # wide vectors, a hundred neighbors each: retrieval of candidates for a later stage
        _search("999 global descriptors, k=100", GLOBALS, 999, 100, False,
                dict(DEFAULTS, read=32, starts=128, waves=2, rerank=256, wave_rerank=256)),
        # a small collection with another shape of lattice
        _search("300 queries, small index", SMALL, 300, 10, False,
                dict(DEFAULTS, read=8, starts=32, waves=2)),
        # building: the exact neighbors of every row, what the neighbor table of a new index is made from
        dict(name="neighbors of 200001 rows", do="neighbors", data="descriptor", rows=200_001, dim=128,
             k=64),
        # ... and the table of an index too large for that: its own search over every row, in three passes
        dict(name="searched table of 100001 rows", do="table", data="embedding", rows=100_001, dim=96,
             copies=32, blocks=4, list_len=32, min_cell=8, log_buckets=14, sketch_width=64, table_len=32),
    ]


# ---- drawn cases ---------------------------------------------------------------------------------


def _log_between(rng, low, high):
    """A whole number between the two, spread evenly over its logarithm."""
    return min(high, int(low * (high / low) ** rng.random()))


def _draw_index(rng):
    """An index of any size and dimension the listed ones span (rows x dimension bounded by theirs)."""
    data = rng.choice(("descriptor", "embedding", "global", "mixture"))
    dim = rng.choice((48, 64, 96, 100, 128, 200, 256, 384, 512, 768, 960))
    # rows that do not start on 16-byte boundaries are scanned without the tensor cores when the
    # table is made: small collections only
    most = 40_000 if dim % 8 else min(400_000, 64_000_000 // dim)
    blocks = rng.choice((4, 4, 4, 2, 3))
    return dict(data=data, rows=_log_between(rng, 20_000, most), dim=dim, copies=rng.randint(8, 64),
                blocks=blocks, list_len=rng.choice((16, 32, 64)), min_cell=rng.choice((4, 8, 16)),
                log_buckets=14, sketch_width=rng.choice([w for w in (32, 48, 64, 96, 128) if w <= dim]),
                table_len=rng.choice((16, 32, 64)))


def _draw_search(rng):
    # one in three on the index of the listed cases, the rest on one of its own
    index = dict(DESCRIPTORS) if rng.random() < 0.33 else _draw_index(rng)
    params = dict(DEFAULTS)
    params["read"] = rng.choice((4, 8, 16, 24, 32))
    params["starts"] = rng.choice((16, 24, 32, 64, 96, 128, 192, 256))
    params["waves"] = rng.choice((0, 1, 1, 2, 2, 3))
    params["rerank"] = rng.choice((64, 128, 256, 512))
    params["wave_rerank"] = rng.choice((64, 128, 256, 384, 512))
    params["sketch_rank"] = rng.random() < 0.15
    params["batch"] = rng.choice((10_000, 10_000, 10_000, 4_096, 1_000))
    k = rng.choice((1, 10, 10, 10, 20, 32))
    heavy = params["starts"] * params["waves"] >= 256 or index["dim"] > 256
    queries = _log_between(rng, 1, 2_000 if heavy else 12_000)
    # a few batches at most, as a program would size them
    params["batch"] = max(params["batch"], (queries + 2) // 3)
    return dict(do="search", queries=queries, k=k, host=rng.random() < 0.3, **index, **params)


def draw(rng):
    what = rng.random()
    if what < 0.10:
        dim = rng.choice((64, 96, 128, 200, 256))
        return dict(do="neighbors", data=rng.choice(("descriptor", "embedding", "mixture")),
                    rows=_log_between(rng, 10_000, min(200_000, 25_600_000 // dim)), dim=dim,
                    k=rng.choice((10, 32, 64)))
    if what < 0.20:
        dim = rng.choice((64, 96, 128))
        return dict(do="table", data=rng.choice(("descriptor", "embedding", "mixture")),
                    rows=_log_between(rng, 20_000, 100_000), dim=dim, copies=rng.randint(8, 32), blocks=4,
                    list_len=rng.choice((16, 32)), min_cell=rng.choice((8, 16)), log_buckets=14,
                    sketch_width=rng.choice((32, 48, 64)), table_len=rng.choice((16, 24, 32)))
    return _draw_search(rng)


# ---- rows and queries ----------------------------------------------------------------------------


def _rows(data, count, dim, seed):
    """``count`` rows of a kind of data, float32 on the GPU. What belongs to the kind (centres of its
    clusters, the matrix of the anisotropic one) is the same for every seed."""
    kind = torch.Generator("cuda").manual_seed(4321)
    g = torch.Generator("cuda").manual_seed(int(seed))

    def normal(*shape, of=g):
        return torch.randn(shape, generator=of, device="cuda")

    def pick(centers):
        return centers[torch.randint(len(centers), (count,), generator=g, device="cuda")]

    if data == "descriptor":  # whole numbers 0 .. 255 around 1 024 centres
        centers = torch.rand(1024, dim, generator=kind, device="cuda") * 120.0
        return (pick(centers) + normal(count, dim).abs() * 40.0).clamp_(0.0, 255.0).round_()
    if data == "embedding":  # unit norm, variances decaying as 1 / i
        q, _ = torch.linalg.qr(normal(dim, dim, of=kind))
        scale = torch.arange(1, dim + 1, device="cuda", dtype=torch.float32).rsqrt()
        return torch.nn.functional.normalize((normal(count, dim) * scale) @ q)
    if data == "global":  # non-negative, 256 centres, little noise
        return pick(normal(256, dim, of=kind).abs() * 0.1) + normal(count, dim).abs() * 0.02
    if data == "mixture":  # 64 Gaussian clusters
        return pick(normal(64, dim, of=kind) * 2.0) + normal(count, dim)
    raise ValueError(data)


# the handles a program keeps: the last two indexes that were asked for
_handles = collections.OrderedDict()


def _index(case):
    key = tuple(case[f] for f in INDEX_FIELDS)
    idx = _handles.get(key)
    if idx is None:
        while len(_handles) >= 2:
            _handles.popitem(last=False)
        idx = _handles[key] = _build(_rows(case["data"], case["rows"], case["dim"], 1), case)
    _handles.move_to_end(key)
    return idx


def _build(rows, case, **other):
    params = {f: case[f] for f in INDEX_FIELDS[3:]}
    params.update(pca_dims=min(64, case["dim"]), seed=7, **other)
    with tempfile.TemporaryDirectory(prefix="octex-perf-") as path:
        octex_b200.build_native(rows, path, **params)
        return octex_b200.load(path, placement="replicate", devices=torch.cuda.current_device())


# ---- one pass ------------------------------------------------------------------------------------


def prepare(case, seed):
    if case["do"] == "search":
        queries = _rows(case["data"], case["queries"], case["dim"], 1000 + seed)
        if case["host"]:
            queries = queries.cpu().numpy()
        return dict(do="search", index=_index(case), queries=queries, k=case["k"],
                    params={f: case[f] for f in SEARCH_FIELDS})
    rows = _rows(case["data"], case["rows"], case["dim"], 1000 + seed)
    if case["do"] == "neighbors":
        return dict(do="neighbors", rows=rows.half(), k=case["k"])
    # the index as the builder has it when it comes to the table
    return dict(do="table", index=_build(rows, case, table_len=0), k=case["table_len"])


def run(state):
    if state["do"] == "search":
        return state["index"].search(state["queries"], state["k"], **state["params"])
    if state["do"] == "neighbors":
        return octex_b200.exact_neighbors(state["rows"], state["k"])
    return state["index"].searched_table(state["k"])


# ---- what a pass cannot do without ---------------------------------------------------------------


def work(case):
    n, dim = case["rows"], case["dim"]
    if case["do"] == "neighbors":
        # every pair's product once (it serves both rows), the rows in, ids and distances out
        return dict(bytes=2 * n * dim + 8 * n * case["k"], flops=n * n * dim)
    width, sketch, table = 8 * case["blocks"], case["sketch_width"], case["table_len"]
    if case["do"] == "table":
        # the index in and the table out; per row three passes of the projections, of the sketch
        # distances (all list entries of distinct rows; half the table entries of two, then three waves
        # of 128 starts) and of the exact distances of the 3k/2 + 1 answers kept
        scored = 3 * 0.85 * case["copies"] * case["list_len"] + 0.5 * 5 * 128 * table
        exact = 3 * (table + table // 2 + 1)
        return dict(bytes=n * (2 * dim + sketch + 4 * table),
                    flops=n * (3 * 2 * dim * (width * case["copies"] + sketch) + 2 * sketch * scored + 3 * dim * exact))
    # A search reads at most an array once, however many queries meet a row of it. About 85 of 100
    # list entries are of distinct rows, and half of the table entries of a wave.
    q, waves = case["queries"], case["waves"]
    entries = case["copies"] * min(case["read"], case["list_len"])
    first, later = 0.85 * entries, 0.5 * case["starts"] * table * waves
    exact = case["final_rerank"] if case["sketch_rank"] else (
        min(case["rerank"], first) + waves * min(case["wave_rerank"], 0.5 * case["starts"] * table))
    rows_of = lambda gathered: min(n, q * gathered)  # noqa: E731
    moved = q * dim * 4 + q * case["k"] * 12 + case["copies"] * width * dim * 2
    moved += q * case["copies"] * (16 + 4 * min(case["read"], case["list_len"]))
    moved += rows_of(case["starts"] * waves) * 4 * table
    moved += rows_of(first + later) * sketch + rows_of(exact) * 2 * dim
    flops = 2 * dim * (width * case["copies"] + sketch) + 2 * sketch * (first + later) + 3 * dim * exact
    return dict(bytes=moved, flops=q * flops)


def tolerance(case):
    # Distances are sums in 32 bits. An id may change places with one at the same distance, and a row
    # at a cut of the int8 sketch may fall on either side when a query's coordinates are rounded
    # another way.
    return {"rel": 1e-5, "max": 1e-3, "differ": 1e-3}
