"""The forms a round takes by size, against the CPU checker bit for bit."""
import numpy as np
import pytest

import octex_b200
from conftest import small_params

pytestmark = pytest.mark.gpu


def against_checker(oracle, idx, arrays, meta, queries, k, **kw):
    """Whole runs (nothing kept for inspection) against the checker, given the GPU's coordinates."""
    idx.set_debug(taps=True)
    apart = idx.search(queries, k, **kw)
    y = idx.fetch("y", np.uint16, (len(queries), -1))
    idx.set_debug()
    want_ids, want_dist, _ = oracle.Index(arrays, meta).search(queries, k, y_in=y, **kw)
    for dist, ids in (apart, idx.search(queries, k, **kw)):
        assert np.array_equal(ids, want_ids), (len(queries), kw)
        assert np.array_equal(dist.view(np.uint32), want_dist.view(np.uint32)), (len(queries), kw)


def shapes(idx):
    """Of the last batch's first round and waves: threads of a block, blocks of a multiprocessor, slots of the
    gather's set, words of its bits, candidates in global memory, fp16 rows leave the L2 cache first."""
    return idx.fetch("shapes", np.int32, (2, 6)).tolist()


def whole_batch(threads):
    """The fewest queries whose rounds run blocks of `threads` (128 to 512) where their shared memory asks for those."""
    import torch
    return 512 * torch.cuda.get_device_properties(0).multi_processor_count // threads + 1


def built(path, count, **params):
    """An index of `count` clustered rows of 32 dimensions made on the GPU, with its arrays for the checker and 60 queries."""
    import torch
    from octex_b200 import index_dir
    g = torch.Generator("cuda").manual_seed(5)
    centers = torch.randn(500, 32, generator=g, device="cuda") * 2
    rows = centers[torch.randint(500, (count,), generator=g, device="cuda")] + torch.randn(count, 32, generator=g, device="cuda")
    octex_b200.build_native(rows, str(path), blocks=2, pca_dims=32, min_cell=4, log_buckets=12, sketch_width=32,
                            table_len=64, seed=3, **params)
    idx = octex_b200.load(str(path), placement="replicate", devices=0)
    arrays, meta = index_dir.read_index(str(path))
    return idx, arrays, meta, (rows[::count // 60][:60] + 0.1).cpu().numpy()


@pytest.fixture(scope="module")
def many_rows(tmp_path_factory):
    """700 000 rows: a bit for each takes 21 876 words, more than most hash sets and fewer than the largest."""
    idx, *rest = built(tmp_path_factory.mktemp("many_rows"), 700_000, copies=8, list_len=16)
    yield idx, *rest
    idx.close()


@pytest.fixture(scope="module")
def more_rows(tmp_path_factory):
    """1 400 000 rows: a bit for each takes 43 752 words, more than any hash set, and 171 KB."""
    idx, *rest = built(tmp_path_factory.mktemp("more_rows"), 1_400_000, copies=16, list_len=64)
    yield idx, *rest
    idx.close()


@pytest.mark.parametrize("kw,threads,slots,words", [
    (dict(starts=16, rerank=64, wave_rerank=64), 128, 2048, 0),                   # half full at most
    (dict(starts=64, rerank=64, wave_rerank=64), 256, 5464, 0),                   # three quarters
    (dict(starts=96, rerank=64, wave_rerank=128), 512, 8192, 0),
    (dict(starts=256, rerank=128, wave_rerank=512), 512, 21848, 0),               # candidates in global memory
    (dict(starts=300, rerank=128, wave_rerank=512), 512, 0, 21876),               # bits, two blocks
    (dict(starts=400, rerank=128, wave_rerank=512), 1024, 0, 21876),              # bits, one
    (dict(starts=512, sketch_rank=True, final_rerank=32), 1024, 0, 21876),        # distances over the bits
])
def test_gathered_ids(oracle, many_rows, kw, threads, slots, words):
    """Every form of the set of gathered ids in blocks of the size a whole batch has, and of 1 024 threads."""
    idx, arrays, meta, queries = many_rows
    kw = dict(read=16, waves=2, **kw)
    against_checker(oracle, idx, arrays, meta, queries, 10, **kw)
    want_d, want_i = idx.search(queries, 10, **kw)
    n = len(queries) if threads == 1024 else whole_batch(threads)
    d, i = idx.search(np.resize(queries, (n, queries.shape[1])), 10, **kw)
    assert [shapes(idx)[1][f] for f in (0, 2, 3)] == [threads, slots, words]
    assert np.array_equal(i, np.resize(want_i, i.shape)) and np.array_equal(d, np.resize(want_d, d.shape))


@pytest.mark.parametrize("starts,wave_rerank,words", [
    (256, 128, 0),      # the set leaves two blocks
    (300, 128, 43752),  # it leaves one: bits, below the last step of shared memory
    (512, 512, 0),      # they would need that
])
def test_bits_that_take_more_room(oracle, more_rows, starts, wave_rerank, words):
    idx, arrays, meta, queries = more_rows
    kw = dict(read=64, starts=starts, waves=2, rerank=512, wave_rerank=wave_rerank)
    idx.search(queries, 10, **kw)
    assert shapes(idx)[1][3] == words
    against_checker(oracle, idx, arrays, meta, queries, 10, **kw)


def test_rows_that_leave_the_cache_first(oracle, many_rows, more_rows):
    """With a sketch of 50 MB, a quarter of the L2 cache, but not of 25 MB, nor when the rows are in host memory."""
    kw = dict(read=16, starts=32, waves=2, rerank=100, wave_rerank=65)
    for (idx, arrays, meta, queries), first in ((many_rows, 0), (more_rows, 1)):
        idx.search(queries, 10, **kw)
        assert [shape[5] for shape in shapes(idx)] == [first, first]
        against_checker(oracle, idx, arrays, meta, queries, 10, **kw)
    idx, arrays, meta, queries = more_rows
    far = octex_b200.load(idx.path, placement="replicate", devices=0, vectors_on_host=True)
    got, want = far.search(queries, 10, **kw), idx.search(queries, 10, **kw)
    assert [shape[5] for shape in shapes(far)] == [0, 0]
    assert np.array_equal(got[1], want[1]) and np.array_equal(got[0], want[0])
    far.close()


@pytest.mark.parametrize("spare", [0, 1, 64])
def test_full_set(oracle, more_rows, spare):
    """A wave that gathers as many ids as its set has slots (32 768 of 512 table rows), none twice but for `spare`."""
    idx, arrays, meta, queries = more_rows
    kw = dict(read=64, starts=512, rerank=512, wave_rerank=512)
    starts = idx.search(queries[7:8], 512, waves=0, **kw)[1][0]
    assert starts.min() >= 0 and len(set(starts)) == 512
    ids = np.random.default_rng(3).permutation(len(arrays["vectors"]))[:512 * 64].astype(np.int32)
    ids[len(ids) - spare:] = ids[:spare]
    table = np.array(arrays["table"])
    table[starts] = ids.reshape(512, 64)
    idx.set_table(table)
    try:
        idx.set_debug(stats=True)
        idx.search(queries[7:8], 10, waves=1, **kw)
        assert idx.fetch("stats", np.int64, (1, 8))[0, 5] == 512 * 64 - spare and shapes(idx)[1][2:4] == [32768, 0]
        idx.set_debug()
        against_checker(oracle, idx, dict(arrays, table=table), meta, queries[:20], 10, waves=1, **kw)
    finally:
        idx.set_table(arrays["table"])


@pytest.mark.parametrize("starts,wave_rerank,threads,in_global", [
    (16, 256, 128, 0), (75, 512, 256, 0), (143, 512, 512, 0), (254, 512, 512, 1)])
def test_set_of_kept_ids_takes_no_room(oracle, many_rows, starts, wave_rerank, threads, in_global):
    """300 kept entries and block sizes at which 2 or 4 KB more a block would make fewer and larger blocks, or send
    the candidates to global memory."""
    idx, arrays, meta, queries = many_rows
    kw = dict(read=16, starts=starts, waves=1, rerank=128, wave_rerank=wave_rerank)
    n = whole_batch(threads)
    d, i = idx.search(np.resize(queries, (n, queries.shape[1])), 300, **kw)
    assert shapes(idx)[1][0] == threads and shapes(idx)[1][4] == in_global
    against_checker(oracle, idx, arrays, meta, queries, 300, **kw)
    want_d, want_i = idx.search(queries, 300, **kw)
    assert np.array_equal(i, np.resize(want_i, i.shape)) and np.array_equal(d, np.resize(want_d, d.shape))


@pytest.mark.parametrize("threads", [128, 256, 512, 1024])
@pytest.mark.parametrize("k,kw", [
    (10, dict(starts=16, waves=3, rerank=16, wave_rerank=16)),    # 16 kept, no more new ones than that: by places
    (10, dict(starts=16, waves=3, rerank=64, wave_rerank=128)),   # more new ones: ranked, or selected first
    (100, dict(starts=16, waves=2, rerank=128, wave_rerank=128)), # the first round's 128 sorted, then by places again
    (100, dict(starts=16, waves=2, rerank=100, wave_rerank=300)),
])
def test_merges_at_every_block_size(oracle, many_rows, k, kw, threads):
    idx, arrays, meta, queries = many_rows
    kw = dict(read=16, **kw)
    n = len(queries) if threads == 1024 else whole_batch(threads)
    against_checker(oracle, idx, arrays, meta, queries, k, **kw)
    want_d, want_i = idx.search(queries, k, **kw)
    d, i = idx.search(np.resize(queries, (n, queries.shape[1])), k, **kw)
    assert [shape[0] for shape in shapes(idx)] == [threads, threads]
    assert np.array_equal(i, np.resize(want_i, i.shape)) and np.array_equal(d, np.resize(want_d, d.shape))


@pytest.mark.parametrize("threads,rerank", [(128, 32), (128, 33), (256, 90), (256, 91), (512, 128), (512, 129), (1024, 181), (1024, 182)])
def test_first_merges_around_the_ranking(oracle, more_rows, threads, rerank):
    """Sixteen kept of a first round's reranked rows: ranked up to rerank^2 = 32 threads (128 threads: sorted up to 32),
    selected first beyond."""
    idx, arrays, meta, queries = more_rows
    kw = dict(read=64, starts=16, waves=1, rerank=rerank, wave_rerank=64)
    n = len(queries) if threads == 1024 else whole_batch(threads)
    against_checker(oracle, idx, arrays, meta, queries, 10, **kw)
    want_d, want_i = idx.search(queries, 10, **kw)
    d, i = idx.search(np.resize(queries, (n, queries.shape[1])), 10, **kw)
    assert shapes(idx)[0][0] == threads
    assert np.array_equal(i, np.resize(want_i, i.shape)) and np.array_equal(d, np.resize(want_d, d.shape))


@pytest.mark.parametrize("queries_at_once", [5, 64, 700])
@pytest.mark.parametrize("starts,rerank,wave_rerank", [
    (65, 128, 65),     # a first merge of 128 keys into 65 (128 threads: two chunks of a warp), new ones counted
    (128, 129, 128),   # 129 of 256 places; the most keys whose places are counted
    (130, 257, 129),   # 257 of 512; one more
    (200, 512, 256),   # more than twice the kept ones: selected, then sorted
    (512, 511, 300),
    (512, 512, 512),   # as many as there is room for
])
def test_merges_of_many_keys(oracle, more_rows, starts, rerank, wave_rerank, queries_at_once):
    """Merges whose keys the network sorts: sizes around its powers of two, blocks of few and of many threads."""
    idx, arrays, meta, queries = more_rows
    kw = dict(read=64, starts=starts, waves=2, rerank=rerank, wave_rerank=wave_rerank)
    against_checker(oracle, idx, arrays, meta, queries, 32, **kw)
    want_d, want_i = idx.search(queries, starts, **kw)
    d, i = idx.search(np.resize(queries, (queries_at_once, queries.shape[1])), starts, **kw)
    assert np.array_equal(i, np.resize(want_i, i.shape)) and np.array_equal(d, np.resize(want_d, d.shape))


@pytest.mark.parametrize("starts,sketch_rank", [(16, False), (128, False), (129, False), (16, True), (32, True), (33, True)])
def test_short_waves(oracle, more_rows, starts, sketch_rank):
    """Waves of few queries and few entries have a form of their own: one query, the most it takes (16 384 entries in all) and
    one more, on both sides of the most entries a query (128 start points of 64 neighbors, 32 by sketch distance), give
    what the same queries give in a large batch, which is the checker's answer."""
    idx, arrays, meta, queries = more_rows
    kw = dict(read=64, starts=starts, waves=3, rerank=64, wave_rerank=64, sketch_rank=sketch_rank, final_rerank=32)
    most = 16384 // (64 * starts)
    if not sketch_rank:
        against_checker(oracle, idx, arrays, meta, queries[:most], 16, **kw)
    many = np.resize(queries, (200, queries.shape[1]))
    want_d, want_i = idx.search(many, 16, **kw)
    assert shapes(idx)[1][0] < 1024
    for n in (1, most, most + 1):
        d, i = idx.search(many[:n], 16, **kw)
        assert np.array_equal(i, want_i[:n]) and np.array_equal(d.view(np.uint32), want_d[:n].view(np.uint32)), n


def test_plans_of_several_indexes(many_rows, more_rows):
    """Two indexes searched in turn, each with a plan of its own size."""
    (one, _, _, queries), (other, _, _, others) = many_rows, more_rows
    large, small = dict(read=16, starts=256, waves=1, wave_rerank=512), dict(read=16, starts=16, waves=1, wave_rerank=16)
    want = one.search(queries, 10, **large), other.search(others, 10, **small)
    for _ in range(2):
        for got, ref in ((one.search(queries, 10, **large), want[0]), (other.search(others, 10, **small), want[1])):
            assert np.array_equal(got[1], ref[1]) and np.array_equal(got[0], ref[0])


@pytest.mark.parametrize("rows", [511, 512, 513, 8191, 8193])
def test_rows_around_a_word_of_bits(oracle, rows):
    """Ids up to the last bit of the last word, where the set would have 256 to 4 096 slots."""
    from octex_b200 import build_index, synth
    arrays, meta = build_index.build_arrays(synth.plumbing(rows, 32, seed=0), small_params(copies=4, table_len=24), device="cpu")
    idx = octex_b200.attach(arrays, meta, borrow=False)
    queries = synth.plumbing(50, 32, seed=1)
    for kw in (dict(read=16, starts=12, waves=2, rerank=48, wave_rerank=32), dict(read=4, starts=100, waves=1, rerank=16, wave_rerank=256)):
        against_checker(oracle, idx, arrays, meta, queries, 7, **kw)
    idx.close()


@pytest.mark.parametrize("distinct", [1, 3, 40, 4000])
def test_selection_among_equal_distances(oracle, distinct):
    """Rows that repeat: fewer candidates than are selected, or a few equal ones at the cut."""
    from octex_b200 import build_index, synth
    rng = np.random.default_rng(2)
    base = synth.plumbing(distinct, 48, seed=0)[rng.integers(0, distinct, 4000)]
    arrays, meta = build_index.build_arrays(base, small_params(table_len=32), device="cpu")
    idx = octex_b200.attach(arrays, meta, borrow=False)
    queries = synth.plumbing(40, 48, seed=1)
    for kw in (dict(read=16, starts=64, waves=2, rerank=40, wave_rerank=200), dict(read=16, starts=64, waves=1, sketch_rank=True)):
        against_checker(oracle, idx, arrays, meta, queries, 10, **kw)
    idx.close()


@pytest.mark.parametrize("threads", [128, 1024])
@pytest.mark.parametrize("near", [40, 200])
@pytest.mark.parametrize("members", [1, 127, 128, 129, 300])
def test_members_of_the_bin_at_the_cut(oracle, members, near, threads):
    """A wave over table rows made by hand: `near` ids of equal rows, `members` of others, the rest of a third kind, and
    the cut of the selection inside the second kind: up to 128 are ranked aside, for more the threshold is found
    digit by digit. Blocks of 128 threads select in the merge too where more than 256 keys meet (200 near
    ones and 127 members or more), 65 of them, all at the same distance."""
    from octex_b200 import build_index, synth
    rng = np.random.default_rng(2)
    base = synth.plumbing(3000, 48, seed=0)
    kinds = [np.arange(i, 2700, 3) for i in range(3)]
    for i in range(3):
        base[kinds[i]] = base[2700 + i]
    query = (base[:1] + 0.05).astype(np.float32)
    arrays, meta = build_index.build_arrays(base, small_params(table_len=32), device="cpu")
    sketched = (query - arrays["mean"]).astype(np.float64) @ np.asarray(arrays["sketch_basis"], np.float64).reshape(48, -1)
    apart = ((arrays["sketch"] * np.asarray(arrays["sketch_scale"], np.float64) - sketched) ** 2).sum(1)
    kinds.sort(key=lambda of: apart[of[0]])
    bits = np.float32([apart[of[0]] for of in kinds]).view(np.uint32).astype(np.int64)
    shift = max(int(bits[2] - bits[0]).bit_length() - 8, 0)
    assert 1 < (bits[1] - bits[0]) >> shift < ((bits[2] - bits[0]) >> shift) - 1  # bins of their own

    kw = dict(read=16, starts=16, rerank=64, wave_rerank=near + (members + 1) // 2)
    idx = octex_b200.attach(arrays, meta, borrow=False)
    starts = idx.search(query, 65, waves=0, **kw)[1][0, :16]  # 65: more than the first round finds or reranks
    assert starts.min() >= 0
    ids = np.concatenate([rng.permutation(of)[:count] for of, count in zip(kinds, (near, members, 512 - near - members))])
    table = np.array(arrays["table"])
    table[starts] = rng.permutation(ids).astype(np.int32).reshape(16, 32)
    idx.set_table(table)
    n = 3 if threads == 1024 else whole_batch(threads)
    idx.set_debug(stats=True)
    idx.search(np.repeat(query, n, axis=0), 65, waves=1, **kw)
    assert shapes(idx)[1][0] == threads and (idx.fetch("stats", np.int64, (n, 8))[:, 5] == 512).all()
    idx.set_debug()
    against_checker(oracle, idx, dict(arrays, table=table), meta, np.repeat(query, n, axis=0), 65, waves=1, **kw)
    idx.close()


def sketch_distances(codes, scale, qs):
    """fp32 sketch distances [..., rows] of int8 codes [..., rows, width] to queries [..., width], bit for bit: chunks of
    eight codes, two fused multiply-adds a code, then a butterfly over the next power of two of them. float64 has every
    product and sum before a rounding exactly, but for an addition that is rounded twice about once in 2^29."""
    t = (codes.astype(np.float64) * scale.astype(np.float64) - qs.astype(np.float64)[..., None, :]).astype(np.float32).astype(np.float64)
    part = np.zeros(t.shape[:-1] + (t.shape[-1] // 8,), np.float32)
    for i in range(8):
        part = (t[..., i::8] ** 2 + part).astype(np.float32)
    lanes = 1
    while lanes < part.shape[-1]:
        lanes *= 2
    part = np.concatenate([part, np.zeros(part.shape[:-1] + (lanes - part.shape[-1],), np.float32)], -1)
    while lanes > 1:
        part = part[..., 0::2] + part[..., 1::2]
        lanes //= 2
    return part[..., 0]


@pytest.mark.parametrize("width", [16, 32, 48, 64, 80, 128, 144, 256, 320])
def test_sketch_distances_of_waves(width):
    """The fp32 sketch distances a wave and a first round give, at every number of lanes a row takes and with lanes past
    the last chunk."""
    from octex_b200 import build_index, synth
    base = synth.plumbing(3000, 320, seed=0)
    arrays, meta = build_index.build_arrays(base, small_params(pca_dims=64, list_len=16, min_cell=2, sketch_width=width, table_len=24),
                                            device="cpu")
    idx = octex_b200.attach(arrays, meta, borrow=False)
    queries = synth.plumbing(40, 320, seed=9)
    kw = dict(read=4, starts=64, sketch_rank=True, final_rerank=0)
    codes = arrays["sketch"].reshape(3000, width)
    for waves in (0, 2):
        d, ids = idx.search(queries, 64, waves=waves, **kw)
        qs = idx.fetch("qs", np.float32).reshape(-1, width)[:40]
        live = ids >= 0
        assert live.sum() > 400  # (the lists of a first round hold about twenty rows a query)
        assert np.array_equal(sketch_distances(codes[ids], arrays["sketch_scale"], qs)[live], d[live]), (waves, width)
    idx.close()


@pytest.mark.parametrize("starts,table_len,queries", [(16, 24, 3), (64, 24, 40), (200, 32, 700), (512, 32, 2), (512, 32, 160),
                                                      (700, 32, 20)])
def test_kept_lists_by_sketch(starts, table_len, queries):
    """Waves that rank by sketch distance: a full kept list lets only nearer candidates through, which a selection
    goes through where they are more than the list takes. Against the rule itself from the first round's candidates
    on: a wave expands the first kept rows that none did before, and the nearest of all stay; blocks of every size,
    fewer candidates than a step of the block's threads and several steps of them."""
    from octex_b200 import build_index, synth
    rows, width = 6000, 32
    base = synth.plumbing(rows, 64, seed=0)
    arrays, meta = build_index.build_arrays(base, small_params(pca_dims=64, list_len=64, min_cell=2, sketch_width=width,
                                                               table_len=table_len), device="cpu")
    idx = octex_b200.attach(arrays, meta, borrow=False)
    q = synth.plumbing(queries, 64, seed=7)
    kw = dict(read=64, starts=starts, waves=3, sketch_rank=True, final_rerank=0)
    d, ids = idx.search(q, starts, **kw)
    idx.set_debug(taps=True)
    idx.search(q, starts, **kw)
    qs = idx.fetch("qs", np.float32).reshape(-1, width)
    n1, cand = idx.fetch("n1", np.int32), idx.fetch("cand1", np.int32)
    cand = cand.reshape(len(n1), -1)
    idx.set_debug()
    codes, scale, table = arrays["sketch"].reshape(rows, width), arrays["sketch_scale"], arrays["table"].reshape(rows, -1)
    for i in range(0, queries, max(1, queries // 20)):
        dist = sketch_distances(codes, scale, qs[i])
        seen, done = set(cand[i, :n1[i]].tolist()), set()
        for _ in range(3):
            kept = sorted(seen, key=lambda r: (dist[r], r))[:starts]
            new = [r for r in kept if r not in done][:starts]
            done |= set(new)
            seen = set(kept) | (set(table[new].ravel().tolist()) - {-1})
        kept = sorted(seen, key=lambda r: (dist[r], r))[:starts]
        assert ids[i, :len(kept)].tolist() == kept, i
        assert np.array_equal(d[i, :len(kept)], dist[kept])
    idx.close()
