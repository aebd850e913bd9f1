"""The forms a kernel or a call takes by size, against each other and against the inspected run of the
same search (coordinates and codes written out, separate lookup kernel), which test_gpu_parity.py
compares with the CPU checker bit for bit.  Whatever the form, the answer is the same: ids and
distances are compared for equality."""
import numpy as np
import pytest

import octex_b200
from conftest import small_params

pytestmark = pytest.mark.gpu


def make_index(dim, rows=4000, **kw):
    from octex_b200 import build_index, synth
    base = synth.plumbing(rows, dim, seed=0)
    base_kw = dict(pca_dims=min(64, dim), list_len=16, min_cell=2, sketch_width=32, table_len=24)
    base_kw.update(kw)
    arrays, meta = build_index.build_arrays(base, small_params(**base_kw), device="cpu")
    return octex_b200.attach(arrays, meta, borrow=False), meta


def same(a, b):
    return np.array_equal(a[1], b[1]) and np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))


def inspected(idx, queries, k, **kw):
    idx.set_debug(taps=True)
    out = idx.search(queries, k, **kw)
    seg = idx.fetch("seg", np.int32)
    idx.set_debug()
    return out, seg


WRITTEN, SPREAD, BULK, ORDERED = range(4)  # how a batch was projected


def forms(idx):
    """Queries from which on a batch goes in two halves, whether the last one did, how it was projected, in tiles of how many
    queries."""
    return idx.fetch("forms", np.int32).tolist()


def halves_from(idx, queries, **kw):
    idx.search(queries[:1], 10, **kw)
    assert forms(idx)[1] == 0
    return forms(idx)[0]


@pytest.mark.parametrize("blocks,dim", [(1, 48), (2, 100), (3, 96), (4, 98), (4, 64), (4, 200), (5, 64), (6, 130), (8, 64)])
def test_projection_forms(blocks, dim):
    """Lookup in the projection: a lane per block of coordinates with the levels side by side (few
    queries), a lane group per (query, copy). (64 dimensions fit the operand stages, 200 do not, and
    rows of 98 floats do not start on 16-byte boundaries.) An odd number of copies leaves the last tile
    half empty."""
    import torch
    from octex_b200 import synth
    idx, meta = make_index(dim, copies=7, blocks=blocks, pca_dims=min(64, dim))
    kw = dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)
    sizes = (1, 2, 12, 13, 64, 65, 129, 400) + ((9600,) if blocks == 4 else ())
    queries = synth.plumbing(max(sizes), dim, seed=1)
    queries[3, 5] = 3.0e6  # a coordinate for the general decode
    for n in sizes:
        want, seg = inspected(idx, queries[:n], 10, **kw)
        got = idx.search(queries[:n], 10, **kw)
        assert same(got, want), n
        assert np.array_equal(idx.fetch("seg", np.int32), seg), n
        # from rows in the middle of a device array, into new arrays
        q = torch.as_tensor(np.concatenate([queries[-1:], queries[:n]]), device="cuda")[1:]
        d, i = idx.search(q, 10, **kw)
        assert same((d.cpu().numpy(), i.cpu().numpy()), want), n
    idx.close()


@pytest.mark.parametrize("halved", [False, True])
@pytest.mark.parametrize("copies,dim,form", [(63, 64, BULK), (63, 98, BULK), (63, 200, BULK), (63, 320, BULK),
                                             (8, 64, SPREAD), (7, 98, SPREAD), (8, 200, SPREAD), (8, 320, SPREAD)])
def test_projection_of_many_queries(copies, dim, form, halved):
    """A thread per (query, copy) in blocks that go through many tiles, whose operands fit the stages (up to 128
    dimensions) or come in again for every tile, and tiles of few copies spread over the GPU, for whole batches and
    for halves, which share it: as the inspected run, which is neither."""
    import torch
    from octex_b200 import synth
    idx, _ = make_index(dim, rows=3000, copies=copies, blocks=4, pca_dims=64)
    kw = dict(read=8, starts=16, waves=0 if copies > 8 else 1, rerank=32, wave_rerank=32)
    queries = synth.plumbing(6000, dim, seed=1)
    queries[3, 5] = queries[2500, 7] = 3.0e6  # a coordinate for the general decode
    line = halves_from(idx, queries, **kw)
    n = line + 515 if halved else line - 1
    want, seg = inspected(idx, queries[:n], 10, **kw)
    d, i = idx.search(torch.as_tensor(queries[:n], device="cuda"), 10, **kw)
    assert forms(idx)[1:3] == [halved, form]
    assert same((d.cpu().numpy(), i.cpu().numpy()), want)
    assert np.array_equal(idx.fetch("seg", np.int32), seg)
    idx.close()


def test_batches_of_any_size_share_a_plan():
    """A plan made for the largest batch serves smaller ones; searches on several streams and threads
    use its buffers in turn."""
    import threading
    import torch
    from octex_b200 import synth
    idx, meta = make_index(64, copies=8, blocks=4)
    kw = dict(read=8, starts=32, waves=2, rerank=64, wave_rerank=64)
    queries = synth.plumbing(700, 64, seed=1)
    want = idx.search(queries, 10, **kw)
    sizes = (700, 1, 33, 300, 699, 2, 700)
    for n in sizes:
        assert same(idx.search(queries[:n], 10, **kw), (want[0][:n], want[1][:n])), n
        assert idx.fetch("kept_ids", np.int64, (n, -1)).shape[1] == 32
    assert same(idx.search(queries, 10, batch=131, **kw), want)
    q = torch.as_tensor(queries, device="cuda")
    failures = []

    def work(seed):
        rng = np.random.default_rng(seed)
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(40):
                a = int(rng.integers(0, 600))
                n = int(rng.integers(1, 700 - a))
                if rng.random() < 0.3:
                    d, i = idx.search(queries[a:a + n], 10, **kw)
                else:
                    d, i = (t.cpu().numpy() for t in idx.search(q[a:a + n], 10, **kw))
                if not same((d, i), (want[0][a:a + n], want[1][a:a + n])):
                    failures.append((seed, a, n))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    idx.close()


def search_at(idx, queries, ids, dist, m, dim, k, on_device=1, wait=True, stream=0, **kw):
    """The C call on addresses, as a program that has no torch tensors makes it."""
    import ctypes as C
    from octex_b200 import _lib
    p = octex_b200.search_params(**kw)
    fn = _lib.lib().octexB200SearchWait if wait else _lib.lib().octexB200Search
    _lib.check(fn(idx._resources(stream).h, C.byref(p), idx._h, C.c_void_p(queries), C.c_int64(m), C.c_int64(dim),
                  C.c_void_p(ids), C.c_void_p(dist), C.c_int64(k), C.c_int32(on_device)))


def in_place(idx, queries, ids, dist):
    import ctypes as C
    from octex_b200 import _lib
    out = C.c_int32(-1)
    _lib.check(_lib.lib().octexB200SearchInPlace(idx._h, C.c_void_p(queries), C.c_void_p(ids), C.c_void_p(dist),
                                                 C.byref(out)))
    return out.value


def test_arrays_outside_the_index_gpu_are_copied():
    """A device search works in place only on aligned memory of the index's own GPU. Page-locked and
    ordinary host memory given as device arrays, and results off the boundaries of their types, are
    copied, as they were when every search copied. The route is asserted before the search: a kernel
    never gets an address it may not use."""
    import torch
    from octex_b200 import synth
    dim, n, k = 64, 97, 10
    idx, _ = make_index(dim, copies=8, blocks=4)
    kw = dict(read=8, starts=32, waves=1, rerank=64, wave_rerank=64)
    queries = synth.plumbing(n, dim, seed=1)
    want = idx.search(queries, k, **kw)
    q = torch.as_tensor(queries, device="cuda")
    ids, dist = torch.empty((n, k), dtype=torch.int64, device="cuda"), torch.empty((n, k), device="cuda")
    assert in_place(idx, q.data_ptr(), ids.data_ptr(), dist.data_ptr()) == 1
    host = (np.ascontiguousarray(queries), np.zeros((n, k), np.int64), np.zeros((n, k), np.float32))
    addresses = [a.ctypes.data for a in host]
    for at in range(3):  # one of the three elsewhere is enough
        three = [q.data_ptr(), ids.data_ptr(), dist.data_ptr()]
        three[at] = addresses[at]
        assert in_place(idx, *three) == 0
    assert in_place(idx, *addresses) == 0
    search_at(idx, *addresses, n, dim, k, **kw)
    assert same((host[2], host[1]), want)
    pinned = [torch.as_tensor(a).pin_memory() for a in (queries, np.zeros((n, k), np.int64), np.zeros((n, k), np.float32))]
    addresses = [t.data_ptr() for t in pinned]
    assert in_place(idx, *addresses) == 0
    search_at(idx, *addresses, n, dim, k, **kw)
    assert same((pinned[2].numpy(), pinned[1].numpy()), want)
    words = torch.zeros(2 * n * k + 1, dtype=torch.int32, device="cuda")  # ids four bytes off
    off = words.data_ptr() + (4 if words.data_ptr() % 8 == 0 else 0)
    assert in_place(idx, q.data_ptr(), off, dist.data_ptr()) == 0
    search_at(idx, q.data_ptr(), off, dist.data_ptr(), n, dim, k, **kw)
    got = words.cpu().numpy()[1:].tobytes()
    assert same((dist.cpu().numpy(), np.frombuffer(got, np.int64).reshape(n, k)), want)
    idx.close()


def test_queries_on_another_gpu():
    """Torch queries on a GPU the index is not on, with either device current: copied, ordered after
    the stream of the queries' device, results there."""
    import torch
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    from octex_b200 import synth
    idx, _ = make_index(64, copies=8, blocks=4)
    kw = dict(read=8, starts=32, waves=1, rerank=64, wave_rerank=64)
    queries = synth.plumbing(300, 64, seed=1)
    want = idx.search(queries, 10, **kw)
    for current in (0, 1):
        with torch.cuda.device(current):
            q = torch.as_tensor(queries, device="cuda:1")
            for batch in (10000, 70):
                d, i = idx.search(q + 0, 10, batch=batch, **kw)
                assert d.device == i.device == q.device
                assert same((d.cpu().numpy(), i.cpu().numpy()), want)
    idx.close()


def test_captured_searches():
    """The C call that does not wait, captured on a stream of the caller and replayed with other queries:
    arrays used in place and arrays copied in and out (page-locked ones given as device arrays), one batch
    (also after a call that brought a second stream in) and several. use_graph = False, as a capture
    always needed."""
    import torch
    from octex_b200 import synth
    dim, k, n = 64, 10, 300
    idx, _ = make_index(dim, copies=8, blocks=4)
    kw = dict(read=8, starts=32, waves=2, rerank=64, wave_rerank=64)
    queries = synth.plumbing(2 * n, dim, seed=1)
    want = idx.search(queries, k, **kw)
    side = torch.cuda.Stream()
    for batch, pinned in ((1000, False), (1000, True), (130, True), (1000, True), (130, False), (1000, False)):
        q, ids, dist = torch.empty((n, dim)), torch.empty((n, k), dtype=torch.int64), torch.empty((n, k))
        q, ids, dist = (t.pin_memory() if pinned else t.cuda() for t in (q, ids, dist))
        q.copy_(torch.as_tensor(queries[:n]))
        at = (q.data_ptr(), ids.data_ptr(), dist.data_ptr())
        assert in_place(idx, *at) == (0 if pinned else 1)

        def call():
            search_at(idx, *at, n, dim, k, wait=False, stream=side.cuda_stream, batch=batch, use_graph=False, **kw)

        with torch.cuda.stream(side):
            call()  # a plan is made outside of a capture
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            call()
        for a in (0, n, 0):
            q.copy_(torch.as_tensor(queries[a:a + n]))
            ids.fill_(-5)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert same((dist.cpu().numpy(), ids.cpu().numpy()), (want[0][a:a + n], want[1][a:a + n])), (batch, pinned, a)
        del graph
    idx.close()


def test_device_batches_alternate_between_two_streams():
    """Several batches of device queries: the same answers as one batch for whole and ragged counts, after
    work on the caller's stream that makes the queries, before work there that reads the results (the
    C call that does not wait), from several threads."""
    import threading
    import torch
    from octex_b200 import synth
    dim, k = 64, 10
    idx, _ = make_index(dim, copies=8, blocks=4)
    kw = dict(read=8, starts=32, waves=2, rerank=64, wave_rerank=64)
    queries = synth.plumbing(1200, dim, seed=1)
    want = idx.search(queries, k, **kw)
    q = torch.as_tensor(queries, device="cuda")
    for batch in (1, 37, 300, 400, 599, 600, 1199):
        m = min(len(queries), 12 * batch)
        d, i = idx.search(q[:m], k, batch=batch, **kw)
        assert same((d.cpu().numpy(), i.cpu().numpy()), (want[0][:m], want[1][:m])), batch
    failures = []

    def work(seed):
        rng = np.random.default_rng(seed)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            for _ in range(20):
                m, batch = int(rng.integers(2, 1200)), int(rng.integers(100, 700))
                mine = torch.empty((m, dim), device="cuda")
                ids, dist = torch.empty((m, k), dtype=torch.int64, device="cuda"), torch.empty((m, k), device="cuda")
                torch.empty(1 << 24, device="cuda").fill_(1.0)
                mine.copy_(q[:m])
                search_at(idx, mine.data_ptr(), ids.data_ptr(), dist.data_ptr(), m, dim, k, wait=False,
                          stream=side.cuda_stream, batch=batch, **kw)
                mine.zero_()
                got = (dist + 0).cpu().numpy(), (ids + 0).cpu().numpy()
                if not same(got, (want[0][:m], want[1][:m])):
                    failures.append((seed, m, batch))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    idx.close()


@pytest.mark.parametrize("where", ["device", "host"])
def test_resident_after_a_call_of_several_batches(where):
    """A resident search repeats queries of the call before it, also when that call was cut into batches: of
    one of two batches the first `batch`. More than the call had are filled with copies of the first."""
    import torch
    from octex_b200 import synth
    dim, k = 64, 10
    idx, _ = make_index(dim, copies=8, blocks=4)
    kw = dict(read=8, starts=32, waves=2, rerank=64, wave_rerank=64)
    queries = synth.plumbing(500, dim, seed=1)
    want = idx.search(queries, k, **kw)[1]
    q = torch.as_tensor(queries, device="cuda") if where == "device" else queries

    def resident(n):
        idx.search_resident(n, k, batch=300, **kw)
        return idx.fetch("kept_ids", np.int64, (n, -1))[:, :k]

    for total in (500, 301, 333):
        idx.search(q[:total], k, batch=300, **kw)
        assert np.array_equal(resident(300), want[:300]), total
        assert np.array_equal(resident(300), want[:300]), total  # the graph of the batch
        assert np.array_equal(resident(20), want[:20]), total
        assert np.array_equal(idx.search(q[100:400], k, batch=300, **kw)[1] if where == "host" else
                              idx.search(q[100:400], k, batch=300, **kw)[1].cpu().numpy(), want[100:400])
        assert np.array_equal(resident(300), want[100:400]), total
    idx.search(q[:40], k, batch=300, **kw)
    got = resident(50)
    assert np.array_equal(got[:40], want[:40]) and (got[40:] == want[0]).all()
    idx.close()


@pytest.mark.parametrize("dim", [64, 960])
def test_host_arrays_of_any_size(dim):
    """Ordinary host memory on both sides of the sizes at which queries stop being staged and results stop
    being stored through: the answers of the same queries in device memory. (4 000 x 100 results are
    above 4 MB, with 128 entries a query from the last round.)"""
    import torch
    from octex_b200 import synth
    idx, _ = make_index(dim, copies=6, blocks=4, table_len=16)
    kw = dict(read=8, starts=8, waves=1, rerank=128, wave_rerank=64)
    queries = synth.plumbing(9000, dim, seed=1)
    edge = (384 << 10) // (4 * dim)
    for n, k, batch in ((1, 1, 10000), (edge - 1, 10, 10000), (edge, 10, 10000), (edge + 1, 100, 10000), (3 * edge + 5, 10, edge),
                        (3 * edge - 7, 10, edge - 1), (3495, 100, 10000), (3496, 100, 10000), (4000, 100, 10000),
                        (9000, 100, 4000), (8000, 100, 4000)):
        q = queries[:n]
        d, i = idx.search(torch.as_tensor(q, device="cuda"), k, **kw)
        want = d.cpu().numpy(), i.cpu().numpy()
        assert same(idx.search(q, k, batch=batch, **kw), want), (n, k, batch)
        out = np.full((n, k), -7, np.int64), np.full((n, k), -7, np.float32)
        idx.search(q, k, batch=batch, neighbors=out[0], distances=out[1], **kw)
        assert same((out[1], out[0]), want), (n, k, batch)
    idx.close()


def test_results_are_plain_tensors():
    """Queries that need gradients, are a parameter or of a subclass of torch.Tensor: the results are plain
    tensors without history."""
    import torch
    from octex_b200 import synth

    class Named(torch.Tensor):
        pass

    idx, _ = make_index(64, copies=8, blocks=4)
    kw = dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)
    queries = synth.plumbing(5, 64, seed=1)
    want = idx.search(queries, 10, **kw)
    for device in ("cuda", "cpu"):
        plain = torch.as_tensor(queries, device=device)
        for q in (plain.as_subclass(Named), torch.nn.Parameter(plain.clone()), torch.nn.Parameter(plain, requires_grad=False),
                  (plain.clone().requires_grad_() * 1)):
            for t in idx.search(q, 10, **kw):
                assert type(t) is torch.Tensor and not t.requires_grad and t.device == q.device
            d, i = idx.search(q, 10, **kw)
            assert same((d.cpu().numpy(), i.cpu().numpy()), want)
    idx.close()


@pytest.mark.parametrize("copies,dim,n", [(64, 128, 149), (64, 128, 300), (64, 64, 1001), (63, 128, 1184), (64, 128, 1700),
                                          (40, 200, 150), (40, 200, 500), (64, 256, 301)])
def test_projection_tiles_of_fewer_queries(copies, dim, n):
    """The spread form of the projection with the tiles that give every place on the GPU a block: rows that are no
    multiple of them, wide rows where they are split and where not, the line to the bulk form."""
    from octex_b200 import synth
    idx, _ = make_index(dim, rows=3000, copies=copies, blocks=4, pca_dims=64)
    kw = dict(read=8, starts=16, waves=0, rerank=32)
    queries = synth.plumbing(n, dim, seed=8)
    want, seg = inspected(idx, queries, 10, **kw)
    assert same(idx.search(queries, 10, **kw), want)
    halved, form, rows = forms(idx)[1:]
    assert not halved and form in (SPREAD, BULK) and (form == SPREAD or rows == 128), (form, rows)
    assert np.array_equal(idx.fetch("seg", np.int32), seg)
    idx.close()


def test_more_plans_than_words():
    """A plan's arrays are pieces of one block and its give-up word one of 64 of the index: many configurations one
    after the other, each the answer of a handle that knows only this one."""
    from octex_b200 import synth
    idx, _ = make_index(64)
    queries = synth.plumbing(70, 64, seed=3)
    kw = dict(read=8, waves=1, rerank=32, wave_rerank=32)
    got = [idx.search(queries[:1 + s], 5, starts=1 + s, **kw) for s in range(70)]
    for s in (0, 1, 33, 63, 64, 69):
        other, _ = make_index(64)
        assert same(other.search(queries[:1 + s], 5, starts=1 + s, **kw), got[s]), s
        other.close()
    idx.close()


@pytest.mark.parametrize("borrow", [False, True])
def test_table_of_the_same_size_is_written_over(borrow):
    """set_table writes over the index's own table where the size is the same, and never over an array that belongs to
    the caller."""
    import torch
    from octex_b200 import build_index, synth
    base = synth.plumbing(4000, 64, seed=0)
    arrays, meta = build_index.build_arrays(base, small_params(pca_dims=64, list_len=16, min_cell=2, sketch_width=32, table_len=24),
                                            device="cpu")
    queries = synth.plumbing(50, 64, seed=4)
    kw = dict(read=4, starts=16, waves=2, rerank=16, wave_rerank=16)
    table = np.ascontiguousarray(arrays["table"])
    turned = np.ascontiguousarray(np.roll(table, 1, axis=0))  # every row the neighbors of the row before
    mine = torch.as_tensor(table, device="cuda")
    idx = octex_b200.attach(dict(arrays, table=mine) if borrow else arrays, meta, borrow=borrow)
    first = idx.search(queries, 10, **kw)
    idx.set_table(turned)
    second = idx.search(queries, 10, **kw)
    idx.set_table(table)
    assert same(idx.search(queries, 10, **kw), first)
    idx.close()
    assert np.array_equal(mine.cpu().numpy(), table)
    fresh = octex_b200.attach(dict(arrays, table=turned), meta, borrow=False)
    assert same(fresh.search(queries, 10, **kw), second)
    assert not same(first, second)
    fresh.close()


@pytest.mark.parametrize("dim,blocks,kw", [
    (64, 2, dict(read=8, starts=16, waves=2, rerank=32, wave_rerank=32)),
    (98, 2, dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)),             # rows on 8-byte boundaries
    (98, 4, dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)),
    (64, 4, dict(read=16, starts=32, waves=2, rerank=64, wave_rerank=64)),
    (64, 4, dict(read=16, starts=512, waves=0, rerank=32)),                           # nothing but a first round
    (48, 2, dict(read=16, starts=512, waves=1, sketch_rank=True, final_rerank=40)),   # a block a multiprocessor
    (64, 4, dict(read=16, starts=32, waves=1, sketch_rank=True, final_rerank=0)),
])
def test_batches_in_halves(dim, blocks, kw):
    """A batch of more query blocks than the multiprocessors hold goes in two halves on two streams: the answer and
    the segments of the inspected run, which does not, for arrays on the GPU, in ordinary and in page-locked memory (those
    from four million entries on; halves that are staged and halves that are not); one query less than the line and
    batches of odd numbers; searches before and after on another stream."""
    import torch
    from octex_b200 import synth
    copies, table_len = 40 if kw["waves"] == 0 else 6, 32
    idx, _ = make_index(dim, copies=copies, rows=6000, blocks=blocks, table_len=table_len)
    entries = copies * kw["read"] + kw["waves"] * kw["starts"] * table_len
    queries = synth.plumbing((1 << 22) // entries + 2000, dim, seed=5)
    line = halves_from(idx, queries, **kw)
    copied = max(line, ((1 << 22) - 1) // entries + 1)  # and for ordinary memory
    for n in (line - 1, line, line + 1, copied - 1, copied, copied + 999):
        want, seg = inspected(idx, queries[:n], 10, **kw)
        on_gpu = torch.as_tensor(queries[:n], device="cuda")
        d, i = idx.search(on_gpu, 10, **kw)
        assert forms(idx)[1] == (n >= line), n
        assert same((d.cpu().numpy(), i.cpu().numpy()), want), n
        assert np.array_equal(idx.fetch("seg", np.int32), seg), n
        assert same(idx.search(queries[:n], 10, **kw), want), n
        assert forms(idx)[1] == (n >= copied), n
        assert np.array_equal(idx.fetch("seg", np.int32), seg), n
        with torch.cuda.stream(torch.cuda.Stream()):
            d, i = idx.search(on_gpu, 10, **kw)
            torch.cuda.current_stream().synchronize()
        assert same((d.cpu().numpy(), i.cpu().numpy()), want), n
        pinned = torch.as_tensor(queries[:n]).pin_memory()
        got = idx.search(pinned, 10, **kw)
        got = [t.cpu().numpy() if torch.is_tensor(t) else t for t in got]
        assert same(got, want), n
    idx.close()


def test_halves_of_several_threads():
    """Two threads whose batches go in halves at the same time, on one handle and the one stream it has for second halves,
    beside a third thread whose stream is under capture; what that captured gives the same answer afterwards."""
    import threading

    import torch
    from octex_b200 import synth
    dim, k, n = 64, 10, 2800
    idx, _ = make_index(dim, copies=6, blocks=4)
    kw = dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)
    queries = torch.as_tensor(synth.plumbing(n, dim, seed=6), device="cuda")
    whole, _ = inspected(idx, queries.cpu().numpy(), k, **kw)
    line = halves_from(idx, queries, **kw)
    idx.search(queries, k, **kw)
    assert forms(idx)[1] == 1 and n > line + 200
    failures, finished = [], []
    began, captured = threading.Barrier(3, timeout=60), threading.Event()
    ids, dist = torch.empty((n, k), dtype=torch.int64, device="cuda"), torch.empty((n, k), device="cuda")
    graph = torch.cuda.CUDAGraph()

    def search(seed):
        rng = np.random.default_rng(seed)
        with torch.cuda.stream(torch.cuda.Stream()):
            began.wait()
            for _ in range(40):
                a = int(rng.integers(0, n - line))
                m = int(rng.integers(line, n - a + 1))
                d, i = (t.cpu().numpy() for t in idx.search(queries[a:a + m], k, **kw))
                if not same((d, i), (whole[0][a:a + m], whole[1][a:a + m])):
                    failures.append((seed, a, m))
        finished.append(seed)

    def capture():
        side = torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side, capture_error_mode="thread_local"):
            began.wait()
            search_at(idx, queries.data_ptr(), ids.data_ptr(), dist.data_ptr(), n, dim, k, wait=False,
                      stream=side.cuda_stream, **kw)
            captured.wait(60)  # the capture stays open until the searches are through
        finished.append("capture")

    torch.cuda.synchronize()
    threads = [threading.Thread(target=search, args=(s,)) for s in range(2)]
    capturing = threading.Thread(target=capture)
    for t in threads + [capturing]:
        t.start()
    for t in threads:
        t.join()
    captured.set()
    capturing.join()
    assert not failures and len(finished) == 3
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert same((dist.cpu().numpy(), ids.cpu().numpy()), whole)
    del graph
    idx.close()


@pytest.mark.parametrize("blocks", [2, 4])
def test_halves_and_graphs(blocks):
    """A search whose stream is captured keeps to it, and the graph gives the answer of the search in halves, also
    while other searches go in halves between its launches; arrays used in place and arrays copied."""
    import torch
    from octex_b200 import synth
    dim, k, n = 64, 10, 2500
    idx, _ = make_index(dim, copies=6, blocks=blocks)
    kw = dict(read=8, starts=16, waves=1, rerank=32, wave_rerank=32)
    queries = torch.as_tensor(synth.plumbing(n, dim, seed=6))
    want = [t.cpu().numpy() for t in idx.search(queries.cuda(), k, **kw)]
    assert forms(idx)[1] == 1
    side = torch.cuda.Stream()
    for pinned in (False, True):
        q, ids, dist = queries, torch.empty((n, k), dtype=torch.int64), torch.empty((n, k))
        q, ids, dist = (t.pin_memory() if pinned else t.cuda() for t in (q, ids, dist))
        at = (q.data_ptr(), ids.data_ptr(), dist.data_ptr())

        def call():
            search_at(idx, *at, n, dim, k, wait=False, stream=side.cuda_stream, use_graph=False, **kw)

        torch.cuda.synchronize()
        call()
        side.synchronize()
        assert forms(idx)[1] == 1
        assert same((dist.cpu().numpy(), ids.cpu().numpy()), want)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            call()
        assert forms(idx)[1] == 0
        for _ in range(2):
            ids.fill_(-5)
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                graph.replay()
            call()  # in halves, behind the graph
            side.synchronize()
            assert same((dist.cpu().numpy(), ids.cpu().numpy()), want)
            ids.fill_(-5)
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert same((dist.cpu().numpy(), ids.cpu().numpy()), want)
        del graph
    idx.close()


@pytest.mark.parametrize("blocks", [2, 4])
def test_resident_batches_in_halves(blocks):
    """The graph of a large batch holds its halves side by side, as the search before it ran them: replayed, with
    fewer queries than the search had, and again after a search of others."""
    from octex_b200 import synth
    idx, _ = make_index(64, copies=6, blocks=blocks)
    kw = dict(read=8, starts=16, waves=2, rerank=32, wave_rerank=32)
    queries = synth.plumbing(2600, 64, seed=6)
    captured = 0
    for first in (0, 100):
        want = idx.search(queries[first:first + 2500], 10, **kw)[1]
        for n in (2500, 2500, 1301, 40, 2500):
            idx.search_resident(n, **kw)
            if n != captured:  # its graph was just made
                assert forms(idx)[1] == (n >= forms(idx)[0]), n
            captured = n
            assert np.array_equal(idx.fetch("kept_ids", np.int64, (n, -1))[:, :10], want[:n]), n
    idx.close()
