"""Calls at the limits of their resources: little free device memory, several host threads,
buffers left by larger calls, candidate ranges near the shared-memory limit."""
import contextlib
import ctypes as C
import threading

import numpy as np
import pytest

from hdgrid_b200 import datasets
from tests.helpers import build_gpu

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def only_free(n_bytes: int):
    """Takes device memory until n_bytes of it (give or take 2 MB) are free."""
    import torch
    rt = C.CDLL("libcudart.so.12")  # (torch's allocator rounds small requests up)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    try:
        for step in (64 * MB, 2 * MB):
            while (over := torch.cuda.mem_get_info()[0] - n_bytes) >= step:
                p = C.c_void_p()
                if rt.cudaMalloc(C.byref(p), C.c_size_t(over // step * step)) != 0:
                    rt.cudaGetLastError()
                    break
                held.append(p)
        yield
    finally:
        torch.cuda.synchronize()
        for p in held:
            rt.cudaFree(p)


def _in_threads(*calls):
    """Runs the calls at the same time, each in a thread of its own; their exceptions."""
    errors = []

    def run(f):
        try:
            f()
        except Exception as e:  # noqa: BLE001 (reported to the test)
            errors.append(e)

    ts = [threading.Thread(target=run, args=(f,)) for f in calls]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    return errors


def _range_ws(n, q, l=4, d=32, m=32, **conf):
    """Points with l integer labels below 1,000 and range filters: half of every dim, or a fiftieth of the one."""
    rng = np.random.default_rng(n + q)
    lab = rng.integers(0, 1000, (n, l)).astype(np.float32)
    lo = rng.integers(0, 500, (q, l)).astype(np.float32)
    box = np.stack([lo, lo + (500 if l > 1 else 20)], axis=2).reshape(q, 2 * l).copy()
    c = dict(clusters=8, sub_clusters=8, pq_dim=m, max_grids=256, filter_dim=2, n_list=8, sub_lists=64, exps0=4, topk=10)
    c.update(conf)
    return dict(base=rng.standard_normal((n, d), dtype=np.float32), labels=lab,
                queries=rng.standard_normal((q, d), dtype=np.float32), query_labels=box,
                hdgrid_conf=datasets.hdgrid_conf(**c),
                filter_conf=f"l = {l}\n" + "".join(f"filter{i}:\n\ttype = 3\n" for i in range(l)), k=int(c["topk"]))


def _io(ws, base, k, cuda, q0=0, q1=None):
    """The queries [q0, q1) of a workload as call arguments: (distances, ids, query input, query output)."""
    import torch
    import hdgrid_b200 as hg
    q = torch.from_numpy(ws["queries"][q0:q1].copy()).to(cuda)
    ql = torch.from_numpy(ws["query_labels"][q0:q1].copy()).to(cuda)
    d = torch.full((q.shape[0], k), -1.0, device=cuda)
    i = torch.full((q.shape[0], k), 7, dtype=torch.int64, device=cuda)
    return d, i, hg.query_input_t(base, q, ql), hg.query_output_t(d, i)


# batches whose kernels ask for different amounts of shared memory, from two threads on two streams
@pytest.mark.parametrize("what", ["query", "bruteforce", "bruteforce_batch", "pq_adc"])
def test_threads_with_different_sizes(cuda, what):
    import torch
    import hdgrid_b200 as hg
    rng = np.random.default_rng(4)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    calls, outs = [], []
    if what == "query":  # subspaces of 16 dims: table slices of 34 KB for one query, 135 KB for 5,000
        ws = _range_ws(2000, 5000, d=512)
        idx, base, _ = build_gpu(ws, cuda)
        for n in (1, 5000):
            d, i, qin, qout = _io(ws, base, 10, cuda, 0, n)
            outs.append((d, i))
            calls.append(lambda st, a=qin, b=qout: idx.query(a, b, stream=st))
        repeat = 300
    elif what == "pq_adc":
        for m in (8, 64):
            codes = torch.from_numpy(rng.integers(0, 256, (m, 5000), dtype=np.uint8)).to(cuda)
            lut = torch.rand((4, m, 256), device=cuda)
            d = torch.zeros((4, 5000), device=cuda)
            outs.append((d,))
            calls.append(lambda st, a=codes, b=lut, c=d, m=m: hg.pq_adc(a, 5000, b, 4, m, 256, None, 5000, c, stream=st))
        repeat = 2000
    else:
        q, n = (4, 2000) if what == "bruteforce" else (64, 190000)
        for dim, l, k in ((16, 1, 5), (96, 5, 200)):
            x = [torch.randn((n, dim), device=cuda), torch.rand((n, l), device=cuda), torch.randn((q, dim), device=cuda),
                 torch.tensor([0.0, 0.7] * l, device=cuda).repeat(q, 1)]
            d = torch.zeros((q, k), device=cuda)
            i = torch.zeros((q, k), dtype=torch.int64, device=cuda)
            outs.append((d, i))
            calls.append(lambda st, x=x, k=k, d=d, i=i: hg.bruteforce_knn(*x, k, d, i, stream=st))
        repeat = 2000 if what == "bruteforce" else 200
    torch.cuda.synchronize()
    want = []
    for c, o, st in zip(calls, outs, streams):
        c(st)
        torch.cuda.synchronize()
        want.append([x.clone() for x in o])

    done = threading.Event()

    def loop(c, st, first):
        try:
            n = 0
            while not done.is_set() if first else n < repeat:  # the first for as long as the second
                c(st)
                n += 1
                if n % 64 == 0:
                    st.synchronize()
            st.synchronize()
        finally:
            done.set()

    errors = _in_threads(*(lambda a=a: loop(*a) for a in zip(calls, streams, (True, False))))
    assert not errors, errors[0]
    for w, o in zip(want, outs):
        assert all(torch.equal(a, b) for a, b in zip(w, o))


def test_estimate_pass_after_a_larger_batch(cuda):
    """The candidate rows of a larger batch hold the memory: the entries of the estimate pass go
    into the part of them that a smaller batch leaves unused."""
    import torch
    ws = datasets.config4(scale=0.04, n_queries=1500, clusters=16, sub_clusters=8, n_list=16, sub_lists=100, exps0=8,
                          max_grids=16384, pq_dim=32)
    idx, base, _ = build_gpu(ws, cuda)
    a, b = _io(ws, base, 100, cuda), _io(ws, base, 100, cuda, 0, 900)
    idx.set_param("BREAK_DOWN", 1)
    idx.query(b[2], b[3])
    assert "estimate" in idx.stage_times()
    want = b[0].clone(), b[1].clone()
    idx, base, _ = build_gpu(ws, cuda)  # (new buffers)
    idx.set_param("BREAK_DOWN", 1)
    idx.set_param("EXPS0", 4096)  # budgets of most of the candidates: no estimate pass
    idx.query(a[2], a[3])
    assert "estimate" not in idx.stage_times()
    idx.set_param("EXPS0", 8)
    with only_free(2 * MB):
        idx.query(b[2], b[3])
        stages = idx.stage_times()
        torch.cuda.synchronize()
    assert "estimate" in stages, stages
    assert torch.equal(b[0], want[0]) and torch.equal(b[1], want[1])


def test_optional_buffers_make_room(cuda):
    """A batch whose rows need the memory of the decoded vectors and the rank planes gets it."""
    import torch
    n, q = 400_000, 600
    ws = _range_ws(n, q, d=128, exps0=2)
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.query(qin, qout)
    torch.cuda.synchronize()
    want = d.clone(), i.clone()
    cands, sel = idx.last_query_stats()["coarse_total"], int(np.frombuffer(idx.debug_fetch("sel_off").tobytes(), np.uint64)[q])
    del idx, qin, qout
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.reserve(q)
    rows = 8 * cands + 4 * sel + (sel // 4096 + q + 1) * 80
    optional = idx.info()["device_bytes"]
    with only_free(rows - 16 * MB):  # (the planes' 64 bytes a point are 25 MB, the decoded vectors 109 MB)
        idx.query(qin, qout)
        torch.cuda.synchronize()
    assert idx.info()["device_bytes"] < optional
    assert torch.equal(d, want[0]) and torch.equal(i, want[1])


def test_room_made_while_another_thread_queries(cuda):
    """The optional buffers go while calls of another stream, captured and plain, are on their way."""
    import torch
    n, q = 400_000, 600
    ws = _range_ws(n, q, d=128, exps0=2)
    idx, base, _ = build_gpu(ws, cuda)
    big, small = _io(ws, base, 10, cuda), _io(ws, base, 10, cuda, 0, 20)
    side = torch.cuda.Stream()
    for graph in (0, 1):
        idx.set_param("QUERY_GRAPH", graph)
        for _ in range(2):
            idx.query(small[2], small[3], stream=side)
    idx.status()
    torch.cuda.synchronize()
    want = small[0].clone(), small[1].clone()
    idx.reserve(q)
    before = idx.info()["device_bytes"]
    done = threading.Event()

    def loop():
        n_calls = 0
        while not done.is_set() or n_calls < 20:
            idx.query(small[2], small[3], stream=side)
            n_calls += 1
        idx.status()
        side.synchronize()

    def large():
        try:
            idx.query(big[2], big[3])
            torch.cuda.default_stream().synchronize()  # (a device-wide wait would break the other's capture)
        finally:
            done.set()

    # the rows of 600 queries take about 1.3 GB: the decoded vectors, then the planes make room for them
    with only_free(1200 * MB):
        errors = _in_threads(loop, large)
        torch.cuda.synchronize()
    assert not errors, errors[0]
    assert idx.info()["device_bytes"] < before
    assert torch.equal(small[0], want[0]) and torch.equal(small[1], want[1])


def test_device_bytes_counts_every_index_array(cuda):
    import torch
    n = 1_000_000
    ws = _range_ws(n, 8, d=128)
    torch.cuda.synchronize()
    base = torch.from_numpy(ws["base"]).to(cuda)
    labels = torch.from_numpy(ws["labels"]).to(cuda)
    import hdgrid_b200 as hg
    idx = hg.SuperGridIndex.from_text(ws["hdgrid_conf"], ws["filter_conf"])
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    idx.build(hg.build_input_t(base, labels))
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    assert abs(idx.info()["device_bytes"] - used) < 32 * MB, (idx.info()["device_bytes"], used)


def test_ranks_tested_without_planes(cuda, tmp_path):
    """An index loaded with no room for the rank planes still rejects candidates by their packed
    ranks before it reads labels."""
    import torch
    import hdgrid_b200 as hg
    n, q = 2_000_000, 2
    ws = _range_ws(n, q, exps0=1)
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.query(qin, qout)
    torch.cuda.synchronize()
    want = d.clone(), i.clone()
    path = str(tmp_path / "index.hdg")
    idx.save(path)
    del idx
    with only_free(n * (64 + 32) + 24 * MB):  # arena and code rows; the planes are another 64 a point
        idx = hg.SuperGridIndex.load(path)
        idx.query(qin, qout)
        torch.cuda.synchronize()
    total = idx.last_query_stats()["coarse_total"]
    read = np.frombuffer(idx.debug_fetch("labels_read").tobytes(), np.uint32)[:q].astype(np.int64).sum()
    tested = np.frombuffer(idx.debug_fetch("ranks_read").tobytes(), np.uint32)[:q].astype(np.int64).sum()
    assert torch.equal(d, want[0]) and torch.equal(i, want[1])
    assert tested == total and read < total // 2, (tested, read, total)


def test_estimate_pass_many_ranges(cuda):
    """2,048 lists in three parts each: 6,144 ranges per query."""
    import torch
    ws = datasets.config4(scale=0.04, n_queries=129, clusters=64, sub_clusters=32, n_list=64, sub_lists=2048, exps0=2,
                          max_grids=1024, pq_dim=32, topk=10, is_split=1, n_split=3)
    ws["query_labels"][:, 0::2] = 0
    ws["query_labels"][:, 1::2] = 1_000_000
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.set_param("BREAK_DOWN", 1)
    idx.query(qin, qout)
    assert "estimate" in idx.stage_times()
    want = d.clone(), i.clone()
    idx.set_param("QUERY_GRAPH", 1)  # the replay scans every candidate
    idx.query(qin, qout)
    d.fill_(-1.0)
    idx.query(qin, qout)
    idx.status()
    torch.cuda.synchronize()
    assert torch.equal(d, want[0]) and torch.equal(i, want[1])


def test_scan_chunk_is_the_largest_item(cuda):
    """SCAN_CHUNK (the autotuner's choice, from one batch) bounds the scan items: a smaller batch
    keeps the items its own size asks for."""
    import torch
    ws = _range_ws(200_000, 100)
    idx, base, _ = build_gpu(ws, cuda)

    def items(q, chunk):
        idx.set_param("SCAN_CHUNK", chunk)
        d, i, qin, qout = _io(ws, base, 10, cuda, 0, q)
        idx.query(qin, qout)
        torch.cuda.synchronize()
        return int(np.frombuffer(idx.debug_fetch("item_off").tobytes(), np.uint32)[q]), d, i

    auto = items(1, 0)
    for chunk in (8192, 65536):
        fixed = items(1, chunk)
        assert fixed[0] == auto[0]
        assert torch.equal(fixed[1], auto[1]) and torch.equal(fixed[2], auto[2])
    assert items(100, 4096)[0] > items(100, 65536)[0]


def test_small_batch_with_little_memory(cuda):
    """A small batch whose rows would be taken for every (query, point) pair runs with the memory
    that its candidates need."""
    import torch
    n, q = 2_000_000, 8
    ws = _range_ws(n, q, l=1)
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.query(qin, qout)
    torch.cuda.synchronize()
    want = d.clone(), i.clone()
    assert idx.last_query_stats()["coarse_total"] < n * q // 8
    side = torch.cuda.Stream()
    with only_free(48 * MB):  # 192 MB for every pair
        idx.query(qin, qout, stream=side)
        torch.cuda.synchronize()
    assert torch.equal(d, want[0]) and torch.equal(i, want[1])


@pytest.mark.parametrize("q,k,n,d", [(64, 100, 190000, 96), (4500, 256, 2000, 16), (1, 10, 100000, 64)])
def test_bruteforce_with_little_memory(cuda, q, k, n, d):
    import torch
    import hdgrid_b200 as hg
    g = torch.Generator(device="cuda").manual_seed(q)
    x = [torch.randn((n, d), device=cuda, generator=g), torch.rand((n, 2), device=cuda, generator=g),
         torch.randn((q, d), device=cuda, generator=g), torch.tensor([0.0, 0.7] * 2, device=cuda).repeat(q, 1)]
    out = []
    for free in (None, 2 * MB):
        dist = torch.full((q, k), -1.0, device=cuda)
        ids = torch.full((q, k), 7, dtype=torch.int64, device=cuda)
        with contextlib.nullcontext() if free is None else only_free(free):
            hg.bruteforce_knn(*x, k, dist, ids)
            torch.cuda.synchronize()
        out.append((dist, ids))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("scale", [1e6, 1e-7])
def test_no_estimate_pass_of_a_useless_scale(cuda, scale):
    """PQ approximations that FP16 cannot hold bound nothing: they are not kept and a batch goes
    straight to the full scan."""
    import torch
    ws = datasets.config4(scale=0.04, n_queries=1500, clusters=16, sub_clusters=8, n_list=16, sub_lists=100, exps0=8,
                          max_grids=16384, pq_dim=32)
    ws["base"] *= np.float32(scale)
    ws["queries"] *= np.float32(scale)
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 100, cuda)
    idx.set_param("BREAK_DOWN", 1)
    idx.query(qin, qout)
    idx.query(qin, qout)
    assert "estimate" not in idx.stage_times()


@pytest.mark.parametrize("entries", [2, 600])
def test_recover_filters_returns_with_its_result(cuda, entries):
    import torch
    import hdgrid_b200 as hg
    conf = "l = 1\nfilter0:\n\ttype = 1\n\tinterval_map = [" + ", ".join(str(i) for i in range(entries)) + "]\n"
    ql = torch.ones((100, 1), device=cuda)
    out = torch.empty((100, 2), device=cuda)
    a = torch.randn((8192, 8192), device=cuda)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(20):
            a @ a
    hg.recover_filters(conf, ql, out, stream=side)
    assert side.query()  # the stream's work, the result with it, has ended
    want = out.clone()
    if entries > 512:
        return
    out.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):  # nothing to wait for
        hg.recover_filters(conf, ql, out, stream=side)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_build_frees_what_its_upload_does_not_need(cuda):
    """Beside the index the upload needs the pool-ordered arrays only: by-id codes, lists, cells
    and Morton codes (36 bytes a point here) are gone by then."""
    import torch
    import hdgrid_b200 as hg
    n = 8_000_000
    ws = _range_ws(1000, 8, d=16, m=16)
    base = torch.randn((n, 16), device=cuda)
    labels = torch.randint(0, 1000, (n, 4), device=cuda).float()
    torch.cuda.synchronize()
    idx = hg.SuperGridIndex.from_text(ws["hdgrid_conf"], ws["filter_conf"])
    # at the upload: code rows, labels, ids, codes, the arena of 48 a point
    with only_free(n * 100 + 48 * MB):
        idx.build(hg.build_input_t(base, labels))
        torch.cuda.synchronize()
    assert idx.info()["n"] == n


def test_rebuild(cuda, tmp_path):
    """A refused build leaves the index as it was; a new one ends the old one's captured graphs; one
    without room for its arrays leaves no index."""
    import torch
    import hdgrid_b200 as hg
    ws = _range_ws(20_000, 50)
    idx, base, labels = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.query(qin, qout)
    torch.cuda.synchronize()
    want, info = (d.clone(), i.clone()), idx.info()
    with pytest.raises(hg.HDGError):
        idx.build(hg.build_input_t(base, -1.0 - labels))
    assert idx.info() == info
    idx.save(str(tmp_path / "index.hdg"))
    again = hg.SuperGridIndex.load(str(tmp_path / "index.hdg"))
    for x in (idx, again):
        d.fill_(-1.0)
        x.query(qin, qout)
        torch.cuda.synchronize()
        assert torch.equal(d, want[0]) and torch.equal(i, want[1])
    idx.set_param("QUERY_GRAPH", 1)
    for _ in range(3):
        idx.query(qin, qout)
    idx.status()
    other = base.flip(0).contiguous()
    fresh = hg.SuperGridIndex.from_text(ws["hdgrid_conf"], ws["filter_conf"])
    fresh.build(hg.build_input_t(other, labels))
    base.copy_(other)  # the same addresses, other vectors
    fresh.query(qin, qout)
    torch.cuda.synchronize()
    want = d.clone(), i.clone()
    idx.build(hg.build_input_t(base, labels))
    for _ in range(3):
        d.fill_(-1.0)
        idx.query(qin, qout)
        idx.status()
        torch.cuda.synchronize()
        assert torch.equal(d, want[0]) and torch.equal(i, want[1])
    n = 8_000_000
    big = hg.build_input_t(torch.randn((n, 32), device=cuda), torch.randint(0, 1000, (n, 4), device=cuda).float())
    with only_free(n * 118):  # pool order takes 112 a point, code rows and labels with the arena 124
        with pytest.raises(hg.HDGError, match="OOM"):
            idx.build(big)
    with pytest.raises(hg.HDGError, match="not built"):
        idx.query(qin, qout)
    idx.build(hg.build_input_t(base, labels))
    d.fill_(-1.0)
    idx.query(qin, qout)
    idx.status()
    torch.cuda.synchronize()
    assert torch.equal(d, want[0]) and torch.equal(i, want[1])


def test_debug_fetch_gemm_err(cuda):
    ws = _range_ws(4000, 8)
    idx, base, _ = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.query(qin, qout)
    assert np.frombuffer(idx.debug_fetch("gemm_err").tobytes(), np.int32)[0] == 0


def test_failed_allocation_is_reported_once(cuda):
    """Neither torch nor the next call of the library finds the status of a build that had no room."""
    import torch
    import hdgrid_b200 as hg
    ws = _range_ws(20_000, 50)
    idx, base, labels = build_gpu(ws, cuda)
    d, i, qin, qout = _io(ws, base, 10, cuda)
    idx.query(qin, qout)
    n = 2_000_000
    big = hg.build_input_t(torch.randn((n, 32), device=cuda), torch.randint(0, 1000, (n, 4), device=cuda).float())
    other = hg.SuperGridIndex.from_text(ws["hdgrid_conf"], ws["filter_conf"])
    with only_free(n * 50):  # (the pool order alone takes 76 a point)
        with pytest.raises(hg.HDGError, match="OOM"):
            other.build(big)
        assert float(torch.ones(8, device=cuda).sum()) == 8.0
        with pytest.raises(hg.HDGError, match="OOM"):
            other.build(big)
        idx.query(qin, qout)
    torch.cuda.synchronize()
