"""Kernels at the sizes where their tiling changes: edges of tiles, remainders, the smallest
and largest of a range, against the oracle or a plain restatement."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from hdgrid_b200 import datasets

pytestmark = pytest.mark.gpu


# 8 / 16 / 32-row tiles: below, at and past one tile, one tile per SM (148) and the next size up
@pytest.mark.parametrize("n", [1, 7, 9, 31, 33, 1184, 1185, 2369, 4737, 9473])
def test_mlp_tiles(cuda, n):
    import torch
    import hdgrid_b200 as hg
    ws = datasets.config1(scale=0.02, n_queries=4)
    idx = hg.SuperGridIndex.from_text(ws["hdgrid_conf"], ws["filter_conf"])
    idx.mlp_init(9)
    w = idx.mlp_weights()
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((n, mo.F)) * 0.7).astype(np.float32)
    y = np.stack([rng.uniform(0, 8, n), rng.integers(0, 2, n)], axis=1).astype(np.float32)
    xt, yt = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    g, loss = idx.mlp_gradients(xt, yt)
    z = idx.mlp_forward(xt).cpu().numpy()
    lo, go = mo.loss_and_grad(w, x, y)
    zo, _ = mo.forward(w, x)
    # one hidden unit's BF16 rounding may flip (2^-8 of it): the bounds of the other MLP tests
    assert np.abs(z - zo).max() <= 1e-2 * (1.0 + np.abs(zo).max())
    assert abs(loss - lo) <= 1e-3 * abs(lo) if n < 32 else abs(loss - lo) <= 1e-4 * abs(lo)
    gg, oo = mo.split(g.cpu().numpy().astype(np.float64)), mo.split(go)
    for name, _ in mo.SHAPES:
        rel = np.linalg.norm(gg[name] - oo[name]) / max(np.linalg.norm(oo[name]), 1e-12)
        assert rel <= (2e-2 if n < 32 else 5e-3), (name, rel)


# one to four queries per shared-memory table, tables from one subspace to the largest that fits
# (and past it: 256), candidate tiles of 128, candidates past the data set
@pytest.mark.parametrize("m,q", [(1, 1), (7, 2), (25, 3), (32, 5), (33, 4), (50, 7), (64, 3), (128, 2), (200, 1), (256, 2)])
@pytest.mark.parametrize("n,n_cand", [(1, 1), (127, 130), (128, 128), (2051, 2051), (40000, 33333)])
def test_pq_adc_all_candidates(cuda, m, q, n, n_cand):
    import torch
    import hdgrid_b200 as hg
    rng = np.random.default_rng(m * 1000 + n)
    codes = rng.integers(0, 256, (m, n), dtype=np.uint8)
    lut = rng.random((q, m, 256), dtype=np.float32)
    out = torch.full((q, n_cand), -1.0, device=cuda)
    hg.pq_adc(torch.from_numpy(codes).to(cuda), n, torch.from_numpy(lut).to(cuda), q, m, 256, None, n_cand, out)
    got = out.cpu().numpy()
    real = min(n, n_cand)
    want = np.zeros((q, real))
    for j in range(m):
        want += lut[:, j, :].astype(np.float64)[:, codes[j, :real]]
    # m positive terms summed in FP32 in some order: relative error below m * 2^-24
    assert np.abs(got[:, :real] - want).max() <= m * 2.0 ** -24 * want.max()
    assert np.all(got[:, real:] == np.finfo(np.float32).max)


@pytest.mark.parametrize("l,q", [(1, 1), (3, 64), (4, 65), (4, 2), (8, 130)])
@pytest.mark.parametrize("n,n_cand", [(1, 1), (5, 3), (1023, 1026), (4097, 4097), (5000, 4096)])
def test_label_mask_all_candidates(cuda, l, q, n, n_cand):
    import torch
    import hdgrid_b200 as hg
    rng = np.random.default_rng(l * 100 + q + n)
    lab = rng.integers(0, 20, (n, l)).astype(np.float32)
    lab[rng.random((n, l)) < 0.02] = np.nan  # a NaN label passes
    lo = rng.integers(-1, 12, (q, l)).astype(np.float32)
    hi = lo + rng.integers(0, 15, (q, l)).astype(np.float32)
    box = np.stack([lo, hi], axis=2).reshape(q, 2 * l).copy()
    out = torch.full((q, n_cand), 7, dtype=torch.int32, device=cuda)
    hg.label_mask(torch.from_numpy(box).to(cuda), torch.from_numpy(lab).to(cuda), l, n, q, None, n_cand, out)
    got = out.cpu().numpy()
    real = min(n, n_cand)
    bad = (lab[None, :real, :] < lo[:, None, :]) | (lab[None, :real, :] > hi[:, None, :])
    assert np.array_equal(got[:, :real], (~bad.any(2)).astype(np.int32))
    assert np.all(got[:, real:] == 0)


@pytest.mark.parametrize("entries", [2, 512, 514, 70000])
def test_recover_filters_map_sizes(cuda, entries):
    import torch
    import hdgrid_b200 as hg
    rng = np.random.default_rng(entries)
    table = rng.integers(0, 1 << 20, entries)
    conf = "l = 1\nfilter0:\n\ttype = 1\n\tinterval_map = [" + ", ".join(map(str, table)) + "]\n"
    ql = np.concatenate([[1.0, entries / 2, entries / 2 + 1], rng.integers(1, entries // 2 + 1, 200)]).astype(np.float32)
    out = torch.empty((ql.size, 2), device=cuda)
    hg.recover_filters(conf, torch.from_numpy(ql[:, None].copy()).to(cuda), out)
    got = out.cpu().numpy()
    v = (ql - 1).astype(np.int64)
    ok = 2 * v + 1 < entries
    assert np.array_equal(got[ok, 0], table[2 * v[ok]].astype(np.float32))
    assert np.array_equal(got[ok, 1], table[2 * v[ok] + 1].astype(np.float32))
    assert np.all(got[~ok, 0] > got[~ok, 1])  # outside the table: an empty box


# queries sharing warps (1 to 16) and two per warp, ragged groups; k at both buffer sizes; tiles of
# 128 rows and their remainders; rows read as float4, as floats, and too long for a staged tile
@pytest.mark.parametrize("q,k", [(1, 1), (2, 100), (3, 256), (9, 10), (16, 128), (17, 129), (33, 100), (70, 5)])
@pytest.mark.parametrize("n,d,l", [(1, 4, 1), (31, 3, 4), (129, 100, 2), (5000, 128, 4), (20011, 96, 8), (1500, 384, 3),
                                   (700, 1001, 1), (300, 6000, 2)])
def test_bruteforce_shapes(cuda, q, k, n, d, l):
    import torch
    import hdgrid_b200 as hg
    rng = np.random.default_rng(q * 31 + n)
    base = rng.standard_normal((n, d), dtype=np.float32)
    qs = rng.standard_normal((q, d), dtype=np.float32)
    lab = rng.integers(0, 1000, (n, l)).astype(np.float32)
    lo = np.where(rng.random((q, l)) < 0.6, 0, rng.integers(0, 1000, (q, l))).astype(np.float32)
    hi = np.where(rng.random((q, l)) < 0.6, 1000, lo + rng.integers(0, 300, (q, l))).astype(np.float32)
    box = np.stack([lo, hi], axis=2).reshape(q, 2 * l).copy()
    dist = torch.full((q, k), -1.0, device=cuda)
    ids = torch.full((q, k), 7, dtype=torch.int64, device=cuda)
    hg.bruteforce_knn(torch.from_numpy(base).to(cuda), torch.from_numpy(lab).to(cuda), torch.from_numpy(qs).to(cuda),
                      torch.from_numpy(box).to(cuda), k, dist, ids)
    gd, gi = dist.cpu().numpy(), ids.cpu().numpy()
    for i in range(q):
        ok = np.all((lab >= lo[i]) & (lab <= hi[i]), axis=1)
        e = ((base[ok].astype(np.float64) - qs[i].astype(np.float64)) ** 2).sum(1)
        m = min(k, e.size)
        tol = (d + 2) * 2.0 ** -24  # d positive terms, one FP32 chain
        np.testing.assert_allclose(gd[i, :m], np.sort(e)[:m], rtol=tol)
        full = np.full(n, np.inf)
        full[ok] = e
        np.testing.assert_allclose(full[gi[i, :m]], gd[i, :m], rtol=tol)
        assert len(set(gi[i, :m].tolist())) == m
        assert np.all(np.isinf(gd[i, m:])) and np.all(gi[i, m:] == -1)


# small batches are enqueued without a host read: their stats are read on demand, whatever ran since
@pytest.mark.parametrize("q", [1, 5, 64])
def test_small_batch_stats_on_demand(cuda, q):
    import torch
    import hdgrid_b200 as hg
    from tests.helpers import build_gpu
    ws = datasets.config1(scale=0.1, n_queries=64)
    idx, base, _ = build_gpu(ws, cuda)
    qs, ql = torch.from_numpy(ws["queries"]).to(cuda), torch.from_numpy(ws["query_labels"]).to(cuda)

    def call(n, stream=None):
        d = torch.empty((n, 20), device=cuda)
        i = torch.empty((n, 20), dtype=torch.int64, device=cuda)
        idx.query(hg.query_input_t(base, qs[:n].contiguous(), ql[:n].contiguous()), hg.query_output_t(d, i), stream=stream)
        return d, i

    idx.set_param("BREAK_DOWN", 1)  # timed calls read the scalars at once
    d0, i0 = call(q)
    want = idx.last_query_stats()
    call(17)
    other = idx.last_query_stats()
    idx.set_param("BREAK_DOWN", 0)
    d1, i1 = call(q)
    assert idx.last_query_stats() == want
    assert torch.equal(d0, d1) and torch.equal(i0, i1)
    call(17)
    idx.query_features(qs, ql, 20)  # reuses the workspace: the call's stats are kept
    assert idx.last_query_stats() == other
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    call(17)
    call(q, side)  # the newest call counts, on whichever stream
    assert idx.last_query_stats() == want
    call(17, side)
    call(q)
    assert idx.last_query_stats() == want
    torch.cuda.synchronize()


def _plain_and_full(cuda, ws, k, conf=()):
    """A batch through the plain call (estimate pass) and through a graph replay (full scan)."""
    import torch
    import hdgrid_b200 as hg
    from tests.helpers import build_gpu
    idx, base, _ = build_gpu(ws, cuda)
    for key, v in conf:
        idx.set_param(key, v)
    q, ql = torch.from_numpy(ws["queries"]).to(cuda), torch.from_numpy(ws["query_labels"]).to(cuda)
    out = []
    for graph in (0, 1):
        idx.set_param("QUERY_GRAPH", graph)
        d = torch.full((q.shape[0], k), -1.0, device=cuda)
        i = torch.full((q.shape[0], k), 7, dtype=torch.int64, device=cuda)
        for _ in range(2):
            idx.query(hg.query_input_t(base, q, ql), hg.query_output_t(d, i))
        if graph:
            idx.status()
            d.fill_(-1.0)
            i.fill_(7)
            idx.query(hg.query_input_t(base, q, ql), hg.query_output_t(d, i))
            idx.status()
        else:
            idx.set_param("BREAK_DOWN", 1)
            idx.query(hg.query_input_t(base, q, ql), hg.query_output_t(d, i))
            stages = idx.stage_times()
            idx.set_param("BREAK_DOWN", 0)
        torch.cuda.synchronize()
        out.append((d, i))
    return idx, stages, out


# one to three groups of 32 subspaces (K of 128, 64 + a remainder chunk, 384), FP16 tables, split
# ranges, ragged query tiles; the estimate pass must select what the full scan selects
@pytest.mark.parametrize("case", ["m32", "m64", "m96", "fp16", "split", "few", "d96"])
def test_estimate_pass_equals_full_scan(cuda, case):
    import torch
    if case in ("m96", "fp16"):
        ws = datasets.config2(scale=0.4, n_queries=2001, max_grids=30_000, exps0=2, lut_fp16=1 if case == "fp16" else 0)
    else:
        ws = datasets.config4(scale=0.04, n_queries=129 if case == "few" else 1500, clusters=16, sub_clusters=8,
                              n_list=16, sub_lists=100, exps0=8, max_grids=16384, pq_dim=64 if case == "m64" else 32,
                              is_split=1 if case == "split" else 0, n_split=3 if case == "split" else 1)
        if case == "few":  # long rows from few queries: open boxes
            ws["query_labels"][:, 0::2] = 0
            ws["query_labels"][:, 1::2] = 1_000_000
        if case == "d96":  # K of 96: one whole chunk of 64 and half of one
            ws["base"] = np.ascontiguousarray(ws["base"][:, :96])
            ws["queries"] = np.ascontiguousarray(ws["queries"][:, :96])
    idx, stages, out = _plain_and_full(cuda, ws, 100)
    assert "estimate" in stages, stages
    assert torch.equal(out[0][1], out[1][1]) and torch.equal(out[0][0], out[1][0])


def test_estimate_pass_threshold_too_low(cuda):
    """One list whose position order is the id order, with the near points exactly at the sampled
    positions: the threshold lies below the budget's share and every query is scanned in full."""
    import torch
    n, d, nq, k, exps0 = 1 << 17, 64, 300, 100, 4
    rng = np.random.default_rng(3)
    base = (rng.standard_normal((n, d)) * 0.1 + 5.0).astype(np.float32)
    K = exps0 * k
    for ms in range(int((5 * np.sqrt(K * n)) ** (2 / 3)) - 1, int((5 * np.sqrt(K * n)) ** (2 / 3)) + 3):
        pos = (np.arange(ms, dtype=np.int64) * n + n // 2) // ms
        base[pos[:: max(1, ms // 24)]] -= 5.0
    ws = dict(base=base, labels=np.full((n, 2), 10, np.float32),
              queries=(rng.standard_normal((nq, d)) * 0.1).astype(np.float32),
              query_labels=np.full((nq, 2), 10, np.float32),
              hdgrid_conf=datasets.hdgrid_conf(clusters=1, sub_clusters=1, pq_dim=32, max_grids=16, n_list=1, sub_lists=1,
                                               exps0=exps0, topk=k),
              filter_conf="l = 2\nfilter0:\n\ttype = 0\n\tshift_val = [5, 5]\nfilter1:\n\ttype = 0\n\tshift_val = [5, 5]\n")
    idx, stages, out = _plain_and_full(cuda, ws, k)
    assert "estimate" in stages, stages
    assert torch.equal(out[0][1], out[1][1]) and torch.equal(out[0][0], out[1][0])
    # every query's kept count was below its budget's share, so every candidate was scanned
    import hdgrid_b200 as hg
    idx.set_param("QUERY_GRAPH", 0)
    b, q, ql = (torch.from_numpy(ws[x]).to(cuda) for x in ("base", "queries", "query_labels"))
    idx.query(hg.query_input_t(b, q, ql), hg.query_output_t(*out[0]))
    nfin = np.frombuffer(idx.debug_fetch("nfin").tobytes(), np.uint32)[:nq]
    assert np.all(nfin == n), nfin


# the tensor-core path: one and several query tiles, row tiles with remainders, K with a remainder
# chunk, label dims of both forms, samples without k passing rows, more passing rows than a list holds
@pytest.mark.parametrize("q,k,n,d,l,kind", [
    (64, 10, 187500, 128, 4, "mixed"), (130, 100, 92311, 96, 4, "mixed"), (257, 256, 46700, 100, 2, "mixed"),
    (65, 1, 185000, 33, 8, "mixed"), (100, 100, 120001, 200, 1, "rare"), (70, 100, 171500, 16, 4, "same"),
    (64, 50, 187501, 64, 1, "sorted"), (32, 100, 375000, 32, 3, "mixed")])
def test_bruteforce_tensor_path(cuda, q, k, n, d, l, kind):
    import torch
    import hdgrid_b200 as hg
    rng = np.random.default_rng(q + n)
    base = rng.standard_normal((n, d), dtype=np.float32)
    qs = rng.standard_normal((q, d), dtype=np.float32)
    if kind == "same":  # every row at one distance: every bound ties, ids decide
        base[:] = base[0]
    if kind == "sorted":  # the near rows lie together: a strided sample sees few of them
        base[:60000] *= np.float32(0.01)
        qs *= np.float32(0.01)
    lab = rng.integers(0, 1000, (n, l)).astype(np.float32)
    lo = np.where(rng.random((q, l)) < 0.6, 0, rng.integers(0, 1000, (q, l))).astype(np.float32)
    hi = np.where(rng.random((q, l)) < 0.6, 1000, lo + rng.integers(0, 300, (q, l))).astype(np.float32)
    if kind == "rare":
        hi = lo + 1
    box = np.stack([lo, hi], axis=2).reshape(q, 2 * l).copy()
    t = [torch.from_numpy(x).to(cuda) for x in (base, lab, qs, box)]
    dist = torch.full((q, k), -1.0, device=cuda)
    ids = torch.full((q, k), 7, dtype=torch.int64, device=cuda)
    hg.bruteforce_knn(*t, k, dist, ids)
    # in groups below the batch rule: the direct path, the same arithmetic and order
    d2, i2 = torch.empty_like(dist), torch.empty_like(ids)
    for a in range(0, q, 31):
        b = min(q, a + 31)
        hg.bruteforce_knn(t[0], t[1], t[2][a:b].contiguous(), t[3][a:b].contiguous(), k, d2[a:b], i2[a:b])
    assert torch.equal(ids, i2) and torch.equal(dist, d2)


# the same with components that FP16 cannot hold, infinities and NaN in queries and base rows, the
# last row tile of every level a part of one and its last row inside the boxes
@pytest.mark.parametrize("n", [187500, 187507, 187649])
def test_bruteforce_tensor_path_not_finite(cuda, n):
    import torch
    import hdgrid_b200 as hg
    q, k, d, l = 64, 10, 128, 4
    rng = np.random.default_rng(n)
    base = rng.standard_normal((n, d), dtype=np.float32)
    qs = rng.standard_normal((q, d), dtype=np.float32)
    lab = rng.integers(0, 1000, (n, l)).astype(np.float32)
    box = np.tile(np.array([0, 1000], np.float32), (q, l))  # every row passes ...
    box[40:, 0] = 700                                       # ... or about a third
    lab[-1] = 800
    for i, v in enumerate((70_000.0, -65_520.0, np.inf, -np.inf, np.nan, 3e19, -3e38, 0.0)):
        qs[5 * i, i] = v
        qs[5 * i + 1] = v
        qs[56 + i, d - 1] = v
    for i, v in enumerate((70_000.0, -1e30, np.inf, -np.inf, np.nan)):
        base[rng.integers(0, n, 40), i] = v
    t = [torch.from_numpy(x).to(cuda) for x in (base, lab, qs, box)]
    dist = torch.full((q, k), -1.0, device=cuda)
    ids = torch.full((q, k), 7, dtype=torch.int64, device=cuda)
    hg.bruteforce_knn(*t, k, dist, ids)
    d2, i2 = torch.empty_like(dist), torch.empty_like(ids)
    for a in range(0, q, 31):  # the direct path
        b = min(q, a + 31)
        hg.bruteforce_knn(t[0], t[1], t[2][a:b].contiguous(), t[3][a:b].contiguous(), k, d2[a:b], i2[a:b])
    assert int(ids.max()) < n
    assert torch.equal(ids, i2) and torch.equal(dist.view(torch.int32), d2.view(torch.int32))


# the predicate pass by bit planes: rank fields of 12 to 3 bits (one plane a rank, or shifted where
# the planes would be too many), ranges of a few rows to whole lists, labels of few values, NaN
# labels (which take the pass without ranks); ids and distances equal the oracle's
@pytest.mark.parametrize("l", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("labels", ["spread", "few", "nan"])
def test_predicate_pass_planes(cuda, l, labels):
    from tests.test_gpu_parity import INV, _parity
    ws = dict(datasets.config4(scale=0.002, n_queries=70, clusters=8, sub_clusters=4, n_list=6, sub_lists=20,
                               max_grids=2048, exps0=1))
    n, q = ws["base"].shape[0], ws["queries"].shape[0]
    rng = np.random.default_rng(l)
    hi = {"spread": 1_000_000, "few": 6, "nan": 1_000_000}[labels]
    lab = rng.integers(0, hi, (n, l)).astype(np.float32)
    if labels == "nan":
        lab[rng.random((n, l)) < 0.01] = np.nan
    a = rng.integers(0, hi, (q, l, 2)).astype(np.float32)
    box = np.sort(a, axis=2)  # from one value to most of the range
    box[:5] = [0, hi]         # nothing excluded
    box[5:10, 0] = [hi + 1, hi + 2]  # nothing passes
    ws["labels"], ws["query_labels"] = lab, box.reshape(q, 2 * l).copy()
    ws["filter_conf"] = f"l = {l}\n" + "".join(f"filter{i}:\n\ttype = 3\n" for i in range(l))
    idx, r = _parity(ws, cuda, exact_ids=True, adc_rotated=True)
    valid = r["g_ids"] != INV
    assert valid.any()
    assert np.array_equal(r["g_ids"], r["o_ids"])
    assert np.array_equal(r["g_dist"][valid].view(np.uint32), r["o_dist"][valid].view(np.uint32))
