"""Timed workloads of the filtered-search path.

Each case is one call that a program using this library makes, with the sizes, filters and
options of the synthetic benchmark configurations (hdgrid_b200/datasets.py), scaled over the
range the library is used in.  ``prepare`` builds what such a program holds beforehand (the
index, the base set, the query batch, output buffers), ``run`` is one call.

Kinds:
* ``shift``   integer labels with +-window filters (config1): one label dim takes the single-dim
              schedule, two or more the post-filter schedule.  A vector or code length that is
              not a multiple of 32 takes the general ADC scan.
* ``mixed``   L2-normalised 384-d vectors with a shift, a map and a div filter (config2; ``fp16``
              is its precision variant config3).
* ``ranges``  four label dims with range filters, selectivity log-uniform in [0.01 %, 90 %]
              (config4): ``schedule`` is ``post``, ``pre`` (exps0 = 1) or ``learned`` (config5).
* ``build``   the index build, then a first batch of queries against it.
* ``truth``   exact filtered kNN (ground truth for recall).
* ``kernels`` filter recovery, PQ lookup table, ADC and label mask in the reference's layouts.
* ``train``   loss gradients of the schedule network over one batch, and its outputs.
"""
from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

import hdgrid_b200 as hg
from hdgrid_b200.datasets import MAP_FRACTIONS, hdgrid_conf

WEIGHTS = Path(hg.__file__).resolve().parent / "learned_weights" / "config5.npy"
MLP_IN, MLP_HID, MLP_OUT = 48, 128, 2


def listed():
    return [
        # a search box: one query against a small collection, latency is all
        dict(name="single_query", kind="shift", n=100_000, d=128, m=32, l=1, q=1, k=10),
        # a few requests gathered by a server, vectors of an odd length (general ADC scan)
        dict(name="odd_small_batch", kind="shift", n=200_003, d=100, m=25, l=2, q=37, k=50),
        # config1: 1,000 queries, one label dim
        dict(name="shift_batch", kind="shift", n=100_000, d=128, m=32, l=1, q=1000, k=100),
        # config2: 10,000 queries over 1M text-embedding-sized vectors, post-filter schedule, a
        # fine grid whose prefix counts are kept as compressed rows
        dict(name="mixed_batch", kind="mixed", n=1_000_000, q=10_000, k=100, fp16=False, cells=3_000_000),
        # config3: its precision variant (FP16 tables, BF16 coarse ranking), a ragged batch, dense counts
        dict(name="mixed_fp16", kind="mixed", n=1_000_000, q=3001, k=100, fp16=True, cells=30_000),
        # the pre-filter schedule: predicate first, ADC distances are the answer
        dict(name="pre_filter", kind="ranges", n=1_000_000, q=4099, k=100, schedule="pre", graph=False),
        # config4's plain schedule with each query's own k
        dict(name="range_post", kind="ranges", n=2_000_000, q=10_000, k=100, schedule="post", graph=False),
        # config5: the learned schedule on 10M vectors, replayed as a captured graph
        dict(name="learned_10m", kind="ranges", n=10_000_000, q=10_000, k=100, schedule="learned", graph=True),
        # a collection is loaded and indexed, and answers its first queries
        dict(name="build_index", kind="build", n=1_000_000, d=128, q=256, k=100),
        # ground truth for a recall measurement
        dict(name="exact_truth", kind="truth", n=1_000_000, d=128, q=1000, k=100),
        # the kernel-level entry points on a batch of candidates
        dict(name="reference_kernels", kind="kernels", n=500_000, d=128, m=32, q=100),
        # one training batch of the schedule network
        dict(name="train_batch", kind="train", n=4096),
    ]


def _spread(rng, lo: int, hi: int) -> int:
    """A whole number in [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["shift", "shift", "mixed", "ranges", "ranges", "build", "truth", "kernels", "train"])
    k = rng.choice([10, 50, 100])
    if kind == "shift":
        d, m = rng.choice([(128, 32), (100, 25), (96, 32), (64, 16), (128, 64)])
        return dict(kind=kind, n=_spread(rng, 20_000, 400_000), d=d, m=m, l=rng.choice([1, 2]),
                    q=_spread(rng, 1, 3000), k=k)
    if kind == "mixed":
        return dict(kind=kind, n=_spread(rng, 100_000, 1_000_000), q=_spread(rng, 8, 10_000), k=k,
                    fp16=rng.random() < 0.5, cells=rng.choice([30_000, 3_000_000]))
    if kind == "ranges":
        schedule = rng.choice(["post", "pre", "learned"])
        return dict(kind=kind, n=_spread(rng, 200_000, 2_000_000), q=_spread(rng, 16, 10_000), k=k,
                    schedule=schedule, graph=schedule == "learned" and rng.random() < 0.5)
    if kind == "build":
        return dict(kind=kind, n=_spread(rng, 50_000, 1_000_000), d=rng.choice([96, 128]), q=_spread(rng, 1, 256), k=k)
    if kind == "truth":
        return dict(kind=kind, n=_spread(rng, 50_000, 1_000_000), d=rng.choice([96, 100, 128]),
                    q=_spread(rng, 1, 1000), k=k)
    if kind == "kernels":
        d, m = rng.choice([(128, 32), (100, 25), (96, 12)])
        return dict(kind=kind, n=_spread(rng, 20_000, 500_000), d=d, m=m, q=_spread(rng, 1, 100))
    return dict(kind=kind, n=_spread(rng, 100, 4096))


# ---- inputs ---------------------------------------------------------------------------------

def _gen(seed: int, salt: int):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1_000_003 + salt)
    return g


def _mixture(g, n: int, d: int, comps: int, normalise: bool = False):
    """Rows of a Gaussian mixture whose centres are those of the benchmark's data sets."""
    centres = torch.from_numpy(np.random.default_rng(7).standard_normal((comps, d), dtype=np.float32)).cuda()
    x = torch.empty((n, d), device="cuda")
    for a in range(0, n, 1 << 20):
        b = min(n, a + (1 << 20))
        comp = torch.randint(0, comps, (b - a,), generator=g, device="cuda")
        x[a:b].normal_(0.0, 0.3, generator=g)
        x[a:b] += centres[comp]
        if normalise:
            x[a:b] /= x[a:b].norm(dim=1, keepdim=True)
    return x


def _ints(g, lo: int, hi: int, shape):
    return torch.randint(lo, hi, shape, generator=g, device="cuda").to(torch.float32)


def _uniform(g, shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _shift_inputs(case, seed):
    n, d, l, q = case["n"], case["d"], case["l"], case["q"]
    base = _mixture(_gen(seed, 1), n, d, 64)
    queries = _mixture(_gen(seed, 2), q, d, 64)
    labels = _ints(_gen(seed, 3), 0, 1_000_000, (n, l))
    qlabels = _ints(_gen(seed, 4), 0, 1_000_000, (q, l))
    window = 30_000 if l == 1 else 150_000
    filt = f"l = {l}\n" + "".join(f"filter{i}:\n\ttype = 0\n\tshift_val = [{window}, {window}]\n" for i in range(l))
    conf = hdgrid_conf(clusters=8, sub_clusters=8, pq_dim=case["m"], max_grids=1_000_000 if l == 1 else 10_000,
                       n_list=8, sub_lists=64, exps0=4, topk=case["k"])
    ranges = torch.stack([qlabels - window, qlabels + window], dim=2).reshape(q, 2 * l)
    return base, labels, queries, qlabels, ranges, conf, filt


def _mixed_inputs(case, seed):
    n, q = case["n"], case["q"]
    base = _mixture(_gen(seed, 1), n, 384, 1024, normalise=True)
    queries = _mixture(_gen(seed, 2), q, 384, 1024, normalise=True)
    g = _gen(seed, 3)
    labels = torch.cat([_ints(g, 0, 30_000_000, (n, 1)), _ints(g, 0, 10_000, (n, 2))], dim=1).contiguous()
    g = _gen(seed, 4)
    # selectivity log-uniform in [0.1 %, 2 %]: the time window gives 2 %, a map interval and
    # the div threshold the rest
    sel = torch.exp(_uniform(g, (q,)) * math.log(20.0) + math.log(0.001))
    r = torch.clamp(sel / (604_800 / 30_000_000), max=1.0)
    fr = torch.tensor(MAP_FRACTIONS, device="cuda", dtype=torch.float64)
    n_ok = (fr[None, :] >= r[:, None]).sum(1)  # the fractions fall, so the usable ones come first
    j = torch.minimum((_uniform(g, (q,)) * n_ok).long(), n_ok - 1).clamp(min=0)
    keep = torch.clamp(r / fr[j], max=1.0)
    q_div = torch.floor((1.0 - keep) * 10_000) * 10
    q_ts = _ints(g, 604_800, 30_000_000, (q,))
    qlabels = torch.stack([q_ts, (j + 1).float(), q_div.float()], dim=1).contiguous()
    table = ", ".join(f"0, {int(round(f * 10_000)) - 1}" for f in MAP_FRACTIONS)
    filt = ("l = 3\nfilter0:\n\ttype = 0\n\tshift_val = [604800, 0]\n"
            f"filter1:\n\ttype = 1\n\tinterval_map = [{table}]\n"
            "filter2:\n\ttype = 2\n\tdiv_value = [10]\n")
    extra = dict(lut_fp16=1, coarse_bf16=1, sub_lists=448, exps0=4) if case["fp16"] else dict(sub_lists=512, exps0=10)
    conf = hdgrid_conf(clusters=64, sub_clusters=8, pq_dim=96, n_list=64, topk=case["k"],
                       max_grids=case["cells"], **extra)
    return base, labels, queries, qlabels, conf, filt


def _range_boxes(g, q: int):
    """[q x 8] lo / hi of four label dims: 1 to 4 random dims bounded, the others open."""
    sel = torch.exp(_uniform(g, (q,)) * (math.log(0.9) - math.log(0.0001)) + math.log(0.0001))
    j = torch.randint(1, 5, (q,), generator=g, device="cuda")
    rank = _uniform(g, (q, 4)).argsort(dim=1).argsort(dim=1)
    bounded = rank < j[:, None]
    width = torch.clamp(torch.round(sel ** (1.0 / j) * 1_000_000), min=1.0)
    lo = torch.floor(_uniform(g, (q, 4)) * (1_000_000 - width[:, None] + 1))
    hi = lo + width[:, None] - 1
    lo = torch.where(bounded, lo, torch.zeros_like(lo))
    hi = torch.where(bounded, hi, torch.full_like(hi, 1_000_000.0))
    return torch.stack([lo, hi], dim=2).reshape(q, 8).float().contiguous()


RANGE_FILTER = "l = 4\n" + "".join(f"filter{i}:\n\ttype = 3\n" for i in range(4))


def _range_inputs(case, seed, d=128):
    n, q = case["n"], case["q"]
    base = _mixture(_gen(seed, 1), n, d, 1024)
    queries = _mixture(_gen(seed, 2), q, d, 1024)
    labels = _ints(_gen(seed, 3), 0, 1_000_000, (n, 4))
    g = _gen(seed, 4)
    boxes = _range_boxes(g, q)
    ks = torch.where(torch.rand((q,), generator=g, device="cuda") < 0.5, max(1, case["k"] // 10), case["k"])
    return base, labels, queries, boxes, ks.to(torch.uint32)


def _range_conf(case):
    big = case["n"] > 4_000_000
    c = dict(clusters=512 if big else 128, sub_clusters=8, pq_dim=32, max_grids=65536 if big else 16384, filter_dim=2,
             topk=case["k"])
    schedule = case.get("schedule", "post")
    if schedule == "post":
        c.update(n_list=64, sub_lists=64, exps0=32)
    elif schedule == "pre":
        c.update(n_list=64, sub_lists=256, exps0=1)
    else:
        c.update(n_list=128 if big else 64, sub_lists=1024 if big else 512, exps0=32, learned=1,
                 query_graph=1 if case["graph"] else 0)
    return hdgrid_conf(**c)


def _index(conf, filt, base, labels):
    idx = hg.SuperGridIndex.from_text(conf, filt)
    idx.build(hg.build_input_t(base, labels))
    return idx


def _outputs(q: int, k: int):
    return (torch.empty((q, k), dtype=torch.float32, device="cuda"),
            torch.empty((q, k), dtype=torch.int64, device="cuda"))


def _mlp_batch(n: int, seed: int):
    g = _gen(seed, 5)
    x = torch.rand((n, MLP_IN), generator=g, device="cuda")
    y = torch.stack([torch.randint(0, 11, (n,), generator=g, device="cuda").float(),
                     (torch.rand((n,), generator=g, device="cuda") < 0.9).float()], dim=1).contiguous()
    return x, y


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("shift", "mixed", "ranges"):
        ks = None
        if kind == "shift":
            base, labels, queries, qlabels, _, conf, filt = _shift_inputs(case, seed)
        elif kind == "mixed":
            base, labels, queries, qlabels, conf, filt = _mixed_inputs(case, seed)
        else:
            base, labels, queries, qlabels, ks = _range_inputs(case, seed)
            conf, filt = _range_conf(case), RANGE_FILTER
        idx = _index(conf, filt, base, labels)
        if kind == "ranges" and case["schedule"] == "learned":
            idx.set_mlp_weights(np.load(WEIGHTS))
        idx.reserve(case["q"])
        dist, ids = _outputs(case["q"], case["k"])
        return dict(kind=kind, idx=idx, k=ks, qin=hg.query_input_t(base, queries, qlabels),
                    qout=hg.query_output_t(dist, ids))
    if kind == "build":
        base, labels, queries, boxes, _ = _range_inputs(case, seed, d=case["d"])
        dist, ids = _outputs(case["q"], case["k"])
        return dict(kind=kind, conf=_range_conf(case), bin=hg.build_input_t(base, labels),
                    qin=hg.query_input_t(base, queries, boxes), qout=hg.query_output_t(dist, ids))
    if kind == "truth":
        base, labels, queries, boxes, _ = _range_inputs(case, seed, d=case["d"])
        dist, ids = _outputs(case["q"], case["k"])
        return dict(kind=kind, base=base, labels=labels, queries=queries, boxes=boxes, k=case["k"], dist=dist, ids=ids)
    if kind == "kernels":
        n, d, m, q = case["n"], case["d"], case["m"], case["q"]
        x = _kernel_inputs(case, seed)
        x.update(kind=kind, n=n, m=m, q=q,
                 ranges=torch.empty((q, 8), device="cuda"), lut=torch.empty((q, m, 256), device="cuda"),
                 dist=torch.empty((q, n), device="cuda"), mask=torch.empty((q, n), dtype=torch.int32, device="cuda"))
        return x
    x, y = _mlp_batch(case["n"], seed)
    idx = hg.SuperGridIndex.from_text(hdgrid_conf(), RANGE_FILTER)
    idx.set_mlp_weights(np.load(WEIGHTS))
    return dict(kind=kind, idx=idx, x=x, y=y)


def _kernel_inputs(case, seed):
    n, d, m, q = case["n"], case["d"], case["m"], case["q"]
    return dict(centers=_mixture(_gen(seed, 1), m * 256, d // m, 64).reshape(m, 256, d // m).contiguous(),
                queries=_mixture(_gen(seed, 2), q, d, 64),
                labels=_ints(_gen(seed, 3), 0, 1_000_000, (n, 4)),
                boxes=_range_boxes(_gen(seed, 4), q),
                codes=torch.randint(0, 256, (m, n), generator=_gen(seed, 6), device="cuda").to(torch.uint8))


def run(state):
    kind = state["kind"]
    if kind in ("shift", "mixed"):
        state["idx"].query(state["qin"], state["qout"])
        return {"distances": state["qout"].distances, "neighbors": state["qout"].neighbors}
    if kind == "ranges":
        state["idx"].query_ex(state["qin"], state["qout"], k=state["k"])
        return {"distances": state["qout"].distances, "neighbors": state["qout"].neighbors}
    if kind == "build":
        idx = _index(state["conf"], RANGE_FILTER, state["bin"].dataset, state["bin"].data_labels)
        idx.query(state["qin"], state["qout"])
        return {"distances": state["qout"].distances, "neighbors": state["qout"].neighbors}
    if kind == "truth":
        hg.bruteforce_knn(state["base"], state["labels"], state["queries"], state["boxes"], state["k"], state["dist"],
                          state["ids"])
        return {"distances": state["dist"], "neighbors": state["ids"]}
    if kind == "kernels":
        s = state
        hg.recover_filters(RANGE_FILTER, s["boxes"], s["ranges"])
        hg.pq_lut(s["centers"], s["queries"], s["m"], s["centers"].shape[2], 256, s["lut"])
        hg.pq_adc(s["codes"], s["n"], s["lut"], s["q"], s["m"], 256, None, s["n"], s["dist"])
        hg.label_mask(s["ranges"], s["labels"], 4, s["n"], s["q"], None, s["n"], s["mask"])
        return {"ranges": s["ranges"], "lut": s["lut"], "distances": s["dist"], "mask": s["mask"]}
    grad, loss = state["idx"].mlp_gradients(state["x"], state["y"])
    return {"gradient": grad, "loss": loss, "outputs": state["idx"].mlp_forward(state["x"])}


def work(case):
    """Bytes and operations one call cannot do without: inputs read once, outputs written once,
    and for a query the exact rows of its own results."""
    kind = case["kind"]
    q, k, n = case.get("q", 0), case.get("k", 0), case["n"]
    if kind in ("shift", "mixed", "ranges"):
        d = case.get("d", 384 if kind == "mixed" else 128)
        l = case.get("l", 3 if kind == "mixed" else 4)
        m = case.get("m", 96 if kind == "mixed" else 32)
        # a batch reads codes and labels of the candidates its lists hold; a small batch may
        # touch a part of the pool only
        pool = min(n, q * max(k, n // 50))
        exact = 0 if case.get("schedule") == "pre" else q * k * d
        return {"bytes": 4 * q * (d + 2 * l) + 12 * q * k + pool * (m + 4 * l) + 4 * min(exact, n * d),
                "flops": 3 * exact + 512 * q * d}
    if kind == "build":
        d, lists, train = case["d"], 1024, max(65536, 64 * 1024)
        # assignment of every point and of the training sample's 20 iterations to the lists,
        # and the PQ encoding (3 operations per value and codeword)
        return {"bytes": 4 * n * (d + 4) + n * (32 + 16 + 12) + 12 * q * k,
                "flops": 2 * (n + 20 * min(train, n)) * lists * d + 3 * (n + 20 * min(65536, n)) * 256 * d}
    if kind == "truth":
        d = case["d"]
        return {"bytes": 4 * n * (d + 4) + 4 * q * (d + 8) + 12 * q * k, "flops": 0.23 * 2 * q * n * d}
    if kind == "kernels":
        d, m = case["d"], case["m"]
        return {"bytes": n * (m + 16) + 8 * q * n + 4 * q * (d + m * 256 + 16) + 4 * 256 * d,
                "flops": q * n * m + 3 * q * 256 * d}
    p = MLP_IN * MLP_HID + MLP_HID * MLP_HID + MLP_HID * MLP_OUT
    return {"bytes": 4 * n * (MLP_IN + 2 * MLP_OUT) + 8 * p, "flops": 2 * p * n * 4}


# ---- the same results in 64 bits ---------------------------------------------------------------

def _exact_knn(base, labels, queries, ranges, k):
    """Filtered kNN: squared distances ascending, ties to the lower id, missing ones inf / -1."""
    q, n, l = queries.shape[0], base.shape[0], labels.shape[1]
    b64 = base.double()
    bn = (b64 * b64).sum(1)
    dist = torch.full((q, k), math.inf, dtype=torch.float64, device="cuda")
    ids = torch.full((q, k), -1, dtype=torch.int64, device="cuda")
    step = max(1, (1 << 28) // n)
    for a in range(0, q, step):
        x = queries[a:a + step].double()
        ok = torch.ones((x.shape[0], n), dtype=torch.bool, device="cuda")
        for i in range(l):
            v = labels[None, :, i]
            ok &= (v >= ranges[a:a + step, 2 * i, None]) & (v <= ranges[a:a + step, 2 * i + 1, None])
        s = (x * x).sum(1)[:, None] - 2.0 * (x @ b64.T) + bn[None, :]
        s.masked_fill_(~ok, math.inf)
        near = s.topk(min(k + 16, n), dim=1, largest=False).indices
        fine = torch.take_along_dim(ok, near, dim=1)
        for r in range(x.shape[0]):  # the differences themselves, free of cancellation
            e = ((b64[near[r]] - x[r]) ** 2).sum(1).masked_fill(~fine[r], math.inf)
            order = torch.argsort(e, stable=True)[:k]
            have = torch.isfinite(e[order])
            dist[a + r, :order.numel()] = e[order]
            ids[a + r, :order.numel()] = torch.where(have, near[r][order], -1)
    return {"distances": dist, "neighbors": ids}


def exact(case, seed):
    kind = case["kind"]
    if kind == "truth":
        base, labels, queries, boxes, _ = _range_inputs(case, seed, d=case["d"])
        return _exact_knn(base, labels, queries, boxes, case["k"])
    if kind == "shift":  # these probe nearly every list and re-rank exactly: the true neighbours
        base, labels, queries, _, ranges, _, _ = _shift_inputs(case, seed)
        return _exact_knn(base, labels, queries, ranges, case["k"])
    if kind == "kernels":
        x = _kernel_inputs(case, seed)
        q, n, m, d = case["q"], case["n"], case["m"], case["d"]
        qs = x["queries"].double().reshape(q, m, 1, d // m)
        lut = ((x["centers"].double()[None] - qs) ** 2).sum(3)
        codes = x["codes"].long()
        dist = torch.zeros((q, n), dtype=torch.float64, device="cuda")
        for j in range(m):
            dist += lut[:, j, :][:, codes[j]]
        lab, box = x["labels"], x["boxes"]
        mask = torch.ones((q, n), dtype=torch.int32, device="cuda")
        for i in range(4):
            mask &= ((lab[None, :, i] >= box[:, 2 * i, None]) & (lab[None, :, i] <= box[:, 2 * i + 1, None])).int()
        return {"ranges": box.double(), "lut": lut, "distances": dist, "mask": mask}
    if kind == "train":
        x, y = _mlp_batch(case["n"], seed)
        return _exact_mlp(np.load(WEIGHTS), x, y)
    return None  # the answer of an approximate search has no value apart from the index that gives it


def _exact_mlp(weights, x, y):
    """The network on weights and activations rounded to BF16 (its definition), sums in 64 bits."""
    def rnd(t):
        return t.float().to(torch.bfloat16).double()
    p = torch.from_numpy(np.ascontiguousarray(weights, np.float32)).cuda()
    sizes = [MLP_HID * MLP_IN, MLP_HID, MLP_HID * MLP_HID, MLP_HID, MLP_OUT * MLP_HID, MLP_OUT]
    w1, b1, w2, b2, w3, b3 = torch.split(p, sizes)
    w1, w2, w3 = rnd(w1).view(MLP_HID, MLP_IN), rnd(w2).view(MLP_HID, MLP_HID), rnd(w3).view(MLP_OUT, MLP_HID)
    b1, b2, b3, y = b1.double(), b2.double(), b3.double(), y.double()
    n = x.shape[0]
    x0 = rnd(x)
    a1 = rnd(torch.relu(x0 @ w1.T + b1))
    a2 = rnd(torch.relu(a1 @ w2.T + b2))
    z = a2 @ w3.T + b3
    loss = ((z[:, 0] - y[:, 0]) ** 2 + torch.clamp(z[:, 1], min=0) - z[:, 1] * y[:, 1]
            + torch.log1p(torch.exp(-z[:, 1].abs()))).mean()
    dz = torch.stack([2 * (z[:, 0] - y[:, 0]), torch.sigmoid(z[:, 1]) - y[:, 1]], dim=1) / n
    d2 = (dz @ w3) * (a2 > 0)
    d1 = (d2 @ w2) * (a1 > 0)
    grad = torch.cat([(d1.T @ x0).reshape(-1), d1.sum(0), (d2.T @ a1).reshape(-1), d2.sum(0), (dz.T @ a2).reshape(-1),
                      dz.sum(0)])
    return {"gradient": grad, "loss": float(loss), "outputs": z}
