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
