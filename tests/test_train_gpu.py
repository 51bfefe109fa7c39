"""The fused training kernels at the edges of their tiling: a single padded row,
one full 128-row tile, a tile and a row, several weight-gradient shares, and
shares of half tiles with more tiles than a 152-SM GPU has CTAs (one then takes two).

Tolerances: those of the gradient comparison with the FP64 MLP (bf16 operands:
relative L2 error <= 5e-2 and cosine >= 0.995 per parameter tensor).  The AdamW
step is compared with its formula on the same kernels' gradient (their sums are
ordered, so a second pass gives the same bits): a dozen FP32 roundings of a
step of at most lr (1 + weight decay |p|) plus one of the parameter.
"""
from contextlib import closing

import numpy as np
import pytest

from oracle import mlp_oracle as MO
from spacetime_gb300.surrogate import Surrogate

pytestmark = pytest.mark.gpu


def _tensors(v):
    o = 0
    for name, shape in MO.SIZES:
        n = int(np.prod(shape))
        yield name, v[o:o + n].astype(np.float64)
        o += n


@pytest.mark.parametrize("n", [1, 128, 129, 27 * 128, 152 * 128 + 1])
def test_gradients_at_tile_edges(built_lib, n):
    rng = np.random.default_rng(n)
    X = rng.uniform(-1, 1, (n, 6)).astype(np.float32)
    T = np.zeros((n, 8), np.float32)
    T[:, :3] = rng.normal(0, 0.3, (n, 3))
    T[:, 3] = rng.uniform(-1, 2, n)
    T[:, 4] = rng.normal(0, 0.2, n)
    T[:, 5] = 1.0
    T[:, 6] = np.arange(n) % 2
    with closing(Surrogate(0, seed=5)) as s:
        loss, g = s.loss_grad(X, T)
        rloss, rg = MO.loss_grad(s.get_params(), X, T)
    assert abs(loss[0] - rloss[0]) <= 2e-2 * abs(rloss[0]) + 1e-6
    for (name, a), (_, b) in zip(_tensors(g), _tensors(rg)):
        rel = np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)
        cos = a @ b / max(np.linalg.norm(a) * np.linalg.norm(b), 1e-30)
        assert rel <= 5e-2 and cos >= 0.995, (name, rel, cos)


@pytest.mark.parametrize("batch", [128, 153 * 128])
def test_adamw_step_is_the_formula_on_the_gradient(built_lib, batch):
    lr, wd = 1e-2, 1e-1
    with closing(Surrogate(0, seed=5)) as s:
        x, t, _ = s.generate(batch, offset=0)
        P = s.get_params()
        loss, g = s.loss_grad(x, t)
        hist = s.train(1, batch=batch, lr=lr, weight_decay=wd)
        Q = s.get_params()
        after, _ = s.loss_grad(x, t)
    assert abs(hist[0] - loss[0]) <= 1e-5 * abs(loss[0])
    p, g = P.astype(np.float64), g.astype(np.float64)
    weight = np.concatenate([np.full(int(np.prod(sh)), len(sh) > 1) for _, sh in MO.SIZES])
    want = p - lr * wd * weight * p - lr * g / (np.abs(g) + 1e-8)
    tol = 2.0 ** -23 * (12 * lr * (1 + wd * np.abs(p)) + np.abs(p))
    # a gradient whose square leaves FP32's normal range keeps fewer bits of it
    ok = (np.abs(Q - want) <= tol) | ((g != 0) & (np.abs(g) < 1e-15))
    assert ok.all(), (np.abs(Q - want) / tol).max()
    assert after[0] != loss[0]
