"""Gradients of the separating-axis MLP at the sizes where the tiled gradient
kernel changes shape: one sample, the edges of a 32-sample tile, the largest
batch with one tile per CTA (296 tiles) and batches whose CTAs take several
tiles, against the float64 oracle; and the same bits on a second run.

Tolerance: a gradient passes through six products of at most 64 terms in
float (fused multiply-adds), each with a relative error of at most 64 * 2^-24
= 4e-6 of its terms' magnitudes; with cancellation of a few times that, 1e-4
of a block's norm bounds it."""
import os
import sys

import numpy as np
import pytest

import reflib
from reactphysics3d_b200 import engine

sys.path.insert(0, os.path.join(reflib.ROOT, "oracle"))
import axis_mlp_oracle as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mlp(cuda_lib):
    ctx = engine.Context(0)
    yield engine.AxisMLP(ctx, seed=17)
    ctx.close()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 4097, 296 * 32, 296 * 32 + 1, 40001])
def test_gradients_match_oracle_at_tile_edges(mlp, n):
    import torch
    p, params, k = mlp.params(), {}, 0
    for name in M.ORDER:
        size = int(np.prod(M.SHAPES[name]))
        params[name] = p[k:k + size].reshape(M.SHAPES[name])
        k += size
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, M.IN)).astype(np.float32)
    y = rng.integers(0, M.OUT, n).astype(np.uint8)
    xd, yd = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    g, loss = mlp.grads(xd, yd)
    g2, loss2 = mlp.grads(xd, yd)
    assert torch.equal(g, g2) and loss == loss2
    ref_loss, ref = M.loss_and_grads(params, x, y.astype(np.int64))
    assert abs(loss - ref_loss) <= 1e-5 * max(1.0, abs(ref_loss))
    g, k = g.cpu().numpy().astype(np.float64), 0
    for name in M.ORDER:
        r = ref[name].ravel()
        assert np.linalg.norm(g[k:k + r.size] - r) <= 1e-4 * np.linalg.norm(r) + 1e-12, name
        k += r.size
