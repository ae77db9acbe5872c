"""The cost model's gradient kernel takes 64 samples at a time: sample counts
around the tile and around a full grid of tiles (304 blocks), with an index
list absent (the training loop passes one), against the 64-bit reference.

Tolerance: a gradient entry is a sum of products whose factors went through at
most 64 + 16 + 64 FP32 additions, so its relative error is below about
150 * 2^-24 = 9e-6 of the terms' size; 2e-5 of the whole gradient's norm."""
import numpy as np
import pytest

from tests import mlp_ref
from toucangpurt_gb300 import sim


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 304 * 64, 304 * 64 + 1, 2 * 304 * 64 + 63])
def test_gradient_around_tiles(built, n):
    rng = np.random.default_rng(n)
    p = rng.normal(0, 0.2, mlp_ref.N_PARAMS).astype(np.float32)
    X = rng.uniform(0, 4, (n, 16)).astype(np.float32)
    y = rng.normal(0, 1, n).astype(np.float32)
    g, loss = sim.mlp_grad(p, X, y)
    gr, lr = mlp_ref.grad(p.astype(np.float64), X.astype(np.float64), y.astype(np.float64))
    assert abs(loss - lr) <= 2e-5 * lr
    assert np.linalg.norm(g - gr) <= 2e-5 * np.linalg.norm(gr)
