"""The gradient kernel fills its last tile up with samples that are none: they
add nothing, also where the biases alone overflow a layer.  And the kernel with
an index list, as the training loop calls it, against the 64-bit reference.

Tolerance as around the tiles: a gradient entry's factors went through at most
64 + 16 + 64 FP32 additions, 150 * 2^-24 = 9e-6 of the terms' size; 2e-5 of the
whole gradient's norm."""
import ctypes as C

import numpy as np
import pytest

from tests import mlp_ref
from toucangpurt_gb300 import capi, sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65])
def test_filled_up_samples_add_nothing(built, n):
    rng = np.random.default_rng(n)
    p = rng.normal(0, 0.2, mlp_ref.N_PARAMS).astype(np.float32)
    w = {name: p[o:o + int(np.prod(s))].reshape(s) for (name, s), o in
         zip(mlp_ref.SHAPES, np.cumsum([0] + [int(np.prod(s)) for _, s in mlp_ref.SHAPES]))}
    # unit 0 is off for every sample and 1e30 for inputs of zero, which unit 0
    # of the second layer takes beyond FP32
    w["b1"][0], w["W1"][0], w["W2"][0, 0] = 1e30, -1e30, 1e10
    X = rng.uniform(1, 4, (n, 16)).astype(np.float32)
    y = rng.normal(0, 1, n).astype(np.float32)
    g, loss = sim.mlp_grad(p, X, y)
    gr, lr = mlp_ref.grad(p.astype(np.float64), X.astype(np.float64), y.astype(np.float64))
    assert abs(loss - lr) <= 2e-5 * lr
    assert np.linalg.norm(g - gr) <= 2e-5 * np.linalg.norm(gr)


# index lists shorter and longer than a tile and than a grid of them, with
# repeats, over a sample set that they do not cover
@pytest.mark.parametrize("n", [1, 32, 63, 64, 65, 1024, 304 * 64 + 1])
def test_gradient_of_listed_samples(built, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    rows = 3000
    p = rng.normal(0, 0.2, mlp_ref.N_PARAMS).astype(np.float32)
    X = rng.uniform(0, 4, (rows, 16)).astype(np.float32)
    y = rng.normal(0, 1, rows).astype(np.float32)
    idx = rng.integers(0, rows, n).astype(np.int32)
    d = [torch.from_numpy(a).to("cuda:0") for a in (p, X, y, idx)]
    grad = torch.zeros(mlp_ref.N_PARAMS, device="cuda:0")
    loss = torch.zeros(1, device="cuda:0")
    torch.cuda.synchronize()
    # cudaError_t tgs::mlpGrad(params, X, y, idx, n, scale, grad, loss, stream)
    fn = capi.lib()["_ZN3tgs7mlpGradEPKfS1_S1_PKjjfPfS4_P11CUstream_st"]
    fn.argtypes = [C.c_void_p] * 4 + [C.c_uint32, C.c_float] + [C.c_void_p] * 3
    fn.restype = C.c_int
    assert fn(*(t.data_ptr() for t in d), n, 1.0 / n, grad.data_ptr(), loss.data_ptr(), None) == 0
    torch.cuda.synchronize()
    gr, lr = mlp_ref.grad(p.astype(np.float64), X[idx].astype(np.float64), y[idx].astype(np.float64))
    assert abs(loss.item() / n - lr) <= 2e-5 * lr
    assert np.linalg.norm(grad.cpu().numpy() - gr) <= 2e-5 * np.linalg.norm(gr)
