"""The tcgen05 tiles of the learned warm start at the edges of a tile and of a
block's run of tiles, against the mma.sync kernels: the same BF16 operands and
rounding points with FP32 sums in another order, where a flipped BF16 rounding
(2^-8 of one of 128 terms) gives 1e-3 of the output scale and, through the
backward pass, 1e-2 of a layer's gradient."""
import numpy as np
import pytest

from test_gpu_mlp import _layers_close, _problem, mlp  # noqa: F401

pytestmark = pytest.mark.gpu


def _both(m, f):
    prev = m.tensor_path(False)
    try:
        want = f()
        m.tensor_path(True)
        return f(), want
    finally:
        m.tensor_path(prev)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 304 * 128 - 1, 304 * 128 + 1, 700 * 128 + 5])
def test_inference(mlp, n):  # noqa: F811
    p, st, X, _ = _problem(21, n)
    if n == 1:
        _, st, _, _ = _problem(21, 64)
    mlp.set_params(p, st)
    got, want = _both(mlp, lambda: mlp.infer(X))
    assert (np.abs(got - want).max(axis=0) <= 1e-3 * np.abs(want).max(axis=0)).all()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1025])
def test_gradient(mlp, n):  # noqa: F811
    """Few and many samples of a larger set, and the same minibatch again after
    a step (the weights in the tensor cores' order follow the others)."""
    p, st, X, T = _problem(22, 2000)
    idx = np.random.default_rng(n).permutation(2000)[:n].astype(np.int32)

    def run():
        mlp.set_params(p, st)
        mlp.set_data(X, T)
        first = mlp.grad(idx)
        mlp.step(idx, 1e-3, 1e-4)
        return first, mlp.grad(idx)

    got, want = _both(mlp, run)
    for (g, loss), (wg, wloss) in zip(got, want):
        assert abs(loss - wloss) <= 1e-3 * wloss
        _layers_close(g, wg, 1e-2)
