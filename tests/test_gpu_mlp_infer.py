"""Inference in one kernel: against the NumPy restatement with bf16 operand
rounding at the tolerance of the layered kernels, and against the layered
kernels themselves bit for bit -- the loss of nlm_mlp_grad (which runs them)
with the predictions as targets is exactly zero.  Hidden widths and row counts
at the edges of tiles, inputs and outputs wider than one tile, weights changed
after a call, and shapes whose weights do not fit (layered path)."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu

SHAPES = [(10, 128, 3, 2), (1, 16, 1, 1), (17, 48, 2, 9), (64, 112, 4, 64), (33, 24, 5, 8),
          (10, 128, 8, 2), (10, 200, 2, 3)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("rows", [1, 16, 129, 2500])
def test_infer(gpu, shape, rows):
    m = gpu.MLP(*shape, seed=4)
    lay, npar = mlp_ref.layout(*shape)
    rng = np.random.default_rng(rows)
    for k in range(2):  # the second time with other weights
        p = m.params()
        p = p + (p != 0) * rng.normal(0, 0.02, p.size).astype(np.float32)
        m.set_params(p)
        x = rng.normal(size=(rows, shape[0])).astype(np.float32)
        y = m.forward(x)
        yr, _ = mlp_ref.forward(p, lay, x, shape[3])
        assert np.abs(y - yr).max() <= 1e-2 * max(np.abs(yr).max(), 1e-3)
        assert m.grad(x, y)[0] == 0.0
