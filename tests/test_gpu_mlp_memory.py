"""Calls with more and more rows keep one set of device buffers, not one per
size seen: at most half as much again as one call with the largest."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _taken(torch, gpu, shape, rows, call):
    """Device bytes that a model holds after calls with these row counts."""
    gc.collect()
    m = gpu.MLP(*shape, seed=1)
    m.forward(np.zeros((16, shape[0]), dtype=np.float32))
    free = torch.cuda.mem_get_info()[0]
    for r in rows:
        x = np.ones((r, shape[0]), dtype=np.float32)
        getattr(m, call)(x, *([np.ones((r, shape[3]), dtype=np.float32)] if call != "forward"
                              else []))
    out = free - torch.cuda.mem_get_info()[0]
    m.close()
    return out


@pytest.mark.parametrize("shape,step,call", [((10, 128, 3, 2), 100000, "forward"),
                                             ((10, 200, 2, 3), 10000, "forward"),
                                             ((10, 64, 2, 2), 20000, "grad"),
                                             ((10, 64, 2, 2), 200000, "set_data")])
def test_growing_row_counts(gpu, shape, step, call):
    torch = pytest.importorskip("torch")
    torch.empty(1, device="cuda")
    rows = [step * k for k in range(1, 13)]
    _taken(torch, gpu, shape, rows[:1], call)
    one = _taken(torch, gpu, shape, rows[-1:], call)
    grown = _taken(torch, gpu, shape, rows, call)
    assert one > 20 << 20
    assert grown <= 1.5 * one + (16 << 20), (grown, one)


def test_values_after_growing(gpu):
    m = gpu.MLP(10, 200, 2, 3, seed=1)
    rng = np.random.default_rng(0)
    x = rng.normal(size=(5000, 10)).astype(np.float32)
    y = m.forward(x)
    for r in (100, 1500, 2100, 5000, 7):
        assert np.array_equal(m.forward(x[:r]), y[:r])
        m2 = gpu.MLP(10, 128, 2, 3, seed=1)
        m2.set_params(m2.params())
        a = m2.forward(x[:7])
        assert np.array_equal(m2.forward(x[:r])[:7], a)
