"""nlm_neighbor_search and its one-search form against every pair in numpy with
the reference's predicate (horizon + 1e-10 definitely greater than the
distance, relative 1e-5): identical rows.  Bonds exactly at the horizon, far
from the origin (where FP32 cannot decide), thin and sparse clouds, coincident
nodes, one and no node."""
import ctypes as C

import numpy as np
import pytest

from nlmech_gb300 import abi, configs

pytestmark = pytest.mark.gpu


def _pairs(x, horizon):
    rows = []
    rad = horizon + 1e-10
    for i in range(len(x)):
        d = x[i] - x
        r = np.sqrt(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2])
        near = (rad - r) > np.maximum(np.abs(r), rad) * 1e-5
        near[i] = False
        rows.append(np.flatnonzero(near).astype(np.int32))
    return np.concatenate([[0], np.cumsum([len(r) for r in rows])]), np.concatenate(rows)


def _cloud(name):
    rng = np.random.default_rng(5)
    if name == "lattice":  # distances equal to the horizon up to rounding
        return configs.grid2d(23, 17, 1e-3, 0.0, 0)[0], 3e-3, 2
    if name == "lattice_inside":  # just past it relative to the tolerance
        return configs.grid2d(23, 17, 1e-3, 0.0, 0)[0], 3e-3 * (1 + 1.0001e-5), 2
    if name == "shuffled_3d":
        x = configs.grid3d(9, 8, 7, 1e-3, 0.05, 1)[0]
        return np.ascontiguousarray(x[rng.permutation(len(x))]), 3e-3, 3
    if name == "far":
        return configs.grid2d(20, 15, 1e-3, 0.05, 2)[0] + [4e5, -3e5, 0.0], 3e-3, 2
    if name == "far_pair":  # one node 1e5 horizons away: FP32 margin of the order of h
        x = configs.grid2d(20, 15, 1e-3, 0.05, 2)[0]
        x[7] += [2e2, 0.0, 0.0]
        return x, 3e-3, 2
    if name == "line":
        x = np.zeros((50, 3))
        x[:, 0] = rng.uniform(0, 1, 50)
        return x, 0.1, 1
    if name == "coincident":
        x = rng.uniform(0, 1, (60, 3))
        x[31] = x[30]
        return x, 0.3, 3
    return np.array([[0.5, 0.25, 0.0]]), 0.1, 2


@pytest.mark.parametrize("name", ["lattice", "lattice_inside", "shuffled_3d", "far", "far_pair",
                                  "line", "coincident", "one"])
def test_rows_equal_all_pairs(gpu, name):
    x, hz, dim = _cloud(name)
    rp, cols = gpu.neighbor_search(x, hz, dim)
    rp0, cols0 = _pairs(x, hz)
    assert np.array_equal(rp, rp0) and np.array_equal(cols, cols0)
    # the two-call form, counts first
    L, x = gpu.load(), np.ascontiguousarray(x)
    rp2 = np.zeros(len(x) + 1, dtype=np.int64)
    cols2 = np.zeros(len(cols0), dtype=np.int32)
    arg = (C.c_int(dim), C.c_int64(len(x)), abi.dptr(x), C.c_double(hz),
           abi.ptr(rp2, C.c_int64))
    assert L.nlm_neighbor_search(*arg, None) == 0 and np.array_equal(rp2, rp0)
    assert L.nlm_neighbor_search(*arg, abi.ptr(cols2, C.c_int32)) == 0
    assert np.array_equal(cols2, cols0)


def test_refusals(gpu):
    rp, cols = gpu.neighbor_search(np.zeros((0, 3)), 0.1)
    assert list(rp) == [0] and len(cols) == 0
    x = configs.grid2d(9, 9, 1e-3, 0.0, 0)[0]
    for bad, hz, code in ((np.nan, 3e-3, 7), (np.inf, 3e-3, 7), (1e-3, -1.0, 1)):
        y = x.copy()
        y[40, 1] = bad
        with pytest.raises(gpu.NLMError) as e:
            gpu.neighbor_search(y, hz)
        assert e.value.code == code
    with pytest.raises(gpu.NLMError) as e:  # a row of more than 512
        gpu.neighbor_search(configs.grid2d(30, 30, 1e-3, 0.0, 0)[0], 1.0)
    assert e.value.code == 1
