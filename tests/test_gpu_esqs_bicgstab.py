"""BiCGSTAB on a system whose first iteration all but solves it: two free nodes,
the first of them loaded, the second with a volume eps times the others.  J is
then [[a, O(eps)], [c, d]], and after one iteration the residual is O(eps) of
the load: above lin_tol, far below what r.r = s.s - omega t.s can resolve
(the square root of 2^-53).  Two unknowns take two iterations."""
import numpy as np
import pytest

from nlmech_gb300 import configs
from nlmech_gb300.decks import BC, MaterialDeck, Problem

pytestmark = pytest.mark.gpu


def _chain(eps, dim, n=9):
    h = 0.1
    x, vol = configs.grid2d(n, 1, h, 0.0, 0)
    x[:, 1] = 0.0
    vol = np.full(n, h)
    vol[5] = eps * h
    one = dict(spatial_fn="constant", spatial_params=[1.0])
    reg = dict(region="line") if dim == 1 else dict(region="rectangle", y1=-1.0, y2=1.0)
    at = lambda i: dict(x1=x[i, 0] - 0.4 * h, x2=x[i, 0] + 0.4 * h, **reg)
    fixed = dict(time_fn="constant", time_params=[0.0], **one)
    dirs = list(range(1, dim + 1))
    ubc = [BC(direction=dirs, **fixed, **at(i)) for i in range(n) if i not in (4, 5)]
    if dim == 2:
        ubc += [BC(direction=[2], **fixed, **at(i)) for i in (4, 5)]
    fbc = [BC(direction=[1], time_fn="linear", time_params=[4.0], **one, **at(4))]
    mat = MaterialDeck(kind="ElasticState", density=1200.0, K=4000.0, G=1500.0, E=4000.0)
    return Problem(dim=dim, x=x, volume=vol, horizon=3 * h, mesh_size=h, material=mat,
                   ubc=ubc, fbc=fbc)


@pytest.mark.parametrize("dim", [1, 2])
def test_two_unknowns_take_two_iterations(gpu, dim):
    its = []
    for k in range(12):
        eps = 10.0 ** (-8.5 - 0.15 * k)  # down to 7e-11, lin_tol 1e-12
        q = gpu.ESQSModel(_chain(eps, dim), gpu.esqs_params(max_iters=1, tol=1e-30, jacobian=1,
                                                            lin_tol=1e-12, dt=0.25))
        its.append(q.solve(1)[1][0])
        u = q.get()[0]
        assert np.isfinite(u).all() and abs(u[4, 0]) > 0 and abs(u[5, 0]) > 0
    assert its == [2] * len(its), its
