"""The quasi-static Jacobian assembled from per-bond differences: the first
Newton iterates equal the oracle's, which takes central differences of full
forces and a dense LU.  Differences of 1e-7 h leave entries good to about 1e-9,
so iterates agree to 1e-6 of the displacement with room for the conditioning; a
missing or misplaced term shows at order one.  1-D, 2-D and 3-D, rows longer
than a warp (horizon 4h, 3-D), both Jacobian forms."""
import numpy as np
import pytest

from nlmech_gb300 import configs
from nlmech_gb300.decks import BC, MaterialDeck, Problem

pytestmark = pytest.mark.gpu


def _problem(dim, n, ratio=3):
    h = 0.1
    if dim == 3:
        x, vol = configs.grid3d(*n, h, 0.05, 3)
    else:
        x, vol = configs.grid2d(n[0], n[1] if dim == 2 else 1, h, 0.05, 3)
        if dim == 1:
            x[:, 1] = 0.0
    hi = x.max(axis=0) + 1.0
    box = dict(y1=-1.0, y2=hi[1], z1=-1.0, z2=hi[2], region="cuboid" if dim == 3 else "rectangle")
    one = dict(spatial_fn="constant", spatial_params=[1.0])
    mat = MaterialDeck(kind="ElasticState", density=1200.0, K=4000.0, G=1500.0, E=4000.0)
    if dim == 1:
        box["region"] = "line"
    ubc = [BC(x1=-1.0, x2=2.5 * h, direction=list(range(1, dim + 1)), time_fn="constant",
              time_params=[0.0], **one, **box)]
    fbc = [BC(x1=hi[0] - 1.0 - 2.4 * h, x2=hi[0], direction=[min(dim, 2)], time_fn="linear",
              time_params=[4.0], **one, **box)]
    return Problem(dim=dim, x=x, volume=vol, horizon=ratio * h, mesh_size=h, material=mat,
                   ubc=ubc, fbc=fbc)


@pytest.mark.parametrize("case", [(1, (14,)), (2, (12, 9)), (2, (11, 9), 4), (3, (7, 5, 4)),
                                  (3, (9, 4, 4))])
@pytest.mark.parametrize("jac", [0, 1])
@pytest.mark.parametrize("iters", [1, 3])
def test_newton_iterates_match_oracle(gpu, oracle, case, jac, iters):
    p = _problem(*case)
    kw = dict(jacobian=jac, max_iters=iters, tol=1e-14, perturbation=1e-7, lin_max_iters=2000,
              lin_tol=1e-12, dt=0.25)
    o = oracle.OracleQS(p, oracle.QSParams(solver=0, tol_relative=0, **kw))
    q = gpu.ESQSModel(p, gpu.esqs_params(**kw))
    io, ro = o.solve(1)
    ig, lg, rg = q.solve(1)
    assert ig[0] == io[0] == iters
    uo, ug = o.get()[0], q.get()[0]
    assert np.abs(uo).max() > 0
    assert np.abs(ug - uo).max() <= 1e-6 * np.abs(uo).max()
