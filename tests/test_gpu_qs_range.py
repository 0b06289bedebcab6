"""The quasi-static solve does not depend on the units: with stiffness and
fracture energy scaled by a power of two, forces and tangent scale exactly, so
the displacements are the same bits.  Scales that take r.r out of FP32's range in
both directions: just past it, where the totals of the two-launch form (FP64) still
hold it, and far past it."""
import dataclasses

import numpy as np
import pytest

from nlmech_gb300 import configs
from test_gpu_qs_resident import _block

pytestmark = pytest.mark.gpu

PLATES = {"2d": lambda: configs.qs_plate(40, h=5e-4, du=4e-8, jitter=0.05, seed=1),
          "3d": lambda: _block((9, 14, 7))}


def _steps(gpu, p, e):
    m = p.material
    p.material = dataclasses.replace(m, E=m.E * 2.0 ** e, Gc=m.Gc * 2.0 ** e)
    q = gpu.QSModel(p, gpu.qs_params(tol=1e-10))
    st = [q.load_step() for _ in range(2)]
    assert all(s["res_final"] <= 1e-10 * s["res_plain"] for s in st), st
    return q.state(), [(s["newton_iters"], s["lin_iters"]) for s in st]


@pytest.mark.parametrize("name", list(PLATES))
def test_power_of_two_units_give_the_same_bits(gpu, name):
    assert PLATES[name]().material.E > 0 and PLATES[name]().material.Gc > 0
    u, its = _steps(gpu, PLATES[name](), 0)
    for e in (28, 30, 32, 50, -100):
        ue, ie = _steps(gpu, PLATES[name](), e)
        assert ie == its, (e, ie, its)
        assert np.array_equal(u, ue), e
