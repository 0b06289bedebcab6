"""The FP32 Krylov solve in one cooperative launch (krylov_launch 0 and 1)
against the two-launch form, which a model falls back to when a wait of that
launch runs out (barrier_extra makes every wait run out): the same Newton
solutions.  Node counts around the blocks' ranges (one block, a last block of
one node, 64 nodes per block, more lanes than bonds), horizon 4h, 3-D."""
import numpy as np
import pytest

from nlmech_gb300 import configs

pytestmark = pytest.mark.gpu


def _run(gpu, p, steps=2, **kw):
    q = gpu.QSModel(p, gpu.qs_params(tol=1e-12, **kw))
    st = [q.load_step() for _ in range(steps)]
    assert all(s["res_final"] <= 1e-12 * s["res_plain"] for s in st), st
    return q.state()


def _block(n):
    p = configs.qs_plate(8, h=5e-4, du=4e-9)
    p.dim, p.cracks = 3, []
    p.x, p.volume = configs.grid3d(*n, 5e-4, 0.02, 3)
    L = n[1] * 5e-4
    for b, (y1, y2) in zip(p.ubc, [(-1.0, 1e-3), (L - 1e-3, 1.0), (L - 1e-3, 1.0)]):
        b.region, b.x1, b.x2, b.y1, b.y2, b.z1, b.z2 = "cuboid", -1.0, 1.0, y1, y2, -1.0, 1.0
    p.ubc[0].direction, p.ubc[1].direction = [1, 2, 3], [1, 3]
    return p


CASES = {"one_block": lambda: configs.qs_plate(8, h=5e-4, du=4e-8),
         "last_block_one_node": lambda: configs.qs_plate(9, h=5e-4, du=4e-8),
         "many": lambda: configs.qs_plate(101, h=5e-4, du=4e-8, jitter=0.05, seed=1),
         "d4h": lambda: configs.qs_plate(60, h=5e-4, ratio=4, du=4e-8, jitter=0.05, seed=2),
         "3d": lambda: _block((9, 14, 7))}


@pytest.mark.parametrize("name", list(CASES))
def test_resident_matches_two_launches(gpu, name):
    """Both end at residuals 1e-12 of the step's, and the displacements differ
    by that times the conditioning of these meshes (below 1e4)."""
    p = CASES[name]()
    ua = _run(gpu, p, krylov_launch=1)
    ub = _run(gpu, p, krylov_launch=0, barrier_extra=1, wait_limit_s=0.02)
    assert np.abs(ua - ub).max() <= 1e-8 * np.abs(ub).max()
