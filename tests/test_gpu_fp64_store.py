"""FP64 steps over the bond store against the kernels that recompute every
bond's geometry (NLM_DECOMP_THREAD1): the same operations rounded in the same
order, so states and bond bits are equal bit for bit.  Rows shorter and longer
than one 32-bit bond word, ragged last slices, every term of the bond force,
and every team size (lanes per node) the rule on the node count gives."""
import numpy as np
import pytest

from nlmech_gb300 import abi, configs

pytestmark = pytest.mark.gpu

RNP = [dict(), dict(contact=True, speed=60.0), dict(nofail=True, speed=40.0),
       dict(infl=(1, [])), dict(infl=(2, [])), dict(irreversible=False, speed=40.0),
       dict(scheme=abi.CENTRAL_DIFFERENCE, speed=40.0), dict(ratio=5, speed=40.0),
       dict(vol=True)]


def _plate(ratio=3, speed=1.0, contact=False, nofail=False, infl=None, irreversible=True,
           scheme=abi.VELOCITY_VERLET, vol=False):
    p = configs.rnp_plate(37, 1e-3, ratio, 0.012, speed, 2e-8, 1, seed=4, ny=29)
    m = p.material
    m.apply_contact, m.irreversible, p.scheme = contact, irreversible, scheme
    if infl:
        m.influence_type, m.influence_params = infl
    if nofail:
        p.no_fail, p.no_fail_tol = abi.NOFAIL_COMPUTE, 2.25 * ratio * 1e-3
    if vol:
        p.volume = p.volume * np.random.default_rng(3).uniform(0.8, 1.2, p.n)
    return p


def _cube(dim, sc, compat=False, strain=False):
    p = configs.elastic_state_cube(9, 1e-3, sc=sc, seed=2, ref_compat=compat)
    p.v0 = 40.0 * p.v0
    if dim == 2:
        p.x, p.volume = configs.grid2d(35, 21, 1e-3, 0.05, 2)
        p.dim, p.cracks = 2, []
        p.v0 = np.random.default_rng(5).uniform(-5, 5, p.x.shape) * [1, 1, 0]
        p.material.plane_strain = strain
    return p


def _same(gpu, p, steps=60):
    a, b = gpu.FDModel(p), gpu.FDModel(p, decomposition=abi.DECOMP_THREAD1)
    for m in (a, b):
        m.run(steps)
    for q, r in zip(a.state(), b.state()):
        assert np.isfinite(r).all() and np.array_equal(q, r)
    assert np.array_equal(a.bond_state(), b.bond_state())
    return b


@pytest.mark.parametrize("opt", RNP, ids=lambda o: "-".join(o) or "plain")
def test_rnp_store_same_bits(gpu, opt):
    p = _plate(**opt)
    cut = gpu.FDModel(p).count_broken()
    b = _same(gpu, p)
    if opt.get("speed", 0) >= 40 and opt.get("irreversible", True):
        assert b.count_broken() > cut  # the slow branch ran


def test_rnp_store_same_bits_3d(gpu):
    p = configs.rnp_plate(2, 1e-3, 3, 0.0, 30.0, 2e-8, 1)
    p.dim, p.ubc = 3, []
    p.x, p.volume = configs.grid3d(11, 9, 7, 1e-3, 0.05, 1)
    p.v0 = np.random.default_rng(6).uniform(-2, 2, p.x.shape)
    _same(gpu, p)


@pytest.mark.parametrize("nx", [64, 140, 190])
def test_rnp_store_same_bits_larger_teams(gpu, nx):
    p = configs.rnp_plate(nx, 1e-3, 3, 0.02, 40.0, 2e-8, 1, seed=5, ny=nx - 3)
    _same(gpu, p, 12)


@pytest.mark.parametrize("n", [16, 24, 33])
def test_es_store_same_bits_larger_teams(gpu, n):
    p = configs.elastic_state_cube(n, 1e-3, sc=5e-4, seed=3)
    p.v0 = 20.0 * p.v0
    _same(gpu, p, 6)


@pytest.mark.parametrize("case", [(3, 5e-4, False, False), (3, 0.0, False, False),
                                  (3, 5e-4, True, False), (2, 5e-4, False, False),
                                  (2, 5e-4, False, True)])
def test_es_store_same_bits(gpu, case):
    _same(gpu, _cube(*case), 40)


@pytest.mark.parametrize("where", ["coincident", "far"])
def test_store_special_values(gpu, where):
    """Two nodes in one place (zero length, 0 / 0) and a displacement whose
    stretch overflows the threshold's range give what the other path gives."""
    p = _plate()
    if where == "coincident":
        p.x[400] = p.x[401]
    else:
        p.u0 = np.zeros_like(p.x)
        p.u0[400, 0] = 1e200
    a, b = gpu.FDModel(p), gpu.FDModel(p, decomposition=abi.DECOMP_THREAD1)
    for m in (a, b):
        m.run(1)
    for q, r in zip(a.state(), b.state()):
        assert np.array_equal(q, r, equal_nan=True)
    assert np.array_equal(a.bond_state(), b.bond_state())
