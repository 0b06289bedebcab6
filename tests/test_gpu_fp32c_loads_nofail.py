"""FP32C steps under force loads, which the step kernel evaluates itself, and with
no-fail regions, where a row takes the break-free loop unless a no-fail bond ends
at it: against the reference's outputs on every decomposition, with and without
graphs; rows that share a warp with rim rows or do not; batches."""
import os

import numpy as np
import pytest

from nlmech_gb300 import abi, configs

from refcases import GOLDEN_CASES
from test_gpu_refgolden import GOLDEN, _pairs

pytestmark = pytest.mark.gpu

DECOMPS = [abi.DECOMP_THREAD, abi.DECOMP_THREAD1, abi.DECOMP_WARP, abi.DECOMP_TILE,
           abi.DECOMP_TILE_LOCAL]


@pytest.mark.parametrize("dec", DECOMPS)
@pytest.mark.parametrize("name", ["loads_nofail_plate", "nofail_regions_plate",
                                  "force_functions_plate", "angled_regions_plate"])
def test_against_reference_golden(gpu, name, dec):
    """The bar of the FP32C golden test: 1e-5 relative L2, 0.1 % of the bonds."""
    make, steps = GOLDEN_CASES[name]
    z = np.load(os.path.join(GOLDEN, "rnp_ref_%s.npz" % name))
    ref = _pairs(z["rowptr"], z["cols"], z["broken"])
    m = gpu.FDModel(make(), precision=abi.FP32C, decomposition=dec)
    assert m.decomposition() == dec
    m.run(steps)
    out = m.state()
    assert np.linalg.norm(out[0] - z["u"]) <= 1e-5 * np.linalg.norm(z["u"])
    diff = len(_pairs(z["rowptr"], z["cols"], m.bond_state()) ^ ref)
    assert diff <= 1e-3 * max(len(ref), 1), (diff, len(ref))
    g = gpu.FDModel(make(), precision=abi.FP32C, decomposition=dec)
    g.set_graph(10)
    g.run(steps)
    for a, b in zip(out, g.state()):
        assert np.array_equal(a, b)
    assert np.array_equal(m.bond_state(), g.bond_state())


def _plate(circles, steps=1, jitter=0.05):
    p = configs.rnp_plate(96, 1e-3, 3, 0.03, 0.2, 2e-8, steps, jitter=jitter)
    p.no_fail = abi.NOFAIL_DATA
    p.no_fail_tol = 1e-3
    p.nofail_regions = [("Circle", [x, y, 0.0, r]) for x, y, r in circles]
    # strains of a tenth of the critical one: nothing breaks
    p.u0 = np.random.default_rng(5).normal(0.0, 2e-8, size=p.x.shape)
    p.u0[:, 2] = 0.0
    return p


def _rim(p, circles, rowptr, cols):
    """Nodes near a circle (a margin for its edge) or next to such a node."""
    tough = np.zeros(p.n, dtype=bool)
    for x, y, r in circles:
        tough |= np.hypot(p.x[:, 0] - x, p.x[:, 1] - y) <= 1.05 * r
    rim = tough.copy()
    rows = np.repeat(np.arange(p.n), np.diff(rowptr))
    rim[rows[tough[cols]]] = True
    return rim


@pytest.mark.parametrize("jitter", [0.0, 0.05])
@pytest.mark.parametrize("dec", [abi.DECOMP_TILE_LOCAL, abi.DECOMP_THREAD])
def test_a_row_does_not_depend_on_its_warp(gpu, dec, jitter):
    """Two models that differ in no-fail circles elsewhere: the forces of rows that
    no circle reaches are the same bits, though most of them share a warp with
    rim rows in one model (full loop) and with none in the other (break-free)."""
    few = [(0.02, 0.02, 2e-3)]
    many = few + [(0.009 * (i + 1), 0.009 * (j + 1), 0.8e-3)
                  for i in range(9) for j in range(9)]
    out = []
    for circles in (few, many):
        m = gpu.FDModel(_plate(circles, jitter=jitter), precision=abi.FP32C, decomposition=dec)
        m.run(0)
        out.append(m.state()[2])
    p = _plate(many, jitter=jitter)
    rim = _rim(p, many, *m.neighbors())
    assert 0.2 < rim.mean() < 0.8
    assert np.array_equal(out[0][~rim], out[1][~rim])
    assert np.abs(out[0][~rim]).max() > 0


@pytest.mark.parametrize("dec", [None, abi.DECOMP_THREAD, abi.DECOMP_TILE_LOCAL])
def test_batch_with_nofail_layers(gpu, oracle, dec):
    """Some plates with a no-fail layer, some with none; the bar of the batch
    tests."""
    plates = configs.ensemble(nplates=5, nmin=600, nmax=3000, seed=3, steps=300)
    for p in plates[1::2]:
        p.no_fail = abi.NOFAIL_COMPUTE
        p.no_fail_tol = 4.25 * p.mesh_size
    b = gpu.Batch(plates, decomposition=dec)
    b.run(300)
    for s, p in enumerate(plates):
        o = oracle.OracleFD(p)
        rowptr, cols = o.neighbors()
        o.run(300)
        u, uo = b.state(s)[0], o.state()[0]
        assert np.linalg.norm(u - uo) <= 1e-5 * np.linalg.norm(uo), s
        d = len(_pairs(rowptr, cols, b.bond_state(s)) ^ _pairs(rowptr, cols, o.bond_state()))
        assert d <= 1e-3 * max(int(o.bond_state().sum()), 1) + 2, s
