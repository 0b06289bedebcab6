"""Which form the FP32 Krylov solve takes (krylov_launch 0: one launch where it
fits, 1: the same with an error for a wait that runs out, 2: two launches), that
the one-launch form is the one that runs on the meshes of test_gpu_qs_resident,
and both forms on a plate that fractures."""
import numpy as np
import pytest

from nlmech_gb300 import configs
from test_gpu_qs_resident import CASES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(CASES))
def test_one_launch_runs_where_it_is_chosen(gpu, name):
    p = CASES[name]()
    for k, form in ((0, 1), (1, 1), (2, 2)):
        q = gpu.QSModel(p, gpu.qs_params(krylov_launch=k))
        assert q.krylov_form() == form
        q.load_step()
        assert q.krylov_form() == form
    # only a launch that waits can run out of time
    kw = dict(barrier_extra=1, wait_limit_s=0.02)
    q = gpu.QSModel(p, gpu.qs_params(krylov_launch=1, **kw))
    with pytest.raises(gpu.NLMError) as e:
        q.load_step()
    assert e.value.code == 4  # NLM_ERR_TIMEOUT
    # krylov_launch = 0 goes over to two launches, and says so: the same solves
    # as with 2
    qa = gpu.QSModel(p, gpu.qs_params(krylov_launch=0, **kw))
    qb = gpu.QSModel(p, gpu.qs_params(krylov_launch=2, **kw))
    assert (qa.krylov_form(), qb.krylov_form()) == (1, 2)
    qa.load_step(), qb.load_step()
    assert (qa.krylov_form(), qb.krylov_form()) == (2, 2)
    assert np.array_equal(qa.state(), qb.state())


def test_forms_agree_on_a_fracturing_plate(gpu):
    """Every load step converges to the 1e-8 relative residual in both; bonds
    break at intermediate iterates, so up to 1 % of the broken bonds and of the
    displacement differ, as between the FP32 solves and the oracle's."""
    p = configs.qs_plate(48, h=5e-4, du=1e-6)
    kw = dict(lin_tol=1e-6, max_newton=60)
    qa = gpu.QSModel(p, gpu.qs_params(krylov_launch=1, **kw))
    qb = gpu.QSModel(p, gpu.qs_params(krylov_launch=2, **kw))
    for k in range(4):
        sa, sb = qa.load_step(), qb.load_step()
        assert sa["res_final"] <= 1e-8 * sa["res_plain"], (k, sa)
        assert sb["res_final"] <= 1e-8 * sb["res_plain"], (k, sb)
    assert (qa.krylov_form(), qb.krylov_form()) == (1, 2)
    ba, bb = qa.bond_state(), qb.bond_state()
    assert np.count_nonzero(bb) > 1000
    assert np.count_nonzero(ba != bb) <= 0.01 * np.count_nonzero(bb)
    ua, ub = qa.state(), qb.state()
    assert np.linalg.norm(ua - ub) <= 1e-2 * np.linalg.norm(ub)
