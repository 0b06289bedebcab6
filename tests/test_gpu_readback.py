"""Read-back of the fields into arrays that a program keeps: their pages are
resident, so no thread is started to make them so."""
import threading

import numpy as np
import pytest

from nlmech_gb300 import abi, configs

pytestmark = pytest.mark.gpu


def _next_thread_id():
    ids = []
    t = threading.Thread(target=lambda: ids.append(threading.get_native_id()))
    t.start()
    t.join()
    return ids[0]


def test_kept_arrays_start_no_thread(gpu):
    """Thread ids are handed out in order: 40 read-backs that start a thread
    each use 40 of them (other processes only add to the count, so the least
    of three attempts is taken)."""
    p = configs.rnp_plate(260, 1e-3, 3, 0.05, 2e-4, 1e-7, 1, ny=260)
    m = gpu.FDModel(p, precision=abi.FP32C)
    m.run(3)
    kept = [np.ones((p.n, 3)) for _ in range(3)]
    assert sum(a.nbytes for a in kept) > 4 << 20
    used = []
    for _ in range(3):
        first = _next_thread_id()
        for _ in range(40):
            gpu._check(gpu.load().nlm_fd_get_state(m.h, *[abi.dptr(a) for a in kept]))
        used.append(_next_thread_id() - first)
    assert min(used) < 40, used
    for a, b in zip(m.state(), kept):  # fresh arrays
        assert np.array_equal(a, b)
