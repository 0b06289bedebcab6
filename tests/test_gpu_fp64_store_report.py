"""An FP64 model for whose bond store there is no room steps all the same, to the
same bits, and its decomposition says so."""
import numpy as np
import pytest

from nlmech_gb300 import abi, configs
from nlmech_gb300.decks import MaterialDeck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["RNPBond", "ElasticState"])
def test_decomposition_tells(gpu, kind):
    torch = pytest.importorskip("torch")
    p = configs.rnp_plate(400, 1e-3, 3, 0.05, 0.1, 2e-8, 5)
    if kind == "ElasticState":
        p.material = MaterialDeck(kind="ElasticState", density=1200.0, K=4e9, G=1.5e9)
        p.cracks = []

    def run():
        m = gpu.FDModel(p, precision=abi.FP64)
        m.run(5)
        return m.decomposition(), m.state()

    dec, ref = run()
    assert dec != abi.DECOMP_THREAD1
    torch.empty(1, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    m = gpu.FDModel(p, precision=abi.FP64)
    taken = free - torch.cuda.mem_get_info()[0]
    m.close()
    torch.cuda.empty_cache()
    # room for the model as it was, not for twice its store
    filler = torch.empty(torch.cuda.mem_get_info()[0] - taken, dtype=torch.uint8, device="cuda")
    try:
        dec, out = run()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert dec == abi.DECOMP_THREAD1
    for a, b in zip(ref, out):
        assert np.array_equal(a, b)
