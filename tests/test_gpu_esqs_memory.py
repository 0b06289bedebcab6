"""What a quasi-static ElasticState model keeps on the device per bond: its block of
J (mdim^2 doubles), the two differences that other rows read (2 mdim doubles), a
column id, and the mesh's own lists."""
import pytest

from nlmech_gb300 import configs
from nlmech_gb300.decks import BC, MaterialDeck, Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, (600, 600)), (3, (48, 48, 48))])
def test_bytes_per_bond(gpu, dim, n):
    torch = pytest.importorskip("torch")
    h = 0.1
    x, vol = (configs.grid3d if dim == 3 else configs.grid2d)(*n, h, 0.05, 3)
    ubc = [BC(region="cuboid" if dim == 3 else "rectangle", x1=-1.0, x2=2.5 * h, y1=-1.0, y2=100.0,
              z1=-1.0, z2=100.0, direction=list(range(1, dim + 1)), time_fn="constant",
              time_params=[0.0], spatial_fn="constant", spatial_params=[1.0])]
    p = Problem(dim=dim, x=x, volume=vol, horizon=3 * h, mesh_size=h, ubc=ubc,
                material=MaterialDeck(kind="ElasticState", density=1200.0, K=4000.0, G=1500.0))
    nnz = int(gpu.neighbor_search(x, p.horizon, dim)[0][-1])
    gpu.ESQSModel(p).close()
    torch.empty(1, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    q = gpu.ESQSModel(p)
    taken = free - torch.cuda.mem_get_info()[0]
    q.close()
    # the mesh: two column lists and their padding (12 bytes); vectors and node
    # data: 120 doubles a node at most
    need = nnz * (8 * dim * dim + 16 * dim + 4 + 12) + 960 * p.n
    assert nnz > 5_000_000
    assert taken <= need + (64 << 20), (taken / nnz, need / nnz)
