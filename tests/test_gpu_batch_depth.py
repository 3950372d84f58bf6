"""A batch whose cases leave the update's depth open (chosen by the blocks of them
all: 4, 8 or 16 planes) next to explicit depths, one and several views per subset:
the volumes of the cases run one after another, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (nx, ny, nz), subsets, planes: 4 planes for the first batch, 8 and 16 for the others
BATCHES = {
    "few": [((40, 24, 9), 6, 0), ((33, 17, 5), 6, 0), ((64, 40, 17), 3, 0), ((30, 9, 8), 6, 8)],
    "more": [((320, 200, 31), 6, 0), ((97, 41, 20), 6, 0)],
    "many": [((500, 380, 17), 6, 0), ((120, 60, 33), 6, 32)],
}


@pytest.mark.parametrize("name", list(BATCHES))
def test_open_depths(name):
    from newrecon_gb300 import native, ostr
    from newrecon_gb300.geometry import Geometry, view_angles

    native.load()
    rng = np.random.default_rng(3)
    cases = []
    for (nx, ny, nz), subsets, planes in BATCHES[name]:
        g = Geometry.dbt(nx, ny, nz, 0.5, 1.0, nx + 9, ny + 7, 0.5, 6)
        n = 6 * g.n_bins
        cases.append((planes, dict(geom=g, angles=view_angles(6, 15.0),
                                   prj=rng.poisson(900.0, n).astype(np.float32),
                                   blank=np.full(n, 1e3, np.float32), subset_num=subsets,
                                   iter_num=2, beta=5.0, delta=0.01, potential="huber",
                                   **({"upd_planes": planes} if planes else {}))))
    one = ostr.Batch([c for _, c in cases], mode="sequential").run()
    shared = ostr.Batch([c for _, c in cases], mode="shared").run()
    for u, v in zip(one, shared):
        assert float(u.max()) > 0 and torch.equal(u, v)
    for (planes, c), u in zip(cases, one):
        plan = ostr.OSTR(c["geom"], subset_num=c["subset_num"], beta=5.0, delta=0.01,
                         potential="huber")
        plan.params.upd_planes = planes
        plan.setup(c["angles"], c["prj"], c["blank"])
        x = torch.zeros(c["geom"].n_voxels, device="cuda")
        assert torch.equal(plan.iterate(x, 2), u.view(-1))
