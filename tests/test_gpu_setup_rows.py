"""gamma * yry of the set-up on detectors of one to eight rows per thread (the
count goes by the detector's size), with rows left over: bit for bit the product
that the reference-shaped calls give; and the view order and status words that the
same launch writes."""
import numpy as np
import pytest
import torch

from test_gpu_setup import product

pytestmark = pytest.mark.gpu

# detectors of 6 views: 1, 2, 5 and 8 rows per thread
BINS = [(33, 35), (129, 330), (200, 611), (705, 301)]


@pytest.mark.parametrize("bins", BINS, ids=lambda b: "%dx%d" % b)
def test_rows_per_thread(bins):
    from newrecon_gb300 import native, ostr
    from newrecon_gb300.geometry import Geometry, view_angles

    native.load()
    g = Geometry.dbt(60, 40, 5, 0.5, 1.0, *bins, 0.25, 6)
    angles = view_angles(6, 15.0)
    rng = np.random.default_rng(bins[0])
    n = 6 * g.n_bins
    y = rng.poisson(40.0, n).astype(np.float32)
    scat = rng.uniform(0.0, 60.0, n).astype(np.float32)
    plan = ostr.OSTR(g, subset_num=3, beta=1.0, delta=0.01, has_scatter=True)
    plan.ws.fill_(255)
    plan.setup(angles, y, np.full(n, 100.0, np.float32), scat)
    got = plan.section("gamma_yry").view(6, bins[1], bins[0]).transpose(1, 2).reshape(-1)
    assert torch.equal(got, product(g, angles, y, scat, "length"))
    assert plan.section("index").tolist() == [0, 3, 1, 4, 2, 5]
    assert plan.check() == 0
