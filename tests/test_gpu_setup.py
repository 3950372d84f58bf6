"""The scan set-up (gamma * yry and the curvature d) where its kernels' tiles end:
volumes of one voxel, rows left over from blocks of 16, detectors one bin wide
or high, more rows than a thread walks, zero counts, scatter above the counts,
both gammas, several subset orders.

gamma * yry is the product that the reference-shaped calls give, bit for bit
(the same slab test, the same roundings; those calls are held against the
oracle in test_gpu_ops).  d, the back projection of random data, against the
FP64 oracle to the operator's bars of test_gpu_ops (relative RMSE 5e-5, maximum
2e-4 of scale).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (nx, ny, nz), (BINSx, BINSy)
SIZES = [((1, 1, 1), (6, 5)), ((33, 15, 3), (1, 30)), ((31, 17, 4), (45, 1)),
         ((40, 33, 5), (52, 67)), ((64, 16, 2), (33, 40))]


def product(g, angles, y, scat, mode):
    """gamma * yry by the reference-shaped calls, [view][i][j]."""
    from newrecon_gb300 import ostr

    ostr.set_geometry(g)
    old, ostr.gamma_mode = ostr.gamma_mode, mode
    gam = torch.zeros(y.size, device="cuda")
    ostr.fprojectCB_1R_GPU_OSTR_normprj(gam, angles, np.arange(6, dtype=np.int32), 0, 6)
    ostr.gamma_mode = old
    yd = torch.from_numpy(y).cuda()
    return ostr.compute_gamma_yry(ostr.compute_yry(yd, scat), gam)


@pytest.mark.parametrize("mode", ["length", "chord"])
@pytest.mark.parametrize("size", SIZES, ids=["%dx%dx%d" % s[0] for s in SIZES])
def test_setup_against_oracle(size, mode):
    from newrecon_gb300 import native, ostr
    from newrecon_gb300.geometry import Geometry, view_angles
    from oracle.oracle import Oracle

    native.load()
    (nx, ny, nz), (bx, by) = size
    g = Geometry.dbt(nx, ny, nz, 0.5, 1.0, bx, by, 0.5, 6)
    angles = view_angles(6, 15.0)
    rng = np.random.default_rng(nx + by)
    n = 6 * g.n_bins
    y = rng.poisson(40.0, n).astype(np.float32)
    y[rng.random(n) < 0.1] = 0.0
    idx = np.arange(6, dtype=np.int32)
    O = Oracle(np.float64)
    gamma = O.fp_gamma(g, angles, idx, 0, 6, mode=mode)
    for scat in (None, rng.uniform(0.0, 60.0, n).astype(np.float32)):
        gy = gamma * O.compute_yry(y, scat)
        d = O.bp_sbp(g, gy, idx, angles, 0, 6)
        for subsets in (6, 3):
            plan = ostr.OSTR(g, subset_num=subsets, beta=1.0, delta=0.01, gamma_mode=mode,
                             has_scatter=scat is not None)
            plan.setup(angles, y, np.full(n, 100.0, np.float32), scat)
            got = plan.section("gamma_yry").view(6, by, bx).transpose(1, 2).reshape(-1)
            assert torch.equal(got, product(g, angles, y, scat, mode))
            e = plan.section("d").cpu().numpy().astype(np.float64) - d.ravel()
            assert np.linalg.norm(e) <= 5e-5 * np.linalg.norm(d)
            assert np.abs(e).max() <= 2e-4 * np.abs(d).max()
