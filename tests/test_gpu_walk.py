"""The subset loop's projection by row lists (walk.cuh) where it can go wrong:
one-voxel and one-row volumes, rays that enter and leave through the sides,
rows parallel to the grid, lists of every length around the 256 entries a warp
holds (longer rows take the general walk), views at the slope where the general
walk takes over.

With no counts and a blank scan of 1 the subset gradient h is -exp(-line).
The lines are held against the FP64 oracle with four times the projector's bars of test_gpu_ops
(relative RMSE 5e-6, maximum 1e-4 of scale at up to 25 degrees: the same
rounding moves a crossing about 1 / cos further at up to 80).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RMSE, TOL = 2e-5, 4e-4


def geometry(nx, ny, nz, vx=0.5, vy=0.5, vz=1.0, bins=(70, 50), off=(0.0, 0.0), b=0.5, **kw):
    from newrecon_gb300.geometry import Geometry

    d = dict(nx=nx, ny=ny, nz=nz, vx=vx, vy=vy, vz=vz, x_p0=-nx * vx / 2, y_p0=-ny * vy, z_p0=0.0,
             nbx=bins[0], nby=bins[1], bx=b, by=b, x_d0=-bins[0] * b / 2 + off[0],
             y_d0=-bins[1] * b + off[1], detectorR=20.0, sourceR=640.0, sourceY=0.0, n_angles=5)
    d.update(kw)
    return Geometry(**d)


SPAN = np.radians([-25.0, -7.0, 0.0, 12.0, 25.0])
CASES = {
    "one_voxel": (geometry(1, 1, 1, bins=(9, 7)), SPAN),
    "one_row": (geometry(40, 1, 12), SPAN),
    "one_plane": (geometry(40, 24, 1), SPAN),
    "sides": (geometry(24, 16, 60, bins=(120, 70), off=(3.0, 6.0)), SPAN),
    # row 20's bin centre is the source's y: the row never crosses a y plane
    "parallel_row": (geometry(40, 40, 20, bins=(60, 40), sourceY=-9.75), SPAN),
    # fine planes: rows of about 240 to 270 list entries
    "list_full": (geometry(32, 64, 240, vz=0.25, bins=(60, 160), sourceR=220.0), SPAN),
    "list_long": (geometry(16, 12, 400, vz=0.25, bins=(40, 30)), SPAN),
    # tan 63.4 deg = 2: views on both sides of the slope limit, and one beyond
    "steep": (geometry(64, 32, 24, bins=(96, 48), n_angles=4),
              np.radians([55.0, 61.0, 66.0, 80.0])),
    "thick": (geometry(36, 20, 18, vz=2.5, bins=(60, 50)), SPAN),
}


@pytest.mark.parametrize("name", list(CASES))
def test_against_oracle(name):
    from newrecon_gb300 import native, ostr
    from oracle.oracle import Oracle

    native.load()
    g, angles = CASES[name]
    angles = np.asarray(angles, np.float32)
    if name == "steep":  # the shadow of a steep view lies far to one side
        g.x_d0 = -g.nbx * g.bx / 2 - 40.0
    rng = np.random.default_rng(len(name))
    x = (rng.random(g.n_voxels, dtype=np.float32) * 0.05).astype(np.float32)
    A, n = g.n_angles, g.n_angles * g.n_bins
    ref = Oracle(np.float64).fp_ostr(g, x, angles, np.arange(A, dtype=np.int32), 0, A)
    ref = ref.reshape(A, g.nbx, g.nby).transpose(0, 2, 1)   # [view][j][i], as h
    plan = ostr.OSTR(g, subset_num=1, beta=1.0, delta=0.01)
    plan.setup(angles, torch.zeros(n, device="cuda"), torch.ones(n, device="cuda"))
    plan.project(torch.from_numpy(x).cuda(), 0)
    h = plan.section("h").cpu().numpy().astype(np.float64).reshape(ref.shape)
    d = -np.log(-h) - ref
    assert np.abs(ref).max() > 0
    assert np.linalg.norm(d) <= RMSE * np.linalg.norm(ref)
    assert np.abs(d).max() <= TOL * np.abs(ref).max()
