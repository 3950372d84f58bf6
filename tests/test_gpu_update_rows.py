"""The fused update's two-rows-per-thread walk where it can go wrong: volumes of
one cell, tiles cut short in x and y (a last row without its partner), chunks
of one to three planes, several views per subset.

Against the FP64 oracle after one iteration (relative RMSE 1e-4, the OSTR
loop's bar), and every chunk depth -- the one chosen by size among them -- bit
for bit.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (3, 2, 1), (31, 8, 4), (33, 9, 5), (64, 7, 3), (97, 17, 9)]


@pytest.mark.parametrize("subsets", [6, 2])
@pytest.mark.parametrize("shape", SHAPES, ids=["x".join(map(str, s)) for s in SHAPES])
def test_edges_against_oracle(shape, subsets):
    from newrecon_gb300 import native, ostr
    from newrecon_gb300.geometry import Geometry, view_angles
    from newrecon_gb300.phantom import poisson_counts
    from oracle.oracle import Oracle

    native.load()
    nx, ny, nz = shape
    g = Geometry.dbt(nx, ny, nz, 0.5, 1.0, nx + 12, ny + 9, 0.5, 6)
    angles = view_angles(6, 15.0)
    rng = np.random.default_rng(nx + 7 * ny)
    xt = (rng.random(g.n_voxels, dtype=np.float32) * 0.05).astype(np.float32)
    O = Oracle(np.float64)
    line = O.fp_ostr(g, xt, angles, np.arange(6, dtype=np.int32), 0, 6)
    y = poisson_counts(line, 1e4, nx)
    b = np.full_like(y, 1e4)
    yd, bd = torch.from_numpy(y).cuda(), torch.from_numpy(b).cuda()
    for pot in ("q2", "lange", "hyperbola", "huber"):
        ref = O.reconstruct(g, angles, y, b, subset_num=subsets, iter_num=1, beta=20.0,
                            delta=0.01, potential=pot)
        outs = []
        for planes in (0, 8, 16, 32):
            plan = ostr.OSTR(g, subset_num=subsets, beta=20.0, delta=0.01, potential=pot)
            plan.params.upd_planes = planes
            plan.setup(angles, yd, bd)
            x = torch.zeros(g.n_voxels, device="cuda")
            plan.iterate(x, 1)
            assert plan.check() == 0
            outs.append(x)
        for o in outs[1:]:
            assert torch.equal(o, outs[0]), (pot, shape)
        got = outs[0].cpu().numpy().astype(np.float64)
        err = np.linalg.norm(got - ref) / max(np.linalg.norm(ref), 1e-30)
        assert err < 1e-4, (pot, err)
