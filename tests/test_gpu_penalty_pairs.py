"""The hyperbola's penalty adds its neighbour terms two to a division; a term whose
partner lies outside the volume, and the thirteenth, have one of their own.  Volumes
of one voxel, row or plane and small blocks, where every combination occurs, against
the sum over pairs in NumPy doubles: 13 terms of at most ten roundings each and the
sum of the partials stay under 1e-13 relative."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (2, 1, 1), (1, 2, 1), (1, 1, 2), (5, 1, 1), (1, 7, 3), (33, 5, 2), (32, 4, 3)]


@pytest.mark.parametrize("pot", ["hyperbola", "lange"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%dx%d" % s)
def test_penalty_pairs(size, pot):
    from newrecon_gb300 import native
    from newrecon_gb300.geometry import POTENTIALS, Geometry

    native.load()
    nx, ny, nz = size
    g = Geometry.dbt(nx, ny, nz, 0.5, 1.0, 8, 8, 0.5, 1)
    v = np.random.default_rng(nx + ny + nz).uniform(0, 0.05, (nz, ny, nx)).astype(np.float32)
    delta, want, zr = float(np.float32(0.003)), 0.0, 2.0
    x = v.astype(np.float64)
    for dz, dy, dx in [(1, a, b) for a in (-1, 0, 1) for b in (-1, 0, 1)] + \
            [(0, 1, b) for b in (-1, 0, 1)] + [(0, 0, 1)]:
        w = 1.0 / np.sqrt(float(dx * dx + dy * dy) + float(dz * dz) * zr * zr)
        for z in range(nz - dz):
            for y in range(max(0, -dy), ny - max(0, dy)):
                for c in range(max(0, -dx), nx - max(0, dx)):
                    u = abs(x[z, y, c] - x[z + dz, y + dy, c + dx]) / delta
                    psi = u * u / (np.sqrt(1 + u * u) + 1) if pot == "hyperbola" else u - np.log1p(u)
                    want += w * delta * delta * psi
    xd = torch.from_numpy(v.ravel()).cuda()
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    gc = g.to_c()
    native.call("nr_penalty_fp64_static", ctypes.byref(gc), ctypes.c_void_p(xd.data_ptr()),
                POTENTIALS[pot], ctypes.c_float(delta), ctypes.c_void_p(out.data_ptr()), None)
    assert abs(float(out.item()) - want) <= 1e-13 * abs(want)
