"""The reference-shaped back projector and OS-SART update by a thread per voxel
(small and thin volumes) give the bits of the tiled forms: parts of a volume, back
projected as volumes of their own, against the whole one's part.  Parts of one
voxel, about the block's 128, one row, column or line of planes; more views than
either form holds at a time."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# whole volume, views: tiles of four columns per thread and of one
WHOLE = [((300, 290, 9), 67), ((64, 64, 30), 33)]
# offset and size of the part
PARTS = [((17, 9, 3), (1, 1, 1)), ((0, 60, 8), (43, 3, 1)), ((7, 1, 5), (16, 8, 1)),
         ((3, 2, 0), (1, 62, 9)), ((0, 31, 0), (64, 1, 9)), ((63, 63, 0), (1, 1, 9)),
         ((1, 0, 2), (33, 33, 7))]


@pytest.mark.parametrize("whole", WHOLE, ids=lambda w: "%dx%dx%d-%d" % (*w[0], w[1]))
def test_parts_have_the_whole_volumes_bits(whole):
    from newrecon_gb300 import native, ostr, sart
    from newrecon_gb300.geometry import Geometry, view_angles

    native.load()
    (nx, ny, nz), A = whole
    # binary sizes, so that the shifted origins are exact; a detector smaller than
    # the volume's shadow
    g = Geometry.dbt(nx, ny, nz, 0.5, 1.0, nx, ny - 9, 0.5, A)
    gen = torch.Generator(device="cuda").manual_seed(nx)
    prj = torch.randn(A * g.n_bins, device="cuda", generator=gen)
    base = torch.rand(nz, ny, nx, device="cuda", generator=gen)
    prior = torch.randn(nz, ny, nx, device="cuda", generator=gen)
    ang = torch.from_numpy(np.asarray(view_angles(A, 30.0), np.float32)).cuda()
    idx = torch.arange(A, dtype=torch.int32, device="cuda").flip(0).contiguous()

    def run(geom, x, pr):
        ostr.set_geometry(geom)
        a, b, c = (x.clone().view(-1) for _ in range(3))
        ostr.bprojectCB_GPU_SBP(a, prj, idx, ang, 0, A)
        sart.bprojectCB_4B_GPU_SART_R(b, prj, pr.contiguous().view(-1), idx, ang, 0, A, 0.7, -0.3)
        ostr.bprojectCB_GPU_SBP(c, prj, idx, ang, 2, 3)
        return [t.view(x.shape) for t in (a, b, c)]

    full = run(g, base, prior)
    for (ox, oy, oz), (px, py, pz) in PARTS:
        s = dataclasses.replace(g, nx=px, ny=py, nz=pz, x_p0=g.x_p0 + 0.5 * ox,
                                y_p0=g.y_p0 + 0.5 * oy, z_p0=g.z_p0 + oz)
        cut = (slice(oz, oz + pz), slice(oy, oy + py), slice(ox, ox + px))
        for w, p in zip(full, run(s, base[cut].contiguous(), prior[cut])):
            assert torch.equal(w[cut], p), (px, py, pz)
