"""The reference-shaped back projector and OS-SART update by tiles of 32 x 32
voxels: a voxel's value depends neither on its place in a tile, nor on the planes
and views its block takes, nor on whether its warp takes the form without edge
tests.  A part of a volume, back projected as a volume of its own (sizes about
the tile's edge, one row, one column; few tiles and many), has the bits of the
whole one's part; the whole one is compared with the FP64 oracle elsewhere."""
import dataclasses

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# whole volume, views: several planes per block, and two chunks of views
WHOLE = [((640, 640, 13), 3), ((100, 70, 9), 33)]
# offset and size of the part
PARTS = [((0, 0, 0), (31, 33, 5)), ((37, 21, 2), (32, 32, 7)), ((5, 3, 1), (95, 1, 8)),
         ((64, 38, 8), (1, 32, 1)), ((3, 0, 0), (97, 65, 9))]


@pytest.mark.parametrize("part", PARTS, ids=lambda p: "%dx%dx%d" % p[1])
@pytest.mark.parametrize("whole", WHOLE, ids=lambda w: "%dx%dx%d-%d" % (*w[0], w[1]))
def test_parts_have_the_whole_volumes_bits(whole, part):
    from newrecon_gb300 import native, ostr, sart
    from newrecon_gb300.geometry import Geometry, view_angles

    native.load()
    (nx, ny, nz), A = whole
    (ox, oy, oz), (px, py, pz) = part
    # binary sizes, so that the shifted origins are exact; a detector smaller than
    # the volume's shadow
    g = Geometry.dbt(nx, ny, nz, 0.5, 1.0, nx, ny - 9, 0.5, A)
    s = dataclasses.replace(g, nx=px, ny=py, nz=pz, x_p0=g.x_p0 + 0.5 * ox,
                            y_p0=g.y_p0 + 0.5 * oy, z_p0=g.z_p0 + oz)
    gen = torch.Generator(device="cuda").manual_seed(nx + px)
    prj = torch.randn(A * g.n_bins, device="cuda", generator=gen)
    base = torch.rand(nz, ny, nx, device="cuda", generator=gen)
    prior = torch.randn(nz, ny, nx, device="cuda", generator=gen)
    ang = torch.from_numpy(np.asarray(view_angles(A, 30.0), np.float32)).cuda()
    idx = torch.arange(A, dtype=torch.int32, device="cuda").flip(0).contiguous()
    cut = (slice(oz, oz + pz), slice(oy, oy + py), slice(ox, ox + px))

    def run(geom, x, pr):
        ostr.set_geometry(geom)
        a, b = x.clone().view(-1), x.clone().view(-1)
        ostr.bprojectCB_GPU_SBP(a, prj, idx, ang, 0, A)
        sart.bprojectCB_4B_GPU_SART_R(b, prj, pr.contiguous().view(-1), idx, ang, 0, A, 0.7, -0.3)
        return a.view(x.shape), b.view(x.shape)

    for w, p in zip(run(g, base, prior), run(s, base[cut].contiguous(), prior[cut])):
        assert torch.equal(w[cut], p)
