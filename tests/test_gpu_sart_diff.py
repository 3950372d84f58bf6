"""The super-sampled OS-SART loop's normalised difference, bit for bit from the
line integrals of nr_fp_4r: (p - m cos theta) with one rounding, then the quotient
by the chord; the regularised step amplifies a last bit, so it is held."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cos", [False, True])
@pytest.mark.parametrize("size", [(23, 7, 8, 9), (158, 117, 36, 5)])
def test_difference_of_the_supersampled_lines(size, cos):
    from newrecon_gb300 import native, ostr, sart
    from newrecon_gb300.geometry import Geometry, view_angles

    native.load()
    nx, ny, nz, A = size
    g = Geometry.dbt(nx, ny, nz, 0.25, 1.0, int(nx * 1.3) + 1, int(ny * 1.2) + 1, 0.25, A)
    gen = torch.Generator(device="cuda").manual_seed(nx)
    x = torch.rand(g.n_voxels, device="cuda", generator=gen) * 0.05
    line = torch.rand(A * g.n_bins, device="cuda", generator=gen)
    angles = np.asarray(view_angles(A, 15.0), np.float32)
    plan = sart.OSSART(g, subset_num=A, lam=0.4, use_cos=cos, supersample=True)
    plan.setup(angles, line)
    ostr.set_geometry(g)
    m = torch.zeros(A * g.n_bins, device="cuda")
    sart.fproject_4R(x, m, angles, np.arange(A, dtype=np.int32), 0, A, use_cos=False,
                     layout="ji")
    m = m.cpu().numpy().reshape(A, -1)
    p = plan.section("line").cpu().numpy().reshape(A, -1)
    norm = plan.section("norm").cpu().numpy().reshape(A, -1)
    assert (norm > 0).any() and (m > 0).any()
    for a in range(A):
        plan.project(x, a)
        got = plan.section("diff").cpu().numpy()
        # a product of two floats and the sum's leading 64 bits are exact in a long double
        ct = np.longdouble(np.float32(np.cos(np.float64(angles[a])))) if cos else np.longdouble(1)
        dif = (p[a] - m[a].astype(np.longdouble) * ct).astype(np.float32)
        ref = np.zeros_like(dif)
        np.divide(dif, norm[a], out=ref, where=norm[a] != 0)
        assert np.array_equal(got, ref), a
