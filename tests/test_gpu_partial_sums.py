"""The objective's partials are summed by one block or, from 8192 on, by one-warp
blocks in the same order: the penalty through the workspace has the bits of the
workspace-free one, which always sums in one block, about the line and at partial
counts that leave a warp's rows ragged."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

# penalty partials: 8190, 8192, 8211 and 262,000, with one data partial beside them
SIZES = [(64, 52, 315), (64, 64, 256), (68, 68, 161), (500, 499, 131)]


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%dx%d" % s)
def test_workspace_penalty_has_the_static_bits(size):
    from newrecon_gb300 import native, ostr
    from newrecon_gb300.geometry import POTENTIALS, Geometry, view_angles

    native.load()
    g = Geometry.dbt(*size, 0.5, 1.0, 32, 4, 0.5, 1)
    gen = torch.Generator(device="cuda").manual_seed(sum(size))
    x = 0.05 * torch.rand(g.n_voxels, device="cuda", generator=gen)
    y = torch.full((g.n_bins,), 100.0, device="cuda")
    plan = ostr.OSTR(g, subset_num=1, beta=1.0, delta=0.003, potential="huber")
    plan.setup(view_angles(1, 0.0), y, y)
    got = plan.objective(x)[1]
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    gc = g.to_c()
    native.call("nr_penalty_fp64_static", ctypes.byref(gc), ctypes.c_void_p(x.data_ptr()),
                POTENTIALS["huber"], ctypes.c_float(0.003), ctypes.c_void_p(out.data_ptr()), None)
    assert float(got) == float(out.item())
