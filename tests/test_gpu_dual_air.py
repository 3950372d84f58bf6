"""The dual-energy subtraction where the low-energy volume is zero in whole warps, in
parts of one and in single voxels, with zeros of both signs, infinities, NaN and the
smallest numbers in the high-energy volume: bit for bit float(double(he) -
double(le) w) (a NaN where that is one)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WEIGHTS = [0.1, 0.5, -0.3, 0.7, 0.0, 1 / 3]


@pytest.mark.parametrize("mask", [None, 0.25])
@pytest.mark.parametrize("n", [1, 127, 128, 132, 1027, 2048, 70001])
def test_zero_low_energy(n, mask):
    from newrecon_gb300 import dual_energy, native
    from oracle import dual_energy_oracle as de

    native.load()
    rng = np.random.default_rng(n)
    he = rng.uniform(-0.2, 1.0, n).astype(np.float32)
    le = rng.uniform(0.0, 0.9, n).astype(np.float32)
    for k in range(0, n, 256):       # every other warp's 128 voxels, and parts of the next's
        le[k:k + 128] = 0.0
        le[k + 150:k + 171] = -0.0
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-45, 3e38], np.float32)
    for k, v in enumerate(special):  # one warp each
        at = 256 * k + 17
        if at < n:
            he[at] = v
    kw = {} if mask is None else dict(mask_level=mask)
    d, _ = dual_energy.subtract(torch.from_numpy(he).cuda(), torch.from_numpy(le).cuda(), WEIGHTS,
                                **kw)
    with np.errstate(invalid="ignore"):
        ref, _ = de.subtract(he, le, WEIGHTS, **kw)
    got = d.cpu().numpy()
    for g, r in zip(got, ref):
        nan = np.isnan(r)
        assert np.array_equal(np.isnan(g), nan)
        assert np.array_equal(g[~nan].view(np.uint32), r[~nan].view(np.uint32))
