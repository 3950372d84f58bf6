"""The dual-energy subtraction's lists of outputs left to FP64: every output of a
warp's 128 voxels on the list (sixteen weights, products that lie on a rounding
tie), none of them, and both, at the sizes where the warp's voxels and the
16-byte form end.  Bit-identical to float(double(he) - double(le) w)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WEIGHTS = [0.1, 0.2, 0.3, 0.4, 0.6, 0.7, 0.8, 0.9, 1.1, 1.3, 1.7, -0.1, -0.3, 0.5, 0.0, 1 / 3]


@pytest.mark.parametrize("n", [1, 3, 4, 31, 127, 128, 129, 132, 1023, 1024, 1028, 624640])
def test_open_outputs(n):
    from newrecon_gb300 import dual_energy, native
    from oracle import dual_energy_oracle as de

    native.load()
    rng = np.random.default_rng(n)
    # ten times a small integer: the products with tenths are whole, and so many
    # ulps below he that the difference is a tie of the float grid
    a = (10.0 * rng.integers(1, 1 << 18, n)).astype(np.float32)
    b = ((1 << 24) + 2.0 * rng.integers(0, 1 << 20, n)).astype(np.float32)
    for le in (a, np.where(rng.random(n) < 0.5, a, np.float32(0.0)), a * np.float32(0.37)):
        le = le.astype(np.float32)
        d, _ = dual_energy.subtract(torch.from_numpy(b).cuda(), torch.from_numpy(le).cuda(),
                                    WEIGHTS)
        ref, _ = de.subtract(b, le, WEIGHTS)
        got = d.cpu().numpy()
        for k in range(len(WEIGHTS)):
            assert np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32)), WEIGHTS[k]
        # one weight in place, over he and over le
        for over in (0, 1):
            v = [torch.from_numpy(b).cuda(), torch.from_numpy(le).cuda()]
            dual_energy.subtract(v[0], v[1], WEIGHTS[:1], out=v[over])
            assert np.array_equal(v[over].cpu().numpy().view(np.uint32), ref[0].view(np.uint32))
