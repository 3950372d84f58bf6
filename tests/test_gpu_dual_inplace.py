"""The dual-energy subtraction written over one of its inputs, with the slice
entropies: the histogram is of the inputs as they were given, so outputs and
entropies are those of the call with an output of its own, bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NX, NY, NZ = 37, 29, 5


@pytest.mark.parametrize("over", ["he", "le"])
@pytest.mark.parametrize("weights", [[0.3], [0.3, 0.7, 0.5]], ids=["one", "three"])
@pytest.mark.parametrize("mask", [None, 0.35])
def test_entropies_over_an_input(over, weights, mask):
    from newrecon_gb300 import dual_energy, native

    native.load()
    rng = np.random.default_rng(3)
    n = NX * NY * NZ
    # he - le w and the histogram's bins differ in every voxel once he or le is lost
    he = rng.uniform(0.3, 1.0, n).astype(np.float32)
    le = rng.uniform(0.0, 0.9, n).astype(np.float32)
    kw = dict(slice_shape=(NX, NY), entropy_slice=3, mask_level=mask)
    ref, ent = dual_energy.subtract(torch.from_numpy(he).cuda(), torch.from_numpy(le).cuda(),
                                    weights, **kw)
    # the input is a row of the output; n is odd, so only row 0 is aligned
    out = torch.empty(len(weights), n, device="cuda")
    v = {"he": torch.from_numpy(he).cuda(), "le": torch.from_numpy(le).cuda()}
    out[0] = v[over]
    v[over] = out[0]
    d, got = dual_energy.subtract(v["he"], v["le"], weights, out=out, **kw)
    assert torch.equal(d, ref)
    assert got == ent
