"""The 32 -> 32 convolution (runs of rows, two planes per run) at the sizes where
its tiles and runs end: one voxel, x tiles of 127, 128 and 129 columns, an odd
plane left over, more runs than SMs, runs longer than the accumulator cycle.

Forward and gradients against the FP64 NumPy network that rounds to BF16 where
the GPU stores BF16.  What is left is the FP32 accumulation order and the BF16
rounding flips it causes: relative L2 error 2e-3 (outputs), 1e-2 (gradients),
the bars of test_gpu_cnn.py.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DIMS = [(1, 1, 1, 1), (127, 5, 3, 1), (128, 23, 2, 1), (129, 7, 1, 80), (3, 9, 7, 3)]


def rel(a, b):
    a = np.asarray(a, np.float64).ravel()
    b = np.asarray(b, np.float64).ravel()
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


@pytest.mark.parametrize("dims", DIMS, ids=["x".join(map(str, d)) for d in DIMS])
def test_row_runs(dims):
    from newrecon_gb300 import native, warmstart
    from oracle import cnn_oracle as co

    native.load()
    nx, ny, nz, nb = dims
    rng = np.random.default_rng(sum(dims))
    x = rng.uniform(0.0, 0.1, size=(nb, nz, ny, nx)).astype(np.float32)
    t = (x + rng.normal(scale=0.01, size=x.shape)).astype(np.float32)
    p = co.init_params(6, last_scale=0.5)
    net = warmstart.WarmStartCNN(p, scale=20.0)
    xd, td = torch.from_numpy(x.ravel()).cuda(), torch.from_numpy(t.ravel()).cuda()
    out = net.forward(xd, dims).cpu().numpy()
    _, grad = net.loss_grad(xd, td, dims)
    net.check()
    grad = grad.cpu().numpy()
    f, _ = co.forward(p, x, 20.0, bf=True)
    ref = np.maximum(x + f / 20.0, 0.0)
    assert rel(out, ref) < 2e-3
    _, gref = co.loss_grad(p, x, t, 20.0, bf=True)
    wo, _, _ = co.param_offsets()
    for l in range(6):
        ni, no = co.LAYERS[l]
        sw = slice(wo[l], wo[l] + 27 * ni * no)
        assert rel(grad[sw], gref[sw]) < 1e-2, (l, rel(grad[sw], gref[sw]))
