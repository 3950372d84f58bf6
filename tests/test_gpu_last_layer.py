"""The last layer's second pass adds the residual itself, four voxels per thread
where the rows and the caller's tensors are 16-byte aligned: every alignment of
the input and the output, and the in-place call, give the same bits.  A row that
is not a multiple of four voxels takes the scalar form at any alignment."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [4, 6, 128, 1028])
def test_alignment_and_in_place(nx):
    import ctypes

    from newrecon_gb300 import native, warmstart
    from oracle import cnn_oracle as co

    native.load()
    dims = (nx, 3, 2, 1)
    n = nx * 6
    rng = np.random.default_rng(nx)
    x = rng.uniform(0.0, 0.1, size=n).astype(np.float32)
    net = warmstart.WarmStartCNN(co.init_params(6, last_scale=0.5), scale=20.0)
    d, ws = net._workspace(dims, False)

    def call(off_in, off_out, in_place=False):
        xin = torch.zeros(n + 4, device="cuda")[off_in:off_in + n]
        xin.copy_(torch.from_numpy(x))
        out = xin if in_place else torch.full((n + 8,), 7.0, device="cuda")[off_out:off_out + n]
        native.call("nr_cnn_forward", ctypes.byref(d),
                    ctypes.c_void_p(net.params.data_ptr()), ctypes.c_void_p(xin.data_ptr()),
                    ctypes.c_float(20.0), ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(ws.data_ptr()),
                    ctypes.c_size_t(ws.numel()), ctypes.c_void_p(0))
        torch.cuda.synchronize()
        return out.cpu()

    want = call(0, 0)
    assert torch.equal(net.forward(torch.from_numpy(x).cuda(), dims).cpu(), want)
    for off_in in (0, 1):
        for off_out in (0, 2, 3):
            assert torch.equal(call(off_in, off_out), want), (off_in, off_out)
        assert torch.equal(call(off_in, 0, in_place=True), want), off_in
