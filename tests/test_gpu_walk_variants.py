"""Every variant of the subset projection gives the same bits: gather batches of
2, 4 and 8, direct or staged by TMA, on rows shorter than a warp's list, around
its length and several lists long, few and many rows per plane, and views that
the general walk takes.

And the direct form against the FP64 oracle at up to 25 degrees to the projector's
own bars of test_gpu_ops (relative RMSE 5e-6, maximum 1e-4 of scale).  With no
counts and a blank scan of 1 the gradient h is -exp(-line); the volume is scaled
to lines of up to 1, where expf's ulp and the product's rounding move
a line by at most 1.8e-7.
"""
import numpy as np
import pytest
import torch

from test_gpu_walk import CASES, SPAN, geometry

pytestmark = pytest.mark.gpu

NARROW = np.radians([-12.0, -5.0, 0.0, 7.0, 12.0])
TALL = {
    # lists of about 225 to 270 entries in rows that TMA can describe
    "nz%d" % nz: (geometry(24, 20, nz, vz=0.25, bins=(40, 36)), SPAN)
    for nz in (225, 240, 245, 247, 248, 249, 250, 252, 254, 256)
}
TALL["five_lists"] = (geometry(32, 48, 900, vz=0.1, bins=(40, 80), sourceR=300.0), SPAN)
# about 110 rows per plane, two planes to a list; and 250, where the general walk takes over
DENSE = {
    "dense": (geometry(8, 400, 4, vx=0.2, vy=0.2, vz=100.0, bins=(20, 90), b=2.0), NARROW),
    "denser": (geometry(8, 400, 4, vx=0.2, vy=0.2, vz=100.0, bins=(20, 90), b=4.0), NARROW),
}
VARIANTS = [(2, False), (4, False), (8, False), (2, True), (4, True)]


def project(g, angles, x, batch, stage):
    from newrecon_gb300 import native, ostr

    native.load()
    n = g.n_angles * g.n_bins
    plan = ostr.OSTR(g, subset_num=1, beta=1.0, delta=0.01, stage=stage)
    plan.params.fp_batch = batch
    plan.setup(np.asarray(angles, np.float32), torch.zeros(n, device="cuda"),
               torch.ones(n, device="cuda"))
    plan.project(x, 0)
    assert plan.check() == 0
    return plan.section("h").clone()


@pytest.mark.parametrize("name", [*CASES, *TALL, *DENSE])
def test_variants_give_the_same_bits(name):
    g, angles = {**CASES, **TALL, **DENSE}[name]
    rng = np.random.default_rng(7)
    x = torch.from_numpy((rng.random(g.n_voxels, dtype=np.float32) * 0.02)).cuda()
    h = [project(g, angles, x, k, stage) for k, stage in VARIANTS]
    assert float((h[0] + 1.0).abs().max()) > 0
    for v, o in zip(VARIANTS[1:], h[1:]):
        assert torch.equal(o, h[0]), v


@pytest.mark.parametrize("name", [n for n in CASES if n != "steep"] + [*TALL])
def test_against_oracle(name):
    from oracle.oracle import Oracle

    g, angles = {**CASES, **TALL}[name]
    angles = np.asarray(angles, np.float32)
    rng = np.random.default_rng(11)
    A = g.n_angles
    x = rng.random(g.n_voxels, dtype=np.float32)
    O, idx = Oracle(np.float64), np.arange(A, dtype=np.int32)
    x = (x / np.abs(O.fp_ostr(g, x, angles, idx, 0, A)).max()).astype(np.float32)
    ref = O.fp_ostr(g, x, angles, idx, 0, A).reshape(A, g.nbx, g.nby).transpose(0, 2, 1)
    h = project(g, angles, torch.from_numpy(x).cuda(), 0, False)
    d = -np.log(-h.cpu().numpy().astype(np.float64).reshape(ref.shape)) - ref
    assert np.linalg.norm(d) <= 5e-6 * np.linalg.norm(ref)
    assert np.abs(d).max() <= 1e-4 * np.abs(ref).max()


def test_batch_modes_give_the_same_bits():
    """Cases whose rows take several lists: shared launches and one after another."""
    from newrecon_gb300 import native, ostr

    native.load()
    rng = np.random.default_rng(5)
    cases = []
    for name in ("nz250", "five_lists"):
        g, angles = TALL[name]
        n = g.n_angles * g.n_bins
        cases.append(dict(geom=g, angles=np.asarray(angles, np.float32),
                          prj=rng.poisson(900.0, n).astype(np.float32),
                          blank=np.full(n, 1e3, np.float32), subset_num=5, iter_num=1, beta=5.0,
                          delta=0.01, potential="huber"))
    a, b = (ostr.Batch(cases, mode=m).run() for m in ("shared", "sequential"))
    for u, v in zip(a, b):
        assert float(u.max()) > 0 and torch.equal(u, v)
