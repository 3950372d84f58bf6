"""The autotuner compares the default update depth (0: by the volume's size) with
the explicit ones and can keep it (host logic: the timings are given, no GPU)."""
import types

import pytest
import torch

from newrecon_gb300 import autotune


class Plan:
    """What tune() needs of a plan."""

    def __init__(self):
        self.geom = types.SimpleNamespace(nx=256, ny=128, nz=24, nbx=320, nby=160, n_angles=9,
                                          n_voxels=8)
        self.params = types.SimpleNamespace(fp_batch=0, fp_stage=0, upd_planes=0, upd_tile=0,
                                            subset_num=9, potential=1, has_scatter=0)
        self.ws = torch.empty(1)

    def project(self, x, a):
        pass

    def update(self, x, xo, a):
        pass


@pytest.mark.parametrize("best", [0, 8, 32])
def test_default_depth_is_timed_and_kept(best, tmp_path, monkeypatch):
    monkeypatch.setenv("NR_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d=None: "gpu")
    plan = Plan()
    ms = {0: 2.0, 8: 2.5, 16: 3.0, 32: 4.0}
    ms[best] = 1.0
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: ms[plan.params.upd_planes])
    _, planes, rec = autotune.tune(plan)
    assert planes == best == plan.params.upd_planes == rec["upd_planes"]
    again = Plan()
    again.params.upd_planes = 16
    assert autotune.apply_cached(again) is not None
    assert again.params.upd_planes == best
