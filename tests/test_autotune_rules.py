"""Which cached picks the tuner applies (no GPU: a stand-in for the solver, its timings
and the device's name)."""
import json
import types

import pytest


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    import torch
    from mpf3d import autotune
    monkeypatch.setenv("MPF3D_TUNING_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "GPU")
    return autotune


def domain(nx, ny, nz, anisotropy=True):
    return types.SimpleNamespace(nx=nx, ny=ny, nz=nz, N=5, slots=8, anisotropy=anisotropy, torque=anisotropy,
                                 device="cuda:0", tuning=None, sweep_tma=False)


def test_picks_of_other_kernels_are_not_applied(tuner, monkeypatch, tmp_path):
    s = domain(128, 128, 128)
    other = tuner.key_of(s).rsplit("|k", 1)[0]
    (tmp_path / "tune.json").write_text(json.dumps({other: {"config": [8, 8, 4, 256, 32, 64]},
                                                    other + f"|k{tuner.KERNELS - 1}": {"config": [2, 8, 4, 256, 32, 64]}}))
    monkeypatch.setattr(tuner, "time_config", lambda *a, **k: 1.0)
    assert tuple(tuner.tune(s)["config"]) == tuner.DEFAULT
    assert tuner.key_of(s) in json.loads((tmp_path / "tune.json").read_text())
