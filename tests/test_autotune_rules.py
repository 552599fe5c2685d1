"""What the tuner searches and which cached picks it applies (no GPU: a stand-in for the
solver, its timings and the device's name)."""
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


@pytest.mark.parametrize("dims,anisotropy,lists", [((64, 64, 64), True, False), ((80, 80, 80), True, False),
                                                   ((128, 128, 128), True, True), ((80, 80, 80), False, True),
                                                   ((32, 32, 32), False, False)])
def test_list_shapes_are_timed_only_where_they_apply(tuner, monkeypatch, dims, anisotropy, lists):
    timed = []

    def time_config(solver, cfg, steps, sweep_tma=False):
        timed.append(tuple(cfg))
        return 1.0 if tuple(cfg) == tuner.DEFAULT else 1.0 - 1e-3 * len(timed)  # noise that favours the latest

    monkeypatch.setattr(tuner, "time_config", time_config)
    rec = tuner.tune(domain(*dims, anisotropy), use_cache=False)
    shapes = {cfg[2:] for cfg in timed}
    assert shapes == ({tuner.DEFAULT[2:]} | set(tuner.QUEUE) if lists else {tuner.DEFAULT[2:]})
    if not lists:
        assert tuple(rec["config"][2:]) == tuner.DEFAULT[2:]


def test_picks_of_other_kernels_are_not_applied(tuner, monkeypatch, tmp_path):
    s = domain(128, 128, 128)
    other = tuner.key_of(s).rsplit("|k", 1)[0]
    (tmp_path / "tune.json").write_text(json.dumps({other: {"config": [8, 8, 4, 256, 32, 64]},
                                                    other + f"|k{tuner.KERNELS - 1}": {"config": [2, 8, 4, 256, 32, 64]}}))
    monkeypatch.setattr(tuner, "time_config", lambda *a, **k: 1.0)
    assert tuple(tuner.tune(s)["config"]) == tuner.DEFAULT
    assert tuner.key_of(s) in json.loads((tmp_path / "tune.json").read_text())


def test_rule_of_batches():
    from mpf3d import _lib
    L = _lib.lib()
    assert L.mpf3d_batched_step_by_kind(1 << 18, 1) == 0 and L.mpf3d_batched_step_by_kind(1 << 20, 1) == 1
    assert L.mpf3d_batched_step_by_kind(1000, 0) == 1
    assert L.mpf3d_compact_step_by_kind(0, 1, 1, 1) == 0
