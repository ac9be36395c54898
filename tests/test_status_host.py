"""A kernel wait that ran out (the TIMEOUT bit of the device status) reaches the
caller as an error at every point that reads the status."""

import types

import pytest
import torch

from nhqg_gb300 import _native as nat
from nhqg_gb300 import ensemble, solver


class _Eng:
    def __init__(self, bits):
        self.bits = bits

    def device_status(self, reset=True):
        bits, self.bits = self.bits, 0 if reset else self.bits
        return bits

    def state_desc(self, *s):
        return nat.StateDesc()


def test_check_band():
    solver._check_band(_Eng(0), "x")
    with pytest.raises(ValueError, match="band"):
        solver._check_band(_Eng(nat.DEVICE_STATUS_OOB), "x")
    for other in (0, nat.DEVICE_STATUS_OOB):
        e = _Eng(nat.DEVICE_STATUS_TIMEOUT | other)
        with pytest.raises(RuntimeError, match="wait"):
            solver._check_band(e, "x")
        solver._check_band(e, "x")  # reported once
    with pytest.raises(nat.NativeError):
        solver._check_band(_Eng(-1), "x")


def test_run_reports_later_chunks(monkeypatch):
    e = _Eng(0)

    def step(s, grid, n, check=False, precision="fp64"):
        e.bits |= 0 if check else nat.DEVICE_STATUS_TIMEOUT
        return s

    monkeypatch.setattr(solver, "sanitize_state", lambda s, g: solver.State(*[torch.zeros(1)] * 4))
    monkeypatch.setattr(solver, "step_inplace", step)
    monkeypatch.setattr(solver, "engine_for", lambda g: e)
    grid = types.SimpleNamespace(dt=0.1)
    solver.run(grid, (), 2, 2)
    with pytest.raises(RuntimeError, match="wait"):
        solver.run(grid, (), 4, 2)


def test_ensemble(monkeypatch):
    ens = ensemble.Ensemble.__new__(ensemble.Ensemble)
    ens.handle = None
    ens.engines = [_Eng(0), _Eng(nat.DEVICE_STATUS_TIMEOUT), _Eng(nat.DEVICE_STATUS_OOB)]
    ens.lib = types.SimpleNamespace(nhqg_batch_load=lambda *a: 0)
    monkeypatch.setattr(ensemble, "to_device", lambda s: s)
    monkeypatch.setattr(ensemble, "_stream_handle", lambda: None)
    monkeypatch.setattr(ensemble.torch.cuda, "synchronize", lambda: None)
    ens.load(0, ())
    with pytest.raises(RuntimeError, match="wait"):
        ens.load(1, ())
    with pytest.raises(ValueError, match="band"):
        ens.load(2, ())
    ens.check()
    ens.engines[2].bits = nat.DEVICE_STATUS_TIMEOUT
    with pytest.raises(RuntimeError, match="wait"):
        ens.check()
