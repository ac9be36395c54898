"""Contexts on several threads and streams whose launches of one kernel differ in
shared memory: full planes and the band's rectangle of one transform length, and
the corrector's 1-D kernel at two time steps."""

import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REPEATS = 600


def _race(jobs):
    """Each job's callable REPEATS times on a thread and stream of its own; returns
    the status codes other than 0."""
    import torch
    bad, go = [], threading.Barrier(len(jobs))

    def work(fn, stream):
        torch.cuda.set_device(0)
        go.wait()
        for _ in range(REPEATS):
            rc = fn(ctypes.c_void_p(stream.cuda_stream))
            if rc:
                bad.append(rc)

    streams = [torch.cuda.Stream() for _ in jobs]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=j) for j in zip(jobs, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return bad


def test_products():
    import torch
    from nhqg_gb300 import NHQGConfig, make_grid, spectral
    from nhqg_gb300.engine import Engine
    g = make_grid(NHQGConfig(Nx=256, Nz=16, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule",
                             nonlinear_advection="flux", nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1, dt=1e-4,
                             thermal_closure="fixed_conduction"))
    e = Engine(g)
    state = [torch.zeros((lv, 256, 129), dtype=torch.complex128, device="cuda") for lv in (17, 15, 15)]
    state.append(torch.zeros(17, dtype=torch.float64, device="cuda"))
    out = [t.clone() for t in state]
    a, b = e.state_desc(*state), e.state_desc(*out)
    kx, ky = np.asarray(g.kx), np.asarray(g.ky)
    plane = spectral._engine(256, kx, ky)
    f = torch.zeros((7, 3, 256, 129), dtype=torch.complex128, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in f]
    bad = _race([lambda st: e.lib.nhqg_explicit_rhs(e.handle, ctypes.byref(a), ctypes.byref(b), 0, 0, st),
                 lambda st: e.lib.nhqg_triple_advection_23(plane.handle, 0, 3, *p, st)])
    assert not bad, (len(bad), set(bad))


def test_correctors():
    import torch
    from nhqg_gb300 import NHQGConfig, make_grid
    from nhqg_gb300.engine import Engine
    g = make_grid(NHQGConfig(Nx=16, Nz=256, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule",
                             nonlinear_advection="flux", nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1, dt=1e-4,
                             thermal_closure="evolve_mean", mean_exchange_discretization="balanced_sbp2_pc",
                             sbp_corrector_substeps=2))
    jobs = []
    for total in (1e-7, 4e-5):  # reaches of the banded inverse, and so its size
        e = Engine(g)
        s = [torch.zeros((lv, 16, 9), dtype=torch.complex128, device="cuda") for lv in (257, 255, 255)]
        s.append(torch.zeros(257, dtype=torch.float64, device="cuda"))
        o = [t.clone() for t in s]
        a, b = e.state_desc(*s), e.state_desc(*o)
        jobs.append(lambda st, e=e, a=a, b=b, s=s, o=o, total=total: e.lib.nhqg_sbp2_corrector(
            e.handle, ctypes.byref(a), ctypes.byref(b), total, st))
    bad = _race(jobs)
    assert not bad, (len(bad), set(bad))
