"""Lazily conjugated and negated tensors as inputs: every entry point answers as
it does for the same values written out."""

import numpy as np
import pytest

import oracle
from oracle.nhqg_oracle import OracleConfig

pytestmark = pytest.mark.gpu

CFG = dict(Nx=16, Nz=12, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule", nonlinear_advection="flux",
           nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1, dt=1e-3, thermal_closure="evolve_mean",
           mean_exchange_discretization="balanced_sbp2_pc", sbp_corrector_substeps=2)


def _state(**kw):
    """(grid, views, the same values written out)"""
    import torch
    from nhqg_gb300 import NHQGConfig, make_grid
    g = make_grid(NHQGConfig(**dict(CFG, **kw)))
    mask = oracle.make_grid(OracleConfig(**CFG)).mask_23
    rng = np.random.default_rng(3)
    views = []
    for lv in (13, 11, 11):
        f = np.fft.rfft2(rng.standard_normal((lv, 16, 16))) * mask[None]
        views.append(torch.from_numpy(f).cuda().conj())
    tb = rng.standard_normal(13) * 1e-2
    views.append(torch._neg_view(torch.from_numpy(tb).cuda()))
    assert all(v.is_conj() for v in views[:3]) and views[3].is_neg()
    return g, views, [v.clone() for v in views]


@pytest.mark.parametrize("call", ["imex_step", "imex_step_mixed", "explicit_rhs", "implicit_tendency", "solve",
                                  "corrector", "sanitize", "ensemble"])
def test_state_views(call):
    import torch
    from nhqg_gb300 import solver as S
    from nhqg_gb300.ensemble import Ensemble
    # the stage solve alone is defined without the split exchange
    alone = dict(thermal_closure="fixed_conduction", mean_exchange_discretization="legacy")
    g, views, plain = _state(**(alone if call == "solve" else {}))

    def run(s):
        if call == "imex_step":
            return S.imex_step(s, g)
        if call == "imex_step_mixed":
            return S.imex_step(s, g, precision="mixed")
        if call == "explicit_rhs":
            return S.explicit_rhs(s, g)
        if call == "implicit_tendency":
            return S.implicit_tendency(s, g)
        if call == "solve":
            return S.imex_implicit_solve(*s[:3], g)
        if call == "corrector":
            return S.apply_balanced_sbp2_corrector(s, g, 1e-4)
        if call == "sanitize":
            return S.sanitize_state(s, g)
        ens = Ensemble([g], autotune=False)
        ens.load(0, s)
        ens.step(1)
        return ens.store(0)

    for a, b in zip(run(views), run(plain)):
        assert torch.equal(a, b)


def test_plane_views():
    import torch
    from nhqg_gb300 import spectral
    _, views, plain = _state()
    kx = (2.0 * np.pi * np.fft.fftfreq(16, d=1.0 / 16))[:, None]
    ky = (2.0 * np.pi * np.arange(9.0))[None]

    def run(s):
        q, w, th = s[0][:11], s[1], s[2]
        return spectral.triple_jacobian(w, q, w, th, kx, ky, 16, 24)

    for a, b in zip(run(views), run(plain)):
        assert torch.equal(a, b)
