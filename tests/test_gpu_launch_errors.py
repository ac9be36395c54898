"""A kernel of the corrector that could not be launched is reported."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_corrector(monkeypatch):
    """Eight modes per CTA at 973 levels want more shared memory than a CTA has: the
    runtime refuses the column kernels' launches, and the call says so."""
    from nhqg_gb300 import NHQGConfig, make_grid
    from nhqg_gb300 import _native as nat
    from nhqg_gb300 import solver as S
    monkeypatch.setenv("NHQG_COLUMN_MODES", "8")
    g = make_grid(NHQGConfig(Nx=8, Nz=972, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule",
                             nonlinear_advection="flux", nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1,
                             dt=1e-4, thermal_closure="evolve_mean",
                             mean_exchange_discretization="balanced_sbp2_pc", sbp_corrector_substeps=2))
    s = [np.zeros((lv, 8, 5), complex) for lv in (973, 971, 971)] + [np.zeros(973)]
    with pytest.raises(nat.NativeError):
        S.apply_balanced_sbp2_corrector(s, g, 1e-5)
    monkeypatch.delenv("NHQG_COLUMN_MODES")
    g = g._replace(imex_inv=np.array(g.imex_inv))  # another context
    assert not S.apply_balanced_sbp2_corrector(s, g, 1e-5)[2].abs().any()
