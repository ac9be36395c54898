"""The plain corrector's 1-D kernel with transfer matrices whose rows are wider than
the package's two entries, past what its shared memory holds."""

import numpy as np
import pytest

import oracle
from oracle.nhqg_oracle import OracleConfig, OracleState

pytestmark = pytest.mark.gpu


def _widen(A, width, seed):
    """A plus `width` small entries around each row's own (end rows kept)"""
    rng = np.random.default_rng(seed)
    A = np.array(A)
    n = len(A)
    for i in range(1, n - 1):
        j0 = min(max(int(np.argmax(np.abs(A[i]))) - width // 2, 0), n - width)
        A[i, j0:j0 + width] += 1e-5 * rng.standard_normal(width)
    return A


# entries a row: 2 as built; 24 and 60 at 257 levels lie on both sides of the 200 KB
# that the tables and vectors may take; 973 levels hold two entries only just
@pytest.mark.parametrize("nz,width", [(256, 2), (256, 24), (256, 60), (63, 40), (972, 2), (972, 4)])
def test_wide_rows(nz, width):
    from nhqg_gb300 import NHQGConfig, make_grid
    from nhqg_gb300 import solver as S
    cfg = dict(Nx=8, Nz=nz, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule",
               nonlinear_advection="flux", nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1, dt=1e-4,
               thermal_closure="evolve_mean", mean_exchange_discretization="balanced_sbp2_pc",
               sbp_corrector_substeps=3)
    g, o = make_grid(NHQGConfig(**cfg)), oracle.make_grid(OracleConfig(**cfg))
    if width > 2:
        kw = dict(cgl_to_sbp=_widen(g.cgl_to_sbp, width, 1), sbp_to_cgl=_widen(g.sbp_to_cgl, width, 2))
        g, o = g._replace(**kw), o.replace(**kw)
    rng = np.random.default_rng(nz)
    s = [np.fft.rfft2(rng.standard_normal((lv, 8, 8))) * o.mask_23[None] *
         np.exp(-8.0 * np.arange(lv) / nz)[:, None, None] for lv in (nz + 1, nz - 1, nz - 1)]
    tb = 0.05 * rng.standard_normal(nz + 1) * np.exp(-np.arange(nz + 1) / 4.0)
    s = OracleState(*s, tb)
    ref = oracle.nhqg_oracle.apply_balanced_sbp2_corrector(s, o, 3e-5)
    got = S.apply_balanced_sbp2_corrector(s, g, 3e-5)
    # the corrector's bound at 256 levels (1e-12), growing as the dense transforms' rounding
    # and the left inverse's sums do, with the depth squared
    for a, b in zip(got[2:], ref[2:]):
        assert np.linalg.norm(a.cpu().numpy() - b) <= 1e-12 * max(1.0, nz / 256.0) ** 2 * np.linalg.norm(b)
