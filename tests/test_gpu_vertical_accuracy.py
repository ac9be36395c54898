"""Accuracy of the plain path's fixed-point vertical transforms: against a long
double restatement they are no further off than the FP64 transforms that
NHQG_FX_VERTICAL=0 selects, at every radix mix and up to their depth limit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _grid(nz):
    from nhqg_gb300 import NHQGConfig, make_grid
    return make_grid(NHQGConfig(Nx=8, Nz=nz, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule",
                                nonlinear_advection="flux", nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1,
                                dt=1e-4, thermal_closure="evolve_mean",
                                mean_exchange_discretization="balanced_sbp2_pc", sbp_corrector_substeps=1))


def _columns(nz, decay):
    """theta planes of 15 random modes, coefficients decaying by e^-decay"""
    rng = np.random.default_rng(nz)
    k = np.fft.fftfreq(8, 1.0 / 8)
    keep = (np.abs(k) <= 2)[:, None] & (np.arange(5) <= 2)[None]
    f = np.fft.rfft2(rng.standard_normal((nz - 1, 8, 8))) * keep[None]
    f[:, 0, 0] = 0.0
    return f * np.exp(-decay * np.arange(nz - 1) / nz)[:, None, None]


def _round_trip(g, th):
    """The corrector with w = 0, one substep: theta -> CGL nodes -> SBP grid (ends
    set to zero) -> CGL nodes -> coefficients -> Galerkin, in long double"""
    nz = g.Nz
    x = np.stack([th.real, th.imag], -1).reshape(nz - 1, -1).astype(LD)
    c = np.zeros((nz + 1, x.shape[1]), LD)
    c[:nz - 1] -= x
    c[2:] += x
    table = np.cos(np.arange(2 * nz).astype(LD) * (LD("3.14159265358979323846264338327950288") / LD(nz)))
    j = np.arange(nz + 1)
    V = table[np.outer(j, j) % (2 * nz)]
    s = np.asarray(g.cgl_to_sbp).astype(LD) @ (V @ c)
    s[0] = s[-1] = 0
    y = np.asarray(g.sbp_to_cgl).astype(LD) @ s
    half = np.ones(nz + 1, LD)
    half[0] = half[nz] = LD(1) / LD(2)
    c = (LD(2) / LD(nz)) * half[:, None] * (V.T @ (half[:, None] * y))
    out = np.zeros_like(x)
    for n in range(nz - 1):
        out[n] = (out[n - 2] if n >= 2 else 0) - c[n]
    return out


def _gpu(nz, th):
    from nhqg_gb300 import solver as S
    g = _grid(nz)
    z = np.zeros_like
    state = (np.zeros((nz + 1, 8, 5), complex), z(th), th, np.zeros(nz + 1))
    got = S.apply_balanced_sbp2_corrector(state, g, 1e-5)[2].cpu().numpy()
    return g, np.stack([got.real, got.imag], -1).reshape(nz - 1, -1)


@pytest.mark.parametrize("nz", [12, 18, 48, 64, 96, 128, 162, 192, 256, 384, 512])
@pytest.mark.parametrize("decay", [14.0, 1.0])
def test_no_further_off_than_fp64(nz, decay, monkeypatch):
    th = _columns(nz, decay)
    g, fixed = _gpu(nz, th)
    monkeypatch.setenv("NHQG_FX_VERTICAL", "0")
    _, plain = _gpu(nz, th)
    assert not np.array_equal(fixed, plain)  # two transforms ran
    ref = _round_trip(g, th)
    err = [float(np.sqrt(np.sum((a - ref) ** 2) / np.sum(ref ** 2))) for a in (fixed, plain)]
    assert err[1] < 1e-11  # the restatement is the corrector's
    assert err[0] <= err[1], err
