"""Sponge and trap terms of the fixed-point products at every transform length: the
explicit tendency against the oracle, and non-finite sponge values."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(nx, rule, eta=0.0, seed=0):
    """A grid with a smooth random sponge and, with eta, a random background PV of
    that size, and the oracle's."""
    import oracle
    from oracle.nhqg_oracle import OracleConfig, _zero_pad
    from nhqg_gb300 import NHQGConfig, make_grid
    cfg = dict(Nx=nx, Nz=4, L=9.0, float_dtype="float64", horizontal_dealiasing=rule + "_rule",
               nonlinear_advection="flux", nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1, dt=1e-3,
               thermal_closure="fixed_conduction")
    g, o = make_grid(NHQGConfig(**cfg)), oracle.make_grid(OracleConfig(**cfg))
    rng = np.random.default_rng(nx + seed)
    k = np.abs(np.fft.fftfreq(nx, 1.0 / nx))
    kk = np.hypot(k[:, None], np.arange(nx // 2 + 1)[None])

    def field(scale):
        return np.fft.rfft2(rng.standard_normal((nx, nx))) * o.mask_23 * np.exp(-0.3 * kk) * scale

    sig = field(1.0)
    npad = 3 * nx // 2
    kw = dict(sponge_phys=np.fft.irfft2(sig, s=(nx, nx)),
              sponge_phys_pad=np.fft.irfft2(_zero_pad(sig, nx, npad), s=(npad, npad)))
    if eta:
        kw["eta_hat"] = field(eta)
    return g._replace(**kw), o.replace(**kw)


def _state(g, mask, seed=1):
    rng = np.random.default_rng(seed)
    return (*(np.fft.rfft2(rng.standard_normal((lv, g.Nx, g.Nx))) * mask for lv in (5, 3, 3)), np.zeros(5))


# transform lengths 48, 64, 96, 128, 192 and the padded 72, 96, 144, 192; a background PV
# 1e4 times q has to cancel out of the sponge's operand
@pytest.mark.parametrize("nx,rule", [(48, "23"), (64, "23"), (96, "23"), (128, "23"), (192, "23"),
                                     (48, "32"), (64, "32"), (96, "32"), (128, "32")])
@pytest.mark.parametrize("eta", [0.0, 1.0, 1e4])
def test_against_oracle(nx, rule, eta):
    import oracle
    from nhqg_gb300 import solver as S
    g, o = _grid(nx, rule, eta)
    s = _state(g, o.mask_23)
    ref = oracle.nhqg_oracle.explicit_rhs(oracle.nhqg_oracle.OracleState(*s), o)
    for got, want in zip(S.explicit_rhs(s, g)[:3], ref[:3]):
        # the operators' bound; with the trap the tendency of q is of its advection's size
        assert np.linalg.norm(got.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)


@pytest.mark.parametrize("nx,rule", [(48, "23"), (64, "23"), (48, "32")])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_sponge(nx, rule, bad, monkeypatch):
    from nhqg_gb300 import solver as S
    g, o = _grid(nx, rule)
    s = _state(g, o.mask_23)
    name = "sponge_phys_pad" if rule == "32" else "sponge_phys"
    sp = np.array(getattr(g, name))
    sp[3, 4] = bad
    for fixed in ("1", "0"):  # the FP64 products say what is expected
        monkeypatch.setenv("NHQG_FX_PRODUCTS", fixed)
        # a copy of the inverse: contexts are kept per grid
        out = S.explicit_rhs(s, g._replace(imex_inv=np.array(g.imex_inv), **{name: sp}))[:3]
        for f in out:
            f = f.cpu().numpy()
            keep = np.broadcast_to(o.mask_23 > 0, f.shape)
            assert not np.isfinite(f[keep].real).any() and not np.isfinite(f[keep].imag).any(), fixed
