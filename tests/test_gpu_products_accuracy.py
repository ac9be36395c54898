"""Accuracy and range of the fixed-point products: against long double FFTs they are
no further off than the FP64 kernels that NHQG_FX_PRODUCTS=0 selects, and rows whose
products reach the bound of their exponent do not overflow."""

import numpy as np
import pytest

from test_gpu_products_fx import L, _call, _grid, _reference

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _planes(nx, rule, kind):
    rng = np.random.default_rng(nx)
    f = rng.standard_normal((4, nx, nx))
    if kind == "line":  # a few active rows
        f = f * np.exp(-((np.arange(nx) - nx / 2) / 2.0) ** 2)[None, :, None]
    f = np.fft.rfft2(f)
    if kind == "few":  # a few active modes
        keep = np.zeros(f.shape[1:], bool)
        keep[rng.integers(-3, 4, 4), rng.integers(0, 4, 4)] = True
        keep[1, 2] = True
        f = f * keep
    return (f * _grid(nx)[2] if rule == "23" else f)[:, None]


def _long_double(form, f, nx, rule):
    n = nx if rule == "23" else 3 * nx // 2
    kx, ky, keep = _grid(nx)
    f = f[:, 0].astype(np.clongdouble)

    def rows(a, width):  # zero-padded to n rows
        if n == nx:
            return a
        out = np.zeros((n, width), a.dtype)
        out[:nx // 2, :a.shape[1]] = a[:nx // 2]
        out[n - nx // 2:, :a.shape[1]] = a[nx // 2:]
        return out

    phys = lambda a: np.fft.irfft2(rows(a, n // 2 + 1), s=(n, n))  # noqa: E731
    kxn = rows(kx.astype(LD), 1)
    kyn = np.zeros((1, n // 2 + 1), LD)
    kyn[:, :nx // 2 + 1] = ky

    def back(a):
        if n == nx:
            return a * keep
        return np.concatenate([a[:nx // 2, :nx // 2 + 1], a[n - nx // 2:, :nx // 2 + 1]]) * (LD(n) / LD(nx)) ** 2

    px, py = phys(1j * kx.astype(LD) * f[0]), phys(1j * ky.astype(LD) * f[0])
    out = []
    for g in f[1:]:
        if form == "flux":
            p = phys(g)
            out.append(back(1j * kxn * np.fft.rfft2(-py * p) + 1j * kyn * np.fft.rfft2(px * p)))
        else:
            out.append(back(np.fft.rfft2(px * phys(1j * ky.astype(LD) * g) - py * phys(1j * kx.astype(LD) * g))))
    return out


@pytest.mark.parametrize("form", ["flux", "jac"])
@pytest.mark.parametrize("kind", ["white", "line", "few"])
@pytest.mark.parametrize("nx,rule", [(48, "23"), (64, "23"), (96, "32"), (128, "32"), (192, "23"), (256, "23")])
def test_no_further_off_than_fp64(nx, rule, kind, form, monkeypatch):
    from nhqg_gb300 import spectral
    f = _planes(nx, rule, kind)
    ref = _long_double(form, f, nx, rule)
    err = []
    for fixed in ("1", "0"):
        monkeypatch.setenv("NHQG_FX_PRODUCTS", fixed)
        monkeypatch.setattr(spectral, "_SPECTRAL", {})  # contexts of this switch's own
        got = _call(form, f, nx, rule)
        err.append(max(float(np.sqrt(np.sum(np.abs(a[0] - r) ** 2) / np.sum(np.abs(r) ** 2)))
                       for a, r in zip(got, ref)))
    assert err[1] < 1e-13  # the restatement is the products'
    assert err[0] <= err[1], err


@pytest.mark.parametrize("form", ["flux", "jac"])
@pytest.mark.parametrize("nx", [48, 96, 192, 256])
@pytest.mark.parametrize("rows", ["all", "even", "one"])
def test_rows_at_the_bound(nx, rows, form):
    """Velocity and scalars of constant size along y: |u f| sums to the Cauchy-Schwarz
    bound of the row (to twice less where both rows of a pair are alike).  The scales
    step the products through the factor of two between exponents."""
    x, y = np.arange(nx), np.arange(nx)
    s = np.where((y // (nx // 8)) % 2 == 0, 1.0, -1.0)  # zero mean
    on = {"all": x >= 0, "even": x % 2 == 0, "one": x == 2}[rows]
    plane = np.fft.rfft2(on[:, None] * s[None])
    kx, ky, keep = _grid(nx)
    psi = np.divide(plane, -1j * ky, out=np.zeros_like(plane), where=ky != 0)
    # modes without energy carry rounding only: removed, the exponents are the wave's
    psi[:, np.abs(plane).max(0) < 1e-9] = 0.0
    for t in range(8):
        f = np.stack([psi * 2.0 ** (t / 8.0), plane, plane * 3.0, plane * 0.7])[:, None]
        for got, ref in zip(_call(form, f, nx, "23"), _reference(form, f, nx, "23")):
            # the bound of the FP64 product tests, of the largest that the products could be:
            # the flux of a constant product is rounding alone
            size = np.linalg.norm(f[1]) * np.abs(np.fft.irfft2(plane, s=(nx, nx))).max() * 2 * np.pi * nx / L
            assert np.linalg.norm(got - ref) <= 1e-13 * max(np.linalg.norm(ref), size)
