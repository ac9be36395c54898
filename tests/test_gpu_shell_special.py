"""The plain path's per-shell solve with matrices and right-hand sides that the
digits of its tensor-core kernel could lose: non-finite matrix entries."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(nx, nz, **kw):
    from nhqg_gb300 import NHQGConfig, make_grid
    return make_grid(NHQGConfig(**dict(dict(
        Nx=nx, Nz=nz, L=10.0, float_dtype="float64", horizontal_dealiasing="23_rule", Ra_tilde=40.0, nu_q=0.3,
        nu_w=0.2, nu_theta=0.1, hyper_order=2, dt=2e-3, thermal_closure="fixed_conduction"), **kw)))


def _modes(g):
    """kept modes and the shell row of each, (Nx, Nk)"""
    k = np.abs(np.fft.fftfreq(g.Nx, 1.0 / g.Nx)) <= g.Nx // 3
    keep = k[:, None] & (np.arange(g.Nx // 2 + 1) <= g.Nx // 3)[None]
    return keep, np.asarray(g.imex_shell_row)


def _solve_w(g, Rw):
    """w of the stage solve with R_q = R_theta = 0: A^-1 R_w, mode by mode"""
    from nhqg_gb300 import solver as S
    zq = np.zeros((g.Nz + 1,) + Rw.shape[1:], complex)
    return S.imex_implicit_solve(zq, Rw, np.zeros_like(Rw), g)[1].cpu().numpy()


def _noise(g, seed, decay=0.0):
    rng = np.random.default_rng(seed)
    shape = (g.Nz - 1, g.Nx, g.Nx // 2 + 1)
    keep, _ = _modes(g)
    f = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * keep[None]
    return f * np.exp(-decay * np.arange(g.Nz - 1) / g.Nz)[:, None, None]


# the second matrix row is in the second tile of 128 rows; 18 and 257 fill no tile
@pytest.mark.parametrize("nz", [18, 140, 257])
def test_non_finite_matrix_rows(nz):
    g = _grid(12, nz)
    keep, row = _modes(g)
    R = _noise(g, nz)
    base = _solve_w(g, R)
    inv = np.array(g.imex_inv)
    shell = row[1, 1]
    hit = keep & (row == shell)
    rows = [3, nz - 4, 5]
    inv[shell, rows[0], 2] = np.nan
    inv[shell, rows[1], nz - 4] = np.nan  # on the diagonal
    inv[shell, rows[2], 0] = np.inf
    got = _solve_w(g._replace(imex_inv=inv), R)
    for r in rows:
        assert not np.isfinite(got[r][hit].real).any() and not np.isfinite(got[r][hit].imag).any()
    same = np.ones(got.shape, bool)
    for r in rows:
        same[r][hit] = False
    assert np.array_equal(got[same], base[same])


def _bound(A, x):
    """Error bound of one column, per row: two roundings of each part (the diagonal's
    product and the rest), the dropped digit groups (2^-55 of row maximum off the
    diagonal times column maximum, powers of two above each included) and the
    rounding of both operands to 2^-61 of those."""
    off = np.abs(A - np.diag(np.diag(A)))
    om, xm = off.max(1), np.abs(x).max()
    rest = np.abs((A - np.diag(np.diag(A))) @ x)
    return (2.0 ** -52 * (np.abs(np.diag(A) * x) + rest) + 2.0 ** -55 * om * xm +
            2.0 ** -61 * (om * np.abs(x).sum() + xm * off.sum(1)))


# coefficients decaying as a resolved column's do: the small ones keep their accuracy
@pytest.mark.parametrize("nz,decay", [(18, 30.0), (128, 14.0), (130, 30.0), (257, 14.0)])
def test_small_coefficients(nz, decay):
    g = _grid(12, nz)
    keep, row = _modes(g)
    R = _noise(g, nz, decay)
    got = _solve_w(g, R)
    for i, j in np.argwhere(keep):
        A = np.asarray(g.imex_inv)[row[i, j]]
        for part in (np.real, np.imag):
            x = np.ascontiguousarray(part(R[:, i, j]))
            ref = A.astype(np.longdouble) @ x.astype(np.longdouble)
            assert np.all(np.abs(part(got[:, i, j]) - ref) <= _bound(A, x))


# equal digits of one sign: every digit sum is as large as the depth allows (255 and 256
# rows), at the limit of the accumulators' exact range
@pytest.mark.parametrize("nz", [256, 257])
@pytest.mark.parametrize("digit", [-128, 127])
def test_saturated_digits(nz, digit):
    g = _grid(8, nz)
    # 32 2^56 at most under the exponent, then six digits; the double's 53 bits hold them
    v = float(sum((digit if k else int(np.sign(digit)) * 31) * 256 ** (6 - k) for k in range(7))) / 2.0 ** 53
    inv = np.full_like(np.asarray(g.imex_inv), v)
    keep, _ = _modes(g)
    R = np.zeros((nz - 1, 8, 5), complex)
    R[:, keep] = v * (1 - 1j)
    got = _solve_w(g._replace(imex_inv=inv), R)
    exact = float(np.longdouble(v) * np.longdouble(v) * (nz - 1))
    for part, sign in ((np.real, 1.0), (np.imag, -1.0)):
        assert np.all(np.abs(part(got[:, keep]) - sign * exact) <= 2.0 ** -51 * exact)
