"""CPU emulation of the plain corrector's 1-D solve (numerical method): FP64
iterative refinement around a banded FP32 inverse whose row i is row i of the
inverse of A's block [i - ov, i + ov] (one FP32 LU without pivoting of the block's
transpose per row, as k_corr_tstep forms it).  The system, the host's rule for ov and
the check are those of the windowed form's test."""

import numpy as np
import pytest

from test_corrector_windows_cpu import _factor, _overlap, _rhs, _solve, _system


def _banded_inverse(A, ov):
    P = len(A)
    M = np.zeros((P, P), np.float32)
    for i in range(P):
        e0, e1 = max(0, i - ov), min(P, i + ov + 1)
        B = np.ascontiguousarray(A[e0:e1, e0:e1].T)
        unit = np.zeros(e1 - e0, np.float32)
        unit[i - e0] = 1.0
        M[i, e0:e1] = _solve(_factor(B, 0, e1 - e0), unit)  # B y = e_i: y is row i
    return M


def _refine(A, b, ov, sweeps=3):
    M = _banded_inverse(A, ov)
    sol, res, last = np.zeros(len(b)), b.copy(), None
    for _ in range(sweeps):
        last = M @ res.astype(np.float32)
        sol = sol + last.astype(np.float64)
        res = b - A @ sol
    return sol, float(np.abs(last).max()) <= 1e-10 * float(np.abs(sol).max())


@pytest.mark.parametrize("N,dt,w2", [(32, 5e-5, 0.0), (64, 5e-5, 10.0), (256, 2e-5, 0.0), (256, 5e-5, 100.0)])
def test_reaches_fp64_roundoff(N, dt, w2):
    A, sub = _system(N, dt, w2)
    ov = _overlap(N, sub)
    assert ov is not None
    b = _rhs(A, N)
    sol, converged = _refine(A, b, ov)
    exact = np.linalg.solve(A, b)
    # the windowed form's bound
    assert np.abs(sol - exact).max() <= 2e-15 * np.abs(exact).max()
    assert converged


@pytest.mark.parametrize("N,dt,ov", [(64, 5e-5, 1), (256, 2e-5, 2)])
def test_small_reach_fails_the_check(N, dt, ov):
    A, _ = _system(N, dt, 0.0)
    _, converged = _refine(A, _rhs(A, 1), ov)
    assert not converged
