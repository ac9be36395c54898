"""Fixed-point products at the ends of the exponent range: a factor in the subnormal
numbers times one large enough is a product like any other."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["flux", "jac"])
@pytest.mark.parametrize("nx", [48, 256])
def test_subnormal_stream_function(nx, form):
    import torch
    from nhqg_gb300 import spectral
    L = 2.0 * np.pi
    kx = (2.0 * np.pi * np.fft.fftfreq(nx, d=L / nx))[:, None]
    ky = (2.0 * np.pi * np.arange(nx // 2 + 1) / L)[None]
    mask = (np.abs(np.fft.fftfreq(nx, 1.0 / nx)) <= nx // 3)[:, None] & (np.arange(nx // 2 + 1) <= nx // 3)[None]
    rng = np.random.default_rng(2)
    f = np.fft.rfft2(rng.standard_normal((4, 2, nx, nx))) * mask
    f[0] /= np.abs(f[0]).max()  # psi at most 1
    fn = spectral.triple_conservative_flux_divergence_23 if form == "flux" else spectral.triple_jacobian_23

    def call(psi, rest):
        t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (psi, *rest)]
        return [o.cpu().numpy() for o in fn(*t, kx, ky, mask, nx)]

    # psi is normal, the velocity i k psi / (N Nx)^2 that the kernels transform is not: typical
    # entries of 2^-3 leave 2^-1030 at 48^2 (44 bits) and 2^-1040 at 256^2 (34 bits, 6e-11)
    low = call(f[0] * 2.0 ** -1005, f[1:] * 2.0 ** 900)
    for a, b in zip(low, call(f[0], f[1:])):
        a = a * 2.0 ** 105
        assert np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(b)
