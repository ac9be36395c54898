"""The plane products' workspace: nothing of it stays with a context, it is as
large as the call needs, and calls with and without one agree."""

import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(nx, L):
    kx = (2.0 * np.pi * np.fft.fftfreq(nx, d=L / nx))[:, None]
    ky = (2.0 * np.pi * np.arange(nx // 2 + 1) / L)[None]
    mask = (np.abs(np.fft.fftfreq(nx, 1.0 / nx)) <= nx // 3)[:, None] & (np.arange(nx // 2 + 1) <= nx // 3)[None]
    return kx, ky, mask


def _planes(nx, levels):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    return torch.fft.rfft2(torch.randn(4, levels, nx, nx, generator=gen, dtype=torch.float64, device="cuda"))


def test_contexts_keep_no_workspace():
    """A few levels at 256^2 for several box lengths: device memory outside torch's
    allocator grows by what a context holds (the same for one level), no more."""
    import torch
    from nhqg_gb300 import spectral
    f = _planes(256, 7)

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    def call(L, lev):
        kx, ky, mask = _grid(256, L)
        spectral.triple_conservative_flux_divergence_23(*f[:, :lev], kx, ky, mask, 256)

    for L in (3.0, 4.0, 5.0):
        call(L, 1)  # makes the context
    before = free()
    for L in (3.0, 4.0, 5.0):
        call(L, 7)
    assert before - free() <= 8 << 20


def test_lent_is_what_the_call_needs():
    from nhqg_gb300 import _native as nat
    from nhqg_gb300 import spectral
    kx, ky, _ = _grid(256, 3.0)
    e = spectral._engine(256, kx, ky)

    def size(kind, lev, rc=0):
        n = ctypes.c_size_t()
        assert e.lib.nhqg_plane_workspace_bytes(e.handle, kind, lev, ctypes.byref(n)) == rc
        return n.value

    assert size(0, 1) == 0  # the context's own buffers
    # 5 input fields of 129 columns, 6 products of 86, their exponents, in units of 256 bytes
    for lev in (7, 33):
        want = lev * 256 * 16 * (5 * 129 + 6 * 86) + 4 * lev * (5 * 129 + 6 * 128)
        assert want <= size(0, lev) <= want + 4 * 256
    for kind in (0, 1, nat.PLANE_SPONGE):
        assert size(kind, 5000) == size(kind, 4000) <= 600 << 20
    size(7, 3, rc=1)
    size(0, 0, rc=1)


@pytest.mark.parametrize("nx,levels", [(48, 33), (256, 9)])
def test_with_and_without(nx, levels):
    import torch
    from nhqg_gb300 import spectral
    kx, ky, mask = _grid(nx, 3.0)
    e = spectral._engine(nx, kx, ky)
    f = _planes(nx, levels)
    for form, fn in ((0, spectral.triple_conservative_flux_divergence_23), (1, spectral.triple_jacobian_23)):
        lent = fn(*f, kx, ky, mask, nx)
        out = [torch.empty_like(f[0]) for _ in range(3)]
        p = [ctypes.c_void_p(t.data_ptr()) for t in (*f, *out)]
        small = torch.empty(64, dtype=torch.uint8, device="cuda")  # too small: not used
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for call in (lambda: e.lib.nhqg_triple_advection_23(e.handle, form, levels, *p, st),
                     lambda: e.lib.nhqg_triple_advection_ws(e.handle, form, levels, *p, small.data_ptr(), 64, st)):
            for o in out:
                o.fill_(1.0)
            assert call() == 0
            for a, b in zip(lent, out):
                assert torch.equal(a, b)
        assert e.lib.nhqg_triple_advection_ws(e.handle, form, levels, *p, small.data_ptr() + 8, 56, st) == 1


def test_beside_another_thread_s_capture():
    """A plane call of the C interface allocates nothing, so that it does not break
    a stream capture that another thread has begun."""
    import torch
    from nhqg_gb300 import spectral
    kx, ky, mask = _grid(128, 6.0)
    e = spectral._engine(128, kx, ky)
    f = _planes(128, 40)
    out = [torch.empty_like(f[0]) for _ in range(3)]
    p = [ctypes.c_void_p(t.data_ptr()) for t in (*f, *out)]
    side = torch.cuda.Stream()
    st = ctypes.c_void_p(side.cuda_stream)
    assert e.lib.nhqg_triple_advection_23(e.handle, 0, 1, *p, st) == 0  # loads the kernels
    torch.cuda.synchronize()
    rc = []
    x = torch.zeros(4, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1.0
        t = threading.Thread(target=lambda: rc.append(e.lib.nhqg_triple_advection_23(e.handle, 0, 40, *p, st)))
        t.start()
        t.join()
    assert rc == [0]
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
    for a, b in zip(out, spectral.triple_conservative_flux_divergence_23(*f, kx, ky, mask, 128)):
        assert torch.equal(a, b)
