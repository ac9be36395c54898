"""Tile autotuning reaches every context whose own products run on the tiled
kernels, whichever other products of it do not."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (form, sponge, Nx, tiles to choose): the Jacobian with a sponge and lengths without
# fixed-point kernels run in FP64
@pytest.mark.parametrize("form,sponge,nx,tuned", [("flux", False, 48, False), ("flux", True, 48, False),
                                                  ("jacobian", False, 48, False), ("jacobian", True, 48, True),
                                                  ("flux", False, 36, True)])
def test_fp64_tiles(form, sponge, nx, tuned):
    from nhqg_gb300 import NHQGConfig, make_grid
    from nhqg_gb300.engine import Engine
    g = make_grid(NHQGConfig(Nx=nx, Nz=4, L=9.0, float_dtype="float64", horizontal_dealiasing="23_rule",
                             nonlinear_advection=form, nu_q=0.1, nu_w=0.1, nu_theta=0.1, hyper_order=1, dt=1e-3,
                             thermal_closure="fixed_conduction"))
    if sponge:
        g = g._replace(sponge_phys=np.ones((nx, nx)))
    e = Engine(g)
    assert e.tiles() == (0, 0, 0, 0)
    tiles = e.autotune()
    assert (tiles[0] > 0 and tiles[1] > 0) == tuned and tiles[2:] == (0, 0)
