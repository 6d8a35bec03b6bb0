"""The level-0 up kernel's 1024-thread tiles against its 256-thread ones: bit for bit the same potential,
residual and cycle count for every sweep count and charge type, on grids of a few tiles and of more than
one wave of them, with edge tiles of one node."""
import numpy as np
import pytest

from pic_cuda_b200 import _lib as L
from pic_cuda_b200 import configs as cf
from pic_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [65, 129, 513])
@pytest.mark.parametrize("deposit", [L.DEPOSIT_F32, L.DEPOSIT_I64])
@pytest.mark.parametrize("nu", [0, 1, 2, 3, 4])
def test_wide_level0_tiles_same_bits(nx, deposit, nu):
    rho = np.random.default_rng(nx + nu).standard_normal((nx, nx)) * 1e-6
    out = []
    for wide in (0, 64):
        e = Engine(0)
        e.set_option(L.OPT_MG_WIDE_TILES, wide)
        cfg = cf.plasma(nx, 0.01, 1000, deposit=deposit, seed=3, tol=1e-6)
        cfg.nu_pre, cfg.nu_post, cfg.max_cycles = max(nu, 1), nu, 6
        j = e.add_job(cfg)
        j.set_grid(L.GRID_RHO, rho)
        j.solve_field()
        d = j.diagnostics()
        out.append((j.get_grid(L.GRID_PHI), d["relres"], d["vcycles"]))
        e.close()
    assert out[0][2] >= 1
    assert out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])


# 65^2 with the one-CTA solver from 33^2 down, so that its level 0 has tiles
@pytest.mark.parametrize("nu", [1, 2, 3, 4])
def test_wide_level0_tiles_of_the_smallest_grid(nu):
    rho = np.random.default_rng(nu).standard_normal((65, 65)) * 1e-6
    out = []
    for wide in (0, 64):
        e = Engine(0)
        e.set_option(L.OPT_MG_COARSE_TOP, 33)
        e.set_option(L.OPT_MG_WIDE_TILES, wide)
        cfg = cf.plasma(65, 0.01, 1000, deposit=L.DEPOSIT_I64, seed=3, tol=1e-6)
        cfg.nu_pre = cfg.nu_post = nu
        cfg.max_cycles = 6
        j = e.add_job(cfg)
        j.set_grid(L.GRID_RHO, rho)
        j.solve_field()
        d = j.diagnostics()
        out.append((j.get_grid(L.GRID_PHI), d["relres"], d["vcycles"]))
        e.close()
    assert out[0][2] >= 1 and out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])
