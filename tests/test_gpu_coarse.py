"""The one-CTA coarse solver with register-resident levels: every first level it takes (65^2 down to
3^2), every depth, and sweep counts from none to more than the tile kernels have, V-cycle by V-cycle
against the FP64 oracle.  Tolerance as for the other multigrid kernels: FP32 corrections, 1e-6 relative
L2 of phi after three cycles."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 5, 9, 17, 33, 65, 129])
@pytest.mark.parametrize("nu", [(2, 2, 2), (0, 1, 3), (1, 0, 20), (6, 5, 1)])
def test_every_depth_matches_oracle(orc, n, nu):
    import torch
    from pic_cuda_b200.engine import solve_multigrid_f64
    h = 0.7 / (n - 1)
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, n))
    phi0 = np.zeros((n, n))
    phi0[0, :] = 0.5
    for levels in range(1 if n <= 65 else 2, int(np.log2(n - 1)) + 1):
        dphi = torch.tensor(phi0, device="cuda")
        cyc, _, _ = solve_multigrid_f64(dphi, torch.tensor(f, device="cuda"), n, n, levels, h, 1.15, *nu, tol=0.0,
                                        max_cycles=3)
        assert cyc == 3
        ref = orc.mg_vcycles(phi0, f, h, 3, levels=levels, omega=1.15, nu1=nu[0], nu2=nu[1], nuc=nu[2])
        assert rel_l2(dphi.cpu().numpy(), ref) < 1e-6, levels
