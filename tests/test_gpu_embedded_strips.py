"""The embedded-boundary multigrid's row-pipeline (strip) kernels, which take levels of more than about
2 million nodes, against the FP64 oracle: ragged and even sizes (strips and row chunks end in
remainders), every sweep count they are built for, with and without phi_bc, and a mask at an odd
address (its words are loaded aligned).  Tolerance as in test_gpu_embedded.py: 1e-12 relative L2 per
V-cycle (FP64 throughout; only the contraction of a multiply-add differs)."""
import numpy as np
import pytest

from conftest import rel_l2
from pic_cuda_b200 import _lib as L
from test_gpu_embedded import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nu,options,with_bc", [
    (2049, 1300, (2, 2), L.EMB_COARSEN_ANY | L.EMB_PROLONG_BILINEAR, True),
    (1302, 2051, (2, 2), 0, True),
    (2200, 1201, (1, 3), L.EMB_COARSEN_ANY, True),
    (2049, 1300, (3, 1), L.EMB_PROLONG_BILINEAR, False),
    (1302, 2051, (0, 2), L.EMB_COARSEN_ANY, True),
    (2200, 1201, (2, 0), L.EMB_COARSEN_ANY | L.EMB_PROLONG_BILINEAR, False),
])
def test_strips_match_oracle(orc, nx, ny, nu, options, with_bc):
    import torch
    from pic_cuda_b200.engine import solve_embedded_f64
    h, levels = 1.0 / (nx - 1), 6
    phi, rhs, mask, bc = problem(nx, ny, seed=nx + ny)
    rng = np.random.default_rng(1)
    mask[rng.integers(1, ny - 1, 60), rng.integers(1, nx - 1, 60)] = rng.integers(1, 3, 60)   # single nodes
    flat = torch.empty(nx * ny + 1, dtype=torch.uint8, device="cuda")
    dm = flat[1:].view(ny, nx)
    dm.copy_(torch.tensor(mask))
    d = [torch.tensor(a, device="cuda") for a in (phi, rhs)]
    solve_embedded_f64(d[0], d[1], dm, torch.tensor(bc, device="cuda") if with_bc else None, levels, h, nu[0], nu[1],
                       options, tol=0.0, max_cycles=1)
    ref = orc.emb_vcycles(phi, rhs, mask, bc if with_bc else None, h, levels, 1, nu1=nu[0], nu2=nu[1], options=options)
    assert rel_l2(d[0].cpu().numpy(), ref) < 1e-12
