"""The embedded-boundary solve's V-cycles behind a tolerance go out in groups, and the first one below
it ends the solve on the device.  Checked against the same number of V-cycles without a tolerance, bit
for bit: the iterate, the residual and the count do not depend on how far ahead the host sent cycles.
Sweep counts with an odd number of launches per level end each level in a copy."""
import pytest

from pic_cuda_b200 import _lib as L
from test_gpu_embedded import problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,levels,nu", [
    (3, 3, 1, (2, 2)), (65, 65, 4, (2, 2)), (130, 97, 5, (1, 2)), (130, 97, 5, (3, 5)), (130, 97, 1, (5, 0)),
    (385, 257, 6, (6, 1)), (2049, 1300, 6, (2, 2)),
])
@pytest.mark.parametrize("tol", [0.9, 1e-2, 1e-7])
def test_cycles_stop_where_they_converge(nx, ny, levels, nu, tol):
    import torch
    from pic_cuda_b200.engine import solve_embedded_f64
    h, opt = 1.0 / (nx - 1), L.EMB_COARSEN_ANY | L.EMB_PROLONG_BILINEAR
    phi, rhs, mask, bc = (torch.tensor(a, device="cuda") for a in problem(nx, ny, seed=nx + ny))
    a = phi.clone()
    cycles, rel, ok = solve_embedded_f64(a, rhs, mask, bc, levels, h, nu[0], nu[1], opt, tol=tol, max_cycles=23)
    assert 1 <= cycles <= 23 and ok == (rel < tol) and (ok or cycles == 23)
    b = phi.clone()
    count, rel_b, _ = solve_embedded_f64(b, rhs, mask, bc, levels, h, nu[0], nu[1], opt, tol=0.0, max_cycles=cycles)
    assert count == cycles and rel_b == rel
    assert torch.equal(a, b)
    if cycles > 1:   # one cycle fewer is not enough
        c = phi.clone()
        _, rel_c, _ = solve_embedded_f64(c, rhs, mask, bc, levels, h, nu[0], nu[1], opt, tol=0.0, max_cycles=cycles - 1)
        assert not rel_c < tol
