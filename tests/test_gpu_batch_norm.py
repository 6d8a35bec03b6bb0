"""A job's residual norm, and with it the cycle its solve stops at, does not depend on the jobs it is
stepped with: relres, cycle count and potential equal the job's alone, bit for bit (int64 deposit)."""
import numpy as np
import pytest

from pic_cuda_b200 import _lib as L
from pic_cuda_b200 import configs as cf
from pic_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _run(jobs, steps=2):
    """jobs: (side, tol, nu_pre, nu_post, seed) each; per step and job phi, relres and cycle count."""
    eng = Engine(0)
    made = []
    for n, tol, nu_pre, nu_post, seed in jobs:
        job = eng.add_job(cf.plasma(n, 0.01, 4000, deposit=L.DEPOSIT_I64, tol=tol, nu_pre=nu_pre, nu_post=nu_post,
                                    omega=1.15, warm_start=seed % 2))
        cf.load_plasma(job, 4000, 0.01, 2.0, 0.03, seed=100 + seed)
        made.append(job)
    out = []
    for _ in range(steps):
        eng.step(1)
        eng.sync()
        for job in made:
            d = job.diagnostics()
            out.append((d["relres"], d["vcycles"], job.get_grid(L.GRID_PHI)))
    eng.close()
    return out


# enough level-0 rows over all jobs for another kernel than a job alone would take; a large job beside
# small ones; pre-smoothing counts of which no kernel with compile-time shapes fits every job
@pytest.mark.parametrize("jobs", [
    [(257, 1e-6, 2, 2, k) for k in range(32)],
    [(513, 1e-7, 1, 3, k) for k in range(10)] + [(129, 1e-8, 1, 3, 10)],
    [(2049, 1e-5, 2, 2, 0), (1025, 1e-6, 2, 2, 1), (257, 1e-7, 2, 2, 2), (65, 1e-8, 2, 2, 3)],
    [(257, 1e-7, 2, 2, 0), (257, 1e-7, 3, 2, 1), (129, 1e-7, 2, 2, 2)],
], ids=["many_257", "many_513", "uneven", "mixed_pre"])
def test_norm_does_not_depend_on_the_batch(jobs):
    batch = _run(jobs)
    for k in sorted({0, 1, len(jobs) // 2, len(jobs) - 1}):
        for step, alone in enumerate(_run([jobs[k]])):
            b = batch[step * len(jobs) + k]
            assert b[1] == alone[1], (k, step)
            assert b[0] == alone[0], (k, step)
            np.testing.assert_array_equal(b[2], alone[2])


# post-smoothing counts of which no kernel with compile-time shapes fits every job: the general kernel
# runs jobs that have such a kernel when alone
@pytest.mark.parametrize("jobs", [
    [(257, 1e-7, 2, 2, 0), (257, 1e-7, 2, 3, 1), (129, 1e-7, 2, 2, 2), (129, 1e-7, 5, 6, 3)],
    [(2049, 1e-5, 2, 2, 0), (257, 1e-7, 2, 3, 1), (65, 1e-8, 1, 1, 2)],
], ids=["tiles", "tiles_and_strips"])
def test_mixed_post_smoothing_keeps_each_result(jobs):
    test_norm_does_not_depend_on_the_batch(jobs)


# every kernel that sums the norm: the one-CTA solver's update, 1024- and 256-thread tiles, strips and the
# general kernel.  Tolerance: the residual's own rounding, a few ulp of phi / h^2 per node, and 1e-13 for the sums.
@pytest.mark.parametrize("n", [3, 33, 65, 129, 257, 1025, 2049])
@pytest.mark.parametrize("nu", [1, 2, 4, 5])
def test_norm_equals_the_residual_of_phi(n, nu):
    import torch
    from pic_cuda_b200.engine import solve_multigrid_f64
    h = 0.3 / (n - 1)
    rho = torch.randn((n, n), dtype=torch.float64, generator=torch.Generator().manual_seed(n)).cuda()
    for cycles in (1, 3):
        phi = torch.zeros_like(rho)
        _, rel, _ = solve_multigrid_f64(phi, rho, n, n, 0, h, 1.15, nu, nu, 2, 0.0, cycles)
        p, f = phi.cpu().numpy().astype(np.longdouble), rho.cpu().numpy().astype(np.longdouble)
        r = f[1:-1, 1:-1] - (p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:] - 4 * p[1:-1, 1:-1]) / (
            np.longdouble(h) * np.longdouble(h))
        rnorm, fnorm = np.sqrt((r * r).sum()), np.sqrt((f * f).sum())
        tol = 1e-13 + 16 * 2.0 ** -53 * n * float(np.abs(p).max() / h / h / rnorm)
        assert abs(rel / float(rnorm / fnorm) - 1) < tol
    zero = torch.zeros_like(rho)
    assert solve_multigrid_f64(zero.clone(), zero, n, n, 0, h, 1.15, nu, nu, 2, 0.0, 2)[1] == 0.0
