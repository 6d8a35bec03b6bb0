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
