"""The row-pipeline (strip) kernels of the multigrid against its tile kernels: jobs stepped in a batch
large enough for the strips give the same bits as each job alone, where the levels run as tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 257^2 ends strips and row chunks in remainders on every level; 24 jobs are enough items for the
# strip kernels at levels 0 (down and up) and, with 513^2, level 1
@pytest.mark.parametrize("n,jobs,nu_pre,nu_post", [(257, 24, 2, 2), (257, 24, 0, 1), (257, 24, 1, 0), (257, 24, 3, 3),
                                                   (257, 24, 4, 4), (513, 24, 2, 2), (513, 24, 4, 3)])
def test_strips_equal_tiles_bitwise(n, jobs, nu_pre, nu_post):
    from pic_cuda_b200 import _lib as L, configs as cf
    from pic_cuda_b200.engine import Engine

    def make(eng, k):
        job = eng.add_job(cf.plasma(n, 0.01, 4000, deposit=L.DEPOSIT_I64, tol=0.0, max_cycles=3, nu_pre=nu_pre,
                                    nu_post=nu_post, omega=1.15, warm_start=k % 2))
        cf.load_plasma(job, 4000, 0.01, 2.0, 0.03, seed=100 + k)
        return job

    eng = Engine(0)
    batch = [make(eng, k) for k in range(jobs)]
    eng.step(2)
    eng.sync()
    for k in (0, 1, jobs - 1):
        alone = Engine(0)
        job = make(alone, k)
        alone.step(2)
        alone.sync()
        np.testing.assert_array_equal(batch[k].get_grid(L.GRID_PHI), job.get_grid(L.GRID_PHI))
        alone.close()
    eng.close()
