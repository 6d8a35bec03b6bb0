"""Jobs of different depth and tolerance in one batch.  Once the deep jobs have converged, the launches of
their levels have nothing to do, and the shallow jobs' remaining V-cycles must still run in order: every
job's potential and cycle count equal the job's alone, bit for bit (int64 deposit)."""
import numpy as np
import pytest

from pic_cuda_b200 import _lib as L
from pic_cuda_b200 import configs as cf
from pic_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu


# (side, tol): the deep jobs stop cycles before the shallow ones; 2049^2 runs as strips, the others as tiles
@pytest.mark.parametrize("specs", [
    [(513, 1e-1), (257, 1e-2), (129, 1e-10), (129, 1e-11)],
    [(257, 1e-1), (129, 1e-10), (65, 1e-11), (33, 1e-11)],
    [(2049, 1e-1), (257, 1e-2), (129, 1e-10)],
])
@pytest.mark.parametrize("graph", [False, True])
def test_shallow_jobs_go_on_after_deep_ones(specs, graph):
    def make(eng, k):
        n, tol = specs[k]
        job = eng.add_job(cf.plasma(n, 0.01, 20_000, deposit=L.DEPOSIT_I64, tol=tol, omega=1.15, seed=k))
        cf.load_plasma(job, 20_000, 0.01, 2.0, 0.03, seed=50 + k)
        return job

    def state(eng, jobs):
        out = []
        for _ in range(4):
            (eng.step_graph if graph else eng.step)(1)
            eng.sync()
            out.append([(j.get_grid(L.GRID_PHI), j.diagnostics()["vcycles"]) for j in jobs])
        return out

    eng = Engine(0)
    batch = state(eng, [make(eng, k) for k in range(len(specs))])
    eng.close()
    assert batch[0][0][1] < batch[0][-1][1]   # the deep job stops first
    for k in range(len(specs)):
        eng = Engine(0)
        alone = state(eng, [make(eng, k)])
        eng.close()
        for b, a in zip(batch, alone):
            assert b[k][1] == a[0][1]
            np.testing.assert_array_equal(b[k][0], a[0][0])
