"""Particles loaded in the middle of a run with step graphs: the sort due after the step takes the band
pass for them (three launches more than the graph's own sort, whose launch that finds the due slots falls
away) and leaves them in cell order, each particle where the stream-ordered steps have it."""
import numpy as np
import pytest

from pic_cuda_b200 import _lib as L
from pic_cuda_b200 import configs as cf
from pic_cuda_b200.engine import Engine

pytestmark = pytest.mark.gpu

N, COUNT = 129, 2_100_003


def _run(graph, reload):
    eng = Engine(0)
    job = eng.add_job(cf.plasma(N, 0.01, COUNT, deposit=L.DEPOSIT_I64, walls=L.WALLS_NONE, sort_every=4, tol=0.0,
                                max_cycles=1))
    cf.load_plasma(job, COUNT, 0.01, 2.0, 0.03, seed=5)
    step = eng.step_graph if graph else eng.step
    step(3)
    if reload:
        job.load_species(0, *cf.maxwellian_state(COUNT, 0.01, 2.0, cf.ME, 9, "cuda"))
    eng.sync()
    eng.stats(reset=True)
    step(1)   # the fourth step ends with the sort
    eng.sync()
    launches = eng.stats()["kernel_launches"]
    raw = {k: v.cpu().numpy() for k, v in job.export_raw(0).items()}
    eng.close()
    return launches, raw


def test_reload_under_step_graph_takes_the_band_pass():
    plain, _ = _run(True, False)
    launches, raw = _run(True, True)
    assert launches == plain + 3 - 1
    cell = raw["cell"].astype(np.int64) & 0xFFFFFFFF
    assert (np.diff((cell >> 16) * N + (cell & 0xFFFF)) >= 0).all()
    _, ref = _run(False, True)
    a, b = np.argsort(raw["pid"]), np.argsort(ref["pid"])
    for k in raw:
        np.testing.assert_array_equal(raw[k][a], ref[k][b])
