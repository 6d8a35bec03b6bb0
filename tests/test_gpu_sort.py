"""Counting sort of freshly loaded slots that take the band pass: the particles come out in cell order,
each with the values it went in with, and those outside the grid last."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 33^2 and 257^2 nodes: fewer cell rows than bands, and bands of two rows; a count that ends chunks and
# warp items in remainders; the loader's place for particles outside the grid
@pytest.mark.parametrize("n,count,outside", [(33, 2_000_001, 0), (257, 2_345_679, 1000), (1025, 2_100_000, 0)])
def test_band_pass_sorts_and_keeps_particles(n, count, outside):
    import torch
    from pic_cuda_b200 import _lib as L, configs as cf
    from pic_cuda_b200.engine import Engine
    eng = Engine(0)
    job = eng.add_job(cf.plasma(n, 0.01, count, walls=L.WALLS_NONE))
    x, y, vx, vy, vz = cf.maxwellian_state(count, 0.01, 2.0, cf.ME, 3, "cuda")
    x[:outside] += 0.02
    job.load_species(0, x, y, vx, vy, vz)
    before = job.export_raw(0)
    torch.cuda.synchronize()
    job.sort()
    after = job.export_raw(0)
    torch.cuda.synchronize()
    key = after["cell"].long() & 0xFFFFFFFF
    key = (key >> 16) * n + (key & 0xFFFF)   # cells outside (all bits set) have the largest key
    assert bool((key[1:] >= key[:-1]).all())
    assert int((after["cell"] == -1).sum()) == outside
    order = torch.argsort(after["pid"])
    for k in ("cell", "fx", "fy", "vx", "vy", "vz", "pid"):
        assert torch.equal(after[k][order], before[k])
    eng.close()
