"""Batches whose grids step resident, one to three side by side (Batch tile 6): every grid bit for bit as
stepped alone, over calls long and short enough for both ways of stepping."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [1, 2, 3])
def test_resident_grids_step_as_alone(gpu, monkeypatch, share):
    scenes = W.batch_grids(count=4, lo=24, hi=64, pml=5, steps=60, seed=11)
    sims = [fdtd.Sim.try_new(*sc.args()) for sc in scenes]
    b = fdtd.Batch(gpu, sims, [sc.pulse for sc in scenes], 60, tune=False, tile=6, blocks_per_sm=share, graph_steps=4)
    assert b.info()["tile"] == "resident grids"
    chunks = (3, 9, 1, 20)   # graphs of single steps, then resident calls of odd and even length
    for k in chunks:
        b.step(k)
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    for q, (sc, sim) in enumerate(zip(scenes, sims)):
        nn = int(np.prod(sc.grid.dims()))
        s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
        s.step(sum(chunks))
        for which, n in (("series", sum(chunks) * 2), ("e", 3 * nn), ("h", 3 * nn)):
            assert np.array_equal(b.read(q, which, n), s.read(which, n)), (q, which)
        s.close()
    b.close()


@pytest.mark.parametrize("tile", [6, 7])
def test_a_grid_that_cannot_step_resident_takes_the_merged_launches(gpu, tile):
    sc = W.spheres(12, pml=5, count=2, rmin=1, rmax=2, steps=10)   # both layers in one 4-node group along k
    sim = fdtd.Sim.try_new(*sc.args())
    b = fdtd.Batch(gpu, [sim], [sc.pulse], 10, tune=False, tile=tile)
    assert b.info()["tile"] == "merged TMA launches"
    b.step(10)
    s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
    s.step(10)
    n = 3 * int(np.prod(sc.grid.dims()))
    for which in ("e", "h"):
        assert np.array_equal(b.read(0, which, n), s.read(which, n))
    s.close()
    b.close()
