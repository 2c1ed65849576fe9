"""Resident grids of a batch side by side (Batch tile 6, blocks_per_sm launches at a time)."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200.grid import Grid

pytestmark = pytest.mark.gpu


def test_launches_side_by_side_fit_an_sm(gpu, monkeypatch):
    """An axis so long that four launches' tables of factors outgrow an SM's shared memory: three run side
    by side, each grid bit for bit as stepped alone."""
    grid = Grid.uniform((0.0,) * 3, (1.3, 0.02, 0.024), (1300, 20, 24), 4)
    mats = fdtd.Materials.new(grid)
    sims = [fdtd.Sim.try_new(grid, mats, None, [], [fdtd.PortDef("a", [[fdtd.Edge(2, (at, 10, 12))]], 50.0)], [], fdtd.Media())
            for at in (200, 650, 1100, 900)]
    pulse = fdtd.Pulse(10e9, 5e9)
    b = fdtd.Batch(gpu, sims, [pulse] * 4, 60, tune=False, tile=6, blocks_per_sm=4)
    assert b.info()["tile"] == "resident grids" and b.info()["blocks_per_sm"] == 3
    b.step(31)
    n = 3 * int(np.prod(sims[0].dims()))
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    for q, sim in enumerate(sims):
        s = fdtd.Session(gpu, sim, 0, pulse, fdtd.Extras(max_steps=60, fused_e=True))
        s.step(31)
        for which in ("e", "h"):
            assert np.array_equal(b.read(q, which, n), s.read(which, n)), (q, which)
        s.close()
    b.close()
