"""Grids that fit the device only without the Debye layout of resident steps (on top of the edge list, by
4-node groups): they are taken, stepped by the one-step kernels, with the same results."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W
from fieldgrid_b200.grid import Grid

pytestmark = pytest.mark.gpu

CELLS, POLES = 150, 12


def _sim(cells, poles):
    grid = Grid.uniform((0.0,) * 3, (cells * 1e-3,) * 3, (cells,) * 3, 8)
    n = cells ** 3
    one = np.ones(n, np.float32)
    media = fdtd.Media(fdtd.Sheets(), fdtd.Debye([(1e9 * 2.0 ** q, 1.0 / poles) for q in range(poles)]), [])
    ports = [fdtd.PortDef("a", [[fdtd.Edge(2, (cells // 2,) * 3)]], 50.0)]
    return fdtd.Sim.try_new(grid, fdtd.Materials(3 * one, 0 * one, 2 * one, one), None, [], ports, [], media)


def _fields(s, sim):
    n = 3 * int(np.prod(sim.dims()))
    return s.read("e", n), s.read("h", n)


def test_a_grid_is_not_refused_for_the_resident_layout(gpu, monkeypatch):
    import torch

    sim, small = _sim(CELLS, POLES), _sim(20, 1)
    pulse, extras = fdtd.Pulse(10e9, 5e9), fdtd.Extras(max_steps=20, fused_e=True)

    def session(x=sim):
        return fdtd.Session(gpu, x, 0, pulse, extras)

    s = session()
    assert "resident" in s.variant
    full = s.device_bytes
    s.step(9)
    want = _fields(s, sim)
    s.close()
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    s = session()
    lean = s.device_bytes
    s.close()
    monkeypatch.delenv("FIELDGRID_RESIDENT")
    assert full - lean > 256 << 20
    session(small).close()   # the arena kept for the next session is a small one

    def leave(size):   # fills the device but for `size` bytes
        torch.cuda.empty_cache()
        return torch.empty(torch.cuda.mem_get_info()[0] - size, dtype=torch.uint8, device="cuda")

    reserve, half = 256 << 20, (full - lean) // 2   # a session leaves 256 MB of the device
    hog = leave(lean + reserve + half)
    try:
        s = session()
        assert "resident" not in s.variant and s.device_bytes == lean
        s.step(9)
        for a, b in zip(_fields(s, sim), want):
            assert np.array_equal(a, b)
        s.close()
        session(small).close()
        del hog
        hog = leave(2 * lean + reserve + half)   # one grid with the layout, not the second beside it
        b = fdtd.Batch(gpu, [sim, sim], [pulse] * 2, 20, tune=False, tile=6)
        assert b.info()["tile"] != "resident grids"
        b.step(9)
        n = 3 * int(np.prod(sim.dims()))
        for q in range(2):
            assert np.array_equal(b.read(q, "e", n), want[0])
        b.close()
    finally:
        del hog
        torch.cuda.empty_cache()
        session(small).close()
