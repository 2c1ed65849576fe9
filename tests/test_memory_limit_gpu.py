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


def test_a_gradient_is_not_refused_for_the_resident_layout(gpu, monkeypatch):
    """The session fits with the layout, the sweep's buffers behind it only without."""
    import torch

    n = CELLS
    one = np.ones(n ** 3, np.float32)
    deb, design = one.copy().reshape(n, n, n), (slice(72, 78),) * 2 + (slice(40, 44),)
    deb[68:82, 68:82, 36:48] = 0.0   # no Debye edge reaches the design
    poles = fdtd.Debye([(1e9 * 2.0 ** q, 1.0 / POLES) for q in range(POLES)])
    grid = Grid.uniform((0.0,) * 3, (n * 1e-3,) * 3, (n,) * 3, 8)
    ports = [fdtd.PortDef("a", [[fdtd.Edge(2, (75, 75, 30))]], 50.0)]
    sim = fdtd.Sim.try_new(grid, fdtd.Materials(2 + deb, 0 * one, 1 + deb, deb), None, [], ports, [],
                           fdtd.Media(fdtd.Sheets(), poles, []))
    pulse = fdtd.Pulse(10e9, 5e9)
    spec = fdtd.FluxSpec(tuple(d.start for d in design), tuple(d.stop for d in design), 50, 10e9, 40)
    want = fdtd.flux_gradient(gpu, sim, 0, pulse, spec)
    sizes = []
    for route in ("1", "0"):
        monkeypatch.setenv("FIELDGRID_RESIDENT", route)
        s = fdtd.Session(gpu, sim, 0, pulse, fdtd.Extras(max_steps=40, freqs=[10e9], plane_k=50, fused_e=True))
        sizes.append(s.device_bytes)
        s.close()
    monkeypatch.delenv("FIELDGRID_RESIDENT")
    small = _sim(20, 1)
    fdtd.Session(gpu, small, 0, pulse, fdtd.Extras(max_steps=4, fused_e=True)).close()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (sizes[0] + (300 << 20)), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):   # the second finds what the first gave back
            got = fdtd.flux_gradient(gpu, sim, 0, pulse, spec)
            assert got.objective == want.objective and np.abs(want.grad_eps).max() > 0
            assert np.array_equal(got.grad_eps, want.grad_eps) and np.array_equal(got.grad_sigma, want.grad_sigma)
    finally:
        del hog
        torch.cuda.empty_cache()
