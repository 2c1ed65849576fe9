"""Runs that outgrow f32 (a region of negative conductivity, so that its fields grow every step): stepped
resident and by the one-step kernels (FIELDGRID_RESIDENT=0) they hold the same values, infinities and
NaNs at every node, from before the first infinity until it has spread."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W
from fieldgrid_b200.grid import Grid

pytestmark = pytest.mark.gpu


def _sim(dims, pml, debye, at, grow):
    grid = Grid.uniform((0.0,) * 3, tuple(d * 1e-3 for d in dims), dims, pml)
    (eps, sig, inf, deb), tau = W.sphere_materials(dims, 10, 2, max(3, min(dims) // 4), pml, 7)
    if not debye:
        eps, inf, deb = eps - deb, np.ones_like(inf), np.zeros_like(deb)
    else:   # ends inside 4-node groups along k, within the region
        eps.reshape(dims)[at[0], at[1] + 1:at[1] + 3, at[2] + 1:at[2] + 3] = 5.0
        deb.reshape(dims)[at[0], at[1] + 1:at[1] + 3, at[2] + 1:at[2] + 3] = 2.0
    sig.reshape(dims)[tuple(slice(a, a + 4) for a in at)] = grow
    media = fdtd.Media(fdtd.Sheets(), fdtd.Debye([(1.0 / tau, 0.7), (2.0 / tau, 0.3)] if debye else []), [])
    mid = tuple(d // 2 for d in dims)
    ports = [fdtd.PortDef("a", [[fdtd.Edge(2, mid)]], 50.0)]
    return fdtd.Sim.try_new(grid, fdtd.Materials(eps, sig, inf, deb), None, [], ports, [], media)


def _states(gpu, dims, pml, fused, debye, at):
    sim = _sim(dims, pml, debye, at, -3.0)
    s = fdtd.Session(gpu, sim, 0, fdtd.Pulse(10e9, 5e9), fdtd.Extras(max_steps=400, fused_e=fused))
    nn = int(np.prod(sim.dims()))
    out = []
    for _ in range(240):
        s.step(1)
        out.append((s.read("e", 3 * nn), s.read("h", 3 * nn)))
    resident = "resident" in s.variant
    s.close()
    return resident, out


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("dims,pml,debye,at", [
    ((30, 33, 28), 0, True, (11, 9, 12)),      # Debye groups, some of their edges not Debye
    ((30, 33, 33), 5, False, (6, 6, 6)),       # beside the layer, whose ends share 4-node groups with other nodes
    ((31, 30, 34), 6, True, (8, 8, 25)),
])
def test_both_routes_overflow_alike(gpu, monkeypatch, dims, pml, debye, at, fused):
    """Resident steps against the one-step kernels (FIELDGRID_RESIDENT=0): the same values, infinities and
    NaNs at every node after every step, from before the first infinity until it has spread."""
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    off, want = _states(gpu, dims, pml, fused, debye, at)
    monkeypatch.delenv("FIELDGRID_RESIDENT")
    on, got = _states(gpu, dims, pml, fused, debye, at)
    assert on and not off
    finite = [bool(np.isfinite(e).all()) for e, _ in want]
    assert finite[0] and not finite[-1]
    first = finite.index(False)
    for q, (a, b) in enumerate(zip(got, want)):
        for name, x, y in zip("eh", a, b):
            assert np.array_equal(x, y, equal_nan=True), (q, first, name)


def test_a_tuned_batch_starts_clean_after_trials_that_overflowed(gpu):
    """The tuner's trials run the grid past f32 before its fields and states go back to step 0."""
    sim = _sim((30, 33, 28), 0, True, (11, 9, 12), -6.0)
    b = fdtd.Batch(gpu, [sim, sim], [fdtd.Pulse(10e9, 5e9)] * 2, 60, tune=True)
    assert b.info()["tile"] == "resident grids"
    b.step(30)
    s = fdtd.Session(gpu, sim, 0, fdtd.Pulse(10e9, 5e9), fdtd.Extras(max_steps=60, fused_e=True))
    s.step(30)
    n = 3 * int(np.prod(sim.dims()))
    for which in ("e", "h"):
        want = s.read(which, n)
        assert np.isfinite(want).all()
        for q in range(2):
            assert np.array_equal(b.read(q, which, n), want), (q, which)
    s.close()
    b.close()
