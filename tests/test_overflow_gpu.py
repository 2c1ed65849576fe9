"""Runs that outgrow f32 (a region of negative conductivity, so that its fields grow every step)."""
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
    sim = fdtd.Sim.try_new(grid, fdtd.Materials(eps, sig, inf, deb), None, [], ports, [], media)
    return sim


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
