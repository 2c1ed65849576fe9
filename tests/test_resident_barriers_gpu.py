"""Small grids by the grid-wide barrier (FIELDGRID_RESIDENT=grid), the resident launch of a device that has
no room for one cluster of 16 blocks, against the cluster launch: the same fields and gradients."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [14, 22])
def test_small_grids_step_by_either_barrier(gpu, monkeypatch, cells):
    sc = W.spheres(cells, pml=4, count=4, rmin=2, rmax=5, steps=40, fused=True)
    sim = fdtd.Sim.try_new(*sc.args())
    n = 3 * int(np.prod(sc.grid.dims()))
    out = []
    for route in (None, "grid"):
        if route:
            monkeypatch.setenv("FIELDGRID_RESIDENT", route)
        s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
        assert ("resident, 16 blocks" in s.variant) == (route is None), s.variant
        assert "resident" in s.variant
        s.step(33)
        out.append((s.read("e", n), s.read("h", n), s.read("series", 66)))
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_small_gradients_sweep_by_either_barrier(gpu, monkeypatch):
    scene, spec, _, _ = W.flux_design(20, 18, 16, pml=0, design=(3, 3, 2), steps=60, checkpoints=0)
    sc = scene()
    sim = fdtd.Sim.try_new(*sc.args())
    a = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec)
    monkeypatch.setenv("FIELDGRID_RESIDENT", "grid")
    b = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec)
    assert a.objective == b.objective and np.abs(a.grad_eps).max() > 0
    assert np.array_equal(a.grad_eps, b.grad_eps) and np.array_equal(a.grad_sigma, b.grad_sigma)
