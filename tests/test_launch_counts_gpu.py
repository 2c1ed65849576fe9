"""Session.launches: what step() enqueues, by the route that steps."""
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_launches_are_those_of_the_route_that_steps(gpu, monkeypatch):
    sc = W.dielectric_box(48, pml=6, steps=4)
    sim = fdtd.Sim.try_new(*sc.args())
    s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
    assert "resident" in s.variant
    assert [s.launches(k) for k in (0, 1, 1000, 1024, 1025, 5000)] == [0, 1, 1, 1, 2, 5]
    s.close()
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
    assert s.launches(7) == 7 * s.launches_per_step >= 28
    s.close()
