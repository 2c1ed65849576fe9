"""Every call that hands out what steps have left reports a bounded wait that ran out: the march's copy
waits (FIELDGRID_TEST_STALL_PLANE: one plane's barrier expects more bytes than are sent) and the resident
kernels' grid barrier (FIELDGRID_TEST_STALL_BARRIER: it waits for one arrival more than there are blocks),
with the limit of 10 ms in place of 2 s. The kernels return, so the device stays usable."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu

TEXT = "bounded wait in the fused step ran out"


def _stall(monkeypatch, route):
    monkeypatch.setenv("FIELDGRID_TEST_WAIT_NS", "10000000")
    if route == "march":
        monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
        monkeypatch.setenv("FIELDGRID_TEST_STALL_PLANE", "20")   # a plane inside the clean box
    else:
        monkeypatch.setenv("FIELDGRID_TEST_STALL_BARRIER", "1")


def _scene(steps=20):
    return W.spheres(40, pml=5, count=8, rmin=3, rmax=9, steps=steps, fused=True)


@pytest.mark.parametrize("route", ["march", "resident"])
def test_sessions_report_it_until_they_are_closed(gpu, monkeypatch, route):
    sc = _scene()
    sim = fdtd.Sim.try_new(*sc.args())
    nn = int(np.prod(sc.grid.dims()))
    with monkeypatch.context() as m:
        _stall(m, route)
        s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
        assert ("resident" in s.variant) == (route == "resident"), s.variant
        s.step(4)
        for call in (s.sync, lambda: s.read("e", 3 * nn), lambda: s.read("series", 8), s.energy, s.sync):
            with pytest.raises(fdtd.FdtdError, match=TEXT):
                call()
        s.close()
        with pytest.raises(fdtd.FdtdError, match=TEXT):
            fdtd.run(gpu, sim, 0, sc.pulse, sc.extras)
    s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
    s.step(4)
    s.sync()
    assert np.isfinite(s.read("e", 3 * nn)).all()
    s.close()


@pytest.mark.parametrize("route,tile", [("march", 3), ("march", 5), ("resident", 6)])
def test_batches_report_it(gpu, monkeypatch, route, tile):
    scenes = [_scene(40) for _ in range(3)]
    sims = [fdtd.Sim.try_new(*sc.args()) for sc in scenes]
    pulses = [sc.pulse for sc in scenes]
    with monkeypatch.context() as m:
        _stall(m, route)
        b = fdtd.Batch(gpu, sims, pulses, 40, tune=False, tile=tile)
        b.step(10)
        for call in (b.sync, lambda: b.read(0, "series", 20), b.sync):
            with pytest.raises(fdtd.FdtdError, match=TEXT):
                call()
        b.close()
        with pytest.raises(fdtd.FdtdError, match=TEXT):   # no trial that ended early is taken for a fast one
            fdtd.Batch(gpu, sims, pulses, 40, tune=True)
    b = fdtd.Batch(gpu, sims, pulses, 40, tune=False, tile=tile)
    b.step(10)
    b.sync()
    assert np.array_equal(b.read(0, "series", 20), b.read(2, "series", 20))
    b.close()


@pytest.mark.parametrize("grad", [False, True])
def test_flux_gradients_report_it(gpu, monkeypatch, grad):
    scene, spec, _, _ = W.flux_design(30, 28, 26, pml=4, design=(4, 4, 3), steps=40)
    sc = scene()
    sim = fdtd.Sim.try_new(*sc.args())
    with monkeypatch.context() as m:
        _stall(m, "resident")
        with pytest.raises(fdtd.FdtdError, match=TEXT):
            fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec, grad=grad)
    assert np.isfinite(fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec, grad=grad).objective)
