"""Gradients whose checkpoints are run again, and sweeps by one launch a step: designs whose history would
take more memory than their checkpoints, and the routes of grids that do not step resident
(FIELDGRID_RESIDENT=0), all against the stored history, bit for bit."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _gradient(gpu, sim, sc, spec, **kw):
    args = dict(checkpoints=spec.checkpoints, transposes=0) | kw
    return fdtd.flux_gradient(gpu, sim, 0, sc.pulse, fdtd.FluxSpec(
        spec.design_lo, spec.design_hi, spec.plane_k, spec.freq, spec.steps, **args))


def _equal(a, b):
    assert a.objective == b.objective and np.abs(a.grad_eps).max() > 0
    assert np.array_equal(a.grad_eps, b.grad_eps)
    assert np.array_equal(a.grad_sigma, b.grad_sigma)


@pytest.mark.parametrize("route", ["resident", "march"])
@pytest.mark.parametrize("dims,pml,design,steps,checkpoints,debye", [
    ((24, 24, 24), 4, (8, 8, 7), 400, 4, False),
    ((26, 24, 30), 4, (9, 8, 7), 401, 4, True),         # the Debye states among what a checkpoint keeps; a short last segment
    ((64, 60, 72), 8, (20, 18, 18), 480, 4, True),      # re-runs of a dependency cone inside the grid
])
def test_re_run_segments_give_the_stored_history(gpu, monkeypatch, dims, pml, design, steps, checkpoints, debye, route):
    scene, spec, _, _ = W.flux_design(*dims, pml=pml, design=design, steps=steps, checkpoints=checkpoints, debye=debye)
    sc = scene()
    sim = fdtd.Sim.try_new(*sc.args())
    stored = _gradient(gpu, sim, sc, spec, checkpoints=0)
    if route == "march":
        monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    again = _gradient(gpu, sim, sc, spec)
    assert stored.recompute_ms == 0.0 and again.recompute_ms > 0.0 and again.segments > 2
    _equal(stored, again)
    _equal(stored, _gradient(gpu, sim, sc, spec, transposes=1))


@pytest.mark.parametrize("dims,debye", [((24, 24, 24), False), ((40, 44, 70), False), ((70, 37, 33), False),
                                        ((40, 44, 70), True)])
def test_the_fused_adjoint_step_equals_the_separate_transposes(gpu, monkeypatch, dims, debye):
    """One launch per adjoint step on extents that leave partial (30, 14) tiles and several x-segments."""
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    scene, spec, _, _ = W.flux_design(*dims, pml=4, design=(4, 4, 3), steps=120, checkpoints=0, debye=debye)
    sc = scene()
    sim = fdtd.Sim.try_new(*sc.args())
    _equal(_gradient(gpu, sim, sc, spec), _gradient(gpu, sim, sc, spec, transposes=1))


def test_a_sweep_of_several_resident_launches(gpu):
    """A launch takes at most 1024 steps."""
    scene, spec, _, _ = W.flux_design(24, 22, 20, pml=3, design=(4, 4, 3), steps=2100, checkpoints=0, debye=True)
    sc = scene()
    sim = fdtd.Sim.try_new(*sc.args())
    _equal(_gradient(gpu, sim, sc, spec), _gradient(gpu, sim, sc, spec, transposes=1))
