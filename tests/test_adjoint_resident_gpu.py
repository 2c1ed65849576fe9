"""The backward sweep as resident launches (adjoint_resident.cuh) and the stored history that replaces
checkpoints where it is the smaller, against the separate transposes (transposes=1) and against
sessions that do not step resident (FIELDGRID_RESIDENT=0): the same sums in the same order, so the
gradients must be equal bit for bit."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _case(dims, pml, design, steps, checkpoints, debye):
    scene, spec, _, _ = W.flux_design(*dims, pml=pml, design=design, steps=steps, checkpoints=checkpoints)
    sc = scene()
    if debye == "slab":       # a slab beside the design, as flux_design's own
        return W.flux_design(*dims, pml=pml, design=design, steps=steps, checkpoints=checkpoints, debye=True)[0](), spec
    if debye == "plane":      # two poles, across the flux plane: Debye edges among its source's nodes
        k = spec.plane_k
        shape = tuple(dims)
        box = (slice(pml + 2, pml + 9), slice(pml + 1, pml + 8), slice(k - 2, k + 2))
        sc.mats.inf.reshape(shape)[box] = 2.0
        sc.mats.debye.reshape(shape)[box] = 3.0
        sc.mats.eps.reshape(shape)[box] = 5.0
        sc.media = fdtd.Media(fdtd.Sheets(), fdtd.Debye([(1.0 / 20e-12, 0.6), (1.0 / 90e-12, 0.4)]), [])
    return sc, spec


@pytest.mark.parametrize("dims,pml,design,steps,checkpoints,debye", [
    ((20, 18, 16), 0, (3, 3, 2), 60, 0, None),          # one cluster, no layer
    ((30, 28, 27), 4, (4, 4, 3), 90, 0, None),          # 28 nodes along k
    ((31, 34, 33), 5, (4, 5, 3), 90, 4, "slab"),        # 34 nodes along k
    ((40, 37, 45), 6, (5, 4, 4), 101, 0, "plane"),      # 46 nodes along k, an odd number of steps
    ((72, 61, 54), 8, (6, 6, 4), 64, 5, "plane"),       # several passes of the launch
])
def test_the_resident_sweep_equals_the_separate_transposes(gpu, monkeypatch, dims, pml, design, steps, checkpoints, debye):
    sc, spec = _case(dims, pml, design, steps, checkpoints, debye)
    sim = fdtd.Sim.try_new(*sc.args())
    a = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec)
    sep = fdtd.FluxSpec(spec.design_lo, spec.design_hi, spec.plane_k, spec.freq, spec.steps, checkpoints=0, transposes=1)
    b = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, sep)
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    c = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec)
    assert a.recompute_ms == 0.0 and np.abs(a.grad_eps).max() > 0
    for other in (b, c):
        assert a.objective == other.objective
        assert np.array_equal(a.grad_eps, other.grad_eps)
        assert np.array_equal(a.grad_sigma, other.grad_sigma)


@pytest.mark.parametrize("debye", [False, True])
def test_a_history_larger_than_the_checkpoints_is_run_again(gpu, debye):
    """A design that fills much of the grid: its whole history would take more than two checkpoints, so
    the segments run again, with the gradient of the stored history."""
    scene, spec, _, _ = W.flux_design(30, 30, 32, pml=4, design=(16, 16, 8), steps=240, checkpoints=4, debye=debye)
    sc = scene()
    sim = fdtd.Sim.try_new(*sc.args())
    b = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, spec)
    full = fdtd.FluxSpec(spec.design_lo, spec.design_hi, spec.plane_k, spec.freq, spec.steps, checkpoints=0)
    a = fdtd.flux_gradient(gpu, sim, 0, sc.pulse, full)
    assert b.segments == 4 and b.recompute_ms > 0.0 and a.recompute_ms == 0.0
    assert np.array_equal(a.grad_eps, b.grad_eps)
    assert np.array_equal(a.grad_sigma, b.grad_sigma)
