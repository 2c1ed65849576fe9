"""Resident stepping (stencil_resident.cuh: many steps of a small grid in one cooperative launch) against
the same session stepped by the captured one-step kernels (FIELDGRID_RESIDENT=0). Both do the
reference's f32 operations in its order, so fields, records and accumulators must agree bit for bit;
the port records are f64 sums rounded to f32, in the same order for up to 32 edges."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W
from fieldgrid_b200.grid import Grid

pytestmark = pytest.mark.gpu


def _scene(dims, pml, poles=1, freqs=0, inductor=False, seed=7):
    """Random spheres (a fifth Debye, with `poles` poles) on a box of uneven sizes, two ports."""
    grid = Grid.uniform((0.0,) * 3, tuple(d * 1e-3 for d in dims), dims, pml)
    (eps, sig, inf, deb), tau = W.sphere_materials(dims, 10, 2, max(3, min(dims) // 4), pml, seed)
    media = fdtd.Media(fdtd.Sheets(), fdtd.Debye([(q / tau, 1.0 / q) for q in range(1, poles + 1)]), [])
    mid = tuple(d // 2 for d in dims)
    ports = [fdtd.PortDef("a", [[fdtd.Edge(2, mid)]], 50.0),
             fdtd.PortDef("b", [[fdtd.Edge(2, (mid[0], mid[1] - 1, mid[2] - 1))]], 75.0)]
    lumped = [fdtd.Lumped("l", [fdtd.Edge(2, (mid[0] + 1, mid[1], mid[2]))], fdtd.Element.Inductor(2e-9))] if inductor else []
    extras = fdtd.Extras(max_steps=60, freqs=[5e9, 9e9][:freqs], plane_k=dims[2] // 2 if freqs else None)
    sim = fdtd.Sim.try_new(grid, fdtd.Materials(eps, sig, inf, deb), None, lumped, ports, [], media)
    if freqs:
        extras.ntff = fdtd.patches(sim, 1).gpu
    return sim, fdtd.Pulse(10e9, 5e9), extras


def _run(gpu, sim, pulse, extras, chunks):
    s = fdtd.Session(gpu, sim, 0, pulse, extras)
    variant, steps = s.variant, sum(chunks)
    for k in chunks:
        s.step(k)
    n = sim.dims()
    nn, nf = int(np.prod(n)), len(extras.freqs)
    out = {"e": s.read("e", 3 * nn), "h": s.read("h", 3 * nn), "series": s.read("series", steps * 4),
           "energy": np.float64(s.energy())}
    if nf:
        out["plane"] = s.read("plane", n[0] * n[1] * nf * 10)
        out["ntff"] = s.read("ntff", len(extras.ntff) // 13 * nf * 12)
    s.close()
    return variant, out


@pytest.mark.parametrize("dims,pml,poles,freqs,inductor,fused", [
    ((12, 9, 7), 0, 1, 0, True, True),          # one cluster, no layer, 8 nodes along k
    ((21, 18, 23), 4, 1, 0, False, False),      # one cluster, 24 nodes along k
    ((30, 33, 28), 5, 2, 1, True, True),        # 29 nodes along k, two poles, every record
    ((30, 33, 33), 5, 1, 2, False, False),      # 34 nodes along k: the k + 4 neighbour outside the last group
    ((24, 40, 54), 6, 3, 1, False, True),       # 55 nodes along k
    ((61, 47, 15), 6, 1, 0, False, True),       # 16 nodes along k, every group in a layer
    ((30, 30, 12), 5, 1, 0, False, True),       # both layers meet in one group: not stepped resident
    ((90, 70, 130), 8, 1, 0, False, True),      # 131 nodes along k, several passes of the launch
    ((1100, 16, 12), 0, 1, 0, False, True),     # a long axis
])
def test_resident_steps_equal_the_one_step_kernels(gpu, monkeypatch, dims, pml, poles, freqs, inductor, fused):
    sim, pulse, extras = _scene(dims, pml, poles, freqs, inductor)
    extras.fused_e = fused
    chunks = (1, 4, 3, 1, 16)   # odd and even launches from either buffer set
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
    v0, ref = _run(gpu, sim, pulse, extras, chunks)
    monkeypatch.delenv("FIELDGRID_RESIDENT")
    v1, got = _run(gpu, sim, pulse, extras, chunks)
    assert "resident" not in v0 and ("resident" in v1) == (dims != (30, 30, 12)), (v0, v1)
    assert np.abs(ref["e"]).max() > 0
    for key, want in ref.items():
        assert np.array_equal(got[key], want), (key, np.abs(got[key] - want).max())


def test_resident_steps_beyond_the_tables_and_per_step_timing_agree(gpu, monkeypatch):
    """Steps past max_steps (the pulse and phases formed on the device, nothing recorded), and a
    session that goes back and forth between resident steps and the one-step kernels."""
    sim, pulse, extras = _scene((30, 26, 29), 5, freqs=1)
    extras.fused_e, extras.max_steps = True, 12
    out = []
    for off in (True, False):
        if off:
            monkeypatch.setenv("FIELDGRID_RESIDENT", "0")
        else:
            monkeypatch.delenv("FIELDGRID_RESIDENT")
        s = fdtd.Session(gpu, sim, 0, pulse, extras)
        s.step(9)
        s.kernel_times(2)   # two steps, one kernel at a time
        s.step(20)
        nn = int(np.prod(sim.dims()))
        out.append((s.steps, s.read("e", 3 * nn), s.read("h", 3 * nn), s.read("series", 12 * 4)))
        s.close()
    assert out[0][0] == out[1][0] == 31
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)
