"""The one-step kernels by themselves (FIELDGRID_RESIDENT=0): grids that would step resident, marched by the
TMA and the direct-load kernels, with their graphs' replays, k-layer tiles and CPML shell."""
import numpy as np
import pytest

from conftest import rel_l2
from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def one_step(monkeypatch):
    monkeypatch.setenv("FIELDGRID_RESIDENT", "0")


def _session(gpu, sc, sim, tma):
    s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
    assert "resident" not in s.variant and s.variant.startswith("TMA") == tma, s.variant
    return s


def test_the_tma_and_the_direct_march_agree_bit_for_bit(gpu, monkeypatch):
    sc = W.spheres(72, pml=6, count=16, rmin=3, rmax=14, steps=120, fused=True)
    sim = fdtd.Sim.try_new(*sc.args())
    _session(gpu, sc, sim, True).close()
    a = fdtd.run(gpu, sim, 0, sc.pulse, sc.extras, keep_fields=True)
    monkeypatch.setenv("FIELDGRID_NO_TMA", "1")
    _session(gpu, sc, sim, False).close()
    b = fdtd.run(gpu, sim, 0, sc.pulse, sc.extras, keep_fields=True)
    for name in ("e", "h", "series"):
        assert np.array_equal(getattr(a, name), getattr(b, name)), name


@pytest.mark.parametrize("fused", [True, False])
def test_graph_replays_of_any_chunks_equal_one_run(gpu, fused):
    """Graphs of 32 steps, pairs, and singles of either parity."""
    sc = W.spheres(40, pml=5, count=8, rmin=3, rmax=8, steps=101, fused=fused)
    sim = fdtd.Sim.try_new(*sc.args())
    rec = fdtd.run(gpu, sim, 0, sc.pulse, sc.extras, keep_fields=True)
    s = _session(gpu, sc, sim, fused)
    for k in (1, 33, 2, 1, 64):
        s.step(k)
    n = 3 * int(np.prod(sc.grid.dims()))
    assert np.array_equal(s.read("e", n), rec.e) and np.array_equal(s.read("h", n), rec.h)
    assert np.array_equal(s.read("series", 202), rec.series)
    s.close()
    ref = O.run_cpu(O.OracleSim(*sc.args(), bits=32), 0, sc.pulse, sc.extras, keep_fields=True)
    for name in ("e", "h", "series"):
        assert rel_l2(getattr(rec, name), getattr(ref, name)) <= 1e-4, name


def test_a_lone_tile_that_reaches_the_k_layer_matches_the_oracle(gpu):
    sc = W.spheres(10, pml=4, count=2, rmin=1, rmax=2, steps=30, fused=True)
    sim = fdtd.Sim.try_new(*sc.args())
    s = _session(gpu, sc, sim, True)
    assert "(1 reaching the k layer)" in s.variant, s.variant
    s.close()
    rec = fdtd.run(gpu, sim, 0, sc.pulse, sc.extras, keep_fields=True)
    ref = O.run_cpu(O.OracleSim(*sc.args(), bits=32), 0, sc.pulse, sc.extras, keep_fields=True)
    for name in ("e", "h", "series"):
        assert rel_l2(getattr(rec, name), getattr(ref, name)) <= 1e-4, name
