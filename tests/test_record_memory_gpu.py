"""Each array of a run's record is a program's own: keeping one keeps no other alive."""
import gc

import numpy as np
import psutil
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_a_kept_plane_does_not_hold_the_fields(gpu):
    sc = W.dielectric_box(180, pml=6, steps=4)
    sc.extras.freqs, sc.extras.plane_k = [5e9, 9e9], 90
    sim = fdtd.Sim.try_new(*sc.args())
    fields = 6 * int(np.prod(sc.grid.dims())) * 4   # bytes of E and H: 142 MB

    def rss():
        gc.collect()
        return psutil.Process().memory_info().rss

    first = fdtd.run(gpu, sim, 0, sc.pulse, sc.extras, keep_fields=True)
    want = first.plane.copy()
    assert first.plane.size >= 1 << 18 and first.e.flags.writeable and first.plane.flags.writeable
    h = first.h
    del first
    start, planes = rss(), []
    for _ in range(4):
        planes.append(fdtd.run(gpu, sim, 0, sc.pulse, sc.extras, keep_fields=True).plane)
    assert rss() - start < fields
    for p in planes:
        assert np.array_equal(p, want)
    assert np.abs(h).max() > 0   # outlives its record and the others
