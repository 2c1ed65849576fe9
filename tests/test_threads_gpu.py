"""Runs from several threads on one device handle: the arena kept from a session that ended goes to one of
them only, and every run's results are those of running alone."""
import threading

import numpy as np
import pytest

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_runs_from_several_threads(gpu):
    scenes = [W.spheres(n, pml=5, count=8, rmin=3, rmax=9, steps=200, fused=q % 2 == 0) for q, n in enumerate((18, 40, 41, 64, 30))]
    sims = [fdtd.Sim.try_new(*sc.args()) for sc in scenes]

    def run(q):
        return fdtd.run(gpu, sims[q], 0, scenes[q].pulse, scenes[q].extras, keep_fields=True)

    want, wrong = [run(q) for q in range(len(sims))], []

    def work(q):
        try:
            for _ in range(6):
                rec = run(q)
                for name in ("e", "h", "series"):
                    if not np.array_equal(getattr(rec, name), getattr(want[q], name)):
                        wrong.append((q, name))
        except Exception as e:   # noqa: BLE001 - reported below, on the main thread
            wrong.append((q, repr(e)))

    threads = [threading.Thread(target=work, args=(q,)) for q in range(len(sims))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
