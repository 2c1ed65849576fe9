"""Session.sync waits for the session's own steps, not for what a program has queued on other streams."""
import time

import pytest
import torch

from fieldgrid_b200 import fdtd
from fieldgrid_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_sync_does_not_wait_for_the_default_stream(gpu):
    sc = W.dielectric_box(32, pml=4, steps=4)
    sim = fdtd.Sim.try_new(*sc.args())
    s = fdtd.Session(gpu, sim, 0, sc.pulse, sc.extras)
    s.step(4)
    s.sync()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    torch.cuda._sleep(1_000_000_000)   # half a second of clocks, one thread
    done.record()
    t = time.perf_counter()
    s.step(4)
    s.sync()
    assert not done.query() and time.perf_counter() - t < 0.2
    torch.cuda.synchronize()
    s.close()
