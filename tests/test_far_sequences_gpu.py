"""Far fields over patches whose lines share few coordinate sequences, or so many that the directions go in
several passes, against the host's sums of the same f64 formula (both sum up to 10^6 terms in f64 in
different orders: 1e-11 of the largest field)."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd

pytestmark = pytest.mark.gpu


def _lines(sequences, share, length):
    """`sequences` sets of coordinates along z of their own, each on `share` lines."""
    rng = np.random.RandomState(5)
    z = np.sort(rng.uniform(0.0, 0.05, (sequences, 1, length)), axis=2)
    pos = np.zeros((sequences, share, length, 3))
    pos[..., 0] = rng.uniform(0.0, 0.05, (sequences, share, 1))
    pos[..., 1] = rng.uniform(0.0, 0.05, (sequences, share, 1))
    pos[..., 2] = z
    return pos.reshape(-1, 3)


@pytest.mark.parametrize("sequences,share,length,dirs", [
    (70000, 1, 8, 3),        # a sequence of its own for every line, more than a launch has parts
    (40, 1, 60, 70),         # few lines, none shared
    (4096, 33, 8, 5),        # as many sequences as the lines' kernel takes
    (4097, 33, 8, 5),        # one more
    (600, 32, 8, 9000),      # partial sums past their room: two passes over the directions
    (2, 40, 700, 40),        # lines longer than the table: cut in three
])
def test_device_far_fields_equal_the_host_sums(gpu, sequences, share, length, dirs):
    pos = _lines(sequences, share, length)
    rng = np.random.RandomState(6)
    area = rng.uniform(0.5e-6, 1e-6, len(pos))
    acc = rng.standard_normal((len(pos), 1, 12)).astype(np.float32)
    d = rng.standard_normal((dirs, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = fdtd.Patches(pos, area, np.zeros(0, np.uint32))
    some = np.unique(np.linspace(0, dirs - 1, 8).astype(int))
    host = fdtd.Far.load(p, acc, 1, 0, 9e9).fields(d[some])
    far = fdtd.Far.load(p, acc, 1, 0, 9e9, gpu=gpu)
    for _ in range(2):
        got = far.fields(d)
        assert np.isfinite(got).all()
        assert np.abs(got[some] - host).max() <= 1e-11 * np.abs(host).max()


def test_the_handles_keep_a_bounded_share_of_the_device(gpu):
    """A layout takes 104 bytes a patch and stays with its handle, of all handles together up to 1 GiB:
    sixteen of 83 MB keep twelve, and the others are laid out by each call."""
    import torch

    pos = _lines(2, 40, 10000)
    p = fdtd.Patches(pos, np.full(len(pos), 1e-6), np.zeros(0, np.uint32))
    acc = np.random.RandomState(7).standard_normal((len(pos), 1, 12)).astype(np.float32)
    d = np.array([[0.6, 0.0, 0.8], [0.0, 1.0, 0.0]])
    free = lambda: torch.cuda.mem_get_info()[0]
    first = fdtd.Far.load(p, acc, 1, 0, 9e9, gpu=gpu)
    want = first.fields(d)
    del first
    start = free()
    fars = [fdtd.Far.load(p, acc, 1, 0, 9e9, gpu=gpu) for _ in range(16)]
    for _ in range(2):
        for far in fars:
            assert np.array_equal(far.fields(d), want)
    assert start - free() < (1 << 30) + (96 << 20)
    del far, fars
    assert start - free() < 64 << 20
