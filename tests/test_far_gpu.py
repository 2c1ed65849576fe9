"""Far fields on the device over patches in lines (k_far_lines) and over patches in no order
(k_far_field), against the host's sums of the same f64 formula. Both sum up to a few 10^4 terms in f64 in
different orders: the difference is held to 1e-12 of the largest field."""
import numpy as np
import pytest

from fieldgrid_b200 import fdtd

pytestmark = pytest.mark.gpu


def _box(n, spacing):
    """The patches of a closed box, face by face, with graded or uniform spacing."""
    lines = [np.concatenate([[0.0], np.cumsum(1e-3 * (1.0 + (0.3 * np.sin(np.arange(k)) if spacing == "graded" else 0.0 * np.arange(k))))])
             for k in n]
    mid = [0.5 * (v[1:] + v[:-1]) for v in lines]
    pos, area = [], []
    for a in range(3):
        u, v = (a + 1) % 3, (a + 2) % 3
        for plane in (lines[a][0], lines[a][-1]):
            p = np.zeros((n[u], n[v], 3))
            p[..., a], p[..., u], p[..., v] = plane, mid[u][:, None], mid[v][None, :]
            pos.append(p.reshape(-1, 3))
            area.append(np.outer(np.diff(lines[u]), np.diff(lines[v])).ravel())
    return np.concatenate(pos), np.concatenate(area)


@pytest.mark.parametrize("n,spacing,order", [
    ((9, 11, 8), "uniform", "lines"),       # the shortest lines that count as lines, groups of less than four
    ((30, 26, 41), "graded", "lines"),      # tiles of eight with a rest
    ((3, 5, 330), "uniform", "lines"),      # lines longer than the table: cut in two
    ((30, 26, 17), "graded", "shuffled"),   # no lines
    ((2, 2, 2), "uniform", "lines"),        # lines too short
])
@pytest.mark.parametrize("dirs", [1, 33, 200])
def test_device_far_fields_equal_the_host_sums(gpu, n, spacing, order, dirs):
    rng = np.random.RandomState(3)
    pos, area = _box(n, spacing)
    if order == "shuffled":
        at = rng.permutation(len(pos))
        pos, area = pos[at], area[at]
    acc = rng.standard_normal((len(pos), 2, 12)).astype(np.float32)
    d = rng.standard_normal((dirs, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = fdtd.Patches(pos, area, np.zeros(0, np.uint32))
    host = fdtd.Far.load(p, acc, 2, 1, 7e9, scale=(0.3, -1.2)).fields(d)
    far = fdtd.Far.load(p, acc, 2, 1, 7e9, scale=(0.3, -1.2), gpu=gpu)
    for _ in range(2):   # the second call on the layout the first one made
        got = far.fields(d)
        assert np.abs(got - host).max() <= 1e-12 * np.abs(host).max()
    assert np.abs(far.fields(d[:1]) - host[:1]).max() <= 1e-12 * np.abs(host).max()
