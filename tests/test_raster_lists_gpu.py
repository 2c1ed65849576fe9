"""The rasteriser's per-column crossing lists at their edges: long lists (a heap sort), coincident
crossings, more crossings than the first allocation holds, one triangle over many columns; every mask
bit for bit the oracle's."""
import numpy as np
import pytest

from fieldgrid_b200 import raster as R
from fieldgrid_b200.grid import uniform
from oracle import oracle as O
from tests.meshes import cuboid, sphere

pytestmark = pytest.mark.gpu


def _plates(n, copies):
    """n thin closed plates one above the other, each `copies` times."""
    z = np.linspace(0.05, 0.95, n)
    return np.concatenate([cuboid([0.11, 0.13, v], [0.87, 0.91, v + 0.4 / n]) for v in z for _ in range(copies)])


@pytest.mark.parametrize("mesh,lines", [
    (lambda: _plates(12, 1), (12, 13, 200)),     # 24 crossings a column: an insertion sort
    (lambda: _plates(40, 1), (12, 13, 200)),     # 80: a heap
    (lambda: _plates(40, 9), (12, 13, 200)),     # 720, coincident by nine: the lists outgrow their first room
    (lambda: cuboid([0.02, 0.03, 0.2], [0.97, 0.96, 0.8]), (160, 150, 9)),   # twelve triangles, many columns
    (lambda: sphere(0.01, 12, (0.51, 0.49, 0.5)), (20, 20, 20)),             # smaller than a cell
])
def test_fill_with_long_short_and_wide_lists_equals_the_oracle(gpu, mesh, lines):
    mesh = mesh()
    samples = [uniform(0.0, 1.0, n) for n in lines]
    got = R.fill(gpu, mesh, samples, "ijk")
    inside, thin = O.raster_fill(mesh, samples, [len(v) for v in samples], 0)
    assert np.array_equal(got.inside, np.nonzero(inside)[0])
    assert np.array_equal(got.thin, np.nonzero(thin)[0])
    assert len(got.inside) + len(got.thin) > 0


def _pieces(lo, hi, axis, parts):
    """The cuboid's surface with the faces along `axis` cut into `parts`."""
    cuts, out = np.linspace(lo[axis], hi[axis], parts + 1), []
    for a, b in zip(cuts[:-1], cuts[1:]):
        l, h = lo.copy(), hi.copy()
        l[axis], h[axis] = a, b
        out.append(cuboid(l, h))
    t = np.concatenate(out).reshape(-1, 3, 3)
    x = t[..., axis]
    return t[~((x == x[:, :1]).all(axis=1) & (x[:, 0] > lo[axis]) & (x[:, 0] < hi[axis]))]


@pytest.mark.parametrize("axis,cells", [(0, 1400), (1, 700), (1, 1400), (2, 1400)])
def test_rays_just_past_the_edge_of_a_wide_face_stay_outside(gpu, axis, cells):
    """The rays run 1.2e-6 of a cell past the box's far edges: within the hit test's 1e-9 of a triangle 1400
    cells wide (along y it fills 30 nodes too many), where the mesh's boxes keep them out. So a box fills as
    one whose faces are short pieces, which no such ray hits."""
    n = [7, 6, 9]
    n[axis] = cells + 3
    lo, hi = np.ones(3), np.array(n) - 2.0
    samples = [np.arange(k, dtype=float) for k in n]
    wide, short = (R.fill(gpu, m, samples, "ijk") for m in (cuboid(lo, hi), _pieces(lo, hi, axis, 14)))
    inside, _ = O.raster_fill(_pieces(lo, hi, axis, 14), samples, n, 0)
    assert np.array_equal(wide.inside, short.inside) and np.array_equal(wide.thin, short.thin)
    assert np.array_equal(wide.inside, np.nonzero(inside)[0]) and len(wide.inside) > 0
