"""A fill that fails (here: no device memory for its masks) returns its error with both masks clear, and the
next one runs."""
import ctypes as C

import numpy as np
import pytest

from fieldgrid_b200._lib import lib
from meshes import cuboid

pytestmark = pytest.mark.gpu


def test_a_failed_fill_leaves_clear_masks(gpu):
    import torch

    n = 300
    line = np.arange(n) + 0.5
    tris = np.ascontiguousarray(cuboid((50.0,) * 3, (120.0,) * 3), np.float64)
    dp, up = C.POINTER(C.c_double), C.POINTER(C.c_uint8)
    inside, thin = np.full(n ** 3, 7, np.uint8), np.full(n ** 3, 7, np.uint8)
    err = C.create_string_buffer(256)
    s = line.ctypes.data_as(dp)

    def fill():
        return lib().fg_raster_fill(gpu._h, tris.ctypes.data_as(dp), len(tris), s, n, s, n, s, n, 0,
                                    inside.ctypes.data_as(up), thin.ctypes.data_as(up), err, 256)

    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert fill() != 0 and b"memory" in err.value, err.value
    finally:
        del hog
        torch.cuda.empty_cache()
    assert not inside.any() and not thin.any()
    assert fill() == 0
    assert inside.sum() == 70 ** 3
