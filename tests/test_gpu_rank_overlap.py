"""Rank filters whose output overlaps their input: minima and maxima go through the scratch
(the tiles of the one-pass kernels would read what their neighbours have written), the
subtraction in one pass is refused."""

import numpy as np
import pytest
from scipy import ndimage

pytestmark = pytest.mark.gpu

CODES = {"uint8": 0, "uint16": 1, "float32": 2, "float64": 3}


def _tensor(a):
    import torch

    return torch.as_tensor(a.view("i2") if a.dtype == np.uint16 else a, device="cuda")


@pytest.mark.parametrize("dtype", list(CODES))
@pytest.mark.parametrize("window", [(1, 9, 7), (1, 30, 31), (3, 1, 1), (3, 2, 3)])
@pytest.mark.parametrize("shift", [0, 1])  # in place; one image row further on
def test_minima_and_maxima_in_place(dtype, window, shift):
    import torch

    from fluidimage_gb300 import _lib as L

    nt, ny, nx = 3, 150, 200
    img = np.random.default_rng(3).integers(0, 255, (nt, ny, nx)).astype(dtype)
    store = _tensor(np.zeros(img.size + nx, dtype))
    scratch = torch.empty(2 * img.size, dtype=torch.int64, device="cuda")
    for rank in (0, int(np.prod(window)) - 1):
        store[:img.size] = _tensor(img.ravel())
        out = store[shift * nx:shift * nx + img.size]
        L.check(L.load().fi_rank_filter(
            L.ptr(store), L.ptr(out), CODES[dtype], nt, ny, nx, *window, rank, 0, 0.0,
            L.ptr(scratch), L.stream_handle()), "fi_rank_filter")
        got = out.cpu().numpy().view(dtype).reshape(img.shape)
        np.testing.assert_array_equal(got, ndimage.rank_filter(img, rank, size=window))


def test_overlap_needs_the_scratch():
    from fluidimage_gb300 import _lib as L

    lib = L.load()
    store = _tensor(np.zeros(64 * 65, np.uint8))
    p, q, s = L.ptr(store), L.ptr(store[64:]), L.stream_handle()
    assert lib.fi_rank_needs_scratch(0, 1, 64, 1, 5, 5, 0) == 0
    for out in (p, q):
        assert lib.fi_rank_filter(p, out, 0, 1, 64, 64, 1, 5, 5, 0, 0, 0.0, None, s) != 0
        assert lib.fi_rank_subtract(p, out, 0, 1, 64, 64, 1, 5, 5, 0, 0, 0.0, 1.0, 0, 0, None,
                                    s) != 0
