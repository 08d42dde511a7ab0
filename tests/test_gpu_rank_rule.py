"""Medians and percentiles of 2-D windows on both sides of the line between the bit-plane
and the select kernel, against the general path (any window of float64 values): equal
values for every boundary mode, odd sizes and window shapes, few and unrelated values."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,nt,ny,nx,sy,sx", [
    ("uint8", 1, 300, 411, 30, 31), ("uint8", 1, 300, 411, 5, 7), ("uint8", 9, 100, 130, 32, 32),
    ("uint16", 1, 517, 523, 31, 30), ("uint16", 1, 517, 523, 12, 20), ("uint16", 1, 40, 33, 32, 3),
    ("float32", 1, 1030, 1021, 32, 29), ("float32", 1, 200, 130, 30, 30)])
@pytest.mark.parametrize("mode", range(5))
def test_both_kernels_match_the_general_path(dtype, nt, ny, nx, sy, sx, mode):
    import torch

    from fluidimage_gb300 import _lib as L

    lib = L.load()
    rng = np.random.default_rng(ny + mode)
    y, x = np.mgrid[0:ny, 0:nx]
    smooth = 90 + 40 * np.sin(x / 23) * np.cos(y / 31)
    image = smooth + rng.integers(0, 60, (nt, ny, nx))
    if mode % 2:  # unrelated values
        image = rng.integers(0, 255 if dtype == "uint8" else 65535, (nt, ny, nx))
    image = image.astype(dtype) if dtype != "float32" else (image * 1.37 - 100).astype(dtype)
    code = {"uint8": 0, "uint16": 1, "float32": 2}[dtype]
    dev = lambda a: torch.as_tensor(a.view("i2") if a.dtype == np.uint16 else a,  # noqa: E731
                                    device="cuda")
    a, wide = dev(image), dev(image.astype(np.float64))
    out, want = torch.empty_like(a), torch.empty_like(wide)
    s = L.stream_handle()
    for rank in (sy * sx // 2, sy * sx // 10, sy * sx - 2):
        for p, q, c in ((a, out, code), (wide, want, 3)):
            L.check(lib.fi_rank_filter(L.ptr(p), L.ptr(q), c, nt, ny, nx, 1, sy, sx, rank, mode,
                                       7.0, None, s), "fi_rank_filter")
        got = out.cpu().numpy()
        got = got.view(np.uint16) if dtype == "uint16" else got
        np.testing.assert_array_equal(got.astype(np.float64), want.cpu().numpy())
