"""fi_sharpen with weights that no gaussian has (outside [0, 1]) against the two filters and
the combination one after the other: equal bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# every weight outside [0, 1]; some; none.  The sums stay within the type: a cast of a
# negative or larger float has no defined value.
@pytest.mark.parametrize("weights", [(1.5,), (1.25, 1.5, 1.25), (-0.25, 1.5, -0.25),
                                     (0.5, 1.5, 0.5), (-0.1, 0.3, 0.6, 0.3, -0.1),
                                     (0.25, 0.5, 0.25)])
@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
def test_any_weights(weights, dtype):
    import torch

    from fluidimage_gb300 import _lib as L

    lib = L.load()
    code = {"uint8": 0, "uint16": 1}[dtype]
    ny, nx = 45, 131
    img = np.random.default_rng(4).integers(8, 11, (ny, nx)).astype(dtype)
    x = torch.as_tensor(img.view("i2") if dtype == "uint16" else img, device="cuda")
    w1, w2 = np.array(weights), np.array([0.25, 0.5, 0.25])
    r1, r2, s = len(w1) // 2, 1, L.stream_handle()
    new = lambda dt=x.dtype: torch.empty((ny, nx), dtype=dt, device="cuda")  # noqa: E731
    # the filter alone, then the same as the second filter of the combination
    for first, second, ra, rb in ((w1, w2, r1, r2), (w2, w1, r2, r1)):
        blurred, out = new(), new(torch.float64)
        L.check(lib.fi_sharpen(L.ptr(x), L.ptr(out), L.ptr(blurred), code, 1, ny, nx,
                               first.ctypes.data, ra, second.ctypes.data, rb, 3.0, s), "sharpen")
        b, f, tmp, want = new(), new(), new(), new(torch.float64)
        da, db = (torch.as_tensor(w, device="cuda") for w in (first, second))
        for src, dst, d, r in ((x, b, da, ra), (b, f, db, rb)):
            L.check(lib.fi_gaussian_filter(L.ptr(src), L.ptr(dst), L.ptr(tmp), code, 1, ny, nx,
                                           L.ptr(d), r, s), "gaussian")
        L.check(lib.fi_sharpen_combine(L.ptr(b), L.ptr(f), code, ny * nx, 3.0, L.ptr(want), s),
                "combine")
        assert int(b.max()) > 0
        assert torch.equal(blurred, b)
        assert torch.equal(out, want)


def test_blurred_apart_from_the_images():
    import torch

    from fluidimage_gb300 import _lib as L

    store = torch.zeros(64 * 64 * 10, dtype=torch.uint8, device="cuda")
    w = np.array([0.25, 0.5, 0.25])
    at = lambda k: L.ptr(store[k * 64 * 64:])  # noqa: E731
    for x, out, blurred in ((0, 2, 0), (0, 1, 2), (1, 2, 0)):
        rc = L.load().fi_sharpen(at(x), at(out), at(blurred) + 64, 0, 1, 64, 64, w.ctypes.data, 1,
                                 w.ctypes.data, 1, 3.0, L.stream_handle())
        assert rc != 0
