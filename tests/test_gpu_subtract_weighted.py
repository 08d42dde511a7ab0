"""The rank filter and fi_subtract_weighted one after the other against fi_rank_subtract:
equal bits for every type, weight and clamp."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float32", "float64"])
@pytest.mark.parametrize("weight", [1.0, 0.7, -3.0, 2])
@pytest.mark.parametrize("clamp", [0, 1])
def test_two_steps_equal_one(dtype, weight, clamp):
    import torch

    from fluidimage_gb300 import _lib as L, preproc as P

    lib, s = L.load(), L.stream_handle()
    nt, ny, nx = 3, 70, 101
    img = np.random.default_rng(5).integers(0, 250, (nt, ny, nx)).astype(dtype)
    x = P.to_device(img)
    code, out_dt = P._DT[img.dtype], P._result_dtype(img.dtype, weight)
    new = lambda dt: P._empty((nt, ny, nx), dt, x.device)  # noqa: E731
    scratch = torch.empty(2 * x.numel(), dtype=torch.int64, device="cuda")
    for window, rank in (((1, 7, 9), 31), ((1, 7, 9), 0), ((3, 1, 1), 2), ((3, 3, 3), 13)):
        filtered, two, one = new(img.dtype), new(out_dt), new(out_dt)
        args = (code, nt, ny, nx, *window, rank, 0, 0.0)
        L.check(lib.fi_rank_filter(L.ptr(x), L.ptr(filtered), *args, L.ptr(scratch), s), "filter")
        L.check(lib.fi_subtract_weighted(L.ptr(x), L.ptr(filtered), code, x.numel(),
                                         float(weight), P._DT[out_dt], clamp, L.ptr(two), s),
                "subtract")
        L.check(lib.fi_rank_subtract(L.ptr(x), L.ptr(one), *args, float(weight), P._DT[out_dt],
                                     clamp, L.ptr(scratch), s), "both")
        assert torch.equal(two, one)
        assert clamp == 0 or float(P._as_float64(two).min()) >= 0.0
