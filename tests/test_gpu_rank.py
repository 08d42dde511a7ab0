"""Rank filters, the fused background subtraction and sharpen at the sizes where their
kernels change (tile edges, windows of one and two words, packed and single pixels,
scratch and no scratch), exact against scipy.ndimage and numpy."""

import numpy as np
import pytest
from scipy import ndimage

pytestmark = pytest.mark.gpu

KINDS = (("min", None), ("median", None), ("percentile", 10.0), ("percentile", 100.0))


def _images(rng, shape, dtype):
    """A smooth background, noise and spots; float images with unrelated values, signs
    and infinities."""
    ny, nx = shape[-2:]
    back = 300 + 100 * np.sin(np.arange(nx) / 17.0)[None, :] + np.arange(ny)[:, None]
    img = back + rng.normal(0, 15, shape)
    img[rng.random(shape) < 0.03] = 4000
    if dtype.startswith("float"):
        img = (img - 350) * rng.normal(1, 0.3, shape)
        img.flat[[3, 50]] = np.inf, -np.inf
        return img.astype(dtype)
    if dtype == "uint8":
        return (img % 256).astype(dtype)
    img[..., : nx // 3] *= 14  # all sixteen bits in a part of the image
    return np.clip(img, 0, 65535).astype(dtype)


def _rank_of(size, kind, q):
    return {"min": 0, "median": size // 2}.get(kind, size - 1 if q == 100.0 else int(size * (q or 0) / 100))


@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float32", "float64"])
@pytest.mark.parametrize("window,shape,mode", [
    ((1, 1), (40, 33), "reflect"), ((2, 3), (32, 64), "mirror"), ((7, 30), (65, 95), "reflect"),
    ((32, 32), (64, 33), "wrap"), ((33, 5), (70, 40), "nearest"), ((30, 31), (31, 128), "constant"),
    ((3, 40), (35, 66), "reflect"),
])
def test_sliding_rank_filters(dtype, window, shape, mode):
    from fluidimage_gb300 import preproc as P

    rng = np.random.default_rng(5)
    img = _images(rng, (2,) + shape, dtype)
    dev = P.to_device(img)
    for kind, q in KINDS:
        r = _rank_of(window[0] * window[1], kind, q)
        want = np.stack([ndimage.rank_filter(im, r, size=window, mode=mode) for im in img])
        got = P.to_host(P.rank_filter(dev, (1,) + window, kind, q, mode=mode))
        np.testing.assert_array_equal(got, want, err_msg=f"{kind} {q}")


@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float32", "float64"])
@pytest.mark.parametrize("shape,st", [((3, 9, 7), 3), ((5, 16, 12), 4), ((8, 31, 8), 8),
                                      ((4, 8, 8), 11), ((40, 6, 10), 9), ((120, 4, 4), 2)])
def test_temporal_rank_filters(dtype, shape, st):
    from fluidimage_gb300 import preproc as P

    img = _images(np.random.default_rng(6), shape, dtype)
    dev = P.to_device(img)
    for mode in ("reflect", "constant"):
        for kind, q in KINDS:
            want = ndimage.rank_filter(img, _rank_of(st, kind, q), size=(st, 1, 1), mode=mode)
            got = P.to_host(P.rank_filter(dev, (st, 1, 1), kind, q, mode=mode))
            np.testing.assert_array_equal(got, want, err_msg=f"{mode} {kind} {q}")


@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float32", "float64"])
@pytest.mark.parametrize("weight", [1.0, 0.7, -3.0, 2])
def test_background_subtraction(dtype, weight):
    """img - weight * filtered in numpy's dtype and rounding, clamped or not."""
    from fluidimage_gb300 import preproc as P

    img = _images(np.random.default_rng(7), (4, 45, 70), dtype)
    img[~np.isfinite(img.astype(float))] = 1
    if dtype.startswith("float") and isinstance(weight, int):
        weight = float(weight)
    dev = P.to_device(img)
    for tool, size, rank in (("temporal_minima", (4, 1, 1), 0), ("temporal_median", (4, 1, 1), 2)):
        want = img - weight * ndimage.rank_filter(img, rank, size=size)
        got = P.to_host(getattr(P, tool)(dev, weight=weight))
        assert got.dtype == want.dtype
        np.testing.assert_array_equal(got, want)
    for tool, rank in (("sliding_minima", 0), ("sliding_median", 40)):
        want = img[0] - weight * ndimage.rank_filter(img[0], rank, size=9)
        want[want < 0] = 0
        got = P.to_host(getattr(P, tool)(dev[0], weight=weight, window_size=9))
        assert got.dtype == want.dtype
        np.testing.assert_array_equal(got, want)


def test_unrelated_values():
    """Images whose windows share no value: every pixel's rank is selected alone."""
    from fluidimage_gb300 import preproc as P

    rng = np.random.default_rng(8)
    for img in (rng.permutation(65536).reshape(256, 256).astype(np.uint16),
                rng.normal(size=(100, 90)).astype(np.float32)):
        want = ndimage.median_filter(img, size=30)
        got = P.to_host(P.rank_filter(P.to_device(img)[None], (1, 30, 30), "median"))[0]
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("shape", [(33, 65), (2, 64, 64), (5, 7), (1, 200)])
@pytest.mark.parametrize("sigmas", [(3.0, 1.0), (0.1, 0.4), (7.0, 2.3), (9.0, 1.0)])
def test_sharpen(dtype, shape, sigmas):
    """Two gaussian filters in the image type and the wrapping difference; half of the
    image constant (line sums next to whole numbers)."""
    from fluidimage_gb300 import preproc as P

    img = _images(np.random.default_rng(9), shape, dtype)
    img[..., shape[-1] // 2:] = np.iinfo(dtype).max
    for alpha in (30.0, 0.3):
        want = []
        for im in img.reshape((-1,) + shape[-2:]):
            b = ndimage.gaussian_filter(im, sigmas[0])
            want.append(b + alpha * (b - ndimage.gaussian_filter(b, sigmas[1])))
        got = P.to_host(P.sharpen(P.to_device(img), *sigmas, alpha))
        np.testing.assert_array_equal(got, np.reshape(want, shape))
