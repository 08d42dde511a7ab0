"""sharpen of 8 and 16 bit images at the sizes where its tiles change height (32 rows, fewer
for small images), exact against scipy."""

import numpy as np
import pytest
from scipy import ndimage

pytestmark = pytest.mark.gpu


# tiles of 8 rows (fewer rows, one more, several), 16 and 32
@pytest.mark.parametrize("shape", [(1, 1), (7, 65), (9, 64), (100, 130), (515, 509), (701, 803)])
@pytest.mark.parametrize("sigmas", [(3.0, 1.0), (8.0, 8.0)])
@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
def test_tile_heights(shape, sigmas, dtype):
    from fluidimage_gb300 import preproc as P

    img = np.random.default_rng(13).integers(0, np.iinfo(dtype).max, shape).astype(dtype)
    img[: shape[0] // 2] = 137
    b = ndimage.gaussian_filter(img, sigmas[0])
    want = b + 30.0 * (b - ndimage.gaussian_filter(b, sigmas[1]))
    got = P.to_host(P.sharpen(P.to_device(img), *sigmas, 30.0))
    np.testing.assert_array_equal(got, want)


def test_small_constant_image():
    """Every line sum in float64, 65 taps: 0.4 ms on two tiles, 0.14 ms on eight."""
    import torch

    from fluidimage_gb300 import preproc as P

    dev = P.to_device(np.full((64, 64), 137, np.uint8))
    times = []
    for _ in range(8):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        begin.record()
        P.sharpen(dev, 8.0, 8.0)
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    assert min(times) < 0.27
