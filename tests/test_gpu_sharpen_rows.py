"""sharpen of images at the largest number of rows of its fused kernel and beyond, exact
against scipy."""

import numpy as np
import pytest
from scipy import ndimage

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [65535 * 32, 65535 * 32 + 1])
@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
def test_rows(rows, dtype):
    from fluidimage_gb300 import preproc as P

    img = np.random.default_rng(5).integers(0, 200, (rows, 2)).astype(dtype)
    b = ndimage.gaussian_filter(img, 1.0)
    want = b + 30.0 * (b - ndimage.gaussian_filter(b, 1.0))
    got = P.to_host(P.sharpen(P.to_device(img), 1.0, 1.0, 30.0))
    np.testing.assert_array_equal(got, want)
