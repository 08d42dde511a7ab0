"""Rank filters along time on stacks too small to fill the chip with one thread per pixel:
the frames are split between blocks."""

import numpy as np
import pytest
from scipy import ndimage

pytestmark = pytest.mark.gpu


# one block of pixels and as many parts as frames; parts of several frames with a short
# last one; one part
@pytest.mark.parametrize("shape,st", [((95, 4, 4), 95), ((90, 16, 20), 7), ((23, 120, 121), 23),
                                      ((50, 150, 154), 5), ((11, 700, 600), 4)])
@pytest.mark.parametrize("dtype", ["uint8", "uint16", "float32", "float64"])
def test_split_frames(shape, st, dtype):
    from fluidimage_gb300 import preproc as P

    rng = np.random.default_rng(11)
    img = (rng.integers(0, 200, shape) * (1 if dtype == "uint8" else 300)).astype(dtype)
    dev = P.to_device(img)
    for kind, rank in (("min", 0), ("median", st // 2)):
        for mode in ("reflect", "constant"):
            want = ndimage.rank_filter(img, rank, size=(st, 1, 1), mode=mode)
            got = P.to_host(P.rank_filter(dev, (st, 1, 1), kind, mode=mode))
            np.testing.assert_array_equal(got, want)


def test_small_stack_is_not_a_serial_chain():
    """A pixel's 95 medians of 95 frames on one thread take 5 ms; spread, under 0.1 ms."""
    import torch

    from fluidimage_gb300 import preproc as P

    img = np.random.default_rng(12).integers(0, 255, (95, 16, 16)).astype(np.uint8)
    dev = P.to_device(img)
    times = []
    for _ in range(6):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        begin.record()
        P.temporal_median(dev)
        end.record()
        end.synchronize()
        times.append(begin.elapsed_time(end))
    assert min(times) < 1.0
