"""Per-window plugin calls above the size that stays in pinned memory: each array is copied
once, so a call costs little more than its copies; results as for the same windows in
small calls."""

import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count", [(48, 300), (32, 513)])
def test_large_calls_equal_small_ones(n, count):
    from fluidimage_gb300.correl import CorrelGB300

    rng = np.random.default_rng(21)
    a = rng.random((count, n, n), dtype=np.float32)
    b = np.roll(a, (2, -1), (1, 2)) + 0.1 * rng.random((count, n, n), dtype=np.float32)
    plugin = CorrelGB300((n, n), nb_peaks_to_search=2)
    planes, norms = plugin.correl_batch(a, b)
    large = plugin.peaks_batch(planes.copy(), norms, apply_subpix=True)
    for k in range(0, count, 7):
        p, q = plugin.correl_batch(a[k:k + 7], b[k:k + 7])
        np.testing.assert_array_equal(planes[k:k + 7], p)
        np.testing.assert_array_equal(norms[k:k + 7], q)
        small = plugin.peaks_batch(p, q, apply_subpix=True)
        for got, want in zip(large[:6], small[:6]):
            np.testing.assert_array_equal(got[k:k + 7], want)
        assert large[6][k:k + 7] == small[6]


def test_large_call_costs_its_copies():
    import torch

    from fluidimage_gb300.correl import CorrelGB300

    n, count = 48, 1024
    rng = np.random.default_rng(22)
    a, b = (rng.random((count, n, n), dtype=np.float32) for _ in range(2))
    plugin = CorrelGB300((n, n))

    def best(call):
        times = []
        for _ in range(8):
            torch.cuda.synchronize()
            begin = time.perf_counter()
            call()
            times.append(time.perf_counter() - begin)
        return min(times)

    def copies():  # two arrays in, one out
        x, _ = (torch.from_numpy(k).cuda() for k in (a, b))
        return x.cpu().numpy()

    copies()
    plugin.correl_batch(a, b)
    # (little more than the copies with each array copied once; through one host buffer
    # for all arrays that is copied back whole, 18 times)
    assert best(lambda: plugin.correl_batch(a, b)) < 2.5 * best(copies)
