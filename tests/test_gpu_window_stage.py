"""The per-window plugin's calls through pinned host memory (up to STAGE_MAX bytes) and
through device memory give the same arrays, for one window and around the limit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (64 px: 21 windows fit the pinned buffer of a correlation, 22 do not)
@pytest.mark.parametrize("n,count,nb_peaks", [(8, 1, 1), (32, 1, 3), (24, 5, 2), (64, 21, 1),
                                              (64, 22, 3), (64, 70, 1)])
@pytest.mark.parametrize("dmax", [None, 5.0])
def test_pinned_and_device_calls_agree(monkeypatch, n, count, nb_peaks, dmax):
    from fluidimage_gb300 import correl as C

    rng = np.random.default_rng(n * count)
    im0 = rng.normal(10, 3, (count, 2 * n, n))[:, ::2]  # float64, strided
    im1 = np.roll(im0, (2, -1), (1, 2)) + rng.normal(0, 0.3, im0.shape)
    plugin = C.CorrelGB300((n, n), displacement_max=dmax, nb_peaks_to_search=nb_peaks)
    results = []
    for limit in (C.STAGE_MAX, 0):
        monkeypatch.setattr(C, "STAGE_MAX", limit)
        planes, norms = plugin.correl_batch(im0, im1)
        after = planes.copy()
        peaks = plugin.peaks_batch(after, norms, apply_subpix=True)
        try:
            sub = plugin.apply_subpix(0, 0, planes[-1])
        except C.PIVError as error:
            sub = error.explanation
        results.append((planes, norms, after, *peaks[:6], peaks[6], sub))
    for got, want in zip(*results):
        if isinstance(got, np.ndarray):
            np.testing.assert_array_equal(got, want)
        else:
            assert got == want
    single, norm = plugin(im0[0], im1[0])  # the arrays are the caller's own
    plugin(im1[0], im0[0])
    np.testing.assert_array_equal(single, results[0][0][0])
    assert norm == results[0][1][0]
