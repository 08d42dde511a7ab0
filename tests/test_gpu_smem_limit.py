"""Kernels whose dynamic shared memory lies between 48 KB less their own static memory and
48 KB, each as the first of its process (a larger launch before it would have raised the
kernel's limit)."""

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

# (31 + sx) x (15 + sy) keys of 4 bytes: 12285, 12288 and 12285 keys (48 KB: 12288)
MEDIAN = """
import numpy as np
from scipy import ndimage
from fluidimage_gb300 import preproc as P
img = np.random.default_rng(0).integers(0, 65535, (40, 70)).astype(np.uint16)
got = P.to_host(P.rank_filter(P.to_device(img)[None], (1, {sy}, {sx}), "median"))[0]
want = ndimage.median_filter(img, size=({sy}, {sx}), mode="reflect")
np.testing.assert_array_equal(got, want)
"""


@pytest.mark.parametrize("sy,sx", [(90, 86), (113, 65), (81, 97)])
def test_median_at_the_default_limit(sy, sx):
    code = MEDIAN.format(sy=sy, sx=sx)
    res = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
