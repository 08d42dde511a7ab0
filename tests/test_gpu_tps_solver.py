"""The TPS solve and evaluation (run_tps) against the oracle's FP64 systems
(compute_tps_weights, thin_plate_spline.py:168-216, and the blended interpolation of
ThinPlateSplineSubdom) at the sizes where the solver changes form: tiles of 32 unknowns
(num_centers - 3) and their remainders, 96 and 97 (one block's products), 192 (where
partial residuals move), one subdomain (clusters) and hundreds (one block each), on each
source of kernel values: the half-pixel lattice of a window grid, an irregular integer
lattice, positions off the lattice."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, rng):
    nx = int(np.ceil(np.sqrt(n)))
    gy, gx = np.meshgrid(np.arange(-(-n // nx)) * 8.0, np.arange(nx) * 10.0, indexing="ij")
    x, y = gx.ravel()[:n] + 16, gy.ravel()[:n] + 16
    if kind == "grid":  # window centres moved by odd shifts' half pixels
        x, y = x + 0.5 * rng.integers(0, 2, n), y + 0.5 * rng.integers(0, 2, n)
    elif kind == "integers":
        x, y = x + rng.integers(-2, 3, n), y + rng.integers(-2, 3, n)
    else:
        x, y = x + rng.uniform(-2, 2, n), y + rng.uniform(-2, 2, n)
    return x.astype(np.float32), y.astype(np.float32)


@pytest.mark.parametrize("kind", ["grid", "integers", "reals"])
@pytest.mark.parametrize("n,subdom", [
    (4, 4), (34, 34), (35, 35), (36, 36), (67, 67), (68, 68), (98, 98), (99, 99), (100, 100),
    (131, 131), (194, 194), (195, 195), (196, 196), (227, 227), (260, 260), (611, 611),
    (9000, 24)])
def test_solution_matches_fp64(kind, n, subdom):
    import torch

    from fluidimage_gb300.engine import run_tps
    from oracle import piv as O

    rng = np.random.default_rng(n)
    x, y = _points(kind, n, rng)
    u = (3 * np.sin(x / 40) + rng.normal(0, 0.3, n)).astype(np.float32)
    v = (2 * np.cos(y / 30) + rng.normal(0, 0.3, n)).astype(np.float32)
    # (inside the buffered subdomains, on the lattice)
    gy, gx = np.meshgrid(np.arange(y.min() + 1, y.max(), 5.0), np.arange(x.min() + 1, x.max(), 6.0),
                         indexing="ij")
    px, py = np.rint(gx.ravel()), np.rint(gy.ravel())
    dev = torch.device("cuda")
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a, dtype=dt), device=dev)  # noqa: E731
    out = run_tps(t(x, "f4"), t(y, "f4"), t(u, "f4"), t(v, "f4"), n, t(px, "f8"), t(py, "f8"),
                  px.size, subdom, 0.5, None, True, None)
    assert int(out.singular.sum()) == 0
    tps = O.TPSSubdom(np.array([y, x], dtype=np.float64), subdom, 0.5)
    assert out.nb_subdom == tps.nb_subdom
    assert tps.nb_subdom <= 2 if n == subdom else tps.nb_subdom > 304
    if min(len(i) for i in tps.indices) < 3:  # two subdomains of two of the four centres:
        return  # systems of rank 4 of 5, whose solution is rounding
    tps.init_new_positions(np.array([py, px]))
    # the refinement stops at 4e-11 of the solution; the evaluation and the oracle's own
    # LU (condition numbers up to 1e5) amplify rounding to a few 1e-10: 1e-8 has a margin
    for values, got, smooth in ((u, out.out_x, out.smooth_x), (v, out.out_y, out.smooth_y)):
        want_s, weights, _ = tps.weights_subdom(values.astype(np.float64))
        atol = 1e-8 * np.abs(values).max()
        np.testing.assert_allclose(smooth.cpu().numpy(), want_s, rtol=0, atol=atol)
        np.testing.assert_allclose(got.cpu().numpy(), tps.interpolate(weights), rtol=0, atol=atol)
