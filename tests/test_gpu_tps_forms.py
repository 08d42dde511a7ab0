"""The mixed-precision TPS solve keeps every subdomain it should (no FP64 fallback) over
sizes, sources of kernel values and smoothing, and is right for the smallest systems: one
subdomain of 4 to 12 centres, and more subdomains of at most 13 centres than SMs."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, rng):
    nx = int(np.ceil(np.sqrt(n)))
    gy, gx = np.meshgrid(np.arange(-(-n // nx)) * 8.0, np.arange(nx) * 10.0, indexing="ij")
    x, y = gx.ravel()[:n] + 16, gy.ravel()[:n] + 16
    if kind == "grid":
        x, y = x + 0.5 * rng.integers(0, 2, n), y + 0.5 * rng.integers(0, 2, n)
    elif kind == "integers":
        x, y = x + rng.integers(-2, 3, n), y + rng.integers(-2, 3, n)
    else:
        x, y = x + rng.uniform(-2, 2, n), y + rng.uniform(-2, 2, n)
    return x.astype(np.float32), y.astype(np.float32)


def _run(kind, n, subdom, smoothing):
    import torch

    from fluidimage_gb300.engine import run_tps

    rng = np.random.default_rng(n)
    x, y = _points(kind, n, rng)
    u = (3 * np.sin(x / 40) + rng.normal(0, 0.3, n)).astype(np.float32)
    v = (2 * np.cos(y / 30) + rng.normal(0, 0.3, n)).astype(np.float32)
    gy, gx = np.meshgrid(np.arange(y.min() + 1, y.max(), 5.0), np.arange(x.min() + 1, x.max(), 6.0),
                         indexing="ij")
    px, py = np.rint(gx.ravel()), np.rint(gy.ravel())
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a, dtype=dt), device="cuda")  # noqa: E731
    out = run_tps(t(x, "f4"), t(y, "f4"), t(u, "f4"), t(v, "f4"), n, t(px, "f8"), t(py, "f8"),
                  px.size, subdom, smoothing, None, True, None)
    return out, (x, y, u, v, px, py)


@pytest.mark.parametrize("kind", ["grid", "integers", "reals"])
@pytest.mark.parametrize("smoothing", [1e-6, 0.5, 5.0, 1e3])
@pytest.mark.parametrize("n,subdom", [(9, 36), (99, 99), (100, 100), (195, 195), (196, 196),
                                      (2000, 40), (2000, 200), (9000, 24)])
def test_no_fallback(kind, smoothing, n, subdom):
    out, _ = _run(kind, n, subdom, smoothing)
    assert int(out.mp_status.sum()) == 0
    assert 2 <= int(out.mp_sweeps.min()) and int(out.mp_sweeps.max()) < 60


# tolerance: entries of K below 1e4 rounded to 2^-48 of it, against a smoothing of 2 and
# more, 2e-11 of the values, with a margin of 50
@pytest.mark.parametrize("kind", ["grid", "integers", "reals"])
@pytest.mark.parametrize("n,subdom", [(k, 4 * k) for k in range(4, 13)] + [(900, 4)])
def test_smallest_systems(kind, n, subdom):
    import torch

    from oracle import piv as O

    out, (x, y, u, v, px, py) = _run(kind, n, subdom, 0.5)
    tps = O.TPSSubdom(np.array([y, x], dtype=np.float64), subdom, 0.5)
    assert out.nb_subdom == tps.nb_subdom
    if n > 12:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert tps.nb_subdom > sms and max(len(i) for i in tps.indices) <= 13
        assert min(len(i) for i in tps.indices) >= 4
    else:
        assert tps.nb_subdom == 1 and int(out.mp_status.sum()) == 0
    tps.init_new_positions(np.array([py, px]))
    for values, got, smooth in ((u, out.out_x, out.smooth_x), (v, out.out_y, out.smooth_y)):
        want_s, weights, _ = tps.weights_subdom(values.astype(np.float64))
        atol = 1e-9 * np.abs(values).max()
        np.testing.assert_allclose(smooth.cpu().numpy(), want_s, rtol=0, atol=atol)
        np.testing.assert_allclose(got.cpu().numpy(), tps.interpolate(weights), rtol=0, atol=atol)
