"""The error of the TPS of small subdomains against the same splines in extended precision
(LU in float64, residuals and kernel values in long double until the corrections vanish).
What limits it should be the rounding of the projected matrix: 2^-48 of kernel values up to
~2e4, 7e-11, against eigenvalues from ~10 on, so a relative rms error below 1e-12; the two
sweeps of refinement that the stopping rule took for enough left 1.5e-12 to 3.2e-12."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _phi(r2):
    out = np.zeros_like(r2)
    out[r2 > 0] = r2[r2 > 0] * np.log(r2[r2 > 0]) / 2
    return out


def _spline(x, y, values, lam, qx, qy):
    """The smoothed spline through (x, y) at (qx, qy)."""
    import scipy.linalg

    n = x.size
    x, y, qx, qy = (q.astype(LD) for q in (x, y, qx, qy))
    mx, my, width = x.mean(), y.mean(), max(np.ptp(x), np.ptp(y))
    affine = lambda a, b: np.stack([np.ones(a.size, LD), (b - my) / width,  # noqa: E731
                                    (a - mx) / width], 1)
    k = _phi((y[:, None] - y) ** 2 + (x[:, None] - x) ** 2) + np.eye(n, dtype=LD) * LD(lam)
    scale = np.abs(k).max()
    a = np.zeros((n + 3, n + 3), LD)
    a[:n, :n], a[:n, n:], a[n:, :n] = k / scale, affine(x, y), affine(x, y).T
    lu = scipy.linalg.lu_factor(a.astype(float))
    b = np.concatenate([values.astype(LD), np.zeros((3, values.shape[1]), LD)])
    z = np.zeros_like(b)
    for _ in range(10):
        z += scipy.linalg.lu_solve(lu, (b - a @ z).astype(float)).astype(LD)
    f = _phi((qy[:, None] - y) ** 2 + (qx[:, None] - x) ** 2)
    return f @ (z[:n] / scale) + affine(qx, qy) @ z[n:]


@pytest.mark.parametrize("kind,subdom", [("grid", 30), ("reals", 30), ("grid", 40),
                                         ("reals", 40)])
def test_small_subdomains(kind, subdom):
    import torch

    from fluidimage_gb300.engine import run_tps
    from oracle import piv as O

    rng = np.random.default_rng(632)
    gy, gx = np.meshgrid(np.arange(24) * 8.0 + 16, np.arange(26) * 8.0 + 16, indexing="ij")
    n = gx.size
    move = (lambda: 0.5 * rng.integers(0, 2, n)) if kind == "grid" else (  # noqa: E731
        lambda: rng.uniform(-1, 1, n))
    x, y = ((a.ravel() + move()).astype(np.float32) for a in (gx, gy))
    u = (3 * np.sin(x / 40) + rng.normal(0, 0.3, n)).astype(np.float32)
    v = (2 * np.cos(y / 30) + rng.normal(0, 0.3, n)).astype(np.float32)
    t = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    py, px = (a.ravel() for a in np.meshgrid(np.arange(18, 196, 8.0), np.arange(18, 210, 8.0),
                                             indexing="ij"))
    out = run_tps(t(x), t(y), t(u), t(v), n, t(px), t(py), px.size, subdom, 0.5, None, True, None)
    assert int(out.mp_status.sum()) == 0
    tps = O.TPSSubdom(np.array([y, x], dtype=np.float64), subdom, 0.5)
    tps.init_new_positions(np.array([py, px]))
    values, want, norm = np.stack([u, v], 1), np.zeros((px.size, 2), LD), np.zeros(px.size)
    for i, (ind, q) in enumerate(zip(tps.indices, tps.ind_new)):
        coefs = tps._coef_norm(px[q], py[q], i)
        norm[q] += coefs
        want[q] += coefs[:, None] * _spline(x[ind], y[ind], values[ind], tps.smoothing_coef,
                                            px[q], py[q])
    want /= norm[:, None]
    got = np.stack([out.out_x.cpu().numpy(), out.out_y.cpu().numpy()], 1)
    error = np.sqrt(((got - want) ** 2).mean() / (want ** 2).mean())
    assert error < 1e-12
