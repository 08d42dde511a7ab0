"""fi_tps_layout reads its plan and nothing else of the plan's buffer: a header copied into
another buffer, whose other bytes are anything, gives the same layout and keeps its bytes."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("centres_on,points_on", [(True, True), (True, False), (False, True)])
def test_copied_header(centres_on, points_on):
    import torch

    from fluidimage_gb300 import _lib as L, engine

    lib, p, dev = L.load(), L.ptr, torch.device("cuda")
    rng = np.random.default_rng(1)
    gy, gx = np.meshgrid(np.arange(30) * 8.0 + 4, np.arange(40) * 8.0 + 4, indexing="ij")
    n = gx.size
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a.ravel(), dtype=dt),  # noqa: E731
                                      device=dev)
    new = lambda k, dt, v: torch.full((k,), v, dtype=dt, device=dev)  # noqa: E731
    i32, i64, f32, f64 = torch.int32, torch.int64, torch.float32, torch.float64
    cx0 = gx + 0.5 * rng.integers(0, 2, gx.shape)
    cx0[17, 23] += 0.0 if centres_on else 0.25
    px0 = gx.copy()
    px0[29, 39] += 0.0 if points_on else 0.25
    xs, ys, u = t(cx0, "f4"), t(gy, "f4"), t(rng.normal(0, 1, gx.shape), "f4")
    plan = torch.zeros(L.TPS_PLAN_BYTES, dtype=torch.uint8, device=dev)
    cx, cy, ux, uy = new(n, f64, 0), new(n, f64, 0), new(n, f32, 0), new(n, f32, 0)
    L.check(lib.fi_tps_plan_make(p(xs), p(ys), p(u), p(u), n, 100, 0.5, 20.0, p(plan), p(cx),
                                 p(cy), p(ux), p(uy), None, None), "plan")
    px, py = t(px0, "f8"), t(gy, "f8")
    tiles, cap = -(-n // 256), engine.tps_subdomain_capacity(n, 100)
    results = []
    for fill in (0, 1, 255):
        copy = torch.full_like(plan, fill)
        copy[:C.sizeof(L.TpsPlan)] = plan[:C.sizeof(L.TpsPlan)]
        before = copy.clone()
        cxy2, pxy2, clat, plat = (new(k, i32, -7) for k in (2 * n, 2 * n, 1, 1))
        cb, pb = new(2 * tiles, f64, 0), new(2 * tiles, f64, 0)
        counts, ncounts, order = (new(cap, i32, 0) for _ in range(3))
        offs = new(4 * cap + 6, i64, 0)
        L.check(lib.fi_tps_layout(p(copy), cap, p(cx), p(cy), n, p(px), p(py), n, 0, p(cxy2),
                                  p(clat), p(pxy2), p(plat), p(cb), p(pb), p(counts), p(ncounts),
                                  p(offs), p(order), None), "layout")
        assert torch.equal(copy, before)
        assert (int(clat), int(plat)) == (int(centres_on), int(points_on))
        results.append((counts, ncounts, offs, order))
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
