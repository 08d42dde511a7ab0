"""fi_tps_layout and fi_tps_members_fill (both point sets together, the y-band tiles)
against fi_tps_members over every point, one set at a time: equal counts, members,
coefficients and flags; the solve order against a stable sort of the counts."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one tile; a remainder; more tiles than are looked at directly (running extremes); an
# order by rank, sorted, and by rank past the sort's shared memory
@pytest.mark.parametrize("ny,nx,shuffled,lattice", [
    (9, 25, False, True), (33, 31, True, False), (70, 90, True, True),
    (360, 370, True, True), (702, 760, False, True), (702, 760, False, False),
    (900, 1000, False, True)])
def test_layout_matches_full_scans(ny, nx, shuffled, lattice):
    import torch

    from fluidimage_gb300 import _lib as L, engine

    lib = L.load()
    dev = torch.device("cuda")
    rng = np.random.default_rng(ny * nx)
    gy, gx = np.meshgrid(np.arange(ny) * 8.0 - 4.0, np.arange(nx) * 8.0 + 4.0, indexing="ij")
    xs = (gx + rng.integers(0, 2, gx.shape) * (0.5 if lattice else 0.25)).ravel()
    ys = (gy + rng.integers(0, 2, gy.shape) * 0.5).ravel()
    if shuffled:
        order = rng.permutation(xs.size)
        xs, ys = xs[order], ys[order]
    n = xs.size
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a, dtype=dt), device=dev)  # noqa: E731
    new = lambda k, dt: torch.empty(max(k, 1), dtype=dt, device=dev)  # noqa: E731
    i32, i64, f32, f64 = torch.int32, torch.int64, torch.float32, torch.float64
    dx = rng.normal(0, 1, n)
    dx[rng.random(n) < 0.05] = np.nan
    tx, ty, tdx, tdy = t(xs, "f4"), t(ys, "f4"), t(dx, "f4"), t(np.zeros(n), "f4")
    plan = torch.empty(L.TPS_PLAN_BYTES, dtype=torch.uint8, device=dev)
    cx, cy, ux, uy = new(n, f64), new(n, f64), new(n, f32), new(n, f32)
    p = L.ptr
    L.check(lib.fi_tps_plan_make(p(tx), p(ty), p(tdx), p(tdy), n, 200, 0.5, 20.0, p(plan), p(cx),
                                 p(cy), p(ux), p(uy), None, None), "plan")
    hdr = L.TpsPlan.from_buffer_copy(plan.cpu().numpy().tobytes())
    nv, nsub = hdr.num_centers, hdr.nb_subdomx * hdr.nb_subdomy
    px, py = t(gx.ravel(), "f8"), t(gy.ravel(), "f8")
    cap = nsub + 7  # capacities above the plan's counts
    ct, pt = -(-n // 256), -(-n // 256)
    cxy2, pxy2, clat, plat = new(2 * n, i32), new(2 * n, i32), new(1, i32), new(1, i32)
    cb, pb = new(2 * ct, f64), new(2 * pt, f64)
    counts, ncounts, offs = new(cap, i32), new(cap, i32), new(4 * cap + 6, i64)
    order = new(cap, i32)
    idx, nidx, co, nco = new(4 * n, i32), new(4 * n, i32), new(4 * n, f64), new(4 * n, f64)
    for _ in range(2):  # twice on one plan
        L.check(lib.fi_tps_layout(p(plan), cap, p(cx), p(cy), n, p(px), p(py), n, 0, p(cxy2),
                                  p(clat), p(pxy2), p(plat), p(cb), p(pb), p(counts), p(ncounts),
                                  p(offs), p(order), None), "layout")
    L.check(lib.fi_tps_members_fill(p(plan), cap, p(cx), p(cy), n, p(px), p(py), n, p(cxy2),
                                    p(clat), p(pxy2), p(plat), p(cb), p(pb), p(offs), p(idx),
                                    p(co), p(nidx), p(nco), None), "fill")
    torch.cuda.synchronize()
    want = torch.sort(counts[:nsub], descending=True, stable=True).indices
    assert torch.equal(order[:nsub], want.to(i32))
    for (qx, qy, k, xy2, lat, cnt, ind, cf, o0) in (
            (cx, cy, nv, cxy2, clat, counts, idx, co, 0),
            (px, py, n, pxy2, plat, ncounts, nidx, nco, cap)):
        wxy2, wlat = engine.lattice_coords(qx, qy, k)
        assert int(lat) == int(wlat)
        assert torch.equal(xy2[:2 * k], wxy2)
        want = new(nsub, i32)
        args = (p(wxy2), p(wlat), None, None, None)
        L.check(lib.fi_tps_members(p(plan), nsub, p(qx), p(qy), k, 0, p(want), None, None, None,
                                   *args), "count")
        assert torch.equal(cnt[:nsub], want)
        total = int(want.sum())
        assert total >= k
        woff = torch.cumsum(want.to(i64), 0) - want
        assert torch.equal(offs[o0:o0 + nsub], woff)
        wind, wcf = new(total, i32), new(total, f64)
        L.check(lib.fi_tps_members(p(plan), nsub, p(qx), p(qy), k, 1, None, p(woff), p(wind),
                                   p(wcf), *args), "members")
        assert torch.equal(ind[:total], wind)
        assert torch.equal(cf[:total], wcf)
