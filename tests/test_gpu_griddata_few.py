"""griddata of few queries, where a block takes four of them instead of sixteen."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vectors(ny, nx, keep, seed=3):
    """Vectors of a window grid of 8 px steps, half a pixel off it here and there; all but
    `keep` of them missing."""
    import torch

    g = np.random.default_rng(seed)
    gy, gx = (a.ravel() for a in np.meshgrid(8.0 * (1 + np.arange(ny)), 8.0 * (1 + np.arange(nx)),
                                             indexing="ij"))
    n = gx.size
    dx, dy = 5 * np.sin(gx / 40), 4 * np.cos(gy / 50)
    gone = g.permutation(n)[keep:]
    dx[gone] = np.nan
    dev = lambda a, t: torch.tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
    f32, i32 = torch.float32, torch.int32
    xs, ys = (dev(a + 0.5 * g.integers(0, 2, n), f32) for a in (gx, gy))
    grid = (dev(gx[:nx], i32), dev(gy[::nx], i32), nx, ny)
    return xs, ys, dev(dx, f32), dev(dy, f32), n, grid


@pytest.mark.parametrize("keep", [600, 480, 60])
@pytest.mark.parametrize("off", [-1, 0, 1, None])
def test_few_as_many(keep, off):
    """The same queries in a call of their own, at both sides of the line and for 3 of them,
    and among four times as many: equal bits."""
    import torch

    from fluidimage_gb300 import engine as E

    line = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    count = 3 if off is None else line + off
    args = _vectors(20, 30, keep)
    g = np.random.default_rng(8)
    px, py = (torch.tensor(0.5 * g.integers(0, top, 4 * line), device="cuda") for top in (520, 360))
    few = E.run_griddata(*args, px[:count].clone(), py[:count].clone(), count, None)
    many = E.run_griddata(*args, px, py, px.numel(), None)
    for name in ("out_x", "out_y", "rx", "ry", "flags"):
        assert torch.equal(getattr(few, name), getattr(many, name)[:count])


def test_time_around_few_vectors(monkeypatch):
    """414 queries around 5 vectors: 65 us with a thread a query, 99 with sixteen queries a
    block, 47 with four."""
    import torch

    from fluidimage_gb300 import _lib as L, engine as E

    lib, times = L.load(), []
    call = lib.fi_griddata

    def timed(*a):
        begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(40000)  # the launches queue behind it
        begin.record()
        status = call(*a)
        end.record()
        times.append((begin, end))
        return status

    monkeypatch.setattr(lib, "fi_griddata", timed)
    args = _vectors(2, 23, 5)
    py, px = (a.ravel() for a in np.meshgrid(8.0 * np.arange(6) / 3 // 1, 8.0 * np.arange(69) / 3 // 1,
                                             indexing="ij"))
    px, py = (torch.tensor(a, device="cuda") for a in (px, py))
    for _ in range(12):
        E.run_griddata(*args, px, py, px.numel(), None)
    torch.cuda.synchronize()
    assert min(b.elapsed_time(e) for b, e in times) < 0.07
