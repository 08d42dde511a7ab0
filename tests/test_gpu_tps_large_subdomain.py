"""fi_tps_interpolate at the largest subdomains it takes: the shared memory for max_members
centres (here a capacity, far above the actual count), equal to the call with the count."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_capacity(monkeypatch):
    import torch

    from fluidimage_gb300 import _lib as L
    from fluidimage_gb300.engine import run_tps

    lib, dev = L.load(), torch.device("cuda")
    rng = np.random.default_rng(2)
    gy, gx = np.meshgrid(np.arange(12) * 8.0, np.arange(15) * 8.0, indexing="ij")
    t = lambda a, dt: torch.as_tensor(np.ascontiguousarray(a.ravel(), dtype=dt),  # noqa: E731
                                      device=dev)
    u = [rng.normal(0, 1, gx.shape) for _ in range(2)]

    def fields():
        o = run_tps(t(gx, "f4"), t(gy, "f4"), t(u[0], "f4"), t(u[1], "f4"), gx.size, t(gx, "f8"),
                    t(gy, "f8"), gx.size, 400, 0.5, None, True, None)
        return o.out_x, o.out_y

    want = fields()
    call = lib.fi_tps_interpolate

    class Lib:
        members = 0

        def __getattr__(self, name):
            return getattr(lib, name)

        def fi_tps_interpolate(self, plan, nsub, maxc, *args):
            return call(plan, nsub, self.members, *args)

    fake = Lib()
    monkeypatch.setattr(L, "load", lambda: fake)
    for fake.members in (800, 3653, 3656):  # (3656: 200 KB at 56 bytes a centre)
        got = fields()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    for fake.members in (3657, -1):
        with pytest.raises(Exception, match="too large"):
            fields()
