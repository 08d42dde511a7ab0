"""The image deformation and its adjoint at ragged sizes (edges of the 32 x 64 tiles, fewer
pixels than a tile) and node spacings (many cells in a tile, one cell over many), against
float64 autograd of the same interpolation; and the pair minima at every alignment."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W,spacing", [(5, 3, 2), (64, 32, 16), (65, 33, 3), (63, 97, 40),
                                         (200, 31, 7), (130, 161, 200)])
def test_warp_and_adjoint_match_float64(H, W, spacing):
    import torch

    from fluidimage_gb300 import _lib as L, deform
    import deform_reference as R

    rng = np.random.default_rng(H * W)
    dev = torch.device("cuda")
    axis = lambda n: np.cumsum(np.concatenate(  # noqa: E731
        [[1.0], spacing * rng.uniform(0.6, 1.4, max(1, n // spacing))])).astype(np.float32)
    xn, yn = (torch.as_tensor(axis(n), device=dev) for n in (W, H))
    nodes = torch.as_tensor(rng.normal(0, 1.5, (2, 2, yn.numel(), xn.numel())),
                            dtype=torch.float32, device=dev)
    y, x = np.mgrid[0:H, 0:W]
    im = np.stack([100 + 30 * np.sin(x / 9 + k) + 20 * np.cos(y / 7) for k in range(2)])
    im = torch.as_tensor(im, dtype=torch.float32, device=dev)
    g_out = torch.as_tensor(rng.normal(0, 1, (2, H, W)), dtype=torch.float32, device=dev)
    got = deform.warp(nodes, xn, yn, im, 0.5)
    g_nodes, g_im = torch.zeros_like(nodes), torch.zeros_like(im)
    L.check(L.load().fi_dc_warp_backward(
        L.ptr(nodes), L.ptr(xn), xn.numel(), L.ptr(yn), yn.numel(), 0.5, L.ptr(im), L.FI_F32, 2, H,
        W, L.ptr(g_out), L.ptr(g_nodes), L.ptr(g_im), L.stream_handle()), "fi_dc_warp_backward")
    d, i = nodes.double().requires_grad_(True), im.double().requires_grad_(True)
    want = R.warp(d, xn, yn, i, 0.5)
    want.backward(g_out.double())
    # positions are good to 2e-5 px: times slopes up to 6 a pixel; the pixels' weights to
    # the same; a node sums up to a cell's pixels, each good to 1e-6 of g times the slope
    # (2e-4 where the slope changes at a pixel's edge)
    assert torch.allclose(got.double(), want.detach(), rtol=0, atol=2e-3)
    assert torch.allclose(g_im.double(), i.grad, rtol=0, atol=1e-3)
    cell = min(4 * spacing**2, H * W)
    assert torch.allclose(g_nodes.double(), d.grad, rtol=0, atol=2e-3 + 2e-5 * cell)


@pytest.mark.parametrize("dtype", ["uint8", "int16", "float32"])
@pytest.mark.parametrize("count", [1, 7, 129, 100003])
def test_pair_minima_at_every_alignment(dtype, count):
    import torch

    from fluidimage_gb300 import _lib as L

    dt = getattr(torch, dtype)
    code = {"uint8": L.FI_U8, "int16": L.FI_U16, "float32": L.FI_F32}[dtype]
    gen = torch.Generator("cuda").manual_seed(count)
    top = 255 if dtype == "uint8" else 32767
    ims = [torch.randint(1, top, (count + 16,), generator=gen, device="cuda").to(dt)
           for _ in range(2)]
    out = torch.empty(2, dtype=torch.float32, device="cuda")
    for a, b in [(0, 0), (1, 0), (0, 1), (3, 3), (2, 5), (8, 4), (13, 15)]:
        p, q = ims[0][a:a + count], ims[1][b:b + count]
        L.check(L.load().fi_images_min(L.ptr(p), L.ptr(q), code, count, L.ptr(out),
                                       L.stream_handle()), "fi_images_min")
        assert out.tolist() == [float(p.min()), float(q.min())]
