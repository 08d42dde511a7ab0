"""The work whose speed this repository measures: PIV works, their blocks and the
preprocessing of images, each through the entry points that a program calls.

A case is a dict of plain values; ``kind`` says which entry point it takes:

* ``window``  one window pair through the per-window plugin (``CorrelGB300``): what an
  installed fluidimage calls for each vector when the plugin is registered there;
* ``piv``     one image pair through ``WorkPIV``: ``calcul_device`` for images that are
  on the device already, ``calcul`` (``host``) from and to host arrays;
* ``batch``   many image pairs of mixed shapes through ``PIVBatch``;
* ``tps``     the thin-plate-spline interpolation of one pass's vectors (``run_tps``);
* ``refine``  forward and backward pass of ``DeformCorrelate`` (one refinement step);
* ``tool``    one preprocessing tool over images, through ``WorkPreproc``.

Images are rendered from the seed on the GPU: Gaussian particles of the densities,
diameters, intensities and noise of the repository's own workloads, moved by a vortex or
a sinusoid.  Particle contributions are added as integers, so that the order of the
additions does not matter.
"""

import math
import random

import numpy as np
import torch

from fluidimage_gb300 import WorkPIV
from fluidimage_gb300.batch import PIVBatch
from fluidimage_gb300.correl import CorrelGB300
from fluidimage_gb300.deform import DeformCorrelate, node_grid
from fluidimage_gb300.engine import run_tps
from fluidimage_gb300.preproc import WorkPreproc

BATCH_SHAPES = ((512, 512), (768, 1024), (600, 811), (1024, 1280), (2048, 2048))
BATCH_WINDOWS = (16, 24, 32, 48, 64)


def _piv(name, height, width, dtype, window, passes, overlap, tps, **more):
    case = {"kind": "piv", "height": height, "width": width, "dtype": dtype, "window": window,
            "passes": passes, "overlap": overlap, "tps": tps, "subdom": 200, "smoothing": 0.5,
            "neighbour": 2.0, "host": False}
    case.update(more)
    return dict(case, name=name) if name else case


def _tool(name, tool, frames, height, width, dtype, **args):
    case = dict({"kind": "tool", "tool": tool, "frames": frames, "height": height,
                 "width": width, "dtype": dtype}, **args)
    return dict(case, name=name) if name else case


def listed():
    return [
        # the smallest call: one vector of an upstream run that uses the plugin; one
        # plane, one peak search, one subpixel fit, from and to host arrays
        {"name": "window_32", "kind": "window", "n": 32},
        # a small single pass (a quick look at one pair, a region of interest): float
        # images, few windows, little work per launch
        _piv("single_512_f32", 512, 512, "float32", 32, 1, 0.5, "last"),
        # the reference's usual run at full size, and the repository's benchmark: three
        # passes 64 -> 32 -> 16 px with the TPS between them, 12-bit camera images
        _piv("multipass_2048_u16", 2048, 2048, "uint16", 64, 3, 0.5, "all"),
        # upstream's default parameters over three passes (48 -> 24 -> 12 px, griddata
        # between them) on an 8-bit camera frame, from and to host memory
        _piv("default_1024x1280_host", 1024, 1280, "uint8", 48, 3, 0.5, "last", smoothing=5.0,
             neighbour=10.0, host=True),
        # the largest call: a 16-megapixel pair at overlap 0.75 (259 081 vectors)
        _piv("single_4096_ov75", 4096, 4096, "uint16", 32, 1, 0.75, "last", subdom=256),
        # a series of pairs of several cameras and settings, kept on the device
        {"name": "batch_12", "kind": "batch", "jobs": 12, "mix": 3},
        # the interpolation of a full-size pass (16 px windows of a 2048^2 pair) on its
        # own grid: the largest single block of a multipass run
        {"name": "tps_255x255", "kind": "tps", "ny": 255, "nx": 255, "step": 8, "zoom": 1,
         "subdom": 200, "smoothing": 0.5},
        # one gradient step of the field refinement on two full-size pairs
        {"name": "refine_2x2048", "kind": "refine", "pairs": 2, "height": 2048, "width": 2048,
         "dtype": "float32"},
        # background removal with the toolbox's defaults (30 px window): the median of a
        # full-size frame, and the minimum over a small series of 8-bit frames
        _tool("sliding_median_2048", "sliding_median", 1, 2048, 2048, "uint16", window=30),
        _tool("sliding_minima_4x512", "sliding_minima", 4, 512, 512, "uint8", window=30),
        # background removal over time: the minimum over a burst of frames
        _tool("temporal_minima_8x2048", "temporal_minima", 8, 2048, 2048, "uint16"),
        # the toolbox's sharpening with its defaults
        _tool("sharpen_2048", "sharpen", 1, 2048, 2048, "uint16"),
    ]


# ------------------------------------------------------------------------ draw
def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("piv", "piv", "piv", "piv", "tool", "tool", "tool", "tps", "batch",
                       "refine", "window"))
    if kind == "window":
        return {"kind": "window", "n": rng.choice((16, 24, 32, 48, 64))}
    if kind == "piv":
        passes = rng.choice((1, 1, 2, 3))
        last = rng.choice((8, 12, 16, 24, 32) if passes > 1 else (8, 12, 16, 24, 32, 48, 64))
        while last * 2 ** (passes - 1) > 64:
            passes -= 1
        window = last * 2 ** (passes - 1)
        overlap = rng.choice((0.25, 0.5, 0.5, 0.75))
        lo = max(160, 5 * window)
        height, width = _log_int(rng, lo, 4096), _log_int(rng, lo, 4096)
        step = last - round(overlap * last)
        while (height // step) * (width // step) > 120000:
            height, width = max(lo, int(0.8 * height)), max(lo, int(0.8 * width))
        tps = rng.choice(("last", "last", "all", "none") if passes > 1 else ("last", "none"))
        return _piv(None, height, width, rng.choice(("uint8", "uint16", "uint16", "float32")),
                    window, passes, overlap, tps, subdom=rng.choice((100, 200, 256)),
                    smoothing=rng.choice((0.5, 2.0, 5.0)), host=rng.random() < 0.3)
    if kind == "batch":
        return {"kind": "batch", "jobs": _log_int(rng, 2, 12), "mix": rng.randrange(10 ** 6)}
    if kind == "tps":
        nx, ny = _log_int(rng, 16, 255), _log_int(rng, 16, 255)
        zoom = 2 if nx * ny < 16000 and rng.random() < 0.5 else 1
        return {"kind": "tps", "ny": ny, "nx": nx, "step": rng.choice((4, 6, 8, 16, 32)),
                "zoom": zoom, "subdom": rng.choice((100, 200, 256)),
                "smoothing": rng.choice((0.5, 2.0, 5.0))}
    if kind == "refine":
        return {"kind": "refine", "pairs": rng.choice((1, 2)), "height": _log_int(rng, 96, 2048),
                "width": _log_int(rng, 96, 2048),
                "dtype": rng.choice(("uint8", "uint16", "float32"))}
    tool = rng.choice(("sliding_minima", "sliding_median", "sliding_percentile",
                       "temporal_minima", "temporal_median", "temporal_percentile", "sharpen"))
    dtype = rng.choice(("uint8", "uint16", "uint16", "float32"))
    height, width = _log_int(rng, 128, 2048), _log_int(rng, 128, 2048)
    if tool.startswith("sliding"):
        return _tool(None, tool, rng.choice((1, 1, 2, 4)) if height * width < 2 ** 20 else 1,
                     height, width, dtype, window=_log_int(rng, 5, 30))
    if tool.startswith("temporal"):
        return _tool(None, tool, rng.randint(3, 8), height, width, dtype)
    return _tool(None, tool, 1, height, width, dtype)


# --------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(gen, count, lo, hi):
    return lo + (hi - lo) * torch.rand(count, generator=gen, device="cuda", dtype=torch.float64)


def _vortex(x, y, height, width, peak):
    """An Oseen vortex at the centre, its core a tenth of the image (peak velocity
    ``peak`` px)."""
    rc = 0.1 * min(height, width)
    x, y = x - 0.5 * (width - 1), y - 0.5 * (height - 1)
    r2 = (x * x + y * y).clamp_min(1e-9)
    u = peak * rc / 0.6382 * (1.0 - torch.exp(-r2 / rc ** 2)) / r2
    return -u * y, u * x


def _sinusoid(x, y, height, width, peak):
    k = 2 * math.pi / 512.0
    return peak * torch.sin(k * y), peak * torch.cos(k * x)


def _render(height, width, x, y, diam, peak):
    out = torch.zeros(height * width, dtype=torch.int32, device="cuda")
    ix, iy = torch.floor(x), torch.floor(y)
    inv = -8.0 / diam ** 2
    for oy in range(-4, 5):
        gy = torch.exp(inv * (iy + oy - y) ** 2) * peak * 256.0
        row = iy + oy
        ok_y = (row >= 0) & (row < height)
        for ox in range(-4, 5):
            col = ix + ox
            ok = ok_y & (col >= 0) & (col < width)
            v = torch.round(gy * torch.exp(inv * (col - x) ** 2)).to(torch.int32)
            at = (row * width + col).to(torch.int64)
            out.index_add_(0, torch.where(ok, at, 0), torch.where(ok, v, 0))
    return out.view(height, width).to(torch.float64) / 256.0


def _storage(im, dtype):
    """Pixel values as the device type of ``dtype`` (uint16 in int16 storage)."""
    if dtype == "uint8":
        return im.clamp(0, 255).to(torch.uint8)
    if dtype == "uint16":
        v = im.clamp(0, 4095).to(torch.int32)
        return torch.where(v > 32767, v - 65536, v).to(torch.int16)
    return im.clamp(0, 4095).to(torch.float32)


def _pair(gen, height, width, dtype, field=_vortex, peak=6.0):
    margin = 16.0
    count = int(0.05 * (height + 2 * margin) * (width + 2 * margin))
    x0 = _uniform(gen, count, -margin, width - 1 + margin)
    y0 = _uniform(gen, count, -margin, height - 1 + margin)
    diam = _uniform(gen, count, 2.0, 3.0)
    top = 255.0 if dtype == "uint8" else 4000.0
    bright = _uniform(gen, count, 0.25 * top, top)
    x1, y1 = x0, y0
    for _ in range(3):
        dx, dy = field(0.5 * (x0 + x1), 0.5 * (y0 + y1), height, width, peak)
        x1, y1 = x0 + dx, y0 + dy
    noise = 2.0 if dtype == "uint8" else 20.0
    ims = []
    for x, y in ((x0, y0), (x1, y1)):
        im = _render(height, width, x, y, diam, bright)
        im = im + noise * torch.randn((height, width), generator=gen, device="cuda",
                                      dtype=torch.float64)
        ims.append(_storage(torch.round(im), dtype))
    return ims


def _frames(gen, case):
    """Frames of a burst: moving particles over an uneven, static background."""
    height, width, dtype = case["height"], case["width"], case["dtype"]
    top = 255.0 if dtype == "uint8" else 4000.0
    yy = torch.arange(height, device="cuda", dtype=torch.float64)[:, None] / height
    xx = torch.arange(width, device="cuda", dtype=torch.float64)[None, :] / width
    back = 0.08 * top * (1.0 + 0.5 * torch.sin(5.0 * xx + 2.0 * yy) + 0.3 * yy)
    out = []
    for _ in range(case["frames"]):
        count = int(0.03 * height * width)
        im = _render(height, width, _uniform(gen, count, 0, width - 1),
                     _uniform(gen, count, 0, height - 1), _uniform(gen, count, 2.0, 3.0),
                     _uniform(gen, count, 0.2 * top, 0.8 * top))
        im = im + back + 0.005 * top * torch.randn((height, width), generator=gen,
                                                   device="cuda", dtype=torch.float64)
        out.append(_storage(torch.round(im), dtype))
    return torch.stack(out) if case["frames"] > 1 else out[0]


def _host(im):
    a = im.cpu().numpy()
    return a.view(np.uint16) if a.dtype == np.int16 else a


#: the works of this program, one per set of parameters (a user builds a work once and
#: gives it the pairs of a series); the oldest is dropped
_WORKS = {}


def _work(case, make):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _WORKS:
        while len(_WORKS) >= 16:
            _WORKS.pop(next(iter(_WORKS)))
        _WORKS[key] = make()
    return _WORKS[key]


def _piv_params(case):
    params = WorkPIV.create_default_params()
    params.piv0.shape_crop_im0 = case["window"]
    params.piv0.grid.overlap = case["overlap"]
    params.multipass.number = case["passes"]
    params.multipass.use_tps = {"all": True, "last": "last", "none": False}[case["tps"]]
    params.multipass.subdom_size = case["subdom"]
    params.multipass.smoothing_coef = case["smoothing"]
    params.fix.threshold_diff_neighbour = case["neighbour"]
    return params


def _preproc_params(case):
    params = WorkPreproc.create_default_params()
    tool = getattr(params.tools, case["tool"])
    tool.enable = True
    if "window" in case:
        tool.window_size = case["window"]
    return params


def _batch_jobs(case):
    """(height, width, window, overlap) of each pair: a property of the case."""
    rng = random.Random(case["mix"])
    return [rng.choice(BATCH_SHAPES) + (rng.choice(BATCH_WINDOWS), rng.choice((0.5, 0.5, 0.75)))
            for _ in range(case["jobs"])]


def _tps_inputs(case, seed):
    """The vectors of a pass: centres on the window grid or half a pixel off it (odd
    window shifts), float32 displacements of a vortex with noise, half a percent of
    outliers and half a percent of missing vectors; and the grid to interpolate at."""
    gen = _generator(seed)
    ny, nx, step = case["ny"], case["nx"], case["step"]
    gy, gx = torch.meshgrid(
        step + step * torch.arange(ny, device="cuda", dtype=torch.float64),
        step + step * torch.arange(nx, device="cuda", dtype=torch.float64), indexing="ij")
    gx, gy = gx.reshape(-1), gy.reshape(-1)
    dx, dy = _vortex(gx, gy, (ny + 1) * step, (nx + 1) * step, 8.0)
    n = nx * ny
    xs = gx + 0.5 * torch.remainder(torch.round(dx), 2.0)
    ys = gy + 0.5 * torch.remainder(torch.round(dy), 2.0)
    dx = dx + 0.05 * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    dy = dy + 0.05 * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    lot, few = torch.randperm(n, generator=gen, device="cuda"), n // 200
    dx = torch.where(lot < few, dx + 4.0, dx)
    dx = torch.where(lot >= n - few, float("nan"), dx)
    dy = torch.where(lot >= n - few, float("nan"), dy)
    z = case["zoom"]
    py, px = torch.meshgrid(
        step + step // z * torch.arange(z * ny, device="cuda", dtype=torch.float64),
        step + step // z * torch.arange(z * nx, device="cuda", dtype=torch.float64),
        indexing="ij")
    return {"xs": xs.float(), "ys": ys.float(), "dx": dx.float(), "dy": dy.float(),
            "px": px.reshape(-1).contiguous(), "py": py.reshape(-1).contiguous()}


def _refine_inputs(case, seed):
    gen = _generator(seed)
    height, width = case["height"], case["width"]
    pairs = [_pair(gen, height, width, case["dtype"], _sinusoid, 4.0)
             for _ in range(case["pairs"])]
    xn, yn = (torch.from_numpy(c).cuda() for c in node_grid(height, width))
    y, x = torch.meshgrid(yn.double(), xn.double(), indexing="ij")
    u, v = _sinusoid(x, y, height, width, 4.0)
    nodes = torch.stack([u, v]).expand(case["pairs"], 2, -1, -1)
    nodes = nodes + 0.4 * torch.randn(nodes.shape, generator=gen, device="cuda",
                                      dtype=torch.float64)
    return {"nodes": nodes.float().contiguous(), "im0": torch.stack([p[0] for p in pairs]),
            "im1": torch.stack([p[1] for p in pairs]), "xn": xn, "yn": yn}


def _window_inputs(case, seed):
    n = case["n"]
    im0, im1 = _pair(_generator(seed), 3 * n, 3 * n, "float32", peak=0.12 * n)
    return tuple(_host(im[n // 2:n // 2 + n, n:2 * n].contiguous()) for im in (im0, im1))


def prepare(case, seed):
    kind = case["kind"]
    state = {"kind": kind, "case": case}
    if kind == "window":
        state["correl"] = _work(case, lambda: CorrelGB300((case["n"],) * 2))
        state["im0"], state["im1"] = _window_inputs(case, seed)
    elif kind == "piv":
        state["work"] = _work(case, lambda: WorkPIV(_piv_params(case)))
        ims = _pair(_generator(seed), case["height"], case["width"], case["dtype"])
        state["im0"], state["im1"] = (_host(im) for im in ims) if case["host"] else ims
    elif kind == "batch":
        gen, jobs = _generator(seed), []
        for height, width, window, overlap in _batch_jobs(case):
            params = _piv_params(_piv(None, height, width, "uint16", window, 1, overlap, "last"))
            jobs.append((*_pair(gen, height, width, "uint16"), params))
        state["batch"] = PIVBatch(jobs)
    elif kind == "tps":
        state.update(_tps_inputs(case, seed))
    elif kind == "refine":
        state.update(_refine_inputs(case, seed))
        state["nodes"].requires_grad_(True)
    else:
        state["work"] = _work(case, lambda: WorkPreproc(_preproc_params(case)))
        state["images"] = _frames(_generator(seed), case)
    return state


# ------------------------------------------------------------------------ run
def _device_outputs(outs):
    res = []
    for p in outs:
        d = {k: getattr(p, k) for k in ("deltaxs_raw", "deltays_raw", "correls_max", "errors",
                                        "xs", "ys", "deltaxs", "deltays", "fix_flags")}
        for tag in ("tps_next", "tps_final"):
            t = getattr(p, tag)
            if t is not None:
                d[tag] = {"x": t.out_x, "y": t.out_y, "rx": t.rx, "ry": t.ry}
        res.append(d)
    return res


def _host_outputs(results):
    res = []
    for p in results.passes:
        d = {k: getattr(p, k) for k in ("deltaxs", "deltays", "correls_max", "xs", "ys")}
        for k in ("deltaxs_approx", "deltays_approx", "deltaxs_final", "deltays_final"):
            v = getattr(p, k, None)
            if v is not None:
                d[k] = v
        res.append(d)
    return res


def run(state):
    kind = state["kind"]
    if kind == "window":
        plugin = state["correl"]
        correl, norm = plugin(state["im0"], state["im1"])
        dx, dy, cmax, _ = plugin.compute_displacements_from_correl(correl, norm=norm)
        sx, sy = plugin.apply_subpix(dx, dy, correl)
        return {"correl": correl, "norm": norm, "dx": dx, "dy": dy, "cmax": cmax, "sx": sx,
                "sy": sy}
    if kind == "piv":
        if state["case"]["host"]:
            return _host_outputs(state["work"].calcul_from_arrays(state["im0"], state["im1"]))
        return _device_outputs(state["work"].calcul_device(state["im0"], state["im1"]))
    if kind == "batch":
        state["batch"].run()
        return [{"dx": j.out.deltaxs, "dy": j.out.deltays, "cmax": j.out.correls_max,
                 "errors": j.out.errors, "fix": j.out.fix_flags} for j in state["batch"].jobs]
    if kind == "tps":
        c = state["case"]
        t = run_tps(state["xs"], state["ys"], state["dx"], state["dy"], state["xs"].numel(),
                    state["px"], state["py"], state["px"].numel(), c["subdom"], c["smoothing"],
                    1.5, c["zoom"] == 1, None)
        out = {"x": t.out_x, "y": t.out_y, "rx": t.rx, "ry": t.ry}
        if c["zoom"] == 1:
            out.update(smooth_x=t.smooth_x, smooth_y=t.smooth_y)
        return out
    if kind == "refine":
        nodes = state["nodes"]
        r = DeformCorrelate.apply(nodes, state["im0"], state["im1"], state["xn"], state["yn"],
                                  0.1, True)
        loss = (r * r).sum(dim=-1).mean()
        (grad,) = torch.autograd.grad(loss, nodes)
        return {"r": r, "loss": loss, "grad": grad}
    return state["work"].calcul_device(state["images"])


# ----------------------------------------------------------------------- work
_SIZE = {"uint8": 1, "uint16": 2, "float32": 4}


def _grid(length, n, overlap):
    """Window centres along one axis."""
    step = n - round(overlap * n)
    top = length - (n // 2 + n % 2)
    at = list(range(n // 2, top, step))
    if top - at[-1] > step // 2.5:
        at.append(top)
    return at


def _correl_flops(n):
    return 3 * 2.5 * n * n * math.log2(n * n) + 5 * n * n


def _tps_flops(vectors, subdom):
    """One Cholesky factor, two refined solutions and the kernel matrix of subdomains
    widened by 20 % on each side."""
    m = 1.96 * subdom
    return vectors / subdom * (m ** 3 / 3 + 30 * m ** 2)


def _pass_work(height, width, n, overlap):
    vectors = len(_grid(height, n, overlap)) * len(_grid(width, n, overlap))
    return vectors, vectors * _correl_flops(n)


def work(case):
    kind = case["kind"]
    if kind == "window":
        n = case["n"]
        return {"bytes": 12 * n * n, "flops": _correl_flops(n)}
    if kind == "piv":
        size = case["height"] * case["width"] * _SIZE[case["dtype"]]
        nbytes, flops = 2 * size, 0.0
        for k in range(case["passes"]):
            vectors, f = _pass_work(case["height"], case["width"], case["window"] >> k,
                                    case["overlap"])
            nbytes, flops = nbytes + 62 * vectors, flops + f
            last = k == case["passes"] - 1
            if case["tps"] == "all" or (case["tps"] == "last" and last):
                flops += _tps_flops(vectors, case["subdom"])
        return {"bytes": nbytes, "flops": flops}
    if kind == "batch":
        nbytes, flops = 0, 0.0
        for height, width, n, overlap in _batch_jobs(case):
            vectors, f = _pass_work(height, width, n, overlap)
            nbytes, flops = nbytes + 4 * height * width + 14 * vectors, flops + f
        return {"bytes": nbytes, "flops": flops}
    if kind == "tps":
        n = case["ny"] * case["nx"]
        pts = n * case["zoom"] ** 2
        return {"bytes": 16 * n + 40 * pts,
                "flops": _tps_flops(n, case["subdom"]) + pts * 1.96 ** 2 * case["subdom"] * 6}
    pixels = case["height"] * case["width"]
    if kind == "refine":
        pixels *= case["pairs"]
        windows = case["pairs"] * (case["height"] // 32) * (case["width"] // 32)
        return {"bytes": 2 * pixels * _SIZE[case["dtype"]],
                "flops": windows * 2 * _correl_flops(32) + 2 * 3 * 20 * pixels}
    pixels *= case["frames"]
    wide = 4 if case["dtype"] == "float32" else 8
    taps = 2 * (25 + 9) if case["tool"] == "sharpen" else 4
    return {"bytes": pixels * (_SIZE[case["dtype"]] + wide), "flops": taps * pixels}


# ---------------------------------------------------------------------- exact
def _planes64(w0, w1):
    """Correlation planes (lags laid out as upstream's: displacement = n/2 - 1 - index),
    norms, of windows [count, n, n] float64."""
    n = w0.shape[-1]
    w0 = w0 - w0.mean(dim=(-1, -2), keepdim=True)
    w1 = w1 - w1.mean(dim=(-1, -2), keepdim=True)
    raw = torch.fft.ifft2(torch.conj(torch.fft.fft2(w0)) * torch.fft.fft2(w1)).real
    at = (n - 1 - torch.arange(n, device=raw.device) + n // 2) % n
    norms = torch.sqrt((w0 * w0).sum(dim=(-1, -2)) * (w1 * w1).sum(dim=(-1, -2)))
    return raw[:, at][:, :, at], norms


def _largest(planes):
    n = planes.shape[-1]
    f = planes.reshape(planes.shape[0], -1).argmax(dim=1)
    i0, i1 = f // n, f % n
    edge = (i0 == 0) | (i0 == n - 1) | (i1 == 0) | (i1 == n - 1)
    return i0, i1, edge


def _displacements64(planes, norms):
    """(dx, dy, correl_max): the largest value, searched again outside 3 px of it where it
    lies on the border, then the '2d_gaussian2' fit or the centroid."""
    count, n, _ = planes.shape
    i0, i1, edge = _largest(planes)
    sel = torch.nonzero(edge)[:, 0]
    if sel.numel():
        k = torch.arange(n, device=planes.device)
        near = (((k[None, :] - i0[sel][:, None]).abs() <= 3)[:, :, None]
                & ((k[None, :] - i1[sel][:, None]).abs() <= 3)[:, None, :])
        # (nothing is left out when 3 px below or left of it is outside the plane: upstream's
        # slice of a negative start is empty)
        near &= ((i0[sel] >= 3) & (i1[sel] >= 3))[:, None, None]
        j0, j1, still = _largest(planes[sel].masked_fill(near, float("-inf")))
        # a second peak that touches what was left out counts as none
        a = torch.arange(sel.numel(), device=planes.device)
        for y in (-1, 0, 1):
            for x in (-1, 0, 1):
                still = still | near[a, (j0 + y).clamp(0, n - 1), (j1 + x).clamp(0, n - 1)]
        i0[sel], i1[sel] = torch.where(still, i0[sel], j0), torch.where(still, i1[sel], j1)
        edge[sel] = still
    a = torch.arange(count, device=planes.device)
    cmax = planes[a, i0, i1] / norms
    o = torch.arange(-1, 2, device=planes.device)
    c0, c1 = i0.clamp(1, n - 2), i1.clamp(1, n - 2)
    crop = planes[a[:, None, None], (c0[:, None] + o)[:, :, None], (c1[:, None] + o)[:, None, :]]
    v = crop - crop.amin(dim=(1, 2), keepdim=True)
    v = v / v.amax(dim=(1, 2), keepdim=True)
    ln = torch.log(torch.where(v == 0, 1e-8, v))
    b = o.double()
    bx, by = b[None, None, :], b[None, :, None]

    def moment(weight, by_):
        return (weight * ln).sum(dim=(1, 2)) / by_

    c10, c01, c11 = moment(bx, 6.0), moment(by, 6.0), moment(bx * by, 4.0)
    c20, c02 = moment(3 * bx * bx - 2, 6.0), moment(3 * by * by - 2, 6.0)
    den = 4 * c20 * c02 - c11 * c11
    gx, gy = (c11 * c01 - 2 * c10 * c02) / den, (c11 * c10 - 2 * c01 * c20) / den
    s = crop.sum(dim=(1, 2))
    mx, my = (bx * crop).sum(dim=(1, 2)) / s, (by * crop).sum(dim=(1, 2)) / s
    far = gx * gx + gy * gy > 4.5
    gx, gy = torch.where(far, mx, gx), torch.where(far, my, gy)
    bad = edge | (gx * gx + gy * gy > 4.5)
    gx, gy = torch.where(bad, 0.0, gx), torch.where(bad, 0.0, gy)
    return n / 2 - 1 - (i1 + gx), n / 2 - 1 - (i0 + gy), cmax


def _values64(im):
    """Pixel values as float64 (uint16 images come in int16 storage)."""
    if im.dtype == torch.int16:
        return (im.to(torch.int32) & 0xFFFF).double()
    return im.double()


def _pass64(im0, im1, n, overlap):
    """The single pass of a pair: displacements, correlation maxima, positions."""
    gy, gx = (torch.tensor(_grid(length, n, overlap), device="cuda") for length in im0.shape)
    xs, ys = gx.repeat(gy.numel()), gy.repeat_interleave(gx.numel())
    im0, im1 = _values64(im0), _values64(im1)
    parts, o = [], torch.arange(n, device="cuda") - n // 2
    for k in range(0, xs.numel(), 8192):
        r = (ys[k:k + 8192, None] + o)[:, :, None]
        c = (xs[k:k + 8192, None] + o)[:, None, :]
        parts.append(_displacements64(*_planes64(im0[r, c], im1[r, c])))
    dx, dy, cmax = (torch.cat(p) for p in zip(*parts))
    return {"dx": dx, "dy": dy, "cmax": cmax, "xs": xs.double(), "ys": ys.double()}


def _exact_window(case, seed):
    w0, w1 = (torch.from_numpy(w).double()[None] for w in _window_inputs(case, seed))
    planes, norms = _planes64(w0, w1)
    dx, dy, cmax = _displacements64(planes, norms)
    return {"correl": planes[0].numpy(), "norm": float(norms[0]), "dx": None, "dy": None,
            "cmax": cmax[0].numpy(), "sx": float(dx[0]), "sy": float(dy[0])}


def _exact_piv(case, seed):
    # later passes look at windows moved by whole pixels, which rest on thresholds and
    # roundings of the passes before: they have no value of their own in 64 bits
    if case["passes"] != 1:
        return None
    ims = _pair(_generator(seed), case["height"], case["width"], case["dtype"])
    p = _pass64(*ims, case["window"], case["overlap"])
    if case["host"]:
        return [{"correls_max": p["cmax"], "xs": None, "ys": None}]
    return [{"deltaxs_raw": p["dx"], "deltays_raw": p["dy"], "correls_max": p["cmax"],
             "xs": p["xs"], "ys": p["ys"]}]


def _exact_batch(case, seed):
    gen, out = _generator(seed), []
    for height, width, window, overlap in _batch_jobs(case):
        p = _pass64(*_pair(gen, height, width, "uint16"), window, overlap)
        out.append({"cmax": p["cmax"]})
    return out


def _phi64(ya, xa, yb, xb):
    r2 = (ya[:, None] - yb[None, :]) ** 2 + (xa[:, None] - xb[None, :]) ** 2
    return torch.where(r2 == 0, 0.0, 0.5 * r2 * torch.log(r2.clamp_min(1e-30)))


def _exact_tps(case, seed):
    """The smoothed splines of the subdomains (LU of the full saddle-point systems), their
    outliers replaced and solved again, blended."""
    s = _tps_inputs(case, seed)
    keep = ~(torch.isnan(s["dx"]) | torch.isnan(s["dy"]))
    xs, ys = s["xs"][keep].double(), s["ys"][keep].double()
    values = torch.stack([s["dx"][keep], s["dy"][keep]], 1).double()
    px, py = s["px"], s["py"]
    x0, x1, y0, y1 = (float(v) for v in (xs.min(), xs.max(), ys.min(), ys.max()))
    n, ratio = xs.numel(), (y1 - y0) / (x1 - x0)
    nb = n / case["subdom"]
    nbx = int(math.floor(math.sqrt(nb / ratio))) or 1
    nby = int(math.ceil(math.sqrt(nb * ratio))) or 1
    xd, yd = np.linspace(x0, x1, nbx + 1), np.linspace(y0, y1, nby + 1)
    lam = case["smoothing"] * math.sqrt((xd[1] - xd[0]) * (yd[1] - yd[0]) / (n / (nbx * nby)))
    bx, by = 0.2 * (x1 - x0) / nbx, 0.2 * (y1 - y0) / nby
    out, wsum = torch.zeros_like(px)[:, None].repeat(1, 2), torch.zeros_like(px)
    smooth, csum = torch.zeros_like(values), torch.zeros_like(xs)
    for iy in range(nby):
        for ix in range(nbx):
            xa, xb, ya, yb = xd[ix] - bx, xd[ix + 1] + bx, yd[iy] - by, yd[iy + 1] + by
            xc, yc = 0.5 * (xa + xb), 0.5 * (ya + yb)

            def inside(x, y):
                sel = torch.nonzero((x >= xa) & (x < xb) & (y >= ya) & (y < yb))[:, 0]
                x, y = x[sel], y[sel]
                w = ((1 - (x - xc) ** 2 / (xb - xc) ** 2) * (1 - (y - yc) ** 2 / (yb - yc) ** 2)
                     + 0.001)
                return sel, x, y, w

            sel, x, y, w = inside(xs, ys)
            m = sel.numel()
            em = torch.cat([_phi64(y, x, y, x), torch.ones_like(x)[:, None], y[:, None],
                            x[:, None]], 1)
            a = torch.zeros((m + 3, m + 3), dtype=torch.float64, device=x.device)
            a[:m] = em
            a[m:, :m] = em[:, m:].T
            a[:m, :m] += lam * torch.eye(m, dtype=torch.float64, device=x.device)
            lu, piv = torch.linalg.lu_factor(a)
            rhs = torch.zeros((m + 3, 2), dtype=torch.float64, device=x.device)
            rhs[:m] = values[sel]
            todo = [True, True]
            sol = torch.linalg.lu_solve(lu, piv, rhs)
            sm = em @ sol
            for _ in range(10):
                bad = (sm - rhs[:m]).abs() > 1.5
                todo = [t and bool(b) for t, b in zip(todo, bad.any(dim=0))]
                if not any(todo):
                    break
                go = torch.tensor(todo, device=x.device)
                rhs[:m] = torch.where(bad & go, sm, rhs[:m])
                new = torch.linalg.lu_solve(lu, piv, rhs)
                sol = torch.where(go, new, sol)
                sm = em @ sol
            smooth[sel] += w[:, None] * sm
            csum[sel] += w
            sel, x2, y2, w = inside(px, py)
            ev = torch.cat([_phi64(y2, x2, y, x), torch.ones_like(x2)[:, None], y2[:, None],
                            x2[:, None]], 1)
            out[sel] += w[:, None] * (ev @ sol)
            wsum[sel] += w
    out, smooth = out / wsum[:, None], smooth / csum[:, None]
    res = {"x": out[:, 0], "y": out[:, 1]}
    if case["zoom"] == 1:
        res.update(smooth_x=smooth[:, 0], smooth_y=smooth[:, 1])
    return res


def _warp64(nodes, xn, yn, im, scale):
    def cell(at, v):
        j = (torch.searchsorted(at, v, right=True) - 1).clamp(0, at.numel() - 2)
        return j, ((v - at[j]) / (at[j + 1] - at[j])).clamp(0.0, 1.0)

    pairs, height, width = im.shape
    xs = torch.arange(width, dtype=torch.float64, device=im.device)
    ys = torch.arange(height, dtype=torch.float64, device=im.device)
    (j, tx), (i, ty) = cell(xn.double(), xs), cell(yn.double(), ys)
    ty = ty[:, None]
    rows = (1 - ty) * nodes[:, :, i] + ty * nodes[:, :, i + 1]
    d = (1 - tx) * rows[:, :, :, j] + tx * rows[:, :, :, j + 1]
    x, y = xs + scale * d[:, 0], ys[:, None] + scale * d[:, 1]
    xf, yf = torch.floor(x).detach(), torch.floor(y).detach()
    fx, fy = x - xf, y - yf
    xa, xb = xf.long().clamp(0, width - 1), (xf.long() + 1).clamp(0, width - 1)
    ya, yb = yf.long().clamp(0, height - 1), (yf.long() + 1).clamp(0, height - 1)
    b = torch.arange(pairs, device=im.device)[:, None, None]
    top = (1 - fx) * im[b, ya, xa] + fx * im[b, ya, xb]
    bot = (1 - fx) * im[b, yb, xa] + fx * im[b, yb, xb]
    return (1 - fy) * top + fy * bot


def _exact_refine(case, seed):
    s = _refine_inputs(case, seed)
    nodes = s["nodes"].double().requires_grad_(True)
    w = []
    for im, scale in ((s["im0"], -0.5), (s["im1"], 0.5)):
        im = _warp64(nodes, s["xn"], s["yn"], _values64(im), scale)
        b, h, v = im.shape[0], im.shape[1] // 32, im.shape[2] // 32
        t = im[:, :32 * h, :32 * v].reshape(b, h, 32, v, 32).permute(0, 1, 3, 2, 4)
        t = t - t.mean(dim=(-1, -2), keepdim=True)
        w.append(t / torch.sqrt((t * t).sum(dim=(-1, -2), keepdim=True)))
    c = torch.fft.ifft2(torch.conj(torch.fft.fft2(w[0])) * torch.fft.fft2(w[1])).real
    m = torch.arange(32, device=c.device)
    lag = torch.where(m < 16, m, m - 32).double()
    off = (m[:, None] == 16) | (m[None, :] == 16)
    p = torch.softmax(c.masked_fill(off, float("-inf")).flatten(-2) / 0.1, -1).view_as(c)
    r = torch.stack([(p * lag).sum(dim=(-1, -2)), (p * lag[:, None]).sum(dim=(-1, -2))], -1)
    loss = (r * r).sum(dim=-1).mean()
    (grad,) = torch.autograd.grad(loss, nodes)
    return {"r": r, "loss": loss, "grad": grad}


def _reflect(i, n):
    """Indices beyond the ends mirrored with the edge repeated."""
    i = i % (2 * n)
    return torch.where(i < n, i, 2 * n - 1 - i)


def _ranked(x, window, rank):
    """The rank-th smallest value of every box (nt, ny, nx) of a stack of whole numbers,
    bit by bit from the top."""
    pads = []
    for axis, size in enumerate(window):
        n = x.shape[axis]
        at = _reflect(torch.arange(-(size // 2), n + size - 1 - size // 2, device=x.device), n)
        pads.append(at)
    p = x[pads[0]][:, pads[1]][:, :, pads[2]]
    nt, ny, nx = x.shape
    best = torch.zeros_like(x)
    for bit in range(int(x.max()).bit_length() - 1, -1, -1):
        cand = best | (1 << bit)
        below = torch.zeros_like(x)
        for a in range(window[0]):
            for b in range(window[1]):
                for c in range(window[2]):
                    below += p[a:a + nt, b:b + ny, c:c + nx] < cand
        best = torch.where(below <= rank, cand, best)
    return best


def _exact_tool(case, seed):
    images = _frames(_generator(seed), case)
    x = _values64(images)
    if case["tool"] == "sharpen":
        return _exact_sharpen(x, case["dtype"])
    stack = x if x.dim() == 3 else x[None]
    n = case.get("window", 1)
    window = (1, n, n) if case["tool"].startswith("sliding") else (stack.shape[0], 1, 1)
    size = window[0] * window[1] * window[2]
    rank = {"minima": 0, "median": size // 2, "percentile": int(size * 10.0 / 100.0)}[
        case["tool"].split("_")[1]]
    # the images' values are whole numbers in every type
    out = stack - _ranked(stack.to(torch.int32), window, rank).double()
    if case["tool"].startswith("sliding"):
        out = out.clamp_min(0.0)
    return out if x.dim() == 3 else out[0]


def _exact_sharpen(x, dtype):
    def cast(v):
        return v.to(torch.float32).double() if dtype == "float32" else torch.trunc(v)

    def blur(v, sigma):
        radius = int(4.0 * sigma + 0.5)
        at = np.arange(-radius, radius + 1)
        phi = np.exp(-0.5 / (sigma * sigma) * at ** 2)
        phi = (phi / phi.sum())[::-1]
        for axis in (0, 1):
            n = v.shape[axis]
            k = torch.arange(n, device=v.device)
            acc = v * float(phi[radius])
            for j in range(radius, 0, -1):
                both = (v.index_select(axis, _reflect(k - j, n))
                        + v.index_select(axis, _reflect(k + j, n)))
                acc = acc + both * float(phi[radius - j])
            v = cast(acc)
        return v

    first = blur(x, 3.0)
    diff = first - blur(first, 1.0)
    if dtype != "float32":
        diff = torch.remainder(diff, 256.0 if dtype == "uint8" else 65536.0)
    return first + 30.0 * diff


def exact(case, seed):
    return {"window": _exact_window, "piv": _exact_piv, "batch": _exact_batch,
            "tps": _exact_tps, "refine": _exact_refine, "tool": _exact_tool}[case["kind"]](
                case, seed)
