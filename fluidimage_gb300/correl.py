"""Correlation plugin with the upstream per-window contract, computed on the GPU.

``CorrelGB300`` follows ``CorrelFFTNumpy`` (calcul/correl.py:665-685) and the
methods it inherits from ``CorrelFFTBase`` / ``CorrelBase``
(calcul/correl.py:167-281, 513-568):

* ``__call__(im0, im1) -> (correl, norm)``: float32 plane in the
  ``_like_fftshift`` layout (so that ``dx = ix0 - ix``) and a Python float with
  ``correl / norm`` in [-1, 1];
* ``compute_displacements_from_correl(correl, norm) -> (dx, dy, correl_max,
  other_peaks)``, raising ``PIVError`` (``explanation``, ``results``) like
  upstream, including the second-chance search that writes NaNs into the
  caller's plane when ``displacement_max`` is None, and the other peaks when
  ``nb_peaks_to_search > 1``;
* ``apply_subpix(dx, dy, correl)`` (any ``SubPix`` method: '2d_gaussian2' with its
  centroid fallback, '2d_gaussian', 'centroid', 'no_subpix');
* ``get_indices_no_displacement()``, ``displacement_max``.

Every computation runs in the CUDA library; the plugin only moves arrays.  It
registers as ``correlation_classes["gb300"]``, and :func:`register_upstream`
adds it to an installed fluidimage's registry so that
``params.piv0.method_correl = "gb300"`` selects it there.  For whole passes, use
``fluidimage_gb300.WorkPIV`` (one launch per pass instead of one per window).
"""

from __future__ import annotations

import math
import threading

import numpy as np

from . import _lib as L
from .engine import SUPPORTED_WINDOWS, displacement_mask, parse_displacement_max
from .errors import ERROR_STRINGS, PIVError


def _dev():
    import torch

    return torch.device("cuda")


#: bytes up to which a call's arrays stay in pinned host memory, which the kernels read
#: and write in place
STAGE_MAX = 1 << 20

_STAGE = threading.local()


class _Arrays:
    """The arrays of one call: ``specs`` is a list of (shape, numpy dtype), ``ptr[i]``
    what the library takes and, after ``finish()``, ``get(i)`` an array of the caller's
    own.

    A small call is bound by the host: each of its five to ten copies to or from the
    device costs 10 to 20 us, for a few kilobytes.  Its arrays lie side by side in a
    pinned buffer (one per thread, at most ``STAGE_MAX``), which the GPU reads and writes
    over its link to the host, so that a call is a launch and one synchronisation: a
    32 px window through correlation, peak and subpixel fit 585 -> 111 us.  Larger calls
    go through device memory, the inputs array by array and the outputs in one copy, so
    that the buffer stays bounded (planes and peaks of 256 windows of 32 px 424 us, of
    1024 of 48 px 1302; with a copy for each array 540 and 1449).
    """

    def __init__(self, specs):
        import torch

        self.spans, total = [], 0
        for shape, dtype in specs:
            nbytes = math.prod(shape) * dtype.itemsize
            self.spans.append((total, nbytes, dtype, shape))
            total += -(-nbytes // 16) * 16
        total = max(total, 16)
        self.stream = torch.cuda.current_stream()
        self.host = self.device = None
        self.first = 0  # where the host's bytes begin
        if total <= STAGE_MAX:
            stage = getattr(_STAGE, "stage", None)
            if stage is None or stage[0].numel() < total:
                buf = torch.empty(max(total, 1 << 16), dtype=torch.uint8, pin_memory=True)
                stage = _STAGE.stage = buf, buf.numpy(), buf.data_ptr()
            _, self.host, base = stage
        else:
            self.device = torch.empty(total, dtype=torch.uint8, device=_dev())
            base = self.device.data_ptr()
        self.ptr = [base + span[0] for span in self.spans]

    def view(self, i):
        at, nbytes, dtype, shape = self.spans[i]
        if at < self.first:  # an input in device memory, as the kernels left it
            raw = self.device[at:at + nbytes].cpu().numpy()
        else:
            raw = self.host[at - self.first:at - self.first + nbytes]
        return raw.view(dtype).reshape(shape)

    def start(self, *inputs):
        """Fills the first arrays; what the library needs before the launch."""
        for i, array in enumerate(inputs):
            if self.device is None:
                self.view(i)[...] = array
            else:
                import torch

                at, nbytes, dtype, _ = self.spans[i]
                raw = np.ascontiguousarray(array, dtype=dtype).reshape(-1).view(np.uint8)
                self.device[at:at + nbytes].copy_(torch.from_numpy(raw))
                self.first = self.spans[i + 1][0]
        return self.stream.cuda_stream

    def finish(self):
        if self.device is None:
            self.stream.synchronize()
        else:  # the outputs in one copy, the caller's own
            self.host = self.device[self.first:].cpu().numpy()

    def get(self, i):
        return self.view(i).copy() if self.device is None else self.view(i)


_F64, _F32, _I32, _U8 = (np.dtype(t) for t in ("f8", "f4", "i4", "u1"))


class CorrelGB300:
    """FFT cross-correlation of one window pair (or a batch) on the GPU."""

    _tag = "gb300"
    #: class of the errors the per-window methods raise; ``register_upstream`` makes
    #: it a subclass of the installed fluidimage's PIVError as well, so that
    #: upstream's ``except PIVError`` (works/piv/singlepass.py:328, 339;
    #: works/piv/fix.py:202) catches it
    _piv_error = PIVError

    def __init__(self, im0_shape, im1_shape=None, method_subpix="2d_gaussian2", nsubpix=None,
                 displacement_max=None, particle_radius=3, nb_peaks_to_search=1, mode=None):
        self.mode = mode
        if im1_shape is None:
            im1_shape = im0_shape
        im0_shape = tuple(int(n) for n in im0_shape)
        im1_shape = tuple(int(n) for n in im1_shape)
        if im0_shape != im1_shape:
            raise ValueError(
                "with this correlation method the input images have to have the same shape."
            )
        if im0_shape[0] != im0_shape[1] or im0_shape[0] not in SUPPORTED_WINDOWS:
            raise NotImplementedError(f"window {im0_shape} not supported: square {SUPPORTED_WINDOWS}")
        if method_subpix == "2d_gaussian2" and nsubpix is not None and nsubpix != 1:
            raise ValueError(
                "Subpixel method '2d_gaussian2' doesn't require nsubpix. "
                "In this case, nsubpix has to be equal to None."
            )
        if method_subpix not in L.SUBPIX_METHODS:
            raise ValueError(f"method has to be in {list(L.SUBPIX_METHODS)}")
        self.nsubpix = 1 if nsubpix is None else int(nsubpix)
        if not 1 <= self.nsubpix <= L.MAX_NSUBPIX:
            raise NotImplementedError(f"nsubpix must be in 1..{L.MAX_NSUBPIX} on this backend")
        if not 1 <= int(nb_peaks_to_search) <= L.MAX_PEAKS:
            raise NotImplementedError(f"nb_peaks_to_search must be in 1..{L.MAX_PEAKS}")
        self.method_subpix = method_subpix
        self._method = L.SUBPIX_METHODS[method_subpix]
        self._minv = None
        self.im0_shape = im0_shape
        self.im1_shape = im1_shape
        self.n = im0_shape[0]
        self.iy0, self.ix0 = (i // 2 - 1 for i in im0_shape)
        self.displacement_max = parse_displacement_max(displacement_max, im0_shape)
        self.particle_radius = particle_radius
        self.nb_peaks_to_search = nb_peaks_to_search
        mask, box = displacement_mask(self.n, self.displacement_max)
        self.where_large_displacement = mask
        self.start_stop_for_search0 = (box[0], box[1])
        self.start_stop_for_search1 = (box[2], box[3])
        self._box = box
        self._mask_dev = None

    # ---------------------------------------------------------------- geometry
    def compute_displacement_from_indices(self, ix, iy):
        return self.ix0 - ix, self.iy0 - iy

    def compute_indices_from_displacement(self, dx, dy):
        return self.ix0 - dx, self.iy0 - dy

    def get_indices_no_displacement(self):
        return self.iy0, self.ix0

    # ---------------------------------------------------------------- planes
    def correl_batch(self, ims0, ims1):
        """Planes and norms of a stack of window pairs ``(count, n, n)``."""
        w0 = np.ascontiguousarray(ims0, dtype=np.float32)
        w1 = np.ascontiguousarray(ims1, dtype=np.float32)
        if w0.ndim == 2:
            w0, w1 = w0[None], w1[None]
        count = w0.shape[0]
        if tuple(w0.shape[1:]) != self.im0_shape or w0.shape != w1.shape:
            raise ValueError("Bad im_crop shape.")
        a = _Arrays([(w0.shape, _F32), (w0.shape, _F32), (w0.shape, _F32), ((count,), _F64)])
        s = a.start(w0, w1)
        L.check(L.load().fi_correl_windows(a.ptr[0], a.ptr[1], count, self.n, a.ptr[2], a.ptr[3],
                                           s), "fi_correl_windows")
        a.finish()
        return a.get(2), a.get(3)

    def __call__(self, im0, im1):
        """Correlation plane and norm of one window pair (correl.py:671-685)."""
        planes, norms = self.correl_batch(im0, im1)
        return planes[0], float(norms[0])

    # ---------------------------------------------------------------- peaks
    def _mask_device(self):
        import torch

        if self.where_large_displacement is not None and self._mask_dev is None:
            self._mask_dev = torch.as_tensor(self.where_large_displacement.astype(np.uint8),
                                             device=_dev())
        return self._mask_dev

    def _minv_device(self):
        import torch

        from .engine import subpix_pinv

        if self.method_subpix == "2d_gaussian" and self._minv is None:
            self._minv = torch.as_tensor(subpix_pinv(self.nsubpix), device=_dev())
        return self._minv

    def peaks_batch(self, planes, norms, apply_subpix=False):
        """Peak search (+ subpixel) of a stack of planes; returns per-plane arrays
        ``(dx, dy, correl_max, err, i0, i1, other_peaks)``; ``planes`` receives the
        second-chance NaN boxes like upstream (no displacement_max only).
        ``other_peaks`` is None (nb_peaks_to_search == 1) or per plane None (search
        raised) or a list of ``(dx, dy, correl_max)``."""
        p = np.ascontiguousarray(planes, dtype=np.float32)
        if p.ndim == 2:
            p = p[None]
        count = p.shape[0]
        nrm = np.asarray(norms, dtype=np.float64).reshape(-1)
        b = self._box
        nb = int(self.nb_peaks_to_search)
        K = nb - 1
        if p.size < count * self.n * self.n or nrm.size < count:
            raise ValueError("planes and norms do not match the windows")
        n1 = (count,)
        specs = [(nrm.shape, _F64), (p.shape, _F32), (n1, _F32), (n1, _F32), (n1, _F32),
                 (n1, _U8), (n1, _I32), (n1, _I32)]
        if K > 0:
            specs += [(n1, _I32), ((count, K, L.PEAK_FIELDS), _F32), ((count, K), _U8)]
        mask, minv = self._mask_device(), self._minv_device()
        a = _Arrays(specs)
        s = a.start(nrm, p)
        L.check(L.load().fi_peaks_from_planes(
            a.ptr[1], a.ptr[0], count, self.n, L.ptr(mask), b[0], b[1], b[2], b[3],
            int(self.particle_radius), int(apply_subpix), self._method, self.nsubpix,
            L.ptr(minv), nb, *a.ptr[2:8], *(a.ptr[8:] if K > 0 else (None,) * 3), s),
            "fi_peaks_from_planes")
        a.finish()
        if isinstance(planes, np.ndarray) and self.where_large_displacement is None:
            planes[...] = a.view(1).reshape(planes.shape)
        other = None
        if K > 0:
            counts, peaks = a.view(8), a.get(9)
            other = [None if counts[k] < 0 else
                     [(int(peaks[k, j, 0]), int(peaks[k, j, 1]), peaks[k, j, 2])
                      for j in range(int(counts[k]))] for k in range(count)]
        return (*(a.get(i) for i in range(2, 8)), other)

    def compute_displacements_from_correl(self, correl, norm=1.0):
        """(dx, dy, correl_max, other_peaks) of one plane (correl.py:226-275, 561-568)."""
        dx, dy, cm, err, i0, i1, other = self.peaks_batch(correl, [norm])
        cmax = 0.0 if norm == 0 else cm[0]
        e = int(err[0])
        if e == 5:
            raise AssertionError("correlation plane without finite value")
        if e:
            error = self._piv_error(explanation=ERROR_STRINGS[e])
            error.results = (int(dx[0]), int(dy[0]), cmax)
            raise error
        return int(dx[0]), int(dy[0]), cmax, (None if other is None else other[0])

    def apply_subpix(self, dx, dy, correl):
        """Subpixel displacement with the plugin's method (correl.py:277-281,
        subpix.py:107-218)."""
        ix, iy = self.compute_indices_from_displacement(dx, dy)
        p = np.ascontiguousarray(correl, dtype=np.float32)
        if p.size < self.n * self.n:
            raise ValueError("the plane does not match the window")
        minv = self._minv_device()
        a = _Arrays([(p.shape, _F32), ((2,), _I32), ((2,), _F32), ((1,), _U8)])
        s = a.start(p, (int(iy), int(ix)))
        L.check(L.load().fi_subpix_at(a.ptr[0], 1, self.n, a.ptr[1], a.ptr[1] + 4, self._method,
                                      self.nsubpix, L.ptr(minv), a.ptr[2], a.ptr[2] + 4,
                                      a.ptr[3], s), "fi_subpix_at")
        a.finish()
        e = int(a.view(3)[0])
        if e:
            raise self._piv_error(explanation=ERROR_STRINGS[e], result_compute_subpix=(iy, ix))
        out = a.view(2)
        return float(out[0]), float(out[1])


correlation_classes = {CorrelGB300._tag: CorrelGB300}


def register_upstream():
    """Add ``CorrelGB300`` to an installed fluidimage's ``correlation_classes``.

    Upstream's ``singlepass`` module imports the same dict object
    (works/piv/singlepass.py:24), so ``params.piv0.method_correl = "gb300"``
    then selects this plugin.  Returns False when fluidimage is not importable.
    """
    try:
        from fluidimage.calcul import correl as upstream
        from fluidimage.calcul.errors import PIVError as UpstreamPIVError
    except Exception:
        return False

    class _PIVError(PIVError, UpstreamPIVError):
        """A PIVError of both packages (upstream's handlers catch their own class)."""

        def __init__(self, *args, **kwargs):
            Exception.__init__(self, *args)
            self.explanation = "General no peak error"
            self.__dict__.update(kwargs)

    CorrelGB300._piv_error = _PIVError
    upstream.correlation_classes[CorrelGB300._tag] = CorrelGB300
    return True
