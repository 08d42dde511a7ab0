"""The minima of image pairs, one pair at a time and batched, with one smallest pixel at a
time where the loads change: first and last pixel, edges of the 16-byte vectors, of a
thread's four vectors in flight, of the vectors and the scalar tail; values of the upper
half of uint16."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

#: dtype: torch storage, smallest and background values
TYPES = {"uint8": ("uint8", 7, 200), "uint16": ("int16", 33000, 60000),
         "float32": ("float32", -3.5, 2.25)}


def _places(count, per, strides):
    vec = count // per * per
    at = {0, 1, per - 1, per, count // 2, vec - 1, vec, count - 1}
    for stride in strides:
        at |= {k * stride * per + d for k in (1, 3, 4) for d in (-1, 0)}
    return sorted(k for k in at if 0 <= k < count)


@pytest.mark.parametrize("dtype", list(TYPES))
@pytest.mark.parametrize("kind", ["small", "one vector", "four vectors"])
def test_smallest_pixel_everywhere(dtype, kind):
    import torch

    from fluidimage_gb300 import _lib as L

    lib = L.load()
    storage, low, high = TYPES[dtype]
    code = {"uint8": L.FI_U8, "uint16": L.FI_U16, "float32": L.FI_F32}[dtype]
    per = {"uint8": 16, "uint16": 8, "float32": 4}[dtype]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    stride = 8 * sms * 256  # threads of the largest launch of one pair
    vectors = {"small": 3, "one vector": stride // 2, "four vectors": 4 * stride + 700}[kind]
    height, width = 1, vectors * per + per - 1
    count = height * width
    ims = [torch.full((count + 16,), high if dtype != "uint16" else high - 65536,
                      dtype=getattr(torch, storage), device="cuda") for _ in range(2)]
    small = low if dtype != "uint16" else low - 65536
    out = torch.empty(2, dtype=torch.float32, device="cuda")
    # a batch of this pair between two others (its launch has fewer threads a pair)
    mins = torch.empty(6, dtype=torch.float32, device="cuda")
    other = torch.full((64,), 1, dtype=getattr(torch, storage), device="cuda")
    keys = torch.empty(6, dtype=torch.int32, device="cuda")
    for place in _places(count, per, (stride, stride // 3)):
        for which in (0, 1):
            a, b = ims[0][:count], ims[1][:count]
            (a, b)[which][place] = small
            want = [float(low if which == k else high) for k in (0, 1)]
            L.check(lib.fi_images_min(L.ptr(a), L.ptr(b), code, count, L.ptr(out),
                                      L.stream_handle()), "fi_images_min")
            assert out.tolist() == want, place
            args = (L.PivPassArgs * 3)()
            for k, (p, q, w) in enumerate(((other, other, 64), (a, b, width), (other, other, 64))):
                args[k].im0, args[k].im1, args[k].dtype = L.ptr(p), L.ptr(q), code
                args[k].height, args[k].width = 1, w
                args[k].im_min = L.ptr(mins[2 * k:])
            dev = torch.from_numpy(np.frombuffer(C.string_at(args, C.sizeof(args)),
                                                 np.uint8).copy()).cuda()
            L.check(lib.fi_images_min_batch(L.ptr(dev), 3, L.ptr(keys), L.stream_handle()),
                    "fi_images_min_batch")
            assert mins.tolist() == [1.0, 1.0, *want, 1.0, 1.0], place
            (a, b)[which][place] = high if dtype != "uint16" else high - 65536
