"""Device memory that the engine reads where it lies (aligned device memory of its own) against the copied route: the
same floats at an offset that is not 16-byte aligned. The results are equal bit for bit."""

import json

import numpy as np
import pytest

from conftest import BASE, sc

pytestmark = pytest.mark.gpu


def shifted(torch, flat, offset):
    """flat on the device, its first element `offset` floats into an allocation with no slack behind it."""
    d = torch.empty(flat.size + offset, dtype=torch.float32, device="cuda")
    d[offset:] = torch.from_numpy(flat)
    torch.cuda.synchronize()
    return d


@pytest.mark.parametrize("w,h", [(1, 1), (33, 21), (257, 64)])
def test_open_device(engine, w, h):
    torch = pytest.importorskip("torch")
    img = sc.synthetic_image(w, h, 3)
    outs = []
    for offset in (0, 1, 4):
        d = shifted(torch, img.ravel(), offset)
        image = sc.SpkDeviceImage(d.data_ptr() + 4 * offset, w, h, 3)
        handle = engine.L.lib.spk_open_device(engine.h, image, json.dumps(dict(BASE)).encode(), None)
        assert handle, engine.L.last_error()
        with sc.Session(engine, handle, None, (h, w)) as s:
            del d
            outs.append(s.develop_debug("full", 1, w, h, counts=False)[0])
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])


@pytest.mark.parametrize("mode,bins", [("fp32", 81), ("bf16x3", 81)])
@pytest.mark.parametrize("w,h", [(33, 21), (257, 64)])
def test_print_negative(engine, w, h, mode, bins):
    torch = pytest.importorskip("torch")
    neg = np.random.default_rng(w).random((h, w, 3), dtype=np.float32) * 2.0
    outs = []
    with engine.open(sc.synthetic_image(w, h, 3), dict(BASE)) as s:
        s.set_print_mode(mode, bins)
        for offset in (0, 1, 4):
            d = shifted(torch, neg.ravel(), offset)
            stride = (w + 31) // 32 * 32
            out = torch.zeros((h, stride, 4), dtype=torch.int16, device="cuda")
            torch.cuda.synchronize()
            s.print_negative(d.data_ptr() + 4 * offset, w, h, out.data_ptr(), stride)
            outs.append(out.cpu().numpy()[:, :w])
    np.testing.assert_array_equal(outs[1], outs[0])
    np.testing.assert_array_equal(outs[2], outs[0])
