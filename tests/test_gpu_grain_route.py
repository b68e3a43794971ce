"""Which renders leave their grain to the print's bands, by the kernels they launch: the film side of a render (its
launches less a reprint's) against the same develop drawn whole. A frame whose print is not in bands (a spectral
print mode, a recursive scanner lens blur, a short frame) is drawn whole; either way the pixels are those of a batch."""

import ctypes

import numpy as np
import pytest

from conftest import BASE, sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,mode,extra,bands", [(2101, 2003, "fp32", {}, 8), (2101, 2003, "fp32_generic", {}, 0),
                                                  (2101, 2003, "fp32", {"scanner_lens_blur": 4.0}, 0),
                                                  (17000, 256, "fp32", {}, 0), (17000, 257, "fp32", {}, 0),
                                                  (8200, 513, "fp32", {}, 3)])
def test_deferred_where_the_print_is_banded(lib, engine, w, h, mode, extra, bands):
    def launched(call):
        n = [ctypes.c_uint64(), ctypes.c_uint64()]
        lib.check(lib.lib.spkx_test_launch_count(ctypes.byref(n[0])))
        out = call()
        lib.check(lib.lib.spkx_test_launch_count(ctypes.byref(n[1])))
        return out, n[1].value - n[0].value

    delta = dict(BASE, film_format_mm=0.009 * max(w, h), **extra)  # a pitch of 9 um
    with engine.open(sc.synthetic_image(w, h, 5), delta) as s:
        s.set_print_mode(mode)
        (out, _), render = launched(lambda: s.render("full"))
        out = out.copy()
        (again, _), reprint = launched(lambda: s.reprint("full"))
        np.testing.assert_array_equal(again, out)
        _, whole = launched(lambda: s.develop_debug("full", 1, w, h, counts=False))
        results, _ = engine.render_batch([s], "full", reprint=True)
        np.testing.assert_array_equal(results[0].pixels, out)
        results[0].free()
    # whole: one draw and one blur; in bands: both for the first 288 rows (all of a frame of 257), and both again
    # for each band that reaches further
    assert (render - reprint - whole > 0) == (bands > 0)
    assert render - reprint - whole <= 2 * bands
