"""Grain drawn in row bands ahead of the print's bands (frames from 4 to 64 megapixels in spk_render) against the
same frames drawn whole (spkx_render_batch): equal bit for bit, and so is a reprint, which reads the whole negative."""

import numpy as np
import pytest

from conftest import BASE, sc

pytestmark = pytest.mark.gpu


# just above one band; a last band of one row, and of a partial tile; just below the range's pixels; odd widths
@pytest.mark.parametrize("w,h", [(16400, 257), (8200, 513), (2101, 2003), (2047, 2048)])
@pytest.mark.parametrize("extra", [{}, {"dir_couplers_active": True, "scanner_lens_blur": 1.5}])
def test_bands_match_whole(engine, w, h, extra):
    delta = dict(BASE, grain_active=True, film_format_mm=0.009 * max(w, h), **extra)  # a pitch of 9 um
    img = sc.synthetic_image(w, h, 5)
    with engine.open(img, delta) as s:
        results, _ = engine.render_batch([s], "full")
        want = results[0].pixels.copy()
        results[0].free()
    with engine.open(img, delta) as s:
        np.testing.assert_array_equal(s.render("full")[0], want)
        np.testing.assert_array_equal(s.reprint("full")[0], want)
