"""Renders when device memory is short: where a faster path takes more scratch than the one it replaced, the call
falls back to that one and gives the same bits. The session's limit stands in for a device without more memory."""

import numpy as np
import pytest

import oracle
from conftest import BASE, sc

pytestmark = pytest.mark.gpu

MIXED = [((0.1, 0.2, 0.3), (3.0 + 0.5 * k, 0.4 * k + 0.3, 4.0)) for k in range(6)]
FIRST_SEED = 0x4ABEA221  # of a session's first develop
SLACK = 1 << 18  # tables and rounding: less than a plane of the frames below


def plane(w, h):
    return 12 * w * h


def test_grain_in_bands_released_for_the_print(engine):
    """A frame whose grain is drawn in bands holds the exposure and grain planes through the print. The frame, the
    negative, the print's output and the glare's two planes fit; with those two they do not."""
    w, h = 2048, 2100
    delta = dict(BASE, halation_active=False, glare_active=True, film_format_mm=0.009 * h)  # a pitch of 9 um
    img = sc.synthetic_image(w, h, 2)
    with engine.open(img, delta) as s:
        want = s.render("full")[0].copy()
    for planes in (5, 6, 7):
        with engine.open(img, delta) as s:
            s.set_scratch_limit(planes * plane(w, h) + SLACK)
            np.testing.assert_array_equal(s.render("full")[0], want)
            s.set_scratch_limit(0)
            negative = s.negative("full", w, h)
            np.testing.assert_array_equal(negative, s.develop_debug("full", FIRST_SEED, w, h, counts=False)[0])


@pytest.mark.parametrize("w,h,tier", [(4421, 300, "preview"), (6601, 201, "preview"), (1001, 1301, "live")])
def test_tier_image_beside_the_frame(engine, w, h, tier):
    """A tier not much smaller than the frame: the tier's image and one more plane of the frame's size fit beside the
    frame, the two filtered rows per output row together would not."""
    img = sc.synthetic_image(w, h, 3)
    delta = dict(BASE, preview_long_edge=800)
    with engine.open(img, delta) as s:
        want = s.tier_image(tier)
    np.testing.assert_array_equal(want, oracle.downscale(img, 3400 if tier == "preview" else 800))
    assert h / 2 < want.shape[0] <= h / 1.25  # a ratio that has a filter
    with engine.open(img, delta) as s:
        s.set_scratch_limit(2 * plane(w, h) + want.nbytes + SLACK)
        np.testing.assert_array_equal(s.tier_image(tier), want)


def test_mixed_components_one_at_a_time(engine):
    """Components with recursive and FIR channels: the frame, the exposure, the mixture's sum and three planes for
    one component fit, the planes of two do not."""
    w, h = 400, 300
    with engine.open(sc.synthetic_image(w, h, 2), dict(BASE, grain_active=False)) as s:
        s.set_halation(MIXED, (0.3, 0.2, 0.1))
        want, _ = s.develop_debug("full", 1, w, h, counts=False)
        s.set_scratch_limit(6 * plane(w, h) + SLACK)
        got, _ = s.develop_debug("full", 1, w, h, counts=False)
        np.testing.assert_array_equal(got, want)
        s.set_scratch_limit(5 * plane(w, h) + SLACK)
        with pytest.raises(sc.SpkError) as e:
            s.develop_debug("full", 1, w, h, counts=False)
        assert e.value.status == sc.SPK_ERR_GPU
        s.set_scratch_limit(0)
        got, _ = s.develop_debug("full", 1, w, h, counts=False)
        np.testing.assert_array_equal(got, want)
