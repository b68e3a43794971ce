"""The print kernel's CTA sizes: a small frame printed alone takes quarter-size CTAs, beside others in a batch full ones.
The pixels are those of a reprint either way, at sizes around a CTA's and around the rule's line."""

import numpy as np
import pytest

from conftest import BASE, sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(7, 9), (33, 31), (128, 4), (131, 97), (333, 250), (391, 194), (640, 460), (641, 473)])
def test_batch_matches_reprint(engine, w, h):
    sessions = [engine.open(sc.synthetic_image(w, h, i), BASE) for i in range(4)]
    try:
        want = [s.render("full")[0].copy() for s in sessions]
        for plan in ("frames:1", "frames:2", "frames:4"):
            engine.batch_plan(plan)
            results, info = engine.render_batch(sessions, "full", reprint=True)
            assert info["plan"] == plan
            for r, x in zip(results, want):
                np.testing.assert_array_equal(r.pixels, x)
                r.free()
    finally:
        engine.batch_plan()
        for s in sessions:
            s.close()
