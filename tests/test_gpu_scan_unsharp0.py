"""The scanner's unsharp mask at a radius of 0: its sigma scales with the tier, and on a tier below about a quarter of
the frame it has a single tap. Against the float64 oracle on the tier's image, with and without a lens blur, alone and
in the batch's launches."""

import numpy as np
import pytest

import oracle
from conftest import BASE, lsb_stats, sc, setup_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(3600, 300), (5001, 165), (130, 3700), (24001, 31)])
@pytest.mark.parametrize("lens", [0.0, 0.1, 0.6, 1.5, 2.9])
def test_single_tap_mask(engine, lib, resources, w, h, lens):
    img = sc.synthetic_image(w, h, 8)
    delta = dict(BASE, grain_active=False, scanner_lens_blur=lens, preview_long_edge=800)
    with engine.open(img, delta) as s:
        got, _ = s.render("live")
        tier = s.tier_image("live")
        try:
            for plan in ("frames:1", "persistent:2048:592"):
                engine.batch_plan(plan)
                results, _ = engine.render_batch([s], "live", reprint=True)
                np.testing.assert_array_equal(results[0].pixels, got)
                results[0].free()
        finally:
            engine.batch_plan()
    th, tw = tier.shape[:2]
    rho = max(tw, th) / max(w, h)
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(tw, th))["f64"]
    assert f64["unsharp_sigma"] * rho < 1 / 6  # a radius of floor(3 sigma + 1/2) = 0
    want, _ = oracle.Oracle(f64, seed=1, rho_tier=rho).render(tier)
    st = lsb_stats(got, want)
    assert st["n_gt1"] <= 2 and st["max"] <= 2, st  # the float64 gate of the other renders
    assert (got[..., 3] == 65535).all()
