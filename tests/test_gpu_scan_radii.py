"""The scanner's register windows at every lens-blur radius (1..9: windows of 12 outputs over 36 rows and
pixels, their remainders, tiles cut by the frame's edges) against the float64 oracle, and the small prints
that run in quarter-size CTAs, at the edges of a pixel pair."""

import numpy as np
import pytest

import oracle
from conftest import BASE, lsb_stats, sc, setup_f64

pytestmark = pytest.mark.gpu


def check(engine, lib, resources, w, h, lens):
    img = sc.synthetic_image(w, h, 12)
    delta = dict(BASE, grain_active=False, scanner_lens_blur=lens)
    with engine.open(img, delta) as s:
        got, _ = s.render("full")
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(w, h))["f64"]
    want, _ = oracle.Oracle(f64, seed=1).render(img)
    st = lsb_stats(got, want)
    assert st["n_gt1"] <= 2 and st["max"] <= 2, st  # the float64 gate of the other renders
    assert (got[..., 3] == 65535).all()


@pytest.mark.parametrize("lens", [0.3, 0.6, 0.9, 1.2, 1.5, 1.9, 2.2, 2.5, 2.9])
@pytest.mark.parametrize("w,h", [(45, 37), (32, 64), (97, 33)])
def test_lens_radii(engine, lib, resources, w, h, lens):
    check(engine, lib, resources, w, h, lens)


@pytest.mark.parametrize("w,h", [(16, 16), (17, 15), (255, 1), (257, 1), (513, 3)])
def test_small_prints(engine, lib, resources, w, h):
    check(engine, lib, resources, w, h, 0.0)
