"""The tier downscale's row and column passes against the oracle's binary32 restatement, bit for bit (widths
of every remainder by 4, the mirrored edges, frames of a few rows, steep ratios), and the meter's
order statistics where whole digits of the keys coincide."""

import numpy as np
import pytest

import oracle
from conftest import BASE, sc, setup_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,L", [(1601, 1067, 1600), (1602, 33, 1600), (1603, 1, 800), (4001, 2667, 1600), (801, 5000, 800),
                                   (2400, 3, 1000), (23900, 40, 800), (32003, 85, 800)])
def test_tier_image_bit_exact(engine, w, h, L):
    img = sc.synthetic_image(w, h, 31)
    with engine.open(img, dict(BASE, preview_long_edge=L)) as s:
        got = s.tier_image("live")
    want = oracle.downscale(img, L)
    assert got.shape == want.shape
    assert np.array_equal(got, want)


@pytest.mark.parametrize("picture", ["flat", "two", "ramp", "one_pixel"])
def test_meter_order_statistics(engine, lib, resources, picture):
    w, h = (1, 1) if picture == "one_pixel" else (401, 77)
    img = np.full((h, w, 3), 0.25, np.float32)
    if picture == "two":  # half the keys equal, the rest equal to another
        img[:, w // 2:] = 0.125
    if picture == "ramp":  # neighbouring keys differ in their last digits
        img *= (1.0 + np.arange(w * h, dtype=np.float32).reshape(h, w, 1) * 2.0 ** -22)
    delta = dict(BASE, auto_exposure=True)
    with engine.open(img, delta) as s:
        got = s.meter()
    m = setup_f64(lib, resources, delta, 10.0)["f64"]["input_rgb_to_xyz"]
    want = oracle.meter(img, m)
    for k, v in want.items():
        assert got[k] == pytest.approx(v, abs=1e-9), k  # binary64 sums of 31,000 terms in another order
