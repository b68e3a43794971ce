"""The column pass with two and with three strips an SM (three where a short frame has more than two for every SM, 296
strips of 4 pixels on a whole B200), against the float64 oracle: both sides of the rule's lines in width and height,
widths whose last strip is cut, one to three components."""

import numpy as np
import pytest

import oracle
from conftest import BASE, sc, setup_f64

pytestmark = pytest.mark.gpu

COMPS = [((1.0, 0.5, 0.25), (3.5, 4.0, 5.0)), ((0.5, 1.0, 0.75), (8.0, 8.0, 8.0)), ((0.25, 0.5, 1.0), (40.0, 30.0, 20.0))]


@pytest.mark.parametrize("w,h,n", [(1184, 3, 2), (1185, 3, 1), (1186, 7, 3), (1187, 64, 2), (1200, 257, 3), (1189, 500, 1),
                                   (1189, 501, 1), (1188, 1100, 2), (1188, 1101, 2), (2403, 130, 3)])
def test_strips_against_fp64(engine, lib, resources, w, h, n):
    hal = (COMPS[:n], (0.3, 0.2, 0.1))
    delta = dict(BASE, grain_active=False)
    img = sc.synthetic_image(w, h, 7)
    with engine.open(img, delta) as s:
        s.set_halation(*hal)
        neg, _ = s.develop_debug("full", 1, w, h, counts=False)
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(w, h))["f64"]
    _, want = oracle.Oracle(f64, seed=1, halation=hal).render(img)
    np.testing.assert_allclose(neg, want, rtol=0, atol=5e-5)  # the float64 gate of the other negatives
