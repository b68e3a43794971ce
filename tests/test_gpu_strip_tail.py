"""The column pass's strips whose last turn leaves part of a warp without a row (three quads a row, 32 lanes), at
widths that send the sum over the strip: one component, whose sum stays in registers, and two, whose sum is in
tensor memory. Against the float64 oracle, and twice with the same bits."""

import numpy as np
import pytest

import oracle
from conftest import BASE, sc, setup_f64

pytestmark = pytest.mark.gpu

COMPS = [((1.0, 0.5, 0.25), (3.5, 4.0, 5.0)), ((0.5, 1.0, 0.75), (8.0, 8.0, 8.0))]


@pytest.mark.parametrize("w,h", [(5, 1), (6, 11), (7, 21), (9, 43), (13, 128), (21, 139)])
@pytest.mark.parametrize("n", [1, 2])
def test_partial_last_warp(engine, lib, resources, w, h, n):
    hal = (COMPS[:n], (0.3, 0.2, 0.1))
    delta = dict(BASE, grain_active=False)
    img = sc.synthetic_image(w, h, 3)
    with engine.open(img, delta) as s:
        s.set_halation(*hal)
        neg, again = (s.develop_debug("full", 1, w, h, counts=False)[0] for _ in range(2))
    np.testing.assert_array_equal(again, neg)
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(w, h))["f64"]
    _, want = oracle.Oracle(f64, seed=1, halation=hal).render(img)
    np.testing.assert_allclose(neg, want, rtol=0, atol=5e-5)  # the float64 gate of the other negatives
