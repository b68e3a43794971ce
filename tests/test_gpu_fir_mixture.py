"""The tiled FIR mixture (fir_mixture) against the float64 oracle: per-channel radii 0..9, frames at the edges
of its 32 x 32 tiles and of the smallest it takes, and its three ways to end (alone, a sum's start, a sum's
continuation)."""

import ctypes

import numpy as np
import pytest

import oracle
from conftest import BASE, sc, setup_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(32, 32), (33, 31), (31, 65), (64, 10), (10, 64), (97, 33), (9, 40)])
@pytest.mark.parametrize("sigma", [(0.2, 1.0, 2.99), (0.5, 0.7, 1.2), (2.4, 1.9, 0.0)])
def test_per_channel_fir_against_fp64(lib, w, h, sigma):
    plane = np.random.default_rng(w * 1000 + h).random((h, w, 3), dtype=np.float32) + 0.1
    out = np.zeros_like(plane)
    lib.check(lib.lib.spkx_gaussian(plane.ctypes.data_as(sc.FP), out.ctypes.data_as(sc.FP), w, h,
                                    (ctypes.c_double * 3)(*sigma)))
    want = oracle.gaussian(plane, sigma)
    assert (np.abs(out - want) / np.abs(want)).max() <= 2e-6  # the reference's tolerance (tests/test_fx.cpp:200)


COMPS = {"start": [((1.0, 0.8, 0.6), (0.6, 1.3, 2.9)), ((0.5, 0.6, 0.7), (2.2, 0.0, 0.9))],
         "continued": [((0.4, 0.5, 0.6), (3.5, 2.0, 9.0)), ((1.0, 0.8, 0.6), (0.6, 1.3, 2.9)),
                       ((0.5, 0.6, 0.7), (1.1, 1.6, 2.6)), ((0.2, 0.3, 0.4), (12.0, 14.0, 16.0))],
         "identity_first": [((1.0, 0.8, 0.6), (0.0, 0.0, 0.0)), ((0.5, 0.6, 0.7), (1.0, 1.5, 0.0))]}


@pytest.mark.parametrize("w,h", [(33, 31), (64, 96), (130, 65)])
@pytest.mark.parametrize("name", sorted(COMPS))
def test_mixture_against_fp64(engine, lib, resources, w, h, name):
    hal = (COMPS[name], (0.3, 0.2, 0.1))
    delta = dict(BASE, grain_active=False)
    img = sc.synthetic_image(w, h, 2)
    with engine.open(img, delta) as s:
        s.set_halation(*hal)
        neg, _ = s.develop_debug("full", 1, w, h, counts=False)
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(w, h))["f64"]
    _, want = oracle.Oracle(f64, seed=1, halation=hal).render(img)
    np.testing.assert_allclose(neg, want, rtol=0, atol=5e-5)  # the float64 gate of the other negatives
