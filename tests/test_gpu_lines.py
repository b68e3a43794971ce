"""The recursive blur's line kernels (k_iir_h, k_iir_v), which take the frames and channels that the
block-parallel kernels do not, against the float64 oracle: sizes at the edges of the row pass's 10-row,
32-pixel chunks and of the column pass's 16-row chunks, and the accumulating modes of the column pass on
lines too long for shared memory."""

import ctypes

import numpy as np
import pytest

import oracle
from conftest import BASE, sc, setup_f64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(9, 31), (10, 32), (11, 33), (16, 64), (17, 65), (15, 96), (31, 97), (1, 33), (33, 1),
                                   (160, 129)])
@pytest.mark.parametrize("sigma", [(2.5, 8.0, 0.0), (3.5, 0.3, 40.0)])
def test_mixed_channels_against_fp64(lib, shape, sigma):
    h, w = shape
    plane = np.random.default_rng(h * 1000 + w).random((h, w, 3), dtype=np.float32) + 0.1
    out = np.zeros_like(plane)
    lib.check(lib.lib.spkx_gaussian(plane.ctypes.data_as(sc.FP), out.ctypes.data_as(sc.FP), w, h,
                                    (ctypes.c_double * 3)(*sigma)))
    err = np.abs(out - oracle.gaussian(plane, sigma))
    for c in range(3):
        # the reference's relative tolerances (tests/test_fx.cpp:200) of values up to 1.1
        assert err[..., c].max() <= (1e-5 if sigma[c] >= 3 else 2e-6) * 1.1, (c, err[..., c].max())


@pytest.mark.parametrize("w,h", [(7, 5000), (20003, 3)])
def test_long_lines_mixture_against_fp64(engine, lib, resources, w, h):
    """A two-component halation on a frame whose lines exceed shared memory: the column pass starts the
    mixture's sum with the first component and adds the second."""
    hal = ([((1.0, 0.5, 0.25),) + ((8, 8, 8),), ((0.5, 1.0, 0.75),) + ((40, 40, 40),)], (0.3, 0.2, 0.1))
    delta = dict(BASE, grain_active=False, film_format_mm=200.0)
    img = sc.synthetic_image(w, h, 4)
    with engine.open(img, delta) as s:
        s.set_halation(*hal)
        neg, _ = s.develop_debug("full", 1, w, h, counts=False)
    f64 = setup_f64(lib, resources, delta, 200000.0 / max(w, h))["f64"]
    _, want = oracle.Oracle(f64, seed=1, halation=hal).render(img)
    np.testing.assert_allclose(neg, want, rtol=0, atol=5e-5)  # the float64 gate of the other negatives


@pytest.mark.parametrize("w,h", [(4, 1), (5, 42), (6, 43), (7, 128), (8, 129), (12, 171), (33, 700), (130, 257), (64, 2560)])
def test_block_mixture_against_fp64(engine, lib, resources, w, h):
    """The block-parallel mixture of three recursive components: strips cut by the frame's edge, frames whose
    rows are not aligned, and the edges of the sum's turns of 128 quads in tensor memory."""
    hal = ([((1.0, 0.5, 0.25), (3.5, 4.0, 5.0)), ((0.5, 1.0, 0.75), (8, 8, 8)), ((0.25, 0.5, 1.0), (40, 30, 20))],
           (0.3, 0.2, 0.1))
    delta = dict(BASE, grain_active=False)
    img = sc.synthetic_image(w, h, 9)
    with engine.open(img, delta) as s:
        s.set_halation(*hal)
        neg, _ = s.develop_debug("full", 1, w, h, counts=False)
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(w, h))["f64"]
    _, want = oracle.Oracle(f64, seed=1, halation=hal).render(img)
    np.testing.assert_allclose(neg, want, rtol=0, atol=5e-5)  # the float64 gate of the other negatives


MIXED = {"run_first": [((0.4, 0.5, 0.6), (3.5, 2.0, 9.0)), ((0.2, 0.3, 0.4), (12.0, 14.0, 16.0)),
                       ((0.5, 0.4, 0.3), (0.0, 5.0, 0.0))],
         "run_after_fir": [((1.0, 0.8, 0.6), (0.6, 1.3, 2.9)), ((0.5, 0.4, 0.3), (0.0, 5.0, 1.1)),
                           ((0.4, 0.5, 0.6), (3.5, 2.0, 9.0)), ((0.2, 0.3, 0.4), (0.7, 0.8, 0.9))],
         "most": [((0.1, 0.2, 0.3), (3.0 + 0.5 * k, 0.4 * k, 4.0)) for k in range(8)]}


@pytest.mark.parametrize("w,h", [(31, 33), (42, 64), (200, 97)])
@pytest.mark.parametrize("name", sorted(MIXED))
def test_joined_line_passes_against_fp64(engine, lib, resources, w, h, name):
    """Components with recursive and FIR channels side by side: their line passes share launches."""
    hal = (MIXED[name], (0.3, 0.2, 0.1))
    delta = dict(BASE, grain_active=False)
    img = sc.synthetic_image(w, h, 2)
    with engine.open(img, delta) as s:
        s.set_halation(*hal)
        neg, _ = s.develop_debug("full", 1, w, h, counts=False)
    f64 = setup_f64(lib, resources, delta, 35000.0 / max(w, h))["f64"]
    _, want = oracle.Oracle(f64, seed=1, halation=hal).render(img)
    np.testing.assert_allclose(neg, want, rtol=0, atol=5e-5)  # the float64 gate of the other negatives
