"""The develop kernel's draws against the shared sampler (bit for bit): partial warps and blocks, pixels far
smaller and far larger than a grain (the product method in lockstep; counts beyond the log(k!) table and
beyond binary32's integers), and a film whose densities' axis has no interval guide."""

import json
import os
import shutil

import numpy as np
import pytest

import oracle
from conftest import BASE, sc

pytestmark = pytest.mark.gpu


def check_draws(counts, lam, seed):
    for c in range(3):
        for l in range(3):
            want = oracle.poisson(lam[..., c * 3 + l].ravel(), c + 10 * l, seed)
            assert np.array_equal(counts[..., c * 3 + l].ravel(), want), (c, l)


@pytest.mark.parametrize("w,h,pitch_um,couplers", [(1, 1, 24.0, False), (31, 3, 24.0, True), (33, 2, 300.0, False),
                                                   (127, 5, 1500.0, True), (800, 3, 5.0, True), (800, 3, 5.0, False),
                                                   (1601, 2, 5.2, True), (129, 2, 31.1, False)])
def test_draws_match_sampler(engine, w, h, pitch_um, couplers):
    mm = min(200.0, max(4.0, pitch_um * max(w, h) / 1000.0))
    delta = dict(BASE, film_format_mm=mm, dir_couplers_active=couplers)
    with engine.open(sc.synthetic_image(w, h, 6), delta) as s:
        counts, lam = s.develop_draws("full", 77, w, h)
    check_draws(counts, lam, 77)


def test_axis_without_guide(lib, engine, resources, tmp_path):
    """A film curve whose first two points are equal has no interval guide: the general lookup then finds the
    same lambdas, bit for bit, for every density above them."""
    folder = str(tmp_path / "resources")
    shutil.copytree(resources, folder)
    path = os.path.join(folder, "profiles", BASE["film_stock"] + ".json")
    profile = json.load(open(path))
    curves = profile["data"]["density_curves"]
    curves[1] = curves[0]
    json.dump(profile, open(path, "w"))
    img = np.maximum(sc.synthetic_image(300, 40, 8), np.float32(0.05))
    for couplers in (False, True):
        delta = dict(BASE, film_format_mm=4.0, dir_couplers_active=couplers)
        with engine.open(img, delta) as s:
            want = s.develop_draws("full", 5, 300, 40)
        with lib.engine(folder) as other, other.open(img, delta) as s:
            counts, lam = s.develop_draws("full", 5, 300, 40)
        check_draws(counts, lam, 5)
        if not couplers:  # the couplers' pre-inverted curve depends on the whole curve
            assert np.array_equal(lam, want[1]) and np.array_equal(counts, want[0])
