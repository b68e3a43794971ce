"""Renders when device memory is short: where a faster path takes more scratch than the one it replaced, the call
falls back to that one and gives the same bits. The session's limit stands in for a device without more memory."""

import numpy as np
import pytest

from conftest import BASE, sc

pytestmark = pytest.mark.gpu

MIXED = [((0.1, 0.2, 0.3), (3.0 + 0.5 * k, 0.4 * k + 0.3, 4.0)) for k in range(6)]
SLACK = 1 << 18  # tables and rounding: less than a plane of the frames below


def plane(w, h):
    return 12 * w * h


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
