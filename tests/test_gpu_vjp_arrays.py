"""spk_render_vjp's host arrays: pageable and pinned ones, and arrays given for two of its arguments, which end as the
calls' order has them (the gradient of the loss is read first, the output written, then the gradient)."""

import numpy as np
import pytest

from conftest import BASE, sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
def test_shared_arrays(engine, pinned):
    torch = pytest.importorskip("torch")
    w, h = 257, 131

    def array(values=None):
        t = torch.zeros((h, w, 3), dtype=torch.float32, pin_memory=pinned).numpy()
        if values is not None:
            t[:] = values
        return t

    with engine.open(sc.synthetic_image(w, h, 4), dict(BASE, grain_active=True)) as s:
        s.set_halation([((0.02,) * 3, (8.0,) * 3), ((0.02,) * 3, (40.0,) * 3)], (0.02,) * 3)
        gy = np.random.default_rng(1).standard_normal((h, w, 3)).astype(np.float32)
        gx, _, y = s.render_vjp(gy, 5, want_output=True)

        def call(grad_output, grad_input, output):
            s.L.check(s.L.lib.spk_render_vjp(s.h, b"full", 5, grad_output.ctypes.data_as(sc.FP),
                                             grad_input.ctypes.data_as(sc.FP), None, 0, output.ctypes.data_as(sc.FP)))

        for _ in range(5):
            a, b, c = array(gy), array(), array()
            call(a, b, c)
            assert np.array_equal(b, gx) and np.array_equal(c, y) and np.array_equal(a, gy)
            a, b = array(gy), array()
            call(a, b, b)  # output and grad_input
            np.testing.assert_array_equal(b, gx)
            a, b = array(gy), array()
            call(a, b, a)  # grad_output and output
            assert np.array_equal(b, gx) and np.array_equal(a, y)
            a, b = array(gy), array()
            call(a, a, b)  # grad_output and grad_input
            assert np.array_equal(a, gx) and np.array_equal(b, y)
