"""The grain sampler on the device against its host build, bit for bit, where its branch-free operations
would leave their range: lambdas at the ends of binary32, a uniform of 1. And those operations against the compiler's."""

import ctypes

import numpy as np
import pytest

import oracle
from conftest import BASE, sc

pytestmark = pytest.mark.gpu


def device_poisson(lib, lam, stream, seed):
    lam = np.ascontiguousarray(lam, np.float32)
    out = np.zeros_like(lam)
    lib.check(lib.lib.spkx_sampler_poisson(lam.ctypes.data_as(sc.FP), out.ctypes.data_as(sc.FP), lam.size, stream, seed))
    return out


@pytest.mark.parametrize("lam", [np.inf, -np.inf, np.nan, np.finfo(np.float32).max, 1e30, 1e20, 0.0, -3.0, 1e-45, 10.0,
                                 np.nextafter(np.float32(10), np.float32(0))])
def test_lambda_at_the_ends_of_binary32(lib, lam):
    lam = np.full(4099, lam, np.float32)
    for stream, seed in ((0, 1), (21, 77)):
        np.testing.assert_array_equal(device_poisson(lib, lam, stream, seed), oracle.poisson(lam, stream, seed))


# (seed, c, l, pixel) whose draw (c, l) starts with a word of 24 leading ones: the squeeze divides by us = 0
TOP_WORDS = [(332, 1, 0, 561), (1155, 2, 1, 1383), (2857, 0, 0, 1755), (3815, 2, 2, 1706)]


@pytest.mark.parametrize("seed,c,l,pixel", TOP_WORDS)
def test_uniform_of_one(lib, engine, seed, c, l, pixel):
    """The attempt is rejected by the sampler and by the develop kernel's queue, whatever its candidate was."""
    assert int(sc.philox_np([pixel], [c + 10 * l], seed)[0]) >> 8 == 0xFFFFFF
    for lam in (10.0, 37.0, 2500.0, 1e5):
        lam = np.full(pixel + 1, lam, np.float32)
        np.testing.assert_array_equal(device_poisson(lib, lam, c + 10 * l, seed), oracle.poisson(lam, c + 10 * l, seed))
    with engine.open(sc.synthetic_image(64, 64, 6), dict(BASE, film_format_mm=4.0)) as s:
        counts, lam = s.develop_draws("full", seed, 64, 64)
    want = oracle.poisson(lam[..., 3 * c + l].ravel(), c + 10 * l, seed)
    assert lam[..., 3 * c + l].ravel()[pixel] >= 10.0
    np.testing.assert_array_equal(counts[..., 3 * c + l].ravel(), want)


RCP, SQRT, DIV, DIV_CONST = range(4)


@pytest.mark.parametrize("op,n,seed", [(RCP, 201 << 23, 0), (SQRT, 227 << 23, 0), (DIV, 1 << 31, 1), (DIV, 1 << 31, 2),
                                       (DIV_CONST, 1 << 31, 3)])
def test_operations_correctly_rounded(lib, op, n, seed):
    """The reciprocal and the root over every significand and exponent that they are used at; the quotients,
    which have two significands, over random ones and those nearest a rounding boundary."""
    wrong = ctypes.c_uint64(1)
    lib.check(lib.lib.spkx_test_sampler_ops(op, n, seed, ctypes.byref(wrong)))
    assert wrong.value == 0
