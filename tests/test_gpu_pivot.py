"""The pivot reciprocal and the pivot search of the Gauss-Jordan kernels."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e180])
@pytest.mark.parametrize("ratio", [1.0, 1e-3, 1e9])
def test_reciprocal(negf, scale, ratio):
    """1 x 1 inverses: each part is rounded once, so the error is at most u of the
    part (u = 2^-53; 2 % for the terms below the rounding of the last addition)."""
    rng = np.random.default_rng(11)
    a = scale * (rng.standard_normal(1000) + 1j * ratio * rng.standard_normal(1000))
    dO = [negf.dzeros(1, 1) for _ in a]
    negf.be_inv_batched_([negf.to_device(np.full((1, 1), x)) for x in a], dO)
    got = np.array([negf.to_host(o)[0, 0] for o in dO])
    x, y = a.real.astype(np.longdouble), a.imag.astype(np.longdouble)
    d = x * x + y * y
    for g, r in ((got.real, x / d), (got.imag, -y / d)):
        assert np.all(np.abs(g - r) <= 1.02 * 2.0 ** -53 * np.abs(r))
