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


@pytest.mark.parametrize("n", [2, 40, 100, 140, 300])
@pytest.mark.parametrize("tiny", [5e-324, 1e-320, 1e-312])
def test_tiny_pivot_is_not_zero(negf, n, tiny):
    """A column of zeros and one subnormal entry has a pivot; its reciprocal
    overflows, so the call may fail in a later column, but not in this one."""
    from libnegf_b200._lib import int_array, ptr_array
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    a[:, 0] = 0.0
    a[n // 2, 0] = tiny
    d, o, info = negf.to_device(a), negf.dzeros(n, n), (ctypes.c_int32 * 1)()
    negf.load().negf_zinv_batched(1, int_array([n]), ptr_array([d.data_ptr()]), int_array([n]), ptr_array([o.data_ptr()]),
                                  int_array([n]), info, None)
    assert info[0] != 1
    assert info[0] > 1 or not np.isfinite(negf.to_host(o)).all()
