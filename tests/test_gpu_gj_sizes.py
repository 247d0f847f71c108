"""Gauss-Jordan inversion at the edges of its tiles: sub-panels of 8 columns,
panels of 32 / 16 / 8, row tiles of 16, one to four rows per thread, update
stripes of 16 and 32 columns, and batches that mix sizes.

Tolerance: a backward-stable inversion's relative error is of the order of
n u cond(A) (u = 2^-53), and no less than the rounding of one complex
reciprocal (|a|^2: 1.5 u, its reciprocal: 1 u, the product: 0.5 u) on either
side of the comparison; the bar is u (n cond(A) + 6)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(negf, mats):
    dA = [negf.to_device(a) for a in mats]
    dO = [negf.dzeros(*a.shape) for a in mats]
    negf.be_inv_batched_(dA, dO)
    for a, da, o in zip(mats, dA, dO):
        ref = np.linalg.inv(a)
        err = np.linalg.norm(negf.to_host(o) - ref) / np.linalg.norm(ref)
        assert err <= 2.0 ** -53 * (a.shape[0] * np.linalg.cond(a) + 6)
        assert np.array_equal(negf.to_host(da), a)


def _mat(rng, n):
    return rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))


@pytest.mark.parametrize("n", [2, 7, 8, 9, 16, 17, 31, 33, 63, 65, 97, 111, 112, 113, 127, 129, 145, 255, 257, 399, 401,
                               513, 801, 1024])
def test_sizes(negf, n):
    rng = np.random.default_rng(n)
    _check(negf, [_mat(rng, n) for _ in range(2)])


@pytest.mark.parametrize("sizes", [[5, 112, 64, 1], [113, 8, 40, 129], [256, 31, 200], [700, 33, 512]])
def test_mixed_sizes(negf, sizes):
    rng = np.random.default_rng(sum(sizes))
    _check(negf, [_mat(rng, n) for n in sizes])


@pytest.mark.parametrize("n", [150, 330])
def test_batches_that_fill_the_gpu(negf, n):
    rng = np.random.default_rng(n)
    base = [_mat(rng, n) for _ in range(3)]
    _check(negf, [base[i % 3] for i in range(70)])


@pytest.mark.parametrize("n", [12, 100, 140])
@pytest.mark.parametrize("scale", [1e-160, 1e150])
def test_scaled(negf, n, scale):
    """|pivot|^2 outside the FP64 range."""
    rng = np.random.default_rng(n)
    a = _mat(rng, n)
    o = negf.dzeros(n, n)
    negf.be_inv_batched_([negf.to_device(a * scale)], [o])
    ref = np.linalg.inv(a)
    err = np.linalg.norm(negf.to_host(o) * scale - ref) / np.linalg.norm(ref)
    assert err <= 2.0 ** -53 * n * np.linalg.cond(a) + 2.0 ** -52


@pytest.mark.parametrize("n", [20, 100, 140, 300])
def test_singular_column(negf, n):
    """A zero column: info names it, and only the singular matrix of a batch fails."""
    import ctypes
    from libnegf_b200._lib import int_array, ptr_array, NEGF_ERR_SINGULAR
    rng = np.random.default_rng(n)
    a = _mat(rng, n)
    z = a.copy()
    z[:, n // 2] = 0.0
    dA = [negf.to_device(a), negf.to_device(z)]
    dO = [negf.dzeros(n, n), negf.dzeros(n, n)]
    info = (ctypes.c_int32 * 2)()
    rc = negf.load().negf_zinv_batched(2, int_array([n, n]), ptr_array([x.data_ptr() for x in dA]), int_array([n, n]),
                                       ptr_array([x.data_ptr() for x in dO]), int_array([n, n]), info, None)
    assert rc == NEGF_ERR_SINGULAR and info[0] == 0 and info[1] == n // 2 + 1
    ref = np.linalg.inv(a)
    assert np.linalg.norm(negf.to_host(dO[0]) - ref) <= 2.0 ** -53 * n * np.linalg.cond(a) * np.linalg.norm(ref)
